"""The extension's whole ops (csrc/native.cc) against the Python text they stand in for: the same bits for what they take, and the
same answer for what they leave to it; and the ops that run without their autograd.Function where no derivative can be asked for."""
import pytest
import torch
from torch.autograd import forward_ad

from pratchya_b200 import _lib
from pratchya_b200._nnx_impl import _glue, _module
from pratchya_b200._nnx_impl._nograph import no_graph
from pratchya_b200._qualia import _ops
from pratchya_b200._qualia._qarr import QArrayImpl

pytestmark = pytest.mark.gpu

WHOLE = {"quantize", "quantize_transposed", "dequantize", "dequantize_bwd", "fake_quantize", "transpose_bytes", "gemm", "linear", "linear_step", "dense_dot"}


class _PythonOnly:
    """The extension with every whole op declining."""
    def __getattr__(self, name):
        return (lambda *args: None) if name in WHOLE else getattr(_REAL, name)


_REAL = None


@pytest.fixture
def both(monkeypatch):
    """both(f): f() with the extension and f() with the Python text."""
    global _REAL
    _REAL = _lib.native()

    def run(f):
        def outcome():
            try:
                return f()
            except Exception as e:                       # noqa: BLE001 -- the kind of refusal is what is compared
                return type(e)
        mine = outcome()
        monkeypatch.setattr(_lib, "_native", _PythonOnly())
        text = outcome()
        monkeypatch.setattr(_lib, "_native", _REAL)
        return mine, text
    return run


def _same(a, b):
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if isinstance(a, torch.Tensor):
        return (isinstance(b, torch.Tensor) and a.shape == b.shape and a.dtype == b.dtype and a.device == b.device and a.stride() == b.stride()
                and a.requires_grad == b.requires_grad
                and torch.equal(a.contiguous().flatten().view(torch.uint8), b.contiguous().flatten().view(torch.uint8)))
    return a == b


def _inputs():
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    base = r(256, 1024)
    yield "f32", base
    yield "bf16", base.bfloat16()
    yield "f64", base.double()
    yield "half", base.half()
    yield "transposed", r(1024, 256).t()
    yield "strided", r(256, 2048)[:, ::2]
    yield "off alignment", r(256 * 1024 + 1)[1:].view(256, 1024)
    yield "leading dims", r(2, 3, 128, 256)
    yield "one dim", r(1024)
    yield "no dim", r(())
    yield "empty", r(0, 128)
    yield "empty lead", r(0, 128, 128)
    yield "one row", r(1, 128)
    yield "expanded", r(1, 1024).expand(128, 1024)
    yield "conjugate view", torch.randn(128, 128, dtype=torch.complex64, device="cuda").conj().imag
    yield "parameter", torch.nn.Parameter(base)
    yield "cpu", torch.zeros(128, 128)
    yield "indivisible", r(100, 130)


@pytest.mark.parametrize("grid", [(1, 128), (128, 128), (128, 1), (16, 16), (1, 1), (0, 128), (1.0, 128.0)])
def test_quantizers_answer_alike(built_lib, both, grid):
    for name, x in _inputs():
        for f in (lambda: _ops.quantize_impl(x, grid), lambda: _ops.quantize_impl(x, grid, "e5m2"), lambda: _ops.quantize_transposed_impl(x, 128),
                  lambda: _ops.fake_quantize_impl(x, grid, torch.float32), lambda: _ops.fake_quantize_impl(x, grid, torch.bfloat16),
                  lambda: _ops.fake_quantize_impl(x, grid, torch.float16), lambda: _ops.fake_quantize_scales_impl(x, grid, torch.float32),
                  lambda: _ops.dequantize_impl(*_ops.quantize_impl(x, grid), torch.bfloat16, grid),
                  lambda: _ops.dequantize_impl(*_ops.quantize_impl(x, grid), torch.float64, grid),
                  lambda: _ops.dequantize_impl(*_ops.quantize_impl(x, (1, 1)), torch.float32, grid),          # scales of another grid
                  lambda: _ops.dequantize_impl_bwd(*_ops.quantize_impl(x, grid)[1:], x, grid)):
            mine, text = both(f)
            assert _same(mine, text), (name, grid, mine, text)


def test_products_answer_alike(built_lib, both):
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    for m, k, n, grid, lead in [(256, 1024, 512, (128, 128), ()), (8, 1024, 256, (128, 128), ()), (64, 128, 48, (128, 1), (2, 3)), (3, 128, 128, (128, 128), ()), (40, 256, 24, (128, 1), ())]:
        x, w, dy = r(*lead, m, k), r(k, n) * 0.02, r(m, n)
        for f in (lambda: _ops.matmul_impl(*_ops.quantize_impl(x, (1, 128)), *_ops.quantize_impl(w, grid), (1, 128), grid),
                  lambda: _ops.matmul_impl(*_ops.quantize_impl(x, (1, 128)), *_ops.quantize_impl(w, grid), (1, 128), grid, out_dtype=torch.bfloat16),
                  lambda: _ops.transpose_bytes(_ops.quantize_impl(w, grid)[0]),
                  lambda: _ops.literal_dots(_ops.quantize_impl(x.reshape(-1, k)[:m], (1, 128)), _ops.quantize_impl(w, grid), (1, 128), grid, dy),
                  lambda: _module.Linear(k, n, grid, kernel=w)(x), lambda: _module.Linear(k, n, grid, kernel=w)(x.bfloat16())):
            mine, text = both(f)
            assert _same(mine, text), (m, k, n, grid)


@pytest.mark.parametrize("grid", [(128, 128), (128, 1)])
@pytest.mark.parametrize("fake", [True, False])
def test_a_linear_without_a_graph_gives_the_bits_of_one_with_it(built_lib, both, grid, fake):
    g = torch.Generator(device="cuda").manual_seed(5)
    w = (torch.randn(1024, 512, generator=g, device="cuda") * 0.02).requires_grad_(True)
    for x in (torch.randn(256, 1024, generator=g, device="cuda"), torch.randn(2, 40, 1024, generator=g, device="cuda"), torch.randn(7, 1024, generator=g, device="cuda").bfloat16(),
              torch.randn(1024, 64, generator=g, device="cuda").t()):
        f = lambda: _module.linear_fp8(x, w, grid, fake_quant_output=fake)
        graph = f()
        assert graph.requires_grad
        with torch.no_grad():
            mine, text = both(f)
            keep = {}
            kept = [_module.linear_fp8(x, w, grid, fake_quant_output=fake, prepared=keep) for _ in range(2)]
        assert not mine.requires_grad and torch.equal(mine, graph.detach()) and torch.equal(text, mine) and mine.dtype == graph.dtype
        assert all(torch.equal(k, mine) for k in kept) and set(keep) == {"wq", "w_t"}


@pytest.mark.parametrize("grid", [(2 ** 32 + 1, 128), (1, 2 ** 32 + 128), (2 ** 64 + 1, 128), (-1, 128), (1, -(2 ** 32) + 128)])
def test_block_sizes_beyond_an_int_are_refused(built_lib, both, grid):
    """Block sizes whose low 32 bits are (1, 128) divide no array."""
    x = torch.randn(8, 1024, device="cuda")
    triple = _ops.quantize_impl(x, (1, 128))
    for f in (lambda: _ops.quantize_impl(x, grid), lambda: _ops.quantize_transposed_impl(x.repeat(16, 1), grid[1]) if grid[1] != 128 else ValueError,
              lambda: _ops.fake_quantize_impl(x, grid, torch.float32), lambda: _ops.fake_quantize_scales_impl(x, grid, torch.float32),
              lambda: _ops.dequantize_impl(*triple, torch.float32, grid)):
        mine, text = both(f)
        assert mine is text and isinstance(mine, type) and issubclass(mine, Exception), (grid, mine, text)


@pytest.mark.parametrize("prepared", [False, True])
def test_a_linear_without_a_graph_prepares_its_weight_once(built_lib, monkeypatch, prepared):
    """The calls that the extension leaves to the Python text, too: one quantization of the weight, and no byte transpose that no product reads."""
    g = torch.Generator(device="cuda").manual_seed(6)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    calls = []
    for name in ("quantize_impl", "transpose_bytes"):
        monkeypatch.setattr(_ops, name, lambda t, *args, _f=getattr(_ops, name), _n=name: (calls.append((_n, t.shape)), _f(t, *args))[1])
    for w, grid, x, fake, turned in [
            (r(1024, 128), (128, 1), r(64, 1024), True, 1), (r(1024, 128), (128, 1), r(64, 1024), False, 1), (r(1024, 512), (128, 128), r(1024, 64).t(), True, 1),
            (r(1024, 512), (128, 128), r(64, 1024).bfloat16(), False, 1), (r(1024, 512), (128, 128), r(64, 1024).half(), True, 1), (r(1024, 512), (128, 128), r(64, 1024), True, 1),
            (r(128, 256), (128, 128), r(3, 128), True, 0), (r(1024, 24), (128, 1), r(64, 1024), True, 0), (r(256, 256), (16, 16), r(64, 256), True, 0)]:
        keep = {} if prepared else None
        with torch.no_grad():
            for again in (False, True):
                calls.clear()
                _module.linear_fp8(x, w, grid, fake_quant_output=fake, prepared=keep)
                n = 0 if again and prepared else 1
                assert sum(name == "quantize_impl" and shape == w.shape for name, shape in calls) == n, (tuple(w.shape), grid, calls)
                assert sum(name == "transpose_bytes" for name, _ in calls) == n * turned, (tuple(w.shape), grid, calls)


def test_ops_keep_their_function_where_a_derivative_can_be_asked_for(built_lib):
    x, w = torch.randn(8, 1024, device="cuda"), torch.randn(1024, 256, device="cuda") * 0.02
    scale = torch.ones(1024, device="cuda")
    assert not no_graph()
    with torch.no_grad():
        assert no_graph()
        assert not torch.vmap(lambda t: torch.ones_like(t) * no_graph())(x[:, 0]).any()
        with forward_ad.dual_level():
            assert not no_graph()
            dual = forward_ad.make_dual(x, torch.ones_like(x))
            for f in (lambda: _module.linear_fp8(dual, w), lambda: _glue.rms_norm(dual, scale, 1e-6)):
                with pytest.raises((RuntimeError, NotImplementedError)):      # no forward-mode rule: refused, not dropped
                    f()
        seen = []
        torch.jit.trace(lambda t: (seen.append(no_graph()), t + 1)[1], torch.zeros(1), check_trace=False)
        assert seen == [False]
    assert torch.equal(_glue.rms_norm(x, scale, 1e-6), _no_grad(lambda: _glue.rms_norm(x, scale, 1e-6)))


def _no_grad(f):
    with torch.no_grad():
        return f()


def test_statuses_and_arguments_raise(built_lib):
    nat = _lib.native()
    x = torch.zeros(4, 128, device="cuda")
    with pytest.raises(_lib.PbError):
        nat.pb_relu2(x, 3, x)                             # no multiple of 4
    with pytest.raises(TypeError):
        nat.pb_relu2(x, 4)
    with pytest.raises(TypeError):
        nat.pb_relu2(x, "4", x)
    with pytest.raises(ValueError):
        QArrayImpl(torch.zeros(4, 130, device="cuda"), (1, 128))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):                         # the current stream, not the default one
        a = _ops.quantize_impl(torch.ones(64, 1024, device="cuda"), (1, 128))
    side.synchronize()
    assert _same(a, _ops.quantize_impl(torch.ones(64, 1024, device="cuda"), (1, 128)))
