"""A Linear's forward and backward pass in one call of the extension each, against the same pass op by op: the same bits and the same
refusals over types, grids, token counts, orders, gradient formats and recipes, with the weight prepared or not."""
import pytest
import torch

from pratchya_b200 import _lib
from pratchya_b200._nnx_impl import _module
from pratchya_b200._qualia import _ops

pytestmark = pytest.mark.gpu


class _OpByOp:
    """The extension with the two calls declining."""
    def __init__(self, native):
        self.native = native

    def __getattr__(self, name):
        return (lambda *args: None) if name in ("linear_forward", "linear_backward") else getattr(self.native, name)


def _both(monkeypatch, f):
    native = _lib.native()

    def outcome():
        try:
            return f()
        except Exception as e:                       # noqa: BLE001 -- the kind of refusal is what is compared
            return type(e)
    mine = outcome()
    monkeypatch.setattr(_lib, "_native", _OpByOp(native))
    text = outcome()
    monkeypatch.setattr(_lib, "_native", native)
    return mine, text


def _same(a, b):
    if isinstance(a, tuple):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if isinstance(a, torch.Tensor):
        return a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b)
    return a is b


@pytest.mark.parametrize("shape,n,grid,fake", [((64, 1024), 512, (128, 128), True), ((1000, 512), 1024, (128, 128), True), ((1024, 1024), 1024, (128, 128), True), ((2048, 256), 640, (128, 128), True),
                                               ((2, 1024, 512), 2048, (128, 128), True), ((1024, 512), 384, (128, 128), False), ((8, 1024), 128, (128, 1), False), ((8, 1024), 128, (128, 1), True), ((704, 128), 1024, (128, 1), False),
                                               ((7, 1024), 48, (128, 1), False), ((5, 384), 128, (128, 128), True), ((3, 8, 256), 256, (64, 64), True), ((16, 1000), 128, (128, 128), True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("how", ["plain", "strided x", "strided gradient", "e5m2", "reference", "prepared", "tf32", "bf16 weight"])
def test_training_step_in_two_calls_gives_the_bits_of_its_ops(built_lib, monkeypatch, shape, n, grid, fake, dtype, how):
    g = torch.Generator(device="cuda").manual_seed(shape[-1] + n)
    k = shape[-1]
    base = torch.randn(*shape[:-1], 2 * k, generator=g, device="cuda").to(dtype)
    x = (base[..., ::2] if how == "strided x" else base[..., :k].contiguous()).detach().requires_grad_(True)
    w = (torch.randn(k, n, generator=g, device="cuda") * 0.02).to(torch.bfloat16 if how == "bf16 weight" else torch.float32).requires_grad_(True)
    gy = torch.randn(*shape[:-1], 2 * n, generator=g, device="cuda") * 1e-3
    gy = gy[..., ::2] if how == "strided gradient" else gy[..., :n].contiguous()
    options = dict(fake_quant_output=fake, grad_format="e5m2" if how == "e5m2" else "e4m3", recipe="reference" if how == "reference" else "fp8")

    def step():
        y = _module.linear_fp8(x, w, grid, prepared={} if how == "prepared" else None, **options)
        return (y.detach(), *torch.autograd.grad(y, (x, w), gy.to(y.dtype)))
    if how == "tf32":
        _ops.set_literal_dot_precision("tf32")
    try:
        mine, text = _both(monkeypatch, step)
    finally:
        _ops.set_literal_dot_precision("f32")
    assert _same(mine, text), (mine, text)


@pytest.mark.parametrize("grid,n,fake", [((128, 128), 512, True), ((128, 1), 48, False)])
def test_a_gradient_format_that_nothing_is_stored_in_is_not_asked_for(built_lib, grid, n, fake):
    """The literal dots store no gradient in fp8: what `grad_format` says is not read there, and refused where it is."""
    x, w = torch.randn(64, 1024, device="cuda", requires_grad=True), (torch.randn(1024, n, device="cuda") * 0.02).requires_grad_(True)
    step = lambda x, fmt: torch.autograd.grad(_module.linear_fp8(x, w, grid, fake_quant_output=fake, grad_format=fmt).sum(), (x, w))
    assert all(torch.equal(a, b) for a, b in zip(step(x, "none"), step(x, "e4m3")))
    if grid == (128, 128):
        with pytest.raises(KeyError):
            step(torch.randn(1024, 1024, device="cuda", requires_grad=True), "none")


class _Counting:
    """The extension, with what its two calls were asked and answered."""
    def __init__(self, native):
        self.native, self.taken, self.left = native, [], []

    def __getattr__(self, name):
        call = getattr(self.native, name)
        if name not in ("linear_forward", "linear_backward"):
            return call

        def counted(*args):
            out = call(*args)
            (self.left if out is None else self.taken).append(name)
            return out
        return counted


def _training_step(x, w, grid, fake, **options):
    y = _module.linear_fp8(x, w, grid, fake_quant_output=fake, **options)
    return (y.detach(), *torch.autograd.grad(y, (x, w), torch.ones_like(y) * 1e-3))


BOTH = ["linear_forward", "linear_backward"]


@pytest.mark.parametrize("rows,k,n,grid,fake,dtype,taken", [
    (64, 1024, 512, (128, 128), True, torch.float32, BOTH), (1000, 512, 1024, (128, 128), True, torch.bfloat16, BOTH), (1024, 1024, 1024, (128, 128), True, torch.bfloat16, BOTH),
    (1024, 512, 384, (128, 128), False, torch.float32, BOTH), (704, 128, 1024, (128, 1), False, torch.float32, BOTH), (7, 1024, 48, (128, 1), False, torch.float32, BOTH),
    (5, 384, 128, (128, 128), True, torch.float32, []), (24, 256, 256, (64, 64), True, torch.float32, []), (64, 1024, 512, (128, 128), True, torch.float16, [])])
def test_which_steps_the_calls_take(built_lib, monkeypatch, rows, k, n, grid, fake, dtype, taken):
    counting = _Counting(_lib.native())
    monkeypatch.setattr(_lib, "_native", counting)
    x, w = torch.randn(rows, k, device="cuda").to(dtype).requires_grad_(True), (torch.randn(k, n, device="cuda") * 0.02).requires_grad_(True)
    _training_step(x, w, grid, fake)
    assert counting.taken == taken


@pytest.mark.parametrize("rows,k,n,grid,fake,dtype", [(600, 1024, 1024, (128, 128), True, torch.bfloat16), (1024, 512, 1024, (128, 128), True, torch.float32), (704, 128, 1024, (128, 1), False, torch.float32)])
def test_the_calls_under_hooks_on_another_stream_and_in_a_graph(built_lib, monkeypatch, rows, k, n, grid, fake, dtype):
    counting = _Counting(_lib.native())
    monkeypatch.setattr(_lib, "_native", counting)
    xs = [torch.randn(rows, k, device="cuda").to(dtype).requires_grad_(True) for _ in range(3)]
    w = (torch.randn(k, n, device="cuda") * 0.02).requires_grad_(True)
    want = [_training_step(x, w, grid, fake) for x in xs]
    packed = []

    def pack(t):
        packed.append(t)
        return t.cpu()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        got = _training_step(xs[0], w, grid, fake)
    assert _same(got, want[0]) and len(packed) == (11 if fake and rows % 1024 == 0 else 8 if fake else 6)      # x's triple, the weight's, x^T's, the output's scales
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = [_training_step(x, w, grid, fake) for x in xs]
    torch.cuda.current_stream().wait_stream(side)
    assert all(_same(a, b) for a, b in zip(got, want))
    static = xs[0].detach().clone().requires_grad_(True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _training_step(static, w, grid, fake)
    for x, ref in zip(xs, want):
        with torch.no_grad():
            static.copy_(x)
        graph.replay()
        assert _same(out, ref)
    assert not counting.left
