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
