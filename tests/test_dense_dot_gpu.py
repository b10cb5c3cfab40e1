"""pb_dense_dot (an fp8 triple against a dense f32 cotangent) against 64-bit products of the dequantized operands: tiles with one row
or column, a contraction shorter than a stage, parts of it on several CTAs, and every grid it takes."""
import pytest
import torch

from pratchya_b200 import _lib
from pratchya_b200._qualia import _ops
from pratchya_b200._qualia import dequantize_impl, quantize_impl

pytestmark = pytest.mark.gpu


def _bound(a, b):
    """Per element: |a| @ |b| times the roundings an f32 dot of this kernel can make -- one of the scaled operand (2^-24; the three
    bf16 terms keep it to 2^-26), the tensor core's within 32 of the contraction (six additions of at most 2^-23) and one
    addition per 32 of it."""
    depth = a.shape[1]
    return (a.abs() @ b.abs()) * 2.0 ** -24 * (14 + (depth + 31) // 32)


@pytest.mark.parametrize("m,k,n,grid", [(1, 128, 16, (128, 1)), (5, 128, 128, (128, 128)), (129, 256, 48, (128, 1)), (64, 1024, 2048, (128, 1)),
                                        (31, 128, 1024, (128, 128)), (130, 384, 640, (128, 128)), (1000, 2048, 128, (128, 1)), (3000, 128, 256, (128, 1))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dense_dot_matches_64_bits(built_lib, m, k, n, grid, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(m, k, generator=g, device="cuda") * torch.randn(1, k, generator=g, device="cuda").exp()
    w = torch.randn(k, n, generator=g, device="cuda") * 0.02
    dy = torch.randn(m, n, generator=g, device="cuda") * torch.randn(m, 1, generator=g, device="cuda").exp() * 1e-3
    dy[0, 0] = 0.0
    dy = dy.to(dtype)
    xq, wq = quantize_impl(x, (1, 128)), quantize_impl(w, grid)
    xh, wh = dequantize_impl(*xq, torch.float32, (1, 128)).double(), dequantize_impl(*wq, torch.float32, grid).double()
    gx, gw = _ops.literal_dots(xq, wq, (1, 128), grid, dy)
    assert gx.shape == (m, k) and gw.shape == (k, n)
    dy64 = dy.double()
    assert ((gx.double() - dy64 @ wh.t()).abs() <= _bound(dy64, wh.t()) + 1e-30).all()
    assert ((gw.double() - xh.t() @ dy64).abs() <= _bound(xh.t(), dy64) + 1e-30).all()
    again = _ops.literal_dots(xq, wq, (1, 128), grid, dy)
    assert torch.equal(gx, again[0]) and torch.equal(gw, again[1])
    assert built_lib.pb_gemm_check(torch.cuda.current_stream().cuda_stream) == 0


def test_infinities_and_nans_spread_as_in_an_f32_dot(built_lib):
    xq, wq = quantize_impl(torch.ones(64, 128, device="cuda"), (1, 128)), quantize_impl(torch.ones(128, 128, device="cuda"), (128, 128))
    dy = torch.ones(64, 128, device="cuda")
    dy[3, 5], dy[9, 7] = float("inf"), float("nan")
    gx, gw = _ops.literal_dots(xq, wq, (1, 128), (128, 128), dy)
    assert torch.isinf(gx[3]).all() and torch.isnan(gx[9]).all() and torch.isfinite(gx[[r for r in range(64) if r not in (3, 9)]]).all()
    assert torch.isinf(gw[:, 5]).all() and torch.isnan(gw[:, 7]).all() and torch.isfinite(gw[:, :5]).all()


def _f32_dot_bound(a, b):
    """As _bound for sums made one f32 product after the other: two roundings of the operand and one addition each, of numbers that
    may be subnormal (2^-149)."""
    return (a.abs() @ b.abs()) * 2.0 ** -24 * (a.shape[1] + 4) + a.shape[1] * 2.0 ** -149


@pytest.mark.parametrize("x_amp,w_amp,g_amp", [(1.0, 0.02, 1e-32), (1.0, 0.02, 1e-35), (1.0, 0.02, 1e-38), (1e-4, 1e-4, 1e-32), (1e-37, 1e-37, 1.0), (1e-30, 1e-30, 1e30),
                                               (1.0, 0.02, 1e34)])
@pytest.mark.parametrize("m,k,n,grid", [(130, 384, 640, (128, 128)), (300, 1024, 48, (128, 1))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cotangents_and_scales_far_from_one(built_lib, x_amp, w_amp, g_amp, m, k, n, grid, dtype):
    """Cotangents, scales or both at the ends of the f32 range: as an f32 dot."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x, w = torch.randn(m, k, generator=g, device="cuda") * x_amp, torch.randn(k, n, generator=g, device="cuda") * w_amp
    dy = (torch.randn(m, n, generator=g, device="cuda") * g_amp).to(dtype)
    dy[5] = 0.0
    xq, wq = quantize_impl(x, (1, 128)), quantize_impl(w, grid)
    xh, wh = dequantize_impl(*xq, torch.float32, (1, 128)).double(), dequantize_impl(*wq, torch.float32, grid).double()
    gx, gw = _ops.literal_dots(xq, wq, (1, 128), grid, dy)
    dy64 = dy.double()
    assert ((gx.double() - dy64 @ wh.t()).abs() <= _f32_dot_bound(dy64, wh.t())).all()
    assert ((gw.double() - xh.t() @ dy64).abs() <= _f32_dot_bound(xh.t(), dy64)).all()


def test_products_that_are_finite_though_the_scaled_cotangent_is_not(built_lib):
    """3e38 against a block of amplitude 300: the block's small values make finite products, its large ones infinities."""
    m, k, n = 64, 256, 128
    w = torch.full((k, n), 1e-3, device="cuda")
    w[7] = 300.0                                         # one row of dX's columns in either block row
    w[200] = -300.0
    x = torch.full((m, k), 1e-3, device="cuda")
    x[:, 9] = 300.0
    dy = torch.zeros(m, n, device="cuda")
    dy[3, 5], dy[11, 6], dy[20, 100] = 3e38, -3.39e38, 1.0
    xq, wq = quantize_impl(x, (1, 128)), quantize_impl(w, (128, 128))
    xh, wh = dequantize_impl(*xq, torch.float32, (1, 128)).double(), dequantize_impl(*wq, torch.float32, (128, 128)).double()
    gx, gw = _ops.literal_dots(xq, wq, (1, 128), (128, 128), dy)
    for got, a, b in ((gx, dy.double(), wh.t()), (gw, xh.t(), dy.double())):
        want = a @ b
        finite = want.abs() < 3.3e38
        assert finite.any() and (~finite).any()
        assert ((got.double() - want).abs() <= _f32_dot_bound(a, b))[finite].all() and torch.isinf(got[~finite]).all()


def test_other_shapes_take_the_library_route(built_lib):
    """A width that is no multiple of 16, a grid the kernel does not take, a cotangent off the 16-byte alignment."""
    for m, k, n, gx_, gw_ in [(32, 64, 24, (1, 64), (64, 1)), (32, 128, 24, (1, 128), (128, 1)), (32, 128, 128, (1, 128), (128, 128))]:
        x, w = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
        dy = torch.randn(m * n + 1, device="cuda")[1:].view(m, n)
        xq, wq = quantize_impl(x, gx_), quantize_impl(w, gw_)
        gx, gw = _ops.literal_dots(xq, wq, gx_, gw_, dy)
        xh, wh = dequantize_impl(*xq, torch.float32, gx_).double(), dequantize_impl(*wq, torch.float32, gw_).double()
        assert (gx.double() - dy.double() @ wh.t()).abs().max() <= 1e-4 and (gw.double() - xh.t() @ dy.double()).abs().max() <= 1e-4


@pytest.mark.parametrize("tokens,rows,cols,grid,free", [(0, 2048, 128, (128, 1), 2433), (0, 3072, 48, (128, 1), 1030), (0, 256, 4112, (128, 1), 129), (1, 100, 2048, (1, 128), 1316), (1, 65, 1024, (1, 128), 2500),
                                                        (1, 1090, 256, (1, 128), 4), (1, 200, 384, (1, 128), 132)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_several_tiles_per_cta_and_ragged_ends(built_lib, tokens, rows, cols, grid, free, dtype):
    """More tiles than SMs (a tile leaves while the next is made), parts of a contraction that end inside a stage, rows of g that end inside
    a chunk of eight; then the sums of one cotangent, in the last tile, that are not finite and made again."""
    gen = torch.Generator(device="cuda").manual_seed(rows + cols + free)
    q, sc8, sc32 = quantize_impl(torch.randn(rows, cols, generator=gen, device="cuda") * 0.02, grid)
    g = (torch.randn(rows if tokens else free, free if tokens else cols, generator=gen, device="cuda") * 1e-3).to(dtype)
    code = _lib.PB_F32 if dtype is torch.float32 else _lib.PB_BF16
    size = built_lib.pb_dense_dot_workspace_size(tokens, rows, cols, *grid, free)
    ws = torch.full((max(size, 16),), 0xff, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    d = dequantize_impl(q, sc8, sc32, torch.float32, grid).double()

    def run():
        out = torch.full(((cols, free) if tokens else (free, rows)), float("nan"), device="cuda")
        _lib.check(built_lib.pb_dense_dot(tokens, q.data_ptr(), sc8.data_ptr(), sc32.data_ptr(), rows, cols, *grid, g.data_ptr(), code, free, out.data_ptr(), ws.data_ptr(), size, stream))
        a, b = (d.t(), g.double()) if tokens else (g.double(), d.t())
        return out.double(), a @ b, _bound(a, b)

    got, want, bound = run()
    assert ((got - want).abs() <= bound + 1e-30).all()
    (g[:, -1] if tokens else g[-1]).mul_(1e33)
    got, want, bound = run()
    finite = torch.ones(free, dtype=torch.bool, device="cuda")
    finite[-1] = False
    got_f, want_f, bound_f = (t[:, finite] if tokens else t[finite] for t in (got, want, bound))
    assert ((got_f - want_f).abs() <= bound_f + 1e-30).all()
    last, want_l = (got[:, -1], want[:, -1]) if tokens else (got[-1], want[-1])      # f32 products one after the other
    bound_l = (bound[:, -1] if tokens else bound[-1]) * (rows if tokens else cols)
    assert ((last - want_l).abs() <= bound_l).all()
    assert built_lib.pb_gemm_check(stream) == 0
