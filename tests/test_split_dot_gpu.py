"""pb_dense_dot's form for operands that many tiles share (the fastest workspace), against 64-bit products and against the form that
needs no workspace: remainders of its tiles in every direction, every tile width, contractions cut and not, several sets and
several rounds of terms, powers of two that bf16 does not hold, infinities and NaNs."""
import pytest
import torch

from pratchya_b200 import _lib
from pratchya_b200._qualia import _ops, dequantize_impl, quantize_impl

pytestmark = pytest.mark.gpu

F32, BF16 = torch.float32, torch.bfloat16
PB_ERR_DEVICE_TIMEOUT = 7


def _dot(lib, tokens, triple, grid, g, best=True):
    """(out, whether the workspace is the fastest form's)"""
    q, sc8, sc32 = triple
    rows, cols = q.shape
    free, code = g.shape[1] if tokens else g.shape[0], _lib.PB_BF16 if g.dtype == BF16 else _lib.PB_F32
    least = lib.pb_dense_dot_workspace_size(tokens, rows, cols, *grid, free)
    size = lib.pb_dense_dot_workspace_best(tokens, rows, cols, *grid, free, code) if best else least
    ws = torch.full((max(size, 16),), 0xff, dtype=torch.uint8, device="cuda")          # NaNs, as bf16 and as f32
    out = torch.full((cols, free) if tokens else (free, rows), float("nan"), device="cuda")
    status = lib.pb_dense_dot(tokens, q.data_ptr(), sc8.data_ptr(), sc32.data_ptr(), rows, cols, *grid, g.data_ptr(), code, free, out.data_ptr(),
                              ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream)
    assert status == 0, lib.pb_last_error()
    return out, size > least


def _sums(tokens, triple, grid, g):
    d = dequantize_impl(*triple, F32, grid).double()
    return (d.t(), g.double()) if tokens else (g.double(), d.t())


def _bound(a, b):
    """Per element, |a| @ |b| times the roundings of this form: one of an operand (2^-24), up to two of a factor on the finished sum, the
    tensor core's within 64 of the contraction (twelve additions of at most 2^-23, of which eight make the low terms) and one
    addition per 64 of it or per part."""
    return (a.abs() @ b.abs()) * 2.0 ** -24 * (27 + (a.shape[1] + 63) // 64 + 16)


def _inputs(rows, cols, grid, free, tokens, dtype, amp=1.0):
    g = torch.Generator(device="cuda").manual_seed(rows + 3 * cols + free)
    x = torch.randn(rows, cols, generator=g, device="cuda") * torch.randn(rows, 1, generator=g, device="cuda").exp() * 0.02
    cot = torch.randn(rows if tokens else free, free if tokens else cols, generator=g, device="cuda") * 1e-3 * amp
    return quantize_impl(x, grid), cot.to(dtype)


# tokens, rows, cols, grid, free: the widths of a tile are chosen by how the tiles fill 148 SMs
CASES = [(0, 2048, 2048, (128, 128), 3001), (0, 1024, 1024, (128, 128), 1031), (0, 512, 2048, (128, 128), 777), (0, 4096, 528, (128, 1), 600), (0, 1024, 4096, (128, 128), 260),
         (0, 1152, 640, (128, 1), 2050), (1, 3001, 2048, (1, 128), 2048), (1, 193, 1024, (1, 128), 1032), (1, 1000, 512, (1, 128), 520), (1, 401, 3072, (1, 128), 648),
         (1, 4100, 2048, (1, 128), 128), (1, 777, 640, (1, 128), 1024), (1, 256, 1024, (1, 128), 2056)]


@pytest.mark.parametrize("tokens,rows,cols,grid,free", CASES)
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_sums_against_64_bits_and_the_other_form(built_lib, tokens, rows, cols, grid, free, dtype):
    triple, g = _inputs(rows, cols, grid, free, tokens, dtype)
    got, shared = _dot(built_lib, tokens, triple, grid, g)
    plain, _ = _dot(built_lib, tokens, triple, grid, g, best=False)
    a, b = _sums(tokens, triple, grid, g)
    want, bound = a @ b, _bound(a, b)
    assert ((got.double() - want).abs() <= bound + 1e-37).all()
    assert ((got - plain).abs().double() <= 2 * bound + 1e-37).all()
    error = lambda o: ((o.double() - want).norm() / want.norm()).item()
    assert error(got) <= error(plain) * 1.02                     # never the less precise of the two
    again, _ = _dot(built_lib, tokens, triple, grid, g)
    assert torch.equal(got, again)
    assert built_lib.pb_gemm_check(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("tokens,depth", [(0, 128), (0, 256), (0, 512), (1, 128), (1, 200), (1, 256), (1, 320), (1, 376), (1, 384), (1, 512), (1, 1000)])
def test_short_sums_of_one_sign_are_no_less_precise_than_the_other_form(built_lib, tokens, depth, dtype):
    """Where nothing cancels, what the tensor core's additions drop adds up, and few f32 additions follow that could hide it."""
    rows, cols, grid = (depth, 2048, (1, 128)) if tokens else (2048, depth, (128, 128))
    gen = torch.Generator(device="cuda").manual_seed(depth)
    triple = quantize_impl(torch.randn(rows, cols, generator=gen, device="cuda").abs() * 0.02, grid)
    g = (torch.randn(depth, 2048, generator=gen, device="cuda").abs() * 1e-3).to(dtype)
    g = g if tokens else g.t().contiguous()
    got, shared = _dot(built_lib, tokens, triple, grid, g)
    assert shared
    a, b = _sums(tokens, triple, grid, g)
    want = a @ b
    assert ((got.double() - want).abs() <= _bound(a, b)).all()
    assert (got.double() - want).norm() <= (_dot(built_lib, tokens, triple, grid, g, best=False)[0].double() - want).norm()


@pytest.mark.parametrize("dtype", [F32, BF16])
def test_a_workspace_off_32_bytes_gives_the_same_form(built_lib, dtype):
    """The workspace's alignment is 16 bytes; the bits do not depend on more of it, and nothing beyond its size is written."""
    rows, cols, grid, free = 1000, 1024, (1, 128), 1032
    (q, sc8, sc32), g = _inputs(rows, cols, grid, free, 1, dtype)
    want, shared = _dot(built_lib, 1, (q, sc8, sc32), grid, g)
    assert shared
    code = _lib.PB_BF16 if dtype == BF16 else _lib.PB_F32
    size = built_lib.pb_dense_dot_workspace_best(1, rows, cols, *grid, free, code)
    room = torch.full((size + 96,), 0xa5, dtype=torch.uint8, device="cuda")
    assert room.data_ptr() % 32 == 0
    for off in (16, 32, 48):
        out = torch.empty_like(want)
        _lib.check(built_lib.pb_dense_dot(1, q.data_ptr(), sc8.data_ptr(), sc32.data_ptr(), rows, cols, *grid, g.data_ptr(), code, free, out.data_ptr(),
                                          room.data_ptr() + off, size, torch.cuda.current_stream().cuda_stream))
        assert torch.equal(out, want) and (room[:16] == 0xa5).all() and (room[off + size:] == 0xa5).all()


def test_the_cases_reach_this_form(built_lib):
    """A changed rule that leaves these cases to the other form would leave this one untested."""
    size = lambda c, code: built_lib.pb_dense_dot_workspace_best(c[0], c[1], c[2], *c[3], c[4], code) - built_lib.pb_dense_dot_workspace_size(c[0], c[1], c[2], *c[3], c[4])
    assert sum(size(c, _lib.PB_BF16) > 0 for c in CASES) >= 11 and sum(size(c, _lib.PB_F32) > 0 for c in CASES) >= 8
    assert size((0, 4096, 528, (128, 1), 600), _lib.PB_F32) == 0           # a factor per column of the contraction
    assert size((1, 777, 640, (1, 128), 1024), _lib.PB_F32) == 0           # super-groups that end inside a row


@pytest.mark.parametrize("tokens,rows,cols,grid,free,dtype", [(1, 8200, 2048, (1, 128), 8192, F32), (1, 8200, 11264, (1, 128), 512, BF16), (0, 11264, 8208, (128, 1), 512, BF16)])
def test_several_rounds_of_terms(built_lib, tokens, rows, cols, grid, free, dtype):
    triple, g = _inputs(rows, cols, grid, free, tokens, dtype)
    got, shared = _dot(built_lib, tokens, triple, grid, g)
    assert shared
    a, b = _sums(tokens, triple, grid, g)
    assert ((got.double() - a @ b).abs() <= _bound(a, b) + 1e-37).all()
    # the sums of one cotangent made again, in the last round too: f32 products, a rounding a term and those of an operand
    (g[:, -7] if tokens else g[-7]).mul_(1e32)
    a, b = _sums(tokens, triple, grid, g)
    got = _dot(built_lib, tokens, triple, grid, g)[0]
    assert ((got.double() - a @ b).abs() <= (a.abs() @ b.abs()) * 2.0 ** -24 * (a.shape[1] + 4) + 1e-37).all()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("tokens", [0, 1])
def test_infinities_nans_and_blocks_far_below_their_group(built_lib, tokens, dtype):
    """Blocks 2^-118 and less of their super-group's largest value (their power of two times an fp8 value has no normal bf16), an
    infinite and a NaN cotangent: what the form without a workspace gives, whose sums are f32 products where they are not finite."""
    rows, cols, grid, free = (512, 1024, (1, 128), 1024) if tokens else (1024, 1024, (128, 128), 600)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(rows, cols, generator=g, device="cuda")
    x[:, 128:256] *= 2.0 ** -118
    if not tokens:
        x[256:384] *= 2.0 ** -120
    triple = quantize_impl(x, grid)
    cot = (torch.randn(rows if tokens else free, free if tokens else cols, generator=g, device="cuda") * 1e20).to(dtype)
    got, shared = _dot(built_lib, tokens, triple, grid, cot)
    assert shared
    a, b = _sums(tokens, triple, grid, cot)
    want = a @ b
    assert ((got.double() - want).abs() <= (a.abs() @ b.abs()) * 2.0 ** -24 * (a.shape[1] + 4) + a.shape[1] * 2.0 ** -149).all()
    cot = cot * 1e-20
    cot[(5, 17) if tokens else (17, 5)], cot[(9, 33) if tokens else (33, 9)] = float("inf"), float("nan")
    got = _dot(built_lib, tokens, triple, grid, cot)[0]
    got = got if tokens else got.t()                             # [i, j]: the cotangents' rows j are 17 and 33
    rest = [j for j in range(got.shape[1]) if j not in (17, 33)]
    assert torch.isnan(got[:, 33]).all() and not torch.isfinite(got[:, 17]).any() and torch.isfinite(got[:, rest]).all()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("tokens", [0, 1])
def test_no_wait_runs_out_while_every_sum_is_made_again(built_lib, diag_lib, tokens, dtype):
    """Cotangents whose sums pass f32's largest number with the terms' 2^40 and do not without it: all sums of every tile are made again.
    Three tiles a CTA, 8192 of the contraction, and waits of eight milliseconds at most: the tiles behind do not wait for it."""
    rows, cols, grid, free = (8192, 2048, (1, 128), 5000) if tokens else (2048, 8192, (128, 128), 5000)
    triple, g = _inputs(rows, cols, grid, free, tokens, dtype, amp=1e32)
    st = torch.cuda.current_stream().cuda_stream
    try:
        assert diag_lib.pb_debug_dot_control(1 << 12, 0) == 0
        got, shared = _dot(diag_lib, tokens, triple, grid, g)
        assert shared and diag_lib.pb_gemm_check(st) == 0
    finally:
        diag_lib.pb_debug_dot_control(0, 0)
    a, b = _sums(tokens, triple, grid, g)
    # f32 products, one after the other: a rounding a term, and those of an operand
    assert ((got.double() - a @ b).abs() <= (a.abs() @ b.abs()) * 2.0 ** -24 * (a.shape[1] + 4)).all()
    wild = torch.full_like(g, float("nan"))
    assert torch.isnan(_dot(built_lib, tokens, triple, grid, wild)[0]).all() and built_lib.pb_gemm_check(st) == 0


@pytest.mark.parametrize("whole_op", [True, False])
@pytest.mark.parametrize("tokens,dtype", [(0, F32), (1, F32), (1, BF16)])
def test_where_its_workspace_does_not_fit_the_other_form_runs(built_lib, monkeypatch, tokens, dtype, whole_op):
    """Torch's allocator is held to 48 MB more than it has: room for out and the least workspace, not for the terms."""
    rows, cols, grid, free = (8192, 2048, (1, 128), 2048) if tokens else (2048, 8192, (128, 128), 2048)
    triple, g = _inputs(rows, cols, grid, free, tokens, dtype)
    want = _dot(built_lib, tokens, triple, grid, g, best=False)[0]
    if not whole_op:                                             # the Python text
        real = _lib.native()
        monkeypatch.setattr(_lib, "_native", type("Declining", (), {"dense_dot": lambda self, *args: None, "__getattr__": lambda self, name: getattr(real, name)})())
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (48 << 20)) / total)
        got = _ops._dense_dot(tokens, *triple, grid, g)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)


@pytest.mark.parametrize("tokens", [0, 1])
def test_a_wait_that_runs_out_is_reported_and_the_next_launch_is_clean(built_lib, diag_lib, tokens):
    """The diagnostics build leaves the first stage of a launch unfilled, with a poll budget of about two milliseconds per wait."""
    rows, cols, grid, free = (600, 1024, (1, 128), 512) if tokens else (1024, 1024, (128, 128), 600)
    triple, g = _inputs(rows, cols, grid, free, tokens, F32)
    st = torch.cuda.current_stream().cuda_stream
    before, shared = _dot(diag_lib, tokens, triple, grid, g)
    assert shared and diag_lib.pb_gemm_check(st) == 0
    try:
        assert diag_lib.pb_debug_dot_control(1 << 10, 1) == 0
        _dot(diag_lib, tokens, triple, grid, g)
        assert diag_lib.pb_gemm_check(st) == PB_ERR_DEVICE_TIMEOUT and b"dense-dot" in diag_lib.pb_last_error()
        assert diag_lib.pb_gemm_check(st) == 0                   # reading the status clears it
    finally:
        diag_lib.pb_debug_dot_control(0, 0)
    after, _ = _dot(diag_lib, tokens, triple, grid, g)
    assert diag_lib.pb_gemm_check(st) == 0 and torch.equal(before, after)
    assert built_lib.pb_gemm_check(st) == 0


@pytest.mark.parametrize("rows,cols,free,amp", [(128, 128, 1, 1.0), (128, 2048, 63, 1.0), (512, 512, 5, 1.0), (1024, 1024, 64, 1e-30), (2048, 2048, 129, 1.0), (8192, 4096, 150, 1.0), (384, 2048, 1000, 1e30),
                                                (640, 640, 200, 1.0), (1152, 896, 333, 1.0), (2048, 1024, 2400, 1.0)])
def test_one_term_for_a_bf16_cotangent(built_lib, rows, cols, free, amp):
    """dX of a bf16 cotangent: the fp8 values times their powers of two, the super-group's factor on the finished sums (of one group, of
    two, of one per row of blocks; 640 and 1152 rows: groups that end inside a row, three terms), few tokens and no whole tile of them."""
    triple, g = _inputs(rows, cols, (128, 128), free, 0, BF16, amp)
    got, _ = _dot(built_lib, 0, triple, (128, 128), g)
    plain, _ = _dot(built_lib, 0, triple, (128, 128), g, best=False)
    a, b = _sums(0, triple, (128, 128), g)
    want, bound = a @ b, _bound(a, b)
    assert ((got.double() - want).abs() <= bound + 1e-37).all()
    if amp == 1.0:
        assert (got.double() - want).norm() <= (plain.double() - want).norm() * 1.02
    assert torch.equal(got, _dot(built_lib, 0, triple, (128, 128), g)[0])
    assert built_lib.pb_gemm_check(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("power", [60, 100, -60])
def test_rows_far_below_a_large_super_group(built_lib, dtype, power):
    """dX of a weight whose super-group's largest value is 2^power, with rows of size one in it, and a cotangent of 2^-power: the sums of
    those rows are as far from f32's ends as an f32 dot's."""
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(1024, 1024, generator=g, device="cuda") * 2.0 ** power
    x[256:384] = torch.randn(128, 1024, generator=g, device="cuda") * 2.0 ** min(power, 0)
    triple = quantize_impl(x, (128, 128))
    cot = (torch.randn(600, 1024, generator=g, device="cuda") * 2.0 ** -power).to(dtype)
    got, shared = _dot(built_lib, 0, triple, (128, 128), cot)
    assert shared
    a, b = _sums(0, triple, (128, 128), cot)
    assert ((got.double() - a @ b).abs() <= _bound(a, b)).all()


@pytest.mark.parametrize("rows,cols,free", [(2048, 2048, 8), (4096, 1024, 64), (8192, 2048, 1), (8192, 2048, 100), (8192, 2048, 128)])
def test_one_term_for_few_rows_of_a_large_weight(built_lib, rows, cols, free):
    """The faster form there, and the more precise one."""
    triple, g = _inputs(rows, cols, (128, 128), free, 0, BF16)
    got, shared = _dot(built_lib, 0, triple, (128, 128), g)
    assert shared
    a, b = _sums(0, triple, (128, 128), g)
    want = a @ b
    assert ((got.double() - want).abs() <= _bound(a, b)).all()
    assert (got.double() - want).norm() <= (_dot(built_lib, 0, triple, (128, 128), g, best=False)[0].double() - want).norm() * 1.02
