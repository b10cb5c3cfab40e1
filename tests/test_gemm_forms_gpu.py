"""The forms of the GEMM that its size chooses between (tiles of 128 x 32, 64, 128 and 224 on one CTA, 256 x 224 on a pair, the
contraction cut over a cluster of two and four): remainders in every direction against a 64-bit product, the same bits from all of
them, and their abort paths."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from pratchya_b200 import _lib
from pratchya_b200._qualia import _ops, dequantize_impl, quantize_impl

pytestmark = pytest.mark.gpu

PB_ERR_DEVICE_TIMEOUT = 7


def _triples(m, k, n, grid):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = torch.randn(m, k, generator=g, device="cuda") * torch.randn(m, 1, generator=g, device="cuda").exp()
    w = torch.randn(k, n, generator=g, device="cuda") * 0.02
    return quantize_impl(x, (1, 128)), quantize_impl(w, grid)


@pytest.mark.parametrize("m,k,n,grid", [
    (1, 1024, 1024, (128, 128)), (8, 2048, 2048, (128, 128)), (127, 2304, 128, (128, 128)), (128, 4096, 512, (128, 128)), (33, 5120, 256, (128, 128)), (100, 3072, 1024, (128, 128)),
    (5, 2048, 8192, (128, 128)), (129, 2048, 2048, (128, 128)), (255, 8192, 2048, (128, 128)), (257, 1024, 896, (128, 128)), (520, 2048, 2048, (128, 128)), (1000, 1024, 1152, (128, 128)),
    (2000, 1024, 1024, (128, 128)), (1031, 2048, 8192, (128, 128)), (8, 256, 640, (128, 128)), (16, 384, 384, (128, 128)), (640, 1280, 256, (128, 128)),
    (1, 2048, 128, (128, 1)), (64, 2048, 48, (128, 1)), (300, 1024, 144, (128, 1)), (1000, 2048, 128, (128, 1)), (72, 640, 16, (128, 1)), (8, 128, 2064, (128, 1)), (8192, 2048, 128, (128, 1)),
    (129, 1152, 4096, (128, 1)), (2056, 128, 1040, (128, 1)), (40, 2048, 8208, (128, 1))])
def test_products_against_64_bits(built_lib, m, k, n, grid):
    xq, wq = _triples(m, k, n, grid)
    if xq[1].shape[-1] != 8:
        xq, _ = _triples(m + 8 - m % 8, k, n, grid)         # whole super-groups
    xd, wd = dequantize_impl(*xq, torch.float32, (1, 128)).double(), dequantize_impl(*wq, torch.float32, grid).double()
    want = xd @ wd
    # per element, |x| @ |w| times what the tensor core's additions of 128 products (2^-23 each k-block at most, of which eight meet in an
    # accumulator) and the f32 additions of the blocks and parts behind them may be off by
    bound = (xd.abs() @ wd.abs()) * 2.0 ** -23 * (k / 128 + 12)
    got = _ops.matmul_impl(*xq, *wq, (1, 128), grid)
    assert got.shape == want.shape and ((got.double() - want).abs() <= bound + 1e-30).all()
    half = _ops.matmul_impl(*xq, *wq, (1, 128), grid, out_dtype=torch.bfloat16)
    assert ((half.double() - want).abs() <= bound + want.abs() * 2.0 ** -8 + 1e-30).all()
    assert torch.equal(got, _ops.matmul_impl(*xq, *wq, (1, 128), grid))
    assert built_lib.pb_gemm_check(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("m,k,n,grid", [(8, 2048, 8192, (128, 1)), (64, 2048, 2048, (128, 128)), (100, 2048, 8192, (128, 128)), (136, 2048, 2048, (128, 128)), (500, 1024, 1024, (128, 128))])
def test_a_workspace_for_more_rows_serves_fewer(built_lib, m, k, n, grid):
    """A host with one workspace for all of its batch sizes: what the largest takes is enough for every other, and the bits are the same."""
    xq, wq = _triples(m, k, n, grid)
    wt, st = _ops.transpose_bytes(wq[0]), torch.cuda.current_stream().cuda_stream
    b = _ops._operand(wt, wq[1], wq[2], n, k, (grid[1], 128), 1)
    a = _ops._operand(*xq, m, k, (1, 128))
    large = _ops._operand(*xq, 1024, k, (1, 128))                      # describes a size: nothing is read through it
    own, size = built_lib.pb_gemm_workspace_size(a, b), built_lib.pb_gemm_workspace_size(large, b)

    def run(size, x=None):
        ws, d = torch.full((size + 512,), 0xa5, dtype=torch.uint8, device="cuda"), torch.full((m, n), float("nan"), device="cuda")
        if x is not None:                                              # A's scales by the quantizer, into the same workspace
            q, s8, s32 = [torch.empty_like(t) for t in xq]
            _lib.check(built_lib.pb_quantize_for_gemm(x.data_ptr(), _lib.PB_F32, m, k, _lib.PB_E4M3, q.data_ptr(), s8.data_ptr(), s32.data_ptr(), b, ws.data_ptr(), size, st))
            _lib.check(built_lib.pb_gemm_tn_ex(_ops._operand(q, s8, s32, m, k, (1, 128)), b, d.data_ptr(), _lib.PB_F32, n, ws.data_ptr(), size, 1, st))
        else:
            _lib.check(built_lib.pb_gemm_tn(a, b, d.data_ptr(), _lib.PB_F32, n, ws.data_ptr(), size, st))
        assert (ws[size:] == 0xa5).all()
        return d

    want = run(own)
    assert torch.equal(run(size), want)
    if grid == (128, 128):
        g = torch.Generator(device="cuda").manual_seed(m + k + n)      # as _triples
        x = torch.randn(m, k, generator=g, device="cuda") * torch.randn(m, 1, generator=g, device="cuda").exp()
        assert torch.equal(run(size, x), want)
    assert built_lib.pb_gemm_check(st) == 0


# remainders of 128 and 256 rows, of 32, 64, 128 and 224 columns, of a chunk of eight k-blocks; contractions cut and not, in halves and not
FORM_SIZES = [(1, 1024, 1024, (128, 128)), (40, 4096, 512, (128, 128)), (127, 2304, 128, (128, 128)), (128, 5120, 384, (128, 128)), (129, 2048, 2048, (128, 128)), (200, 8192, 2048, (128, 128)),
              (257, 4096, 896, (128, 128)), (500, 1024, 1024, (128, 128)), (1000, 3072, 1152, (128, 128)), (2048, 1024, 640, (128, 128)),
              (8, 2048, 144, (128, 1)), (64, 640, 48, (128, 1)), (136, 2048, 128, (128, 1)), (300, 1024, 2064, (128, 1)), (1000, 2048, 240, (128, 1)), (2056, 128, 1040, (128, 1))]


def _products(lib):
    out = {}
    for m, k, n, grid in FORM_SIZES:
        xq, wq = _triples(m, k, n, grid)
        wt = _ops.transpose_bytes(wq[0])
        a, b = _ops._operand(*xq, m, k, (1, 128)), _ops._operand(wt, wq[1], wq[2], n, k, (grid[1], 128), 1)
        size, st = lib.pb_gemm_workspace_size(a, b), torch.cuda.current_stream().cuda_stream
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        out[m, k, n, grid, "workspace"] = torch.tensor([size])
        for dtype, code in ((torch.float32, _lib.PB_F32), (torch.bfloat16, _lib.PB_BF16)):
            d = torch.full((m, n), float("nan"), dtype=dtype, device="cuda")
            assert lib.pb_gemm_tn(a, b, d.data_ptr(), code, n, ws.data_ptr(), size, st) == 0, lib.pb_last_error()
            out[m, k, n, grid, code] = d.cpu()
        assert lib.pb_gemm_check(st) == 0
    return out


@pytest.mark.parametrize("form", ["32", "64", "128", "224", "pair"])
def test_every_form_gives_the_same_bits(built_lib, diag_lib, tmp_path, form):
    """The diagnostics build's switches force one form on every size, in a process of its own (they are read once)."""
    env = dict(os.environ, PB_GEMM_BN="224" if form == "pair" else form, PB_GEMM_SINGLE="0" if form == "pair" else "1")
    here = Path(__file__).resolve().parent
    code = "import sys; sys.path[:0] = sys.argv[2:]\nimport test_gemm_forms_gpu as t, torch\ntorch.save(t._products(t._lib.load_diagnostics()), sys.argv[1])"
    r = subprocess.run([sys.executable, "-c", code, str(tmp_path / "d.pt"), str(here), str(here.parent)], env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    forced = torch.load(tmp_path / "d.pt")
    chosen, compared = _products(built_lib), 0
    sizes = [key for key in chosen if key[-1] == "workspace"]
    assert sum(not torch.equal(forced[key], chosen[key]) for key in sizes) >= 5            # the switch is heard: another tile width, another layout
    for key, want in ((key, d) for key, d in chosen.items() if key not in sizes):
        # an f32 product of more than 128 rows may be the sum of two halves, which the wide single tiles do not make
        if form in ("128", "224") and key[0] > 128 and key[-1] == _lib.PB_F32:
            continue
        assert torch.equal(forced[key].view(torch.uint8), want.view(torch.uint8)), (form, key)
        compared += 1
    assert compared >= 20


def test_outputs_with_longer_rows_and_off_the_store_alignment(built_lib):
    """ldd beyond n, and rows that are no multiple of 16 bytes: nothing but [m, n] is written."""
    for m, k, n, ldd in [(40, 4096, 512, 640), (40, 2048, 512, 513), (130, 1024, 256, 300), (7, 1024, 128, 129)]:
        xq, wq = _triples(m, k, n, (128, 128))
        wt = _ops.transpose_bytes(wq[0])
        a, b = _ops._operand(*xq, m, k, (1, 128)), _ops._operand(wt, wq[1], wq[2], n, k, (128, 128), 1)
        size = built_lib.pb_gemm_workspace_size(a, b)
        ws = torch.full((size,), 0xff, dtype=torch.uint8, device="cuda")
        want = dequantize_impl(*xq, torch.float32, (1, 128)).double() @ dequantize_impl(*wq, torch.float32, (128, 128)).double()
        for dtype, code in ((torch.float32, _lib.PB_F32), (torch.bfloat16, _lib.PB_BF16)):
            d = torch.full((m + 1, ldd), 7.0, dtype=dtype, device="cuda")
            _lib.check(built_lib.pb_gemm_tn(a, b, d.data_ptr(), code, ldd, ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream))
            assert (d[:m, n:] == 7).all() and (d[m:] == 7).all()
            assert ((d[:m, :n].double() - want).norm() / want.norm()).item() <= (1e-6 if code == _lib.PB_F32 else 4e-3)


@pytest.mark.parametrize("m,k,n", [(40, 4096, 512), (40, 2048, 2048), (40, 1024, 256), (200, 8192, 2048), (100, 1024, 8192), (2048, 2048, 2048)])
def test_a_wait_that_runs_out_is_reported_and_the_next_launch_is_clean(built_lib, diag_lib, m, k, n):
    """The diagnostics build leaves a launch's first stage (of a cluster's last rank) unfilled, with a poll budget of about two milliseconds."""
    xq, wq = _triples(m, k, n, (128, 128))
    wt = _ops.transpose_bytes(wq[0])
    a, b = _ops._operand(*xq, m, k, (1, 128)), _ops._operand(wt, wq[1], wq[2], n, k, (128, 128), 1)
    size, st = diag_lib.pb_gemm_workspace_size(a, b), torch.cuda.current_stream().cuda_stream
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")

    def run():
        d = torch.zeros(m, n, device="cuda")
        assert diag_lib.pb_gemm_tn(a, b, d.data_ptr(), _lib.PB_F32, n, ws.data_ptr(), size, st) == 0
        return d

    before = run()
    assert diag_lib.pb_gemm_check(st) == 0 and before.abs().max().item() > 0
    try:
        assert diag_lib.pb_debug_gemm_control(1 << 10, 8) == 0
        run()
        assert diag_lib.pb_gemm_check(st) == PB_ERR_DEVICE_TIMEOUT
        assert diag_lib.pb_gemm_check(st) == 0               # reading the status clears it
    finally:
        diag_lib.pb_debug_gemm_control(0, 0)
    after = run()
    assert diag_lib.pb_gemm_check(st) == 0 and torch.equal(before, after)
    assert built_lib.pb_gemm_check(st) == 0
