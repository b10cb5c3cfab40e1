"""The abort path of the dense-dot kernel: a bounded wait that runs out is reported by pb_gemm_check.

The diagnostics build fills the first stage of a launch and never announces it, with a poll budget of about two milliseconds per
wait: the issuing lane gives up on the stage, the emptying warps on its accumulator, the converting warps on its buffer, and
the kernel releases tensor memory and returns.  Nothing is in flight for the stage, nothing traps or faults."""
import pytest
import torch

from helpers import synth, to_torch
from pratchya_b200 import _lib
from pratchya_b200._qualia import quantize_impl

pytestmark = pytest.mark.gpu

PB_ERR_DEVICE_TIMEOUT = 7


@pytest.mark.parametrize("tokens", [0, 1])
@pytest.mark.parametrize("m,k,n", [(200, 1024, 512), (40, 128, 64)])      # more stages than buffers, and a single one
def test_a_wait_that_runs_out_is_reported_and_the_next_launch_is_clean(built_lib, diag_lib, tokens, m, k, n):
    grid, rows, cols = ((1, 128), m, k) if tokens else ((128, 1), k, n)
    q, sc8, sc32 = quantize_impl(to_torch(synth((rows, cols), seed=rows)), grid)
    g = to_torch(synth((m, n), seed=n, scale=1e-3))
    free = n if tokens else m
    st = torch.cuda.current_stream().cuda_stream
    ws_bytes = diag_lib.pb_dense_dot_workspace_size(tokens, rows, cols, *grid, free)
    ws = torch.empty(max(ws_bytes, 16), dtype=torch.uint8, device="cuda")

    def run():
        out = torch.zeros((k, n) if tokens else (m, k), device="cuda")
        assert diag_lib.pb_dense_dot(tokens, q.data_ptr(), sc8.data_ptr(), sc32.data_ptr(), rows, cols, *grid, g.data_ptr(), _lib.PB_F32, free,
                                     out.data_ptr(), ws.data_ptr(), ws_bytes, st) == 0
        return out

    before = run()
    assert diag_lib.pb_gemm_check(st) == 0 and before.abs().max().item() > 0
    try:
        assert diag_lib.pb_debug_dot_control(1 << 10, 1) == 0
        run()
        assert diag_lib.pb_gemm_check(st) == PB_ERR_DEVICE_TIMEOUT
        assert b"dense-dot" in diag_lib.pb_last_error()
        assert diag_lib.pb_gemm_check(st) == 0           # reading the status clears it
    finally:
        diag_lib.pb_debug_dot_control(0, 0)
    after = run()
    assert diag_lib.pb_gemm_check(st) == 0 and torch.equal(before, after)
    assert built_lib.pb_gemm_check(st) == 0              # the product library has a word of its own
