"""The prepared scales of an activation whose rows do not fill the GEMM's tiles: whatever the workspace held in the rows of padding
(NaN and Inf scales among it), the product has the bits of the path that prepares them itself."""
import pytest
import torch

from helpers import synth, to_torch
from pratchya_b200._qualia import LinearStep, matmul_impl, quantize_impl
from pratchya_b200._qualia import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 127, 129, 255, 300, 1000])
@pytest.mark.parametrize("n,k", [(1024, 2048), (256, 4096)])
@pytest.mark.parametrize("garbage", [0xFF, 0x7F, 0x00])
def test_rows_of_padding_do_not_matter(built_lib, rows, n, k, garbage):
    x = to_torch(synth((rows, k), seed=rows + k))
    wq = quantize_impl(to_torch(synth((k, n), seed=n, scale=0.02, outliers=0)), (128, 128))
    w_t = _ops.transpose_bytes(wq[0])
    want = matmul_impl(*quantize_impl(x, (1, 128)), *wq, (1, 128), (128, 128), y_fp8_t=w_t)
    step = LinearStep(w_t, wq[1], wq[2], rows=rows, out_dtype=torch.float32)
    step.ws.fill_(garbage)
    assert torch.equal(step(x)[0], want)
    assert torch.equal(step(x)[0], want)             # the weight's scales are in the workspace now
