"""Small kernels around a Linear's products: the byte transpose of a weight (16-byte form and the other), and the fake quantization
that also leaves its scales, against the calls they stand for."""
import pytest
import torch

from helpers import synth, to_torch
from pratchya_b200._qualia import _ops
from pratchya_b200._qualia import dequantize_impl, quantize_impl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(16, 16), (128, 128), (144, 272), (2048, 128), (128, 8192), (112, 16), (130, 64), (64, 130), (1, 1)])
def test_transpose_bytes(built_lib, rows, cols):
    q = torch.randint(0, 256, (rows, cols), device="cuda", dtype=torch.uint8).view(torch.float8_e4m3fn)
    assert torch.equal(_ops.transpose_bytes(q).view(torch.uint8), q.view(torch.uint8).t())


@pytest.mark.parametrize("shape,dtype", [((1, 1024), torch.float32), ((3, 2048), torch.bfloat16), ((8, 128), torch.float32), ((2, 5, 1024), torch.float32),
                                         ((3, 128), torch.float32), ((4, 384), torch.bfloat16)])
def test_fake_quantize_with_its_scales(built_lib, shape, dtype):
    x = to_torch(synth(shape, seed=shape[-1]))
    out, sc8, sc32 = _ops.fake_quantize_scales_impl(x, (1, 128), dtype)
    q, want8, want32 = quantize_impl(x, (1, 128))
    assert torch.equal(out, dequantize_impl(q, want8, want32, dtype, (1, 128)))
    assert torch.equal(sc8.view(torch.uint8), want8.view(torch.uint8)) and torch.equal(sc32, want32) and sc8.shape == want8.shape


@pytest.mark.parametrize("shape,grid", [((128, 128), (128, 128)), ((384, 640), (128, 128)), ((2048, 128), (128, 1)), ((128, 132), (128, 1)),
                                        ((192, 320), (64, 64)), ((3, 128, 272), (128, 16)), ((64, 260), (64, 4)), ((100, 256), (50, 128)), ((128, 6), (128, 1)),
                                        ((1024, 320), (1024, 1)), ((768, 144), (768, 1)), ((2, 1024, 192), (1024, 1))])
def test_fake_quantize_on_a_weights_grid(built_lib, shape, grid):
    x = to_torch(synth(shape, seed=shape[-1], scale=1e-3))
    x.view(-1)[::41] = -0.0
    x.view(-1)[: shape[-1]] = 0.0
    got, want = _ops.fake_quantize_impl(x, grid, torch.float32), dequantize_impl(*quantize_impl(x, grid), torch.float32, grid)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
