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


@pytest.mark.parametrize("rows,cols,grid,one_call", [(128, 128, (128, 128), True), (128, 4, (128, 1), True), (1024, 3840, (1024, 128), True), (2048, 128, (2048, 128), False),
                                                     (4096, 256, (4096, 1), False), (1024, 2048, (512, 16), False)])
def test_tall_blocks_that_few_ctas_would_walk_go_by_two_calls(built_lib, rows, cols, grid, one_call):
    """The library's rule, and the same bits on both sides of it; the one call still takes what the rule sends elsewhere."""
    x = to_torch(synth((rows, cols), seed=cols, scale=1e-3))
    blocks = rows * cols // (grid[0] * grid[1])
    assert built_lib.pb_fake_quantize_blocks_workspace_size(1, rows, cols, *grid) == (4 * blocks if one_call else 0)
    want = dequantize_impl(*quantize_impl(x, grid), torch.float32, grid)
    out, ws = torch.empty_like(x), torch.empty(blocks, device="cuda")
    assert built_lib.pb_fake_quantize_blocks(x.data_ptr(), 1, rows, cols, *grid, out.data_ptr(), ws.data_ptr(), 4 * blocks, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, want) and torch.equal(_ops.fake_quantize_impl(x, grid, torch.float32), want)
