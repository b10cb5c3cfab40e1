"""The two-kernel quantizer of tall blocks (64 rows or more) against the oracle, bit for bit: part-filled column groups, one-column
blocks, blocks narrower than a warp's row, super-groups inside a CTA and across many, stacks, and both dtypes and formats."""
import numpy as np
import pytest
import torch

from helpers import BF16, assert_triple_equal, bytes_of, oracle, synth, to_torch
from pratchya_b200._qualia import quantize_impl

pytestmark = pytest.mark.gpu

CASES = [
    ((128, 132), (128, 1)), ((256, 4), (128, 1)), ((64, 520), (64, 1)), ((128, 2056), (128, 1)),      # the last column group part full
    ((128, 128), (128, 128)), ((384, 640), (128, 128)), ((2048, 1152), (128, 128)),                   # bf16: an odd number of 128-column blocks
    ((128, 272), (128, 16)), ((64, 264), (64, 8)), ((192, 320), (64, 64)), ((1024, 2048), (64, 32)),  # several blocks per warp, K above and below 32
    ((100, 256), (100, 128)), ((66, 128), (66, 64)), ((3, 128, 256), (128, 128)), ((2, 256, 136), (64, 1)),
    ((63, 128), (63, 64)), ((128, 6), (128, 1)), ((128, 96), (128, 48)),                              # the three-kernel form's side of the rule
]


@pytest.mark.parametrize("shape,grid", CASES)
@pytest.mark.parametrize("dtype", [np.float32, BF16])
@pytest.mark.parametrize("fmt", ["e4m3", "e5m2"])
def test_tall_blocks_bit_exact(built_lib, shape, grid, dtype, fmt):
    x = synth(shape, seed=len(shape) * 1000 + shape[-1] + grid[1], scale=0.02, dtype=dtype)
    x.reshape(-1)[::37] = -0.0
    assert_triple_equal(quantize_impl(to_torch(x), grid, out_format=fmt), oracle.quantize_impl(x, grid, out_format=fmt), f"{shape} {grid}")


@pytest.mark.parametrize("grid", [(128, 128), (128, 1)])
def test_a_nan_stays_in_its_block(built_lib, grid):
    x = synth((128, 256), seed=3)
    x[5, 7] = np.nan
    clean = x.copy()
    clean[5, 7] = 0.0
    got, want = quantize_impl(to_torch(x), grid), quantize_impl(to_torch(clean), grid)
    assert bytes_of(got[0])[5, 7] & 0x7F == 0x7F
    cols = [c for c in range(256) if (c != 7 if grid[1] == 1 else c >= 128)]
    assert np.array_equal(bytes_of(got[0])[:, cols], bytes_of(want[0])[:, cols])
    assert torch.isfinite(got[2]).all()


def test_views_off_the_vector_alignment(built_lib):
    base = to_torch(synth((128 * 256 + 1,), seed=9))
    x = base[1:].view(128, 256)                        # four bytes off sixteen: the scalar form of the three-kernel path
    assert_triple_equal(quantize_impl(x, (128, 128)), oracle.quantize_impl(x.cpu().numpy(), (128, 128)), "offset view")
