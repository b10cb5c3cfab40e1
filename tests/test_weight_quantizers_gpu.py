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
    ((1024, 320), (1024, 1)), ((768, 144), (768, 1)), ((2, 1024, 192), (1024, 1)), ((1024, 2048), (512, 64)),      # K above 32, with super-groups that end inside a CTA's blocks
    ((2048, 3200), (2048, 128)), ((1024, 9472), (512, 1)), ((192, 3200), (96, 128)),                  # many rows on many CTAs
    ((4096, 256), (4096, 128)), ((2048, 256), (2048, 1)), ((512, 2048), (256, 32)), ((128, 128), (128, 1)),      # ... and on few: three kernels
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


@pytest.mark.parametrize("shape,grid", [((128, 256), (128, 128)), ((256, 256), (128, 1)), ((128, 128), (64, 16)), ((130, 256), (65, 4)), ((32, 256), (4, 64)), ((16, 1024), (2, 512))])
@pytest.mark.parametrize("dtype", [np.float32, BF16])
def test_nans_are_dropped_on_every_route(built_lib, shape, grid, dtype):
    """A row, a column and single elements of NaN: everything else has the scales and bytes that it has beside zeros, and a copy off
    the vector alignment has those of the aligned array.  A block of nothing but NaNs keeps the scale byte 255."""
    x = synth(shape, seed=grid[1], dtype=np.float32)
    nan = np.zeros(shape, bool)
    nan[5] = True
    nan[: grid[0], 8 * grid[1] % shape[1] : 8 * grid[1] % shape[1] + grid[1]] = True      # one whole block
    nan[:, 3] = True
    nan[7, 9] = nan[11, 40] = True
    clean, x = np.where(nan, 0, x).astype(dtype), np.where(nan, np.nan, x).astype(dtype)
    got, want = quantize_impl(to_torch(x), grid), quantize_impl(to_torch(clean), grid)
    q, wq = bytes_of(got[0]), bytes_of(want[0])
    assert (q[nan] & 0x7F == 0x7F).all() and np.array_equal(q[~nan], wq[~nan])
    whole = nan.reshape(shape[0] // grid[0], grid[0], shape[1] // grid[1], grid[1]).all(axis=(1, 3)).reshape(-1)
    sc8, wsc8 = bytes_of(got[1]).reshape(-1), bytes_of(want[1]).reshape(-1)
    assert whole.any() and (sc8[whole] == 255).all() and np.array_equal(sc8[~whole], wsc8[~whole])
    assert torch.equal(got[2], want[2])
    t = to_torch(x)
    base = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    off = base[1:].view(shape)
    off.copy_(t)
    assert all(np.array_equal(bytes_of(a), bytes_of(b)) for a, b in zip(quantize_impl(off, grid)[:2], got[:2]))
