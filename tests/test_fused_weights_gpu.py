"""The byte transpose of a weight: its 16-byte form and the other."""
import pytest
import torch

from pratchya_b200._qualia import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(16, 16), (128, 128), (144, 272), (2048, 128), (128, 8192), (112, 16), (130, 64), (64, 130), (1, 1)])
def test_transpose_bytes(built_lib, rows, cols):
    q = torch.randint(0, 256, (rows, cols), device="cuda", dtype=torch.uint8).view(torch.float8_e4m3fn)
    assert torch.equal(_ops.transpose_bytes(q).view(torch.uint8), q.view(torch.uint8).t())
