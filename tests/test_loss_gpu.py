"""The loss kernels' one-pass row reduction and its two block sizes: vocabularies around the unrolled step of either, few rows (1024
threads each) and many (256), and logits of -inf, which a masked vocabulary has."""
import pytest
import torch

from pratchya_b200 import _lib

pytestmark = pytest.mark.gpu


def _run(z, target, weight, alpha):
    lib = _lib.load()
    rows, vocab = z.shape
    loss, lse = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.pb_smoothed_xent(z.data_ptr(), target.data_ptr(), weight.data_ptr(), rows, vocab, alpha, loss.data_ptr(), lse.data_ptr(), st))
    dz, up = torch.full_like(z, float("nan")), torch.ones(1, device="cuda")       # an element that is not written shows
    _lib.check(lib.pb_smoothed_xent_bwd(z.data_ptr(), target.data_ptr(), weight.data_ptr(), lse.data_ptr(), up.data_ptr(), 2.0, rows, vocab, alpha, dz.data_ptr(), st))
    return loss, lse, dz


@pytest.mark.parametrize("rows,vocab", [(3, 4), (2, 1020), (5, 4092), (5, 4096), (3, 4100), (2, 16384), (2, 16388), (1, 65536), (1000, 4096), (1000, 4100), (1000, 8), (400, 4092), (400, 8192), (500, 32768)])
def test_rows_of_any_length(built_lib, rows, vocab):
    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    z = torch.randn(rows, vocab, generator=g, device="cuda") * 4
    z[0] -= 1000.0                                     # a row far from zero: the running maximum has to carry it
    z[-1, -1] = 60.0                                   # ... and one whose maximum is its last value
    target = torch.randint(0, vocab, (rows,), generator=g, device="cuda")
    weight = torch.rand(rows, generator=g, device="cuda")
    loss, lse, dz = _run(z, target, weight, 0.1)
    z64 = z.double()
    want = torch.logsumexp(z64, -1)
    # a thread adds at most 64 + 10 terms of relative error 2^-24 each and expf's 2 ulp, and lse itself rounds
    assert (lse.double() - want).abs().max() <= 8e-6 + 2 ** -23 * want.abs().max()
    logp = z64 - want[:, None]
    ref = weight.double() * (-0.9 * logp.gather(1, target[:, None])[:, 0] - 0.1 * logp.mean(-1))
    assert (loss.double() - ref).abs().max() <= 2e-5 + 2 ** -21 * z64.abs().max()
    # dz by its own terms: the softmax carries the error of z - lse (lse's own, and the rounding of the difference) and expf's
    # 2 ulp; it, the one-hot and alpha / V meet in two additions and are scaled by a factor of two roundings
    hot, p, x = torch.zeros_like(z64).scatter_(1, target[:, None], 0.9), logp.exp(), logp.abs()
    softmax_error = p * ((lse.double() - want).abs()[:, None] + 2.0 ** -24 * x + 2.0 ** -22)
    bound = weight.double()[:, None] / 2 * (softmax_error + 2.0 ** -22 * (p + hot + 0.1 / vocab))
    assert ((dz.double() - weight.double()[:, None] / 2 * (p - hot - 0.1 / vocab)).abs() <= bound + 1e-38).all()


@pytest.mark.parametrize("rows", [4, 1000])
def test_masked_logits(built_lib, rows):
    z = torch.randn(rows, 5000, device="cuda")
    z[:, :4500] = -float("inf")                        # whole threads see nothing else
    z[1] = -float("inf")                               # a row without any logit: not a number, as its softmax is
    target = torch.full((rows,), 4999, device="cuda", dtype=torch.int64)
    _, lse, _ = _run(z, target, torch.ones(rows, device="cuda"), 0.0)
    want = torch.logsumexp(z.double(), -1)
    keep = [i for i in range(rows) if i != 1]
    assert torch.isnan(lse[1]) and (lse.double()[keep] - want[keep]).abs().max() <= 1e-5
