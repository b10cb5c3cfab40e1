"""A scan cut after any timestep and continued from the state that it left gives the bits of the whole one: a prompt in pieces of any
length, and decoding a token at a time, are the prefill."""
import pytest
import torch

from pratchya_b200._nnx_impl._wkv7 import _forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [2, 60, 100, 160, 230])      # every form of the forward kernel
@pytest.mark.parametrize("save", [False, True])
def test_a_scan_cut_anywhere_is_the_whole_one(built_lib, heads, save):
    steps = 19
    g = torch.Generator(device="cuda").manual_seed(heads)
    rn = lambda: torch.randn(1, steps, heads * 64, generator=g, device="cuda")
    kap = torch.nn.functional.normalize(rn().view(1, steps, heads, 64), dim=-1).reshape(1, steps, heads * 64)
    ins = [torch.sigmoid(rn()), torch.sigmoid(rn()), kap, rn(), rn(), rn()]
    state = torch.randn(1, heads, 64, 64, generator=g, device="cuda")
    s_all, y_all, _, sa_all = _forward(state, ins, heads, save)
    for cuts in [[c] for c in range(1, steps)] + [list(range(1, steps)), [3, 5, 6, 13]]:
        s, ys, sas = state, [], []
        for lo, hi in zip([0, *cuts], [*cuts, steps]):
            s, y, _, sa = _forward(s, [t[:, lo:hi].contiguous() for t in ins], heads, save)
            ys.append(y)
            sas.append(sa)
        assert torch.equal(torch.cat(ys, 1), y_all) and torch.equal(s, s_all), cuts
        if save:
            assert torch.equal(torch.cat(sas, 1), sa_all), cuts
