"""The forward scan's forms by head count give the bits of one head's call, in what they leave for the backward pass too: a head's sums
have one order in all of them."""
import pytest
import torch

from pratchya_b200._nnx_impl._wkv7 import _forward, wkv_state_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [18, 19, 37, 38, 74, 75, 148, 149, 185, 186])
@pytest.mark.parametrize("steps", [1, 7, 8, 9, 11, 12, 13, 14, 16, 26])
@pytest.mark.parametrize("with_grad", [False, True])
def test_head_counts_agree(built_lib, heads, steps, with_grad):
    g = torch.Generator(device="cuda").manual_seed(heads + steps)
    rn = lambda: torch.randn(1, steps, heads * 64, generator=g, device="cuda")
    kap = torch.nn.functional.normalize(rn().view(1, steps, heads, 64), dim=-1).reshape(1, steps, heads * 64)
    ins = [torch.sigmoid(rn()), torch.sigmoid(rn()), kap, rn(), rn(), rn()]
    state = torch.randn(1, heads, 64, 64, generator=g, device="cuda")
    full = [t.clone().requires_grad_(with_grad) for t in ins]
    s_all, y_all = wkv_state_scan(state, *full, heads)
    if with_grad:
        _, _, ckpt_all, sa_all = _forward(state, ins, heads, True)
    for h in {0, 1, heads // 2, heads - 1}:
        one = [t[..., h * 64:(h + 1) * 64].contiguous() for t in ins]
        s_one, y_one = wkv_state_scan(state[:, h:h + 1].contiguous(), *one, 1)
        if with_grad:
            _, _, ckpt_one, sa_one = _forward(state[:, h:h + 1].contiguous(), one, 1, True)
            assert torch.equal(sa_all[..., h * 64:(h + 1) * 64], sa_one) and torch.equal(ckpt_all.view(heads, -1)[h], ckpt_one)
        assert torch.equal(y_all[..., h * 64:(h + 1) * 64], y_one) and torch.equal(s_all[:, h:h + 1], s_one)


@pytest.mark.parametrize("heads", [222, 223])
@pytest.mark.parametrize("steps", [1, 2, 6, 7, 8, 9, 15, 17, 23])
@pytest.mark.parametrize("with_grad", [False, True])
def test_heads_around_one_and_a_half_waves_agree(built_lib, heads, steps, with_grad):
    """Halves of a head per CTA up to three on an SM, whole heads above: the bits of one head's call, and of the same scan cut at a
    multiple of eight timesteps and continued."""
    g = torch.Generator(device="cuda").manual_seed(heads + steps)
    rn = lambda: torch.randn(1, steps, heads * 64, generator=g, device="cuda")
    kap = torch.nn.functional.normalize(rn().view(1, steps, heads, 64), dim=-1).reshape(1, steps, heads * 64)
    ins = [torch.sigmoid(rn()), torch.sigmoid(rn()), kap, rn(), rn(), rn()]
    state = torch.randn(1, heads, 64, 64, generator=g, device="cuda")
    s_all, y_all, ckpt_all, sa_all = _forward(state, ins, heads, with_grad)
    for h in (0, heads - 1):
        one = [t[..., h * 64:(h + 1) * 64].contiguous() for t in ins]
        s_one, y_one, ckpt_one, sa_one = _forward(state[:, h:h + 1].contiguous(), one, 1, with_grad)
        assert torch.equal(y_all[..., h * 64:(h + 1) * 64], y_one) and torch.equal(s_all[:, h:h + 1], s_one)
        if with_grad:
            assert torch.equal(sa_all[..., h * 64:(h + 1) * 64], sa_one) and torch.equal(ckpt_all.view(heads, -1)[h], ckpt_one)
    if steps > 8:
        s_cut, y_a, _, _ = _forward(state, [t[:, :8].contiguous() for t in ins], heads, with_grad)
        s_end, y_b, _, _ = _forward(s_cut, [t[:, 8:].contiguous() for t in ins], heads, with_grad)
        assert torch.equal(torch.cat([y_a, y_b], 1), y_all) and torch.equal(s_end, s_all)
