"""The scan's forward layouts (16 or 32 rows of a head per CTA for few heads, halves of a head around one wave of them, a whole head for many)
and the backward kernel's half chunks, over lengths around the chunk of eight, against the recurrence in 64 bits."""
import pytest
import torch

from pratchya_b200._nnx_impl._wkv7 import wkv_state_scan

pytestmark = pytest.mark.gpu


def _recurrence(state, ins, n):
    b, t, c = ins[0].shape
    w, a, kap, kt, v, r = (x.reshape(b, t, n, 64) for x in ins)
    ys = []
    for i in range(t):
        sa = torch.einsum("bnij,bnj->bni", state, kap[:, i])
        state = state * w[:, i].unsqueeze(-2) - sa.unsqueeze(-1) * (a[:, i] * kap[:, i]).unsqueeze(-2) + v[:, i].unsqueeze(-1) * kt[:, i].unsqueeze(-2)
        ys.append(torch.einsum("bnij,bnj->bni", state, r[:, i]))
    return state, torch.stack(ys, 1).reshape(b, t, c)


@pytest.mark.parametrize("batch,steps,heads", [(1, 1, 1), (1, 2, 3), (2, 8, 2), (1, 9, 2), (1, 17, 5), (3, 24, 32), (4, 12, 33), (1, 13, 130)])
@pytest.mark.parametrize("with_grad", [False, True])
def test_scan_against_the_recurrence(built_lib, batch, steps, heads, with_grad):
    g = torch.Generator(device="cuda").manual_seed(steps * 100 + heads)
    rn = lambda: torch.randn(batch, steps, heads * 64, generator=g, device="cuda")
    k = rn()
    kap = torch.nn.functional.normalize(k.view(batch, steps, heads, 64), dim=-1).reshape(k.shape)
    ins = [torch.exp(-torch.exp(rn() - 2)), torch.sigmoid(rn()), kap, k, rn(), rn()]
    state = torch.randn(batch, heads, 64, 64, generator=g, device="cuda") * 0.3
    leaves = [t.clone().requires_grad_(with_grad) for t in (state, *ins)]
    s_out, y = wkv_state_scan(leaves[0], *leaves[1:], heads)
    ref = [t.double().requires_grad_(with_grad) for t in (state, *ins)]
    s_ref, y_ref = _recurrence(ref[0], ref[1:], heads)
    # 64-term f32 sums of values of this size, their errors carried over `steps` contracting updates: 1e-7 observed, 64 * 2^-24 allowed
    close = lambda got, want: (got.double() - want).abs().max() <= 4e-6 * want.abs().max()
    assert close(s_out.detach(), s_ref.detach()) and close(y.detach(), y_ref.detach())
    if with_grad:
        gy, gs = rn(), torch.randn_like(state)
        got = torch.autograd.grad((y, s_out), leaves, (gy, gs))
        want = torch.autograd.grad((y_ref, s_ref), ref, (gy.double(), gs.double()))
        for name, u, v in zip(("state", "decay", "iclr", "removal_k", "replacement_k", "v", "r"), got, want):
            assert (u.double() - v).abs().max() <= 2e-5 * v.abs().max(), name


@pytest.mark.parametrize("heads,steps", [(1, 5), (2, 64), (40, 13), (130, 24)])
def test_what_a_timestep_writes_where_it_erases_something_larger(built_lib, heads, steps):
    """w = a = 1 and unit keys: every timestep erases a column of a state near 1e4 exactly and writes v there, of size one.  The
    column and the output are v to the last bit, and dr = S_t^T dy is as accurate as a sum of that column (64 products and
    additions), none of which survives where the write meets the old state before the erasure does."""
    g = torch.Generator(device="cuda").manual_seed(heads)
    shape = (1, steps, heads * 64)
    unit = torch.zeros(1, steps, heads, 64, device="cuda")
    for t in range(steps):
        unit[:, t, :, (5 * t) % 64] = 1.0
    unit = unit.reshape(shape)
    ones, v = torch.ones(shape, device="cuda"), torch.randn(shape, generator=g, device="cuda")
    state = 1e4 * torch.randn(1, heads, 64, 64, generator=g, device="cuda")
    leaves = [t.clone().requires_grad_(True) for t in (state, ones, ones, unit, unit, v, unit)]
    s_out, y = wkv_state_scan(leaves[0], *leaves[1:], heads)
    assert torch.equal(y, v)
    want = state.clone()
    for t in range(steps):
        want[..., (5 * t) % 64] = v.view(1, steps, heads, 64)[:, t]
    assert torch.equal(s_out, want)
    dy = torch.randn(shape, generator=g, device="cuda")
    dr = torch.autograd.grad(y, leaves[6], dy)[0].view(1, steps, heads, 64).double()
    v64, dy64 = v.view(1, steps, heads, 64).double(), dy.view(1, steps, heads, 64).double()
    for t in range(steps):
        got = dr[:, t, :, (5 * t) % 64]
        assert ((got - (v64[:, t] * dy64[:, t]).sum(-1)).abs() <= 65 * 2.0 ** -24 * (v64[:, t] * dy64[:, t]).abs().sum(-1)).all(), t


@pytest.mark.parametrize("heads", [1, 60, 100, 160, 230])
@pytest.mark.parametrize("iclr,decay,outlier", [(1.0, 1.0, 64.0), (1.0, 1.0, 1e6), (0.95, 0.99, 64.0), (0.95, 0.99, 1e4)])
def test_the_timesteps_after_a_large_value_is_erased(built_lib, heads, iclr, decay, outlier):
    """One key for all timesteps, read by itself, and a value far larger than the others in one of them.  The timestep behind it erases
    what it wrote and keeps that write's rounding, 2^-24 of its size, which the next one reads in the stored state and erases with
    it.  From there on each timestep is as accurate as its own sums: some twenty roundings of what it reads and of what it writes,
    as a 2-norm over the rows no more than 8 * 2^-24 of both (1 to 2 seen)."""
    steps = 24
    g = torch.Generator(device="cuda").manual_seed(heads)
    shape = (1, steps, heads * 64)
    key = torch.nn.functional.normalize(torch.randn(1, 1, heads, 64, generator=g, device="cuda"), dim=-1).expand(1, steps, heads, 64).reshape(shape).contiguous()
    full = lambda x: torch.full(shape, x, device="cuda")
    v0 = torch.randn(shape, generator=g, device="cuda")
    norm = lambda x: x.view(steps, heads, 64).double().norm(dim=-1)
    for at in range(5, 13):           # wherever in a chunk of eight it comes
        v = v0.clone()
        v[:, at] *= outlier
        ins = [full(decay), full(iclr), key, key, v, key]
        _, y = wkv_state_scan(None, *ins, heads)
        _, ref = _recurrence(torch.zeros(1, heads, 64, 64, device="cuda", dtype=torch.float64), [x.double() for x in ins], heads)
        error, size = norm(y - ref), norm(ref)
        for t in [*range(1, at), *range(at + 2, steps)]:
            assert (error[t] <= 8 * 2.0 ** -24 * (size[t] + size[t - 1])).all(), (at, t, (error[t] / (size[t] + size[t - 1])).max().item())
