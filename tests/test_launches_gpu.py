"""Chains of kernels that are launched behind one another, over the same buffers again and again: the results of the same calls with
the device waited for in between, on one stream, on two, and from a graph."""
import pytest
import torch

from pratchya_b200._nnx_impl import _glue, _module
from pratchya_b200._nnx_impl._wkv7 import wkv_state_scan
from pratchya_b200._qualia import _ops, dequantize_impl, quantize_impl

pytestmark = pytest.mark.gpu


def _chain(xs, w, sync):
    outs = []
    for x in xs:
        layer = [lambda t: quantize_impl(t, (1, 128)), lambda t: dequantize_impl(*t, torch.float32, (1, 128)), lambda t: _module.linear_fp8(t, w, (128, 128)),
                 lambda t: _ops.fake_quantize_impl(t, (1, 128), torch.float32)]
        t = x
        for f in layer:
            t = f(t)
            if sync:
                torch.cuda.synchronize()
        outs.append(t)
    return outs


@pytest.mark.parametrize("rows,k,n", [(1, 1024, 512), (64, 1024, 1024), (1000, 512, 2048), (4096, 1024, 1024)])
def test_a_chain_without_waits_gives_the_same_bits(built_lib, rows, k, n):
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.randn(k, n, generator=g, device="cuda") * 0.02
    xs = [torch.randn(rows, k, generator=g, device="cuda") for _ in range(6)]
    with torch.no_grad():
        want = _chain(xs, w, True)
        for _ in range(5):
            assert all(torch.equal(a, b) for a, b in zip(_chain(xs, w, False), want))
        streams = [torch.cuda.Stream() for _ in range(2)]
        for _ in range(5):
            got = []
            for s in streams:
                s.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(s):
                    got.append(_chain(xs, w, False))
            for s in streams:
                torch.cuda.current_stream().wait_stream(s)
            for outs in got:
                assert all(torch.equal(a, b) for a, b in zip(outs, want))
        static = [x.clone() for x in xs]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = _chain(static, w, False)
        for shift in range(3):
            for i, t in enumerate(static):
                t.copy_(xs[(i + shift) % len(xs)])
            graph.replay()
            assert all(torch.equal(o, want[(i + shift) % len(xs)]) for i, o in enumerate(outs))


class _Step:
    """A training step of what a block is made of, over `steps` tokens of 16 heads: three kernels with a memset in front, a Linear whose cotangent is bf16
    (its literal dots with operands made ready and parts that are added, or fp8 gradients from 1024 tokens on), a low-rank layer (the other literal
    dots), a deep product of few rows (a cluster's), the scan with the kernels around it, the loss; forward and all gradients."""
    heads, chans = 16, 1024

    def __init__(self, steps):
        g = torch.Generator(device="cuda").manual_seed(steps)
        rn = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std
        self.steps, c = steps, self.chans
        self.w = [rn(c, c, std=0.03), rn(c, 128, std=0.03), rn(128, c, std=0.03), rn(4096, 512, std=0.02), rn(c, 2048, std=0.03), torch.rand(c, generator=g, device="cuda"), 1 + rn(c, std=0.1),
                  rn(c, std=0.1), 1 + rn(c, std=0.1), rn(c, std=0.1)]
        angles = torch.outer(torch.arange(steps, device="cuda", dtype=torch.float32), 1e4 ** (-torch.arange(0, 64, 2, device="cuda", dtype=torch.float32) / 64))
        self.tables = torch.cos(angles), torch.sin(angles)
        self.ids = torch.randint(0, 2048, (1, steps), generator=g, device="cuda")
        self.xs = [rn(1, steps, c) for _ in range(3)]
        self.deep = rn(64, 4096)

    def __call__(self, x, wait=False):
        def done(t):                  # the device is waited for behind this op, and behind what makes this gradient
            if wait:
                torch.cuda.synchronize()
                if t.requires_grad:
                    t.register_hook(lambda g: torch.cuda.synchronize())
            return t
        x = x.detach().requires_grad_(True)
        w1, down, up, deep, head, mix, rk, bias, scale, bonus = w = [t.detach().requires_grad_(True) for t in self.w]
        blocks = [done(t) for t in quantize_impl(x.detach()[0, :self.steps // 8 * 8], (8, 64))]
        few = done(_module.linear_fp8(self.deep, deep, (128, 128)))
        a = done(done(_module.linear_fp8(x.bfloat16(), w1, (128, 128))).float())
        b = done(_module.linear_fp8(done(torch.tanh(done(_module.linear_fp8(a, down, (128, 1), fake_quant_output=False)))), up, (128, 1), fake_quant_output=False))
        decay, iclr, kappa, kt, v, r, k = [done(t) for t in _glue.wkv_prepare(a, b, x, a, b, x, a, *self.tables, rk, mix, self.heads)]
        state, y = [done(t) for t in wkv_state_scan(None, decay, iclr, kappa, kt, v, r, self.heads)]
        out = done(_glue.wkv_finish(y, r, k, v, a, scale, bias, bonus, 1e-5 * self.heads, self.heads))
        loss = done(_glue.smoothed_cross_entropy(done(_module.linear_fp8(out, head, (128, 128))), self.ids))
        leaves = [x, *w]
        grads = torch.autograd.grad(loss + 1e-3 * (state.mean() + few.mean()), leaves)
        if wait:
            torch.cuda.synchronize()
        return [*(t.view(torch.uint8) if t.element_size() == 1 else t for t in blocks), few.detach(), out.detach(), state.detach(), loss.detach(), *grads]


@pytest.mark.parametrize("steps", [40, 600, 1024])
def test_training_steps_without_waits_give_the_same_bits(built_lib, steps):
    step = _Step(steps)
    want = [step(x, wait=True) for x in step.xs]
    same = lambda got, ref: all(torch.equal(a, b) for a, b in zip(got, ref, strict=True))
    assert not same(want[0], want[1])
    for _ in range(4):                # buffers of one step serve the next with other values
        assert all(same(step(x), ref) for x, ref in zip(step.xs, want))
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(3):
        got = []
        for s, x in zip(streams, step.xs):
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(step(x))
        for s in streams:
            torch.cuda.current_stream().wait_stream(s)
        assert all(same(outs, ref) for outs, ref in zip(got, want))
    # captured, one step on the capturing stream and one on a stream that leaves it and comes back, between kernels of both
    static = [x.clone() for x in step.xs[:2]]
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        first = quantize_impl(static[0][0], (1, 128))
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            b = step(static[1])
        a = step(static[0])
        torch.cuda.current_stream().wait_stream(side)
        last = dequantize_impl(*first, torch.float32, (1, 128)) + b[-1].sum() * 0
    for shift in range(3):
        for i, t in enumerate(static):
            t.copy_(step.xs[(i + shift) % 3])
        graph.replay()
        torch.cuda.synchronize()
        assert same(a, want[shift % 3]) and same(b, want[(1 + shift) % 3])
        assert torch.equal(last, dequantize_impl(*quantize_impl(static[0][0], (1, 128)), torch.float32, (1, 128)))
