"""Chains of kernels that are launched behind one another, over the same buffers again and again: the results of the same calls with
the device waited for in between, on one stream, on two, and from a graph."""
import pytest
import torch

from pratchya_b200._nnx_impl import _module
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
