"""Calls with little work overlap the start of each kernel with the end of the one ahead. Calls of both kinds, queued one after the
other in one stream and in two without waiting in between, give the bits that they give alone."""

import pytest
import torch

from fast_diffusion_attention import diffusion_attn_func, diffusion_attn_varlen_func

pytestmark = pytest.mark.gpu

# rows x heads x head dim below, at and above 2^23
SHAPES = [(1, 40, 2, 2, 64), (2, 256, 4, 2, 128), (1, 512, 4, 4, 256), (4, 512, 16, 8, 128), (4, 520, 16, 8, 128)]


def _call(x, bs=16):
    q, k, v, g, cu = x
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    if cu is None:
        out = diffusion_attn_func(*leaves, bs)
    else:
        n = int(leaves[0].shape[0] // (cu.numel() - 1))
        out = diffusion_attn_varlen_func(*leaves, cu, cu, n, n, bs)
    _, dk, dv = torch.autograd.grad(out, leaves, g)
    return out, dk, dv


def _inputs(shape, packed):
    b, n, h, hk, d = shape
    lead = (b * 2 * n,) if packed else (b, 2 * n)
    q, k, v, g = (torch.randn(*lead, x, d, device="cuda", dtype=torch.bfloat16) for x in (h, hk, hk, h))
    cu = torch.arange(0, b + 1, device="cuda", dtype=torch.int32) * (2 * n) if packed else None
    return q, k, v, g, cu


@pytest.mark.parametrize("streams", [1, 2])
def test_queued_calls_give_the_bits_of_calls_alone(streams):
    torch.manual_seed(0)
    xs = [_inputs(s, packed) for s in SHAPES for packed in (False, True)]
    want = []
    for x in xs:
        want.append(_call(x))
        torch.cuda.synchronize()
    queues = [torch.cuda.Stream() for _ in range(streams)]
    got = []
    for i in range(60):
        with torch.cuda.stream(queues[i % streams]):
            got.append((i * 7 % len(xs), _call(xs[i * 7 % len(xs)])))
    torch.cuda.synchronize()
    for j, out in got:
        assert all(torch.equal(a, b) for a, b in zip(out, want[j]))
