"""Calls with little work overlap the start of each kernel with the end of the one ahead. Calls of both kinds and all forms, queued one
after the other in one stream and in two without waiting in between, or replayed from a CUDA graph, give the bits that they give alone;
dq of the single-pass backward, whose partial sums are added in scheduling order, within one rounding step."""

import pytest
import torch

from _util import assert_same_gradients
from fast_diffusion_attention import _lib, diffusion_attn_func, diffusion_attn_varlen_func
from test_launch_choices import _overlaps

pytestmark = pytest.mark.gpu

BF, HF, F8 = torch.bfloat16, torch.float16, torch.float8_e4m3fn
# batch (or half lengths of packed samples), n, heads, heads_k, dim, dtype, softcap, deterministic, whether forward and backward overlap:
# rows x heads x head dim below, at and above 2^23, and every form of the backward (single pass with and without parts, split, dV apart)
CALLS = [
    (1, 40, 2, 2, 64, BF, 0.0, False, (True, True)), (2, 256, 4, 2, 128, HF, 0.0, False, (True, True)),
    (1, 700, 8, 2, 128, BF, 0.0, False, (True, True)), (2, 300, 4, 4, 96, BF, 20.0, False, (True, True)),
    (1, 512, 4, 4, 256, BF, 0.0, False, (True, True)), (2, 256, 4, 2, 128, BF, 0.0, True, (True, True)),
    (3, 200, 4, 4, 64, HF, 20.0, True, (True, True)), (2, 1400, 10, 10, 136, BF, 0.0, False, (True, True)),
    (1, 700, 30, 30, 192, BF, 0.0, False, (True, True)), (4, 512, 16, 16, 128, BF, 0.0, False, (True, False)),
    (4, 512, 16, 8, 128, BF, 0.0, False, (True, True)), (4, 520, 16, 8, 128, BF, 0.0, False, (False, False)),
    ((17, 300, 1, 128, 513), 0, 6, 2, 64, BF, 0.0, False, (True, True)), ((200, 0, 431, 77), 0, 4, 4, 256, BF, 0.0, False, (True, True)),
    ((90, 650, 3), 0, 4, 2, 128, HF, 20.0, True, (True, True)),
    (2, 300, 4, 2, 128, F8, 0.0, False, (True, True)), ((300, 64, 129), 0, 4, 4, 256, F8, 0.0, False, (True, True)),
]


def _inputs(call):
    b, n, h, hk, d, dtype, softcap, deterministic, overlap = call
    packed = isinstance(b, tuple)
    lead = (2 * sum(b),) if packed else (b, 2 * n)
    shape = dict(seqlen=2 * max(b), batch=len(b), total=2 * sum(b)) if packed else dict(seqlen=2 * n, batch=b)
    assert _overlaps(heads=h, heads_k=hk, d=d, bs=16, softcap=softcap, deterministic=int(deterministic), **shape) == overlap
    q, k, v = (torch.randn(*lead, x, d, device="cuda").to(dtype) for x in (h, hk, hk))
    g = None if dtype == F8 else torch.randn_like(q)
    cu = torch.tensor((0,) + b, device="cuda").cumsum(0).int() * 2 if packed else None
    return q, k, v, g, cu, (2 * max(b) if packed else 0), dict(softcap=softcap, deterministic=deterministic)


def _call(x, bs=16):
    q, k, v, g, cu, longest, kw = x
    leaves = [t.detach().requires_grad_(g is not None) for t in (q, k, v)]
    if cu is None:
        out = diffusion_attn_func(*leaves, bs, **kw)
    else:
        out = diffusion_attn_varlen_func(*leaves, cu, cu, longest, longest, bs, **kw)
    return (out.detach(),) + (torch.autograd.grad(out, leaves, g) if g is not None else ())


def _same(got, want, x):
    single_pass = x[0].shape[-1] <= 128 and not x[-1]["deterministic"]
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        assert_same_gradients(name, a, b, exact=name != "dq" or not single_pass)


@pytest.mark.parametrize("streams", [1, 2])
def test_queued_calls_give_the_bits_of_calls_alone(streams):
    torch.manual_seed(0)
    xs = [_inputs(c) for c in CALLS]
    want = []
    for x in xs:
        want.append(_call(x))
        torch.cuda.synchronize()
    queues = [torch.cuda.Stream() for _ in range(streams)]
    got = []
    for i in range(6 * len(xs)):
        with torch.cuda.stream(queues[i % streams]):
            got.append((i * 7 % len(xs), _call(xs[i * 7 % len(xs)])))
    torch.cuda.synchronize()
    for j, out in got:
        _same(out, want[j], xs[j])
    assert _lib.device_status()[0] == 0


@pytest.mark.parametrize("call", [CALLS[0], CALLS[2], CALLS[4], CALLS[7], CALLS[12]])
def test_captured_calls_give_the_bits_of_calls_alone(call):
    torch.manual_seed(1)
    x = _inputs(call)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            want = [t.clone() for t in _call(x)]
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _call(x)
    for _ in range(10):
        graph.replay()
    torch.cuda.synchronize()
    _same(got, want, x)
    assert _lib.device_status()[0] == 0
    del graph
