"""The same inputs many times over: every role of the kernels (TMA warp, MMA issuers, compute and epilogue
warpgroups) hands work to the others through barriers, and a missing dependency would show up as a result that
changes with the timing of a run. Outputs and gradients must be bitwise the same in every repetition, on shapes
that make the CTAs take many items each (item boundaries are where buffers change owners). The one exception is
dq of the default (deterministic=False) backward for head dims up to 128: its fp32 partial sums are added with
global reductions in scheduling order, as in the reference (mainloop_bwd_sm90_tma_gmma_ws.hpp:605-664 there), so
it may differ by one rounding step; with deterministic=True it is bitwise stable too."""

import pytest
import torch

from _util import assert_same_gradients
from fast_diffusion_attention import _lib, diffusion_attn_func, diffusion_attn_varlen_func

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _step(q, k, v, do, bs, cu=None, max_len=None, **kw):
    q, k, v = (t.detach().clone().requires_grad_(True) for t in (q, k, v))
    if cu is None:
        out, lse = diffusion_attn_func(q, k, v, bs, return_attn_probs=True, **kw)
    else:
        out, lse = diffusion_attn_varlen_func(q, k, v, cu, cu, max_len, max_len, bs, return_attn_probs=True, **kw)
    out.backward(do)
    return out.detach(), lse.detach(), q.grad, k.grad, v.grad


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("heads,heads_k,d,bs,n,batch", [
    (16, 16, 128, 256, 2048, 8),    # the benchmark shape: about 14 / 28 items per CTA
    (8, 2, 128, 96, 1100, 3),       # grouped heads, masked tiles, partial last tile
    (6, 6, 64, 32, 1500, 4),
    (4, 4, 256, 128, 1024, 2),
    (10, 10, 256, 64, 1500, 2),     # wide heads, samples long and heads many enough for dK and dV items in launches of their own
    (20, 10, 136, 96, 2100, 2),
])
def test_bitwise_stable_over_repetitions(heads, heads_k, d, bs, n, batch, deterministic):
    torch.manual_seed(7)
    q = torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    do = torch.randn_like(q)
    first = _step(q, k, v, do, bs, deterministic=deterministic)
    junk = torch.empty(64 << 20, device=DEV, dtype=torch.uint8)
    for rep in range(6):
        if rep % 2:
            junk.random_(0, 255)   # other work in between shifts the timing and the cache state
        again = _step(q, k, v, do, bs, deterministic=deterministic)
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), again, first):
            assert_same_gradients(f"{name} (repetition {rep})", a, b, exact=deterministic or d > 128 or name != "dq")
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0


@pytest.mark.parametrize("deterministic", [False, True])
def test_bitwise_stable_varlen_with_softcap(deterministic):
    torch.manual_seed(8)
    ns = [700, 64, 1300, 0, 257, 2048, 5, 900]
    cu = torch.tensor([0] + list(torch.tensor([2 * x for x in ns]).cumsum(0)), device=DEV, dtype=torch.int32)
    total = 2 * sum(ns)
    q = torch.randn(total, 8, 128, device=DEV, dtype=torch.float16)
    k = torch.randn(total, 4, 128, device=DEV, dtype=torch.float16)
    v = torch.randn(total, 4, 128, device=DEV, dtype=torch.float16)
    do = torch.randn_like(q)
    first = _step(q, k, v, do, 80, cu=cu, max_len=2 * max(ns), softcap=15.0, deterministic=deterministic)
    for rep in range(4):
        again = _step(q, k, v, do, 80, cu=cu, max_len=2 * max(ns), softcap=15.0, deterministic=deterministic)
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), again, first):
            assert_same_gradients(f"{name} (repetition {rep})", a, b, exact=deterministic or name != "dq")
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0


def test_sm_margin_changes_the_grid_not_the_result():
    """sm_margin leaves SMs free for other work (flash_api.cpp:168-170, :300-301 of the reference): fewer
    persistent CTAs walk the same items, every output is still produced by one item in one fixed order."""
    torch.manual_seed(9)
    q = torch.randn(2, 2 * 900, 8, 128, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(2, 2 * 900, 4, 128, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(2, 2 * 900, 4, 128, device=DEV, dtype=torch.bfloat16)
    do = torch.randn_like(q)
    base = _step(q, k, v, do, 64)
    for margin in (1, 20, 140, 1000):   # more than there are SMs leaves one CTA
        got = _step(q, k, v, do, 64, sm_margin=margin)
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, base):
            assert_same_gradients(f"{name} with sm_margin={margin}", a, b, exact=name != "dq")
    base = _step(q, k, v, do, 64, deterministic=True)
    for margin in (20, 1000):
        got = _step(q, k, v, do, 64, sm_margin=margin, deterministic=True)
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, base):
            assert_same_gradients(f"{name} with sm_margin={margin}, deterministic", a, b, exact=True)
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0


@pytest.mark.parametrize("dtype,softcap", [(torch.bfloat16, 0.0), (torch.bfloat16, 20.0), (torch.float16, 0.0),
                                           (torch.float8_e4m3fn, 0.0)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,bs", [(900, 64), (333, 20), (128, 1024)])
def test_one_or_two_query_tiles_per_item_give_the_same_result(n, bs, d, dtype, softcap):
    """A forward whose items of one 128-row query tile all find an SM takes those; with fewer SMs left to it the same call
    takes items of two. Each query tile sees the same sub-steps in the same order either way, batched or packed."""
    torch.manual_seed(12)
    heads, heads_k = 4, 2
    q, k, v = (torch.randn(1, 2 * n, h, d, device=DEV).to(dtype) for h in (heads, heads_k, heads_k))
    cu = torch.tensor([0, 2 * n], device=DEV, dtype=torch.int32)
    results = []
    for margin in (0, 147):
        results.append(diffusion_attn_func(q, k, v, bs, softcap=softcap, sm_margin=margin, return_attn_probs=True))
        out, lse = diffusion_attn_varlen_func(q[0], k[0], v[0], cu, cu, 2 * n, 2 * n, bs, softcap=softcap, sm_margin=margin,
                                              return_attn_probs=True)
        results.append((out[None], lse[None]))
    for out, lse in results[1:]:
        assert torch.equal(out, results[0][0]) and torch.equal(lse, results[0][1])


@pytest.mark.parametrize("heads,heads_k,d", [(32, 8, 64), (8, 8, 64), (32, 8, 128)])
def test_no_wait_expires_over_many_backward_passes(heads, heads_k, d):
    """The roles of the single-pass backward run a step apart; where one of them can be lapped by another, a wait by
    parity misses its phase now and then (a few launches in a thousand) and gives up after two seconds."""
    torch.manual_seed(10)
    n = 2048
    q = torch.randn(4, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(4, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(4, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    do = torch.randn_like(q)
    for _ in range(400):
        torch.autograd.grad(diffusion_attn_func(q, k, v, 64), (q, k, v), do)
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0


def test_first_call_of_a_new_thread():
    """A thread that has done no CUDA work has no current context, and with every allocation out of the cache nothing
    binds one before the tensor maps are encoded. Autograd threads are such threads."""
    import threading
    torch.manual_seed(11)
    q, k, v = (torch.randn(1, 512, 2, 64, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    want = diffusion_attn_func(q, k, v, 32)
    del want
    torch.cuda.synchronize()
    want = diffusion_attn_func(q, k, v, 32)
    spare = diffusion_attn_func(q, k, v, 32)
    del spare   # the thread's output comes from here
    got = []
    thread = threading.Thread(target=lambda: got.append(diffusion_attn_func(q, k, v, 32)))
    thread.start()
    thread.join()
    assert len(got) == 1 and torch.equal(got[0], want)


@pytest.mark.parametrize("heads,heads_k,d,deterministic", [(8, 2, 256, False), (10, 10, 256, False), (8, 2, 128, True)])
def test_no_wait_expires_over_many_split_backward_passes(heads, heads_k, d, deterministic):
    torch.manual_seed(12)
    n = 1500
    q = torch.randn(2, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k, v = (torch.randn(2, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
    do = torch.randn_like(q)
    for _ in range(300):
        torch.autograd.grad(diffusion_attn_func(q, k, v, 48, deterministic=deterministic), (q, k, v), do)
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0
