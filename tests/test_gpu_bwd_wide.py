"""Backward of heads wider than 128 that makes dK and dQ in one kernel and dV in another: the shapes that take it (as the workspace
shows, no GPU needed) and, at the edges of its tiles (64 queries, 128 keys, the 64 columns of a panel, a head dimension that ends in
the first or second half of dQ^T), its gradients against the split form. dK and dV have the same products in the same order there,
so they are the same bits; dQ's partial sums are added in another order, in fp32: one rounding step, and where terms cancel a few
2^-24 of the largest."""

import pytest
import torch

from fast_diffusion_attention import diffusion_attn_func, diffusion_attn_varlen_func
from test_parts_rule import _bytes, _packed


def _wide(seqlen, heads, heads_k, d, **kw):
    return _bytes(seqlen, heads, heads_k, d, **kw) > _bytes(seqlen, heads, heads_k, d, deterministic=1, **kw)


@pytest.mark.parametrize("d", [136, 192, 256])
def test_who_takes_it(d):
    assert _wide(16384, 8, 8, d, batch=2)
    assert _wide(2800, 20, 10, d, batch=2)
    assert _wide(heads=32, heads_k=8, d=d, **_packed([4095, 1203, 2750, 3391, 1876, 2049]))
    assert not _wide(2798, 20, 10, d, batch=2)                                  # short samples
    assert not _wide(heads=8, heads_k=8, d=d, **_packed([8192] + [500] * 40))   # most of them short
    assert not _wide(heads=8, heads_k=8, d=d, **_packed([512] * 64, 16384))     # a loose bound
    assert not _wide(8192, 16, 4, d, batch=1)                                   # chains of four heads, most of the chip idle
    assert not _wide(4096, 8, 1, d, batch=4)


def _check(q, k, v, bs, *, softcap=0.0, cu=None):
    g = torch.randn_like(q)

    def grads(deterministic):
        leaves = [t.detach().requires_grad_() for t in (q, k, v)]
        kw = dict(softcap=softcap, deterministic=deterministic)
        if cu is None:
            out = diffusion_attn_func(*leaves, bs, **kw)
        else:
            longest = int((cu[1:] - cu[:-1]).max())
            out = diffusion_attn_varlen_func(*leaves, cu, cu, longest, longest, bs, **kw)
        return torch.autograd.grad(out, leaves, g)

    (dq, dk, dv), (dq0, dk0, dv0) = grads(False), grads(True)
    assert torch.equal(dk, dk0) and torch.equal(dv, dv0)
    step = 2.0 ** (-7 if q.dtype == torch.bfloat16 else -10)
    a, b = dq.float(), dq0.float()
    assert bool(((a - b).abs() <= step * b.abs() + 1e-5 * b.abs().max()).all())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,bs,heads,heads_k,d", [(1400, 1, 10, 10, 256), (1409, 64, 20, 10, 136), (1473, 300, 10, 10, 192),
                                                  (1536, 1536, 10, 10, 256), (1471, 2000, 20, 10, 200), (1503, 17, 30, 10, 256)])
def test_wide_heads(n, bs, heads, heads_k, d, dtype):
    torch.manual_seed(n)
    assert _wide(2 * n, heads, heads_k, d, batch=2, bs=bs)
    q, k, v = (torch.randn(2, 2 * n, h, d, device="cuda", dtype=dtype) for h in (heads, heads_k, heads_k))
    _check(q, k, v, bs)


@pytest.mark.gpu
@pytest.mark.parametrize("softcap", [0.0, 4.0])
def test_wide_heads_packed(softcap):
    torch.manual_seed(7)
    ns = [2100, 1, 63, 2050, 1985, 2777]
    kw = _packed(ns)
    assert _wide(heads=12, heads_k=6, d=256, **kw)
    cu = torch.tensor([0] + ns, device="cuda").cumsum(0).int() * 2
    q, k, v = (torch.randn(2 * sum(ns), h, 256, device="cuda", dtype=torch.bfloat16) for h in (12, 6, 6))
    _check(q, k, v, 48, softcap=softcap, cu=cu)


@pytest.mark.gpu
def test_rows_of_other_samples_stay_out():
    torch.manual_seed(9)
    n, bs = 1430, 40
    q, k, v = (torch.randn(2, 2 * n, 10, 256, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    g = torch.randn_like(q)

    def grads(x):
        leaves = [t.detach().requires_grad_() for t in x]
        return torch.autograd.grad(diffusion_attn_func(*leaves, bs), leaves, g)

    want = grads((q, k, v))
    loud = [t.clone() for t in (q, k, v)]
    for t in loud:
        t[1] *= 100.0                                 # the other sample lies right behind the first
    dq, dk, dv = grads(loud)
    assert torch.equal(dk[0], want[1][0]) and torch.equal(dv[0], want[2][0])
    assert (dq[0].float() - want[0][0].float()).abs().max() <= 2.0 ** -7 * want[0][0].float().abs().max()
