"""Backward of heads wider than 128 whose dV items have a launch of their own (three dO slots, no V tile) beside one for dK: who takes it
(no GPU needed), its gradients at the edges of its tiles (64 queries, 128 keys, padded head dimensions) against the oracle in float32,
and against the form that makes both in one launch, which the same heads take one by one. Each item has the same products in the same order
either way, so the gradients are the same bits."""

import pytest
import torch

from _util import assert_within_2x
from fast_diffusion_attention import _lib, diffusion_attn_func, diffusion_attn_varlen_func
from oracle import diffusion_oracle as orc
from test_launch_choices import _choices
from test_parts_rule import _packed


def _apart(seqlen, heads, heads_k, d, **kw):
    return bool(_choices(seqlen, heads, heads_k, d, **kw) & _lib.FDA_CHOICE_DV_APART)


@pytest.mark.parametrize("d", [136, 192, 256])
def test_who_takes_it(d):
    for deterministic in (0, 1):
        assert _apart(16384, 8, 8, d, batch=2, deterministic=deterministic)
        assert _apart(1400, 16, 16, d, batch=2, deterministic=deterministic)
    assert _apart(heads=32, heads_k=8, d=d, **_packed([4095, 1203, 2750, 3391, 1876, 2049]))
    assert not _apart(1398, 16, 16, d, batch=2)                                  # short samples
    assert not _apart(heads=8, heads_k=8, d=d, **_packed([8192] + [300] * 40))   # most of them short
    assert not _apart(8192, 16, 4, d, batch=1)                                   # chains of four heads, most of the chip idle
    assert not _apart(16384, 8, 8, 128, batch=2)


def _grads(q, k, v, g, bs, softcap, cu, **kw):
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    if cu is None:
        out = diffusion_attn_func(*leaves, bs, softcap=softcap, **kw)
    else:
        longest = int((cu[1:] - cu[:-1]).max())
        out = diffusion_attn_varlen_func(*leaves, cu, cu, longest, longest, bs, softcap=softcap, **kw)
    return torch.autograd.grad(out, leaves, g)


def _check(q, k, v, bs, *, softcap=0.0, cu=None, picked=(0, -1)):
    g = torch.randn_like(q)
    heads_k, group = k.shape[-2], q.shape[-2] // k.shape[-2]
    got = _grads(q, k, v, g, bs, softcap, cu)
    again = _grads(q, k, v, g, bs, softcap, cu, deterministic=True)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
    assert _lib.device_status()[0] == 0
    for h in picked:
        h %= heads_k
        mine = [slice(h * group, (h + 1) * group), slice(h, h + 1), slice(h, h + 1)]
        one = [t[..., s, :].contiguous() for t, s in zip((q, k, v, g), mine + mine[:1])]
        mine = [t[..., s, :] for t, s in zip(got, mine)]
        for a, b in zip(mine, _grads(*one, bs, softcap, cu)):
            assert torch.equal(a, b)
        if cu is None:
            truth, plain = (orc.backward(*one, bs, softcap=softcap, **kw) for kw in ({}, dict(compute_dtype=q.dtype)))
        else:
            truth, plain = (orc.backward_varlen(*one, cu.tolist(), bs, softcap=softcap, **kw) for kw in ({}, dict(compute_dtype=q.dtype)))
        for name, a, t, pl in zip(("dq", "dk", "dv"), mine, truth, plain):
            assert_within_2x(name, a, t, pl)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,bs,heads,heads_k,d", [(700, 1, 16, 16, 256), (703, 9, 16, 16, 192), (1409, 64, 20, 10, 136),
                                                  (1471, 2000, 20, 10, 200), (1536, 1536, 10, 10, 256), (1473, 300, 10, 10, 256)])
def test_wide_heads(n, bs, heads, heads_k, d, dtype):
    torch.manual_seed(n)
    assert _apart(2 * n, heads, heads_k, d, batch=2, bs=bs) and not _apart(2 * n, heads // heads_k, 1, d, batch=2, bs=bs)
    q, k, v = (torch.randn(2, 2 * n, h, d, device="cuda", dtype=dtype) for h in (heads, heads_k, heads_k))
    _check(q, k, v, bs)


@pytest.mark.gpu
@pytest.mark.parametrize("softcap", [0.0, 4.0])
def test_wide_heads_packed(softcap):
    torch.manual_seed(7)
    ns = [2100, 1, 63, 2050, 1985, 2777]
    assert _apart(heads=12, heads_k=6, d=256, **_packed(ns)) and not _apart(heads=2, heads_k=1, d=256, **_packed(ns))
    cu = torch.tensor([0] + ns, device="cuda").cumsum(0).int() * 2
    q, k, v = (torch.randn(2 * sum(ns), h, 256, device="cuda", dtype=torch.bfloat16) for h in (12, 6, 6))
    _check(q, k, v, 48, softcap=softcap, cu=cu, picked=(3,))


@pytest.mark.gpu
def test_rows_of_other_samples_stay_out():
    torch.manual_seed(9)
    n, bs = 1430, 40
    q, k, v = (torch.randn(2, 2 * n, 10, 256, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    g = torch.randn_like(q)
    want = _grads(q, k, v, g, bs, 0.0, None)
    loud = [t.clone() for t in (q, k, v)]
    for t in loud:
        t[1] *= 100.0                                 # the other sample lies right behind the first
    assert all(torch.equal(a[0], b[0]) for a, b in zip(_grads(*loud, g, bs, 0.0, None), want))
