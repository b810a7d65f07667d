"""Single-pass backward where the query heads of a group are dealt out to several CTAs and their dK and dV added up afterwards:
few tokens, few KV heads, more than 32 steps a key tile (the smallest shapes here, with smaller groups, are just below that and
stay whole). One head a part and several, groups with and without small divisors, head dimensions that do not fill a piece,
ends of halves inside a piece of 32 rows, packed batches with empty samples, strided outputs; dk and dv are the same in every
run."""

import pytest
import torch

from fast_diffusion_attention import diffusion_attn_func
from fast_diffusion_attention.interface import diffusion_attn_varlen_qkvpacked_func
from oracle import diffusion_oracle as orc
from test_gpu_bwd import check_backward
from test_parts_rule import parts

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("d", [128, 64, 96, 40, 8])
@pytest.mark.parametrize("heads,heads_k", [(32, 1), (24, 2), (5, 1), (8, 1), (12, 2)])
@pytest.mark.parametrize("batch,n,bs", [(1, 1, 1), (1, 100, 32), (2, 129, 129), (1, 300, 8), (2, 511, 64)])
def test_parts_of_a_group(batch, n, bs, heads, heads_k, d):
    torch.manual_seed(n + heads)
    q, k, v = (torch.randn(batch, 2 * n, h, d, device=DEV, dtype=torch.bfloat16) for h in (heads, heads_k, heads_k))
    check_backward(q, k, v, bs)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    runs = [torch.autograd.grad(diffusion_attn_func(*leaves, bs), leaves, torch.ones_like(q)) for _ in range(3)]
    for run in runs[1:]:
        assert torch.equal(run[1], runs[0][1]) and torch.equal(run[2], runs[0][2])


@pytest.mark.parametrize("d", [128, 64, 96])
@pytest.mark.parametrize("layout", ["batched", "packed"])
@pytest.mark.parametrize("heads,heads_k,batch,n,bs,n_parts", [
    (64, 8, 4, 300, 24, 2),      # four heads a part
    (24, 4, 3, 700, 64, 3),      # two
    (32, 2, 3, 1000, 300, 4),    # four
    (24, 4, 6, 400, 100, 2),     # three
])
def test_parts_of_several_heads(heads, heads_k, batch, n, bs, n_parts, layout, d):
    lead = (batch, 2 * n) if layout == "batched" else (2 * batch * n,)
    cu = None if layout == "batched" else torch.arange(0, 2 * batch * n + 1, 2 * n, device=DEV, dtype=torch.int32)
    assert parts(2 * n, heads, heads_k, d, batch=batch, total=None if cu is None else 2 * batch * n, bs=bs)[0] == n_parts
    torch.manual_seed(n)
    q, k, v = (torch.randn(*lead, h, d, device=DEV, dtype=torch.bfloat16) for h in (heads, heads_k, heads_k))
    first = check_backward(q, k, v, bs, cu=cu)
    torch.manual_seed(n)
    q, k, v = (torch.randn(*lead, h, d, device=DEV, dtype=torch.bfloat16) for h in (heads, heads_k, heads_k))
    again = check_backward(q, k, v, bs, cu=cu)
    assert torch.equal(again[1], first[1]) and torch.equal(again[2], first[2])


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("softcap", [0.0, 8.0])
def test_parts_packed(d, softcap):
    torch.manual_seed(d)
    ns = [70, 0, 1, 400, 33, 128]
    cu = torch.tensor([0] + list(torch.tensor([2 * x for x in ns]).cumsum(0)), device=DEV, dtype=torch.int32)
    q, k, v = (torch.randn(2 * sum(ns), h, d, device=DEV, dtype=torch.float16) for h in (6, 1, 1))
    check_backward(q, k, v, 16, softcap=softcap, cu=cu)


def test_parts_into_one_packed_gradient():
    """The gradient of a packed projection is written in place, with strides of its own."""
    torch.manual_seed(1)
    ns, heads, heads_k, d, bs = [90, 200], 32, 2, 64, 16
    cu = torch.tensor([0, 180, 580], device=DEV, dtype=torch.int32)
    qkv = torch.randn(580, heads + 2 * heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = diffusion_attn_varlen_qkvpacked_func(qkv, cu, 400, bs, num_heads_q=heads)
    g = torch.randn_like(out)
    grad, = torch.autograd.grad(out, qkv, g)
    parts = qkv.detach().split([heads, heads_k, heads_k], 1)
    want = torch.cat(orc.backward_varlen(*parts, g, cu.tolist(), bs), 1)
    plain = torch.cat(orc.backward_varlen(*parts, g, cu.tolist(), bs, compute_dtype=torch.bfloat16), 1)
    for a, t, p in zip(grad.split([heads, heads_k, heads_k], 1), want.split([heads, heads_k, heads_k], 1),
                       plain.split([heads, heads_k, heads_k], 1)):
        assert (a.float() - t).abs().max() <= 2 * (p.float() - t).abs().max() + 1e-3
