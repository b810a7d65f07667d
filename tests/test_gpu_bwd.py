"""Backward parity on the GPU through the public API (autograd -> C ABI) against the oracle's explicit
gradients. Tolerance, as in the reference's tests (tests/test_diffusion_attn.py:76-104 there): for dq, dk, dv
max|got - truth| <= 2 * max|plain - truth| + a few ulps, with truth = float32 oracle on the same inputs and
plain = the oracle evaluated in the input precision. Also: bitwise reproducibility, packed == batched."""

import pytest
import torch

from _util import assert_same_gradients, assert_within_2x
from fast_diffusion_attention import _lib, diffusion_attn_func, diffusion_attn_varlen_func
from oracle import diffusion_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [(2, 128, 4), (1, 256, 32), (3, 100, 3), (2, 333, 16), (1, 517, 7), (1, 64, 64), (1, 300, 128),
          (2, 191, 200), (1, 1, 1), (2, 5, 2), (1, 1024, 1), (1, 777, 64), (1, 512, 256), (1, 640, 128)]


def check_backward(q, k, v, bs, softcap=0.0, cu=None, deterministic=False):
    g = torch.randn_like(q)
    q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
    if cu is None:
        out = diffusion_attn_func(q, k, v, bs, softcap=softcap, deterministic=deterministic)
        truth = orc.backward(q.detach(), k.detach(), v.detach(), g, bs, softcap=softcap)
        plain = orc.backward(q.detach(), k.detach(), v.detach(), g, bs, softcap=softcap, compute_dtype=q.dtype)
    else:
        ms = int((cu[1:] - cu[:-1]).max().item())
        out = diffusion_attn_varlen_func(q, k, v, cu, cu, ms, ms, bs, softcap=softcap, deterministic=deterministic)
        truth = orc.backward_varlen(q.detach(), k.detach(), v.detach(), g, cu.tolist(), bs, softcap=softcap)
        plain = orc.backward_varlen(q.detach(), k.detach(), v.detach(), g, cu.tolist(), bs, softcap=softcap,
                                    compute_dtype=q.dtype)
    grads = torch.autograd.grad(out, (q, k, v), g)
    assert _lib.device_status()[0] == 0
    for name, got, t, pl in zip(("dq", "dk", "dv"), grads, truth, plain):
        assert not torch.isnan(got.float()).any(), name
        assert_within_2x(name, got, t, pl)
    return grads


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("heads,heads_k", [(4, 4), (6, 2), (4, 1)])
@pytest.mark.parametrize("batch,n,bs", SHAPES)
def test_backward_bf16(batch, n, bs, heads, heads_k, d):
    torch.manual_seed(n * 1000 + bs)
    q = torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("batch,n,bs", [(2, 333, 16), (1, 300, 128), (1, 777, 64)])
def test_backward_fp16_softcap(batch, n, bs, d):
    torch.manual_seed(n + bs)
    q, k, v = (torch.randn(batch, 2 * n, h, d, device=DEV, dtype=torch.float16) for h in (4, 2, 2))
    check_backward(q, k, v, bs, softcap=15.0)
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("bs", [1, 4, 13, 64, 160])
def test_backward_varlen(bs, deterministic, d):
    torch.manual_seed(bs)
    ns = [17, 300, 1, 128, 513, 64, 2, 255, 0]
    cu = torch.tensor([0] + list(torch.tensor([2 * x for x in ns]).cumsum(0)), device=DEV, dtype=torch.int32)
    total = 2 * sum(ns)
    q = torch.randn(total, 6, d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(total, 2, d, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(total, 2, d, device=DEV, dtype=torch.bfloat16)
    check_backward(q, k, v, bs, cu=cu, deterministic=deterministic)


@pytest.mark.parametrize("d", [64, 128])
def test_packed_equals_batched_bitwise(d):
    """Packing equal-length samples gives exactly the batched result (out, lse and all gradients)."""
    torch.manual_seed(0)
    batch, n, heads, heads_k, bs = 3, 200, 4, 2, 8
    q = torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn_like(q)
    out, lse = diffusion_attn_func(q, k, v, bs, deterministic=True, return_attn_probs=True)
    grads = torch.autograd.grad(out, (q, k, v), g)
    cu = torch.arange(0, batch * 2 * n + 1, 2 * n, device=DEV, dtype=torch.int32)
    qv, kv, vv = [x.detach().reshape(-1, *x.shape[2:]).requires_grad_() for x in (q, k, v)]
    out_v, lse_v = diffusion_attn_varlen_func(qv, kv, vv, cu, cu, 2 * n, 2 * n, bs, deterministic=True,
                                              return_attn_probs=True)
    grads_v = torch.autograd.grad(out_v, (qv, kv, vv), g.reshape(-1, *g.shape[2:]))
    assert torch.equal(out.reshape(-1, *out.shape[2:]), out_v)
    assert torch.equal(lse.permute(1, 0, 2).reshape(heads, -1), lse_v)
    for x, y in zip(grads, grads_v):
        assert torch.equal(x.reshape(-1, *x.shape[2:]), y)


@pytest.mark.parametrize("heads,heads_k", [(4, 4), (8, 2)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_backward_bitwise_reproducible(heads, heads_k, deterministic):
    torch.manual_seed(1)
    batch, n, bs, d = 2, 700, 4, 128
    q = torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn_like(q)

    def run():
        out = diffusion_attn_func(q, k, v, bs, deterministic=deterministic)
        return torch.autograd.grad(out, (q, k, v), g)

    ref = run()
    for _ in range(4):
        for name, x, y in zip(("dq", "dk", "dv"), run(), ref):
            # without `deterministic` dq comes from global fp32 adds in scheduling order (one rounding step of slack)
            assert_same_gradients(name, x, y, exact=deterministic or name != "dq")


def test_backward_matches_golden_fixture():
    """Gradients of the bf16 golden case produced by the reference's reference.py + autograd (tests/golden)."""
    from _util import load_golden, make_inputs
    from golden.make_golden import DENSE_CASES
    name = "bf16_gqa"
    B, n, H, Hk, d, bs, cap, scale, dt = DENSE_CASES[name]
    gold = load_golden("attention_golden.npz")
    q, k, v, do = make_inputs(int(gold[f"{name}/seed"]), (B, 2 * n, H, d), (B, 2 * n, Hk, d), torch.bfloat16, DEV)
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    out = diffusion_attn_func(q, k, v, bs)
    grads = torch.autograd.grad(out, (q, k, v), do)
    plain = orc.backward(q.detach(), k.detach(), v.detach(), do, bs, compute_dtype=torch.bfloat16)
    for key, got, pl in zip(("dq", "dk", "dv"), grads, plain):
        truth = torch.from_numpy(gold[f"{name}/{key}"]).to(DEV)
        # the golden gradients were taken through a bf16-rounded forward output; allow that rounding too
        assert_within_2x(key, got, truth, pl, atol=3e-2)


@pytest.mark.parametrize("heads,heads_k", [(4, 4), (4, 2)])
@pytest.mark.parametrize("batch,n,bs", [(1, 256, 32), (2, 333, 16), (1, 517, 7), (1, 300, 128), (1, 640, 256), (2, 5, 2)])
def test_backward_head_dim_256(batch, n, bs, heads, heads_k):
    """Head dimension 256: the dK/dV kernel makes two passes over the d halves, the dQ kernel uses 64-key tiles."""
    torch.manual_seed(n * 7 + bs)
    q = torch.randn(batch, 2 * n, heads, 256, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(batch, 2 * n, heads_k, 256, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(batch, 2 * n, heads_k, 256, device=DEV, dtype=torch.bfloat16)
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("d", [80, 96, 112, 160, 192, 224])
@pytest.mark.parametrize("bs", [1, 4, 37])
def test_backward_padded_head_dims(bs, d):
    """Head dimensions between the kernel sizes are padded inside the kernels (zero-filled TMA columns); the
    reference tests the same dims (tests/test_diffusion_attn.py:124-134 there)."""
    torch.manual_seed(d)
    batch, n, heads, heads_k = 2, 211, 4, 2
    q = torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(batch, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16)
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("d", [136, 256])
@pytest.mark.parametrize("n,bs", [(1, 1), (63, 63), (64, 64), (65, 8), (129, 300), (700, 9)])
def test_backward_wide_heads_sub_steps(n, bs, d):
    """Head dimensions above 128: dK and dV are items of their own over sub-steps of 64 queries, with two slots for Q, one
    for dO and four for the statistics. From one sub-step to more than the slots, whole and partial ones."""
    torch.manual_seed(n + d)
    q, k, v = (torch.randn(2, 2 * n, h, d, device=DEV, dtype=torch.bfloat16) for h in (4, 1, 1))
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("d", [96, 128])
@pytest.mark.parametrize("bs", [5, 64])
def test_backward_many_short_items(bs, d):
    """Items of one or two steps, several per CTA: the next item is taken, worked out and its V loaded while the last steps of
    the one before are still under way, and the drain warps go from one item's dK and dV to the next one's dQ."""
    torch.manual_seed(bs + d)
    ns = [(i * 37) % 131 + 1 for i in range(160)]
    cu = torch.tensor([0] + list(torch.tensor([2 * x for x in ns]).cumsum(0)), device=DEV, dtype=torch.int32)
    q, k, v = (torch.randn(2 * sum(ns), h, d, device=DEV, dtype=torch.bfloat16) for h in (4, 2, 2))
    check_backward(q, k, v, bs, cu=cu)


@pytest.mark.parametrize("n,max_n", [(512, 512), (512, 1500), (500, 1600), (512, 5000)])
def test_backward_loose_max_seqlen(n, max_n):
    """max_seqlen may be any upper bound. The dQ accumulator (67 MB here) is zeroed by the preprocess up to a padding of three
    times the rows and by a fill of its own beyond; twice in a row, so that the second call finds the first one's sums."""
    torch.manual_seed(n + max_n)
    batch, heads, d, bs = 8, 16, 128, 64
    q, k, v, g = (torch.randn(batch, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16) for _ in range(4))
    leaves = [x.requires_grad_() for x in (q, k, v)]
    want = torch.autograd.grad(diffusion_attn_func(*leaves, bs), leaves, g)
    cu = torch.arange(0, batch * 2 * n + 1, 2 * n, device=DEV, dtype=torch.int32)
    flat = [x.detach().flatten(0, 1).requires_grad_() for x in (q, k, v)]
    for _ in range(2):
        out = diffusion_attn_varlen_func(*flat, cu, cu, 2 * max_n, 2 * max_n, bs)
        got = torch.autograd.grad(out, flat, g.flatten(0, 1))
        for name, a, b in zip(("dq", "dk", "dv"), got, want):
            assert_same_gradients(name, a.unflatten(0, (batch, -1)), b, exact=name != "dq")
    assert _lib.device_status()[0] == 0
