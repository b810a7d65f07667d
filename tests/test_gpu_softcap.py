"""Capped scores: far below the cap, around half of it, far above, exactly at half, scales that are negative, zero, tiny or
huge, and scores that are not finite. A capped score hangs on that score alone: nothing that the mask hides changes a bit. The
backward caps as the forward did, in both of its forms."""

import pytest
import torch

from _util import assert_same_gradients, assert_within_2x
from fast_diffusion_attention import _lib, diffusion_attn_func, diffusion_attn_varlen_func
from oracle import diffusion_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(n, d, heads=4, heads_k=2, dtype=torch.bfloat16):
    torch.manual_seed(n + d)
    return [torch.randn(2, 2 * n, h, d, device=DEV, dtype=dtype) for h in (heads, heads_k, heads_k)]


# scores have a standard deviation of `gain`: the largest of a warp's 32 x 64 are some 3.5 * gain, half of the cap is 2.5
@pytest.mark.parametrize("gain", [0.25, 0.7, 1.6, 6.0])
@pytest.mark.parametrize("d", [64, 128, 96, 256])
@pytest.mark.parametrize("n,bs", [(64, 64), (300, 16), (1000, 256)])
def test_capped_step(n, bs, d, gain):
    q, k, v = _inputs(n, d)
    g = torch.randn_like(q)
    cap, scale = 5.0, gain * d ** -0.5
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    out, lse = diffusion_attn_func(*leaves, bs, softmax_scale=scale, softcap=cap, return_attn_probs=True)
    truth, lse_t = orc.forward(q, k, v, bs, softmax_scale=scale, softcap=cap)
    plain, _ = orc.forward(q, k, v, bs, softmax_scale=scale, softcap=cap, compute_dtype=q.dtype)
    assert_within_2x("out", out, truth, plain)
    # a score's error is at most the cap times tanh.approx's 2^-11, and the log-sum-exp averages such errors
    assert (lse - lse_t).abs().max().item() <= cap * 2.0 ** -11 + 1e-5
    grads = torch.autograd.grad(out, leaves, g)
    gt = orc.backward(q, k, v, g, bs, softmax_scale=scale, softcap=cap)
    gp = orc.backward(q, k, v, g, bs, softmax_scale=scale, softcap=cap, compute_dtype=q.dtype)
    for name, a, t, pl in zip(("dq", "dk", "dv"), grads, gt, gp):
        assert_within_2x(name, a, t, pl)
    assert _lib.device_status()[0] == 0


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale", [-0.2, 0.0, 1e-8, 3e4])
def test_unusual_scales(scale, d):
    q, k, v = _inputs(200, d)
    out, lse = diffusion_attn_func(q, k, v, 32, softmax_scale=scale, softcap=2.0, return_attn_probs=True)
    truth, lse_t = orc.forward(q, k, v, 32, softmax_scale=scale, softcap=2.0)
    plain, _ = orc.forward(q, k, v, 32, softmax_scale=scale, softcap=2.0, compute_dtype=q.dtype)
    assert_within_2x("out", out, truth, plain)
    assert (lse - lse_t).abs().max().item() <= 2.0 ** -10 + 1e-5


@pytest.mark.parametrize("d", [64, 128])
def test_scores_at_half_the_cap_and_not_finite(d):
    n, bs, cap = 256, 256, 6.0
    q = torch.zeros(1, 2 * n, 2, d, device=DEV, dtype=torch.bfloat16)
    k = torch.zeros_like(q)
    v = torch.randn_like(q)
    q[..., 0] = 1.0
    k[..., 0] = 3.0                                   # scale 1: every score is 3 = cap / 2
    out = diffusion_attn_func(q, k, v, bs, softmax_scale=1.0, softcap=cap)
    mean = torch.stack([v[:, :n].float().mean(1), v[:, n:].float().mean(1)], 1).repeat_interleave(n, 1)
    assert (out.float() - mean).abs().max().item() <= 2.0 ** -8    # equal weights, bf16 result below 1
    k[:, n + 5, :, 0] = float("inf")                  # a clean key: infinite scores are capped, the result stays finite
    out = diffusion_attn_func(q, k, v, bs, softmax_scale=1.0, softcap=cap)
    assert torch.isfinite(out[:, n:]).all()
    w = torch.full((n,), float(torch.exp(cap * torch.tanh(torch.tensor(3.0 / cap)))), device=DEV)
    w[5] = float(torch.exp(torch.tensor(cap)))
    want = torch.einsum("k,bkhd->bhd", w / w.sum(), v[:, n:].float())
    # the weights differ by the cap times tanh.approx's 2^-11, P and the result are rounded to bf16
    assert (out[:, n:].float() - want[:, None]).abs().max().item() <= 2.0 ** -7
    q[:, n + 9, 0, 0] = float("nan")                  # a query row: its own result is NaN, its neighbours' are not
    out = diffusion_attn_func(q, k, v, bs, softmax_scale=1.0, softcap=cap)
    assert torch.isnan(out[:, n + 9, 0]).all()
    rest = torch.ones(2 * n, dtype=torch.bool, device=DEV)
    rest[n + 9] = False
    assert torch.isfinite(out[:, rest]).all()


def _step(q, k, v, g, bs, cu=None, **kw):
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    if cu is None:
        out, lse = diffusion_attn_func(*leaves, bs, return_attn_probs=True, **kw)
    else:
        longest = int((cu[1:] - cu[:-1]).max())
        out, lse = diffusion_attn_varlen_func(*leaves, cu, cu, longest, longest, bs, return_attn_probs=True, **kw)
    return (out.detach(), lse) + torch.autograd.grad(out, leaves, g)


# Scores of the first sample have a standard deviation of 0.4, under a cap of 5; those of the second, 40.
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("n,bs", [(200, 24), (33, 8), (300, 512)])
def test_rows_of_other_samples_do_not_count(n, bs, d, deterministic):
    """Behind a sample lie zeros (batched) or the next sample (packed): how a score is capped does not hang on them."""
    q, k, v = _inputs(n, d)
    q[1] *= 100.0
    g = torch.randn_like(q)
    kw = dict(softmax_scale=0.4 * d ** -0.5, softcap=5.0, deterministic=deterministic)
    batched = _step(q, k, v, g, bs, **kw)
    cu = torch.tensor([0, 2 * n, 4 * n], device=DEV, dtype=torch.int32)
    packed = _step(*(t.flatten(0, 1) for t in (q, k, v, g)), bs, cu=cu, **kw)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), packed, batched):
        a = a.unflatten(1, (2, -1)).transpose(0, 1) if name == "lse" else a.unflatten(0, (2, -1))
        assert_same_gradients(name, a, b, exact=deterministic or name != "dq")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 128])
def test_hidden_keys_do_not_count(d, dtype):
    """Keys of the last block in both halves: all other queries have the same results to the bit whatever those keys are."""
    n, bs = 300, 40
    q, k, v = _inputs(n, d, dtype=dtype)
    g = torch.randn_like(q)
    seen = torch.ones(2 * n, dtype=torch.bool, device=DEV)
    seen[280:n] = seen[n + 280:] = False
    kw = dict(softmax_scale=0.4 * d ** -0.5, softcap=5.0, deterministic=True)
    want = _step(q, k, v, g, bs, **kw)
    k[:, ~seen] *= 100.0
    got = _step(q, k, v, g, bs, **kw)
    assert torch.equal(got[0][:, seen], want[0][:, seen]) and torch.equal(got[1][..., seen], want[1][..., seen])
    assert torch.equal(got[2][:, seen], want[2][:, seen])


@pytest.mark.parametrize("gain", [0.4, 1.6, 6.0])
@pytest.mark.parametrize("d", [40, 64, 96, 128])
def test_both_backward_forms_cap_alike(d, gain):
    """dk and dv of the single-pass and of the split backward are the same bits."""
    q, k, v = _inputs(300, d)
    g = torch.randn_like(q)
    kw = dict(softmax_scale=gain * d ** -0.5, softcap=5.0)
    one, split = (_step(q, k, v, g, 48, deterministic=x, **kw) for x in (False, True))
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), one, split):
        assert_same_gradients(name, a, b, exact=name != "dq")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cap", [30.0, 50.0])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("d", [64, 96, 128, 256])
def test_backward_caps_like_the_forward(d, deterministic, cap, dtype):
    """Rows that see one key have the probability 1, in the backward too, which makes it anew from the score and the
    log-sum-exp (a few 1e-6 off by the rounding of those): dv is the gradient of the output to the bit. Two tanh that differ
    by 2^-11 would make it up to cap * 2^-11 wrong, 1 to 2 %."""
    torch.manual_seed(d)
    q, k, v, g = (torch.randn(512, 2, 4, d, device=DEV, dtype=dtype) for _ in range(4))
    _, lse, _, _, dv = _step(q, k, v, g, 1, softmax_scale=0.3 * cap * d ** -0.5, softcap=cap, deterministic=deterministic)
    assert torch.equal(dv, g)
    score = torch.einsum("bqhd,bqhd->bhq", q.double(), k.double()) * (0.3 * cap * d ** -0.5)
    # tanh.approx is good to 2^-11 of its result
    want = cap * torch.tanh(score / cap)
    assert ((lse - want).abs() <= 2.0 ** -10.9 * want.abs() + 1e-5).all()
