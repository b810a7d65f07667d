"""Capped scores on both sides of the line where the kernels change from a polynomial to the unit's tanh (|score * scale| of
half the cap, decided for a warp and step): all below, some warps below, all above, a score exactly on it, scales that are
negative, zero or out of the polynomial's range, and scores that are not finite."""

import pytest
import torch

from _util import assert_within_2x
from fast_diffusion_attention import _lib, diffusion_attn_func
from oracle import diffusion_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(n, d, heads=4, heads_k=2, dtype=torch.bfloat16):
    torch.manual_seed(n + d)
    return [torch.randn(2, 2 * n, h, d, device=DEV, dtype=dtype) for h in (heads, heads_k, heads_k)]


# scores have a standard deviation of `gain`: the largest of a warp's 32 x 64 are some 3.5 * gain, the line is at 2.5
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
def test_scales_outside_the_polynomial(scale, d):
    q, k, v = _inputs(200, d)
    out, lse = diffusion_attn_func(q, k, v, 32, softmax_scale=scale, softcap=2.0, return_attn_probs=True)
    truth, lse_t = orc.forward(q, k, v, 32, softmax_scale=scale, softcap=2.0)
    plain, _ = orc.forward(q, k, v, 32, softmax_scale=scale, softcap=2.0, compute_dtype=q.dtype)
    assert_within_2x("out", out, truth, plain)
    assert (lse - lse_t).abs().max().item() <= 2.0 ** -10 + 1e-5


@pytest.mark.parametrize("d", [64, 128])
def test_scores_on_the_line_and_not_finite(d):
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
