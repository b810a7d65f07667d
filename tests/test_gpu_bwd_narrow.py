"""Single-pass backward at head dimensions up to 64: dQ is made with a query on every lane, in tensor-memory columns of its own.
Sizes where that can go wrong: one step, two, three (the ring of Q); quarters of a step without queries; head dimensions that end
inside or before the second 32 columns; several heads of a group; ends of samples."""

import pytest
import torch

from fast_diffusion_attention import diffusion_attn_func
from test_gpu_bwd import check_backward

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("d", [8, 24, 32, 40, 56, 64])
@pytest.mark.parametrize("n,bs", [(1, 1), (31, 31), (33, 8), (96, 96), (97, 5), (129, 129), (160, 64), (257, 256), (385, 400),
                                  (511, 32)])
def test_narrow_heads(n, bs, d):
    torch.manual_seed(n + d)
    q, k, v = (torch.randn(2, 2 * n, h, d, device=DEV, dtype=torch.bfloat16) for h in (6, 2, 2))
    check_backward(q, k, v, bs)


@pytest.mark.parametrize("softcap", [0.0, 4.0])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_narrow_heads_packed(dtype, softcap):
    torch.manual_seed(3)
    ns = [1, 0, 63, 65, 700, 128, 127, 2, 300]
    cu = torch.tensor([0] + list(torch.tensor([2 * x for x in ns]).cumsum(0)), device=DEV, dtype=torch.int32)
    q, k, v = (torch.randn(2 * sum(ns), h, 64, device=DEV, dtype=dtype) for h in (4, 1, 1))
    check_backward(q, k, v, 24, softcap=softcap, cu=cu)


def test_rows_of_other_samples_stay_out():
    """The rows that a step reads past the end of a half or sample add nothing, whatever they hold."""
    torch.manual_seed(5)
    n, bs = 100, 20
    q, k, v = (torch.randn(2, 2 * n, 2, 64, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    g = torch.randn_like(q)

    def grads(x):
        leaves = [t.detach().requires_grad_() for t in x]
        return torch.autograd.grad(diffusion_attn_func(*leaves, bs), leaves, g)

    want = grads((q, k, v))
    loud = [t.clone() for t in (q, k, v)]
    for t in loud:
        t[1] *= 100.0                                 # the other sample lies right behind the first
    got = grads(loud)
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        if name == "dq":                              # order of the adds: one rounding step
            assert (a[0].float() - b[0].float()).abs().max() <= 2.0 ** -7 * b[0].float().abs().max()
        else:
            assert torch.equal(a[0], b[0]), name
