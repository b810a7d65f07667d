"""The eager host path against what the operators do: every input a caller may hold (expanded, strided and negated views),
every context that wants to see the calls (modes, hooks on saved tensors, compiled autograd, threads), and the values the
operators hand back. Where nothing but the route differs, results are compared bitwise (deterministic backward)."""

import math
import threading

import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from fast_diffusion_attention import diffusion_attn_func, diffusion_attn_varlen_func
from fast_diffusion_attention.interface import diffusion_attn_qkvpacked_func, diffusion_attn_varlen_qkvpacked_func

pytestmark = pytest.mark.gpu
DEV = "cuda"
B, N, H, HK, D, BS = 2, 96, 4, 2, 64, 16
LAYOUTS = ["batched", "varlen", "qkv", "varlen_qkv"]


def _inputs(layout, seed=0, requires_grad=True):
    """(leaves, cu, dout) of one small problem."""
    g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, device=DEV, dtype=torch.bfloat16, generator=g)

    lead = (B, 2 * N) if layout in ("batched", "qkv") else (B * 2 * N,)
    leaves = [normal(*lead, H + 2 * HK, D)] if "qkv" in layout else [normal(*lead, h, D) for h in (H, HK, HK)]
    cu = None if layout in ("batched", "qkv") else torch.arange(0, B * 2 * N + 1, 2 * N, device=DEV, dtype=torch.int32)
    return [t.requires_grad_(requires_grad) for t in leaves], cu, normal(*lead, H, D)


def _call(layout, leaves, cu, **kw):
    kw.setdefault("deterministic", True)
    if layout == "batched":
        return diffusion_attn_func(*leaves, BS, **kw)
    if layout == "varlen":
        return diffusion_attn_varlen_func(*leaves, cu, cu, 2 * N, 2 * N, BS, **kw)
    if layout == "qkv":
        return diffusion_attn_qkvpacked_func(*leaves, BS, num_heads_q=H, **kw)
    return diffusion_attn_varlen_qkvpacked_func(*leaves, cu, 2 * N, BS, num_heads_q=H, **kw)


def _expected(layout):
    leaves, cu, do = _inputs(layout)
    out = _call(layout, leaves, cu)
    return (out.detach(),) + torch.autograd.grad(out, leaves, do)


def _assert_all_equal(got, want):
    assert len(got) == len(want)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), i


# ------------------------------------------------------------------------------------------ values handed back
@pytest.mark.parametrize("varlen", [False, True])
@pytest.mark.parametrize("d,deterministic", [(64, False), (128, False), (96, True), (256, False)])
def test_backward_operator_returns_the_row_sums(d, deterministic, varlen):
    """(batch, heads, 2, n_pad) of rowsum(dO * O), zero in the padding rows."""
    torch.manual_seed(d)
    n, n_pad, heads, heads_k = 150, 256, 4, 2
    q, do = (torch.randn(B, 2 * n, heads, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, 2 * n, heads_k, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    cu = max_len = None
    if varlen:
        q, k, v, do = (t.flatten(0, 1) for t in (q, k, v, do))
        cu, max_len = torch.arange(0, B * 2 * n + 1, 2 * n, device=DEV, dtype=torch.int32), 2 * n
    out, lse = torch.ops.fda._diffusion_attn_forward(q, k, v, 32, cu, max_len)
    grads = [torch.empty_like(t) for t in (q, k, v)]
    got = torch.ops.fda._diffusion_attn_backward(do, q, k, v, out, lse, *grads, 32, cu, max_len, deterministic=deterministic)
    terms = (do.double() * out.double()).view(B, 2, n, heads, d).permute(0, 3, 1, 2, 4)
    assert got.shape == (B, heads, 2, n_pad) and got.dtype == torch.float32
    # fp32 sums of d exact products, in any order
    assert ((got[..., :n] - terms.sum(-1)).abs() <= d * 2.0 ** -24 * terms.abs().sum(-1)).all()
    assert (got[..., n:] == 0).all()


@pytest.mark.parametrize("d", [64, 128, 256])
def test_fp8_largest_probability_is_exact(d):
    """The largest probability of a row is held as 2^8, which e4m3 has, also where the maximum creeps up by less than a
    rounding step of the type: the row's result then errs by the rounding of the bf16 output (and of the fp32 sum)."""
    n, small, big = 192, 0, 100                    # keys in different sub-steps, the larger score second
    step = 0.09                                    # log2 of the ratio of the two probabilities
    q = torch.zeros(1, 2 * n, 1, d, device=DEV)
    k, v = torch.zeros_like(q), torch.zeros_like(q)
    q[..., 0] = 1
    k[..., 0] = -448                               # everything else: 2^-40 of the row
    for half in (0, n):
        k[:, half + small, :, 0] = 0
        k[:, half + big, :, 0] = 1
        v[:, half + big] = 1
    out = diffusion_attn_func(*(t.to(torch.float8_e4m3fn) for t in (q, k, v)), n, softmax_scale=step * math.log(2))
    want = 1 / (1 + 2.0 ** -step)
    assert (out.double() - want).abs().max().item() <= want * 2.0 ** -8


@pytest.mark.parametrize("dtype,digits", [(torch.bfloat16, 8), (torch.float16, 11)])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("big", [40, 100])
def test_largest_probability_of_the_first_keys_is_exact(d, dtype, digits, big):
    """Where the largest score of a row is among its first 128 keys, its probability is held as 1: with one other key that
    counts and has no value, the result errs by the rounding of the output alone."""
    n = 192
    step = torch.linspace(0.02, 0.98, n, device=DEV).to(dtype)     # log2 of the ratio of the two probabilities, by row
    q = torch.zeros(1, 2 * n, 1, d, device=DEV, dtype=dtype)
    k, v = torch.zeros_like(q), torch.zeros_like(q)
    q[0, :, 0, 0] = step.repeat(2)
    k[..., 0] = -10000                                             # everything else: 2^-200 of the row
    for half in (0, n):
        k[:, half, :, 0] = 0
        k[:, half + big, :, 0] = 1
        v[:, half + big] = 1
    out = diffusion_attn_func(q, k, v, n, softmax_scale=math.log(2))[0, :, 0].double()
    want = (1 / (1 + torch.exp2(-step.double()))).repeat(2)[:, None]
    assert ((out - want).abs() <= want * 2.0 ** -digits * 1.001).all()


# ------------------------------------------------------------------------------------------ views as inputs
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("axis", [-3, -2])
def test_gradient_of_the_output_with_a_zero_stride(layout, axis):
    """The gradient that a sum over tokens or heads hands back is an expanded view."""
    grads = []
    for expanded in (True, False):
        leaves, cu, do = _inputs(layout)
        w = do.select(axis, 0)
        out = _call(layout, leaves, cu)
        if expanded:
            grads.append(torch.autograd.grad((out.sum(axis) * w).sum(), leaves))
        else:
            grads.append(torch.autograd.grad(out, leaves, w.unsqueeze(axis).expand_as(out).contiguous()))
    _assert_all_equal(*grads)


@pytest.mark.parametrize("layout", ["batched", "varlen"])
@pytest.mark.parametrize("axis", [-2, -3])
def test_expanded_keys_and_values(layout, axis):
    results = []
    for expanded in (True, False):
        (q, k, v), cu, do = _inputs(layout, requires_grad=False)
        k, v = (t.narrow(axis, 0, 1).clone().requires_grad_() for t in (k, v))
        shape = list(k.shape)
        shape[axis] = q.shape[axis]
        ke, ve = (t.expand(shape) if expanded else t.expand(shape).contiguous() for t in (k, v))
        out = _call(layout, (q, ke, ve), cu)
        results.append((out.detach(),) + torch.autograd.grad(out, (k, v), do))
    _assert_all_equal(*results)


@pytest.mark.parametrize("layout", ["varlen", "varlen_qkv"])
def test_strided_offsets(layout):
    leaves, cu, do = _inputs(layout)
    out = _call(layout, leaves, torch.stack([cu, -cu], 1)[:, 0])
    _assert_all_equal((out.detach(),) + torch.autograd.grad(out, leaves, do), _expected(layout))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_lazily_negated_views(layout):
    """A tensor whose values are negated by a flag on the view (as the imaginary part of a conjugate is)."""
    leaves, cu, do = _inputs(layout)
    want = _expected(layout)
    with torch.no_grad():
        negated = [torch._neg_view(-t).requires_grad_() for t in leaves]
    assert negated[0].is_neg()
    out = _call(layout, negated, cu)
    _assert_all_equal((out.detach(),) + torch.autograd.grad(out, negated, do), want)
    out = _call(layout, leaves, cu)
    _assert_all_equal((out.detach(),) + torch.autograd.grad(out, leaves, torch._neg_view(-do)), want)


def test_scale_that_is_not_a_number_reaches_the_output():
    leaves, cu, _ = _inputs("batched", requires_grad=False)
    for call in (lambda: diffusion_attn_func(*leaves, BS, softmax_scale=math.nan),
                 lambda: torch.ops.fda._diffusion_attn_forward(*leaves, BS, softmax_scale=math.nan)[0]):
        assert call().isnan().all()


def test_packed_head_count_is_checked():
    qkv = torch.randn(1, 64, 3, 2, 64, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="num_heads_q disagrees"):
        diffusion_attn_qkvpacked_func(qkv, 16, num_heads_q=-1)


# ------------------------------------------------------------------------------------------ who wants to see the calls
class _FunctionLog(TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


class _DispatchLog(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_function_mode_sees_the_operator(layout):
    leaves, cu, do = _inputs(layout)
    with _FunctionLog() as log:
        out = _call(layout, leaves, cu)
    assert any("_diffusion_attn_forward" in s for s in log.seen), log.seen
    _assert_all_equal((out.detach(),) + torch.autograd.grad(out, leaves, do), _expected(layout))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_dispatch_mode_around_the_backward_alone(layout):
    leaves, cu, do = _inputs(layout)
    out = _call(layout, leaves, cu)
    with _DispatchLog() as log:
        grads = torch.autograd.grad(out, leaves, do)
    assert any("_diffusion_attn_backward" in s for s in log.seen), log.seen
    _assert_all_equal((out.detach(),) + grads, _expected(layout))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_hooks_on_saved_tensors_see_all_of_them(layout):
    """Everything that the node keeps goes through the hooks, in the order in which the Python twin saves it."""
    leaves, cu, do = _inputs(layout)
    packed, unpacked = [], []

    def pack(t):
        packed.append(t.dtype)
        return t.cpu()

    def unpack(t):
        unpacked.append(t.dtype)
        return t.to(DEV)

    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        out = _call(layout, leaves, cu)
    result = (out.detach(),) + torch.autograd.grad(out, leaves, do)
    saved = [torch.bfloat16] * (len(leaves) + 1) + [torch.float32] + ([torch.int32] if cu is not None else [])
    assert packed == saved and unpacked == saved
    _assert_all_equal(result, _expected(layout))


@pytest.mark.parametrize("layout", ["varlen", "varlen_qkv"])
def test_offsets_changed_before_the_backward_are_noticed(layout):
    leaves, cu, do = _inputs(layout)
    out = _call(layout, leaves, cu)
    cu.add_(0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, leaves, do)


@pytest.mark.parametrize("layout", LAYOUTS)
def test_checkpointed_region(layout):
    leaves, cu, do = _inputs(layout)
    out = torch.utils.checkpoint.checkpoint(lambda *x: _call(layout, x, cu), *leaves, use_reentrant=False)
    _assert_all_equal((out.detach(),) + torch.autograd.grad(out, leaves, do), _expected(layout))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_backward_under_compiled_autograd(layout):
    from torch._dynamo import compiled_autograd
    leaves, cu, do = _inputs(layout)
    out = _call(layout, leaves, cu)
    with compiled_autograd._enable(torch.compile(backend="eager", fullgraph=False)):
        out.backward(do)
    _assert_all_equal([out.detach()] + [t.grad for t in leaves], _expected(layout))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_gradients_are_constants_under_create_graph(layout):
    """The backward has no derivative; with the native node and with the Python one its results do not require grad."""
    results = []
    for mode in (_FunctionLog(), None):
        leaves, cu, do = _inputs(layout)
        if mode is not None:
            with mode:
                out = _call(layout, leaves, cu)
        else:
            out = _call(layout, leaves, cu)
        results.append(torch.autograd.grad(out, leaves, do.requires_grad_(), create_graph=True))
        assert not any(g.requires_grad for g in results[-1])
    _assert_all_equal(*results)


def test_two_threads_over_one_graph():
    """Each thread gets the gradients or, where the other has freed the graph before it, the error that says so."""
    want = _expected("batched")[1:]
    for _ in range(30):
        leaves, cu, do = _inputs("batched")
        out = _call("batched", leaves, cu)
        results, start = [], threading.Barrier(2)

        def run():
            start.wait()
            try:
                results.append(torch.autograd.grad(out, leaves, do))
            except RuntimeError as e:
                results.append(str(e))

        threads = [threading.Thread(target=run) for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(results) == 2 and any(not isinstance(r, str) for r in results)
        for r in results:
            if isinstance(r, str):
                assert "second time" in r
            else:
                _assert_all_equal(r, want)
