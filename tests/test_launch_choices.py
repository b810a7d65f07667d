"""Which forms of the kernels a call takes, by the launchers' own rules (no GPU needed), and, on the GPU, that forms chosen for speed
alone give the same bits."""

import ctypes as C
import os

import pytest
import torch

from fast_diffusion_attention import _lib, diffusion_attn_varlen_func


def _choices(seqlen, heads, heads_k, d, bs=64, *, batch=1, total=None, dtype=_lib.FDA_BF16, softcap=0.0, sm_margin=0, deterministic=0):
    packed = total is not None
    p = _lib.FdaProblem(dtype, batch, seqlen, total if packed else batch * seqlen, heads, heads_k, d, bs, 0.1, softcap, sm_margin,
                        deterministic, C.c_void_p(256) if packed else None)
    return _lib.load().fda_launch_choices(C.byref(p))


@pytest.mark.parametrize("dtype,d,softcap,line", [(_lib.FDA_BF16, 64, 0.0, 4096), (_lib.FDA_FP16, 40, 0.0, 4096),
                                                      (_lib.FDA_BF16, 64, 30.0, 4096), (_lib.FDA_E4M3, 64, 0.0, 3000),
                                                      (_lib.FDA_E4M3, 256, 30.0, 3000)])
def test_only_long_samples_have_a_loop_for_full_sub_steps(dtype, d, softcap, line):
    def takes(n, bs=64, heads=16, **kw):
        return bool(_choices(2 * n, heads, heads, d, bs, dtype=dtype, softcap=softcap, **kw) & _lib.FDA_CHOICE_FORWARD_FULL_LOOP)

    assert takes(line, batch=4) and takes(line, batch=16) and takes(8192, bs=2048, batch=4)
    for n in (64, 256, 512, 1024, 1500, 2048, line - 1):
        assert not takes(n, batch=128)
    assert takes(600, heads=2) and not takes(599, heads=2) and not takes(512, heads=1)   # few items a CTA
    assert not takes(8192, batch=41, total=2 * (8192 + 40 * 300))     # one long sample among short ones
    assert not takes(32768, batch=64, total=2 * 64 * 512)             # max_seqlen is an upper bound
    assert takes(8192, bs=8192, batch=4) == (dtype == _lib.FDA_E4M3)  # noisy rows of one block see no clean key


def test_who_has_no_such_loop():
    for kw in (dict(d=256), dict(d=136), dict(d=128), dict(d=72, softcap=30.0)):
        assert not _choices(16384, 16, 8, **kw) & _lib.FDA_CHOICE_FORWARD_FULL_LOOP
    assert _choices(16384, 16, 8, d=60) == 0   # refused


def _overlaps(*args, **kw):
    """(forward, backward)"""
    c = _choices(*args, **kw)
    return bool(c & _lib.FDA_CHOICE_FORWARD_OVERLAP), bool(c & _lib.FDA_CHOICE_BACKWARD_OVERLAP)


def test_small_calls_overlap_and_leave_the_sms_free_that_the_caller_wants():
    for kw in (dict(seqlen=512, heads=4, heads_k=4, d=64, batch=2), dict(seqlen=1400, heads=16, heads_k=4, d=128),
               dict(seqlen=2048, heads=8, heads_k=8, d=256, deterministic=1), dict(seqlen=600, heads=8, heads_k=2, d=96, batch=5, total=1900)):
        assert _overlaps(**kw) == (True, True)
        assert _overlaps(sm_margin=1, **kw) == _overlaps(sm_margin=140, **kw) == (False, False)
    assert _overlaps(seqlen=8192, heads=16, heads_k=16, d=128) == (False, False)


def test_long_samples_do_not_overlap():
    """Few rows and heads are little data, but not little work. The single-pass backward of head dims 65 to 128 overlaps with at
    most two items a CTA (a part of a group is an item)."""
    for n, h, hk, d, b, want in ((1500, 8, 8, 128, 1, True), (2048, 8, 8, 96, 1, True), (4096, 4, 4, 128, 1, True), (1500, 8, 2, 128, 1, True),
                                 (1500, 16, 16, 128, 1, False), (512, 16, 16, 128, 4, False), (3000, 8, 2, 96, 1, False),
                                 (4096, 8, 2, 128, 1, False), (8192, 4, 4, 128, 1, False), (2048, 16, 4, 128, 1, False)):
        assert _overlaps(2 * n, h, hk, d, batch=b)[1] is want, (n, h, hk, d, b)
    assert _overlaps(4096, 16, 16, 128, deterministic=1) == _overlaps(8192, 16, 16, 64) == _overlaps(8192, 4, 4, 256) == (True, True)
    for d, h in ((64, 8), (128, 4), (256, 2)):
        for deterministic in (0, 1):
            assert _overlaps(16384, h, h, d, deterministic=deterministic) == (False, False)
    assert _overlaps(1 << 20, 4, 4, 64, batch=2, total=1024) == (True, True)      # max_seqlen is an upper bound


@pytest.mark.gpu
@pytest.mark.parametrize("n,bs", [(601, 16), (777, 150), (4096, 1), (4097, 64), (4100, 300), (4159, 1024)])
@pytest.mark.parametrize("dtype,d,softcap", [(torch.bfloat16, 64, 0.0), (torch.float16, 64, 0.0), (torch.bfloat16, 64, 20.0),
                                             (torch.float8_e4m3fn, 128, 0.0), (torch.float8_e4m3fn, 256, 20.0)])
def test_both_loops_give_the_same_bits(n, bs, dtype, d, softcap):
    """A sample alone, and in front of short ones that take the mean length below the line."""
    torch.manual_seed(n)
    q, k, v = (torch.randn(2 * n + 512, h, d, device="cuda").to(dtype) for h in (4, 2, 2))
    code = {torch.bfloat16: _lib.FDA_BF16, torch.float16: _lib.FDA_FP16}.get(dtype, _lib.FDA_E4M3)
    outs = []
    for ns in ([n], [n] + [32] * 8):
        total = 2 * sum(ns)
        assert bool(_choices(2 * n, 4, 2, d, bs, batch=len(ns), total=total, dtype=code, softcap=softcap) & 1) == (len(ns) == 1)
        cu = torch.tensor([0] + ns, device="cuda").cumsum(0).int() * 2
        out, lse = diffusion_attn_varlen_func(q[:total], k[:total], v[:total], cu, cu, 2 * n, 2 * n, bs, softcap=softcap,
                                              return_attn_probs=True)
        outs.append((out[:2 * n], lse[:, :2 * n]))
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_no_block_ends_before_it_has_waited_for_the_stream():
    """A kernel that may start early must not be complete before those ahead of it: the next one waits for this one only. So no kernel
    (the self tests launch in plain order) returns ahead of ptx::wait_for_stream."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__))), "csrc")
    kernels = 0
    for name in os.listdir(csrc):
        if name.endswith(".cu") and not name.startswith("selftest"):
            for body in open(os.path.join(csrc, name)).read().split("__global__ void")[1:]:
                if "{" in body.split(";")[0]:   # a definition
                    head, found, _ = body.partition("ptx::wait_for_stream();")
                    assert found and "return;" not in head, (name, body[:120])
                    kernels += 1
    assert kernels == 7
