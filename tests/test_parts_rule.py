"""Into how many parts the default backward deals a group's query heads, as the workspace it asks for shows it: few tokens and
few KV heads get parts, a batch with enough work of its own none, whatever the packed lengths or a loose max_seqlen look
like, and the parts never take more than 512 MiB (256 MiB for samples of unlike lengths). No GPU needed."""

import ctypes as C
import random

import pytest

from fast_diffusion_attention import _lib

MIB = 1 << 20


def _bytes(seqlen, heads, heads_k, d, *, batch, total=None, deterministic=0, bs=64):
    packed = total is not None
    p = _lib.FdaProblem(_lib.FDA_BF16, batch, seqlen, total if packed else batch * seqlen, heads, heads_k, d, bs, 0.1, 0.0, 0,
                        deterministic, C.c_void_p(256) if packed else None)
    return _lib.load().fda_bwd_workspace_bytes(C.byref(p))


def parts(seqlen, heads, heads_k, d, **kw):
    """(number of parts, their bytes). The workspace is the deterministic one, the dQ accumulator (the same without groups)
    and the parts: dK and dV of each in the accumulator's layout."""
    fixed = _bytes(seqlen, heads, heads_k, d, deterministic=1, **kw)
    acc = _bytes(seqlen, heads, heads, d, **kw) - fixed
    extra = _bytes(seqlen, heads, heads_k, d, **kw) - fixed - acc
    n = extra * heads / (2 * heads_k * acc)
    assert n == int(n)
    return max(1, int(n)), extra


def _packed(ns, max_n=None):
    return dict(seqlen=2 * (max_n or max(ns)), batch=len(ns), total=2 * sum(ns))


def test_few_tokens_and_few_heads_are_dealt_out():
    assert parts(2000, 8, 1, 128, batch=1)[0] == 8
    assert parts(8192, 8, 2, 128, batch=1)[0] == 4
    assert parts(4096, 32, 8, 128, batch=1)[0] == 2
    assert parts(6000, 14, 2, 128, batch=4)[0] == 7           # 337 MiB
    assert parts(4096, 8, 8, 128, batch=1)[0] == 1            # no groups


@pytest.mark.parametrize("heads,heads_k,d,ns,max_n", [
    (32, 8, 128, [16384] + [256] * 100, None),       # one long sample among many short ones
    (32, 8, 128, [512] * 64, 32768),                 # an upper bound for max_seqlen
    (32, 8, 64, [512] * 64, 1 << 20),
    (8, 1, 128, [8192] * 4 + [64] * 500, None),
    (32, 8, 128, [2048] * 4, None),
])
def test_batches_with_enough_work_stay_whole(heads, heads_k, d, ns, max_n):
    assert parts(heads=heads, heads_k=heads_k, d=d, **_packed(ns, max_n)) == (1, 0)


def test_parts_stay_small():
    rng = random.Random(0)
    seen = set()
    for _ in range(3000):
        heads_k = rng.choice([1, 1, 2, 3, 4, 8])
        group = rng.choice([2, 3, 4, 7, 8, 16, 31])
        d = rng.choice([64, 128])
        ns = [int(2 ** rng.uniform(0, 16)) for _ in range(rng.choice([1, 2, 5, 40]))]
        kw = _packed(ns, rng.choice([None, 2 * max(ns), 1 << 17])) if rng.random() < 0.5 else dict(seqlen=2 * ns[0], batch=len(ns))
        n, extra = parts(heads=heads_k * group, heads_k=heads_k, d=d, **kw)
        alike = "total" not in kw or kw["total"] == kw["batch"] * kw["seqlen"]
        assert group % n == 0 and extra <= (512 if alike else 256) * MIB
        seen.add(n)
    assert {1, 2, 4, 8, 31} <= seen


@pytest.mark.parametrize("n", [127, 333, 1000, 4096])
@pytest.mark.parametrize("batch", [1, 2, 5, 12])
def test_packed_samples_of_one_length_are_dealt_like_a_batch(n, batch):
    for heads, heads_k in [(8, 1), (8, 2), (32, 8), (12, 4), (31, 1)]:
        assert parts(2 * n, heads, heads_k, 128, batch=batch)[0] == parts(heads=heads, heads_k=heads_k, d=128, **_packed([n] * batch))[0]


def test_the_convert_grid_holds_every_head():
    """dQ of each head and, with parts, dK and dV of each KV head are (half, head) rows of one grid, 65535 at most: a call that
    the rest of the backward takes must not fail there."""
    for heads, heads_k in [(32766, 6), (32767, 7), (32767, 1), (32760, 8), (16000, 1)]:
        n, _ = parts(512, heads, heads_k, 64, batch=1)
        assert n == 1 or 2 * (heads + 2 * heads_k) <= 65535, (heads, heads_k, n)
