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


@pytest.mark.parametrize("d", [136, 192, 256])
def test_wide_heads_need_no_accumulator(d):
    """Above head dim 128 the default backward is the deterministic one: the same bits in every run, and the same workspace."""
    for kw in (dict(seqlen=16384, heads=8, heads_k=8, batch=2), dict(seqlen=2800, heads=20, heads_k=10, batch=2),
               dict(heads=32, heads_k=8, **_packed([4095, 1203, 2750, 3391, 1876, 2049]))):
        assert _bytes(d=d, **kw) == _bytes(d=d, deterministic=1, **kw)


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


def _whole_without_parts(n, batch, bs, heads_k):
    """(steps of the longest chain, of all chains) of one query head a group, counted tile pair by tile pair."""
    tiles, chains = -(-n // 128), []
    span = [(128 * t, min(128 * t + 128, n)) for t in range(tiles)]
    for k0, k1 in span:
        first, last = k0 // bs, (k1 - 1) // bs
        noisy = sum(q0 // bs <= last and (q1 - 1) // bs >= first for q0, q1 in span)
        clean = sum((q1 - 1) // bs >= first for q0, q1 in span)
        cross = sum((q1 - 1) // bs > first for q0, q1 in span)
        chains += [noisy, clean + cross]
    return max(chains), sum(chains) * heads_k * batch


@pytest.mark.parametrize("bs", [1, 32, 128, 200, 256, 512, 1000, 4096])
def test_the_rule_follows_the_steps(bs):
    """Parts where the longest chain is well above a CTA's share of all steps, none where it is well below, and with blocks of half
    a sample or more only where they save a number of steps."""
    for n in (300, 1000, 1500, 2048, 4096):
        for batch in (1, 2, 4, 8):
            for heads, heads_k in [(8, 2), (32, 8), (12, 4), (8, 1), (32, 1), (14, 2)]:
                group, tiles = heads // heads_k, -(-n // 128)
                chain, steps = _whole_without_parts(n, batch, bs, heads_k)
                got, nbytes = parts(2 * n, heads, heads_k, 64, batch=batch, bs=bs)
                case = (n, batch, heads, heads_k, chain, steps, got)
                if 2 * bs >= n:
                    assert got == 1 or (chain - steps / 148) * group >= 10, case   # the host's count is off by a tile's edges
                elif bs <= 128:
                    if steps < 0.8 * 120 * chain and 2 * tiles * group > 32 and group < 30:
                        assert got > 1, case
                    if steps > 1.25 * 120 * chain:
                        assert got == 1, case


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
