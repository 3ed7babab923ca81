"""The long pairs' 16-bit kernel (A, C, G, T bytes) against the oracle.

Query lengths around its strips (2-8 rows a half, 64 strips a warp, 8 warps),
windows around its edge steps and stages, no alignment at all, equal maxima in
several rows and columns, alignments that cross every warp boundary with gaps,
lower case, and the longest query its cells hold with the one past it.
"""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300
    return swift_gb300


@pytest.fixture(scope="module")
def ctx(sg):
    return sg.Context(0)


def rand(rng, n):
    return bytes(rng.choice(b"ACGT") for _ in range(n))


def noisy(rng, s, sub, indel):
    out = bytearray()
    for c in s:
        u = rng.random()
        if u < indel / 2:
            continue
        if u < indel:
            out += rand(rng, rng.randint(1, 3))
        out.append(rng.choice(b"ACGT") if rng.random() < sub else c)
    return bytes(out)


def check(ctx, oracle, qs, ws, sc=(2, -1, -10, -1)):
    off = lambda v: np.concatenate([[0], np.cumsum([len(s) for s in v])[:-1]]).astype(np.int64)
    res, _ = ctx.sw_pairs(b"".join(qs), off(qs), [len(q) for q in qs], b"".join(ws), off(ws),
                          [len(w) for w in ws], *sc)
    for i, (q, w) in enumerate(zip(qs, ws)):
        want = oracle.sw(q, w, len(q), len(w), *sc)
        for k in ("score", "start", "end", "len", "qcons", "rcons"):
            assert res[k][i] == want[k], (i, len(q), len(w), k)


@pytest.mark.parametrize("Q", [1, 63, 127, 128, 129, 257, 1023, 1024, 1025, 2047, 2049, 3072, 3073, 4070])
def test_shapes(ctx, oracle, Q):
    rng = random.Random(Q)
    qs, ws = [], []
    for R in (1025, 1040, 1088, 1151, 2003 + Q % 7):
        w = rand(rng, R)
        at = rng.randrange(max(1, R - Q + 1))
        q = (noisy(rng, w[at:at + Q], 0.03, 0.02) + rand(rng, Q))[:Q]
        if len(qs) == 2:
            q, w = q.lower(), w[:500].lower() + w[500:]
        if len(qs) == 3:
            q = rand(rng, Q)  # chance alignments only
        qs.append(q)
        ws.append(w)
    if Q > 256:  # windows shorter than the wavefront
        for R in (1, 2, 61, 62, 63, 64, 65, 130):
            w = rand(rng, R)
            qs.append((rand(rng, Q // 2) + w + rand(rng, Q))[:Q])
            ws.append(w)
    check(ctx, oracle, qs, ws)


def test_ties_and_repeats(ctx, oracle):
    rng = random.Random(7)
    unit = rand(rng, 37)
    qs = [b"A" * 600, b"A" * 1500, unit * 12, unit * 40, rand(rng, 700) + unit + rand(rng, 700) + unit,
          b"C" * 400 + b"G" * 3, b"AC" * 400]
    ws = [b"C" * 1100, b"C" * 700 + b"A" * 3 + b"C" * 600 + b"A" * 3 + b"C" * 30, unit * 60,
          unit * 45, unit + rand(rng, 1000) + unit + rand(rng, 300),
          b"T" * 100 + b"G" + b"T" * 900 + b"GG" + b"T" * 300, b"CA" * 900]
    check(ctx, oracle, qs, ws)
    check(ctx, oracle, qs, ws, (3, -2, -5, -2))
    check(ctx, oracle, qs, ws, (1, -1, -1, -1))


@pytest.mark.parametrize("sc", [(2, -1, -10, -1), (31, -32, -120, -3), (7, -1, -2, -1)])
def test_largest_queries_of_a_scoring(ctx, oracle, sc):
    # the longest query that fits 16 bits, and one more (the int32 kernel)
    m, _, o, e = sc
    bias = (-(4 * o + 1) + 3) // 4 * 4
    most = min((32767 - bias - 4 * (e - o) - 8) // (4 * m), 4095)
    rng = random.Random(m)
    qs, ws = [], []
    for Q in (most, most + 1):
        w = rand(rng, max(Q + 150, 1300))
        qs.append((noisy(rng, w[70:70 + Q], 0.0, 0.0005) + rand(rng, 50))[:Q])
        ws.append(w)
        qs.append(w[20:20 + Q])  # all of it matches: the largest cell there is
        ws.append(w)
    check(ctx, oracle, qs, ws, sc)
