"""The gapless pass: pairs settled from one diagonal.

CPU: on pairs where gaps, repeats and mismatches at every place compete, the
rule (a gapless local score above match * Q + gap_open is the pair's score,
its first row-major place and run its alignment; otherwise the score is at
most that bound) holds against the oracle's Smith-Waterman.

GPU: the aligner's output with the pass equals the generic kernel's for every
pair and the oracle's, at the edges of the pass: shortest queries it takes,
word-size query lengths, mismatches up to one more than it takes and at the
read's ends, windows at a sequence's ends, tandem repeats (equal diagonals),
lower case and N nearby, scorings at and past its mismatch limit.
"""
import random

import numpy as np
import pytest


def gapless(q: bytes, w: bytes, m: int, x: int):
    """(score, row, column, first row) of the first row-major maximum over
    the diagonals' local sums, rows and columns from 1."""
    best = (0, 0, 0, 0)
    for d in range(-len(q) + 1, len(w)):
        u, first = 0, 0
        for i in range(len(q)):
            if not 0 <= i + d < len(w):
                continue
            if u == 0:
                first = i
            u = max(0, u + (m if q[i] == w[i + d] else x))
            if u > best[0] or (u == best[0] > 0 and (i + 1, i + d + 1) < best[1:3]):
                best = (u, i + 1, i + d + 1, first)
    return best


def mutated(rng, s: bytes, subs: int, indel: bool) -> bytes:
    b = bytearray(s)
    for _ in range(subs):
        # the ends as often as the middle
        i = rng.choice([rng.randrange(len(b)), rng.randrange(min(4, len(b))),
                        len(b) - 1 - rng.randrange(min(4, len(b)))])
        b[i] = rng.choice([c for c in b"ACGT" if c != b[i]])
    if indel:
        i, n = rng.randrange(len(b)), rng.randint(1, 3)
        if rng.random() < 0.5:
            del b[i:i + n]
        else:
            b[i:i] = bytes(rng.choice(b"ACGT") for _ in range(n))
    return bytes(b)


@pytest.mark.parametrize("m,x,o,e", [(2, -1, -10, -1), (1, -1, -4, -4), (3, -2, -7, -1),
                                     (2, -5, -3, -2)])
def test_rule_against_smith_waterman(oracle, m, x, o, e):
    rng = random.Random(1000 * m + 100 * -x + 10 * -o - e)
    settled = bounded = 0
    for case in range(400):
        Q, R = rng.randint(8, 40), rng.randint(20, 90)
        if case % 4 == 3:  # a repeat: several diagonals score alike
            unit = bytes(rng.choice(b"ACGT") for _ in range(rng.randint(1, 9)))
            w = mutated(rng, (unit * R)[:R], rng.randint(0, 3), False)
        else:
            w = bytes(rng.choice(b"ACGT") for _ in range(R))
        R = len(w)
        at = rng.randint(-3, max(R - Q + 3, 0))
        q = mutated(rng, (w[max(at, 0):at + Q] + w + b"A" * Q)[:Q], rng.randint(0, 6),
                    rng.random() < 0.3)
        q = (q + b"C" * Q)[:Q]
        got = oracle.sw(q, w, Q, R, m, x, o, e)
        score, row, col, first = gapless(q, w, m, x)
        if score > max(m * Q + o, 0):
            settled += 1
            n = row - first
            assert (got["score"], got["len"]) == (score, n)
            assert (got["start"], got["end"]) == (col - n + 1, col)
            assert bytes(got["qcons"])[::-1] == q[first:row]
            assert bytes(got["rcons"])[::-1] == w[col - n:col]
        else:
            bounded += 1
            assert got["score"] <= max(m * Q + o, 0)
    assert settled > 40 and bounded > 40


# ---------------------------------------------------------------------------
# GPU

@pytest.fixture(scope="module")
def sg():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300
    return swift_gb300


@pytest.fixture(scope="module")
def ctx(sg):
    return sg.Context(0)


def fasta(seqs, width=60):
    return b"".join(b">chr%d\n" % i + b"".join(s[k:k + width] + b"\n" for k in range(0, len(s), width))
                    for i, s in enumerate(seqs))


def revcomp(s: bytes) -> bytes:
    return s[::-1].translate(bytes.maketrans(b"ACGT", b"TGCA"))


def workload(seed, L, n=400):
    """Reads of L bases from a reference with tandem and dispersed repeats,
    lower case, N, and sequences that end near a read's window."""
    rng = random.Random(seed)
    rand = lambda k: bytes(rng.choice(b"ACGT") for _ in range(k))
    unit = rand(350)
    a = rand(3000) + unit + rand(500) + mutated(rng, unit, 4, False) + rand(800)
    tandem = rand(23) * 30
    b = rand(700) + tandem + rand(900) + unit + rand(310)
    c = bytearray(rand(2500))
    c[400:460] = bytes(c[400:460]).lower()
    c[1500:1504] = b"NNNN"
    d = rand(300 + L)
    seqs = [a, b, bytes(c), d]
    reads = []
    for i in range(n):
        s = rng.choice(seqs)
        at = rng.choice([rng.randrange(len(s) - L + 1), 0, len(s) - L, rng.randrange(0, 12),
                         len(s) - L - rng.randrange(0, 12)])
        at = min(max(at, 0), len(s) - L)
        r = mutated(rng, s[at:at + L].upper().replace(b"N", b"A"), i % 7, i % 11 == 5)
        r = (r + rand(L))[:L]
        if i % 3 == 1:
            r = revcomp(r)
        if i % 50 == 49:
            r = r[:L // 2] + b"N" + r[L // 2 + 1:]
        reads.append(b">r%d\n%s\n" % (i, r))
    return fasta(seqs), b"".join(reads)


@pytest.mark.gpu
@pytest.mark.parametrize("L", [35, 36, 48, 63, 64, 65, 100, 129, 199])
def test_output_equals_generic_and_oracle(ctx, sg, oracle, L):
    ref, reads = workload(10 + L, L)
    ix = ctx.index(ref)
    for fmt in (0, 1):
        p = sg.default_params(out_format=fmt)
        got = ctx.align(ix, reads, p)
        ctx.set_sw_path(1)
        try:
            generic = ctx.align(ix, reads, p)
        finally:
            ctx.set_sw_path(0)
        assert got == generic
        o = oracle.default_params(device_mem=ctx.info()["total_mem"], out_format=fmt)
        assert got == oracle.align(ref, reads, o)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(gap_open=-2), dict(gap_open=-1, gap_ext=-1),
                                dict(match=1, gap_open=-7), dict(match=1, gap_open=-8),
                                dict(match=3, mismatch=-4, gap_open=-20, gap_ext=-3),
                                dict(gap_open=-2, gap_ext=-4)])
def test_scorings(ctx, sg, oracle, kw):
    ref, reads = workload(77, 90)
    ix = ctx.index(ref)
    got = ctx.align(ix, reads, sg.default_params(**kw))
    assert got == oracle.align(ref, reads, oracle.default_params(
        device_mem=ctx.info()["total_mem"], **kw))


@pytest.mark.gpu
def test_reads_settled_without_smith_waterman(ctx, sg):
    # clean reads: nothing is left to the Smith-Waterman passes
    rng = random.Random(5)
    s = bytes(rng.choice(b"ACGT") for _ in range(40_000))
    reads = b"".join(b">r%d\n%s\n" % (i, s[500 + 30 * i:600 + 30 * i]) for i in range(1024))
    got, st = ctx.align(ctx.index(fasta([s])), reads, stats=True)
    assert st["printed"] == 1024 == st["traced_pairs"]
    assert st["sw_cells_computed"] == 0 and got.count(b"Score: 200.0") == 1024


@pytest.mark.gpu
@pytest.mark.parametrize("L,frag", [(36, (50, 400)), (64, (99, 600)), (100, (180, 320))])
def test_paired_steps(ctx, sg, oracle, L, frag):
    # mate pairs with 0-6 substitutions among repeats: steps settled whole,
    # steps with one unsettled mate, sums that tie, fragments at the limits
    rng = random.Random(900 + L)
    rand = lambda k: bytes(rng.choice(b"ACGT") for _ in range(k))
    unit = rand(400)
    s = rand(900) + unit + rand(300) + unit + mutated(rng, unit, 3, False) + rand(900)
    r1, r2 = [], []
    for i in range(300):
        f = rng.choice([rng.randint(L, 500), frag[0], frag[1], frag[0] - 1, frag[1] + 1])
        f = max(f, L)
        at = rng.randrange(len(s) - f)
        a = mutated(rng, s[at:at + L], i % 4, i % 13 == 4)
        b = mutated(rng, s[at + f - L:at + f], i % 7, False)
        if i % 10 == 9:
            b = rand(L)
        m1, m2 = (a + rand(L))[:L], revcomp((b + rand(L))[:L])
        if i % 5 == 2:
            m1, m2 = m2, m1
        r1.append(b">p%d/1\n%s\n" % (i, m1))
        r2.append(b">p%d/2\n%s\n" % (i, m2))
    r1, r2, ref = b"".join(r1), b"".join(r2), fasta([s])
    ix = ctx.index(ref)
    for fmt in (0, 1):
        got = ctx.align_paired(ix, r1, r2, sg.default_params(out_format=fmt), *frag)
        o = oracle.default_params(device_mem=ctx.info()["total_mem"], out_format=fmt)
        assert got == oracle.align_paired(ref, r1, r2, o, *frag)


@pytest.mark.gpu
@pytest.mark.parametrize("L,sub", [(60, 0.05), (100, 0.04), (201, 0.01), (230, 0.02), (251, 0.01),
                                   (300, 0.03)])
def test_settled_by_the_lcs_bound(ctx, sg, L, sub):
    # reads the first pass leaves (more mismatches than it takes, or cut off
    # by their window) in numbers that run the LCS pass: as the int32 kernel
    from swift_gb300 import synth
    names, seqs = synth.make_reference(200_000, 3, sigma=0.4, repeat_frac=0.2, n_units=15, seed=L)
    seqs[0][5000:5900] = np.frombuffer(b"ACGTTGCAAC" * 90, np.uint8)  # diagonals alike
    rn, rs, _ = synth.make_reads(seqs, 9000, L, sub, 0.0005, 0.05, seed=L + 1)
    reads = synth.reads_fasta(rn, rs)
    ix = ctx.index(synth.fasta_bytes(names, seqs))
    for kw in (dict(), dict(out_format=1), dict(match=3, mismatch=-2, gap_open=-6, gap_ext=-2)):
        p = sg.default_params(max_read_len=300, **kw)
        got = ctx.align(ix, reads, p)
        ctx.set_sw_path(1)
        try:
            assert got == ctx.align(ix, reads, p), kw
        finally:
            ctx.set_sw_path(0)
