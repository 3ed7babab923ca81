"""Both sides of lines between routes: SAM output with scorings the gapless pass
does not take, reads around the length cut off by their windows, every trace
shape in two calls of one context, reads files around one block's size."""
import random

import numpy as np
import pytest

import test_gapless
import test_parse_small

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


def by_int32(ctx, call):
    ctx.set_sw_path(1)
    try:
        return call()
    finally:
        ctx.set_sw_path(0)


@pytest.mark.parametrize("kw", [dict(match=1, gap_open=-8), dict(gap_open=-15), dict(match=1, gap_open=-7)])
def test_sam_scorings(ctx, sg, oracle, kw):
    ref, reads = test_gapless.workload(31, 90, n=1600)
    ix = ctx.index(ref)
    p = sg.default_params(out_format=1, **kw)
    got, st = ctx.align(ix, reads, p, stats=True)
    # the packed passes took the pairs that hold bases only and were not settled
    assert st["records"] > 1100 and st["trace_cells"] > 0
    assert got == by_int32(ctx, lambda: ctx.align(ix, reads, p))
    assert got == oracle.align(ref, reads, oracle.default_params(
        device_mem=ctx.info()["total_mem"], out_format=1, **kw))


@pytest.mark.parametrize("L", [204, 205])
@pytest.mark.parametrize("n", [700, 9000])
def test_reads_cut_off(ctx, sg, L, n):
    # few and many left to the Smith-Waterman passes
    from swift_gb300 import synth
    names, seqs = synth.make_reference(200_000, 3, sigma=0.4, repeat_frac=0.2, n_units=15, seed=L)
    seqs[0][5000:5900] = np.frombuffer(b"ACGTTGCAAC" * 90, np.uint8)  # diagonals alike
    rn, rs, _ = synth.make_reads(seqs, n, L, 0.015, 0.0005, 0.05, seed=L + 1)
    reads = synth.reads_fasta(rn, rs)
    ix = ctx.index(synth.fasta_bytes(names, seqs))
    for fmt in (0, 1):
        p = sg.default_params(max_read_len=300, out_format=fmt)
        assert ctx.align(ix, reads, p) == by_int32(ctx, lambda: ctx.align(ix, reads, p)), fmt


@pytest.mark.parametrize("q", [36, 96, 104, 120, 128, 160, 250])
def test_every_shape_twice(sg, q):
    # scratch sized for the shape that runs, the first time and the second
    rng = np.random.default_rng(q)
    n, r = 2500, q + 128
    ref = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 400_000)].tobytes()
    ro = rng.integers(0, len(ref) - r, n)
    qo = ro + rng.integers(0, 128, n)
    ql, rl = np.full(n, q, np.int32), np.full(n, r, np.int32)
    c = sg.Context(0)
    shapes = set()
    for mode in (0, *range(2, 14)):
        c.set_tuning(mode)
        calls = [c.sw_pairs(ref, qo, ql, ref, ro, rl, consensus=False) for _ in range(2)]
        shapes |= set(calls[0][1]["shapes"].values())
        for res, st in calls:
            assert (res["score"] == 2 * q).all() and (res["len"] == q).all()
            assert np.array_equal(res["start"], qo - ro + 1) and st["generic_pairs"] == 0
    c.close()
    assert len(shapes) > 1


@pytest.mark.parametrize("size", [300, 65535, 65536, 65537])
def test_reads_file_sizes(ctx, oracle, size):
    rng = random.Random(3)
    ref = bytes(rng.choice(b"ACGT") for _ in range(60_000))
    fa = b">chr\n" + b"\n".join(ref[k:k + 60] for k in range(0, len(ref), 60)) + b"\n"
    ix = ctx.index(fa)
    text = test_parse_small.reads_of(ref, size)
    for t in (text, text[:-1]):
        want = oracle.align(fa, t, oracle.default_params(device_mem=ctx.info()["total_mem"]))
        assert len(want) > 900 and ctx.align(ix, t) == want


@pytest.mark.parametrize("L", [100, 204, 205, 250])
@pytest.mark.parametrize("fmt", [0, 1])
def test_no_packed_pair(ctx, sg, L, fmt):
    # windows cut short by their sequence's end: every pair is the int32 kernel's
    rng = random.Random(L)
    seqs = [bytes(rng.choice(b"ACGT") for _ in range(L + 40)) for _ in range(3)]
    reads = b"".join(b">r%d\n%s\n" % (i, seqs[i % 3][i:i + L]) for i in range(30))
    ix = ctx.index(test_gapless.fasta(seqs))
    p = sg.default_params(max_read_len=300, out_format=fmt)
    got, st = ctx.align(ix, reads, p, stats=True)
    assert st["sw_generic_pairs"] == st["records"] >= 30
    assert got == by_int32(ctx, lambda: ctx.align(ix, reads, p))
