"""The int32 kernel and swift_sw_batch's packed pairs against the oracle at
their edges: query lengths around the rows per lane and lanes, scorings whose
values fit the coded cells and ones that do not, gap scores above zero, bytes
outside ACGT, batches around the packed passes' smallest size.
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


def pairs(n, Q, R, seed, odd=0.5):
    rng = random.Random(seed)
    qs, ws = [], []
    for i in range(n):
        w = bytearray(rng.choice(b"ACGT") for _ in range(R))
        at = rng.randrange(max(1, R - Q + 1))
        q = bytearray((w[at:at + Q] + bytes(rng.choice(b"ACGT") for _ in range(Q)))[:Q])
        for _ in range(i % 6):
            q[rng.randrange(Q)] = rng.choice(b"ACGT")
        if i % 5 == 2 and Q > 8:
            k = rng.randrange(1, Q - 4)
            q = (q[:k] + q[k + 2:] + b"GT")[:Q]
        if rng.random() < odd:
            q[rng.randrange(Q)] = rng.choice(b"NnRacgt")
            w[rng.randrange(R)] = rng.choice(b"NnY\0acgt")
        qs.append(bytes(q))
        ws.append(bytes(w))
    return qs, ws


def check(got, want):
    assert got["score"] == want["score"]
    for key in ("start", "end", "len", "qcons", "rcons"):
        assert got[key] == want[key], key


@pytest.mark.parametrize("sc", [(2, -1, -10, -1), (2, -1, -1, -10), (1, 1, -2, -3), (3, -2, 1, -1),
                                (2, -3, -4, 2), (32767, -32767, -32767, -1), (0, -1, -2, -2)])
@pytest.mark.parametrize("Q,R", [(1, 1), (3, 40), (4, 5), (5, 33), (127, 130), (129, 64), (257, 300)])
def test_batch_scorings(ctx, oracle, Q, R, sc):
    m, x, o, e = sc
    qs, ws = pairs(12, Q, R, 7 * Q + R)
    got = ctx.sw_batch(qs, ws, Q, R, m, x, o, e)
    for g, q, w in zip(got, qs, ws):
        check(g, oracle.sw(q, w, Q, R, m, x, o, e))


@pytest.mark.parametrize("big", [1 << 20, 1 << 21])
def test_scores_beyond_the_coded_cells(ctx, oracle, big):
    m, x, o, e = 2 * big, -big, -4 * big, -big
    qs, ws = pairs(20, 90, 120, 31)
    off = lambda v: np.concatenate([[0], np.cumsum([len(s) for s in v])[:-1]])
    res, _ = ctx.sw_pairs(b"".join(qs), off(qs), [90] * 20, b"".join(ws), off(ws), [120] * 20,
                          m, x, o, e)
    for i in range(20):
        want = oracle.sw(qs[i], ws[i], 90, 120, m, x, o, e)
        check({k: res[k][i] for k in res}, want)


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 3278, 3279, 6200])
def test_batch_sizes(ctx, oracle, n):
    # every size gives each pair its own result: the first, the last and a
    # sample against the oracle, all of them against halves of the batch
    Q, R = 61, 150
    qs, ws = pairs(n, Q, R, n, odd=0.02)
    q = np.zeros((n, Q + 1), np.uint8)
    w = np.zeros((n, R + 1), np.uint8)
    q[:, :Q] = np.frombuffer(b"".join(qs), np.uint8).reshape(n, Q)
    w[:, :R] = np.frombuffer(b"".join(ws), np.uint8).reshape(n, R)
    got = ctx.sw_batch_arrays(q, w, Q, R)
    h = n // 2
    if h:
        halves = [ctx.sw_batch_arrays(q[s].copy(), w[s].copy(), Q, R)
                  for s in (slice(0, h), slice(h, n))]
        for k in range(4):
            assert np.array_equal(got[k], np.concatenate([halves[0][k], halves[1][k]]))
    for i in sorted({0, n - 1, n // 3, n // 2}):
        check(ctx.sw_batch([qs[i]], [ws[i]], Q, R)[0], oracle.sw(qs[i], ws[i], Q, R))
        want = oracle.sw(qs[i], ws[i], Q, R)
        assert tuple(int(got[k][i]) for k in range(4)) == tuple(
            int(want[k]) for k in ("score", "start", "end", "len"))


@pytest.mark.parametrize("n", [40, 4100])
def test_batch_leaves_bytes_past_the_strings(sg, ctx, n):
    # device buffers: only len bytes of each consensus row are written
    torch = pytest.importorskip("torch")
    Q, R = 50, 97
    qs, ws = pairs(n, Q, R, 5, odd=0.1)
    q = torch.zeros((n, Q + 1), dtype=torch.uint8)
    w = torch.zeros((n, R + 1), dtype=torch.uint8)
    q[:, :Q] = torch.from_numpy(np.frombuffer(b"".join(qs), np.uint8).reshape(n, Q).copy())
    w[:, :R] = torch.from_numpy(np.frombuffer(b"".join(ws), np.uint8).reshape(n, R).copy())
    q, w = q.cuda(), w.cuda()
    score = torch.zeros(n, device="cuda")
    st, en, ln = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
    qc, rc = (torch.full((n, Q + R + 2), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx._check(sg.lib().swift_sw_batch(ctx._h, q.data_ptr(), w.data_ptr(), Q, R, n, 2, -1, -10, -1,
                                       score.data_ptr(), st.data_ptr(), en.data_ptr(),
                                       ln.data_ptr(), qc.data_ptr(), rc.data_ptr()))
    past = torch.arange(Q + R + 2, device="cuda")[None, :] >= ln[:, None]
    for c in (qc, rc):
        assert bool((c[past] == 0x7E).all()) and not bool((c[~past] == 0x7E).any())


@pytest.mark.parametrize("Q", [20, 33, 64, 65, 100, 128, 150, 199])
@pytest.mark.parametrize("n_reads", [900, 2600, 9000])
def test_packed_paths_of_the_aligner(ctx, sg, Q, n_reads):
    # reads with too many differences for the gapless pass: few, some and many
    # pairs left (the int32 kernel, the trace of them all in 32 or 16 lanes,
    # bounded selection) print what the int32 kernel prints for every pair
    from swift_gb300 import synth
    names, seqs = synth.make_reference(150_000, 2, sigma=0.3, repeat_frac=0.2, n_units=20, seed=Q)
    ref = synth.fasta_bytes(names, seqs)
    rn, rs, _ = synth.make_reads(seqs, n_reads, Q, 0.06, 0.004, 0.05, seed=Q + 1)
    reads = synth.reads_fasta(rn, rs)
    ix = ctx.index(ref)
    for fmt in (0, 1):
        p = sg.default_params(out_format=fmt)
        got = ctx.align(ix, reads, p)
        ctx.set_sw_path(1)
        try:
            assert got == ctx.align(ix, reads, p), fmt
        finally:
            ctx.set_sw_path(0)
