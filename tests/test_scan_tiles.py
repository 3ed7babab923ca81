"""Index bucket starts are prefix sums over 4^k buckets: seed lengths on both
sides of one tile (2,048 sums) and of the tile count whose sums every block
adds up itself (2,048)."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5, 6, 9, 11, 12])
def test_bucket_starts(k):
    from swift_gb300 import build as b
    b.build()
    import swift_gb300
    rng = random.Random(k)
    seq = bytes(rng.choice(b"ACGT") for _ in range(600_000))
    code = np.zeros(256, np.int64)
    code[list(b"ACGT")] = range(4)
    c = code[np.frombuffer(seq, np.uint8)]
    n = len(seq) // k
    h = (c[:n * k].reshape(n, k) << (2 * np.arange(k))).sum(axis=1)
    want = np.bincount(h, minlength=4 ** k)
    look, rep, ri, rp = swift_gb300.Context(0).index(b">s\n" + seq + b"\n", k, 1 << 20).export()
    occ = want > 0
    assert np.array_equal(np.asarray(rep)[occ], want[occ])
    assert np.array_equal(np.asarray(look)[occ], (np.cumsum(want) - want + 1)[occ])  # (1-based)
    assert len(rp) == n + 1
