"""Reads files around the size that one block parses whole: the same output as
the oracle, and the same errors as the larger files' path."""
import random
import re

import pytest

pytestmark = pytest.mark.gpu

LIMIT = 65536


@pytest.fixture(scope="module")
def sg():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300
    return swift_gb300


@pytest.fixture(scope="module")
def ctx(sg):
    return sg.Context(0)


@pytest.fixture(scope="module")
def ref():
    rng = random.Random(3)
    return bytes(rng.choice(b"ACGT") for _ in range(60_000))


def reads_of(ref, size):
    """A reads file of exactly `size` bytes: reads of 100 bases, names of about
    20 letters."""
    rng = random.Random(size)
    m, out = max(1, size // 125), []
    for i in range(m):
        n = size // m + (1 if i < size % m else 0)
        at = rng.randrange(len(ref) - 100)
        out.append(b">" + (b"r%05d" % i + b"x" * 48)[:n - 103] + b"\n" + ref[at:at + 100] + b"\n")
    return b"".join(out)


@pytest.mark.parametrize("size", [300, LIMIT - 1, LIMIT, LIMIT + 1])
def test_valid_files(ctx, oracle, ref, size):
    text = reads_of(ref, size)
    assert len(text) == size
    fa = b">chr\n" + b"\n".join(ref[k:k + 60] for k in range(0, len(ref), 60)) + b"\n"
    ix = ctx.index(fa)
    p = oracle.default_params(device_mem=ctx.info()["total_mem"])
    for t in (text, text[:-1]):  # with and without the last newline
        try:
            want = oracle.align(fa, t, p)
        except Exception:
            continue
        assert ctx.align(ix, t) == want


BAD = [b">a\nACGT\x00" + b"A" * 95 + b"\n", b">a\n" + b"A" * 50 + b">" + b"C" * 49 + b"\n",
       b">a\n\n", b"ACGT\n", b">a\n>b\n" + b"A" * 100 + b"\n", b">a\n" + b"A" * 300 + b"\n",
       b">" + b"n" * 60 + b"\n" + b"A" * 100 + b"\n", b">tail\n", b"\n\n\n"]


@pytest.mark.parametrize("k", range(len(BAD)))
def test_errors_alike(ctx, sg, ref, k):
    fa = b">chr\n" + ref + b"\n"
    ix = ctx.index(fa)
    said = []
    for n in (0, 300, 900):  # alone, within one block, beyond it
        good = b"".join(b">r%d\n%s\n" % (i, ref[i:i + 100]) for i in range(n))
        with pytest.raises(sg.SwiftError) as e:
            ctx.align(ix, good + BAD[k])
        said.append((e.value.code, re.sub(r"offset \d+", "offset", str(e.value)),
                     [int(v) - len(good) for v in re.findall(r"offset (\d+)", str(e.value))]))
    # (a first line that is no header is reported as such, a later one as a second line)
    assert said[1] == said[2] and (said[0] == said[1] or k in (3, 8))
