"""A call that fails, for want of memory or of the device it names, leaves nothing
behind: the thread's next call gives its own result."""
import random

import numpy as np
import pytest

from test_long_scratch import CappedPool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pairs", "align"])
def test_call_after_out_of_memory(kind):
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    rng = random.Random(11)
    ref = bytes(rng.choice(b"ACGT") for _ in range(100_000))
    ctx = sg.Context(0)
    if kind == "align":
        ix = ctx.index(b">chr\n" + ref + b"\n")
        reads = b"".join(b">r%d\n%s\n" % (i, ref[i:i + 100]) for i in range(60_000))
        call = lambda: ctx.align(ix, reads)
    else:
        off = np.arange(60_000, dtype=np.int64)
        ql, rl = np.full(len(off), 100, np.int32), np.full(len(off), 300, np.int32)
        call = lambda: ctx.sw_pairs(ref, off, ql, ref, off, rl, consensus=False)[0]["score"].tobytes()
    want = call()
    with CappedPool(16 << 20):
        with pytest.raises(sg.SwiftError):
            call()
    assert call() == want


def test_call_after_a_device_that_is_not_there():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    rng = random.Random(4)
    ref = bytes(rng.choice(b"ACGT") for _ in range(3000))
    ctx = sg.Context(0)
    ix = ctx.index(b">chr\n" + ref + b"\n")
    reads = b">r\n" + ref[500:600] + b"\n"
    want = ctx.align(ix, reads)
    with pytest.raises(sg.SwiftError):
        sg.Context(4096)
    assert ctx.align(ix, reads) == want
    with pytest.raises(sg.SwiftError):
        sg.Server(ix, 4096)
    assert ctx.align(ix, reads) == want
