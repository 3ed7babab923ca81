"""Best-per-read groups of the gapless pass: consecutive reads of one name make
one group, inside a warp's 32 records, across its end and longer than it; names
that differ in their last character or before it."""
import re

import pytest

from test_gapless import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run,suffix", [(1, b""), (1, b"x"), (2, b""), (5, b"x*"), (12, b""),
                                        (33, b"*"), (100, b"")])
def test_groups(oracle, run, suffix):
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    ref, reads = workload(300 + run, 100, n=1300)
    reads = re.sub(rb">r(\d+)", lambda m: b">r%d" % (int(m[1]) // run) + suffix, reads)
    ctx = sg.Context(0)
    got = ctx.align(ctx.index(ref), reads)
    assert got == oracle.align(ref, reads, oracle.default_params(
        device_mem=ctx.info()["total_mem"]))
