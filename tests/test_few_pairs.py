"""Calls that leave few pairs to the Smith-Waterman passes: which kernel takes
them, what the statistics say of it, and the same output either way."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300
    return swift_gb300


def workload(n, L):
    """(reference, reads): reads with too many mismatches for the gapless pass."""
    from swift_gb300 import synth
    names, seqs = synth.make_reference(300_000, 3, sigma=0.4, repeat_frac=0.1, n_units=12, seed=L)
    rn, rs, _ = synth.make_reads(seqs, n, L, 0.06, 0.002, 0.05, seed=n)
    return synth.fasta_bytes(names, seqs), synth.reads_fasta(rn, rs)


@pytest.mark.parametrize("n", [30, 300, 1500])
def test_no_first_pass_in_small_calls(sg, n):
    # traced at once by the packed passes, or (the second) all on the int32 kernel
    ref, reads = workload(n, 100)
    ctx = sg.Context(0)
    _, st = ctx.align(ctx.index(ref), reads, stats=True)
    assert (st["sw_generic_pairs"] > 100) == (n == 300)
    assert (st["first_pass_kind"], st["first_pass_cells"], st["first_pass_ms"]) == (0, 0, 0.0)


@pytest.mark.parametrize("L,fmt,n,int32", [
    (128, 0, 300, True), (129, 0, 300, False), (204, 1, 300, False), (205, 1, 300, True),
    (224, 0, 300, False), (225, 0, 300, True), (225, 0, 560, False), (256, 0, 300, True),
    (256, 1, 560, True), (257, 0, 300, False), (257, 1, 300, True), (257, 1, 560, False)])
def test_kernel_by_rows(sg, L, fmt, n, int32):
    # by rows per lane, at the edges; the same bytes as the int32 kernel's
    ref, reads = workload(n, L)
    ctx = sg.Context(0)
    ix = ctx.index(ref)
    p = sg.default_params(max_read_len=300, out_format=fmt)
    got, st = ctx.align(ix, reads, p, stats=True)
    assert 100 < st["records"] <= 1024 and (st["sw_generic_pairs"] > 100) == int32
    ctx.set_sw_path(1)
    assert got == ctx.align(ix, reads, p)
