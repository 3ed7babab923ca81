"""Pairs the LCS bound keeps: few are traced at once, many are scored and the
printed ones traced again; a call that leaves few pairs traces them all.
Either way the output is that of scoring every pair."""
import pytest

pytestmark = pytest.mark.gpu

ROWS = 1_500_000


@pytest.mark.parametrize("n,L,many", [(5_000, 100, None), (9_000, 100, False),
                                      (7_000, 230, False), (130_000, 100, True)])
def test_kept_pairs(n, L, many):
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    from swift_gb300 import synth
    names, seqs = synth.make_reference(400_000, 4, sigma=0.5, repeat_frac=0.3, n_units=40,
                                       unit_len=300, divergence=0.02, seed=211)
    rn, rs, _ = synth.make_reads(seqs, n, L, 0.02, 0.004, 0.05, seed=n)
    ctx = sg.Context(0)
    ix = ctx.index(synth.fasta_bytes(names, seqs))
    reads = synth.reads_fasta(rn, rs)
    p = sg.default_params(max_read_len=300)
    got, st = ctx.align(ix, reads, p, stats=True)
    assert (st["first_pass_kind"] == 3) == (many is not None)
    if many is not None:
        assert st["retraced_pairs"] > 0 and (st["lcs_kept"] * L > ROWS) == many
    ctx.set_sw_path(2)
    assert got == ctx.align(ix, reads, p)
