"""The shape a launch of several row classes was tuned to is not taken for a
launch of its tallest class alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shape_of_a_mixed_launch_is_its_own():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    rng = np.random.default_rng(5)
    ref = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 400_000)].tobytes()

    def call(ctx, ql):
        rl = np.full(len(ql), 232, np.int32)
        ro = rng.integers(0, len(ref) - 232, len(ql))
        res, st = ctx.sw_pairs(ref, ro + 60, ql, ref, ro, rl, consensus=False)
        assert (res["score"] == 2 * ql).all() and st["segments"] == 1
        return st["tune_ms"] > 0

    mixed = np.repeat([96, 104], 1500).astype(np.int32)  # too few each for a launch of its own
    tall = np.full(3000, 104, np.int32)
    ctx = sg.Context(0)
    assert call(ctx, mixed) and not call(ctx, mixed)
    assert call(ctx, tall) and not call(ctx, tall) and not call(ctx, mixed)
    other = sg.Context(0)  # the tallest class's own choice serves the mix
    assert call(other, tall) and not call(other, mixed)
