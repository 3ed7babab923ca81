"""Contexts of several threads whose calls use one kernel with different amounts
of shared memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_int32_kernel_with_two_window_lengths():
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    rng = np.random.default_rng(3)
    Q, errors = 200, []

    def work(R):
        ctx = sg.Context(0)
        w = np.zeros((4, R + 1), np.uint8)
        w[:, :R] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, (4, R))]
        q = np.zeros((4, Q + 1), np.uint8)
        q[:, :Q] = w[:, 50:50 + Q]
        try:
            for _ in range(4000):
                score, start, end, ln = ctx.sw_batch_arrays(q, w, Q, R)
                assert (score == 2 * Q).all() and (start == 51).all() and (ln == Q).all()
        except Exception as e:
            errors.append(e)
        ctx.close()

    threads = [threading.Thread(target=work, args=(R,)) for R in (900, 950, 1000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
