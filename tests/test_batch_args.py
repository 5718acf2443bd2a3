"""Argument structures of a batch, filled by column, against one filled field by
field (as single joins' are): also for windows that the engine refuses, which have
to reach it to be refused there."""
import numpy as np
import pytest


@pytest.mark.parametrize("windows", [[64, 32, 100], [np.int64(64), 32.0, 7], [-5, 0, 3],
                                     [64, -1, 2 ** 62], [2 ** 63, 2 ** 64 + 5, 64]])
def test_batch_args_by_column(windows):
    import scamp_gb300 as s

    series = [np.arange(n, dtype=np.float64) for n in (200, 0, 90)]
    arrs, _, got = s._batch_args(series, windows, "mixed", 0)
    for x, m, ca in zip(arrs, windows, got):
        want = s._args(x, None, m, "1NN_INDEX", "mixed", True, True, False, False, 0.0, -1, -1,
                       max(128000, 2 * int(m)), 0, 0, True)
        for name, _ in ca._fields_[:-1]:  # (but the reserved words)
            assert getattr(ca, name) == getattr(want, name), (m, name)
