"""An operator and its sparse layouts are on the device before the first kernel that reads them: a
recursion right after the layout is built, on fresh operators with other values in the memory that
the last ones gave back, equals the same recursion on the layout that is there already."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [lq.FORMAT_SELL, lq.FORMAT_LOCAL, lq.FORMAT_CSR])
def test_first_use_equals_the_second(fmt):
    N = 40003
    st = lattices.random_phase_states(N, 1, seed=3)
    i = np.arange(N)
    rows, cols = np.concatenate([i, i, i]), np.concatenate([i, (i + 1) % N, (i + 2) % N])
    for trial in range(12):
        vals = np.concatenate([0.2 * (lattices.uniform(trial, N) - 0.5), np.full(N, 0.3), np.full(N, 0.1 + 0.05j)])
        H = lq.Operator.from_csr(N, *lattices.upper_csr(N, rows, cols, vals))
        a, b = (lq.moments2d(H, None, None, st, 8, opts=lq.make_opts(fmt=fmt)) for _ in range(2))
        assert np.array_equal(a, b), trial
