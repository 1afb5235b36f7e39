"""The recursions of small lattices in one cluster (vectors in shared memory) against the grid
kernels, which the SELL layout and a forced thread shape select: the L/R blocks are the same bits,
so the 2D tables are equal; the 1D moments sum the same terms in another order (M = 60 sums of at
most 33k terms below 1: 1e-13)."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def ring(N, seed=5):
    """Closed ring with disorder and second neighbours, and its current operator."""
    i = np.arange(N)
    eps = 0.2 * (lattices.uniform(seed, N) - 0.5)
    rows, cols, vals = [i], [i], [eps.astype(complex)]
    for d, t in ((1, 0.3), (2, 0.1 + 0.05j)):
        if N > 2 * d:
            rows.append(i)
            cols.append((i + d) % N)
            vals.append(np.full(N, t))
    H = lattices.upper_csr(N, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))
    V = lattices.upper_csr(N, i, (i + 1) % N, np.full(N, 0.3j)) if N > 2 else H
    return lq.Operator.from_csr(N, *H), lq.Operator.from_csr(N, *V)


# one CTA to sixteen, rows that do not divide among them (the last CTAs without any), one pass and
# several per thread, the last sizes on either side of the dispatch's line
SIZES = [(1, 1), (2, 1), (3, 2), (31, 1), (127, 1), (129, 1), (130, 3), (257, 4), (513, 1), (999, 2), (1025, 8), (2047, 1),
         (65, 32), (33, 64), (2000, 5), (16000, 1), (16001, 1)]


@pytest.mark.parametrize("N,R", SIZES)
@pytest.mark.parametrize("precision", [lq.PREC_FP64, lq.PREC_MIXED])
def test_tables_equal_the_grid_kernels(N, R, precision):
    H, V = ring(N)
    st = lattices.random_phase_states(N, R, seed=3)
    for opl, opr in ((V, V), (None, None)):
        a, b = (lq.moments2d(H, opl, opr, st, 24, opts=lq.make_opts(precision=precision, fmt=f))
                for f in (lq.FORMAT_CSR, lq.FORMAT_SELL))
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N,R", SIZES)
@pytest.mark.parametrize("precision", [lq.PREC_FP64, lq.PREC_MIXED])
@pytest.mark.parametrize("M", [1, 2, 60, 61])
def test_moments_equal_the_grid_kernels(N, R, precision, M):
    H, V = ring(N)
    st = lattices.random_phase_states(N, R, seed=3)
    for op in (None, V):
        a, b = (lq.moments1d(H, op, st, M, opts=lq.make_opts(precision=precision, thread_shape=t)) for t in (0, 1))
        assert np.abs(a - b).max() <= 1e-13 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("N,R", [(1, 1), (31, 1), (257, 4), (2000, 5)])
def test_time_correlations(oracle_lib, N, R):
    """The evolution series and the recursions from evolved states."""
    i = np.arange(N)
    Hc = lattices.upper_csr(N, i, (i + 1) % N, np.full(N, 0.3)) if N > 2 else lattices.upper_csr(N, i, i, np.full(N, 0.3))
    H, Ho = lq.Operator.from_csr(N, *Hc), oracle_lib.Op(*Hc)
    st = lattices.random_phase_states(N, R, seed=3)
    got = lq.moments_td(H, None, None, st, 20, 3, 0.7, 8.0, 0.3)
    want = oracle_lib.moments_td(Ho, None, None, st, 20, 3, 0.7, 8.0, 0.3)
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()
