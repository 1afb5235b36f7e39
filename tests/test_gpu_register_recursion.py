"""1D moments with the operator's entries in registers, one value of the block a thread, against the
kernel that a forced thread shape selects.  The vectors are the same bits; the moments sum the same
terms, whose absolute values add up to at most 1, in another order and in chains of fewer than 400
additions: 400 x 1.1e-16, doubled by the moment formula, is below 1e-13."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def banded(N, row, seed=5):
    """Hermitian operator of at most `row` entries a row: the diagonal, for even `row` half of the
    rows paired over N / 2, and bonds to the next sites; open at both ends, so that rows differ in
    length.  Norm below 1."""
    i = np.arange(N)
    rows, cols, vals = [i], [i], [(0.2 * (lattices.uniform(seed, N) - 0.5)).astype(complex)]
    far = (row - 1) // 2
    for d in range(1, far + 1):
        rows.append(i[:-d])
        cols.append(i[d:])
        vals.append(np.full(N - d, (0.35 + 0.02j * d) / far))
    if row % 2 == 0:
        h = N // 2
        rows.append(i[:h])
        cols.append(i[:h] + h)
        vals.append(np.full(h, 0.1j))
    return lq.Operator.from_csr(N, *lattices.upper_csr(N, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)))


# longest rows on both sides of every variant; blocks beyond the cluster's sizes, up to one thread
# beyond what two, three and four CTAs of 256 threads on each of 148 SMs cover
CASES = [(4, 17000, 1), (3, 25000, 1), (4, 75776, 1), (4, 75777, 1), (4, 14000, 8), (4, 113665, 1), (4, 151552, 1), (4, 151553, 1),
         (5, 9001, 2), (6, 37889, 2), (6, 56832, 2), (6, 56833, 2), (7, 2500, 4), (8, 75776, 1), (8, 75777, 1), (9, 37888, 1),
         (15, 1100, 5), (16, 37888, 1), (16, 37889, 1), (17, 9000, 1)]


@pytest.mark.parametrize("row,N,R", CASES)
@pytest.mark.parametrize("precision", [lq.PREC_FP64, lq.PREC_MIXED])
def test_moments_equal_the_other_kernel(row, N, R, precision):
    H = banded(N, row)
    i = np.arange(N)
    V = lq.Operator.from_csr(N, *lattices.upper_csr(N, i, (i + 1) % N, np.full(N, 0.3j)))
    st = lattices.random_phase_states(N, R, seed=3)
    for op, M in ((None, 41), (V, 24), (None, 2), (V, 1)):
        a, b = (lq.moments1d(H, op, st, M, opts=lq.make_opts(precision=precision, thread_shape=t)) for t in (0, 1))
        assert np.abs(a - b).max() <= 1e-13 * max(1.0, np.abs(b).max())
