"""The persistent recursions take a row's entries four at a time and the one to three that remain at
once: operators whose rows have 1 to 9 entries, in every layout and thread shape, against the oracle.

FP64: both sides round each of at most 9 products and sums of a row, and a rounding of step m grows at
most m-fold over the steps that follow: 2 x 18 x (1 + ... + 11) x 1.1e-16 < 3e-13 of the moments' bound.
FP32 vectors: one rounding of 2^-24 a value and step, for both vectors of a product: 2 x 66 x 6e-8
< 1e-5."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu

M, R = 12, 8
TOL = {lq.PREC_FP64: 3e-13, lq.PREC_MIXED: 1e-5}


def operators(oracle, N, row):
    """Hermitian band of at most `row` entries a row, open at both ends, norm below 1."""
    i = np.arange(N)
    rows, cols, vals = [i], [i], [(0.2 * (lattices.uniform(7, N) - 0.5)).astype(complex)]
    far = (row - 1) // 2
    for d in range(1, far + 1):
        rows.append(i[:-d])
        cols.append(i[d:])
        vals.append(np.full(N - d, (0.3 + 0.02j * d) / far))
    if row % 2 == 0:
        h = N // 2
        rows.append(i[:h])
        cols.append(i[:h] + h)
        vals.append(np.full(h, 0.1j))
    csr = lattices.upper_csr(N, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))
    return lq.Operator.from_csr(N, *csr), oracle.Op(*csr)


@pytest.mark.parametrize("row", range(1, 10))
@pytest.mark.parametrize("precision", [lq.PREC_FP64, lq.PREC_MIXED])
def test_moments(oracle_lib, row, precision):
    N = 5003
    H, Ho = operators(oracle_lib, N, row)
    V, Vo = operators(oracle_lib, N, 10 - row)
    st = lattices.random_phase_states(N, R, seed=4)
    one, two = oracle_lib.moments1d(Ho, Vo, st, M), oracle_lib.moments2d(Ho, Vo, Vo, st, M)
    for fmt in (0, 1, 3):  # CSR, SELL, locality order
        for shape in (1, 2, 3, 4):
            got = lq.moments1d(H, V, st, M, opts=lq.make_opts(precision=precision, fmt=fmt, thread_shape=shape))
            assert np.abs(got - one).max() <= TOL[precision] * 2
        got = lq.moments2d(H, V, V, st, M, opts=lq.make_opts(precision=precision, fmt=fmt))
        assert np.abs(got - two).max() <= TOL[precision] * 4
