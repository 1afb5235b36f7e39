"""The real energy sums (one FP64 tensor-core product with the left coefficients in its epilogue)
at the edges of its 128 x 64 tiles and K slices of 16, against the oracle.  1e-11 of the maximum:
sums of at most 2 x 130 products with coefficients up to m / f0^3 (3e4 at xbound 0.95), each
rounded once on both sides."""
import numpy as np
import pytest

import linqt_b200 as lq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M0,M1,num_div", [(7, 8, 127), (8, 7, 128), (63, 65, 129), (64, 16, 257), (65, 17, 300),
                                           (128, 9, 384), (130, 128, 1000)])
@pytest.mark.parametrize("variant", ["bastin", "greenwood", "bastin_I", "bastin_II", "bastin_sea", "bastin_surf"])
def test_edges(oracle_lib, M0, M1, num_div, variant):
    rng = np.random.default_rng(M0 * 1000 + M1)
    mu = rng.standard_normal((M0, M1)) + 1j * rng.standard_normal((M0, M1))
    bw, bc, broad = 6.0, 0.2, 1e-3  # no truncation
    muj = oracle_lib.jackson2d(mu, bw, broad, broad)
    assert muj.shape == mu.shape
    E, out = lq.kubo_from_moments(mu, 500, bw, bc, broad, variant=variant, xbound=0.95, num_div=num_div)
    Eo, oo = oracle_lib.kubo_from_moments(muj, 500, bw, bc, variant, xbound=0.95, num_div=num_div)
    assert len(E) == len(Eo) == num_div - 1
    assert np.abs(out - oo).max() <= 1e-11 * np.abs(oo).max()
