"""sigma(E) from the moment table in double-double, at sizes the dispatch sends there, against the
oracle's site-by-site transforms (1e-10 of the maximum over all energies, the repository's bar
for conductivities; both sides round p and w to FP64 at least once, which the division by
(1 - E^2)^2 carries into sigma at 1e-13 and into the integrand's edge at 1e-12 here)."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def setup(orc, Lx, Ly):
    N, H, V = lattices.honeycomb(Lx, Ly, t=-2.7, W=1.0, seed=21)
    lo, hi = lattices.gershgorin_bounds(N, *H)
    bw, bc = 1.05 * (hi - lo), (hi + lo) / 2
    Hg = lq.Operator.from_csr(N, *H)
    Hg.rescale_to_chebyshev(bw, bc)
    return N, bw, bc, Hg, lq.Operator.from_csr(N, *V), orc.Op(*H).rescale(2 / bw, -bc / (bw / 2)), orc.Op(*V)


# energies: even and odd, prime (the only split of 2 n is 2), above the shared-memory transforms'
# range, equal to M; moments: 3, a remainder of the split, more than one row group
@pytest.mark.parametrize("Lx,Ly,R,M,nump", [(24, 20, 2, 64, 250), (24, 20, 2, 65, 301), (24, 20, 2, 61, 251),
                                            (24, 20, 2, 250, 250), (80, 80, 1, 3, 1000), (32, 36, 4, 170, 1024),
                                            (16, 16, 2, 70, 2100)])
@pytest.mark.parametrize("formula", [lq.KUBO_BASTIN, lq.KUBO_GREENWOOD])
def test_sigma_matches_oracle(oracle_lib, Lx, Ly, R, M, nump, formula):
    N, bw, bc, H, V, Ho, Vo = setup(oracle_lib, Lx, Ly)
    st = lattices.random_phase_states(N, R, seed=22)
    E, s, integ = lq.kubo_fft(H, V, V, st, M, nump, formula, bw, bc)
    Eo, so, io, _ = oracle_lib.kubo_fft(Ho, Vo, Vo, st, M, nump, formula, N, bw, bc)
    assert np.abs(E - Eo).max() <= 1e-13 * np.abs(Eo).max()
    assert np.abs(s - so).max() <= 1e-10 * np.abs(so).max()
    if formula == lq.KUBO_BASTIN:
        assert np.abs(integ - io).max() <= 1e-10 * np.abs(io).max()


def test_chunks_of_vectors_and_both_results(oracle_lib):
    """Blocks of one vector each add into one table; the moments come from the same table."""
    N, bw, bc, H, V, Ho, Vo = setup(oracle_lib, 24, 20)
    st = lattices.random_phase_states(N, 3, seed=5)
    M, nump = 70, 300
    mu, (E, s, integ) = lq.kubo_bastin(H, V, V, st, M, nump, bw, bc, opts=lq.make_opts(block_width=1))
    Eo, so, io, _ = oracle_lib.kubo_fft(Ho, Vo, Vo, st, M, nump, lq.KUBO_BASTIN, N, bw, bc)
    muo = oracle_lib.moments2d(Ho, Vo, Vo, st, M)
    assert np.abs(s - so).max() <= 1e-10 * np.abs(so).max()
    assert np.abs(mu - muo).max() <= 1e-12 * np.abs(muo).max()


def test_fp32_vectors(oracle_lib):
    """The mixed solve's table of its FP32 blocks: sigma at the mode's bound."""
    N, bw, bc, H, V, Ho, Vo = setup(oracle_lib, 24, 20)
    st = lattices.random_phase_states(N, 2, seed=5)
    M, nump = 64, 300
    _, s, _ = lq.kubo_fft(H, V, V, st, M, nump, lq.KUBO_BASTIN, bw, bc, opts=lq.make_opts(precision=lq.PREC_MIXED))
    _, so, _, _ = oracle_lib.kubo_fft(Ho, Vo, Vo, st, M, nump, lq.KUBO_BASTIN, N, bw, bc)
    lo, hi = nump // 20, nump - nump // 20
    assert 0 < np.abs(s - so)[lo:hi].max() < 1e-6 * np.abs(so[lo:hi]).max()


def test_too_many_moments_stay_refused(oracle_lib):
    """More moments than the direct transforms take are an error before and after."""
    N, bw, bc, H, V, _, _ = setup(oracle_lib, 4, 4)
    with pytest.raises(lq.LinqtError):
        lq.kubo_fft(H, V, V, lattices.random_phase_states(N, 1, 1), 7300, 7300, lq.KUBO_BASTIN, bw, bc)
