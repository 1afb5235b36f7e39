"""FP64 tables and conductivities whose products come from sites where both sides are small: two
operators on separate regions of a strongly disordered chain, whose states hardly reach from one to the
other, and a local state seen from a distant region.  Every value of the recursions is known to its own
last bits there, and so are FP64 products: 1e-12 of the table's largest entry, as elsewhere (steps
below 300, each rounding once), and 1e-10 of the largest value for conductivities; and ten times what
changes of the Hamiltonian's values in their last bits make of the oracle's result, since the far tails
of the recursions multiply roundings."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def chain(N, W, seed=5):
    """Closed chain with on-site disorder of width W, rescaled; upper CSR."""
    i = np.arange(N)
    half = 1.05 * (2 + W / 2)
    eps = W * (lattices.uniform(seed, N) - 0.5) / half
    return lattices.upper_csr(N, np.concatenate([i, i]), np.concatenate([i, (i + 1) % N]),
                              np.concatenate([eps, np.full(N, 1 / half)]))


def current(N, first, width):
    """Bond currents of `width` bonds from site `first`; rows elsewhere are empty."""
    i = (first + np.arange(width)) % N
    return lattices.upper_csr(N, i, (i + 1) % N, np.full(width, 0.3j))


def operators(orc, *csr):
    N = len(csr[0][0]) - 1
    return [lq.Operator.from_csr(N, *c) for c in csr], [orc.Op(*c) for c in csr]


def reach(f, H, eps=2.0 ** -52):
    """f(oracle's H), and the largest change by relative changes eps of H's values."""
    rng = np.random.default_rng(3)
    want = f(H)
    moved = [f((H[0], H[1], H[2] * (1 + eps * (2 * rng.random(len(H[2])) - 1)))) for _ in range(3)]
    return want, max(np.abs(m - want).max() for m in moved)


@pytest.mark.parametrize("W,gap", [(1.0, 60), (8.0, 10), (8.0, 60), (20.0, 10), (20.0, 60)])
@pytest.mark.parametrize("N,R,M,block_width", [(1001, 2, 163, 0), (1001, 2, 163, 1), (701, 1, 40, 0), (35000, 1, 161, 0)])
def test_regions_apart(oracle_lib, N, R, M, block_width, W, gap):
    (H, A, B), (_, Ao, Bo) = operators(oracle_lib, chain(N, W), current(N, 100, 10), current(N, 110 + gap, 10))
    st = lattices.random_phase_states(N, R, seed=9)
    mu = lq.moments2d(H, A, B, st, M, opts=lq.make_opts(block_width=block_width))
    ref, last_bits = reach(lambda h: oracle_lib.moments2d(oracle_lib.Op(*h), Ao, Bo, st, M), chain(N, W))
    assert np.abs(mu - ref).max() <= 1e-12 * np.abs(ref).max() + 10 * last_bits


@pytest.mark.parametrize("W", [8.0, 20.0])
def test_local_state_and_a_distant_region(oracle_lib, W):
    N, M = 901, 200
    (H, B), (_, Bo) = operators(oracle_lib, chain(N, W), current(N, 490, 10))
    st = np.zeros((1, N), np.complex128)
    st[0, 450] = 1.0
    mu = lq.moments2d(H, None, B, st, M)
    ref, last_bits = reach(lambda h: oracle_lib.moments2d(oracle_lib.Op(*h), None, Bo, st, M), chain(N, W))
    assert np.abs(mu - ref).max() <= 1e-12 * np.abs(ref).max() + 10 * last_bits


@pytest.mark.parametrize("formula", [lq.KUBO_BASTIN, lq.KUBO_GREENWOOD])
@pytest.mark.parametrize("N,R,M,nump,block_width", [(960, 2, 64, 250, 0), (960, 3, 70, 300, 1), (9000, 4, 170, 1024, 0)])
@pytest.mark.parametrize("W,gap", [(20.0, 10), (8.0, 60)])
def test_conductivity_of_regions_apart(oracle_lib, N, R, M, nump, block_width, formula, W, gap):
    bw = 2 * 1.05 * (2 + W / 2)
    (H, A, B), (_, Ao, Bo) = operators(oracle_lib, chain(N, W), current(N, 100, 10), current(N, 110 + gap, 10))
    st = lattices.random_phase_states(N, R, seed=9)
    o = lq.make_opts(block_width=block_width)
    want = {k: reach(lambda h: oracle_lib.kubo_fft(oracle_lib.Op(*h), Ao, Bo, st, M, nump, formula, N, bw, 0.0)[k],
                     chain(N, W)) for k in ((1, 2) if formula == lq.KUBO_BASTIN else (1,))}

    def check(got):
        for k, (ref, last_bits) in want.items():
            assert np.abs(got[k] - ref).max() <= 1e-10 * np.abs(ref).max() + 10 * last_bits, k

    check(lq.kubo_fft(H, A, B, st, M, nump, formula, bw, 0.0, opts=o))
    if formula == lq.KUBO_BASTIN:
        mu, got = lq.kubo_bastin(H, A, B, st, M, nump, bw, 0.0, opts=o)
        check(got)
        ref, last_bits = reach(lambda h: oracle_lib.moments2d(oracle_lib.Op(*h), Ao, Bo, st, M), chain(N, W))
        assert np.abs(mu - ref).max() <= 1e-12 * np.abs(ref).max() + 10 * last_bits


def test_fp32_conductivity_of_regions_apart(oracle_lib):
    """Mixed precision: an integrand in the band's inner half is not lost, within ten times what changes of
    the Hamiltonian's values by 2^-24 make of it.  (The far tails, 1e-20, are within FP32's range.)"""
    N, R, M, nump, W = 960, 2, 70, 300, 20.0
    bw = 2 * 1.05 * (2 + W / 2)
    (H, A, B), (_, Ao, Bo) = operators(oracle_lib, chain(N, W), current(N, 100, 10), current(N, 140, 10))
    st = lattices.random_phase_states(N, R, seed=9)
    E, _, integ = lq.kubo_fft(H, A, B, st, M, nump, lq.KUBO_BASTIN, bw, 0.0, opts=lq.make_opts(precision=lq.PREC_MIXED))
    inner = np.abs(E) < 0.5 * bw / 2
    want, last_bits = reach(lambda h: oracle_lib.kubo_fft(oracle_lib.Op(*h), Ao, Bo, st, M, nump, lq.KUBO_BASTIN, N, bw,
                                                          0.0)[2][inner], chain(N, W), 2.0 ** -24)
    assert 10 * last_bits < np.abs(want).max()
    assert np.abs(integ[inner] - want).max() <= 10 * last_bits


def test_sums_beyond_the_range_are_those_of_fp64_products(oracle_lib):
    """States of 1e155: products overflow, and come out infinite or NaN, not as some finite sum."""
    N, M = 600, 170
    (H, V), _ = operators(oracle_lib, chain(N, 1.0), current(N, 0, N))
    st = lattices.random_phase_states(N, 1, seed=3)
    ok = lq.moments2d(H, V, V, st, M)
    mu = lq.moments2d(H, V, V, st * 1e156, M)
    large = np.abs(ok) > 1e-3 * np.abs(ok).max()
    assert not np.isfinite(mu[large]).any()
