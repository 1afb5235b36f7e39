"""The FP64 moment contraction in residues on the INT8 tensor cores, at the edges of its tiles,
K chunks and dispatch, against numpy's FP64 products of the same recursion.

Tolerance 1e-12 of max|mu|: both sides round each of at most 300 recursion steps (300 eps, with
a growth below the square of that number over 300 in the three-term recursion, ~1e-13) and numpy
its sums; the contraction itself adds at most 2^-53 of each row's norm.
"""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def chain(N, seed=5):
    """Closed chain with disorder, and its current operator (upper CSR)."""
    i = np.arange(N)
    eps = 0.3 * (lattices.uniform(seed, N) - 0.5)
    rows, cols = np.concatenate([i, i]), np.concatenate([i, (i + 1) % N])
    H = lattices.upper_csr(N, rows, cols, np.concatenate([eps, np.full(N, 0.45)]))
    V = lattices.upper_csr(N, i, (i + 1) % N, np.full(N, 0.45j))
    return H, V


def table(N, H, V, states, M):
    """The symmetrised table in numpy."""
    def full(csr):
        rp, c, v = csr
        r = np.repeat(np.arange(N), np.diff(rp))
        off = r != c
        order = np.argsort(np.concatenate([r, c[off]]), kind="stable")
        rows = np.concatenate([r, c[off]])[order]
        cols = np.concatenate([c, r[off]])[order]
        vals = np.concatenate([v, v[off].conj()])[order]
        start = np.searchsorted(rows, np.arange(N))
        return lambda x: np.add.reduceat(vals[:, None] * x[cols], start, axis=0)

    h, vel = full(H), full(V)
    x = states.T

    def blocks(t):
        out = [t, h(t)]
        for _ in range(M - 2):
            out.append(2 * h(out[-1]) - out[-2])
        return out[:M]

    L = np.array([t.ravel() for t in blocks(vel(x))])
    R = np.array([vel(t).ravel() for t in blocks(x)])
    raw = L.conj() @ R.T
    mu = (raw + raw.conj().T) / 2 * 4 / len(states)
    mu[0] /= 2
    mu[:, 0] /= 2
    return mu


# M: below, at and above the 128-row halves and the 256 x 256 tile, and the lower ends of the
# dispatch; K = N R: around the 128-value block, the 4096-value part, the 8192 line of small
# tables and the 32768-value chunk (odd N with one vector: rows 16-byte aligned only)
@pytest.mark.parametrize("N,R,M", [(192, 1, 8), (193, 1, 31), (1021, 2, 100), (4097, 2, 9), (129, 2, 127),
                                   (128, 2, 128), (255, 1, 129), (257, 1, 161), (4095, 1, 160), (4096, 1, 255),
                                   (4097, 1, 256), (1025, 4, 257), (32768, 1, 160), (32769, 1, 163), (8209, 8, 170)])
def test_edges(N, R, M):
    H, V = chain(N)
    st = lattices.random_phase_states(N, R, seed=9)
    mu = lq.moments2d(lq.Operator.from_csr(N, *H), lq.Operator.from_csr(N, *V), lq.Operator.from_csr(N, *V), st, M)
    ref = table(N, H, V, st, M)
    assert np.abs(mu - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("power", [-400, 300])
def test_scaled_states_scale_the_table_exactly(power):
    """States scaled by a power of two: the same integers under other exponents."""
    N, M = 600, 170
    H, V = chain(N)
    ops = [lq.Operator.from_csr(N, *a) for a in (H, V, V)]
    st = lattices.random_phase_states(N, 1, seed=3)
    want = lq.moments2d(*ops, st, M)
    got = lq.moments2d(*ops, st * 2.0 ** power, M)
    assert np.array_equal(got, want * 2.0 ** (2 * power))


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_input_is_not_lost(value):
    """A non-finite entry of a state is in every row of both sides, as in FP64 products."""
    N, M = 700, 170
    H, V = chain(N)
    st = lattices.random_phase_states(N, 1, seed=3)
    st[0, 17] = value
    mu = lq.moments2d(lq.Operator.from_csr(N, *H), lq.Operator.from_csr(N, *V), lq.Operator.from_csr(N, *V), st, M)
    assert not np.isfinite(mu.real).any() and not np.isfinite(mu.imag).any()


def test_localised_state(oracle_lib):
    """LinQT's default state: values over hundreds of decades in one row."""
    N, M = 901, 200
    H, V = chain(N)
    st = np.zeros((1, N), np.complex128)
    st[0, N // 2] = 1.0
    mu = lq.moments2d(lq.Operator.from_csr(N, *H), lq.Operator.from_csr(N, *V), lq.Operator.from_csr(N, *V), st, M)
    ref = oracle_lib.moments2d(oracle_lib.Op(*H), oracle_lib.Op(*V), oracle_lib.Op(*V), st, M)
    assert np.abs(mu - ref).max() <= 1e-12 * np.abs(ref).max()
