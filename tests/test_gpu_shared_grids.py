"""Server slots size their persistent grids from shares of the device: a request that gets all the share
it asks for runs on the grid that it needs, to the last CTA, and so gives the bits of the same solve
without a server."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices, serve

pytestmark = pytest.mark.gpu

# CTAs of 256 rows whose share of the 2 x 148 CTAs of rows of 7 entries, multiplied back in FP64, falls
# short of them
SHORT = [c for c in range(86, 260) if int(296 * (c / 296)) < c]


@pytest.mark.parametrize("ctas", SHORT)
def test_a_granted_share_is_the_whole_grid(ctas):
    N = 256 * ctas
    i = np.arange(N)
    H = lq.Operator.from_csr(N, *lattices.upper_csr(
        N, np.concatenate([i] * 4), np.concatenate([(i + d) % N for d in range(4)]),
        np.concatenate([0.2 * (lattices.uniform(5, N) - 0.5)] + [np.full(N, 0.13)] * 3)))
    st = lattices.random_phase_states(N, 1, seed=3)
    want = lq.moments1d(H, None, st, 64)
    srv = serve.Server(0, 0, 2)
    t = srv.submit(serve.REQ_DOS, H, None, st, 64)
    srv.wait_all()
    assert srv.poll(t)[0] == 2
    got = srv.result(t).copy()
    srv.close()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("share", [0.02, 0.3, 0.7])
@pytest.mark.parametrize("R", [1, 2])
def test_a_share_too_small_for_the_registers(share, R):
    """Blocks that the register recursion takes on the whole device, of a session whose share covers a part
    of its grid: the other kernel's moments (the same terms in another order, below 1e-13)."""
    N = 256 * 230 // R
    i = np.arange(N)
    H = lq.Operator.from_csr(N, *lattices.upper_csr(
        N, np.concatenate([i] * 4), np.concatenate([(i + d) % N for d in range(4)]),
        np.concatenate([0.2 * (lattices.uniform(5, N) - 0.5)] + [np.full(N, 0.13)] * 3)))
    st = lattices.random_phase_states(N, R, seed=3)
    want = lq.moments1d(H, None, st, 64)
    s = lq.Session(0)
    s.set_sm_share(share)
    got = lq.moments1d(H, None, st, 64, session=s)
    s.close()
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
