"""FP64 solves when the device has little memory left: the residue planes of the contraction are an
option, never what a solve fails for, only the call that runs short of memory is the worse for it, and the
same call gives the same blocks and bits whatever planes an earlier one has left in the session.  A
torch buffer takes the rest of the device."""
import contextlib

import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices, serve

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, R, M = 16384, 8, 512  # 2.15 GB of Chebyshev blocks at width 8, planes of 1.14 GB a chunk and 4.6 GB in all
NUMP = 1024
BW = 2 * 1.05 * 8.6


@pytest.fixture(scope="module")
def solve():
    n, H, V = lattices.honeycomb(128, 64, t=-2.7, W=1.0, seed=21)
    assert n == N
    Hg, Vg = lq.Operator.from_csr(n, *H), lq.Operator.from_csr(n, *V)
    Hg.rescale_to_chebyshev(BW, 0.0)
    st = torch.from_numpy(lattices.random_phase_states(n, R, seed=4).view(np.float64)).cuda()
    mu = torch.zeros(2 * M * M, dtype=torch.float64, device="cuda")
    out = torch.zeros(3 * NUMP, dtype=torch.float64, device="cuda")

    def run(session, sigma=False, precision=lq.PREC_FP64):
        o = lq.make_opts(precision=precision)
        if sigma:
            lq.kubo_bastin_dev(Hg, Vg, Vg, st, R, M, NUMP, BW, 0.0, mu, out, opts=o, session=session)
        else:
            lq.moments2d_dev(Hg, Vg, Vg, st, R, M, mu, opts=o, session=session)
        session.synchronize()
        return np.concatenate([mu.cpu().numpy(), out.cpu().numpy()] if sigma else [mu.cpu().numpy()])

    torch.cuda.synchronize()
    run.operators = Hg, Vg
    return run


@contextlib.contextmanager
def only(free_bytes):
    """About this much of the device free meanwhile."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    if free < free_bytes:
        pytest.skip("not enough free memory on the device")
    pad = torch.empty(free - free_bytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del pad
        torch.cuda.synchronize()
        torch.cuda.empty_cache()


@pytest.fixture
def session():
    s = lq.Session(0)
    yield s
    s.close()


@pytest.fixture(scope="module")
def wanted(solve):
    """Of a session that is never short of memory: moments; moments and conductivity; mixed moments."""
    s = lq.Session(0)
    out = solve(s), solve(s, sigma=True), solve(s, precision=lq.PREC_MIXED)
    s.close()
    return out


def test_a_call_repeats_its_blocks_and_bits(solve, wanted, session):
    """Room for the blocks at full width, not for the planes besides."""
    with only(int(2.8e9)):
        got = [solve(session) for _ in range(3)]
    assert np.abs(got[0] - wanted[0]).max() <= 1e-12 * np.abs(wanted[0]).max()
    assert np.array_equal(got[1], got[0]) and np.array_equal(got[2], got[0])
    # memory is back: the kernels and the bits of a session that never was short
    assert np.array_equal(solve(session), wanted[0])


def test_planes_left_behind_do_not_narrow_the_next_solve(solve, wanted, session):
    """A session that holds planes from a solve with room for them, and then the device fills up."""
    assert np.array_equal(solve(session), wanted[0])
    with only(int(0.2e9)):
        assert np.array_equal(solve(session), wanted[0])
        assert np.array_equal(solve(session, precision=lq.PREC_MIXED), wanted[2])


@pytest.mark.parametrize("sigma", [False, True])
def test_one_chunk_of_planes_at_a_time_gives_the_same_bits(solve, wanted, session, sigma):
    """Room for one of the four chunks' planes, and then for all."""
    with only(int(6e9)):
        assert np.array_equal(solve(session, sigma), wanted[sigma])
    assert np.array_equal(solve(session, sigma), wanted[sigma])


@pytest.mark.parametrize("sigma", [False, True])
def test_no_size_of_the_rest_fails(solve, wanted, sigma):
    """The planes may take the rest of the memory, or nearly, but not what the solve needs besides."""
    n, ref = 2 * M * M, wanted[sigma]
    for extra in range(0, 160, 4):
        session = lq.Session(0)
        with only(int(2.74e9) + (extra << 20)):
            got = solve(session, sigma)
        session.close()
        assert np.abs(got[:n] - ref[:n]).max() <= 1e-12 * np.abs(ref[:n]).max(), extra
        if sigma:
            s, r = got[n + NUMP:n + 2 * NUMP], ref[n + NUMP:n + 2 * NUMP]
            assert np.abs(s - r).max() <= 1e-10 * np.abs(r).max(), extra


def test_a_served_request_does_not_change_kernels_for_its_neighbours(solve):
    """A request whose planes do not fit when it runs goes back to run alone, as for any other buffer."""
    Hg, Vg = solve.operators
    srv = serve.Server(0, 16 << 30, 2)
    try:
        with only(int(3.3e9)):
            t = srv.submit(serve.REQ_KUBO_BASTIN, Hg, Vg, None, M, lq.PREC_FP64, R=R, seed=4)
            srv.wait_all()
            assert srv.poll(t)[0] == 2
            assert srv.retries()[1] == 1
    finally:
        srv.close()


def test_a_solve_that_just_fits_is_not_refused_the_second_time(solve):
    """One vector a block: what the arithmetic leaves after the first call is less than before it."""
    n, H, V = lattices.honeycomb(256, 256, t=-2.7, W=1.0, seed=21)
    Hg, Vg = lq.Operator.from_csr(n, *H), lq.Operator.from_csr(n, *V)
    Hg.rescale_to_chebyshev(BW, 0.0)
    st = torch.from_numpy(lattices.random_phase_states(n, 1, seed=4).view(np.float64)).cuda()
    mu = torch.zeros(2 * M * M, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    blocks = 16 * n * (2 * M + 4) + 16 * 66 * M * M  # what a solve counts
    session = lq.Session(0)
    with only(int(blocks / 0.9) + (48 << 20)):
        got = []
        for _ in range(4):
            lq.moments2d_dev(Hg, Vg, Vg, st, 1, M, mu, session=session)
            session.synchronize()
            got.append(mu.cpu().numpy().copy())
    session.close()
    assert all(np.array_equal(g, got[0]) for g in got)
