"""A captured solve is replayed only for calls with the same options: the same pointers with another
operator precision or thread shape are another solve."""
import numpy as np
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_options_are_part_of_the_key():
    N, Hc = lattices.square_lattice(40, t=1.0, W=1.0, seed=11)
    H = lq.Operator.from_csr(N, *Hc)
    H.rescale_to_chebyshev(2 * 1.05 * 4.5, 0.0)
    st = torch.from_numpy(lattices.random_phase_states(N, 2, seed=3).view(np.float64)).cuda()
    mu = torch.zeros(2 * 64, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sess = lq.Session(0)

    def run(**kw):
        lq.moments1d_dev(H, None, st, 2, 64, mu, opts=lq.make_opts(**kw), session=sess)
        sess.synchronize()
        return mu.cpu().numpy().copy()

    kinds = [dict(), dict(operator_precision=lq.OP_C64), dict(thread_shape=1), dict(thread_shape=2)]
    want = [run(**k) for k in kinds]
    assert not np.array_equal(want[0], want[1])
    for k, w in zip(kinds, want):
        for _ in range(4):  # eager, captured, replayed
            assert np.array_equal(run(use_graphs=1, **k), w)
