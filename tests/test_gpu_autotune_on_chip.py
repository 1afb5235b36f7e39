"""The autotuner times what the solve will run: with a thread shape asked for, the kernels that have
shapes; without, the on-chip kernels of small blocks, which have none, once and not once a shape."""
import pytest

import linqt_b200 as lq
from linqt_b200 import lattices

pytestmark = pytest.mark.gpu


def tuned(H, st, **kw):
    lq.moments1d(H, None, st, 200, opts=lq.make_opts(fmt=lq.FORMAT_AUTO, block_width=8, **kw))
    return {k: v for k, v in H.tuned().items() if k.startswith("1d")}


def test_a_forced_shape_is_tuned_by_itself():
    N, Hc = lattices.square_lattice(24, t=1.0, W=1.0, seed=11)
    H = lq.Operator.from_csr(N, *Hc)
    H.rescale_to_chebyshev(2 * 1.05 * 4.5, 0.0)
    st = lattices.random_phase_states(N, 8, seed=3)
    first = tuned(H, st)
    both = tuned(H, st, thread_shape=2)
    assert len(first) == 1 and len(both) == 2
