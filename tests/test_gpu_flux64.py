"""The FP64 flux kernel's row split (1, 2 or 4 rows of a tile per block) and
its ordinary-cell reconstruction: bit for bit the oracle's state on domains
whose edges fall at every position in a tile, with and without a ring inlet,
minmod (divided differences per face) and another limiter (per side)."""
import numpy as np
import pytest

import oracle
from imex_sflow2d_dev_gb300 import lib as L
from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP64

pytestmark = pytest.mark.gpu


def _compare(p, B, q, steps):
    o = oracle.Oracle(p, B)
    o.set_q(W.to_aos(q))
    o.run(max_steps=steps)
    with L.Solver(p, B) as s:
        s.upload_q(W.to_aos(q))
        st = s.advance(max_steps=steps)
        np.testing.assert_array_equal(s.download_q(), o.q())
    assert st.steps == steps and st.t == o.t


# 16 tiles and fewer: 1 row; up to 151: 2 rows; more: 4 rows (152 SMs)
@pytest.mark.parametrize("nx,ny,ns", [(5, 5, 1), (33, 9, 2), (64, 64, 3), (65, 63, 1), (97, 130, 2), (31, 257, 1),
                                      (223, 181, 1)])
@pytest.mark.parametrize("limiter", [1, 3])
def test_dam_break_bits(nx, ny, ns, limiter):
    p, B, q = W.dam_break(nx=nx, ny=ny, precision=PREC_FP64, t_end=1e9, n_solid=ns)
    for i in range(8):
        p.limiter[i] = limiter
    _compare(p, B, q, 6)


@pytest.mark.parametrize("n,dx", [(70, 10.0), (131, 7.3), (200, 10.0)])
def test_current_bits(n, dx):
    p, B, _ = W.pyroclastic(nx=n, ny=n - 3, dx=dx, precision=PREC_FP64, t_end=1e9)
    q = W.developed_current_state(p, B, radius=0.3 * n * dx)
    _compare(p, B, q, 3)
