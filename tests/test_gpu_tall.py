"""Narrow tall domains: block rows past grid.y's limit of 65,535 (FP64 blocks
are parts of a tile: the pointwise kernels from 131,070 rows on, the flux
kernel from 262,140; check_solve's block after the last tile in a domain of
65,535 tile rows with a source)."""
import numpy as np
import pytest

import oracle
from imex_sflow2d_dev_gb300 import lib as L
from imex_sflow2d_dev_gb300 import slabs as S
from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP32, PREC_FP64

pytestmark = pytest.mark.gpu


def _channel(nx, ny, n_rk):
    """Liquid in the first and in the last rows and across the middle."""
    p, B, _ = W.dam_break(nx=nx, ny=ny, n_rk=n_rk, t_end=1e9)
    h = np.zeros((ny, nx))
    h[:9] = 1.0
    h[ny // 2:ny // 2 + 3] = 2.0
    h[-13:-2] = 1.5
    return p, B, W.rest_state_q(p, h, 300.0, [0.0])


def _oracle(p, B, q, steps):
    o = oracle.Oracle(p, B)
    o.set_q(W.to_aos(q))
    o.run(max_steps=steps)
    return o.q()


@pytest.mark.parametrize("ny,n_rk", [(131070, 3), (131083, 3), (262155, 2), (262155, 1)])
def test_fused_step_bits(ny, n_rk):
    p, B, q = _channel(5, ny, n_rk)
    with L.Solver(p, B) as s:
        s.upload_q(W.to_aos(q))
        s.advance(max_steps=3)
        np.testing.assert_array_equal(s.download_q(), _oracle(p, B, q, 3))


def test_call_sites_bits():
    p, B, q = _channel(5, 131083, 2)
    t, dt_old, dt_old_old, t_out = p.t_start, p.dt0, p.dt0, p.t_start + p.dt_output
    with L.Solver(p, B) as s:
        s.upload_q(W.to_aos(q))
        for _ in range(2):
            s.check_solve(False)
            dt, t_out = S.clamp_dt(s.timestep(), t, p.t_end, t_out, dt_old, dt_old_old)
            dt_old_old, dt_old = dt_old, dt
            s.imex_rk_solver(t, dt)
            s.update_erosion_deposition_cell(dt)
            t = s.post_step().t
        np.testing.assert_array_equal(s.download_q(), _oracle(p, B, q, 2))


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_FP32])
def test_source_in_the_tallest_domain(prec):
    """65,535 tile rows and a ring inlet at the low end: the rows there are
    those of a short domain."""
    rows = []
    for ny in (64, 65535 * 8):
        p, _, _ = W.pyroclastic(nx=8, ny=8, dx=20.0, precision=prec, n_rk=3, settling=False, t_end=1e9)
        p.comp_cells_y = ny
        with L.Solver(p, np.zeros((ny, 8))) as s:
            s.upload_q(np.zeros(p.n_vars * 8 * ny))
            s.advance(max_steps=8)
            rows.append(s.download_q().reshape(ny, -1)[:32].copy())
    assert rows[0][:, 0].max() > 0.0
    np.testing.assert_array_equal(rows[1], rows[0])
