"""Sizes on both sides of the step kernels' dispatch lines: check_solve by
groups of tiles, the FP32 stage's block heights, the FP64 list of active
cells, the timestep pass without fluxes."""
import numpy as np
import pytest

import oracle
from imex_sflow2d_dev_gb300 import lib as L
from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP32, PREC_FP64

pytestmark = pytest.mark.gpu

# 32 x 8 tiles: 1,209 (one per block, 4-row stage blocks on 152 SMs: up to
# 1,216) and 1,254 (groups, 8-row blocks), with ragged edges
SIZES = [(13 * 32 - 5, 93 * 8 - 3), (11 * 32 - 31, 114 * 8 - 7)]


def _case(nx, ny, precision, n_rk=2):
    """A dry domain with a liquid block off its centre: most tiles dry,
    a moving edge, tiles that become active."""
    p, B, _ = W.dam_break(nx=nx, ny=ny, precision=precision, n_rk=n_rk, t_end=1e9)
    y, x = np.mgrid[0:ny, 0:nx]
    h = np.where((abs(x - 0.4 * nx) < 60) & (abs(y - 0.7 * ny) < 90), 3.0, 0.0)
    h[0, :5] = 1.0   # and a corner of the domain
    return p, B, W.rest_state_q(p, h, 300.0, [0.0])


def _run(p, B, q, steps, tile_h=0):
    with L.Solver(p, B) as s:
        if tile_h:
            s.set_tile_shape(tile_h)
        s.upload_q(W.to_aos(q))
        s.advance(max_steps=steps)
        return s.download_q(), s.counters()


@pytest.mark.parametrize("nx,ny", SIZES)
def test_fp64_bits(nx, ny):
    p, B, q = _case(nx, ny, PREC_FP64)
    o = oracle.Oracle(p, B)
    o.set_q(W.to_aos(q))
    o.run(max_steps=6)
    np.testing.assert_array_equal(_run(p, B, q, 6)[0], o.q())


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("n_rk", [2, 3])
def test_fp32_against_fp64_and_tile_heights(nx, ny, n_rk):
    ref, cr = _run(*_case(nx, ny, PREC_FP64, n_rk), 6)
    for th in (8, 16, 4):
        got, c = _run(*_case(nx, ny, PREC_FP32, n_rk), 6, th)
        assert c["steps"] == cr["steps"] and c["cell_updates"] == cr["cell_updates"]
        g, r = got.reshape(-1, 5), ref.reshape(-1, 5)
        for i in range(5):   # the FP32 form's bar against FP64
            assert np.abs(g[:, i] - r[:, i]).sum() <= 1e-4 * np.abs(r[:, i]).sum() + 1e-12, (th, i)
