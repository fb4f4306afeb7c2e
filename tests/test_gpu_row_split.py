"""The FP64 flux kernel's three row splits (1, 2 or 4 rows of a tile per block
by the number of tiles against the device's SMs), each with minmod (divided
differences per face) and another limiter (per side), 1 to 3 classes, and a
last block that the last row cuts; check_solve by 1, 2, 4 and 8 tiles per
block with a ragged last block, with and without a ring inlet: bit for bit the
oracle's state."""
import numpy as np
import pytest

import oracle
from imex_sflow2d_dev_gb300 import lib as L
from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP64

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _tiles(nx, ny):
    return ((nx + 31) // 32) * ((ny + 7) // 8)


def _rows(tiles, sms):   # flux64_rows
    return 4 if 2 * tiles >= 2 * sms else 2 if 4 * tiles >= 2 * sms else 1


def _group(tiles, sms):   # mask_group
    g = 1
    while g < 8 and tiles > 8 * sms * g:
        g *= 2
    return g


def _compare(p, B, q, steps):
    o = oracle.Oracle(p, B)
    o.set_q(W.to_aos(q))
    o.run(max_steps=steps)
    with L.Solver(p, B) as s:
        s.upload_q(W.to_aos(q))
        st = s.advance(max_steps=steps)
        np.testing.assert_array_equal(s.download_q(), o.q())
    assert st.steps == steps and st.t == o.t


@pytest.mark.parametrize("rows,ns,cut", [(1, 3, 5), (2, 1, 3), (2, 2, 5), (2, 3, 1), (4, 2, 7), (4, 3, 3)])
@pytest.mark.parametrize("limiter", [1, 3])
def test_flux_row_split(rows, ns, cut, limiter):
    sms = _sms()
    tiles_y = {1: sms // 3, 2: 3 * sms // 4, 4: 5 * sms // 4}[rows] // 5
    nx, ny = 5 * 32 - 29, 8 * tiles_y - cut   # cut % rows rows of the last block are outside
    assert _rows(_tiles(nx, ny), sms) == rows
    p, B, q = W.dam_break(nx=nx, ny=ny, precision=PREC_FP64, t_end=1e9, n_solid=ns)
    y = np.arange(ny)[None, :, None]
    q *= 1.0 + 0.3 * np.sin(0.21 * y)   # slopes along y too
    for i in range(8):
        p.limiter[i] = limiter
    _compare(p, B, q, 6)


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("ring", [False, True])
def test_check_solve_groups(group, ring):
    sms = _sms()
    nx = 13 * 32 - 17
    tiles_y = 8 * sms * group // 13 if group == 1 else (4 * sms * group // 13 + 3) | 1   # an odd number of tiles
    ny = 8 * tiles_y - 5
    tiles = _tiles(nx, ny)
    assert _group(tiles, sms) == group and (group == 1 or tiles % group)
    if ring:
        p, _, _ = W.pyroclastic(nx=8, ny=8, dx=10.0, settling=False, t_end=1e9)
        p.comp_cells_x, p.comp_cells_y = nx, ny
        p.x_source, p.y_source = 0.3 * nx * 10.0, 0.6 * ny * 10.0
        B, q = np.zeros((ny, nx)), np.zeros((p.n_vars, ny, nx))
    else:
        p, B, _ = W.dam_break(nx=nx, ny=ny, precision=PREC_FP64, t_end=1e9)
        y, x = np.mgrid[0:ny, 0:nx]
        h = np.where((abs(x - 0.4 * nx) < 60) & (abs(y - 0.7 * ny) < 90), 3.0, 0.0)
        h[0, :5] = h[-1, -3:] = 1.0   # in the first and in the last group
        q = W.rest_state_q(p, h, 300.0, [0.0])
    _compare(p, B, q, 12 if ring else 6)
