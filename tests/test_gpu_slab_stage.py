"""Row slabs of a domain whose stage kernel has another block shape than the
slabs' own size would give (the FP32 form's line of 1,216 blocks of 32 x 8
cells): bit for bit the undivided run, because the shape goes by the whole
domain."""
import numpy as np
import pytest
from test_gpu_slabs import _split, _undivided

from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP32, PREC_FP64

pytestmark = pytest.mark.gpu


# blocks of 32 x 8 cells, whole and each of two slabs: 16 x 80 = 1,280, 16 x 41
@pytest.mark.parametrize("nx,ny,settling", [(512, 640, False), (512, 637, True)])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_FP32])
def test_slabs_of_a_domain_past_the_line(nx, ny, settling, prec):
    p, B, _ = W.pyroclastic(nx=nx, ny=ny, dx=10.0, settling=settling, precision=prec, t_end=1e9)
    q = W.developed_current_state(p, B, radius=2000.0)
    q_ref, t_ref, st_ref = _undivided(p, B, q, 12)
    q_s, t_s, st_s = _split(p, B, q, 12, 2)
    assert t_s == t_ref
    np.testing.assert_array_equal(q_s, q_ref)
    assert sum(s.solve_cells for s in st_s) == st_ref.solve_cells
