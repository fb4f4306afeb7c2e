"""Settling in a liquid carrier: its velocities are solved once per run and
its hindrance once per cell.  FP64: bit for bit the oracle, which solves them
per class, cell and step.  FP32, a batch and a general tableau against the
single FP64 run."""
import numpy as np
import pytest

import oracle
from imex_sflow2d_dev_gb300 import lib as L
from imex_sflow2d_dev_gb300 import workloads as W
from imex_sflow2d_dev_gb300.params import PREC_FP32, PREC_FP64

pytestmark = pytest.mark.gpu


def _debris(ns, precision, n_rk=2, collective=0):
    p, B, _ = W.dam_break(nx=45, ny=21, dx=5.0, n_solid=ns, precision=precision, n_rk=n_rk, t_end=1e9)
    p.settling_flag, p.collective_settling_flag = 1, collective
    p.A_drag, p.B_drag = 0.01, 1.0
    h = np.where(np.arange(45)[None, :] < 20, 2.0, 0.2) * np.ones((21, 1))
    return p, B, W.rest_state_q(p, h, 300.0, [0.2, 0.05, 0.01][:ns])


def _run(p, B, q, steps):
    with L.Solver(p, B) as s:
        s.upload_q(W.to_aos(q))
        s.advance(max_steps=steps)
        return s.download_q()


@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("collective", [0, 1])
@pytest.mark.parametrize("n_rk", [2, 3])
def test_liquid_settling_bits(ns, collective, n_rk):
    p, B, q = _debris(ns, PREC_FP64, n_rk, collective)
    o = oracle.Oracle(p, B)
    o.set_q(W.to_aos(q))
    o.run(max_steps=5)
    np.testing.assert_array_equal(_run(p, B, q, 5), o.q())


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32])
def test_liquid_settling_batch_and_fp32(precision):
    runs = [_debris(ns, precision) for ns in (1, 2, 3)]
    b = L.Batch(precision, max_runs=4, max_cells=1 << 16)
    ids = [b.submit(p, B, W.to_aos(q), max_steps=5) for p, B, q in runs]
    assert b.advance(8) == 3
    got = [b.collect(i) for i in ids]
    b.close()
    for ns, g in zip((1, 2, 3), got):
        ref = _run(*_debris(ns, PREC_FP64), 5)
        if precision == PREC_FP64:
            np.testing.assert_array_equal(g, ref)
            continue
        g, r = g.reshape(-1, 4 + ns), ref.reshape(-1, 4 + ns)
        for i in range(4 + ns):   # the FP32 form's bar against FP64
            assert np.abs(g[:, i] - r[:, i]).sum() <= 1e-4 * np.abs(r[:, i]).sum() + 1e-12, i
