"""What a failed solve leaves behind, whichever solver the system runs on.

A solve fails by its iteration limit (max_iter = 1: the reference's rule not
met) or by a bounded wait that runs out (wait_polls = 1); nothing faults or
hangs.  The solver of small systems reports its status later than the launch,
so each case is compared with the tiled solver (CAPAC_SOLVER_TILED at
creation), which is waited for inside the force call.
"""
import numpy as np
import pytest

import capacmd_b200 as cm
from conftest import golden_paths

pytestmark = pytest.mark.gpu

PRECS = [cm.PREC_FP64, cm.PREC_MIXED]


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _tight(prec):
    return dict(solver_tol=1e-26) if prec == cm.PREC_FP64 else dict(refine_tol=1e-11)


def _both(monkeypatch, desc, **options):
    """The same system on the small systems' solver and on the tiled one."""
    small = cm.Simulation(desc, **options)
    monkeypatch.setenv("CAPAC_SOLVER_TILED", "1")
    tiled = cm.Simulation(desc, **options)
    monkeypatch.delenv("CAPAC_SOLVER_TILED")
    return small, tiled


@pytest.mark.parametrize("prec", PRECS)
def test_no_gradient_after_a_wait_that_ran_out(prec, monkeypatch):
    d = cm.Desc.from_paths(golden_paths("t_2np"))
    for sim in _both(monkeypatch, d, precision=prec, **_tight(prec)):
        sim.force()
        sim.energy_grad()
        sim.set("wait_polls", [1])
        sim.set("vec_pq", np.zeros(d.n_mat))
        with pytest.raises(cm.CapacError) as e:
            sim.force()
        assert e.value.code == cm.ERR_CUDA
        with pytest.raises(cm.CapacError) as e:
            sim.energy_grad()
        assert e.value.code == cm.ERR_INVALID
        sim.set("wait_polls", [0])
        sim.set("vec_pq", np.zeros(d.n_mat))
        sim.force()
        sim.energy_grad()
