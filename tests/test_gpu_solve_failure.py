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
from conftest import golden_paths, impossible_constraints, rel_err, variant

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


def _mpi_force(sim, pos, pq):
    """capac_mpi_force on arrays of known contents; returns the status and the outputs."""
    out = {k: np.full(sim.n_atoms, -7.0) for k in ("fx", "fy", "fz")}
    out.update(potential=np.full(15, -7.0), virial=np.full(9, -7.0), vec_pq=pq.copy(), vec_ext=np.full(sim.n_mat, -7.0),
               diag_relay=np.full(sim.n_mat, -7.0), inv_sqrt_dens=np.full(sim.desc.n_metal, -7.0))
    xyz = [np.ascontiguousarray(pos[:, a]) for a in range(3)]
    rc = cm.lib().capac_mpi_force(sim._p, *[a.ctypes.data for a in xyz], *[a.ctypes.data for a in out.values()])
    return rc, out


@pytest.mark.parametrize("how,code", [("max_iter", cm.ERR_NOT_CONVERGED), ("wait_polls", cm.ERR_CUDA)])
def test_drop_in_call_leaves_the_callers_arrays(how, code, monkeypatch):
    d = cm.Desc.from_paths(golden_paths("t_2np"))
    pq = np.random.default_rng(5).normal(scale=1e-3, size=d.n_mat)
    for sim in _both(monkeypatch, d, **{how: 1}, solver_tol=1e-26):
        rc, out = _mpi_force(sim, sim.positions(), pq)
        assert rc == code
        assert np.array_equal(out.pop("vec_pq"), pq)
        for name, v in out.items():
            assert np.all(v == -7.0), name


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


STATE = ("rx", "ry", "rz", "vx", "vy", "vz", "fx", "fy", "fz", "virial", "thermo", "vQ")


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("case", ["t_2np", "t_au55w"])
def test_failed_step_is_the_last_one(case, prec, monkeypatch):
    """md_steps stops in the step whose solve failed: positions, velocities,
    thermostat and step count are that step's, as after a solve that is
    waited for at once."""
    d = cm.Desc.from_paths(golden_paths(case))
    small, tiled = _both(monkeypatch, d, precision=prec, **_tight(prec))
    for sim in (small, tiled):
        sim.md_init()
        sim.md_steps(2)
        sim.set("wait_polls", [1])
        with pytest.raises(cm.CapacError) as e:
            sim.md_steps(4)
        assert e.value.code == cm.ERR_CUDA
        assert sim.stats().md_step == 3
    for name in STATE:
        if name not in ("fx", "fy", "fz", "virial"):  # of a vector that no solve has left defined
            assert rel_err(small.get(name), tiled.get(name)) < 1e-9, name
    # and goes on from there once the limit is gone
    for sim in (small, tiled):
        sim.set("wait_polls", [0])
        sim.md_steps(2)
        assert sim.stats().md_step == 5
        assert np.all(np.isfinite(sim.positions()))


@pytest.mark.parametrize("case", ["t_2np", "t_au55w"])
def test_unconverged_step_is_the_last_one(case, monkeypatch):
    """The same with the reference's iteration limit: two iterations of the
    same recurrence, so the forces agree too."""
    d = cm.Desc.from_paths(golden_paths(case))
    small, tiled = _both(monkeypatch, d, max_iter=1, solver_tol=1e-26)
    rng = np.random.default_rng(9)
    f = {k: rng.normal(scale=100.0, size=d.n_atoms) for k in ("fx", "fy", "fz")}
    for sim in (small, tiled):
        for k, v in f.items():
            sim.set(k, v)
        with pytest.raises(cm.CapacError) as e:
            sim.md_steps(3)
        assert e.value.code == cm.ERR_NOT_CONVERGED
        assert "bicg_stab not converged" in str(e.value)
        assert sim.stats().md_step == 1
    for name in STATE:
        assert rel_err(small.get(name), tiled.get(name)) < 1e-9, name


def test_failed_solve_comes_before_failed_constraints(tmp_path, monkeypatch):
    """A step in which the solve and RATTLE fail reports the solve (the force
    call comes first), and no later call reports it again."""
    d = cm.Desc.from_paths(variant("t_au55w", tmp_path, par=impossible_constraints))
    for sim in _both(monkeypatch, d, solver_tol=1e-26):
        sim.md_init()
        sim.set("wait_polls", [1])
        with pytest.raises(cm.CapacError) as e:
            sim.md_steps(1)
        assert e.value.code == cm.ERR_CUDA
        sim.set("wait_polls", [0])
        sim.set("vec_pq", np.zeros(d.n_mat))
        try:
            sim.force()
        except cm.CapacError as later:  # the constraints' own failure, not read yet
            assert later.code == cm.ERR_RATTLE
            sim.force()
        assert np.all(np.isfinite(sim.forces()))
