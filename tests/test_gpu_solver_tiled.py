"""The tiled solvers on small systems, and which systems the small systems'
solver takes.

Systems whose FP64 matrix fits the chip are solved by a kernel of their own
(k_solve_dense.cu), the sizes of test_gpu_solver.py among them.  Here the cases
of that file that are about the tiled solvers (k_solve_coop.cu: group order,
tiles in tensor memory, coarse space, L2 policy) and the bounded wait of
test_gpu_errors.py run with CAPAC_SOLVER_TILED set, and every context is asked
which solver it has.
"""
import os

import numpy as np
import pytest

import capacmd_b200 as cm
import test_gpu_dense_solver as small
import test_gpu_errors as errors
import test_gpu_solver as solver
from capacmd_b200 import configs
from conftest import rel_err

pytestmark = pytest.mark.gpu

PRECS = [cm.PREC_FP64, cm.PREC_MIXED]


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


@pytest.fixture
def tiled(monkeypatch):
    """Contexts keep the tiled solvers; at the end, that each one did."""
    made = []

    class Tiled(cm.Simulation):
        def __init__(self, *a, **k):
            super().__init__(*a, **k)
            made.append(self.get("dense_solver")[0])

    monkeypatch.setenv("CAPAC_SOLVER_TILED", "1")
    monkeypatch.setattr(cm, "Simulation", Tiled)
    yield monkeypatch
    assert made and not any(made), made


@pytest.mark.parametrize("case", ["t_au55w", "t_2np", "c1_field"])
@pytest.mark.parametrize("prec", PRECS)
def test_persistent_solver_matches_stepwise(case, prec, tiled):
    solver.test_persistent_solver_matches_stepwise_tight(case, prec)


@pytest.mark.parametrize("case", ["t_au55w", "t_2np", "c1_field", "t_au13"])
def test_grouped_solver(case, tiled):
    solver.test_grouped_solver_matches_ungrouped(case, tiled)


@pytest.mark.parametrize("case", ["t_au55w", "t_2np", "c1_field"])
def test_tmem_tiles(case, tiled):
    solver.test_tmem_tiles_match_streamed(case, tiled)


@pytest.mark.parametrize("precond", [2, 3])
@pytest.mark.parametrize("case", ["t_2np", "c1_field", "c2"])
def test_two_level(case, precond, tiled):
    solver.test_two_level_inner_solves(case, precond)


@pytest.mark.parametrize("case", ["c2", "t_2np"])
def test_coarse_inversion(case, tiled):
    solver.test_coarse_inversion_by_a_cluster(case, tiled)


@pytest.mark.parametrize("prec", PRECS)
def test_tile_l2_policy(prec, tiled):
    solver.test_tile_l2_policy_changes_no_result(prec, tiled)


@pytest.mark.parametrize("prec", PRECS)
def test_wait_timeout(prec, tiled):
    errors.test_persistent_solver_wait_timeout(prec)


def _cluster(atoms, out_dir):
    """The inner atoms of a bare Au561 in a field, off their sites."""
    w = configs.Workload("cut", [5], 0, 9.0, seed=51, ensemble="nve", efield_vnm=(0.1, 0.2, 0.5))
    s = configs.build(w)
    centre = s["pos"].mean(0)
    keep = np.argsort(((s["pos"] - centre) ** 2).sum(1), kind="stable")[:atoms]
    pos = s["pos"][keep] + np.random.default_rng(52).normal(scale=0.004, size=(atoms, 3))
    paths = {k: os.path.join(str(out_dir), k) for k in ("gro", "par", "mds")}
    texts = {"gro": configs.gro_text(pos, s["vel"][keep], atoms, w.box),
             "par": configs.param_text(atoms, 0, [(0, atoms - 1)]), "mds": configs.mdset_text(w)}
    for k, text in texts.items():
        with open(paths[k], "w") as f:
            f.write(text)
    return cm.Desc.from_paths(paths)


# four columns a thread (769 and 1,021 unknowns, on the five-column kernel), and
# the last size of 148 blocks of 12 rows (1,773) with the first beyond it (1,777)
@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("atoms,dense", [(192, 1.0), (255, 1.0), (443, 1.0), (444, 0.0)])
def test_edges_of_the_small_systems_solver(atoms, dense, prec, tmp_path, monkeypatch):
    d = _cluster(atoms, tmp_path)
    tol = dict(solver_tol=1e-26) if prec == cm.PREC_FP64 else dict(refine_tol=1e-11)
    a = cm.Simulation(d, precision=prec, **tol)
    assert a.get("dense_solver")[0] == dense
    monkeypatch.setenv("CAPAC_SOLVER_TILED", "1")
    b = cm.Simulation(d, precision=prec, **tol)
    assert b.get("dense_solver")[0] == 0.0
    for s in (a, b):
        s.force()
    bar = 1e-10 if prec == cm.PREC_FP64 else 1e-8  # as test_gpu_dense_solver.py
    assert rel_err(a.get("vec_pq"), b.get("vec_pq")) < bar
    assert rel_err(a.forces(), b.forces()) < bar


@pytest.mark.parametrize("prec", PRECS)
def test_which_systems_the_comparisons_solve_so(prec, tmp_path):
    """Every system that test_gpu_dense_solver.py compares but its last, which is beyond."""
    got = [cm.Simulation(small._desc(s, tmp_path), precision=prec).get("dense_solver")[0] for s in small.SHELLS]
    assert got == [1.0] * (len(got) - 1) + [0.0]
