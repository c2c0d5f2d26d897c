"""The solver of small CPIM systems against the tiled one.

Both run the reference's BiCGSTAB (bicg_stab.c:253-573) on the same matrix and
differ in the order of the sums only, so at rTr < 1e-26 bTb the induced
vectors agree to the 1e-10 of the other tight solver comparisons.  Every block
has 12 rows; the kernel's variants are its columns per thread (256 unknowns
each): 13 atoms in one particle (53 unknowns, 5 blocks) and 55 (221) have one
column, two of 55 (442) two, 147 (589) three, two of 147 (1,178) and 309 (1,237)
five, 309 + 55 (1,458) seven, and 309 + 147 (1,826) is beyond, tiled both times.
Four columns and the last size that fits: test_gpu_solver_tiled.py.
"""
import os

import numpy as np
import pytest

import capacmd_b200 as cm
from capacmd_b200 import configs
from conftest import rel_err

pytestmark = pytest.mark.gpu

SHELLS = [(1,), (2,), (2, 2), (3,), (3, 3), (4,), (4, 2), (4, 3)]


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _desc(shells, out_dir):
    """Bare particles in a field, off their symmetric sites."""
    w = configs.Workload("dense", shells, 0, 9.0, seed=21, ensemble="nve", efield_vnm=(0.1, 0.2, 0.5), gap_z=0.9)
    s = configs.build(w)
    pos = s["pos"] + np.random.default_rng(22).normal(scale=0.004, size=s["pos"].shape)
    paths = {k: os.path.join(str(out_dir), k) for k in ("gro", "par", "mds")}
    texts = {"gro": configs.gro_text(pos, s["vel"], s["n_metal"], w.box),
             "par": configs.param_text(s["n_metal"], 0, s["np_ranges"]), "mds": configs.mdset_text(w)}
    for k, text in texts.items():
        with open(paths[k], "w") as f:
            f.write(text)
    return cm.Desc.from_paths(paths)


@pytest.mark.parametrize("shells", SHELLS, ids=lambda s: "+".join(map(str, s)))
def test_dense_solver_matches_tiled(shells, tmp_path, monkeypatch):
    d = _desc(shells, tmp_path)
    dense = cm.Simulation(d, solver_tol=1e-26)
    monkeypatch.setenv("CAPAC_SOLVER_TILED", "1")
    tiled = cm.Simulation(d, solver_tol=1e-26)
    monkeypatch.delenv("CAPAC_SOLVER_TILED")
    for s in (dense, tiled):
        s.force()
    assert dense.stats().solver_iterations > 0
    assert rel_err(dense.get("vec_pq"), tiled.get("vec_pq")) < 1e-10
    assert rel_err(dense.forces(), tiled.forces()) < 1e-10
    # warm starts, several launches in a row
    for s in (dense, tiled):
        s.md_init()
        s.md_steps(3)
    assert rel_err(dense.get("vec_pq"), tiled.get("vec_pq")) < 1e-9
    # the same call twice is the same to the bit
    x = []
    for _ in range(2):
        dense.set("vec_pq", np.zeros(d.n_mat))
        dense.force()
        x.append(dense.get("vec_pq"))
    assert np.array_equal(x[0], x[1])


@pytest.mark.parametrize("shells", SHELLS, ids=lambda s: "+".join(map(str, s)))
def test_dense_mixed_solve_matches_tiled(shells, tmp_path, monkeypatch):
    """The mixed path: both refine to 1e-11 and agree with a tight FP64 solve
    within the mixed path's bar (the bars of test_grouped_solver_matches_ungrouped),
    through warm-started steps and a preconditioner refresh."""
    d = _desc(shells, tmp_path)
    dense = cm.Simulation(d, precision=cm.PREC_MIXED, refine_tol=1e-11)
    monkeypatch.setenv("CAPAC_SOLVER_TILED", "1")
    tiled = cm.Simulation(d, precision=cm.PREC_MIXED, refine_tol=1e-11)
    f64 = cm.Simulation(d, solver_tol=1e-26)
    monkeypatch.delenv("CAPAC_SOLVER_TILED")
    for s in (dense, tiled, f64):
        s.force()
    assert rel_err(dense.get("vec_pq"), f64.get("vec_pq")) < 1e-8
    assert rel_err(dense.forces(), tiled.forces()) < 1e-8
    assert dense.stats().solver_rel_residual <= 1e-11
    dense.md_init()
    tiled.md_init()
    for _ in range(12):
        dense.md_steps(1)
        tiled.md_steps(1)
    assert rel_err(dense.get("vec_pq"), tiled.get("vec_pq")) < 1e-7
    assert rel_err(dense.get("rx"), tiled.get("rx")) < 1e-9
