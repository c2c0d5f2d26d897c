"""Several contexts alive in one process.

The solver of small systems has one kernel per range of sizes; what a launch
needs of it (dynamic shared memory) depends on the system.  A context's solves
must not depend on which others were created after it: a larger system, then a
smaller one of the same kernel, then the larger one again (it solves the same
system as before, to the mixed path's bar).
"""
import os

import numpy as np
import pytest

import capacmd_b200 as cm
from capacmd_b200 import configs
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _desc(shells, out_dir):
    w = configs.Workload("ctx", shells, 0, 9.0, seed=31, ensemble="nve", efield_vnm=(0.0, 0.0, 0.5), gap_z=0.9)
    s = configs.build(w)
    pos = s["pos"] + np.random.default_rng(32).normal(scale=0.004, size=s["pos"].shape)
    os.makedirs(str(out_dir), exist_ok=True)
    paths = {k: os.path.join(str(out_dir), k) for k in ("gro", "par", "mds")}
    texts = {"gro": configs.gro_text(pos, s["vel"], s["n_metal"], w.box),
             "par": configs.param_text(s["n_metal"], 0, s["np_ranges"]), "mds": configs.mdset_text(w)}
    for k, text in texts.items():
        with open(paths[k], "w") as f:
            f.write(text)
    return cm.Desc.from_paths(paths)


# (larger, smaller): 221 and 53 unknowns in one column, 1,237 and 1,178 in five, 1,458 and 1,458 - 4 * 42 in seven
@pytest.mark.parametrize("large,small", [((2,), (1,)), ((4,), (3, 3)), ((4, 2), (4, 1))],
                         ids=["one column", "five columns", "seven columns"])
def test_smaller_system_after_a_larger_one(large, small, tmp_path):
    da, db = _desc(large, tmp_path / "a"), _desc(small, tmp_path / "b")
    assert da.n_mat > db.n_mat
    a = cm.Simulation(da, precision=cm.PREC_MIXED, refine_tol=1e-11)
    a.force()
    x = a.get("vec_pq")
    b = cm.Simulation(db, precision=cm.PREC_MIXED, refine_tol=1e-11)
    b.force()
    a.set("vec_pq", np.zeros(da.n_mat))
    a.force()
    assert rel_err(a.get("vec_pq"), x) < 1e-8
    b.set("vec_pq", np.zeros(db.n_mat))
    b.force()
    assert b.stats().solver_rel_residual <= 1e-11
