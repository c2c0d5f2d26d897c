"""Branches of the integrator kernels against the oracle (plain C).

The Nose-Hoover chain with thermostat velocities on both sides of the bound up
to which its exponentials are Taylor sums, and RATTLE's three-atom iteration
with one, two and three constraints in other orders and orientations.  FP64 on
both sides, a few steps: trajectories agree to rounding, held to the 1e-9 of
the other coupled traces.
"""
import pytest

import capacmd_b200 as cm
from oracle.oracle import Oracle
from conftest import rel_err, variant

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _compare(d, steps, names):
    s, o = cm.Simulation(d), Oracle(d)
    s.md_init()
    assert o.force() == 0
    o.md_init()
    s.md_steps(steps)
    assert o.md_steps(steps) == 0
    for k in names:
        assert rel_err(s.get(k), o.get(k)) < 1e-9, k


@pytest.mark.parametrize("vq0", [0.0, 20.0, 230.0, 400.0])
def test_nose_hoover_chain(vq0, tmp_path):
    # dt 1 fs: the largest argument is 6.6e-5 vQ, 1/64 at 237 per ps; at 230
    # the chain starts below the bound
    paths = variant("t_water", tmp_path)
    text = open(paths["gro"]).read().splitlines()
    assert "vQ" in text[0]
    text[0] = f"step  0  vQ  {vq0:.6f}  vP  0.000000"
    with open(paths["gro"], "w") as f:
        f.write("\n".join(text) + "\n")
    _compare(cm.Desc.from_paths(paths), 3, ("vQ", "rx", "vx", "vz", "thermo"))


ALL = "SOL_CSTRS           3\n0 1   0.100000\n0 2   0.100000\n1 2   0.163298\n"


@pytest.mark.parametrize("cstrs", ["0 1   0.100000", "2 0   0.100000\n0 1   0.100000",
                                   "2 1   0.163298\n0 2   0.100000\n1 0   0.100000"], ids=["one", "two", "three"])
def test_rattle_three_atom_molecules(cstrs, tmp_path):
    def edit(text):
        return text.replace(ALL, f"SOL_CSTRS           {len(cstrs.splitlines())}\n{cstrs}\n")
    _compare(cm.Desc.from_paths(variant("t_water", tmp_path, par=edit)), 3, ("rx", "ry", "vx", "vz", "virial"))
