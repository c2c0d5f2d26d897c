"""The atom-list pair kernel (k_pair.cu, k_pair) over its routes, FP64.

Pairs with funct 1, the shifted-force van der Waals and the damped Coulomb form
with alpha rc < 5 take terms of their own (dsf_terms); all others the general
ones.  Both are compared with the oracle at the same induced vector, on a
system with all pair forms, for alpha rc on both sides of the limit.

Tolerance: a term of either side carries a few units of 2^-53, at most 5 in
erfc; the terms exceed the largest net force by less than a factor of 100
(oxygen pairs inside a hydrogen bond), and some hundred are summed: 100 x (10 +
sqrt(300)) 2^-53 = 3e-13, taken as 1e-12 of the largest force; as much of the
sum of the energy terms.
"""
import numpy as np
import pytest

import capacmd_b200 as cm
from oracle.oracle import Oracle
from conftest import rel_err, variant
from test_gpu_pair_half import OPTIONS, _replace

pytestmark = pytest.mark.gpu

ALPHAS = {f"alpha_{a}": dict(mds=_replace("coulomb_alpha     2.0", f"coulomb_alpha     {a}"))
          for a in ("4.16", "4.17")}  # alpha rc = 4.992 and 5.004


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


@pytest.mark.parametrize("name", [*OPTIONS, *ALPHAS])
def test_routes_match_the_oracle(name, tmp_path):
    d = cm.Desc.from_paths(variant("t_2np", tmp_path, **{**OPTIONS, **ALPHAS}[name]))
    s, o = cm.Simulation(d, solver_tol=1e-24), Oracle(d)
    s.force()
    o.force()  # its lists and matrix
    if name != "no_cpim":
        o.set("vec_pq", s.get("vec_pq"))
    o.force_given_pq()
    assert rel_err(s.forces(), o.forces()) < 1e-12
    p, q = s.get("potential"), o.get("potential")
    for k in (7, 8):
        assert abs(p[k] - q[k]) <= 1e-12 * np.abs(q[1:]).sum()
    assert rel_err(s.get("virial"), o.get("virial")) < 1e-12


@pytest.mark.parametrize("precision", [cm.PREC_FP64, cm.PREC_MIXED])
@pytest.mark.parametrize("shift", [64.0, 2.0 ** 20])
def test_far_from_the_origin(shift, precision, tmp_path):
    """Coordinates that FP32 does not resolve: the candidates are still those of
    FP64.  Positions are multiples of 2^-30, so the shifted differences are the
    same bits and only the order of the sums may differ."""
    d = cm.Desc.from_paths(variant("t_2np", tmp_path, **OPTIONS["no_cpim"]))
    out = []
    for by in (0.0, shift):
        s = cm.Simulation(d, precision=precision, pair_list=1)
        r = np.round(s.positions() * 2.0 ** 30) / 2.0 ** 30 + by
        for a, k in enumerate(("rx", "ry", "rz")):
            s.set(k, r[:, a])
        s.force()
        out.append(s.forces())
    assert rel_err(out[1], out[0]) < (1e-12 if precision == cm.PREC_FP64 else 1e-6)
