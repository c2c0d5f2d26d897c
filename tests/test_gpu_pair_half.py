"""The half-list pair kernel's two routes (k_pair.cu, k_pair_half).

Clusters whose pairs all have funct 1 with the shifted-force van der Waals and
the damped Coulomb form take a short path; every other combination of options
(plain cut-offs, a Gaussian beyond the fitted range of the complementary error
function, Buckingham and Morse or erf-damped pairs next to metal) takes the
general one.  Both are compared with the FP64 path, on a system whose clusters
have between one and four members and list lengths that are no multiple of 32,
and with the atom-list kernel where a pair is so close that its FP32 force is
huge or infinite.

Tolerance: a pair term carries a relative error of a few 2^-24 (r^2, 1/r, the
Gaussian's argument up to 6, r^-14 by products: below 32 x 2^-24 = 2e-6 of the
term), and the terms exceed an atom's net force by less than a factor of five
here: 1e-5 of the largest force, the bound of the mixed path.
"""
import numpy as np
import pytest

import capacmd_b200 as cm
from conftest import rel_err, variant

pytestmark = pytest.mark.gpu

MORSE_BUCK = (" 2    1.0e+05    30.0    2.0e-03", " 3    5.0    20.0    0.28")


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _replace(a, b):
    return lambda text: text.replace(a, b)


def _morse_buck(text):
    out = []
    for line in text.split("\n"):
        if line.startswith(" 4  0.0025"):
            line = MORSE_BUCK[0]
        elif line.startswith(" 4  0.0010"):
            line = MORSE_BUCK[1]
        out.append(line)
    return "\n".join(out)


def _all_plain(text):
    return "\n".join(" 1  0.0025  3.6e-06" if line.startswith(" 4  ") else line for line in text.split("\n"))


OPTIONS = {
    "vdw_cut_off": dict(mds=_replace("shifted", "cut_off")),
    "coulomb_cut_off": dict(mds=_replace("wolf_sum", "cut_off")),
    "narrow_gaussian": dict(mds=_replace("coulomb_alpha     2.0", "coulomb_alpha     4.5")),
    "wide_gaussian": dict(mds=_replace("coulomb_alpha     2.0", "coulomb_alpha     0.7")),
    "no_cpim": dict(mds=_replace("use_cpff          1", "use_cpff          0")),
    "morse_buckingham": dict(par=_morse_buck),
    "metal_plain": dict(par=_all_plain),
}


@pytest.mark.parametrize("split", ["0", "1"])
@pytest.mark.parametrize("name", OPTIONS)
def test_routes_match_fp64(name, split, tmp_path, monkeypatch):
    monkeypatch.setenv("CAPAC_PAIR_SPLIT", split)
    d = cm.Desc.from_paths(variant("t_2np", tmp_path, **OPTIONS[name]))
    half = cm.Simulation(d, precision=cm.PREC_MIXED, refine_tol=1e-11)
    f64 = cm.Simulation(d, precision=cm.PREC_FP64, solver_tol=1e-24)
    for s in (half, f64):
        s.force()
    assert half.get("pair_list")[0] == 1.0
    assert rel_err(half.forces(), f64.forces()) < 1e-5
    p, q = half.get("potential"), f64.get("potential")
    scale = np.abs(q[1:]).sum()
    for k in (7, 8):
        assert abs(p[k] - q[k]) <= 1e-5 * scale
    assert rel_err(half.get("virial"), f64.get("virial")) < 1e-5


@pytest.mark.parametrize("gap", [5e-3, 1e-5])
def test_overlapping_atoms(gap, tmp_path):
    """One water's oxygen at `gap` nm from another's: a force of 1e26 and an
    infinite one.  The same atoms as with the atom list have a finite force,
    and the finite ones agree.  The FP32 difference of coordinates near 1 nm is
    off by up to 1.2e-7, 2.4e-5 of the gap, which r^-14 makes 3.4e-4 in each
    kernel: 1e-3 of the largest for the two atoms."""
    d = cm.Desc.from_paths(variant("t_2np", tmp_path, mds=_replace("use_cpff          1", "use_cpff          0")))
    out = []
    for pair_list in (0, 1):
        s = cm.Simulation(d, precision=cm.PREC_MIXED, pair_list=pair_list)
        r = s.positions()
        o = d.n_metal
        r[o + 30:o + 33] += (r[o] - r[o + 30]) + np.array([gap, 0.0, 0.0])
        s.set("rx", r[:, 0]), s.set("ry", r[:, 1]), s.set("rz", r[:, 2])
        s.force()
        out.append(s.forces())
    finite = [np.isfinite(f).all(axis=1) for f in out]
    assert np.array_equal(*finite)
    assert finite[0].sum() == d.n_atoms - (0 if gap > 1e-3 else 2)
    a, b = (f[finite[0]] for f in out)
    big = np.abs(b).max(axis=1) > 1e10
    assert gap < 1e-3 or big.sum() == 2
    assert np.allclose(a[big], b[big], rtol=0.0, atol=1e-3 * np.abs(b).max())
    assert rel_err(a[~big], b[~big]) < 2e-6
