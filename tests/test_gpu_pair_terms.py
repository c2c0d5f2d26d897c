"""Errors of the pair terms on isolated ion pairs.

4,096 pairs of opposite charges, more than the cut-off from each other, at
separations r between 0.7 and 1.0 nm (alpha r between 1.7 and 2.45, where the
Gaussian carries most of the force).  A Gaussian 2^(c r^2) with c = -alpha^2
log2 e rounded to FP32 has the relative error (alpha r)^2 dc / c of one sign,
and alpha is chosen where that rounding is near its largest (dc / c = 5.0e-8).
The test fits the slope of the force's relative error, against the FP64 path,
over (alpha r)^2.  What else has a slope: the fit of erfc (below 7e-9 on this
range, so below 5e-9 over the 3.1 of (alpha r)^2), the rounded constants of
the two terms (6e-8 of a share that varies by a tenth: 2e-9), and the rounding
of r^2, the Gaussian and the products, zero on average, 4e-7 a pair and so
7e-9 on the slope of 4,096.  In all below 1.5e-8; half the rounded constant's
slope, 2.5e-8, is the bound.

FP64 path: the force of each pair over its separation against decimal
arithmetic on the same r^2.  Its roundings: the Gaussian and erfc 1.1e-16 each
(rms; a quarter of the force is erfc's), the sum, the two products with 1/r and
1/r itself 0.5e-16 each, the constants 1e-16, the product with the component and
the test's division by it 0.5e-16 each: 2.5e-16.  A Gaussian of a rounded r has
2 (alpha r)^2, about nine, times that rounding's 0.6e-16 and more: above 5e-16.
The bound is 4e-16.
"""
import decimal
import os

import numpy as np
import pytest

import capacmd_b200 as cm

pytestmark = pytest.mark.gpu

ALPHA, SIDE, STEP = 2.453125, 16, 2.5

PARAM = """SCALE_LJ_QQ    0.50000000     0.83333333

MOLECULES      2
CAT          4096
ANI          4096

CAT_ATOMS           1
     1.000000    22.990000       0

ANI_ATOMS           1
    -1.000000    35.450000       1

NONBONDED      2         3
 1    0.00000000e+00      0.00000000e+00
 1    0.00000000e+00      0.00000000e+00
 1    0.00000000e+00      0.00000000e+00

""" + "\n".join("\n".join(f"{m}_{s:<14s} 0" for s in ("BONDS", "PAIRS", "ANGLES", "DIHEDRALS", "VSITES", "CSTRS")) + "\n"
                for m in ("CAT", "ANI")) + """
MM_METAL  -1  -1
QSC_METAL  10  8  1.234336909  34.408000  0.408000
CPFF_METAL  39.529700  1.215900   ;  Note: atomic unit

NANOPARTICLES   0
"""


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _ions(out_dir):
    from capacmd_b200 import configs
    rng = np.random.default_rng(41)
    n = SIDE ** 3
    at = (np.stack(np.meshgrid(*[np.arange(SIDE)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * STEP
    axis = rng.normal(size=(n, 3))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    r = rng.uniform(0.7, 1.0, size=(n, 1))
    pos = np.concatenate([at - 0.5 * r * axis, at + 0.5 * r * axis])
    box = SIDE * STEP
    lines = ["step  0  vQ  0.000000  vP  0.000000", f"{len(pos):5d}"]
    for i, p in enumerate(pos):
        lines.append("%5d%-5s%5s%5d %.12f %.12f %.12f 0.0 0.0 0.0"
                     % (i + 1, "CAT" if i < n else "ANI", "Na" if i < n else "Cl", i + 1, *p))
    lines.append(f"{box:10.5f}{box:10.5f}{box:10.5f}")
    w = configs.Workload("ions", [], 0, box, seed=0, ensemble="nve", use_cpff=0)
    texts = {"gro": "\n".join(lines) + "\n", "par": PARAM,
             "mds": configs.mdset_text(w).replace("coulomb_alpha     2.0", f"coulomb_alpha     {ALPHA}")}
    paths = {k: os.path.join(str(out_dir), k) for k in texts}
    for k, text in texts.items():
        with open(paths[k], "w") as f:
            f.write(text)
    d = pos[n:] - pos[:n]
    return cm.Desc.from_paths(paths), n, d


def test_half_list_gaussian_has_no_systematic_error(tmp_path):
    desc, n, d = _ions(tmp_path)
    mixed, f64 = cm.Simulation(desc, precision=cm.PREC_MIXED), cm.Simulation(desc)
    for s in (mixed, f64):
        s.force()
    assert mixed.get("pair_list")[0] == 1.0
    f = [(s.forces()[:n] * d).sum(1) for s in (mixed, f64)]
    assert np.all(f[1] > 0.0)  # each pair attracts, nothing else in reach
    rel = f[0] / f[1] - 1.0
    assert np.abs(rel).max() < 5e-6
    x2 = ALPHA ** 2 * (d * d).sum(1)
    slope = np.polyfit(x2, rel, 1)[0]
    assert abs(slope) < 2.5e-8, slope


def _decimal_force(r2, alpha, rc):
    """Damped shifted Coulomb force over r of unit charges, in 40 digits (alpha r below 3)."""
    D = decimal.Decimal
    with decimal.localcontext() as ctx:
        ctx.prec = 40
        isp = D("0.56418958354775628694807945156077258584405")
        isp_field = D("0.564189583547756")  # the force field's constant, in fifteen digits (typedef.h:44)

        def erfc(x):
            t = s = x
            k = 0
            while abs(t) > D("1e-38"):
                k += 1
                t *= -x * x / k
                s += t / (2 * k + 1)
            return 1 - 2 * isp * s

        def f(v):
            r = v.sqrt()
            return erfc(alpha * r) / v + 2 * alpha * isp_field * (-alpha * alpha * v).exp() / r

        alpha, rc = D(alpha), D(rc)
        shift = f(rc * rc)
        return [(f(D(float(v))) - shift) / D(float(v)).sqrt() for v in r2]


def test_fp64_damped_terms(tmp_path):
    desc, n, _ = _ions(tmp_path)
    s = cm.Simulation(desc)
    x = s.positions()  # as read from the file
    s.force()
    d = x[n:] - x[:n]
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]  # rounded as the kernel rounds it
    at, axis = np.arange(0, n, 4), np.abs(d).argmax(1)[::4]
    got = s.forces()[at, axis] / d[at, axis]
    exact = _decimal_force(r2[at], ALPHA, "1.2")
    fqq = decimal.Decimal("138.935457696552")
    rel = np.array([float(decimal.Decimal(float(g)) / (fqq * e) - 1) for g, e in zip(got, exact)])
    assert np.sqrt((rel * rel).mean()) < 4e-16
