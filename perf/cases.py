"""The work users of this package have it do, as cases to measure.

Four uses, each through the package's public Python entry points:

* ``md``: resident MD, ten steps (one reference ``save_step``) and the frame and
  status values a driver writes after them;
* ``force``: the drop-in force call on a configuration held in host arrays,
  the induced vector solved from zero (a single point, or one frame of a
  trajectory file);
* ``fit``: one frame of a force-matching fit through the autograd wrapper, the
  loss forward and its parameter and position gradients backward;
* ``grad``: a force call on the resident state and the total energy gradient.

Inputs are what the package's own workloads are made of (Mackay gold
icosahedra, rigid 3-site water, a uniform field, 1.2 nm cut-off), written in
the input formats and parsed by the package.  FP64 cases solve the induced
vector tight (rTr < 1e-24 bTb): under the reference's 1e-4 stopping rule the
converged iterate is not a continuous function of rounding, so two correct
programs differ by more than FP64 results can be compared to.  Results of the
mixed-precision path are FP32 pair sums and are handed back as float32.

``exact`` restates the energy, the induced-charge system, RATTLE and the
Nose-Hoover chain in plain FP64 torch; forces and gradients come from autograd.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import capacmd_b200 as cm
from capacmd_b200 import configs, fit

SPACING = 0.3107  # nm between water lattice sites: 33.3 molecules per nm^3
RC, ALPHA, DT, TEMP = 1.2, 2.0, 0.001, 300.0
STEPS = 10
TIGHT = 1e-24


# ------------------------------------------------------------------ the cases

def _case(name, use, shells, waters, *, mixed, field=0.0, ensemble="nvt", gap=0.0, cpim=1):
    return {"name": name, "use": use, "shells": shells, "gap": gap, "waters": waters, "mixed": mixed, "field": field,
            "ensemble": ensemble, "cpim": cpim}


def listed():
    return [
        # a bare particle, the smallest system one runs for long: 147 atoms, no
        # solve (no field), all launch latency
        _case("md_au147_vacuum_fp64", "md", 3, 0, mixed=False, ensemble="nve"),
        # a small solvated particle in a field, as the correctness runs use
        _case("md_au55_water_mixed", "md", 2, 150, mixed=True, field=0.2),
        # the 9k-atom production size, in both precisions
        _case("md_9k_fp64", "md", 4, 3000, mixed=False),
        _case("md_9k_mixed", "md", 4, 3000, mixed=True),
        # two particles in a field, 91k atoms: the mixed path's ordinary size
        _case("md_91k_field_mixed", "md", 5, 30000, mixed=True, field=0.5, gap=1.5),
        # the largest workload of the repository: 452k atoms, 8,229 unknowns
        _case("md_452k_mixed", "md", 8, 150000, mixed=True),
        # solvent alone, FP64: equilibration and energy-drift floors
        _case("md_water_24k_fp64", "md", 0, 8000, mixed=False, ensemble="nve", cpim=0),
        # drop-in force calls: a fit frame's size in FP64, and 91k atoms mixed
        _case("force_3k_fp64", "force", 3, 1000, mixed=False, field=0.5),
        _case("force_91k_mixed", "force", 5, 30000, mixed=True, field=0.5, gap=1.5),
        # a large bare particle polarised by a field, one single point
        _case("force_au1415_field_mixed", "force", 7, 0, mixed=True, field=0.5),
        # force matching on a frame of the fitting workload (3.1k atoms)
        _case("fit_3k_mixed", "fit", 3, 1000, mixed=True),
        # the energy gradient in FP64 at 9k atoms
        _case("grad_9k_fp64", "grad", 4, 3000, mixed=False),
    ]


def draw(rng):
    """One more case: any use, particle, amount of water and precision of the
    listed ranges (FP64 up to 20,000 waters, gradients up to 3,000)."""
    use = rng.choice(["md", "md", "md", "force", "force", "fit", "grad"])
    mixed = use == "fit" or rng.random() < 0.6
    most = 3000 if use in ("fit", "grad") else 150000 if mixed else 20000
    if use == "fit":
        most = 1500
    bare = use in ("md", "force") and rng.random() < 0.2
    waters = 0 if bare else int(round(math.exp(rng.uniform(math.log(120), math.log(most)))))
    top = (7 if mixed else 5) if bare else max(2, min(8, int((waters / 60.0) ** (1.0 / 3.0) * 1.6)))
    shells = rng.randint(2, min(top, 4) if use in ("fit", "grad") else top)
    pair = shells <= 5 and waters >= 40 * shells ** 3 and use in ("md", "force") and rng.random() < 0.3
    cpim = 1
    if use == "md" and waters > 0 and rng.random() < 0.15:
        shells, pair, cpim = 0, False, 0
    field = 0.0 if cpim == 0 else 0.5 if bare else rng.choice([0.0, 0.2, 0.5])
    case = _case("", use, shells, waters, mixed=mixed, field=field, gap=1.5 if pair else 0.0, cpim=cpim,
                 ensemble=rng.choice(["nvt", "nve"]))
    del case["name"]
    return case


# ----------------------------------------------------------------- the inputs

def _system(case, seed):
    """Positions, velocities, masses and charges of a case, from the seed."""
    rng = np.random.default_rng(seed)
    np_pos = configs.icosahedron(case["shells"]) if case["shells"] else np.zeros((0, 3))
    radius = float(np.sqrt((np_pos ** 2).sum(1).max())) if len(np_pos) else 0.0
    shift = np.array([0.0, 0.0, 0.5 * case["gap"] + radius if case["gap"] else 0.0])
    centres = [-shift, shift] if case["gap"] else [0.0 * shift] if case["shells"] else []
    if case["waters"]:
        n = math.ceil(case["waters"] ** (1.0 / 3.0))
        while True:
            box = round(max(n * SPACING, 1.7), 3)
            g = (np.arange(n) + 0.5) * (box / n) - 0.5 * box
            sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
            free = np.ones(len(sites), bool)
            for c in centres:
                free &= ((sites - c) ** 2).sum(1) > (radius + 0.36) ** 2
            room = 2.0 * (radius + shift[2]) + 0.6
            if int(free.sum()) >= case["waters"] and box > room:
                break
            n += 1
        keep = np.sort(rng.choice(np.flatnonzero(free), size=case["waters"], replace=False))
        q = rng.normal(size=(case["waters"], 4))
        q /= np.linalg.norm(q, axis=1, keepdims=True)
        w, x, y, z = q.T
        rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)
        half = math.radians(configs.HOH_DEG) / 2.0
        ref = configs.OH * np.array([[0.0, 0.0, 0.0], [math.sin(half), 0.0, math.cos(half)],
                                     [-math.sin(half), 0.0, math.cos(half)]])
        local = np.einsum("nij,kj->nki", rot, ref)
        water = sites[keep][:, None, :] + local
    else:
        box, water, local = 6.0, np.zeros((0, 3, 3)), np.zeros((0, 3, 3))
    # thermal displacements take the metal off its symmetric sites
    metal = [np_pos + c + rng.normal(scale=0.005, size=np_pos.shape) for c in centres]
    sizes = [len(m) for m in metal]
    M = sum(sizes)
    pos = np.concatenate(metal + [water.reshape(-1, 3)]) + 0.5 * box
    mass = np.concatenate([np.full(M, configs.M_AU), np.tile([configs.M_O, configs.M_H, configs.M_H], len(water))])
    vel = np.zeros_like(pos)
    vel[:M] = rng.normal(size=(M, 3)) * math.sqrt(configs.K_BOLTZ * TEMP / configs.M_AU)
    if len(water):
        # rigid molecules: a centre-of-mass velocity and an angular velocity
        mw = np.array([configs.M_O, configs.M_H, configs.M_H])
        com = (local * mw[None, :, None]).sum(1, keepdims=True) / mw.sum()
        arm = local - com
        vc = rng.normal(size=(len(water), 1, 3)) * math.sqrt(configs.K_BOLTZ * TEMP / mw.sum())
        inertia = np.einsum("k,nka,nkb->nab", mw, arm, arm)
        inertia = np.trace(inertia, axis1=1, axis2=2)[:, None, None] * np.eye(3) - inertia
        ev, axes = np.linalg.eigh(inertia)
        omega = np.einsum("nab,nb->na", axes, rng.normal(size=(len(water), 3)) * np.sqrt(configs.K_BOLTZ * TEMP / ev))
        vel[M:] = (vc + np.cross(omega[:, None, :], arm)).reshape(-1, 3)
    first = np.cumsum([0] + sizes)
    return {"pos": np.round(pos, 12), "vel": np.round(vel, 12), "mass": mass, "box": box, "M": M,
            "ranges": [(int(first[k]), int(first[k + 1]) - 1) for k in range(len(sizes))], "waters": len(water)}


def _gro(s):
    M, rows = s["M"], np.concatenate([s["pos"], s["vel"]], 1)
    heads = ["%5dAU      Au%5d" % ((i + 1) % 100000, (i + 1) % 100000) for i in range(M)]
    names = ("   OW", "  HW1", "  HW2")
    heads += ["%5dSOL  %s%5d" % ((M + k // 3 + 1) % 100000, names[k % 3], (M + k + 1) % 100000)
              for k in range(3 * s["waters"])]
    line = "%s %.12f %.12f %.12f %.12f %.12f %.12f"
    body = "\n".join([line % (h, *r) for h, r in zip(heads, rows.tolist())])
    return "step  0  vQ  0.000000  vP  0.000000\n%5d\n%s\n%s\n" % (len(rows), body, "%10.5f" % s["box"] * 3)


def _desc(case, s):
    w = configs.Workload("case", [], s["waters"], s["box"], seed=0, ensemble=case["ensemble"], dt=DT,
                         efield_vnm=(0.0, 0.0, case["field"]), temperature=TEMP, save_step=STEPS,
                         use_cpff=case["cpim"])
    folder = tempfile.mkdtemp(prefix="capac_case_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
    try:
        paths = {k: os.path.join(folder, k) for k in ("gro", "par", "mds")}
        for k, text in (("gro", _gro(s)), ("par", configs.param_text(s["M"], s["waters"], s["ranges"], case["cpim"])),
                        ("mds", configs.mdset_text(w))):
            with open(paths[k], "w") as f:
                f.write(text)
        return cm.Desc.from_paths(paths)
    finally:
        shutil.rmtree(folder, ignore_errors=True)


def _target(s, seed):
    """Force-matching targets of the size of thermal forces, and parameters a few percent off."""
    rng = np.random.default_rng([seed, 1])
    return rng.normal(scale=800.0, size=s["pos"].shape), 1.0 + 0.03 * rng.normal(size=9)


def prepare(case, seed):
    s = _system(case, seed)
    desc = _desc(case, s)
    sim = cm.Simulation(desc, precision=cm.PREC_MIXED if case["mixed"] else cm.PREC_FP64,
                        solver_tol=0.0 if case["mixed"] else TIGHT)
    state = {"case": case, "sim": sim, "cpim": case["shells"] > 0 and case["cpim"]}
    if case["use"] == "md":
        sim.md_init()
    elif case["use"] == "force":
        state["xyz"] = [np.ascontiguousarray(s["pos"][:, a]) for a in range(3)]
        state["pq"] = np.zeros(desc.n_mat)
    elif case["use"] == "fit":
        target, factor = _target(s, seed)
        params = fit.current_params(sim) * torch.from_numpy(factor)
        state["params"] = params.requires_grad_(True)
        state["pos"] = torch.from_numpy(s["pos"].copy()).requires_grad_(True)
        state["target"] = torch.from_numpy(target)
    else:
        state["pq"] = np.zeros(desc.n_mat)
    return state


# ------------------------------------------------------------------- one pass

def _kind(state, out):
    """FP32 pair sums come back as float32, FP64 results as they are."""
    if not state["case"]["mixed"]:
        return out
    return {k: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32) for k, v in out.items()}


def run(state):
    sim, use = state["sim"], state["case"]["use"]
    if use == "md":
        sim.md_steps(STEPS)
        # what the driver writes at a save step: the frame, the energies, the temperature
        out = {"pos": sim.positions(), "vel": np.stack([sim.get(k) for k in ("vx", "vy", "vz")], 1),
               "force": sim.forces(), "potential": sim.get("potential"), "thermo": sim.get("thermo")}
        if state["cpim"]:
            out["vec_pq"] = sim.get("vec_pq")
    elif use == "force":
        out = sim.mpi_force(*state["xyz"], vec_pq=state["pq"] if len(state["pq"]) else None)
    elif use == "fit":
        params, pos = state["params"], state["pos"]
        params.grad = pos.grad = None
        loss = fit.force_match_loss(sim, params, state["target"], pos)
        loss.backward()
        out = {"loss": loss.detach(), "params": params.grad, "pos": pos.grad}
    else:
        sim.set("vec_pq", state["pq"])
        sim.force()
        params, pos = sim.energy_grad()
        out = {"force": sim.forces(), "potential": sim.get("potential"),
               "params": np.array([params[k] for k in cm.PARAMS]), "pos": pos}
    return _kind(state, out)


def work(case):
    """Pairs inside the cut-off at about 30 operations each, and the bytes of
    the atoms' state and of the symmetric induced-charge matrix, read once per
    product of the solve (about 30 products in FP32 per solve, 150 in FP64)."""
    n_np = 0 if not case["shells"] else 2 if case["gap"] else 1
    M = n_np * (1 + sum(10 * k * k + 2 for k in range(1, case["shells"] + 1)))
    N = M + 3 * case["waters"]
    pairs = 0.5 * 3 * case["waters"] * min(3 * case["waters"], 100.0 * 4.19 * RC ** 3) + 0.5 * M * min(M, 430)
    solve = M > 0 and case["cpim"] and (case["waters"] > 0 or case["field"] > 0)
    word = 4 if case["mixed"] else 8
    products = (30 if case["mixed"] else 150) if solve else 0
    matrix = 5.0 * word * M * M if M else 0.0
    times = {"md": STEPS, "force": 1, "fit": 3, "grad": 2}[case["use"]]
    return {"bytes": times * (N * 24.0 * 4 + matrix * products + pairs * 0.5),
            "flops": times * (pairs * 30.0 + 10.0 * M * M * products + 200.0 * M * M)}


# ------------------------------------------------- the same in 64 bits, plainly

FQQ, BOHR, KB = 138.935457696552, 18.8972612456506, configs.K_BOLTZ
ISP = 0.564189583547756
CONV_E, CONV_V = 2.01552955019358e-05, 3.80879884583368e-04
LJ_OO = (2.48970844e-03, 2.43509761e-06)
ERF_AU = {1: (0.002522219544, 3.624859037184e-06, 2.25), 2: (0.001028707002, 1.45541995368e-06, 2.25)}
W_ERFC = math.erfc(ALPHA * RC) / RC
W_A2 = 2.0 * ALPHA * ISP
W_CONST = math.erfc(ALPHA * RC) / RC ** 2 + W_A2 * math.exp(-(ALPHA * RC) ** 2) / RC


class _Exact:
    """The force field on FP64 tensors; metal atoms first, then O H H triples."""

    def __init__(self, case, s, dev):
        self.case, self.box, self.M, self.N = case, s["box"], s["M"], len(s["pos"])
        self.ranges, self.dev = s["ranges"], dev
        t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
        self.pos, self.vel, self.mass = t(s["pos"]), t(s["vel"]), t(s["mass"])
        nw = s["waters"]
        self.q = torch.cat([t(np.zeros(self.M)), t([configs.Q_O, configs.Q_H, configs.Q_H]).repeat(nw)])
        self.mol = torch.cat([torch.arange(self.M, device=dev),
                              self.M + torch.arange(nw, device=dev).repeat_interleave(3)])
        self.oxygen = torch.zeros(self.N, dtype=torch.bool, device=dev)
        self.oxygen[self.M::3] = True
        self.field = case["field"] * configs.EV2KJMOL
        self.par = t([1.2159, 39.5297, 0.0, 0.0, float("%.9f" % (0.012793 * configs.EV2KJMOL)), 34.408, 0.408, 10.0, 8.0])
        self.cpim = self.M > 0 and case["cpim"]

    def image(self, d):
        return d - self.box * torch.round(d.detach() / self.box)

    def pairs(self, pos):
        """Index pairs inside the cut-off, not both metal, not of one molecule, in chunks."""
        M, N, dev = self.M, self.N, self.dev
        nc = int(self.box / RC)

        def close(i, j):
            d = self.image(pos[j] - pos[i])
            ok = ((d * d).sum(-1) < RC * RC) & (self.mol[i] != self.mol[j]) & (torch.maximum(i, j) >= M)
            return i[ok], j[ok]

        if nc < 3 or N < 4000:
            for lo in range(0, N, 1024):
                i, j = torch.meshgrid(torch.arange(lo, min(lo + 1024, N), device=dev), torch.arange(N, device=dev),
                                      indexing="ij")
                up = j > i
                yield close(i[up], j[up])
            return
        c3 = torch.clamp((torch.remainder(pos, self.box) / self.box * nc).long(), 0, nc - 1)
        cell = (c3[:, 0] * nc + c3[:, 1]) * nc + c3[:, 2]
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=nc ** 3)
        start = torch.cumsum(count, 0) - count
        width = int(count.max())
        table = torch.full((nc ** 3, width), -1, dtype=torch.long, device=dev)
        table[cell[order], torch.arange(N, device=dev) - start[cell[order]]] = order
        ids = torch.arange(nc ** 3, device=dev)
        cx, cy, cz = ids // (nc * nc), ids // nc % nc, ids % nc
        around = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) >= (0, 0, 0)]
        step = max(1, 20_000_000 // (width * width))
        for a, b, c in around:
            other = (((cx + a) % nc) * nc + (cy + b) % nc) * nc + (cz + c) % nc
            for lo in range(0, nc ** 3, step):
                i = table[lo:lo + step, :, None].expand(-1, -1, width)
                j = table[other[lo:lo + step]][:, None, :].expand(-1, width, -1)
                ok = (i >= 0) & (j >= 0)
                if (a, b, c) == (0, 0, 0):
                    ok &= i < j
                yield close(i[ok], j[ok])

    def pair_energy(self, i, j, d):
        """(Coulomb, van der Waals) energies of pairs with r_j - r_i = d, and what the forces' potential has beside them.

        The shifted Lennard-Jones force of the reference is (f(r) r - f(rc) rc) / r (force.c:710-816), the
        derivative of f(rc) rc ln r where its energy has f(rc) (r - rc)."""
        r2 = (d * d).sum(-1)
        r = r2.sqrt()
        both = (i >= self.M) & (j >= self.M)
        qq = torch.where(both, self.q[i] * self.q[j], 0.0)
        coul = FQQ * qq * (torch.erfc(ALPHA * r) / r - W_ERFC + W_CONST * (r - RC))
        oo = both & self.oxygen[i] & self.oxygen[j]
        c6, c12 = LJ_OO
        fc = 12.0 * c12 / RC ** 12 - 6.0 * c6 / RC ** 6
        lj = c12 / r2 ** 6 - c6 / r2 ** 3 + (r - RC) * fc / RC - (c12 / RC ** 12 - c6 / RC ** 6)
        vdw = torch.where(oo, lj, 0.0)
        wat = torch.maximum(i, j)
        for ty, (e6, e12, w) in ERF_AU.items():
            sel = ~both & (self.oxygen[wat] if ty == 1 else ~self.oxygen[wat])
            vdw = vdw + torch.where(sel, (e12 / r2 ** 6 - e6 / r2 ** 3) * torch.erf(r / w), 0.0)
        return coul.sum(), vdw.sum(), torch.where(oo, fc * (r.log() - (r - RC) / RC), 0.0).sum()

    # -- metal: differences of every ordered pair; the diagonal shifted off zero and masked
    def metal_d(self, pos):
        m = pos[:self.M]
        return self.image(m[None, :, :] - m[:, None, :])

    def qsc(self, d, par):
        eps, c, a, n, m = par[4:]
        eye = torch.eye(self.M, dtype=torch.bool, device=self.dev)
        r2 = torch.where(eye, 1.0, (d * d).sum(-1))
        ok = ~eye & (r2 < RC * RC)
        ar = a / r2.sqrt()
        rho = torch.where(ok, ar ** m, 0.0).sum(1)
        return 0.5 * eps * torch.where(ok, ar ** n, 0.0).sum() - eps * c * rho.sqrt().sum()

    def widths(self, par):
        k = math.sqrt(2.0 / math.pi)
        rq = k * par[0] + par[2]  # entries 2 and 3 are 0: widths tied to capacitance and polarizability
        rp = (k * par[1] / 3.0) ** (1.0 / 3.0) + par[3]
        return 1.0 / (2.0 * rq * rq).sqrt(), 1.0 / (rp * rp + rq * rq).sqrt(), 1.0 / (2.0 * rp * rp).sqrt()

    def tensors(self, d, par):
        """erf-damped T0, T1/r, and the dipole tensor, atomic units, zero on the diagonal."""
        iqq, ipq, ipp = self.widths(par)
        eye = torch.eye(self.M, dtype=torch.bool, device=self.dev)
        b = d * BOHR
        r2 = torch.where(eye, 1.0, (b * b).sum(-1))
        r = r2.sqrt()
        off = (~eye).double()
        t0 = torch.erf(r * iqq) / r * off
        s = lambda i: torch.erf(r * i) - 2.0 * ISP * i * r * torch.exp(-r2 * i * i)  # noqa: E731
        t1 = s(ipq) / r ** 3 * off
        c1 = s(ipp) / r ** 5 * off
        c2 = 4.0 * ISP * ipp ** 3 / r2 * torch.exp(-r2 * ipp * ipp) * off
        rr = b[..., :, None] * b[..., None, :]
        t2 = c1[..., None, None] * (3.0 * rr - torch.eye(3, dtype=torch.float64, device=self.dev) * r2[..., None, None])
        return b, t0, t1, t2 - c2[..., None, None] * rr

    def matrix(self, d, par):
        M, n = self.M, 4 * self.M + len(self.ranges)
        b, t0, t1, t2 = self.tensors(d, par)
        pp = (-t2).permute(0, 2, 1, 3).reshape(3 * M, 3 * M)
        pp = pp + torch.eye(3 * M, dtype=torch.float64, device=self.dev) / par[1]
        pq = (t1[..., None] * b).permute(0, 2, 1).reshape(3 * M, M)
        qp = (-(t1[..., None] * b)).reshape(M, 3 * M)
        qq = -t0 - torch.eye(M, dtype=torch.float64, device=self.dev) / par[0]
        lam = torch.zeros(4 * M, n - 4 * M, dtype=torch.float64, device=self.dev)
        for k, (lo, hi) in enumerate(self.ranges):
            lam[3 * M + lo:3 * M + hi + 1, k] = 1.0
        top = torch.cat([torch.cat([pp, pq], 1), torch.cat([qp, qq], 1)], 0)
        zero = torch.zeros(n - 4 * M, n - 4 * M, dtype=torch.float64, device=self.dev)
        return torch.cat([torch.cat([top, lam], 1), torch.cat([lam.T, zero], 1)], 0)

    def charge_pairs(self, pos):
        """(metal, water) index pairs inside the cut-off."""
        got = [[], []]
        for lo in range(self.M, self.N, 30000):
            j = torch.arange(lo, min(lo + 30000, self.N), device=self.dev)
            for m0 in range(0, self.M, 512):
                i = torch.arange(m0, min(m0 + 512, self.M), device=self.dev)
                d = self.image(pos[i][:, None, :] - pos[j][None, :, :])
                a, b = torch.nonzero((d * d).sum(-1) < RC * RC, as_tuple=True)
                got[0].append(i[a])
                got[1].append(j[b])
        return (torch.cat(got[0]), torch.cat(got[1])) if got[0] else (torch.zeros(0, dtype=torch.long, device=self.dev),) * 2

    def charge_terms(self, d):
        """Potential and field (per unit charge, MD units) of water charges at the metal atoms, d = r_metal - r_water."""
        r2 = (d * d).sum(-1)
        r = r2.sqrt()
        ec = torch.erfc(ALPHA * r)
        v = ec / r - W_ERFC + W_CONST * (r - RC)
        a0 = (ec / r2 + W_A2 * torch.exp(-ALPHA * ALPHA * r2) / r - W_CONST) / r
        return v, a0[:, None] * d

    def rhs(self, pos, i, j, d):
        M = self.M
        v, e = self.charge_terms(d)
        E = torch.zeros(M, 3, dtype=torch.float64, device=self.dev).index_add(0, i, FQQ * self.q[j][:, None] * e * CONV_E)
        V = torch.zeros(M, dtype=torch.float64, device=self.dev).index_add(0, i, FQQ * self.q[j] * v * CONV_V)
        f = torch.tensor([0.0, 0.0, self.field], dtype=torch.float64, device=self.dev)
        E = E + f * CONV_E
        V = V - (pos[:M] * f).sum(1) * CONV_V
        return torch.cat([E.reshape(-1), V, torch.zeros(len(self.ranges), dtype=torch.float64, device=self.dev)])

    def solve(self, pos, par, ext):
        i, j = ext
        b = self.rhs(pos, i, j, self.image(pos[i] - pos[j]))
        if float((b * b).sum()) < 1e-10:
            return torch.zeros_like(b), b
        return torch.linalg.solve(self.matrix(self.metal_d(pos), par), b), b

    def induced_energies(self, x, par, i, j, d_ext, d_mm):
        """The energy slots 10..14 of an induced vector x."""
        M = self.M
        p, q = x[:3 * M].reshape(M, 3), x[3 * M:4 * M]
        v, e = self.charge_terms(d_ext)
        e10 = (FQQ * self.q[j] * q[i] * v).sum()
        e11 = -(FQQ / BOHR * self.q[j][:, None] * p[i] * e).sum()
        b, t0, t1, t2 = self.tensors(d_mm, par)
        au = FQQ * BOHR
        e12 = 0.5 * au * (q @ t0 @ q) + 0.5 * au * (q * q).sum() / par[0]
        pb = torch.einsum("ia,ija->ij", p, b) * t1
        e13 = au * (pb * q[None, :]).sum()
        e14 = -0.5 * au * torch.einsum("ia,ijab,jb->", p, t2, p) + 0.5 * au * (p * p).sum() / par[1]
        return e10, e11, e12, e13, e14

    def force(self, pos, par=None):
        """Forces, the 15 energy slots, the virial, and the induced vector with its right-hand side."""
        par = self.par if par is None else par
        M, N = self.M, self.N
        F = torch.zeros(N, 3, dtype=torch.float64, device=self.dev)
        pot = torch.zeros(15, dtype=torch.float64, device=self.dev)
        vir = torch.zeros(3, 3, dtype=torch.float64, device=self.dev)
        for i, j in self.pairs(pos):
            if not len(i):
                continue
            d = self.image(pos[j] - pos[i]).requires_grad_(True)
            c, v, w = self.pair_energy(i, j, d)
            g, = torch.autograd.grad(c + v + w, d)
            F.index_add_(0, i, g)
            F.index_add_(0, j, -g)
            pot[7] += c.detach()
            pot[8] += v.detach()
            vir += d.detach().T @ g
        x = b = None
        if M:
            d = self.metal_d(pos).requires_grad_(True)
            e = self.qsc(d, par)
            g, = torch.autograd.grad(e, d)
            F[:M] += g.sum(1) - g.sum(0)
            pot[1] = e.detach()
            vir += torch.einsum("ija,ijb->ab", d.detach(), g)
        if self.cpim:
            i, j = self.charge_pairs(pos)
            x, b = self.solve(pos, par, (i, j))
            de = self.image(pos[i] - pos[j]).requires_grad_(True)
            dm = self.metal_d(pos).requires_grad_(True)
            es = self.induced_energies(x, par, i, j, de, dm)
            ge, = torch.autograd.grad(es[0] + es[1], de, retain_graph=True)
            gm, = torch.autograd.grad(es[2] + es[3] + es[4], dm)
            F.index_add_(0, i, -ge)
            F.index_add_(0, j, ge)
            F[:M] += gm.sum(1) - gm.sum(0)
            F[:M, 2] += self.field * x[3 * M:4 * M]
            vir += de.detach().T @ ge
            # the metal-metal virial is summed with r in Bohr, as the reference does (cpff.c:752-926)
            vir += BOHR * torch.einsum("ija,ijb->ab", dm.detach(), gm)
            pot[10:15] = torch.stack([v.detach() for v in es])
            pot[9] -= self.field * ((x[3 * M:4 * M] * pos[:M, 2]).sum() + x[2:3 * M:3].sum())
        F[:, 2] += self.field * self.q
        pot[9] -= self.field * (self.q * pos[:, 2]).sum()
        return F, pot, vir.reshape(-1), x, b

    def total(self, pos, par, x, pairs, ext):
        """The potential of the forces as one differentiable value (fixed pair lists)."""
        i, j = pairs
        d = self.metal_d(pos)
        e = sum(self.pair_energy(i, j, self.image(pos[j] - pos[i]))) + self.qsc(d, par) - self.field * (self.q * pos[:, 2]).sum()
        if self.cpim:
            M = self.M
            e = e + sum(self.induced_energies(x, par, *ext, self.image(pos[ext[0]] - pos[ext[1]]), d))
            e = e - self.field * ((x[3 * M:4 * M] * pos[:M, 2]).sum() + x[2:3 * M:3].sum())
        return e

    def lists(self, pos):
        chunks = list(self.pairs(pos))
        return (torch.cat([c[0] for c in chunks]), torch.cat([c[1] for c in chunks])), self.charge_pairs(pos)


def _rattle(f, pos, old, vel, second):
    """Both RATTLE stages on every water at once, constraint by constraint."""
    M, box = f.M, f.box
    X, V = pos[M:].reshape(-1, 3, 3).clone(), vel[M:].reshape(-1, 3, 3).clone()
    O = old[M:].reshape(-1, 3, 3) if old is not None else None
    oh = configs.OH
    # lengths as the input file gives them, six decimals
    hh = float("%.6f" % (2.0 * oh * math.sin(math.radians(configs.HOH_DEG) / 2.0)))
    im = [1.0 / configs.M_O, 1.0 / configs.M_H, 1.0 / configs.M_H]

    def wrap(d):
        return d - box * (d > 0.5 * box) + box * (d < -0.5 * box)

    for _ in range(1001):
        moved = False
        for a, b, ln in ((0, 1, oh), (0, 2, oh), (1, 2, hh)):
            p = wrap(X[:, a] - X[:, b])
            if second:
                g = -(p * (V[:, a] - V[:, b])).sum(1) / ((im[a] + im[b]) * ln * ln)
                g = torch.where(g.abs() > 1e-5, g, 0.0)
                dv = p * g[:, None]
            else:
                diff = ln * ln - (p * p).sum(1)
                q = wrap(O[:, a] - O[:, b])
                g = torch.where(diff.abs() > ln * ln * 2e-5, diff / (2.0 * (im[a] + im[b]) * (q * p).sum(1)), 0.0)
                dx = q * g[:, None]
                X[:, a] += im[a] * dx
                X[:, b] -= im[b] * dx
                dv = dx / DT
            V[:, a] += im[a] * dv
            V[:, b] -= im[b] * dv
            moved = moved or bool((g != 0).any())
        if not moved:
            break
    return torch.cat([pos[:M], X.reshape(-1, 3)]), torch.cat([vel[:M], V.reshape(-1, 3)])


def _chain(ek, vq, ndf):
    """The Nose-Hoover chain of ten links over one half step (thermostat.c:117-191); returns the velocity scale."""
    n, kt = 10, KB * TEMP
    Q = ndf * kt * 0.1 * 0.1
    nkt, scale = kt * ndf, 1.0
    aq = [(ek - nkt) / Q] + [(Q * vq[m] ** 2 - kt) / Q for m in range(n - 1)]
    w1, w3 = 0.41449077179437571194, -0.65796308717750284778
    for _ in range(5):
        for w in (w1, w1, w3, w1, w1):
            h2, h4, h8 = w * DT / 10.0, w * DT / 20.0, w * DT / 40.0
            vq[n - 1] += aq[n - 1] * h4
            for m in range(n - 2, -1, -1):
                e = math.exp(-h8 * vq[m + 1])
                vq[m] = vq[m] * e * e + h4 * aq[m] * e
            scale *= math.exp(-h2 * vq[0])
            aq[0] = (ek * scale * scale - nkt) / Q
            for m in range(n - 1):
                e = math.exp(-h8 * vq[m + 1])
                vq[m] = vq[m] * e * e + h4 * aq[m] * e
                aq[m + 1] = (Q * vq[m] ** 2 - kt) / Q
            vq[n - 1] += aq[n - 1] * h4
    return scale


def _md(f, case):
    pos, vel, m, M = f.pos.clone(), f.vel.clone(), f.mass[:, None], f.M
    rigid = f.N > M
    nvt = case["ensemble"] == "nvt"
    ndf = 3 * f.N - 3 - (f.N - M)
    kinetic = lambda v: float((m * v * v).sum())  # noqa: E731
    no_com = lambda v: v - (m * v).sum(0) / m.sum()  # noqa: E731
    F = f.force(pos)[0]
    vel = no_com(vel)
    ek, vq = kinetic(vel), [0.0] * 10
    for _ in range(STEPS):
        if nvt:
            s = _chain(ek, vq, ndf)
            vel = vel * s
        vel = vel + 0.5 * DT * F / m
        old = pos
        pos = pos + DT * vel
        if rigid:
            pos, vel = _rattle(f, pos, old, vel, False)
        F, pot, _, x, _ = f.force(pos)
        vel = vel + 0.5 * DT * F / m
        if rigid:
            vel = _rattle(f, pos, None, vel, True)[1]
        ek = kinetic(vel)
        if nvt:
            s = _chain(ek, vq, ndf)
            vel = vel * s
        vel = no_com(vel)
        ek = kinetic(vel)
    # the frame is written with molecules whole around their middle atom
    L = f.box
    single = pos[:M]
    single = single - L * (single > L) + L * (single < 0.0)
    W = pos[M:].reshape(-1, 3, 3).clone()
    W[:, 1] += L * (W[:, 1] < 0.0).double() - L * (W[:, 1] > L).double()
    for a in (0, 2):
        d = W[:, a] - W[:, 1]
        W[:, a] += L * (d < -0.5 * L).double() - L * (d > 0.5 * L).double()
    pos = torch.cat([single, W.reshape(-1, 3)])
    pot[0] = pot[1:].sum()
    out = {"pos": pos, "vel": vel, "force": F, "potential": pot, "thermo": np.array([ek, ek / (KB * ndf), TEMP, ndf])}
    if f.cpim:
        out["vec_pq"] = x
    return out


def exact(case, seed):
    s = _system(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = _Exact(case, s, dev)
    if case["use"] == "md":
        if f.N > 200_000:
            return None  # eleven force calls and dense solves: over 20 seconds
        return _md(f, case)
    if case["use"] == "force":
        F, pot, vir, x, b = f.force(f.pos)
        M, one = f.M, torch.ones(f.M, dtype=torch.float64)
        diag = torch.cat([(one / 39.5297).repeat(3), -one / 1.2159, one[:len(f.ranges)]])
        return {"fx": F[:, 0], "fy": F[:, 1], "fz": F[:, 2], "potential": pot, "virial": vir, "vec_pq": x, "vec_ext": b,
                "diag_relay": diag}
    par, pos = f.par.clone(), f.pos.clone()
    if case["use"] == "fit":
        target, factor = _target(s, seed)
        par = par * torch.as_tensor(factor, device=dev)
    par.requires_grad_(True)
    pos.requires_grad_(True)
    pairs, ext = f.lists(pos.detach())
    x = f.solve(pos, par, ext)[0]
    if case["use"] == "grad":
        F, pot, *_ = f.force(f.pos)
        gpos, gpar = torch.autograd.grad(f.total(pos, par, x, pairs, ext), (pos, par))
        return {"force": F, "potential": pot, "params": gpar, "pos": gpos}
    # the forces are -dE/dr at a fixed induced vector; the loss then also
    # depends on the positions through that vector
    at = pos.detach().clone().requires_grad_(True)
    F = -torch.autograd.grad(f.total(at, par, x, pairs, ext), at, create_graph=True)[0]
    loss = ((F - torch.as_tensor(target, device=dev)) ** 2).mean()
    gat, gpar, gx = torch.autograd.grad(loss, (at, par, x), retain_graph=True)
    gpos, = torch.autograd.grad(x, pos, gx)
    gpar[2:4] = 0.0  # the widths follow the capacitance and the polarizability
    return {"loss": loss.detach(), "params": gpar, "pos": gat + gpos}
