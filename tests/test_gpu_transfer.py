"""State and force arrays handed to memory of each kind.

capac_get, capac_get_xyz and capac_mpi_force fill the caller's arrays: pageable
ones in chunks through a pinned buffer, pinned and device ones directly.  Each
must hold the same bytes.  9,309 atoms: 74 and 223 KB, one and several chunks of
at most 256 KB; 91,122 atoms' 2.2 MB of positions pass the 2 MB buffer.
"""
import numpy as np
import pytest
import torch

import capacmd_b200 as cm
from capacmd_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_available):
    if not gpu_available:
        pytest.fail("no sm_100 GPU: GPU tests must run on a B200")


def _memory(kind, n):
    t = torch.full((n,), -7.0, dtype=torch.float64, device="cuda" if kind == "device" else "cpu")
    return t.pin_memory() if kind == "pinned" else t


KINDS = ["pageable", "pinned", "device"]


@pytest.mark.parametrize("case", ["c2", "c3"])
def test_arrays_in_every_kind_of_memory(case):
    desc = cm.Desc.from_paths(configs.cached(case))
    sim = cm.Simulation(desc, precision=cm.PREC_MIXED)
    n = desc.n_atoms
    for k, key in enumerate("xyz"):  # no force call: the state as created, and forces of known values
        sim.set("f" + key, np.arange(n) + 0.25 * k)
    want = {w: np.stack([sim.get(w.decode() + a) for a in "xyz"], 1) for w in (b"r", b"v", b"f")}
    assert want[b"f"][7].tolist() == [7.0, 7.25, 7.5]
    assert np.abs(want[b"v"]).max() > 0.0
    for kind in KINDS:
        t = _memory(kind, n)
        assert cm.lib().capac_get(sim._p, b"vy", t.data_ptr()) == n
        assert np.array_equal(t.cpu().numpy(), want[b"v"][:, 1])
        for what, v in want.items():
            t = _memory(kind, 3 * n)
            assert cm.lib().capac_get_xyz(sim._p, what, t.data_ptr()) == 0
            assert np.array_equal(t.cpu().numpy().reshape(n, 3), v)
    t = _memory("pageable", 3 * n)
    assert cm.lib().capac_get_xyz(sim._p, b"q", t.data_ptr()) == cm.ERR_INVALID
    assert cm.lib().capac_get_xyz(sim._p, b"r", None) == cm.ERR_INVALID
    assert float(t.min()) == float(t.max()) == -7.0


@pytest.mark.parametrize("kind", KINDS)
def test_drop_in_call_into_every_kind_of_memory(kind):
    desc = cm.Desc.from_paths(configs.cached("c2"))
    sim = cm.Simulation(desc, solver_tol=1e-26)
    xyz = [sim.get(k) for k in ("rx", "ry", "rz")]
    ref = sim.mpi_force(*xyz, vec_pq=np.zeros(desc.n_mat))
    out = {k: _memory(kind, desc.n_atoms) for k in ("fx", "fy", "fz")}
    out.update(potential=_memory(kind, 15), virial=_memory(kind, 9), vec_pq=_memory(kind, desc.n_mat),
               vec_ext=_memory(kind, desc.n_mat), diag_relay=_memory(kind, desc.n_mat),
               inv_sqrt_dens=_memory(kind, desc.n_metal))
    out["vec_pq"].zero_()
    torch.cuda.synchronize()
    rc = cm.lib().capac_mpi_force(sim._p, *[a.ctypes.data for a in xyz], *[t.data_ptr() for t in out.values()])
    assert rc == 0
    for name, t in out.items():
        if name in ref:
            assert np.array_equal(t.cpu().numpy(), ref[name]), name
    assert float(out["inv_sqrt_dens"].min()) > 0.0
