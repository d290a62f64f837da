"""The ion pass (ion_pipe) over pools that end inside a tile: FP64 tiles of 64
cells, FP32 tiles of 128, pools of a multiple of 32 slots.  The
padded matrix sizes it is compiled for (3N = 24 -> 32, 30 -> 32, 48, 63 -> 64,
where FP64 takes the plain kernel), fewer tiles than SMs and more than the ring
holds, and cells of a second material with the lattice's DMM and effective
charges of its own, whose coefficients come from global memory.  FP64 against
the update inside the E sweep, FP32 against FP64."""
import os

import numpy as np
import pytest

import harness as H
from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_data

pytestmark = pytest.mark.gpu


def _sim(precision, natom, shape, cells, fused):
    rng = np.random.default_rng(natom)
    z = rng.uniform(-0.5, 0.5, size=(natom, 3, 3)) + rng.choice([-3.0, 3.0], size=natom)[:, None, None] * np.eye(3)
    z -= z.mean(axis=0)
    qv, qm, dmm = lattice_data(z, rng.uniform(10.0, 90.0, natom), list(rng.uniform(300.0, 1000.0, 3 * natom)), natom, 12.0 * natom)
    eps = (4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95)
    mats = [Material(), Material(eps_re=eps, natom=natom, qezv=qv, qezm=qm, dmm=dmm, anglez=0.3),
            Material(eps_re=eps, natom=natom, qezv=0.7 * qv, qezm=0.8 * qm, dmm=dmm)]
    nx, ny, nz = shape
    med = np.zeros((nz, ny, nx), np.int32)
    flat = med.reshape(-1)                    # pool order: k, j, i
    first = nx * ny * 2 + ny // 2 * nx - 16
    flat[first:][:cells] = 1
    flat[first + cells // 2:][:7] = 2
    med = np.ascontiguousarray(med.transpose(2, 1, 0))
    dl = 10e-9
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=3, component="z", frequency=4.0e13)]
    desc = make_desc(med, mats, src, dx=dl, dy=dl, dz=dl, dt=dl / (299792458.0 * np.sqrt(3.0)) * 0.99, pml_thickness=0,
                     precision=precision, source_frequency=4.0e13)
    old = os.environ.get("PHP_IONS")
    if fused:
        os.environ["PHP_IONS"] = "fused"
    try:
        return Simulation(desc), np.argwhere(med > 0), np.argwhere(med == 2)
    finally:
        if old is None:
            os.environ.pop("PHP_IONS", None)
        else:
            os.environ["PHP_IONS"] = old


def _state(args, fused=False):
    sim, cells, other = _sim(*args, fused)
    with sim:
        sim.step(40)
        e = np.stack([sim.read_volume(c) for c in ("Ex", "Ey", "Ez")])
        pick = np.concatenate([cells[::max(1, len(cells) // 40)], cells[-34:], other])
        st = [sim.read_cell_state(*(int(q) for q in c)) for c in pick]
        return e, np.stack([s["r"] for s in st]), np.stack([s["v"] for s in st])


@pytest.mark.parametrize("natom,shape,cells", [(8, (40, 20, 8), 33), (10, (40, 20, 8), 96), (16, (40, 20, 9), 1), (16, (97, 65, 30), 65 * 97 * 24 + 13),
                                               (8, (130, 60, 20), 130 * 60 * 15 + 50), (21, (40, 30, 9), 4033)])
def test_pools_that_end_inside_a_tile(natom, shape, cells):
    e, r, v = _state(("fp64", natom, shape, cells))
    e0, r0, v0 = _state(("fp64", natom, shape, cells), fused=True)
    for x, y in ((e, e0), (r, r0), (v, v0)):
        assert np.abs(y).max() > 0
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()          # as between the two forms elsewhere
    e1, r1, _ = _state(("fp32", natom, shape, cells))
    assert H.rel_l2(e1, e) <= 1e-4 and np.abs(r1 - r).max() <= 1e-3 * np.abs(r).max()
