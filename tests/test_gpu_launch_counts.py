"""Launches of one step where the E sweep is a launch per kind of block: a
domain large enough for the interior launch whose interior is too small a share
of it, and a many-atom lattice whose ion pass runs apart; the latter's fields
against the same domain with its atom blocks on the general path."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom, lattice_data

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99
EPS = (4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95)


def _desc(shape, lattice, atoms_to, precision, pml=6):
    nx, ny, nz = shape
    qv, qm, dmm, natom = lattice
    med = np.zeros(shape, np.int32)
    med[:, :, :atoms_to] = 1
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=atoms_to + 2, component="z", frequency=1.5e15)]
    return make_desc(med, [Material(), Material(eps_re=EPS, natom=natom, qezv=qv, qezm=qm, dmm=dmm)], src, dx=DL, dy=DL, dz=DL,
                     dt=DT, pml_thickness=pml, precision=precision, source_frequency=3e13)


def test_large_domain_of_a_small_interior():
    with Simulation(_desc((256, 256, 128), (*lattice_2atom(0), 2), 100, "fp32")) as sim:
        sim.profile()
        sim.step(1)
        assert sim.profile_read()["step"]["launches"] == 0      # no interior launch
        sim.profile(False)
        c = sim.block_census()
        kinds = (c["e_general"] > 0) + (c["e_atoms"] > 0) + (c["e_plain"] + c["e_plain_cpml"] + c["e_tensor"] > 0)
        sim.step(3)
        assert kinds == 3 and sim.last_launch_count == 3 * (1 + kinds)


@pytest.mark.parametrize("natom", [8, 16])
@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_class_launches_with_the_ion_pass_apart(precision, rtol, natom, monkeypatch):
    rng = np.random.default_rng(natom)
    z = rng.uniform(-0.5, 0.5, size=(natom, 3, 3)) + rng.choice([-3.0, 3.0], size=natom)[:, None, None] * np.eye(3)
    z -= z.mean(axis=0)
    qv, qm, dmm = lattice_data(z, rng.uniform(10.0, 90.0, natom), list(rng.uniform(300.0, 1000.0, 3 * natom)), natom, 12.0 * natom)
    out = []
    for plain, kinds in (("1", 3), ("0", 1)):
        monkeypatch.setenv("PHP_PLAIN_ATOMS", plain)
        with Simulation(_desc((97, 65, 66), (qv, qm, dmm, natom), 30, precision)) as sim:
            sim.step(70)
            sim.step(7)
            assert sim.last_launch_count == 7 * (1 + kinds + 1)
            out.append([sim.read_volume(q) for q in range(9)]
                       + [np.stack([sim.read_cell_state(48, j, k)[s] for j in (0, 5, 31, 64) for k in (3, 29)]) for s in "rv"])
    for q, (x, y) in enumerate(zip(*out)):
        assert np.abs(y).max() > 0
        np.testing.assert_allclose(x, y, rtol=0, atol=rtol * np.abs(y).max(), err_msg=f"output {q}")
