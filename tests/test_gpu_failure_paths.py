"""The bounded waits of the launches that the other failure test does not
reach, without a GPU fault: a wait on a barrier that nothing arrives on gives
up, the launch finishes (its loads in flight and the launches beside it
awaited), the status comes back, and the device and a new context work on.
The H sweep beside the interior launch, and a group of the ion pass that leaves
its first tile behind while the other groups finish later ones."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, PhpError, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_data

pytestmark = pytest.mark.gpu

PHP_ERR_TIMEOUT = -5
DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _stalls_and_recovers(desc, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with monkeypatch.context() as m:
        m.setenv("PHP_TEST_STALL_WAIT", "1")
        stalled = Simulation(desc)
    stalled.step(4)
    with pytest.raises(PhpError) as e:
        stalled.sync()
    assert e.value.code == PHP_ERR_TIMEOUT
    assert stalled.read_volume("Ez").shape == (desc.nx, desc.ny, desc.nz)   # still answers
    stalled.close()
    a, b = Simulation(desc), Simulation(desc)
    a.step(9)
    b.step(4)
    b.step(5)
    np.testing.assert_array_equal(a.read_volume("Ez"), b.read_volume("Ez"))
    a.sync()
    assert np.abs(a.read_volume("Ez")).max() > 0
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_h_sweep_beside_the_interior_launch(precision, monkeypatch):
    med = np.zeros((97, 65, 40), np.int32)
    src = [Source(type=1, x=50, y=30, z=20, component="z", frequency=1.5e15)]
    desc = make_desc(med, [Material()], src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=5, precision=precision)
    _stalls_and_recovers(desc, monkeypatch, PHP_FUSED="2")


# tiles per block: one (a group without a second tile), and more than the ring holds
@pytest.mark.parametrize("cells", [100, 130 * 60 * 18])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_group_of_the_ion_pass(precision, cells, monkeypatch):
    natom, (nx, ny, nz) = 16, (130, 60, 20)
    rng = np.random.default_rng(natom)
    z = rng.uniform(-0.5, 0.5, size=(natom, 3, 3)) + rng.choice([-3.0, 3.0], size=natom)[:, None, None] * np.eye(3)
    z -= z.mean(axis=0)
    qv, qm, dmm = lattice_data(z, rng.uniform(10.0, 90.0, natom), list(rng.uniform(300.0, 1000.0, 3 * natom)), natom, 12.0 * natom)
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=natom, qezv=qv, qezm=qm, dmm=dmm)]
    med = np.zeros((nz, ny, nx), np.int32)
    med.reshape(-1)[nx * ny:][:cells] = 1
    med = np.ascontiguousarray(med.transpose(2, 1, 0))
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=3, component="z", frequency=4.0e13)]
    desc = make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=0, precision=precision, source_frequency=4.0e13)
    _stalls_and_recovers(desc, monkeypatch)
