"""The bounded waits of the launches that the other failure test does not
reach, without a GPU fault: a wait on a barrier that nothing arrives on gives
up, the launch finishes (its loads in flight and the launches beside it
awaited), the status comes back, and the device and a new context work on.
The H sweep beside the interior launch."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, PhpError, Simulation, Source, make_desc

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
