"""Read-outs of what the device did not write: an output frame of a domain whose
diagnostics found no displacement, after the same page-locked memory held
another context's."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99
SHAPE = (33, 20, 12)


def _desc(mats, precision="fp32", **source):
    med = np.full(SHAPE, len(mats) - 1, np.int32)
    src = [Source(**{**dict(type=1, x=16, y=10, z=6, component="z", frequency=1.5e15), **source})]
    return make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=3, precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_frame_without_a_displacement_is_zero(precision):
    qv, qm, dmm = lattice_2atom(0)
    atoms = Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm)
    with Simulation(_desc([Material(), atoms], precision)) as sim:
        for _ in range(6):                                # every slot's memory takes a displaced cell's state
            sim.step(20)
            fr = sim.frame_wait(sim.frame_begin(diag=True, cell=(16, 10, 6)))
        assert np.abs(fr["diag_cell"]["point"]).max() > 0 and np.abs(fr["diag_cell"]["r"]).max() > 0
    with Simulation(_desc([Material()], precision)) as sim:
        for _ in range(6):
            sim.step(2)
            fr = sim.frame_wait(sim.frame_begin(diag=True, cell=(16, 10, 6)))
            assert fr["diag"]["max_e"] > 0 and fr["diag"]["argmax_r"][0] == -1
            np.testing.assert_array_equal(fr["diag_cell"]["point"], np.zeros(9))
            assert not len(fr["diag_cell"]["r"]) or not np.any(fr["diag_cell"]["r"])
            assert not len(fr["cell"]["r"]) or not np.any(fr["cell"]["r"])
