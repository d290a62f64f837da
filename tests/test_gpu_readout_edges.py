"""Read-outs of what the device did not write or cannot represent: an output
frame of a domain whose diagnostics found no displacement, after the same
page-locked memory held another context's, and D of a cell whose E overflowed in
one component."""
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


@pytest.mark.parametrize("mat", [Material(), Material(eps_re=(2.0, 0, 0, 0, 3.0, 0, 0, 0, 2.5))])
def test_d_of_the_components_that_stayed_finite(mat):
    """A source so strong that Ez of its cell overflows single precision in the
    first step: Dx and Dy of the cell do not depend on Ez."""
    with Simulation(_desc([mat], amplitude=1e60, type=0, t0=0.0, tau=1e-15)) as sim:
        sim.step(1)
        p = sim.read_point(16, 10, 6)
        assert np.isinf(p[2]) and p[0] == 0 and p[1] == 0
        assert p[3] == 0 and p[4] == 0 and np.isinf(p[5])
        assert np.array_equal(sim.read_volume("Dx"), np.zeros(SHAPE))
