"""Host to device uploads of a context: many small ones and one of several
staging buffers (4 MB pieces), into buffers that are not cleared first.  A
domain whose material ids take more than two buffers steps like the same domain
created in other company, cell for cell, and its ids come back as given."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _desc(shape, seed):
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    med = rng.integers(0, 4, size=shape).astype(np.int32)
    mats = [Material(), Material(eps_re=(2.0, 0, 0, 0, 2.0, 0, 0, 0, 2.0)),
            Material(eps_re=(-300, 0, 0, 0, -300, 0, 0, 0, -300), eps_im=(150, 0, 0, 0, 150, 0, 0, 0, 150), use_ade=1),
            Material(eps_re=(9.0, 0, 0, 0, 2.0, 0, 0, 0, 2.0), anglez=0.6)]
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=nz // 2, component="z", frequency=1.5e15)]
    return make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=6, precision="fp32", source_frequency=3e13)


def test_contexts_made_after_others_hold_their_own_data():
    shape = (224, 210, 205)                                   # 9.6 MB of ids, 38 MB of slots
    with Simulation(_desc(shape, 1)) as sim:
        sim.step(30)
        want = [sim.read_volume(c) for c in ("Ez", "Dx", "Hy")]
    assert all(np.abs(w).max() > 0 for w in want)
    with Simulation(_desc(shape, 2)) as sim:                  # leaves other contents in the device's pool and the staging
        sim.step(30)
        assert not np.array_equal(sim.read_volume("Ez"), want[0])
    for small in ((33, 20, 9), (64, 64, 64)):
        Simulation(_desc(small, 3)).close()
    with Simulation(_desc(shape, 1)) as sim:
        sim.step(30)
        for c, w in zip(("Ez", "Dx", "Hy"), want):
            np.testing.assert_array_equal(sim.read_volume(c), w)
