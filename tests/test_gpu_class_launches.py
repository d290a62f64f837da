"""The E sweep of a mid-size domain with a lattice as one launch per kind of
block (from 400 000 cells), against the same domain with the lattice's blocks
left to the general path, whose E sweep is one launch (PHP_PLAIN_ATOMS=0 at
create).  Runs of several output intervals cross the graphs' length."""
import os

import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom

pytestmark = pytest.mark.gpu


def _run(precision, shape, z_chunk, atoms):
    nx, ny, nz = shape
    qv, qm, dmm = lattice_2atom(0)
    med = np.zeros(shape, np.int32)
    med[:, :, :nz // 3] = 1
    med[nx // 2:nx // 2 + 20, ny // 2:ny // 2 + 9, nz // 3:] = 2
    dl = 10e-9
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm),
            Material(eps_re=(-300, 0, 0, 0, -300, 0, 0, 0, -300), eps_im=(150, 0, 0, 0, 150, 0, 0, 0, 150), use_ade=1)]
    src = [Source(type=1, x=nx // 3, y=ny // 3, z=nz // 3 + 2, component="z", frequency=1.5e15)]
    desc = make_desc(med, mats, src, dx=dl, dy=dl, dz=dl, dt=dl / (299792458.0 * np.sqrt(3.0)) * 0.99, pml_thickness=6,
                     precision=precision, source_frequency=3.0e13, z_chunk=z_chunk)
    old = os.environ.get("PHP_PLAIN_ATOMS")
    os.environ["PHP_PLAIN_ATOMS"] = atoms
    try:
        sim = Simulation(desc)
    finally:
        if old is None:
            os.environ.pop("PHP_PLAIN_ATOMS")
        else:
            os.environ["PHP_PLAIN_ATOMS"] = old
    pid = sim.dft_add("Dz", nz // 3 - 1, [1.5e15])
    sim.probe_set(nx // 3, ny // 3, nz // 3, nz // 3 - 1)
    for n in (1, 70, 66):
        sim.step(n)
    out = [sim.read_volume(c) for c in range(9)] + [sim.probe_read(), sim.dft_read(pid)[0]]
    sim.step(1)
    launches = sim.last_launch_count
    sim.close()
    return out, launches


# just past the size from which the launches are taken, remainders of one cell past a tile of 32 x 16
@pytest.mark.parametrize("shape,z_chunk", [((97, 65, 64), 0), ((65, 81, 77), 5)])
@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_class_launches_match_one_launch(precision, rtol, shape, z_chunk):
    (a, na), (b, nb) = _run(precision, shape, z_chunk, "1"), _run(precision, shape, z_chunk, "0")
    assert na > nb
    for q, (x, y) in enumerate(zip(a, b)):
        scale = np.abs(y).max()
        assert scale > 0
        np.testing.assert_allclose(x, y, rtol=0, atol=rtol * scale, err_msg=f"output {q}")
