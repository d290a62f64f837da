"""The launches of recorded steps overlap (programmatic launches, some of them
beside the one before), against the same launches one behind the other, which
php_profile_enable records: fields, D, monitor rows and running DFT must be the
same, bit for bit, after a few hundred steps of a domain of several waves of
blocks with a CPML on every side, so that the CPML slabs and the pools of the
atom cells change SM from step to step.  The E sweep's class launches in place,
and the interior launch with the two sweeps beside it."""
import os

import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom

pytestmark = pytest.mark.gpu


def _run(precision, fused, chained, steps):
    shape = nx, ny, nz = (194, 138, 130)
    qv, qm, dmm = lattice_2atom(0)
    med = np.zeros(shape, np.int32)
    med[:, :, :nz // 3] = 1
    med[nx // 2:nx // 2 + 20, ny // 2:ny // 2 + 9, nz // 3:] = 2
    med[:, :, 2 * nz // 3:2 * nz // 3 + 12] = 3
    dl = 10e-9
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm),
            Material(eps_re=(-300, 0, 0, 0, -300, 0, 0, 0, -300), eps_im=(150, 0, 0, 0, 150, 0, 0, 0, 150), use_ade=1),
            Material(eps_re=(3.0, 0, 0, 0, 2.5, 0, 0, 0, 2.2), eps_im=(0.1, 0, 0, 0, 0.1, 0, 0, 0, 0.1), anglez=0.5)]
    src = [Source(type=1, x=nx // 3, y=ny // 3, z=nz // 3 + 2, component="z", frequency=1.5e15)]
    desc = make_desc(med, mats, src, dx=dl, dy=dl, dz=dl, dt=dl / (299792458.0 * np.sqrt(3.0)) * 0.99, pml_thickness=9,
                     precision=precision, source_frequency=3.0e13)
    old = os.environ.get("PHP_FUSED")
    os.environ["PHP_FUSED"] = fused
    try:
        sim = Simulation(desc)
    finally:
        if old is None:
            os.environ.pop("PHP_FUSED")
        else:
            os.environ["PHP_FUSED"] = old
    with sim:
        ids = [sim.dft_add(c, z, [3e13, 1.5e15]) for c, z in (("Dz", nz // 3 - 1), ("Ex", 2), ("Ey", nz // 2))]
        sim.probe_set(nx // 3, ny // 3, nz // 3, nz // 3 - 1)
        if not chained:
            sim.profile()
        sim.step(steps)
        sim.sync()
        return ([sim.read_volume(c) for c in range(9)] + [sim.probe_read()] + [sim.dft_read(p)[0] for p in ids]
                + [sim.read_cell_state(nx // 3 + 4, ny // 3, 3)["v"]])


@pytest.mark.parametrize("fused", ["0", "2"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_chained_launches_equal_launches_in_order(precision, fused):
    want = _run(precision, fused, False, 300)
    assert all(np.abs(x).max() > 0 for x in want)
    for _ in range(2):
        for q, (x, y) in enumerate(zip(_run(precision, fused, True, 300), want)):
            np.testing.assert_array_equal(x, y, err_msg=f"output {q}")
