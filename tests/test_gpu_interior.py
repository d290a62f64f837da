"""The interior of a large domain in a launch of its own (interior_sweep_tma:
H and E of plain and tensor blocks in one march, E and H double buffered)
with the rest in the two sweeps, against the two sweeps alone: the fields, the
CPML and lattice state, the monitor rows and the running DFT must be the same,
bit for bit.  PHP_FUSED=2 at create takes the interior launch at any size,
PHP_FUSED=0 never."""
import os

import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom

pytestmark = pytest.mark.gpu


def _desc(precision, shape, pml, z_chunk=0):
    nx, ny, nz = shape
    qv, qm, dmm = lattice_2atom(0)
    med = np.zeros(shape, np.int32)
    med[:, :, :nz // 4] = 1                                        # two-atom slab
    med[:, :, nz // 4:nz // 2] = 2                                 # rotated lossy tensor layer
    med[nx // 2:nx // 2 + 9, ny // 2:ny // 2 + 9, nz // 2:] = 3    # metal (ADE) through the vacuum
    med[nx // 3, ny // 3, nz // 2 + 3] = 4                         # one cell of another tensor material
    med[nx // 4, ny // 4, nz // 2 + 2] = 5                         # a material whose E is no invertible map of D
    dl = 10e-9
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm),
            Material(eps_re=(6.0, 0, 0, 0, 3.5, 0, 0, 0, 2.8), eps_im=(0.4, 0, 0, 0, 0.2, 0, 0, 0, 0.1), anglez=0.52),
            Material(eps_re=(-300, 0, 0, 0, -300, 0, 0, 0, -300), eps_im=(150, 0, 0, 0, 150, 0, 0, 0, 150), use_ade=1),
            Material(eps_re=(4.0, 0.7, 0, 0.7, 3.0, 0, 0, 0, 2.5), anglex=0.3),
            Material(eps_re=(1.0, 0, 0, 0, 1.0, 0, 0, 0, 1e6))]
    src = [Source(type=1, x=nx // 2, y=ny // 2 - 3, z=nz // 2 + 4, component="z", frequency=1.5e15),
           Source(type=1, x=nx // 3, y=ny // 3, z=2, component="x", frequency=1.0e15)]
    return make_desc(med, mats, src, dx=dl, dy=dl, dz=dl, dt=dl / (299792458.0 * np.sqrt(3.0)) * 0.99, pml_thickness=pml,
                     precision=precision, source_frequency=3.0e13, z_chunk=z_chunk)


def _run(desc, mode, probe, steps):
    old = os.environ.get("PHP_FUSED")
    os.environ["PHP_FUSED"] = mode
    try:
        sim = Simulation(desc)
    finally:
        if old is None:
            os.environ.pop("PHP_FUSED")
        else:
            os.environ["PHP_FUSED"] = old
    ids = [sim.dft_add(c, z, [3e13, 1.5e15]) for c, z in (("Ez", desc.nz // 2 + 3), ("Dx", desc.nz // 2 - 2), ("Dz", 1))]
    sim.probe_set(*probe)
    out = {}
    for n in steps:
        sim.step(n)
    out["volumes"] = [sim.read_volume(c) for c in range(9)]
    out["rows"] = sim.probe_read()
    out["dft"] = [sim.dft_read(p)[0] for p in ids]
    nx, ny, nz = desc.nx, desc.ny, desc.nz
    for cell in ((nx // 2 + 1, ny // 2 + 1, nz // 2 + 1), (5, 6, 1), (nx // 3, ny // 3, nz // 2 + 3), (nx // 4, ny // 4, nz // 2 + 2)):
        out[cell] = list(sim.read_cell_state(*cell).values()) + [sim.read_point(*cell)]
    out["slice"] = sim.read_slice("Dy", "x", nx // 2, f64=True)
    sim.sync()
    sim.profile()
    sim.step(3)
    split = sim.profile_read()["step"]["launches"] == 3
    sim.close()
    return out, split


def _equal(a, b, what):
    if isinstance(a, (list, tuple)):
        for q, (x, y) in enumerate(zip(a, b)):
            _equal(x, y, f"{what}[{q}]")
    else:
        np.testing.assert_array_equal(np.asarray(a), np.asarray(b), err_msg=what)


# tiles of 32 x 16 cells: the smallest grid with one interior tile, remainders of one cell past a tile, z runs cut
# into several ranges, no CPML at all (a run that starts at plane 0)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape,pml,z_chunk", [((65, 49, 40), 0, 0), ((97, 65, 41), 5, 0), ((130, 72, 150), 6, 0),
                                               ((129, 81, 37), 12, 3)])
def test_interior_launch_equals_the_two_sweeps(shape, pml, z_chunk, precision):
    d = _desc(precision, shape, pml, z_chunk)
    nx, ny, nz = shape
    # the monitor: fields and atoms of one block, then of two (slab top), then fields in the interior
    for probe in ((40, 20, 3, 2), (40, 20, nz // 4, nz // 4 - 1), (40, 20, nz - 14, nz - 14)):
        a, na = _run(d, "2", probe, (7, 12, 2))
        b, nb = _run(d, "0", probe, (7, 12, 2))
        assert na and not nb  # the interior's launch, in each of the three steps
        assert np.abs(b["volumes"][2]).max() > 0 and np.abs(b["volumes"][3]).max() > 0
        for k in b:
            _equal(a[k], b[k], f"{k}")


def test_large_domain_takes_the_interior_launch_and_holds_its_planes():
    """By size alone, unless its planes' addresses have been handed out."""
    nx, ny, nz = 224, 224, 176
    med = np.zeros((nx, ny, nz), np.int32)
    dl = 10e-9
    d = make_desc(med, [Material()], [Source(type=1, x=112, y=112, z=80, component="z", frequency=1e15)], dx=dl, dy=dl, dz=dl,
                  dt=dl / (299792458.0 * np.sqrt(3.0)) * 0.99, pml_thickness=8, precision="fp32")
    sim = Simulation(d)
    sim.profile()
    sim.step(5)
    assert sim.profile_read()["step"]["launches"] == 5
    vol = sim.read_volume("Ez")
    from php_fdtd_b200.slab import Slab
    slab = Slab(d, 0, nz)
    slab.step(2)
    planes = [slab.planes(0)[2].data_ptr()]
    slab.step(3)
    assert slab.last_launch_count == 6 and planes == [slab.planes(0)[2].data_ptr()]
    np.testing.assert_array_equal(slab.read_volume("Ez"), vol)
    sim.close()
    slab.close()
