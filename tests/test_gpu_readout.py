"""Read-outs at the sizes where their kernels can go wrong: the diagnostics'
maxima and the argmax's loop order (rows shorter than a vector, odd widths,
fewer rows than warps, equal maxima), the running DFT in the caller's order
(one and several chunks of the device's scratch), and frames whose slice and
monitor rows the device writes to host memory itself or that go by a copy."""
import numpy as np
import pytest

import harness as H
from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.workloads import lattice_2atom

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _sim(shape, precision, pml=0):
    nx, ny, nz = shape
    qv, qm, dmm = lattice_2atom(0)
    med = np.zeros(shape, np.int32)
    med[nx // 3:, :, :] = 1
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm)]
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=nz // 2, component="z", frequency=1.5e15)]
    return Simulation(make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=pml, precision=precision,
                                source_frequency=3.0e13)), med


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(3, 21, 5), (33, 17, 9), (66, 5, 3)])
def test_diagnostics_are_the_first_maxima_in_loop_order(precision, shape):
    """The source sits in the mirror plane of y and z, so maxima come in equal
    pairs; the maximum of the fields read back, and the first of the largest
    |r| in the order i, j, k, coordinate, exactly."""
    sim, med = _sim(shape, precision)
    with sim:
        for n in (2, 25):
            sim.step(n)
            d = sim.diagnostics()
            ex, ey, ez = (sim.read_volume(c) for c in ("Ex", "Ey", "Ez"))
            assert d["max_e"] == np.sqrt(ex * ex + ey * ey + ez * ez).max() > 0
            assert d["max_ex"] == np.abs(ex).max()
            best, where = 0.0, (-1,) * 5
            for i, j, k in np.ndindex(shape):
                if not med[i, j, k]:
                    continue
                r = np.abs(sim.read_cell_state(i, j, k)["r"])
                if r.max() > best:
                    q = int(r.argmax())
                    best, where = float(r.max()), (i, j, k, q // 3, q % 3)
            assert (d["max_r"], d["argmax_r"]) == (best, where)


@pytest.mark.parametrize("shape,freqs", [((33, 70, 5), [3e13]), ((130, 71, 3), [3e13, 1.5e15, 4e14]), ((4, 300, 3), [1e15, 3e13])])
def test_dft_read_in_the_callers_order(shape, freqs):
    z = shape[2] // 2
    sim, _ = _sim(shape, "fp64")
    ref, _ = _sim(shape, "fp64")
    pid = sim.dft_add("Ez", z, freqs)
    acc = np.zeros((len(freqs),) + shape[:2], complex)
    for t in range(25):
        ref.step(1)
        acc += ref.read_volume("Ez")[:, :, z] * np.exp(-2j * np.pi * np.array(freqs) * (t * DT))[:, None, None]
    sim.step(25)
    got, ns = sim.dft_read(pid)
    assert np.abs(acc).max() > 0
    assert ns == 25 and got.shape == acc.shape and np.iscomplexobj(got)
    assert H.rel_l2(got, acc) < 1e-12                 # 25 FP64 samples: rounding of the sums alone
    sim.close()
    ref.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape,steps", [((33, 20, 9), (1, 40)), ((260, 260, 4), (3, 420))])
def test_frames_hold_what_the_synchronous_reads_return(precision, shape, steps):
    """A slice of 260 x 260 (264 KB) and 420 monitor rows (69 KB) go by a copy,
    the smaller ones by the device's own writes."""
    a, _ = _sim(shape, precision)
    b, _ = _sim(shape, precision)
    cell = (shape[0] // 2, shape[1] // 2, shape[2] // 2)
    for s in (a, b):
        s.probe_set(*cell, cell[2])
    for n in steps:
        for s in (a, b):
            s.step(n)
        for axis, pos, rows in (("z", 1, True), ("x", 5, True)):
            fr = a.frame_wait(a.frame_begin(diag=True, slice=("Ez", axis, pos), probe=rows, point=cell, cell=cell))
            assert fr["step"] == b.t and fr["diag"] == b.diagnostics()
            np.testing.assert_array_equal(fr["slice"], b.read_slice("Ez", axis, pos).ravel())
            np.testing.assert_array_equal(fr["rows"], b.probe_read())     # the second time: none left
            np.testing.assert_array_equal(fr["point"], b.read_point(*cell))
            np.testing.assert_array_equal(fr["cell"]["r"], b.read_cell_state(*cell)["r"])
            i, j, k = fr["diag"]["argmax_r"][:3]
            if i >= 0:
                np.testing.assert_array_equal(fr["diag_cell"]["r"], b.read_cell_state(i, j, k)["r"])
    a.close()
    b.close()
