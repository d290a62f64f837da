"""The cells of which the fast modes keep E alone: only where D, read out as
M^-1 E, is as accurate as a stored D within a factor of two.  Rotated materials
of higher contrast keep D in the pool; diagonal ones of any contrast to 256 need
not."""
import numpy as np
import pytest

import harness as H
from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.serving import estimate_bytes

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _desc(material, precision, shape=(40, 36, 33)):
    med = np.zeros(shape, np.int32)
    med[6:-6, 6:-6, 6:-6] = 1
    nx, ny, nz = shape
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=nz // 2, component=c, frequency=f) for c, f in (("z", 1.5e15), ("x", 1e15), ("y", 2e15))]
    return make_desc(med, [Material(), material], src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=4, precision=precision), int(med.sum())


def _turned(c, axis="z", angle=0.6):
    eps = (c, 0, 0, 0, 1.5, 0, 0, 0, 1.5) if axis == "z" else (1.5, 0, 0, 0, 1.5, 0, 0, 0, c)
    return Material(eps_re=eps, **{f"angle{axis}": angle})


@pytest.mark.parametrize("precision,word", [("fp64", 8), ("fp32", 4)])
@pytest.mark.parametrize("material,pooled", [
    (Material(eps_re=(2.25, 0, 0, 0, 2.25, 0, 0, 0, 2.25)), False),
    (Material(eps_re=(1.5, 0, 0, 0, 2.0, 0, 0, 0, 300.0)), False),                 # diagonal, contrast of 200
    (Material(eps_re=(6.0, 0, 0, 0, 3.5, 0, 0, 0, 2.8), anglez=np.pi / 6), False),  # 1.7 in the turned plane
    (_turned(12.0), True), (_turned(48.0, "x"), True), (_turned(300.0, "z", 0.8), True),
    (Material(eps_re=(9.0, 3.0, 0, 3.0, 2.0, 0, 0, 0, 2.5)), True),                # full tensor, eigenvalues 10.1, 0.9
    (Material(eps_re=(1.0, 0, 0, 0, 1.0, 0, 0, 0, 1e6)), True)])                   # no read-out from E
def test_which_materials_keep_d(material, pooled, precision, word):
    desc, ncell = _desc(material, precision)
    plain, _ = _desc(Material(eps_re=(2.0, 0, 0, 0, 2.0, 0, 0, 0, 2.0)), precision)
    more = estimate_bytes(desc) - estimate_bytes(plain)
    assert (more >= 3 * word * ncell) if pooled else (more == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("c,axis,angle", [(12.0, "z", 0.6), (48.0, "x", 0.6), (300.0, "z", 0.8), (2.9, "z", 0.8)])
def test_fp32_d_is_as_accurate_as_h(c, axis, angle):
    """D and H are both sums of single-precision increments of one stencil, so
    their errors against FP64, relative to their size, agree within a small
    factor; 4 is allowed (D is a sum of the same length as H, in one cell in
    six of other materials)."""
    got, want = {}, {}
    for out, precision in ((got, "fp32"), (want, "fp64")):
        with Simulation(_desc(_turned(c, axis, angle), precision)[0]) as sim:
            sim.step(400)
            for name, comps in (("D", "Dx Dy Dz"), ("H", "Hx Hy Hz")):
                out[name] = np.stack([sim.read_volume(q)[6:-6, 6:-6, 6:-6] for q in comps.split()])
    err = {k: H.rel_l2(got[k], want[k]) for k in got}
    assert 0 < err["H"] < 1e-4
    assert err["D"] <= 4 * err["H"], err


@pytest.mark.gpu
@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("fp32", 1e-5)])   # as between the block paths elsewhere
@pytest.mark.parametrize("shape", [(41, 33, 29), (97, 65, 64)])                 # one E sweep; a launch per kind of block
def test_blocks_of_a_material_that_keeps_d(shape, precision, rtol, monkeypatch):
    """The blocks of that material alone against the general path, in the two
    sweeps and in the one-launch step, with the material lossy, and a metal (ADE)
    of fewer cells beside it."""
    nx, ny, nz = shape
    med = np.zeros(shape, np.int32)
    med[:, :, nz // 4:nz // 2] = 1
    med[nx // 2:nx // 2 + 4, ny // 2:ny // 2 + 4, nz // 2:] = 2
    mats = [Material(), Material(eps_re=(12.0, 0, 0, 0, 1.5, 0, 0, 0, 2.0), eps_im=(0.3, 0, 0, 0, 0.2, 0, 0, 0, 0.1), anglez=0.6),
            Material(eps_re=(-300, 0, 0, 0, -300, 0, 0, 0, -300), eps_im=(150, 0, 0, 0, 150, 0, 0, 0, 150), use_ade=1)]
    src = [Source(type=1, x=nx // 3, y=ny // 3, z=nz // 2 + 1, component="z", frequency=1.5e15)]
    desc = make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=4, precision=precision, source_frequency=3e13)
    out = []
    for plain, fused in (("0", "0"), ("1", "0"), ("1", "1")):
        monkeypatch.setenv("PHP_PLAIN_ATOMS", plain)
        monkeypatch.setenv("PHP_FUSED", fused)
        with Simulation(desc) as sim:
            pid = sim.dft_add("Dx", nz // 3, [1.5e15])
            sim.step(150)
            out.append([sim.read_volume(c) for c in range(9)] + [sim.dft_read(pid)[0]])
            assert (sim.block_census()["e_atoms"] > 0) == (plain == "1")
    for q, (y, *others) in enumerate(zip(*out)):
        assert np.abs(y).max() > 0
        for x in others:
            np.testing.assert_allclose(x, y, rtol=0, atol=rtol * np.abs(y).max(), err_msg=f"output {q}")
