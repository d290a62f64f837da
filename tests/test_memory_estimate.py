"""The second field level of the interior launch in the memory estimate: counted
where php_create takes that launch, and only there."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.serving import estimate_bytes
from php_fdtd_b200.workloads import lattice_2atom

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _desc(shape, precision, atoms_to=0, pml=8, tensor_to=0):
    nx, ny, nz = shape
    qv, qm, dmm = lattice_2atom(0)
    med = np.zeros(shape, np.int32)
    med[:, :, :tensor_to] = 2
    med[:, :, :atoms_to] = 1
    mats = [Material(), Material(eps_re=(4.9, 0, 0, 0, 4.9, 0, 0, 0, 2.95), natom=2, qezv=qv, qezm=qm, dmm=dmm),
            Material(eps_re=(6.0, 0, 0, 0, 3.5, 0, 0, 0, 2.8), eps_im=(0.4, 0, 0, 0, 0.2, 0, 0, 0, 0.1), anglez=0.5)]
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=nz // 2, component="z", frequency=1.5e15)]
    return make_desc(med, mats, src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=pml, precision=precision)


# interior share of the 32 x 16 tiles: about 0.7 of the vacuum box; the lattice takes it below 0.4; a CPML of 60 cells too
CASES = [((224, 224, 176), dict(), True), ((224, 224, 176), dict(tensor_to=80), True), ((224, 224, 160), dict(), False),
         ((224, 224, 176), dict(atoms_to=130), False), ((224, 224, 176), dict(pml=60), False)]


@pytest.mark.parametrize("precision,word", [("fp64", 8), ("fp32", 4)])
@pytest.mark.parametrize("shape,kw,taken", CASES)
def test_second_level_is_counted_where_it_is_taken(shape, kw, taken, precision, word, monkeypatch):
    desc = _desc(shape, precision, **kw)
    est = estimate_bytes(desc)
    monkeypatch.setenv("PHP_FUSED", "0")
    without = estimate_bytes(desc)
    nx, ny, nz = shape
    nxp, L = -(-nx // 32) * 32, kw.get("pml", 8)
    level = 6 * nxp * ny * (nz + 2) * word
    # what every such context holds: one level, the CPML state, D, r and v of the lattice
    least = level + (4 * 2 * L * (nz * ny + nz * nxp + ny * nxp) + 15 * nx * ny * kw.get("atoms_to", 0)) * word
    assert without >= least and without - level < least
    assert level <= est - without <= 1.05 * level if taken else est == without


def test_strict_mode_has_no_second_level(monkeypatch):
    desc = _desc((224, 224, 176), "fp64-strict")
    est = estimate_bytes(desc)
    monkeypatch.setenv("PHP_FUSED", "2")
    assert estimate_bytes(desc) == est


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape,kw,taken", CASES)
def test_estimate_covers_the_context(shape, kw, taken, precision):
    desc = _desc(shape, precision, **kw)
    est = estimate_bytes(desc)
    with Simulation(desc) as sim:
        used = sim.memory_bytes
        sim.profile()
        sim.step(2)
        assert (sim.profile_read()["step"]["launches"] > 0) == taken
    assert used <= est <= 1.1 * used + (2 << 20), (used, est)


def test_domains_too_long_for_the_block_lists_keep_the_grid_launches(monkeypatch):
    """A list entry has 15 bits for the tile's y: rows of 262 144 cells and more
    have tiles beyond them."""
    for ny, taken in ((262136, True), (262152, False)):
        desc = _desc((65, ny, 9), "fp32", pml=0)
        est = estimate_bytes(desc)
        with monkeypatch.context() as m:
            m.setenv("PHP_FUSED", "0")
            assert (est > estimate_bytes(desc)) == taken
