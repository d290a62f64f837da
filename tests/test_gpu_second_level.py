"""Whether a large domain gets the second field level of the interior launch:
memory that the device's pool holds and nothing uses counts as free."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.serving import Server, estimate_bytes

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


def _desc(precision="fp32", shape=(224, 224, 176)):
    nx, ny, nz = shape
    src = [Source(type=1, x=nx // 2, y=ny // 2, z=nz // 2, component="z", frequency=1.5e15)]
    return make_desc(np.zeros(shape, np.int32), [Material()], src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=8, precision=precision)


def _interior_launch(sim):
    sim.profile()
    sim.step(1)
    taken = sim.profile_read()["step"]["launches"] > 0
    sim.profile(False)
    return taken


def test_memory_that_the_pool_keeps_is_free():
    torch = pytest.importorskip("torch")
    rt = pytest.importorskip("cuda.bindings.runtime")
    torch.cuda.init()
    free, total = torch.cuda.mem_get_info(0)
    take = int(0.55 * total)
    if free < take + (4 << 30):
        pytest.skip("device memory in use")

    def ck(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1] if len(r) > 1 else None
    pool = ck(rt.cudaDeviceGetMemPool(0))
    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrReleaseThreshold
    old = ck(rt.cudaMemPoolGetAttribute(pool, attr))
    stream = ck(rt.cudaStreamCreate())
    try:
        from cuda.bindings import driver
        ck(rt.cudaMemPoolSetAttribute(pool, attr, driver.cuuint64_t(2 ** 63)))
        p = ck(rt.cudaMallocAsync(take, stream))
        ck(rt.cudaFreeAsync(p, stream))
        ck(rt.cudaStreamSynchronize(stream))
        assert torch.cuda.mem_get_info(0)[0] < total / 2          # the pool kept it
        with Simulation(_desc()) as sim:
            assert _interior_launch(sim)
    finally:
        ck(rt.cudaMemPoolSetAttribute(pool, attr, old))
        ck(rt.cudaMemPoolTrimTo(pool, 0))
        ck(rt.cudaStreamDestroy(stream))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_domain_is_created_without_it_where_it_cannot_be_had(precision, monkeypatch):
    with Simulation(_desc(precision)) as sim:
        assert _interior_launch(sim)
        sim.step(20)
        with_it, vol = sim.memory_bytes, sim.read_volume("Ez")
    monkeypatch.setenv("PHP_TEST_NO_SECOND_LEVEL", "1")     # its allocation fails, after a part of it
    with Simulation(_desc(precision)) as sim:
        assert not _interior_launch(sim)
        sim.step(20)
        level = 6 * 224 * 224 * 178 * (4 if precision == "fp32" else 8)
        assert sim.memory_bytes <= with_it - level
        assert np.abs(vol).max() > 0
        np.testing.assert_array_equal(sim.read_volume("Ez"), vol)


def test_server_charges_it_to_the_budget_only_where_it_is_held(monkeypatch):
    """Two such jobs under a budget of one with it and one without: the second
    runs beside the first only once the first's unused bytes come back."""
    desc = _desc()
    full = estimate_bytes(desc)
    with monkeypatch.context() as m:
        m.setenv("PHP_FUSED", "0")
        bare = estimate_bytes(desc)

    def serve():
        with Server(memory_budget=full + bare - 1) as srv:
            for _ in range(2):
                srv.submit(desc, 2000)
            done = []
            while len(done) < 2:
                done += srv.poll(timeout_ms=20000)
            return [d["device_bytes"] for d in done], srv.stats()
    got, stats = serve()
    assert got[0] == full and stats["peak_running"] == 1
    monkeypatch.setenv("PHP_TEST_NO_SECOND_LEVEL", "1")
    got, stats = serve()
    assert got == [bare, bare] and stats["peak_running"] == 2
