"""Planes per block that php_create chooses: few blocks keep short marches, the
strict mode shorter ones than the fast modes."""
import numpy as np
import pytest

from php_fdtd_b200 import Material, Simulation, Source, make_desc

pytestmark = pytest.mark.gpu

DL = 10e-9
DT = DL / (299792458.0 * np.sqrt(3.0)) * 0.99


@pytest.mark.parametrize("n,precision,planes", [(48, "fp64", 1), (80, "fp64", 2), (80, "fp32", 2), (80, "fp64-strict", 1),
                                                (128, "fp64", 4), (128, "fp64-strict", 2), (160, "fp32", 4),
                                                (160, "fp64-strict", 4), (192, "fp32", 8)])
def test_planes_per_block(n, precision, planes):
    src = [Source(type=1, x=n // 2, y=n // 2, z=n // 2, component="z", frequency=1.5e15)]
    desc = make_desc(np.zeros((n, n, n), np.int32), [Material()], src, dx=DL, dy=DL, dz=DL, dt=DT, pml_thickness=4, precision=precision)
    with Simulation(desc) as sim:
        assert sim.block_census()["blocks"] == -(-n // 32) * -(-n // 8) * -(-n // planes)
