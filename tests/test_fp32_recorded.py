"""FP32-bulk FV results are their FP32 roundings: the WENO indicators' cancellation
moves a face by up to 1e-7 of the stencil's differences, so another form of them,
or another order of a sum, is another result (2e-8 here).  The states are held to
what the register-tiled (small grids) and the pipelined kernel gave at commit
9cacf60, three steps from rough data.

Tolerance: FP64 sums may be ordered differently (1e-13), and where that turns one
FP32 rounding of an increment of at most 0.05 over, a cell moves by 6e-8 x 0.05 =
3e-9; such turns are rare (1e-16 / 6e-8 of the cells a stage)."""
import os

import numpy as np
import pytest

from tests._util import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,nz,nvz,bc", [
    (False, 48, 5, "periodic"), (False, 40, 6, "open"), (True, 64, 5, "periodic"),
    (True, 32, 6, "open")])
def test_fv_fp32_bulk_keeps_its_recorded_results(gpu_lib, monkeypatch, large, nz, nvz, bc):
    from cosenu_b200 import NuOsc
    if large:  # the order of a grid of at least one tile per SM, at a small size
        monkeypatch.setenv("COSENU_KERNEL", "tma")
    rng = np.random.default_rng(nz)
    base = 0.5 + 0.2 * np.sin(2 * np.pi * np.arange(nz) / nz) * rng.uniform(0.5, 1, (8, nvz, 1))
    st = np.zeros((8, nvz, nz + 8))
    st[:, :, 4:-4] = base + rng.uniform(-0.05, 0.05, (8, nvz, nz))
    want = np.load(os.path.join(GOLDEN, "fv_bulk_rough.npz"))[f"{nz}x{nvz}_{bc}"]
    for tile in ({}, {"tile_z": 8, "tile_v": 4}) if not large else ({},):
        with NuOsc(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme="fv", bc=bc, omega=1e-2,
                   theta_deg=37.0, mat=True, mu=0.5, precision="fp32", **tile) as sim:
            sim.upload(st)
            sim.evolve(3)
            d = np.abs(sim.download()[:, :, 4:-4] - want)
        assert d.max() <= 3e-9 and (d > 1e-13).mean() <= 0.01
