"""FV faces in FP64: the range of the shared division, and what it must not change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# States in other units (an amplitude of 1e15 is 1/cm^3 scale): without the source
# terms the scheme is linear in the amplitude up to WENO's absolute epsilon.  The
# product of four neighbouring faces' denominators leaves the FP64 range at
# differences of 1e5.  Mixed: rows and stretches of ordinary size beside large
# ones.  Tolerance as for amplitude 1 (tests/test_stage_kernels.py), relative to
# the row's amplitude.
@pytest.mark.parametrize("bc", ["periodic", "open"])
@pytest.mark.parametrize("amp", [1.0, 1e4, 3e5, 1e7, 1e15, "mixed"])
def test_large_amplitudes(gpu_lib, amp, bc):
    from cosenu_b200 import NuOsc
    from oracle.oracle import Case
    from tests import _longdouble as longdouble
    nz, nvz = 72, 10
    case = Case(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme="fv", bc=bc, omega=0.0,
                mu=0.0)
    rng = np.random.default_rng(11)
    size = np.full((8, nvz, 1), 1.0 if amp == "mixed" else amp)
    if amp == "mixed":
        size[:] = 10.0 ** rng.uniform(0, 15, size.shape)
    st = size * (0.5 + 0.2 * np.sin(2 * np.pi * np.arange(nz) / nz) +
                 rng.uniform(-0.05, 0.05, (8, nvz, nz)))
    if amp == "mixed":
        st[:, :, 20:24] *= 1e-3
    x = np.zeros((8, nvz, case.ld))
    x[:, :, 4:-4] = st
    with NuOsc(nz=nz, nvz=nvz, gz=4, z0=case.z0, z1=case.z1, scheme="fv", bc=bc, mu=0.0,
               vac=False, coll=False) as sim:
        sim.upload(x)
        sim.evolve(3)
        got = sim.download()
    want = longdouble.step(case, st, 3)
    assert np.isfinite(got).all()
    assert (np.abs(got - want) / size).max() <= 1e-12


# What leaves a cell enters its neighbour: a face has the same bits whether its tile
# computes it among its neighbours or the next tile by itself, at its upwind edge.
# Moving a periodic state by four cells (the faces that share a division) moves
# every tile edge and no quad, so the steps of the moved state are the moved steps,
# bit for bit.  Partial last tiles included.
@pytest.mark.parametrize("nz,nvz", [(64, 16), (72, 9), (1000, 37), (4736, 10)])
def test_tile_edges_leave_no_trace(gpu_lib, nz, nvz):
    from cosenu_b200 import NuOsc
    rng = np.random.default_rng(nz)
    st = 0.5 + 0.2 * np.sin(2 * np.pi * np.arange(nz) / nz) * rng.uniform(0.5, 1, (8, nvz, 1)) + \
        rng.uniform(-0.05, 0.05, (8, nvz, nz))
    out = []
    for shift in (0, 4):
        x = np.zeros((8, nvz, nz + 8))
        x[:, :, 4:-4] = np.roll(st, shift, -1)
        with NuOsc(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme="fv", omega=1e-2,
                   theta_deg=37.0, mu=0.5) as sim:
            sim.upload(x)
            sim.evolve(3)
            out.append(np.roll(sim.download()[:, :, 4:-4], -shift, -1))
    assert np.array_equal(*out)
