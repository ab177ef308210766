"""The pipelined stage kernels at the sizes where their tiling can go wrong:
one tile (whose cells are copied to both ghost zones), row counts around the
8-row chunk, rows of both signs of v in a chunk, both boundaries, on rough data
(random differences of 0.1 between neighbours), against long double (FV) or the
CPU oracle (FD).

Tolerances.  FP64: the differences are rounding, a few 1e-16 per operation and
stage; 1e-12 leaves four orders for three steps.  FP32-bulk: an increment
dt k <= 0.5 is held to 6e-8, and the WENO correction (at most the neighbour
differences, 0.4 over a stencil) to about ten roundings of 6e-8 times the
Courant number 0.4: 1e-7 a stage, 12 stages.
"""
import numpy as np
import pytest

from tests import _longdouble as longdouble

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 2e-6}


def _rough(case, oracle, seed):
    rng = np.random.default_rng(seed)
    st = np.zeros((8, case.nvz, case.ld))
    z = 2 * np.pi * np.arange(case.nz) / case.nz
    base = 0.5 + 0.2 * np.sin(z)[None, None, :] * rng.uniform(0.5, 1, (8, case.nvz, 1))
    st[:, :, case.gz:case.gz + case.nz] = base + rng.uniform(-0.05, 0.05,
                                                            (8, case.nvz, case.nz))
    return oracle.fill_ghosts(case, st)


def _compare(oracle, case, precision, steps=3, seed=0, **kw):
    from tests._util import gpu_from_case
    st0 = _rough(case, oracle, seed)
    if case.scheme == "fv":
        ref = longdouble.step(case, st0[..., case.gz:case.gz + case.nz], steps)
    else:
        ref = oracle.step(case, st0, steps)
    with gpu_from_case(case, precision=precision, **kw) as sim:
        tile = sim.tile()
        sim.upload(st0)
        sim.evolve(steps)
        got = sim.download()
    assert np.abs(got - ref).max() <= TOL[precision]
    return tile


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("bc", ["periodic", "open"])
# partial last tiles of 8, 16 and 24 cells (down to a lone one), tiles shared by
# as many blocks as they have chunks, and (968, 77): 310 chunks on 296 block
# slots, so that blocks straddle tiles
@pytest.mark.parametrize("nz,nvz", [(32, 1), (32, 7), (64, 8), (64, 9), (96, 33), (160, 264),
                                    (16, 3), (24, 8), (40, 17), (72, 9), (968, 77)])
def test_fv_pipelined_kernel_edges(gpu_lib, oracle, monkeypatch, nz, nvz, bc, precision):
    from oracle.oracle import Case
    monkeypatch.setenv("COSENU_KERNEL", "tma")
    case = Case(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme="fv", bc=bc, omega=1e-2,
                theta_deg=37.0, mat=True, mu=0.5)
    assert _compare(oracle, case, precision)[0] == 32


# FD: as above with its chunks of 8 and 12 rows, and bands of v (200 x 37: 7
# tiles in bands of 12 rows; 1000 x 100: 32 tiles on 148 SMs)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("bc,fd_advec,ko", [("periodic", "center", 3), ("open", "center", 3),
                                            ("open", "lopsided", 5), ("periodic", "upwind", 5)])
@pytest.mark.parametrize("nz,nvz", [(16, 1), (24, 13), (32, 8), (40, 25), (200, 37), (1000, 100)])
def test_fd_pipelined_kernel_edges(gpu_lib, oracle, nz, nvz, bc, fd_advec, ko, precision):
    from oracle.oracle import Case
    case = Case(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme="fd", bc=bc, omega=1e-2,
                theta_deg=37.0, mat=True, mu=0.5, fd_advec=fd_advec, ko_order=ko)
    assert _compare(oracle, case, precision)[0] == 32


# A call's launches overlap (a stage's blocks start before the previous stage has
# ended); single-stage calls are launched one after the other.  Same bits, at one
# tile, at less and more than a block per SM, and over a replayed step.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("scheme", ["fv", "fd"])
@pytest.mark.parametrize("nz,nvz", [(32, 8), (1000, 37), (9600, 40)])
def test_overlapping_launches_keep_order(gpu_lib, oracle, nz, nvz, scheme, precision):
    from oracle.oracle import Case
    from tests._util import gpu_from_case
    case = Case(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme=scheme, omega=1e-2,
                theta_deg=37.0, mu=0.5)
    st0 = _rough(case, oracle, 1)
    out = []
    for overlap in (True, False):
        with gpu_from_case(case, precision=precision) as sim:
            sim.upload(st0)
            if overlap:
                for n in (1, 3, 19, 1):
                    sim.evolve(n)
            else:
                for i in range(4 * 24):
                    sim.step_stage(i % 4)
            out.append(sim.download())
    assert np.array_equal(*out)
