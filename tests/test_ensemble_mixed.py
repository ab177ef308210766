"""Ensembles whose members differ in more than size, or are stepped by themselves
between the shared runs, against the same members alone, from rough data.

Tolerances.  FP64: moments are summed in other pieces, a few 1e-16 a stage; 1e-12
leaves three orders.  FP32-bulk: such a difference may turn the FP32 rounding of an
increment (at most 0.05: 3e-9) over, now and then in more than one stage: 1e-8."""
import numpy as np
import pytest

from cosenu_b200 import _lib as L
from cosenu_b200.ensemble import Instance

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 1e-8}


class _Flagged(Instance):
    flags = 0

    def params(self, *args, **kw):
        p = super().params(*args, **kw)
        p.flags |= self.flags
        return p


def _member(nz, nvz, nsteps, flags=0):
    x = _Flagged(nz=nz, nvz=nvz, alpha=1.0, sig_nu=0.6, sig_nubar=0.5, mu=0.5, seed=0,
                 nsteps=nsteps, z0=-nz / 4, z1=nz / 4)
    x.flags = flags
    return x


def _rough(x, seed):
    rng = np.random.default_rng(seed)
    base = 0.5 + 0.2 * np.sin(2 * np.pi * np.arange(x.nz) / x.nz) * \
        rng.uniform(0.5, 1, (8, x.nvz, 1))
    st = np.zeros((8, x.nvz, x.nz + 8))
    st[:, :, 4:-4] = base + rng.uniform(-0.05, 0.05, (8, x.nvz, x.nz))
    return st


def _alone(x, i, precision, nsteps, monkeypatch):
    from cosenu_b200 import NuOsc
    monkeypatch.setenv("COSENU_KERNEL", "tma")
    with NuOsc(x.params("fv", precision)) as sim:
        sim.upload(_rough(x, i))
        sim.evolve(nsteps)
        return sim.download()


# 148 tiles a member: three members share each of the 296 block slots, so that
# blocks go from members with advection to members without it and back, after odd
# and even numbers of chunks.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_members_with_and_without_advection(gpu_lib, monkeypatch, precision):
    from cosenu_b200.ensemble import Ensemble
    xs = [_member(4736, nvz, 4, flags) for nvz, flags in
          ((24, 0), (24, L.ADVEC_OFF), (16, 0), (40, L.ADVEC_OFF), (9, 0))]
    with Ensemble(xs, precision=precision) as ens:
        for i, (x, m) in enumerate(zip(xs, ens.members)):
            m.upload(_rough(x, i))
        ens.run()
        ens.synchronize()
        got = [m.download() for m in ens.members]
    for i, x in enumerate(xs):
        want = _alone(x, i, precision, x.nsteps, monkeypatch)
        assert np.abs(got[i] - want).max() <= TOL[precision], i


# The shared launches and a member's own read each other's moments of the state.
# Step by step, as a stretch and stage by stage between two shared runs; row counts
# that are and are not multiples of the 8-row chunk, and fewer rows than one.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("scheme", ["fv", "fd"])
@pytest.mark.parametrize("tiled", [False, True])
def test_members_step_on_their_own_between_runs(gpu_lib, monkeypatch, scheme, precision, tiled):
    from cosenu_b200.ensemble import Ensemble
    xs = [_member(nz, nvz, 0) for nz, nvz in ((256, 37), (512, 64), (96, 5), (4736, 24))]
    with Ensemble(xs, scheme=scheme, precision=precision) as ens:
        if tiled:
            ens.set_config(False, 16, [16, 24, 5, 8])
        for i, (x, m) in enumerate(zip(xs, ens.members)):
            m.upload(_rough(x, i))
        ens.run([2, 3, 1, 2])
        for m in ens.members:
            m.step_rk4()
            m.evolve(2)
            for s in range(4):
                m.step_stage(s)
        ens.run([1, 2, 2, 1])
        ens.synchronize()
        got = [m.download() for m in ens.members]
    from cosenu_b200 import NuOsc
    monkeypatch.setenv("COSENU_KERNEL", "tma")
    for i, (x, n) in enumerate(zip(xs, (7, 9, 7, 7))):
        p = x.params(scheme, precision)
        if tiled:
            p.tile_z, p.tile_v = 16, (16, 24, 5, 8)[i]
        with NuOsc(p) as sim:
            sim.upload(_rough(x, i))
            sim.evolve(n)
            assert np.abs(got[i] - sim.download()).max() <= 3 * TOL[precision], i
