"""Routes through the stage kernels that sizes near one tile do not reach: blocks
that go from one work item to the next with partial tiles, the register-tiled kernel
on the reference's recorded snapshots, and ensemble phases long enough to be
replayed from a graph."""
import numpy as np
import pytest

from tests import _longdouble as longdouble
from tests._util import gpu_from_case, load_golden, maxabs_per_comp, with_ghosts
from tests.test_gpu_parity import SMALL, TOL_PRE
from tests.test_stage_kernels import TOL, _rough

pytestmark = pytest.mark.gpu


# 151 tiles, the last of 8 cells, by three chunks of 8 rows, the last of 5: more
# items than block slots (two blocks per SM for FV, one for FD).  Tolerances as for
# the small grids; two steps.
@pytest.mark.parametrize("bc", ["periodic", "open"])
@pytest.mark.parametrize("scheme", ["fv", "fd"])
def test_blocks_of_several_ragged_items(gpu_lib, oracle, scheme, bc):
    import torch
    from oracle.oracle import Case
    nz, nvz = 4808, 21
    case = Case(nz=nz, nvz=nvz, gz=4, z0=-nz / 4, z1=nz / 4, scheme=scheme, bc=bc, omega=1e-2,
                theta_deg=37.0, mat=True, mu=0.5)
    st0 = _rough(case, oracle, 2)
    if scheme == "fv":
        ref = longdouble.step(case, st0[..., case.gz:case.gz + nz], 2)
    else:
        ref = oracle.step(case, st0, 2)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for precision in ("fp64", "fp32"):
        with gpu_from_case(case, precision=precision) as sim:
            tz, tv = sim.tile()
            assert -(-nz // tz) * -(-nvz // tv) > sms * (2 if scheme == "fv" else 1)
            sim.upload(st0)
            sim.evolve(2)
            assert np.abs(sim.download() - ref).max() <= TOL[precision], precision


@pytest.mark.parametrize("name", SMALL)
def test_register_tiled_kernel_matches_reference(gpu_lib, oracle, monkeypatch, name):
    monkeypatch.setenv("COSENU_KERNEL", "ldg")
    case, d = load_golden(name)
    with gpu_from_case(case) as sim:
        sim.upload(with_ghosts(case, d["state0"], oracle))
        t_prev = 0
        for t in d["dump_steps"]:
            sim.evolve(int(t) - t_prev)
            t_prev = int(t)
            got = sim.download()[..., case.gz:case.gz + case.nz]
            assert np.all(maxabs_per_comp(got, d[f"rho_{t}"]) <= TOL_PRE), (name, int(t))


# Phases of 131 and 170 steps (graphs of 16 steps and a rest launched directly),
# then a short one that starts from the other buffer parity (FP32-bulk).  Smooth
# states far from saturation: rounding only, 1e-12 leaves three orders.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("scheme", ["fv", "fd"])
def test_long_ensemble_phases(gpu_lib, monkeypatch, scheme, precision):
    from cosenu_b200 import NuOsc
    from cosenu_b200.ensemble import Ensemble, Instance
    xs = [Instance(nz=nz, nvz=nvz, alpha=0.9, sig_nu=0.6, sig_nubar=0.5, mu=0.05, seed=i,
                   nsteps=n, z0=-nz / 4, z1=nz / 4)
          for i, (nz, nvz, n) in enumerate(((256, 16, 131), (512, 24, 301), (320, 9, 308)))]
    with Ensemble(xs, scheme=scheme, precision=precision) as ens:
        ens.init_seeded(amp=1e-2)
        ens.run()
        ens.synchronize()
        got = [m.download() for m in ens.members]
    monkeypatch.setenv("COSENU_KERNEL", "tma")
    for i, x in enumerate(xs):
        with NuOsc(x.params(scheme, precision)) as sim:
            sim.init_seeded(x.seed, instance=i, sig_nu=x.sig_nu, sig_nubar=x.sig_nubar,
                            alpha=x.alpha, amp=1e-2)
            sim.evolve(x.nsteps)
            assert np.abs(got[i] - sim.download()).max() <= 1e-12, i
