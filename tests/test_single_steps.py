"""One step per call: launched directly at first, then as a replay of the captured
step.  The routes launch the same kernels on the same data, so states agree bit for
bit."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(precision="fp64", **kw):
    from cosenu_b200 import NuOsc
    sim = NuOsc(nz=96, nvz=16, gz=4, z0=-24.0, z1=24.0, omega=1e-2, theta_deg=37.0, mu=0.5,
                precision=precision, **kw)
    rng = np.random.default_rng(3)
    st = np.zeros((8, 16, 104))
    st[:, :, 4:-4] = 0.5 + rng.uniform(-0.1, 0.1, (8, 16, 96))
    sim.upload(st)
    return sim


def _set_mu(sim, mu):
    sim._check(sim.lib.cosenu_set_collective_pars(sim.h, mu))


@pytest.mark.parametrize("scheme", ["fv", "fd"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("every", [0, 1, 10])
def test_single_steps_equal_a_stretch(gpu_lib, scheme, precision, every):
    n = 40
    mus = [0.5 + (0.01 * (i // every) if every else 0.0) for i in range(n)]
    out = []
    for single in (True, False):
        with _sim(precision, scheme=scheme) as sim:
            i = 0
            while i < n:
                k = 1 if single else (every or n)
                if every and i % every == 0:
                    _set_mu(sim, mus[i])
                sim.step_rk4() if single else sim.evolve(k)
                i += k
            assert sim.steps == n
            out.append(sim.download())
    assert np.array_equal(*out)


# within a caller's own capture a step is launched into it, before and after the
# context has a graph of its own
@pytest.mark.parametrize("before", [0, 12])
def test_step_inside_a_callers_capture(gpu_lib, before):
    import torch
    stream = torch.cuda.Stream()
    with _sim() as sim, _sim() as plain:
        sim.synchronize()
        sim.set_stream(stream.cuda_stream)
        for _ in range(before):
            sim.step_rk4()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            sim.step_rk4()
            sim.step_rk4()
        with torch.cuda.stream(stream):
            g.replay()
            g.replay()
        torch.cuda.synchronize()
        plain.evolve(before + 4)
        assert np.array_equal(sim.download(), plain.download())
        del g


# A parameter changed between any two steps drops the captured step.  Capturing it
# again each time takes about 0.5 ms a step; directly a step takes about 0.05 ms with
# the change's synchronisation.
def test_changing_a_parameter_every_step_does_not_capture(gpu_lib, monkeypatch):
    def best(n=200):
        t = []
        with _sim() as sim:
            for _ in range(3):
                t0 = time.perf_counter()
                for i in range(n):
                    _set_mu(sim, 0.5 + 1e-3 * i)
                    sim.step_rk4()
                sim.synchronize()
                t.append(time.perf_counter() - t0)
        return min(t)
    ours = best()
    monkeypatch.setenv("COSENU_NO_GRAPH", "1")
    assert ours < 3 * best()
