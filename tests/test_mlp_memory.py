"""The fused training path's own buffers (a shuffled copy of the data among them)
are an option, not a condition: with no room left for them training runs on the
separate launches, with the same parameters bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_training_with_device_memory_nearly_full(gpu_lib):
    import torch
    from cosenu_b200.surrogate import MLP
    rng = np.random.default_rng(0)
    rows, shape = 200_000, (258, 64, 1, 128)  # the copy: 211 MB
    x = rng.normal(size=(rows, shape[0])).astype(np.float32)
    t = rng.uniform(0, 1, (rows, shape[3])).astype(np.float32)
    out = []
    for full in (False, True):
        net = MLP(*shape, seed=7)
        net.set_data(x, t)
        hold = None
        if full:
            hold = torch.empty(torch.cuda.mem_get_info()[0] - (150 << 20), dtype=torch.uint8,
                               device="cuda")
        try:
            losses = net.train(epochs=1, batch=512, lr=2e-3, seed=4)
        finally:
            del hold
            torch.cuda.empty_cache()
        out.append((losses, net.params()))
        net.close()
    (la, pa), (lb, pb) = out
    assert np.array_equal(pa, pb)
    assert np.abs(la / lb - 1).max() <= 64 * 6e-8
