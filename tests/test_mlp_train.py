"""The fused training kernels against the separate ones (which the timing mode
keeps): the same operations in the same order, so the parameters agree bit for
bit; the epoch loss is summed in another order, over at most 64 FP32 additions
before FP64 takes over (64 x 6e-8).  Batches around the 64- and 128-row tiles,
ragged last batches, output widths that leave half a 16-column tile, K below and
at multiples of the 64-deep groups, one hidden layer, and a batch beyond the
fused path's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,batch,rows", [
    ((258, 512, 3, 128), 64, 200), ((258, 512, 3, 128), 50, 130), ((258, 512, 3, 128), 200, 450),
    ((30, 32, 2, 24), 1, 5), ((30, 48, 1, 8), 65, 131), ((64, 64, 2, 16), 128, 128),
    ((17, 80, 4, 40), 129, 300), ((30, 32, 2, 16), 513, 600)])
def test_fused_training_equals_separate_kernels(gpu_lib, shape, batch, rows):
    from cosenu_b200.surrogate import MLP
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, shape[0])).astype(np.float32)
    t = rng.uniform(0, 1, (rows, shape[3])).astype(np.float32)
    out = []
    for separate in (False, True):
        net = MLP(*shape, seed=7)
        net.set_data(x, t)
        net.set_timing(separate)
        losses = net.train(epochs=3, batch=batch, lr=2e-3, weight_decay=1e-2, seed=4)
        out.append((losses, net.params()))
        net.close()
    (la, pa), (lb, pb) = out
    assert np.array_equal(pa, pb)
    assert np.abs(la / lb - 1).max() <= 64 * 6e-8
