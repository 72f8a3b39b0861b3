"""The strict FP32 backward takes the records 32 at a time through its MLP
products and 64 at a time through its weight-gradient reductions.

The gradient of a few rays, whose records end anywhere in a tile, is the mean of
the gradients of its rays alone: each sample's own arithmetic is the same in
every place of a tile, so only the order of the FP32 sums differs (relative L2
1e-4, the bound of FP32 accumulation with atomics; 1e-5 on the loss)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOG2T = 12
TABLE_FLOATS = 16 * (1 << LOG2T) * 2
W = H = 16


@pytest.mark.parametrize("n", [2, 3, 5, 9])
def test_records_ending_anywhere_in_a_tile(nes_lib, cuda, n):
    f = nes_lib.focal_from_fov(W, 30.0)
    views = [nes_lib.make_view(M, W, H, f) for M in nes_lib.shell_poses(1, 2, 1.3, 1.6)]
    g = cuda.Generator(device="cuda").manual_seed(n)
    rgb = cuda.rand((2 * W * H, 3), device="cuda", generator=g)
    dep = 1.0 + 0.5 * cuda.rand((2 * W * H,), device="cuda", generator=g)
    r = nes_lib.Renderer(precision=nes_lib.PREC_FP32, seed=4, log2_table_size=LOG2T, max_pixels=W * H * 2)
    t = nes_lib.Trainer(r, batch_rays=16, exact_weight_grads=1)
    t.set_targets(views, rgb.data_ptr(), dep.data_ptr())
    rng = np.random.default_rng(n)
    pairs = np.stack([rng.integers(0, 2, n), rng.integers(0, W * H, n)], 1).astype(np.int32)
    loss, gt, gw = t.grad(pairs, TABLE_FLOATS)
    samples = t.last_samples()
    alone, count = [], 0
    for k in range(n):
        alone.append(t.grad(pairs[k:k + 1], TABLE_FLOATS))
        count += t.last_samples()
    t.close()
    r.close()
    assert count == samples > 0
    assert abs(loss - np.mean([a[0] for a in alone])) <= 1e-5 * loss
    for whole, k in ((gt, 1), (gw, 2)):
        want = np.mean([a[k].astype(np.float64) for a in alone], 0)
        assert np.linalg.norm(whole - want) <= 1e-4 * np.linalg.norm(want)
