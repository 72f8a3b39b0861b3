"""The training pass lists, encodes and evaluates as many blocks of 256 rays at
a time as its sample list holds (2^26 samples), and runs the backward's MLP,
scatter-add and weight-gradient kernels over chunks of the records.

A batch of 2^18 rays with over 2^26 samples goes in several parts: its loss
and gradient are the means of those of its four quarters, which fit the list
(FP32 sums in another order: relative 1e-5 on the loss, relative L2 1e-4 on the
gradients, the bound of FP32 accumulation with atomics).  Ray counts around a
warp, a 128-record tile and a 256-ray block: the tensor-core mode against the
strict FP32 mode within the few-ray TF32 bounds of the oracle comparison (3e-2
relative L2, 0.25 of the largest entry), the same samples in both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOG2T = 14
TABLE_FLOATS = 16 * (1 << LOG2T) * 2
W = H = 16


@pytest.fixture(scope="module")
def targets(nes_lib, cuda):
    f = nes_lib.focal_from_fov(W, 30.0)
    views = [(M, W, H, f) for M in nes_lib.shell_poses(1, 2, 1.3, 1.6)]
    g = cuda.Generator(device="cuda").manual_seed(5)
    rgb = cuda.rand((2 * W * H, 3), device="cuda", generator=g)
    dep = 1.0 + 0.5 * cuda.rand((2 * W * H,), device="cuda", generator=g)
    return views, rgb, dep


def _trainer(nes_lib, targets, rays, exact):
    views, rgb, dep = targets
    r = nes_lib.Renderer(precision=nes_lib.PREC_FP32, seed=2, log2_table_size=LOG2T, max_pixels=W * H * 2)
    t = nes_lib.Trainer(r, batch_rays=rays, exact_weight_grads=exact)
    t.set_targets([nes_lib.make_view(*v) for v in views], rgb.data_ptr(), dep.data_ptr())
    return r, t


def _pairs(n, seed):
    rng = np.random.default_rng(seed)
    return np.stack([rng.integers(0, 2, n), rng.integers(0, W * H, n)], 1).astype(np.int32)


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64))


@pytest.mark.parametrize("exact", [0, 1])
def test_batch_beyond_the_sample_list_is_the_mean_of_its_quarters(nes_lib, targets, exact):
    n = 1 << 18
    r, t = _trainer(nes_lib, targets, n, exact)
    pairs = _pairs(n, 3)
    loss, gt, gw = t.grad(pairs, TABLE_FLOATS)
    samples = t.last_samples()
    assert samples > 1 << 26
    parts = []
    count = 0
    for h in np.split(pairs, 4):
        parts.append(t.grad(h, TABLE_FLOATS))
        assert t.last_samples() <= 1 << 26
        count += t.last_samples()
    t.close()
    r.close()
    assert count == samples
    assert abs(loss - np.mean([p[0] for p in parts])) <= 1e-5 * loss
    for whole, k in ((gt, 1), (gw, 2)):
        assert _rel(whole, np.mean([p[k].astype(np.float64) for p in parts], 0)) <= 1e-4


@pytest.mark.parametrize("n", [1, 31, 33, 129, 255, 257])
def test_ray_counts_around_a_block(nes_lib, targets, n):
    pairs = _pairs(n, n)
    got = {}
    for exact in (0, 1):
        r, t = _trainer(nes_lib, targets, 300, exact)
        got[exact] = t.grad(pairs, TABLE_FLOATS) + (t.last_samples(),)
        t.close()
        r.close()
    (l0, t0, w0, s0), (l1, t1, w1, s1) = got[0], got[1]
    assert s0 == s1 > 0
    assert abs(l0 - l1) <= 1e-5 * l1
    for a, b in ((t0, t1), (w0, w1)):
        assert _rel(a, b) <= 3e-2
        assert np.abs(a.astype(np.float64) - b).max() <= 0.25 * np.abs(b).max()
