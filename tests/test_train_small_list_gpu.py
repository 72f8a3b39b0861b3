"""A small trainer lists 512 samples a ray (at least a block of 32 rays), so a
batch of rays along the cube's diagonal, some 1,000 occupied steps each, goes in
parts, whose sample state lies where the backward of the part before has staged
its records.  Loss and gradient equal those of a trainer whose list holds the
batch at once (FP32 sums in another order: relative 1e-5 on the loss, relative L2
1e-4 on the gradients, the bound of FP32 accumulation with atomics)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOG2T = 14
TABLE_FLOATS = 16 * (1 << LOG2T) * 2
W = H = 16


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("n", [33, 64])
def test_parts_of_a_small_batch(nes_lib, cuda, n, exact):
    f = nes_lib.focal_from_fov(W, 2.0)
    view = nes_lib.make_view(nes_lib.look_at((-0.3, -0.3, -0.3)), W, H, f)
    g = cuda.Generator(device="cuda").manual_seed(n)
    rgb = cuda.rand((W * H, 3), device="cuda", generator=g)
    dep = 1.0 + 0.5 * cuda.rand((W * H,), device="cuda", generator=g)
    pairs = np.stack([np.zeros(n), np.random.default_rng(n).integers(0, W * H, n)], 1).astype(np.int32)
    got = {}
    for rays in (n, 4096):  # lists of 32,768 and 2,097,152 samples
        r = nes_lib.Renderer(precision=nes_lib.PREC_FP32, seed=2, log2_table_size=LOG2T, max_pixels=W * H)
        t = nes_lib.Trainer(r, batch_rays=rays, exact_weight_grads=exact)
        t.set_targets([view], rgb.data_ptr(), dep.data_ptr())
        t.grad(pairs, TABLE_FLOATS)
        got[rays] = t.grad(pairs, TABLE_FLOATS) + (t.last_samples(),)
        t.close()
        r.close()
    (l0, t0, w0, s0), (l1, t1, w1, s1) = got[n], got[4096]
    assert s0 == s1 > 512 * n
    assert n == 33 or s0 > 32768
    assert abs(l0 - l1) <= 1e-5 * l1
    for a, b in ((t0, t1), (w0, w1)):
        assert np.linalg.norm(a.astype(np.float64) - b) <= 1e-4 * np.linalg.norm(b)
