"""The marches take several steps of a ray at a time, as many as the number of
rays in the batch asks for (tensor cores: 4, 8 or 32; plain FP32: 8 or 32).  A
ray's samples are composited in one order whatever that number is, so a view's
pixels must not depend on what it is batched with: the same view alone (32
steps), behind a batch of some 40,000 rays (8) and behind one of 160,000 (4 or
8), bit for bit, and the sample counts add up.  Against the oracle: a partial
grid (windows with gaps), an opaque field (rays that end inside a tile) and ray
counts around a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _render(r, torch, nes_lib, views):
    out = [(torch.full((h * w, 3), -1.0, device="cuda"), torch.full((h * w,), -1.0, device="cuda"))
           for _, w, h, _ in views]
    r.render_views([nes_lib.make_view(*v) for v in views], [a.data_ptr() for a, _ in out],
                   [b.data_ptr() for _, b in out])
    torch.cuda.synchronize()
    return [(a.cpu().numpy(), b.cpu().numpy()) for a, b in out], r.last_sample_count()


@pytest.mark.parametrize("field", ["seeded", "partial", "opaque"])
@pytest.mark.parametrize("prec", ["fp32", "tc"])
def test_steps_at_a_time_do_not_change_a_view(nes_lib, oracle_mod, cuda, field, prec):
    poses = nes_lib.shell_poses(21, 4, 1.3, 1.5)
    view = (poses[0], 37, 29, nes_lib.focal_from_fov(37, 80.0))
    inside = [1, 0, 0, .5, 0, -1, 0, .5, 0, 0, -1, .5]  # every ray hits: 40,000 and 160,000 rays
    mid = (inside, 200, 200, nes_lib.focal_from_fov(200, 100.0))
    large = (inside, 400, 400, nes_lib.focal_from_fov(400, 100.0))
    p = nes_lib.PREC_FP32 if prec == "fp32" else nes_lib.PREC_FP16_TC
    with nes_lib.Renderer(precision=p, record_levels=10, max_pixels=200000) as r:
        sc = oracle_mod.Scene(0, 19)
        if field == "partial":
            r.rebuild_occupancy(0.37)
        if field == "opaque":
            w2 = r.scene_param(2, 16 * 64).reshape(16, 64)
            w2[0, :] = 2.0
            r.set_scene_param(2, w2)
            sc.set_param(2, w2)
        occ = r.occupancy()
        ((rgb, dep),), alone = _render(r, cuda, nes_lib, [view])
        for other in (mid, large):
            _, count = _render(r, cuda, nes_lib, [other])
            (_, (rgb2, dep2)), both = _render(r, cuda, nes_lib, [other, view])
            assert np.array_equal(rgb, rgb2) and np.array_equal(dep, dep2)
            assert both == count + alone
    orgb, odep, _ = sc.render(*view, occ=occ)
    assert oracle_mod.psnr(rgb, orgb) >= 45.0
    # The opaque field's bound in FP16 is one march step (its logit weights scale the rounding into sigma).
    assert np.abs(dep - odep).max() <= (oracle_mod.dt() if field == "opaque" and prec == "tc" else 1e-3)
    if field != "opaque":  # FP16: a ray's T may cross the threshold one sample earlier or later
        # The other precision's march visits the same steps (the oracle looks the grid up at FP64 positions, where a
        # step on a cell's border may fall to the other side).
        other = nes_lib.PREC_FP16_TC if prec == "fp32" else nes_lib.PREC_FP32
        with nes_lib.Renderer(precision=other, record_levels=10, max_pixels=37 * 29) as r:
            if field == "partial":
                r.rebuild_occupancy(0.37)
            assert np.array_equal(r.occupancy(), occ)
            assert _render(r, cuda, nes_lib, [view])[1] == alone


@pytest.mark.parametrize("w,h", [(5, 1), (8, 4), (33, 1), (16, 9)])
def test_few_rays_vs_oracle(nes_lib, renderer, cuda, scene0, oracle_mod, w, h):
    view = (nes_lib.shell_poses(5, 2, 1.2, 1.3)[1], w, h, nes_lib.focal_from_fov(w, 60.0))
    ((rgb, dep),), samples = _render(renderer, cuda, nes_lib, [view])
    orgb, odep, osamples = scene0.render(*view)
    assert samples == osamples
    assert oracle_mod.psnr(rgb, orgb) >= 45.0
    assert np.abs(dep - odep).max() <= 1e-3
