"""Samples on the unit cube's far faces, at a coordinate of exactly 1: every
level's cell there is its last one, at fraction 1.

A camera on the face, one float below 1, whose rays rise by 0.6 x 2^-24 over the
cube: FP32 rounds the face's coordinate of each ray's last sixth to 1.  The
same rays without the rise stay below it, 2^-24 away: less than a step of any
level's FP16 fraction (2^-11 of a cell, at most 2,048 cells), so the two renders
agree to the rounding of a few FP16 colour inputs (2e-3); and the first agrees
with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BELOW = 1.0 - 2.0 ** -24
RISE = float(np.float32(0.6 * 2.0 ** -24))
W, H = 16, 12


def _pose(axis, rise):
    b, c = (axis + 1) % 3, (axis + 2) % 3
    m = np.zeros((3, 4))
    m[axis] = [0.0, 0.0, rise, BELOW]
    m[b] = [0.8, 0.0, 0.0, 0.5]
    m[c] = [0.0, 0.3, 1.0, 0.0]
    return m.reshape(-1).tolist()


@pytest.mark.parametrize("prec", ["fp32", "tc"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_coordinate_of_one(nes_lib, oracle_mod, cuda, scene0, request, prec, axis):
    r = request.getfixturevalue("r32" if prec == "fp32" else "rtc")
    f = nes_lib.focal_from_fov(W, 60.0)
    assert np.count_nonzero((BELOW + RISE * np.linspace(0, 1, 101)).astype(np.float32) == 1.0) >= 16
    out = []
    for rise in (RISE, 0.0):
        rgb = cuda.full((H * W, 3), -1.0, device="cuda")
        dep = cuda.full((H * W,), -1.0, device="cuda")
        r.render_views([nes_lib.make_view(_pose(axis, rise), W, H, f)], [rgb.data_ptr()], [dep.data_ptr()])
        cuda.cuda.synchronize()
        out.append((rgb.cpu().numpy(), dep.cpu().numpy(), r.last_sample_count()))
    (rgb, dep, samples), (rgb0, dep0, samples0) = out
    assert samples == samples0 > 100 * W * H
    assert np.abs(rgb - rgb0).max() <= 2e-3
    assert np.abs(dep - dep0).max() <= 1e-3
    orgb, odep, _ = scene0.render(_pose(axis, RISE), W, H, f)
    assert oracle_mod.psnr(rgb, orgb) >= 45.0
    assert np.abs(dep - odep).max() <= 1e-3
