"""RenderedFrame payloads below and above the size up to which a frame is
written straight into pinned host memory (512 KiB), and at pixel counts that
leave a tail after the 4-element words: bytes equal to the quantised device
render, and the call's sample count its own."""
import numpy as np
import pytest

from test_wire_gpu import decode_rendered_frame, frame_request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (5, 7), (33, 31), (362, 362), (363, 362), (481, 275)])
def test_payload(nes_lib, cuda, oracle_mod, w, h):
    M = nes_lib.shell_poses(3, 1, 1.5, 1.5)[0]
    r = nes_lib.Renderer(seed=1, log2_table_size=14, max_pixels=w * h)
    rgb = cuda.empty(w * h * 3, device="cuda")
    dep = cuda.empty(w * h, device="cuda")
    r.render_views([nes_lib.make_view(M, w, h, nes_lib.focal_from_fov(w, r.cfg.fov_deg))], [rgb.data_ptr()],
                   [dep.data_ptr()])
    cuda.cuda.synchronize()
    samples = r.last_sample_count()
    for _ in range(2):
        out = decode_rendered_frame(r.render(frame_request(5, False, w, h, M)))
        assert r.last_sample_count() == samples
        assert np.array_equal(np.frombuffer(out[6], np.uint8), oracle_mod.rgb_to_rgb24(rgb.cpu().numpy()))
        assert np.array_equal(np.frombuffer(out[7], np.uint8),
                              oracle_mod.depth_to_gray8(dep.cpu().numpy(), r.cfg.depth_gray_max))
    r.close()
