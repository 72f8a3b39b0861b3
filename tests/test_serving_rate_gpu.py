"""Admission by expected delay under overload with views of very different
sizes: batches of small views finish together with the batch before them, which
must not make the measured service rate look unbounded.  The median latency of
the admitted requests stays within 1.25 times the bound (0.8 measured; a rate
averaged over each batch's own time let it reach 2.3)."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND_MS = 100.0


def test_median_latency_stays_near_the_bound(nes_lib, cuda):
    poses = nes_lib.shell_poses(9, 1000, 1.2, 2.0)
    rng = np.random.default_rng(5)
    kind, gap = rng.integers(0, 4, len(poses)), rng.exponential(1.0 / 360.0, len(poses))
    kinds = [(640, 360, 1), (1280, 720, 1), (1920, 1080, 1), (1920, 1832, 2)]
    queue, lat = [], []
    done = threading.Event()
    with nes_lib.Renderer(precision=nes_lib.PREC_FP16_TC, max_pixels=2 * 1920 * 1832) as r:
        srv = nes_lib.Server(r, max_inflight_batches=2, max_batch_pixels=2 * 1920 * 1832, hbm_budget_bytes=20 << 30,
                             max_pending=16, max_queue_ms=BOUND_MS)

        def collect():
            i = 0
            while i < len(queue) or not done.is_set():
                if i >= len(queue):
                    time.sleep(0.0005)
                    continue
                lat.append(srv.wait(queue[i]).latency_ms)
                srv.release(queue[i])
                i += 1

        t = threading.Thread(target=collect)
        t.start()
        try:
            due = time.perf_counter()
            for i, m in enumerate(poses):
                due += gap[i]
                while time.perf_counter() < due:
                    time.sleep(max(0.0, min(0.001, due - time.perf_counter())))
                w, h, n = kinds[kind[i]]
                f = nes_lib.focal_from_fov(w, 90.0)
                mats = nes_lib.stereo_pair(m, 0.063) if n == 2 else [m]
                ticket = srv.submit([nes_lib.make_view(q, w, h, f) for q in mats])
                if ticket is not None:
                    queue.append(ticket)
        finally:
            done.set()
            t.join()
            srv.close()
    assert len(lat) >= 40
    late = sorted(lat[20:])  # after the first batches have set the rate
    assert late[len(late) // 2] <= 1.25 * BOUND_MS
