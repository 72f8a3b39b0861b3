"""YUV conversion in words of 16, 8 and 2 pixels per thread (by the alignment of
rows and planes) at widths and heights around a word's edges: bytes equal to the
oracle's, the rows' padding untouched.  Depth packing at element counts around a
thread block's share (4,096), aligned and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("align", [16, 8, 1])
@pytest.mark.parametrize("w", [1, 15, 16, 17, 31, 32, 33, 47])
def test_word_edges(cuda, nes_lib, oracle_mod, align, w):
    torch = cuda
    for h in (1, 2, 3):
        for gray in (False, True):
            rng = np.random.default_rng([w, h, align])
            row = w if gray else 3 * w
            src_ls = -(-row // align) * align
            if align == 8 and src_ls % 16 == 0:
                src_ls += 8
            if align == 1 and src_ls % 8 == 0:
                src_ls += 1
            ls, ch, cw = nes_lib.linesizes(w), (h + 1) // 2, (w + 1) // 2
            buf = rng.integers(0, 256, (h, src_ls), dtype=np.uint8)
            src = torch.from_numpy(buf.reshape(-1)).cuda()
            planes = [torch.full((k,), 7, dtype=torch.uint8, device="cuda")
                      for k in (ls[0] * h, ls[1] * ch, ls[2] * ch)]
            fn = nes_lib.gray8_to_yuv420p if gray else nes_lib.rgb24_to_yuv420p
            fn(src.data_ptr(), w, h, src_ls, *[p.data_ptr() for p in planes], ls)
            torch.cuda.synchronize()
            ref = (oracle_mod.gray8_to_yuv420p if gray else oracle_mod.rgb24_to_yuv420p)(buf, w, h, src_ls, ls)
            for p, r, s, pw in zip(planes, ref, ls, (w, cw, cw)):
                got = p.cpu().numpy().reshape(-1, s)
                assert np.array_equal(got[:, :pw], np.asarray(r).reshape(-1, s)[:, :pw])
                assert np.all(got[:, pw:] == 7)


@pytest.mark.parametrize("n", [1, 3, 4095, 4096, 4097, 8195])
@pytest.mark.parametrize("offset", [0, 1])
def test_depth_pack_counts(cuda, nes_lib, oracle_mod, n, offset):
    torch = cuda
    x = np.random.default_rng(n).uniform(-1.0, 70.0, n).astype(np.float32)
    src = torch.zeros(n + 8, device="cuda")
    src[offset:offset + n] = torch.from_numpy(x).cuda()
    out = torch.zeros(n + 8, dtype=torch.int16, device="cuda")
    nes_lib.depth_pack_u16mm(src.data_ptr() + 4 * offset, n, out.data_ptr() + 2 * offset)
    torch.cuda.synchronize()
    got = out.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[offset:offset + n], oracle_mod.depth_pack_u16mm(x))
    assert not got[:offset].any() and not got[offset + n:].any()
