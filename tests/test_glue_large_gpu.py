"""The frame glue's paths for inputs that fill the chip: YUV conversion in
16-pixel words (77,824 threads of 16 x 2 pixels and more: 1.25 M pixels a
launch) at widths and heights around a word's edges, single and batched, and
depth packing with four groups per thread (1,245,184 elements and more) around a
block's share of 4,096, aligned and not: bytes equal to the oracle's, the rows'
padding untouched.  An image of more 2 x 2 blocks than one launch numbers
(2^31) goes in bands of rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planes(torch, ls, h):
    ch = (h + 1) // 2
    return [torch.full((k,), 7, dtype=torch.uint8, device="cuda") for k in (ls[0] * h, ls[1] * ch, ls[2] * ch)]


def _check(planes, ref, ls, w):
    for p, r, s, pw in zip(planes, ref, ls, (w, (w + 1) // 2, (w + 1) // 2)):
        got = p.cpu().numpy().reshape(-1, s)
        assert np.array_equal(got[:, :pw], np.asarray(r).reshape(-1, s)[:, :pw])
        assert np.all(got[:, pw:] == 7)


@pytest.mark.parametrize("gray", [False, True])
@pytest.mark.parametrize("w,h", [(1840, 1361), (1841, 1361), (1855, 1362), (1856, 1363)])
def test_sixteen_pixel_words_at_the_edges(cuda, nes_lib, oracle_mod, gray, w, h):
    torch = cuda
    rng = np.random.default_rng([w, h])
    src_ls = -(-(w if gray else 3 * w) // 16) * 16
    buf = rng.integers(0, 256, (h, src_ls), dtype=np.uint8)
    ls = nes_lib.linesizes(w)
    src, planes = torch.from_numpy(buf.reshape(-1)).cuda(), _planes(torch, ls, h)
    fn = nes_lib.gray8_to_yuv420p if gray else nes_lib.rgb24_to_yuv420p
    fn(src.data_ptr(), w, h, src_ls, *[p.data_ptr() for p in planes], ls)
    torch.cuda.synchronize()
    _check(planes, (oracle_mod.gray8_to_yuv420p if gray else oracle_mod.rgb24_to_yuv420p)(buf, w, h, src_ls, ls), ls, w)


@pytest.mark.parametrize("gray", [False, True])
@pytest.mark.parametrize("w,h", [(157, 303), (175, 302)])
def test_sixteen_pixel_words_of_a_batch(cuda, nes_lib, oracle_mod, gray, w, h):
    torch = cuda
    n = 64
    rng = np.random.default_rng([w, h])
    src_ls = -(-(w if gray else 3 * w) // 16) * 16
    buf = rng.integers(0, 256, (n, h, src_ls), dtype=np.uint8)
    ls = nes_lib.linesizes(w)
    src = [torch.from_numpy(b.reshape(-1)).cuda() for b in buf]
    planes = [_planes(torch, ls, h) for _ in range(n)]
    nes_lib.yuv420p_batch([s.data_ptr() for s in src], w, h, src_ls, *[[p[k].data_ptr() for p in planes]
                                                                       for k in range(3)], ls, gray=gray)
    torch.cuda.synchronize()
    for b, p in zip(buf, planes):
        _check(p, (oracle_mod.gray8_to_yuv420p if gray else oracle_mod.rgb24_to_yuv420p)(b, w, h, src_ls, ls), ls, w)


@pytest.mark.parametrize("extra", [0, 1, 3, 4095, 4097])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("frames", [1, 3])
def test_four_groups_of_depths(cuda, nes_lib, oracle_mod, extra, offset, frames):
    torch = cuda
    n = 1245184 + extra
    rng = np.random.default_rng([extra, offset])
    x = rng.uniform(-1.0, 70.0, (frames, n)).astype(np.float32)
    src = torch.zeros((frames, n + 8 - n % 8 + 8), device="cuda")
    src[:, offset:offset + n] = torch.from_numpy(x).cuda()
    out = torch.zeros(src.shape, dtype=torch.int16, device="cuda")
    ins, outs = [s.data_ptr() + 4 * offset for s in src], [o.data_ptr() + 2 * offset for o in out]
    if frames == 1:
        nes_lib.depth_pack_u16mm(ins[0], n, outs[0])
    else:
        nes_lib.depth_pack_u16mm_batch(ins, n, outs)
    torch.cuda.synchronize()
    got = out.cpu().numpy().view(np.uint16)
    for g, f in zip(got, x):
        assert np.array_equal(g[offset:offset + n], oracle_mod.depth_pack_u16mm(f))
        assert not g[:offset].any() and not g[offset + n:].any()


def test_image_in_bands(cuda, nes_lib, oracle_mod):
    torch = cuda
    w, h = 65540, 131070  # 32,770 x 65,535 blocks of 2 x 2: a band of 65,531 rows of blocks and one of 4
    src_ls, ls, ch, cw = w + 1, [w + 1, w // 2 + 1, w // 2 + 1], h // 2, w // 2
    table = oracle_mod.gray8_to_yuv420p(np.arange(256, dtype=np.uint8).reshape(1, 256), 256, 1, 256, [256, 128, 128])[0]
    table = torch.from_numpy(np.asarray(table)[:256].copy()).cuda()
    gen = torch.Generator(device="cuda").manual_seed(3)
    src = torch.randint(0, 256, (h, src_ls), dtype=torch.uint8, device="cuda", generator=gen)
    y, u, v = (torch.full((rows, s), 7, dtype=torch.uint8, device="cuda") for rows, s in zip((h, ch, ch), ls))
    nes_lib.gray8_to_yuv420p(src.data_ptr(), w, h, src_ls, y.data_ptr(), u.data_ptr(), v.data_ptr(), ls)
    for r in range(0, h, 1024):
        assert torch.equal(y[r:r + 1024, :w], table[src[r:r + 1024, :w].int()])
    assert (y[:, w:] == 7).all()
    for p in (u, v):
        assert (p[:, :cw] == 128).all() and (p[:, cw:] == 7).all()


def test_taller_images_are_refused(cuda, nes_lib):
    p = cuda.zeros(1 << 20, dtype=cuda.uint8, device="cuda").data_ptr()
    for fn in (nes_lib.rgb24_to_yuv420p, nes_lib.gray8_to_yuv420p):
        with pytest.raises(nes_lib.NesError):
            fn(p, 1, 131071, 3, p, p, p, [1, 1, 1])
