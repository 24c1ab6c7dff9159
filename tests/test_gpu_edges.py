"""Edges of the kernels' tiles and of the sizes their launch rules turn on, against the oracle, byte for byte."""
import numpy as np
import pytest
import torch

import zap_b200

pytestmark = pytest.mark.gpu


def _image(w, h, seed):
    """Half smooth, half noise, in a row pitch of its own (as a view when `w` is odd)."""
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[: (h + 1) // 2] = np.sort(img[: (h + 1) // 2], axis=1)
    return img


@pytest.mark.parametrize("size", [(1, 1), (1, 9), (70, 1), (64, 64), (65, 63), (127, 130), (3, 300), (129, 256), (640, 71), (1030, 517)])
@pytest.mark.parametrize("srgb", [0, 1])
def test_mip_chain_edges(cuda_lib, oracle, size, srgb):
    """Chains around the 64x64 tile and the six levels of a launch; 16-byte, 4-byte and 1-byte aligned rows."""
    w, h = size
    for pad in (0, 1):  # pad: the image as a view of wider rows, one texel in
        img = _image(w, h, 10 * w + h + srgb)
        wide = torch.zeros(h, w + 2 * pad, 4, dtype=torch.uint8, device="cuda")
        wide[:, pad:pad + w] = torch.from_numpy(img).cuda()
        view = wide[:, pad:pad + w]
        want, got = img, zap_b200.mip_chain_dev(view, srgb)
        for level in got:
            want = oracle.mip_next(want, srgb)
            assert np.array_equal(level.cpu().numpy(), want), (size, srgb, pad, want.shape)
        if max(w, h) > 1:
            assert np.array_equal(zap_b200.mip_next_dev(view, srgb).cpu().numpy(), oracle.mip_next(img, srgb))


@pytest.mark.parametrize("fmt,channels", [(zap_b200.BC4, 1), (zap_b200.BC5, 2), (zap_b200.BC4, 4), (zap_b200.BC3, 4)])
@pytest.mark.parametrize("size", [(4, 4), (7, 5), (36, 12), (1000, 600)])
def test_channel_blocks(cuda_lib, oracle, fmt, channels, size):
    """Flat blocks, ranges from 1 to 255 levels (palettes with repeated entries below 7), every row alignment."""
    w, h = size
    rng = np.random.default_rng(w + fmt)
    bw, bh = (w + 3) // 4, (h + 3) // 4
    lo = np.kron(rng.integers(0, 256, (bh, bw)), np.ones((4, 4), int))[:h, :w]
    span = np.kron((256.0 ** rng.random((bh, bw))).astype(int) - 1, np.ones((4, 4), int))[:h, :w]
    img = np.zeros((h, w, 4), np.uint8)
    img[..., 3] = 255
    for c in ((0, 1, 3) if channels == 4 else range(channels)):
        img[..., c] = np.clip(lo + (rng.random((h, w)) * (span + 1)).astype(int), 0, 255)
    for x0 in (0, 1):  # a view one texel in: the next alignment down
        sub = np.ascontiguousarray(img[:, x0:])
        t = torch.from_numpy(img[..., :channels].copy()).cuda()[:, x0:]
        if sub.shape[1]:
            assert np.array_equal(zap_b200.bc_encode_dev(t, fmt).cpu().numpy(), oracle.bc_encode(sub, fmt)), (fmt, size, x0)


def test_scratch_pool_across_streams_threads_and_capture(cuda_lib, oracle):
    """Scratch from the context's pool: calls on several streams and threads at once, and a captured call replayed."""
    import threading
    imgs = [_image(64 + 16 * k, 80, 40 + k) for k in range(4)]
    want = [oracle.bc_encode(i, zap_b200.BC7) for i in imgs]
    texs = [torch.from_numpy(i).cuda() for i in imgs]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            outs = [zap_b200.bc_encode_dev(texs[k], zap_b200.BC7) for _ in range(8)]
        s.synchronize()
        bad.extend(k for o in outs if not np.array_equal(o.cpu().numpy(), want[k]))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
    out = torch.zeros(want[0].size, dtype=torch.uint8, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        zap_b200.bc_encode_dev(texs[0], zap_b200.BC7, out=out)
    for _ in range(3):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want[0])


@pytest.mark.parametrize("fmt", [zap_b200.BC1, zap_b200.BC3])
@pytest.mark.parametrize("size", [(1, 1), (4, 4), (13, 6), (64, 20), (252, 260), (640, 592), (640, 596), (1200, 1060)])
def test_colour_blocks_around_the_launch_rule(cuda_lib, oracle, fmt, size):
    """Eight threads per block up to 23680 blocks (160 per SM of 148), one above: both sides of the line, partial CTAs, noise
    (wide channels, long climbs), flat and two-colour blocks."""
    w, h = size
    rng = np.random.default_rng(w * 7 + h + fmt)
    img = _image(w, h, w + h)
    bw, bh = (w + 3) // 4, (h + 3) // 4
    kind = np.kron(rng.integers(0, 4, (bh, bw)), np.ones((4, 4), int))[:h, :w]
    flat = np.kron(rng.integers(0, 256, (bh, bw, 4)), np.ones((4, 4, 1), int))[:h, :w].astype(np.uint8)
    near = (flat.astype(int) + rng.integers(-6, 7, (h, w, 4))).clip(0, 255).astype(np.uint8)
    img = np.where((kind == 1)[..., None], flat, np.where((kind == 2)[..., None], near, img))
    img = np.where(((kind == 3) & (rng.random((h, w)) < 0.5))[..., None], flat, img)
    assert np.array_equal(zap_b200.bc_encode_dev(torch.from_numpy(img).cuda(), fmt).cpu().numpy(), oracle.bc_encode(img, fmt))


def _hard_opaque(w, h, seed, share):
    """An opaque image of which about `share` of the blocks are noise or two far colours (the second searches of ASTC and BC7),
    the rest smooth."""
    rng = np.random.default_rng(seed)
    bw, bh = (w + 3) // 4, (h + 3) // 4
    y, x = np.mgrid[0:h, 0:w]
    img = np.stack([x * 255 // max(w, 2), y * 255 // max(h, 2), (x + y) % 256, np.full((h, w), 255)], 2).astype(np.uint8)
    pick = np.kron(rng.random((bh, bw)) < share, np.ones((4, 4), bool))[:h, :w]
    two = np.kron(rng.random((bh, bw)) < 0.5, np.ones((4, 4), bool))[:h, :w]
    a, b = (np.kron(rng.integers(0, 256, (bh, bw, 3)), np.ones((4, 4, 1), int))[:h, :w] for _ in range(2))
    mix = np.where((rng.random((h, w)) < 0.5)[..., None], a, b)
    noise = rng.integers(0, 256, (h, w, 3))
    img[..., :3] = np.where(pick[..., None], np.where(two[..., None], mix, noise), img[..., :3])
    return img


@pytest.mark.parametrize("size,share", [((4, 4), 1.0), ((21, 13), 1.0), ((64, 64), 0.3), ((136, 136), 1.0), ((140, 140), 1.0),
                                        ((1024, 512), 0.01), ((1024, 512), 0.2)])
@pytest.mark.parametrize("opaque", [True, False])
def test_second_search_around_the_list_rule(cuda_lib, oracle, size, share, opaque):
    """ASTC's two-partition search and BC7's modes 5 and 1, a CTA per listed block while the list has no more blocks than the
    launch CTAs (1184), a group of lanes per block above: lists of one block, on either side of the line, and long ones."""
    w, h = size
    img = _hard_opaque(w, h, w + h, share)
    if not opaque:
        img[..., 3] = np.random.default_rng(3).integers(200, 256, (h, w))
    t = torch.from_numpy(img).cuda()
    assert np.array_equal(zap_b200.astc_encode_dev(t).cpu().numpy(), oracle.astc_encode(img))
    assert np.array_equal(zap_b200.bc_encode_dev(t, zap_b200.BC7).cpu().numpy(), oracle.bc_encode(img, zap_b200.BC7))


@pytest.mark.parametrize("size", [(1, 1), (9, 5), (61, 33), (532, 532), (536, 536), (1500, 1212), (1504, 1212)])
def test_bc7_around_the_launch_rules(cuda_lib, oracle, size):
    """Mode 6 by eight threads per block up to 17760 blocks (120 per SM of 148), in small CTAs up to 113664, in large ones
    above; channels wide enough that their sums are taken in float order, flat blocks and smooth ones in one image."""
    w, h = size
    rng = np.random.default_rng(w + h)
    bw, bh = (w + 3) // 4, (h + 3) // 4
    kind = np.kron(rng.integers(0, 8, (bh, bw)), np.ones((4, 4), int))[:h, :w, None]
    flat = np.kron(rng.integers(0, 256, (bh, bw, 4)), np.ones((4, 4, 1), int))[:h, :w]
    near = flat + rng.integers(-9, 10, (h, w, 4))
    wide = np.where(rng.random((h, w, 4)) < 0.5, flat, 255 - flat)
    img = np.where(kind == 0, wide, np.where(kind == 1, flat, near)).clip(0, 255).astype(np.uint8)
    img[..., 3] = np.where(kind[..., 0] % 3 == 0, 255, img[..., 3])
    assert np.array_equal(zap_b200.bc_encode_dev(torch.from_numpy(img).cuda(), zap_b200.BC7).cpu().numpy(), oracle.bc_encode(img, zap_b200.BC7))


@pytest.mark.parametrize("fmt", [zap_b200.BC1, zap_b200.BC3, zap_b200.BC4, zap_b200.BC5, zap_b200.BC7])
@pytest.mark.parametrize("rdo", [1.0, 30.0, 300.0])
def test_rdo_chains_of_every_short_length(cuda_lib, oracle, fmt, rdo):
    """Chains of 1 to 21 blocks (the loader works four blocks ahead, the window holds 16), and a longer one with repeats, flat
    stretches and noise, so that every candidate kind and match distance wins somewhere."""
    rng = np.random.default_rng(int(rdo) + fmt)
    for n in list(range(1, 22)) + [150]:
        pool = rng.integers(0, 256, (5, 4, 4, 4), dtype=np.uint8)
        pool[0] = pool[0, 0, 0]
        blocks = [pool[rng.integers(0, 5)] if rng.random() < 0.5 else
                  (pool[0].astype(int) + rng.integers(-12, 13, (4, 4, 4))).clip(0, 255).astype(np.uint8) for _ in range(n)]
        img = np.ascontiguousarray(np.concatenate(blocks, axis=1))
        got = zap_b200.bc_encode_rdo_dev(torch.from_numpy(img).cuda(), fmt, rdo)
        assert np.array_equal(got.cpu().numpy(), oracle.bc_encode(img, fmt, rdo=rdo)), (fmt, rdo, n)


@pytest.mark.parametrize("size", [(1, 1), (10, 7), (132, 4), (576, 572), (576, 580)])
@pytest.mark.parametrize("opaque", [True, False])
def test_astc_around_the_launch_rule(cuda_lib, oracle, size, opaque):
    """A warp per trial up to 20720 blocks (140 per SM of 148), one thread for all three above; opaque and transparent blocks in one
    image (they take different configurations), flat, near-flat and wide ones."""
    w, h = size
    rng = np.random.default_rng(w * 3 + h)
    bw, bh = (w + 3) // 4, (h + 3) // 4
    kind = np.kron(rng.integers(0, 5, (bh, bw)), np.ones((4, 4), int))[:h, :w, None]
    flat = np.kron(rng.integers(0, 256, (bh, bw, 4)), np.ones((4, 4, 1), int))[:h, :w]
    img = np.where(kind == 0, flat, np.where(kind == 1, rng.integers(0, 256, (h, w, 4)), flat + rng.integers(-9, 10, (h, w, 4)))).clip(0, 255).astype(np.uint8)
    img[..., 3] = 255 if opaque else np.where(kind[..., 0] % 2 == 0, 255, img[..., 3])
    assert np.array_equal(zap_b200.astc_encode_dev(torch.from_numpy(img).cuda()).cpu().numpy(), oracle.astc_encode(img))


@pytest.mark.parametrize("size", [(1, 1), (5, 6), (66, 20), (688, 688), (688, 692)])
@pytest.mark.parametrize("form", ["rgb16f", "rgba16f", "rgba32f"])
def test_bc6h_around_the_launch_rule(cuda_lib, oracle, size, form):
    """A warp per start up to 29600 blocks (200 per SM of 148), one thread for both above; every input form at full and lesser
    alignment, smooth and wild blocks, negatives, NaN and infinities."""
    w, h = size
    rng = np.random.default_rng(w + h + len(form))
    bw, bh = (w + 3) // 4, (h + 3) // 4
    base = np.kron(2.0 ** rng.uniform(-12, 14, (bh, bw, 3)), np.ones((4, 4, 1)))[:h, :w]
    img = np.ones((h, w, 4), np.float32)
    img[..., :3] = base * (1 + rng.uniform(-0.2, 0.2, (h, w, 3)))
    wild = rng.random((h, w)) < 0.02
    img[wild, 0] = rng.choice(np.array([np.nan, np.inf, -np.inf, -3.0, 0.0, 1e-7, 7e4], np.float32), int(wild.sum()))
    if form != "rgba32f":
        with np.errstate(over="ignore"):
            img = img.astype(np.float16).astype(np.float32)
    want = oracle.bc6h_encode(np.ascontiguousarray(img))
    t = torch.from_numpy(img if form == "rgba32f" else img.astype(np.float16))[..., : 3 if form == "rgb16f" else 4].contiguous().cuda()
    for pad in (0, 1):  # the image one texel into wider rows
        wide = torch.zeros(h, w + 2 * pad, t.shape[2], dtype=t.dtype, device="cuda")
        wide[:, pad:pad + w] = t
        assert np.array_equal(zap_b200.bc6h_encode_dev(wide[:, pad:pad + w]).cpu().numpy(), want), (size, form, pad)
