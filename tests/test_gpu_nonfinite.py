"""A camera whose value at one pixel is infinite is left out of that pixel's
average and weights, as one with a very large finite value is: alpha and the
port weights have the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHOT = dict(min_shot=10.0, scale_shot=0.0)  # the shot-noise step maps infinity to NaN
TOP = float(np.finfo(np.float32).max)
# One coefficient A of a tile (the lowest of the first quadrant) is A cos(9 pi / 32)^2 / 4 at the tile's corner
# before the window is taken out, which divides by 4 sin(pi / 32)^2: 2.6 A there, less than A up to that step
BIG = 0.6 * TOP


@pytest.fixture(scope="module")
def frame(native):
    import gpu_runner as R
    from cases import Case
    fr = R.Frame(Case(128, 96, seed=61, border_mode=1))
    R.convert(fr)
    return fr


def _with(fr, values, call):
    """call() with the CLT of tile 100, colour 0 of camera k replaced by the one coefficient values[k]"""
    from tile_processor_gpu_b200 import api
    clt = [x.clone() for x in fr.clt]
    for k, v in values.items():
        t = clt[k].view(-1, 3, 256)[100, 0]
        t.zero_()
        t[0] = v
    saved, fr.p_clt = fr.p_clt, api.PointerArray(clt)
    try:
        return call()
    finally:
        fr.p_clt = saved


# two cameras of the same infinite value stand beside two of large values far from each other
PAIRS = [({2: BIG}, {2: BIG / 4}), ({2: BIG, 3: BIG}, {2: BIG / 4, 3: -BIG / 4})]


@pytest.mark.parametrize("infinite,finite", PAIRS, ids=["one", "two"])
def test_tiles(frame, infinite, finite):
    import gpu_runner as R
    idx = np.array([(100 << 8) | 0x8F], dtype=np.int32)
    got, want = (_with(frame, v, lambda: R.textures_tiles(frame, idx, keep_weights=1, **SHOT))[0, :8, 0, 0]
                 for v in (infinite, finite))
    assert not np.isfinite(got[0]) and np.isfinite(want).all()
    assert np.array_equal(got[3:], want[3:])


@pytest.mark.parametrize("infinite,finite", PAIRS, ids=["one", "two"])
def test_rgba(frame, infinite, finite):
    import gpu_runner as R
    img = []
    for v in (infinite, finite):
        out, woi, stride, _ = _with(frame, v, lambda: R.rgba(frame, **SHOT))
        img.append(out[:(woi[3] + 1) * 32].reshape(4, -1, stride)[:, 100 // 16 * 8, 100 % 16 * 8])
    assert not np.isfinite(img[0][0]) and np.isfinite(img[1]).all()
    assert img[0][3] == img[1][3]


@pytest.mark.parametrize("on_chip", [False, True])
def test_one_call_frame(frame, on_chip):
    """Camera 2 sees white noise and its kernel around the middle of the frame is one coefficient, as large as an
    infinite value needs (at a tile's corner, as above)"""
    import torch
    import gpu_runner as R
    from tile_processor_gpu_b200 import api
    fr, c = frame, frame.case
    cx, cy = c.tasks["xy"][100][2]
    kidx = (int(np.rint(cx / 16 + 1)) + int(np.rint(cy / 16 + 1)) * (c.W // 16 + 2)) * 3

    def kernels(value):
        k = [x.clone() for x in fr.kernels]
        t = k[2].view(-1, 256)[kidx]
        t.zero_()
        t[0] = value
        return api.PointerArray(k)

    # the un-windowed values per unit of the coefficient (large: the other tiles' values do not matter)
    unit = 2.0 ** 20
    keep = fr.p_kernels, fr.p_clt, fr.p_images
    saved = [x.clone() for x in fr.clt]
    noise = torch.randn(fr.images[2].shape, generator=torch.Generator().manual_seed(62)).cuda()
    images = api.PointerArray([noise if k == 2 else x for k, x in enumerate(fr.images)])
    fr.p_kernels, fr.p_images = kernels(unit), images
    R.convert(fr)
    fr.p_clt = api.PointerArray([fr.clt[2]] * 4)
    plain = R.textures_tiles(fr, c.tex_idx, **SHOT)[:, 0].astype(np.float64)
    top = float(fr.clt[2].abs().max()) / unit
    fr.p_kernels, fr.p_clt, fr.p_images = keep
    for a, b in zip(fr.clt, saved):
        a.copy_(b)
    w = np.sin(np.pi * (2 * np.arange(16) + 1) / 32) ** 2
    t = np.abs(plain / w[:, None] / w[None, :]) / unit
    n, r, col = np.unravel_index(np.argmax(t), t.shape)
    assert r in (0, 15)
    big = 1.1 * TOP / t.max()
    assert big * top < 0.6 * TOP
    stride = (c.TX + 1) * 8
    y, x = int(c.tex_idx[n] >> 8) // c.TX * 8 + r, int(c.tex_idx[n] >> 8) % c.TX * 8 + col
    img = []
    for value in (big, big / 4):
        ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
        corrs = torch.zeros((c.num_tiles, 6, 225), device="cuda")
        rgba = torch.zeros((4, (c.TY + 1) * 8, stride), device="cuda")
        clt = api.PointerArray([torch.zeros_like(x) for x in fr.clt]) if on_chip else None
        api.process_frame(fr.g, fr.p_extra, kernels(value), images, c.dstride, api.tasks_to_device(c.tasks),
                          c.num_tiles, corrs, 225, fr.port_offsets, *ints, stride, rgba, fat_zero=0.05, gpu_clt=clt,
                          **SHOT)
        img.append(rgba[:, y, x].cpu().numpy())
    assert not np.isfinite(img[0][0]) and np.isfinite(img[1]).all()
    assert img[0][3] == img[1][3]
