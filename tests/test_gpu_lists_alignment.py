"""Ragged lists and unaligned buffers through the stage kernels: entries of one
list do not influence each other, whatever block they share, and the wide
loads' fallbacks give the same bits as the wide loads (exact comparisons)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def frame(native):
    import gpu_runner as R
    from cases import Case
    fr = R.Frame(Case(128, 96, seed=31, border_mode=1))
    R.convert(fr)
    return fr


def _at_offset(tensors, floats):
    """copies whose first element lies `floats` floats past a 256-byte boundary"""
    import torch
    out = []
    for t in tensors:
        x = torch.zeros(t.numel() + 64, dtype=t.dtype, device=t.device)
        y = x[floats:floats + t.numel()]
        y.copy_(t.reshape(-1))
        out.append(y)
    return out


@pytest.mark.parametrize("colors", [1, 3])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9])
def test_texture_entries_are_independent(frame, colors, count):
    """A list of `count` entries, every third one invalid (no texture bit, or a
    tile outside the frame), gives each entry what a list of it alone gives."""
    import gpu_runner as R
    c = frame.case
    rng = np.random.default_rng(count)
    tiles = rng.choice(c.TX * c.TY, count, replace=False)
    idx = ((tiles << 8) | 0x8F).astype(np.int32)
    idx[2::6] &= ~0x80
    idx[5::6] = ((c.TX * c.TY + 3) << 8) | 0x8F
    got = R.textures_tiles(frame, idx, keep_weights=1, colors=colors)
    for i in range(count):
        assert np.array_equal(got[i], R.textures_tiles(frame, idx[i:i + 1], keep_weights=1, colors=colors)[0]), i
    assert np.all(got[2::6] == -7.0) and np.all(got[5::6] == -7.0)


@pytest.mark.parametrize("colors", [1, 3])
@pytest.mark.parametrize("floats", [1, 4])
def test_textures_of_unaligned_clt(frame, colors, floats):
    import gpu_runner as R
    from tile_processor_gpu_b200 import api
    c = frame.case
    want = R.textures_tiles(frame, c.tex_idx, keep_weights=1, colors=colors)
    moved, saved = _at_offset(frame.clt, floats), frame.p_clt
    frame.p_clt = api.PointerArray(moved)
    try:
        got = R.textures_tiles(frame, c.tex_idx, keep_weights=1, colors=colors)
    finally:
        frame.p_clt = saved
    assert np.array_equal(got, want)


@pytest.mark.parametrize("impl", ["rgba", "process"])
@pytest.mark.parametrize("rows,cols", [(1, 12), (12, 1), (3, 3)])
def test_rgba_with_empty_parities(native, oracle, impl, rows, cols):
    """Task lists that leave some of the four tile parities without a tile: the
    image of the passes that have tiles is complete when the call's last
    launch is, and equals the oracle's."""
    import torch
    import gpu_runner as R
    from cases import Case, rel_err
    from tile_processor_gpu_b200 import api
    m = np.zeros((12, 16), dtype=bool)
    m[4:4 + rows, 2:2 + cols] = True
    c = Case(128, 96, seed=32, border_mode=1, mask=m)
    fr = R.Frame(c)
    clt = R.convert(fr)
    if impl == "rgba":
        out, woi, stride, used = R.rgba(fr)
    else:
        stride, used = (c.TX + 1) * 8 + 40, (c.TY + 1) * 8 * 4
        rgba = torch.full((used + 8, stride), 3.0, device="cuda")
        ints = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (c.TX * c.TYA + 256, 8, 4)]
        corrs = torch.zeros((c.num_tiles * 6, 225), device="cuda")
        api.process_frame(fr.g, fr.p_extra, fr.p_kernels, fr.p_images, c.dstride, fr.tasks, c.num_tiles, corrs, 225,
                          fr.port_offsets, *ints, stride, rgba)
        torch.cuda.synchronize()
        out, woi = rgba.cpu().numpy(), ints[2].cpu().numpy()
    want, _, _, _, woi_o = oracle.generate_RBGA(c.geom, c.tasks, c.TX, c.TY, [x.astype(np.float64) for x in clt],
                                                c.port_offsets, stride, used)
    assert np.array_equal(woi, woi_o)
    h, w = (woi[3] + 1) * 8 * 4, (woi[2] + 1) * 8
    assert rel_err(out[:h, :w], want[:h, :w]) < 1e-4


@pytest.mark.parametrize("count", [1, 3, 4, 5, 739, 741, 768])
@pytest.mark.parametrize("floats", [0, 1, 4])
def test_convert_counts_and_alignment(native, oracle, count, floats):
    """Task counts on both sides of the one-colour / three-colour item rule, not
    multiples of the four tasks of an item among them, with the kernel tables,
    images and the CLT on and off 32-byte boundaries: the same bits as the
    one-colour items on aligned buffers give tile by tile, and within 1e-5 of
    the oracle."""
    import torch
    import gpu_runner as R
    from cases import Case, rel_err
    from tile_processor_gpu_b200 import api
    c = Case(256, 192, seed=33, border_mode=0)
    fr = R.Frame(c)
    want = R.convert(fr, num_tiles=count)
    o = oracle.convert_correct_tiles(c.geom, c.extra, c.kernels, c.pitched, c.dstride, c.tasks[:count])
    assert max(rel_err(want[k], o[k]) for k in range(4)) < 1e-5
    for name in ("images", "kernels", "extra", "clt"):
        moved = _at_offset(getattr(fr, name), floats)
        setattr(fr, name, moved)
        setattr(fr, "p_" + name, api.PointerArray(moved))
    got = R.convert(fr, num_tiles=count)
    for k in range(4):
        assert np.array_equal(got[k], want[k]), k
    # the last four tasks alone, as items of one colour
    n = min(4, count)
    saved = fr.tasks
    fr.tasks = saved[count - n:count].contiguous()
    alone = R.convert(fr, num_tiles=n)
    fr.tasks = saved
    for k in range(4):
        assert np.array_equal(alone[k][(count - n) * 768:count * 768], want[k][(count - n) * 768:count * 768]), k
    torch.cuda.synchronize()


@pytest.mark.parametrize("radius,colors", [(7, 3), (7, 1), (3, 3), (0, 3)])
@pytest.mark.parametrize("floats", [1, 4])
def test_correlate_of_unaligned_clt(frame, radius, colors, floats):
    """The narrower loads of a CLT off 32-byte boundaries give the bits of the
    wide ones, in single entries as in the whole list."""
    import gpu_runner as R
    from tile_processor_gpu_b200 import api
    c = frame.case
    want = R.correlate(frame, c.corr_idx, colors=colors, radius=radius)
    moved, saved = _at_offset(frame.clt, floats), frame.p_clt
    frame.p_clt = api.PointerArray(moved)
    try:
        got = R.correlate(frame, c.corr_idx, colors=colors, radius=radius)
        one = R.correlate(frame, c.corr_idx[13:14], colors=colors, radius=radius)
    finally:
        frame.p_clt = saved
    assert np.array_equal(got, want) and np.array_equal(one[0], want[13])


@pytest.mark.parametrize("width,height,marks,floats,pitch", [
    (32, 32, 0, 0, 0), (40, 48, 1, 1, 3), (120, 128, 0, 4, 1), (248, 32, 1, 0, 8), (1304, 904, 1, 0, 5)])
def test_imclt_all_is_the_twelve_passes(native, width, height, marks, floats, pitch):
    """The one-launch image equals the twelve parity passes bit for bit: odd and
    even tile counts, strips and segments of one cell, the debug marks, an
    unaligned CLT, an odd pitch, and an image that held other values before
    (cells that pass (0, 0) does not cover accumulate onto them)."""
    import torch
    from tile_processor_gpu_b200 import api
    g = api.Geometry(width, height, debug_marks=marks)
    gen = torch.Generator(device="cuda").manual_seed(width)
    clt = torch.randn(g.num_tiles * 768, generator=gen, device="cuda")
    clt = _at_offset([clt], floats)[0]
    stride = width + 8 + pitch
    before = torch.randn((3 * (height + 8), stride), generator=gen, device="cuda")
    want, got = before.clone(), before.clone()
    for color in range(3):
        for v in range(2):
            for h in range(2):
                api.imclt_rbg(g, clt, want, color, v, h, stride)
    api.imclt_rbg_all(g, clt, got, stride)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
