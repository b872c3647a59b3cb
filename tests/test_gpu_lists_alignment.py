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
def test_textures_do_not_depend_on_the_grid(native, colors):
    """One block per SM or the built-in number: tiles and RGBA image have the
    same bits, whether a block holds one entry or all its mono slots are full
    (lists of 3200 and of a few more entries than blocks)."""
    import gpu_runner as R
    from cases import Case
    from tile_processor_gpu_b200 import autotune
    c = Case(512, 400, seed=36, border_mode=1)
    fr = R.Frame(c)
    R.convert(fr)
    lists = [c.tex_idx, c.tex_idx[:1037], c.tex_idx[:151]]
    got = []
    for cap in (0, 1):
        autotune.set_shape("textures", cap)
        try:
            got.append([R.textures_tiles(fr, idx, keep_weights=1, colors=colors) for idx in lists] +
                       [R.rgba(fr, colors=colors)[0]])
        finally:
            autotune.reset()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    one = [R.textures_tiles(fr, c.tex_idx[k:k + 1], keep_weights=1, colors=colors)[0] for k in (0, 1036, 3199)]
    assert all(np.array_equal(got[0][0][k], x) for k, x in zip((0, 1036, 3199), one))


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


@pytest.mark.parametrize("count", [1, 31, 33, 1024, 8191, 8192, 8193, 12288])
def test_texture_list_lengths(native, oracle, count):
    """Task lists on both sides of the one-kernel rule, shuffled, some without
    texture bits: tasks, counts and window equal the oracle's, each sub-list
    holds the oracle's entries, on buffers that held another list before."""
    import torch
    from tile_processor_gpu_b200 import api, synth
    geom = synth.geometry(1024, 768)
    g = api.Geometry.from_dict(geom)
    TX, TY, TYA = synth.tiles(geom)
    rng = np.random.default_rng(count)
    tasks = synth.tasks_grid(geom, rng)[rng.permutation(TX * TY)][:count].copy()
    tasks["task"][rng.random(count) < 0.1] = 0x3F0
    idx = torch.full((TX * TYA,), 0x7F, dtype=torch.int32, device="cuda")
    counts = torch.full((8,), 5, dtype=torch.int32, device="cuda")
    woi = torch.full((4,), -3, dtype=torch.int32, device="cuda")
    t = api.tasks_to_device(tasks)
    api.prepare_texture_list(g, t, count, idx, counts, woi, TX, TY)
    torch.cuda.synchronize()
    want_t, want_i, want_c, want_w = oracle.prepare_texture_list(geom, tasks, TX, TY)
    assert np.array_equal(api.tasks_from_device(t)["task"], want_t["task"])
    assert np.array_equal(woi.cpu().numpy(), want_w)
    got_c, got_i, q = counts.cpu().numpy(), idx.cpu().numpy(), TX * (TYA >> 2)
    assert np.array_equal(got_c, want_c)
    for s in range(8):
        lo = (s >> 1) * q if not s & 1 else (s >> 1) * q + q - want_c[s]
        assert np.array_equal(np.sort(got_i[lo:lo + want_c[s]]), np.sort(want_i[lo:lo + want_c[s]])), s


@pytest.mark.parametrize("radius", [7, 3])
def test_disparity_runs_across_windows(native, oracle, radius):
    """Runs that straddle the 32-entry windows the fit and the features work
    in: tiles with one to six pairs, pair codes of other kinds between them,
    longer runs of repeated pairs, against the oracle, in any window phase."""
    import torch
    from tile_processor_gpu_b200 import api, disparity_net as D, synth
    geom = synth.geometry(256, 192)
    g = api.Geometry.from_dict(geom)
    tiles = 32 * 24
    rng = np.random.default_rng(radius)
    n2 = (2 * radius + 1) ** 2
    for lead in (0, 1, 5):
        codes = [(tiles - 1 << 8) | (i % 6) for i in range(lead)]
        for tile in range(200):
            pairs = [p for p in range(6) if rng.random() < 0.8] or [2]
            if tile % 17 == 3:
                pairs = pairs + [7]
            if tile % 23 == 5:
                pairs = [i % 6 for i in range(11 + tile % 40)]
            codes += [(tile << 8) | p for p in pairs]
        codes += [(tiles + 3 << 8) | 0]
        idx = np.array(codes, np.int32)
        co = rng.random((len(idx), n2)).astype(np.float32)
        po = torch.from_numpy(synth.PORT_OFFSETS.reshape(-1).copy()).cuda()
        dd, ss = (torch.full((tiles,), np.nan, device="cuda") for _ in range(2))
        feat = torch.full((tiles, 6 * n2 + 2), -5.0, device="cuda")
        dco, didx = torch.from_numpy(co).cuda(), torch.from_numpy(idx).cuda()
        api.disparity_fit(g, dco, n2, radius, len(idx), didx, po, dd, ss)
        D.features(g, dco, n2, radius, len(idx), didx, feat, feature_stride=6 * n2 + 2)
        torch.cuda.synchronize()
        want_d, want_s = oracle.disparity_fit(geom, co, idx, radius)
        got_d, got_s = dd.cpu().numpy(), ss.cpu().numpy()
        assert np.array_equal(np.isnan(got_d), np.isnan(want_d))
        ok = ~np.isnan(want_d)
        assert np.max(np.abs(got_d[ok] - want_d[ok])) < 1e-4 and np.max(np.abs(got_s[ok] - want_s[ok])) < 1e-5
        got = feat.cpu().numpy()
        for tile in list(range(200)) + [tiles - 1]:
            run = [(e, c & 0xFF) for e, c in enumerate(codes) if c >> 8 == tile and (c & 0xFF) < 6]
            row = np.zeros(6 * n2, np.float64)
            for e, p in run:
                row[p * n2:(p + 1) * n2] = co[e]
            if run:
                row /= max(np.abs(co[e]).max() for e, _ in run)
                assert np.max(np.abs(got[tile, :6 * n2] - row)) < 1e-6, tile
        assert np.all(got[:, 6 * n2:] == -5.0) and np.all(got[200:tiles - 1] == -5.0)


@pytest.mark.parametrize("impl", ["tc_fp16", "tc_bf16"])
@pytest.mark.parametrize("floats", [1, 4])
def test_tensor_core_stages_of_unaligned_buffers(native, impl, floats):
    """The precision form on buffers off 32-byte boundaries (kernel tables, CLT,
    tile scratch) gives the bits of aligned ones, stage by stage; entry counts
    that leave a block of 128 rows and a warp's 32 entries part full."""
    import gpu_runner as R
    from cases import Case
    from tile_processor_gpu_b200 import api
    c = Case(128, 96, seed=35, border_mode=1)
    fr, un = R.Frame(c), R.Frame(c)
    for name in ("kernels", "clt"):
        moved = _at_offset(getattr(un, name), floats)
        setattr(un, name, moved)
        setattr(un, "p_" + name, api.PointerArray(moved))
    un.tile_scratch()
    un._tiles = _at_offset(un._tiles, floats)
    un.p_tiles = api.PointerArray(un._tiles)
    for n in (13, c.num_tiles):
        a, b = R.convert(fr, impl=impl, num_tiles=n), R.convert(un, impl=impl, num_tiles=n)
        assert all(np.array_equal(a[k], b[k]) for k in range(4)), n
    idx = c.corr_idx[:333].copy()
    idx[7] = (3 << 8) | 6
    idx[40] = (c.TX * c.TY + 1) << 8
    for radius in (7, 2):
        assert np.array_equal(R.correlate(fr, idx, impl=impl, radius=radius),
                              R.correlate(un, idx, impl=impl, radius=radius))
    for colors in (3, 1):
        assert np.array_equal(R.textures_tiles(fr, c.tex_idx, keep_weights=1, impl=impl, colors=colors),
                              R.textures_tiles(un, c.tex_idx, keep_weights=1, impl=impl, colors=colors))
    assert api.tc_status() == 0
