"""The whole frame in stages through a workspace against the form with the CLT
on chip (same device code): the same correlation bits, the image up to the
order of at most four additions per pixel and pass group."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(case):
    import gpu_runner as R
    return R.Frame(case)


def _run(fr, tasks, radius=7, on_chip=False, short_by=None):
    """one frame; on_chip: a CLT output, which the staged form does not write.  short_by: the C entry with a
    workspace of that many bytes too few; its contents come back too"""
    import torch
    from tile_processor_gpu_b200 import _native, api
    c, n = fr.case, len(tasks)
    sz = (2 * radius + 1) ** 2
    t = api.tasks_to_device(tasks)
    corrs = torch.full((n, 6, sz + 3), -7.0, device="cuda")
    stride = (c.TX + 1) * 8 + 40
    ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
    rgba = torch.full(((c.TY + 1) * 8 * 4 + 8, stride), 3.0, device="cuda")
    ws = None
    if short_by is not None:
        need = _native.call("tp_process_frame_workspace", n)
        ws = torch.full((need - short_by,), 77, dtype=torch.uint8, device="cuda")
        _native.call("tp_process_frame_ws", fr.g.ptr, fr.p_extra.dev.data_ptr(), fr.p_kernels.dev.data_ptr(),
                     fr.p_images.dev.data_ptr(), c.dstride, t.data_ptr(), n, 0, 3, 0.25, 0.25, 0.5, 0.05, radius,
                     sz + 3, corrs.data_ptr(), fr.port_offsets.data_ptr(), 10.0, 3.0, 1.5, 0.294118, 0.117647,
                     0.588235, 1, ints[0].data_ptr(), ints[1].data_ptr(), ints[2].data_ptr(), stride,
                     rgba.data_ptr(), None, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    else:
        clt = [torch.zeros_like(x) for x in fr.clt] if on_chip else None
        api.process_frame(fr.g, fr.p_extra, fr.p_kernels, fr.p_images, c.dstride, t, n, corrs, sz + 3,
                          fr.port_offsets, *ints, stride, rgba, fat_zero=0.05, corr_radius=radius, gpu_clt=clt)
    torch.cuda.synchronize()
    woi = ints[2].cpu().numpy()
    h, w = (int(woi[3]) + 1) * 8 * 4, (int(woi[2]) + 1) * 8
    return corrs.cpu().numpy(), woi, rgba.cpu().numpy()[:h, :w], ws, t.cpu().numpy()


def _compare(a, b):
    from cases import rel_err
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert rel_err(a[2], b[2]) < 1e-6
    assert np.array_equal(a[4], b[4])


@pytest.mark.parametrize("shape,count", [((32, 32), 1), ((256, 192), 3), ((256, 192), 739), ((256, 192), 768),
                                         ((512, 400), 3200)])
def test_staged_frame_matches_on_chip(native, shape, count):
    """Counts on both sides of the one-colour / three-colour items; pair and texture bits left out at random,
    tasks of nothing, outside the frame and (without texture bits) of a tile that another task has too."""
    from cases import Case
    c = Case(*shape, seed=41, border_mode=1)
    rng = np.random.default_rng(count)
    tasks = c.tasks[:count].copy()
    if count > 3:
        tasks["task"] = np.where(rng.random(count) < 0.7, tasks["task"], tasks["task"] & ~0xF)
        tasks["task"] &= (rng.integers(0, 64, count) << 4) | 0xF
        tasks["task"][5::31] = 0
        tasks["txy"][7::37] = c.TX + (1 << 16)
        tasks["txy"][9::41] = c.TY << 16
        dup = np.arange(11, count, 43)
        tasks["txy"][dup] = tasks["txy"][dup - 3]
        tasks["task"][dup] &= ~0xF
    fr = _frame(c)
    for radius in (7, 2):
        _compare(_run(fr, tasks, radius), _run(fr, tasks, radius, on_chip=True))


def test_staged_frame_in_two_parts(native):
    """A list longer than the workspace's tasks: the image's tiles lie in both parts."""
    from cases import Case
    c = Case(256, 192, seed=42, border_mode=0)
    n = 131072 + 37
    tasks = np.tile(c.tasks, n // len(c.tasks) + 1)[:n].copy()
    tasks["task"] = 0x10  # one pair, no texture
    own = np.random.default_rng(1).permutation(n)[:len(c.tasks)]
    own[:20] = 131072 + np.arange(20)
    own = np.unique(own)
    tasks["txy"][own] = c.tasks["txy"][:len(own)]
    tasks["task"][own] = c.tasks["task"][:len(own)]
    fr = _frame(c)
    _compare(_run(fr, tasks, 1), _run(fr, tasks, 1, on_chip=True))


def test_frame_with_a_short_workspace(native):
    """One byte too few: the frame runs on chip and leaves the workspace alone."""
    from cases import Case
    c = Case(256, 192, seed=43, border_mode=0)
    fr = _frame(c)
    got = _run(fr, c.tasks, short_by=1)
    _compare(got, _run(fr, c.tasks, on_chip=True))
    assert bool((got[3] == 77).all())
    _compare(_run(fr, c.tasks, short_by=0), got)


def test_frames_without_memory_for_the_workspace(native):
    """Frames that find no memory for their workspace run on chip, and only the
    first of them empties torch's cache; once there is memory they run in stages."""
    import torch
    from cases import Case
    from tile_processor_gpu_b200 import _native, api
    gc.collect()
    torch.cuda.empty_cache()  # before the frame's buffers are cut from a block of an earlier test
    c = Case(800, 720, seed=44, border_mode=0)
    n, stride = c.num_tiles, (c.TX + 1) * 8
    need = _native.call("tp_process_frame_workspace", n)
    fr = _frame(c)
    want = _run(fr, c.tasks, on_chip=True)[0][:, :, :225]
    t = api.tasks_to_device(c.tasks)
    corrs = torch.zeros((n, 6, 225), device="cuda")
    ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
    rgba = torch.zeros(((c.TY + 1) * 8 * 4, stride), device="cuda")

    def frame():
        corrs.zero_()
        api.process_frame(fr.g, fr.p_extra, fr.p_kernels, fr.p_images, c.dstride, t, n, corrs, 225, fr.port_offsets,
                          *ints, stride, rgba, fat_zero=0.05)

    def count(what):
        return torch.cuda.memory_stats()[what]

    torch.cuda.empty_cache()
    spare = torch.empty(need // 2, dtype=torch.uint8, device="cuda")
    limit = (torch.cuda.memory_reserved() + (2 << 20)) / torch.cuda.mem_get_info()[1]
    del spare  # in torch's cache, too small for the workspace
    largest = max((b["size"] for seg in torch.cuda.memory_snapshot() for b in seg["blocks"] if b["state"] == "inactive"),
                  default=0)
    assert largest < need
    try:
        torch.cuda.set_per_process_memory_fraction(limit)
        before = count("num_alloc_retries")
        for _ in range(4):
            frame()
        torch.cuda.synchronize()
        assert count("num_alloc_retries") == before + 1
        assert np.array_equal(corrs.cpu().numpy(), want)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    frame()
    assert torch.cuda.max_memory_allocated() - base >= need
    torch.cuda.synchronize()
    assert np.array_equal(corrs.cpu().numpy(), want)


@pytest.mark.parametrize("shape", [(256, 192), (800, 720)])
def test_captured_frame_after_an_eager_one(native, shape):
    """An eager first call (in stages) prepares the kernels of a captured one (on
    chip, without a workspace): the graph's replays, on new images and tasks in
    the same buffers, give the eager call's frames."""
    import torch
    from cases import Case
    from tile_processor_gpu_b200 import api
    cases = [Case(*shape, seed=k, border_mode=1) for k in (45, 46)]
    frs = [_frame(c) for c in cases]
    c, fr, n, stride = cases[0], _frame(cases[0]), cases[0].num_tiles, (cases[0].TX + 1) * 8
    t = api.tasks_to_device(c.tasks)
    corrs = torch.zeros((n, 6, 228), device="cuda")
    ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
    rgba = torch.zeros(((c.TY + 1) * 8 * 4, stride), device="cuda")

    def frame():
        api.process_frame(fr.g, fr.p_extra, fr.p_kernels, fr.p_images, c.dstride, t, n, corrs, 228, fr.port_offsets,
                          *ints, stride, rgba, fat_zero=0.05)

    want = []
    for k in (1, 0):
        _load(fr, t, frs[k], cases[k])
        frame()
        torch.cuda.synchronize()
        want.insert(0, (corrs.cpu().numpy(), ints[2].cpu().numpy(), rgba.cpu().numpy(), None, t.cpu().numpy()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        frame()
    for k in (0, 1, 0):
        _load(fr, t, frs[k], cases[k])
        corrs.zero_()
        rgba.fill_(3.0)
        graph.replay()
        torch.cuda.synchronize()
        _compare((corrs.cpu().numpy(), ints[2].cpu().numpy(), rgba.cpu().numpy(), None, t.cpu().numpy()), want[k])


def _load(fr, t, src, case):
    """another frame's inputs into fr's buffers (kernel tables, offsets, images) and the task tensor"""
    from tile_processor_gpu_b200 import api
    for name in ("images", "kernels", "extra"):
        for a, b in zip(getattr(fr, name), getattr(src, name)):
            if a is not b:
                a.copy_(b)
    t.copy_(api.tasks_to_device(case.tasks))
