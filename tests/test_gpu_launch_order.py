"""The order in which generate_RBGA_tc's kernels run: the first texture pass
reads the pixel tiles of the tensor-core inverse transform at once, so it must
not be launched as a programmatic dependent of it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(graph):
    """edge types along a captured chain of launches, in launch order (0 complete, 1 programmatic)"""
    cu = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph), ctypes.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(handle, None, None, None, ctypes.byref(n)) == 0
    src, dst = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)()
    data = (ctypes.c_ubyte * (8 * n.value))()  # from port, to port, type, five reserved bytes
    assert cu.cuGraphGetEdges_v2(handle, src, dst, data, ctypes.byref(n)) == 0
    after = {src[i]: (dst[i], data[8 * i + 2]) for i in range(n.value)}
    assert len(after) == n.value  # one successor each
    node = (set(after) - {d for d, _ in after.values()}).pop()
    types = []
    while node in after:
        node, t = after[node]
        types.append(t)
    return types


@pytest.mark.parametrize("fmt", [0, 1])
def test_first_pass_waits_for_the_pixel_tiles(native, fmt):
    """Captured, not run: list -> clear (dependent), clear -> inverse transform
    and inverse transform -> first pass (complete), pass -> pass (dependent)."""
    import torch
    import gpu_runner as R
    from cases import Case
    from tile_processor_gpu_b200 import api
    c = Case(256, 192, seed=51, border_mode=1)
    fr = R.Frame(c)
    # the stage's tables and attributes are set up outside the capture
    R.textures_tiles(fr, c.tex_idx, impl="tc_fp16" if fmt == 0 else "tc_bf16")
    p = R.TEX
    stride = (c.TX + 1) * 8
    out = torch.zeros(((c.TY + 1) * 8 * 4, stride), device="cuda")
    ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        api.generate_RBGA_tc(fr.g, fr.tasks, c.num_tiles, *ints, c.TX, c.TY, fr.p_clt, fr.port_offsets, p["colors"],
                             0, p["min_shot"], p["scale_shot"], p["diff_sigma"], 10.0, 3.0, p["weight0"],
                             p["weight1"], p["weight2"], 1, 0, stride, out, fr.tile_scratch(), fmt=fmt)
    assert _chain(graph.raw_cuda_graph()) == [1, 0, 0, 1, 1, 1]


@pytest.mark.parametrize("impl", ["tc_fp16", "tc_bf16"])
def test_images_back_to_back_share_a_scratch(native, impl):
    """Two frames in turn through the same scratch, without a wait between them:
    each image has the bits of a call alone."""
    import torch
    import gpu_runner as R
    from cases import Case
    from tile_processor_gpu_b200 import api
    c = Case(512, 384, seed=52, border_mode=1)
    fr = R.Frame(c)
    R.convert(fr)
    rng = np.random.default_rng(52)
    clts = [[x.clone() for x in fr.clt], [x * float(rng.uniform(0.5, 2.0)) + 0.25 for x in fr.clt]]
    ptrs = [api.PointerArray(x) for x in clts]
    p, n = R.TEX, c.num_tiles
    stride = (c.TX + 1) * 8
    ints = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (c.TX * c.TYA + 256, 8, 4)]
    tasks = api.tasks_to_device(c.tasks)

    def call(i, out):
        api.generate_RBGA_tc(fr.g, tasks, n, *ints, c.TX, c.TY, ptrs[i], fr.port_offsets, p["colors"], 0,
                             p["min_shot"], p["scale_shot"], p["diff_sigma"], 10.0, 3.0, p["weight0"], p["weight1"],
                             p["weight2"], 1, 0, stride, out, fr.tile_scratch(), fmt=R._tc_fmt(impl))

    image = lambda: torch.zeros(((c.TY + 1) * 8 * 4, stride), device="cuda")  # noqa: E731
    alone = [image(), image()]
    for i in range(2):
        call(i, alone[i])
        torch.cuda.synchronize()
    assert not torch.equal(*alone)
    turns = [image() for _ in range(12)]
    for k, out in enumerate(turns):
        call(k & 1, out)
    torch.cuda.synchronize()
    for k, out in enumerate(turns):
        assert torch.equal(out, alone[k & 1]), k
    assert api.tc_status() == 0
