"""The work that users of the tile processor have it do, as cases that can be timed and checked.

A case is one call or one short sequence of calls through the public entry points (`api`, `disparity_net`), at
frame sizes from a single 32x32 crop to the full 2592x1936 quad frame.  `kind` names the work:

  frame      one quad-camera frame through the drop-in stages: convert_correct_tiles, correlate2D, generate_RBGA
  convert    the forward CLT with aberration correction alone
  correlate  the pairwise phase correlation alone, on a CLT that is there already
  rgba       texture list and overlapped RGBA image alone, on a CLT that is there already
  tiles      non-overlapped texture tiles with their port weights and rms (what a consumer of single tiles asks for)
  imclt      the inverse CLT of one camera into an image (the check picture of a converted frame)
  process    the whole frame in one call (process_frame)
  precision  the three stages with their transforms on the tensor cores
  disparity  plain fit, features, network inference and fallback on a frame's correlations
  train      one training step of the disparity network: forward, backward, Adam

Scenes are a textured slanted plane seen by four cameras with Poisson-Gaussian noise, pixel values around 0..1;
kernels are anisotropic Gaussian point spreads; task centres are jittered and follow the scene's disparity.
"""
import math

import torch

from tile_processor_gpu_b200 import api, disparity_net

PORTS = ((-0.5, -0.5), (0.5, -0.5), (-0.5, 0.5), (0.5, 0.5))
PAIRS = ((0, 1), (2, 3), (0, 2), (1, 3), (0, 3), (2, 1))
SCALES = (0.25, 0.25, 0.5)
FAT_ZERO = 0.05
WEIGHTS = (0.294118, 0.117647, 0.588235)
MIN_SHOT, SCALE_SHOT, DIFF_SIGMA = 10.0, 3.0, 1.5
ADAM = dict(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8)
ADAM_STEPS = 1000  # steps taken before the timed one: moments of a network in mid-training
MAX_W, MAX_H = 2592, 1936


def _frame(name, kind, w, h, active=1.0, **kw):
    """active: the share of the tiles that have a task (a dense frame, or blobs of interest)"""
    return dict(dict(name=name, kind=kind, width=w, height=h, active=active, radius=7, colors=3, border=0), **kw)


def listed():
    return [
        # a small dense frame: a preview, or a region of interest followed at a high rate; launches and latency count
        _frame("frame_small", "frame", 256, 256),
        # an ordinary frame of odd tile counts, tasks only where something is of interest
        _frame("frame_sparse", "frame", 1608, 1208, active=0.35),
        # the three stages of a full 5-megapixel quad frame, each by itself, as a pipeline with its own
        # work between them calls them
        _frame("convert_full", "convert", MAX_W, MAX_H, lpf=0),
        _frame("correlate_full", "correlate", MAX_W, MAX_H),
        _frame("rgba_full", "rgba", MAX_W, MAX_H),
        # texture tiles with weights and rms for a consumer that does its own blending
        _frame("tiles_weights", "tiles", 1024, 768, keep_weights=1),
        # monochrome (infrared) cameras of a smaller format
        _frame("tiles_mono", "tiles", 640, 512, colors=1, keep_weights=0),
        # the check picture of one camera of a full frame
        _frame("imclt_full", "imclt", MAX_W, MAX_H),
        # the full frame in one call
        _frame("process_full", "process", MAX_W, MAX_H),
        # the tensor-core form of the three stages on an ordinary frame
        _frame("precision_fp16", "precision", 1024, 768, fmt=0),
        # disparity of every tile of a full frame: plain fit, network, fallback
        _frame("disparity_full", "disparity", MAX_W, MAX_H),
        # one training step at the trainer's default batch
        dict(name="train_4096", kind="train", rows=4096),
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "convert", "correlate", "rgba", "tiles", "imclt", "process", "precision",
                       "disparity", "train"])
    if kind == "train":
        return dict(kind=kind, rows=int(round(math.exp(rng.uniform(math.log(64), math.log(8192))))))
    # area over its logarithm, aspect between 1:2 and 2:1, sides multiples of 8
    most = 0.4 if kind == "precision" else 1.0
    area = math.exp(rng.uniform(math.log(32 * 32), math.log(MAX_W * MAX_H * most)))
    aspect = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    w = min(MAX_W, max(32, int(math.sqrt(area * aspect)) // 8 * 8))
    h = min(MAX_H, max(32, int(math.sqrt(area / aspect)) // 8 * 8))
    c = _frame("", kind, w, h, active=rng.choice([1.0, round(rng.uniform(0.05, 1.0), 3)]), border=rng.randint(0, 1))
    del c["name"]
    if kind == "imclt":
        c["active"] = 1.0
    if kind in ("frame", "correlate"):
        c["radius"] = rng.choice([7, 7, rng.randint(2, 6)])
    if kind in ("correlate", "rgba", "tiles"):
        c["colors"] = rng.choice([3, 3, 1])
    if kind == "convert":
        c["lpf"] = rng.choice([0, 7])
    if kind == "tiles":
        c["keep_weights"] = rng.randint(0, 1)
    if kind == "precision":
        c["fmt"] = rng.randint(0, 1)
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _noise(g, n, h, w, scales, weights):
    """n smooth random fields in 0..1"""
    out = 0.0
    for s, k in zip(scales, weights):
        coarse = torch.randn((1, n, h // s + 2, w // s + 2), generator=g, device="cuda")
        out = out + k * torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)[0]
    lo, hi = out.amin((1, 2), keepdim=True), out.amax((1, 2), keepdim=True)
    return (out - lo) / (hi - lo)


def _dct4(k, n):
    return 0.5 * math.cos(math.pi * (2 * k + 1) * (2 * n + 1) / 32)


def _dst4(k, n):
    return 0.5 * math.sin(math.pi * (2 * k + 1) * (2 * n + 1) / 32)


def _dct2(k, n):
    return 0.5 * math.cos(math.pi * (2 * n + 1) * k / 16)


def _dst2(k, n):
    return 0.5 * math.sin(math.pi * (2 * n + 1) * (k + 1) / 16)


def _mat(f):
    return torch.tensor([[f(k, n) for n in range(8)] for k in range(8)], dtype=torch.float64, device="cuda")


def _tiles(case):
    return case["width"] // 8, case["height"] // 8


def _pool(g, count=64):
    """CLT tables of `count` anisotropic Gaussian point spreads, sigma 0.5..1.5 px, [count][4][8][8]"""
    t = torch.arange(-7, 8, device="cuda", dtype=torch.float64)
    y, x = torch.meshgrid(t, t, indexing="ij")
    r = _rand(g, 5, count, 1, 1)
    sx, sy, th, ox, oy = 0.5 + r[0], 0.5 + r[1], math.pi * r[2], 0.5 * r[3] - 0.25, 0.5 * r[4] - 0.25
    xr = (x - ox) * th.cos() + (y - oy) * th.sin()
    yr = (y - oy) * th.cos() - (x - ox) * th.sin()
    p = torch.exp(-0.5 * ((xr / sx) ** 2 + (yr / sy) ** 2))
    p = p / p.sum((1, 2), keepdim=True)
    a = math.pi / 16 * torch.outer(2 * torch.arange(8, device="cuda", dtype=torch.float64) + 1, t)
    cs = (a.cos(), a.sin())
    return torch.stack([torch.einsum("um,kmn,vn->kuv", cs[q >> 1], p, cs[q & 1]) for q in range(4)], 1).float()


def _scene(case, seed):
    """What a frame comes with: images, kernel tables, offsets, tasks, all on the GPU."""
    g = _gen(seed)
    W, H = case["width"], case["height"]
    TX, TY = _tiles(case)
    KH, KV = W // 16 + 2, H // 16 + 2
    rows, dstride = H + 16, W + 64
    # a slanted plane of up to 16 px of disparity
    r = _rand(g, 3).tolist()
    d0, gx, gy = 4 * r[0], 8 * r[1] / W, 4 * r[2] / H
    tex = _noise(g, 3, H + 64, W + 64, (24, 8, 4, 2), (0.6, 0.8, 1.0, 1.0))[None]
    yy, xx = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    red, blue = ((yy & 1) == 0) & ((xx & 1) == 1), ((yy & 1) == 1) & ((xx & 1) == 0)
    d = d0 + gx * xx + gy * yy
    images = []
    for ox, oy in PORTS:
        grid = torch.stack([(xx - d * ox + 32) * (2 / (W + 63)) - 1, (yy - d * oy + 32) * (2 / (H + 63)) - 1], -1)
        c = torch.nn.functional.grid_sample(tex, grid[None].float(), align_corners=True)[0]
        v = torch.where(red, c[0], torch.where(blue, c[1], c[2]))
        v = v + torch.sqrt(0.01 * v) * torch.randn((H, W), generator=g, device="cuda")
        v = v + 0.002 * torch.randn((H, W), generator=g, device="cuda")
        image = torch.rand((rows, dstride), generator=g, device="cuda")
        image[:H, :W] = v
        images.append(image)
    nk = KH * KV * 3
    pool = _pool(g)
    kernels = [pool[torch.randint(0, 64, (nk,), generator=g, device="cuda")].reshape(-1) for _ in range(4)]
    extra = []
    for _ in range(4):
        e = torch.zeros((nk, 8), device="cuda")
        e[:, :2] = torch.randint(-16, 17, (nk, 2), generator=g, device="cuda") / 64
        e[:, 4:] = torch.randint(-40, 41, (nk, 4), generator=g, device="cuda") / 4096
        extra.append(e.reshape(-1))
    # the tiles with a task: all, or the highest of a smooth field (blobs)
    n = max(1, round(case["active"] * TX * TY))
    field = _noise(g, 1, TY, TX, (16, 6), (1.0, 0.5)).reshape(-1)
    tile = torch.sort(torch.argsort(field, stable=True)[TX * TY - n:])[0]
    tx, ty = tile % TX, tile // TX
    rec = torch.zeros((n, 10), dtype=torch.int32, device="cuda")
    rec[:, 0] = 0x3FF
    rec[:, 1] = (tx + (ty << 16)).int()
    cx, cy = (8 * tx + 4).double(), (8 * ty + 4).double()
    dd = d0 + gx * cx + gy * cy + (_rand(g, n) - 0.5)
    xy = torch.zeros((n, 8), device="cuda")
    for k, (ox, oy) in enumerate(PORTS):
        j = _rand(g, 2, n) - 0.5
        xy[:, 2 * k] = torch.round((cx + dd * ox + j[0]) * 256).float() / 256
        xy[:, 2 * k + 1] = torch.round((cy + dd * oy + j[1]) * 256).float() / 256
    rec[:, 2:] = xy.view(torch.int32)
    return dict(images=images, kernels=kernels, extra=extra, tasks=rec, tile=tile, xy=xy, dstride=dstride, rows=rows,
                KH=KH, KV=KV)


def _corr_list(tile):
    """(tile << 8) | pair for the six pairs of every tile"""
    return ((tile[:, None] << 8) | torch.arange(6, device="cuda")).reshape(-1).int().contiguous()


def _clt(case, seed):
    """A frame's CLT as a converted frame leaves it, from the 64-bit form of the forward transform"""
    s = _scene(case, seed)
    return s, [c.float().contiguous() for c in _exact_convert(case, s)]


def _corr_planes(case, seed):
    """Correlation tiles of a frame: a peak at each pair's residual disparity, on noise"""
    g = _gen(seed)
    TX, TY = _tiles(case)
    n = max(1, round(case["active"] * TX * TY))
    field = _noise(g, 1, TY, TX, (16, 6), (1.0, 0.5)).reshape(-1)
    tile = torch.sort(torch.argsort(field, stable=True)[TX * TY - n:])[0]
    rho = (3.0 * (torch.rand((n, 1, 1, 1), generator=g, device="cuda") - 0.5))
    b = torch.tensor([[PORTS[j][0] - PORTS[i][0], PORTS[j][1] - PORTS[i][1]] for i, j in PAIRS], device="cuda")
    t = torch.arange(-7, 8, device="cuda", dtype=torch.float32)
    width = 1.0 + 0.5 * torch.rand((n, 1, 1, 1), generator=g, device="cuda")
    px = torch.exp(-0.5 * ((t.view(1, 1, 1, 15) - rho * b[:, 0].view(1, 6, 1, 1)) / width) ** 2)
    py = torch.exp(-0.5 * ((t.view(1, 1, 15, 1) - rho * b[:, 1].view(1, 6, 1, 1)) / width) ** 2)
    c = (0.3 * px * py).reshape(n * 6, 225)
    c += 0.01 * torch.randn((n * 6, 225), generator=g, device="cuda")
    return tile, c


def _weights(seed):
    """Host weights of the network: He-scaled normal, small biases"""
    g = torch.Generator().manual_seed(seed + 77)
    p = {}
    for k in disparity_net.PARAMS:
        shape = disparity_net.SHAPES[k]
        x = torch.randn(shape, generator=g)
        p[k] = (x * (math.sqrt(2 / shape[0]) if k[0] == "W" else 0.05)).numpy()
    p["W3"] *= 0.1
    return p


def _train_inputs(case, seed):
    g = _gen(seed)
    rows = case["rows"]
    x = 0.1 * torch.randn((rows, 1350), generator=g, device="cuda")
    x[:, 112::225] += torch.rand((rows, 6), generator=g, device="cuda")
    target = 0.3 * torch.randn(rows, generator=g, device="cuda")
    m, v = {}, {}
    for k in disparity_net.PARAMS:
        shape = disparity_net.SHAPES[k]
        m[k] = 1e-3 * torch.randn(shape, generator=g, device="cuda")
        v[k] = 1e-5 * (0.5 + torch.rand(shape, generator=g, device="cuda"))
    return x.contiguous(), target, m, v


def _geometry(case):
    return api.Geometry(case["width"], case["height"], image_rows=case["height"] + 16, border_mode=case["border"])


def _ports():
    return torch.tensor(PORTS, dtype=torch.float32, device="cuda").reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        net = disparity_net.DisparityMLP(_weights(seed))
        x, target, m, v = _train_inputs(case, seed)
        net.m, net.v, net.step_count = m, v, ADAM_STEPS
        return dict(case=case, net=net, x=x, target=target)
    TX, TY = _tiles(case)
    st = dict(case=case, g=_geometry(case), po=_ports())
    if kind == "disparity":
        tile, st["corrs"] = _corr_planes(case, seed)
        st["idx"] = _corr_list(tile)
        st["net"] = disparity_net.DisparityMLP(_weights(seed))
        st["net"].pack()
        zeros = lambda *n: torch.zeros(n, device="cuda")  # noqa: E731
        st.update(disp=zeros(TX * TY), strength=zeros(TX * TY), feat=zeros(TX * TY, disparity_net.TC_LDX),
                  out=zeros(TX * TY, 2), rho=zeros(TX * TY))
        return st
    if kind in ("correlate", "rgba", "tiles", "imclt"):
        s, clt = _clt(case, seed)
    else:
        s = _scene(case, seed)
        clt = None if kind == "process" else [torch.zeros(TX * TY * 768, device="cuda") for _ in range(4)]
    n = s["tile"].numel()
    st.update(n=n, dstride=s["dstride"], tasks=s["tasks"])
    if kind in ("frame", "convert", "process", "precision"):
        st.update(keep=(s["images"], s["kernels"], s["extra"]), images=api.PointerArray(s["images"]),
                  kernels=api.PointerArray(s["kernels"]), extra=api.PointerArray(s["extra"]))
    if clt is not None:
        st.update(clt=clt, p_clt=api.PointerArray(clt))
    if kind in ("frame", "correlate", "process", "precision"):
        st["idx"] = _corr_list(s["tile"])
        st["corrs"] = torch.zeros((6 * n, (2 * case["radius"] + 1) ** 2), device="cuda")
    if kind in ("frame", "rgba", "process", "precision"):
        stride = (TX + 1) * 8
        st.update(stride=stride, rgba=torch.zeros(((TY + 1) * 8 * (case["colors"] + 1), stride), device="cuda"),
                  list=torch.zeros(TX * ((TY + 3) & ~3), dtype=torch.int32, device="cuda"),
                  counts=torch.zeros(8, dtype=torch.int32, device="cuda"),
                  woi=torch.zeros(4, dtype=torch.int32, device="cuda"))
    if kind == "precision":
        st["scratch"] = [torch.zeros(TX * TY * 768, device="cuda") for _ in range(4)]
        st["p_scratch"] = api.PointerArray(st["scratch"])
    if kind == "tiles":
        st["list"] = ((s["tile"] << 8) | 0x80).int().contiguous()
        st["tiles"] = torch.zeros((n, _slices(case), 16, 16), device="cuda")
    if kind == "imclt":
        st["stride"] = case["width"] + 8
        st["rbg"] = torch.zeros((3 * (case["height"] + 8), st["stride"]), device="cuda")
    return st


def _slices(case):
    if case["colors"] == 3:
        return 12 if case["keep_weights"] else 4
    return 8 if case["keep_weights"] else 2


# ---- the work ----------------------------------------------------------------------------------------------------


def _fusion(case, keep_weights=0):
    return (case["colors"], 0, MIN_SHOT, SCALE_SHOT, DIFF_SIGMA, 10.0, 3.0) + WEIGHTS + (1, keep_weights)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "train":
        net, rows = st["net"], case["rows"]
        net.forward(st["x"], rows)
        loss = net.loss_backward(st["x"], rows, st["target"])
        net.adam_step(**ADAM)
        return {"loss": loss, "grads": net.g, "params": net.p}
    g = st["g"]
    TX, TY = _tiles(case)
    if kind == "disparity":
        net, tiles = st["net"], TX * TY
        count = st["idx"].numel()
        api.disparity_fit(g, st["corrs"], 225, 7, count, st["idx"], st["po"], st["disp"], st["strength"])
        disparity_net.features(g, st["corrs"], 225, 7, count, st["idx"], st["feat"],
                               feature_stride=disparity_net.TC_LDX)
        net.infer_tc(st["feat"], tiles, st["out"])
        net.combine(st["disp"], st["out"], tiles, st["rho"])
        return {k: st[k] for k in ("disp", "strength", "feat", "out", "rho")}
    n, r = st["n"], case["radius"]
    size = (2 * r + 1) ** 2
    if kind == "process":
        api.process_frame(g, st["extra"], st["kernels"], st["images"], st["dstride"], st["tasks"], n, st["corrs"],
                          size, st["po"], st["list"], st["counts"], st["woi"], st["stride"], st["rgba"],
                          fat_zero=FAT_ZERO, corr_radius=r)
        return {k: st[k] for k in ("corrs", "rgba", "counts", "woi", "tasks")}
    out = {}
    if kind in ("frame", "convert"):
        api.convert_correct_tiles(g, st["extra"], st["kernels"], st["images"], st["tasks"], st["p_clt"], st["dstride"],
                                  n, case.get("lpf", 0))
        out["clt"] = st["clt"]
    if kind in ("frame", "correlate"):
        api.correlate2D(g, st["p_clt"], case["colors"], *SCALES, FAT_ZERO, 6 * n, st["idx"], size, r, st["corrs"])
        out["corrs"] = st["corrs"]
    if kind in ("frame", "rgba"):
        api.generate_RBGA(g, st["tasks"], n, st["list"], st["counts"], st["woi"], TX, TY, st["p_clt"], st["po"],
                          *_fusion(case), st["stride"], st["rgba"])
        out.update({k: st[k] for k in ("rgba", "counts", "woi", "tasks")})
    if kind == "tiles":
        api.textures_accumulate(g, None, st["p_clt"], n, st["list"], st["po"], *_fusion(case, case["keep_weights"]),
                                0, None, _slices(case) * 256, st["tiles"])
        out["tiles"] = st["tiles"]
    if kind == "imclt":
        api.imclt_rbg_all(g, st["clt"][0], st["rbg"], st["stride"])
        out["rbg"] = st["rbg"]
    if kind == "precision":
        f = case["fmt"]
        api.convert_correct_tiles_tc(g, st["extra"], st["kernels"], st["images"], st["tasks"], st["p_clt"],
                                     st["dstride"], n, 0, fmt=f)
        api.correlate2D_tc(g, st["p_clt"], 3, *SCALES, FAT_ZERO, 6 * n, st["idx"], size, r, st["corrs"], fmt=f)
        api.generate_RBGA_tc(g, st["tasks"], n, st["list"], st["counts"], st["woi"], TX, TY, st["p_clt"], st["po"],
                             *_fusion(case), st["stride"], st["rgba"], st["p_scratch"], fmt=f)
        out.update({k: st[k] for k in ("clt", "corrs", "rgba", "counts", "woi", "tasks")})
    return out


def work(case):
    if case["kind"] == "train":
        rows, params = case["rows"], 1350 * 256 + 256 + 256 * 128 + 128 + 128 * 2 + 2
        macs = rows * (2 * 1350 * 256 + 3 * (256 * 128 + 128 * 2))
        return {"bytes": 4.0 * (rows * 1351 + 8 * params), "flops": 2.0 * macs}
    W, H = case["width"], case["height"]
    TX, TY = _tiles(case)
    n = max(1, round(case["active"] * TX * TY))
    c, size = case["colors"], (2 * case["radius"] + 1) ** 2
    share = n / (TX * TY)
    fetch = share * 16.0 * W * H + min(n * 12, 12 * (W // 16 + 2) * (H // 16 + 2)) * 1056.0 + 40.0 * n
    clt, corrs, image = 12288.0 * n * c / 3, 6.0 * n * (4 + 4 * size), share * 4.0 * (W + 8) * (H + 8) * (c + 1)
    ops = {"convert": 75776.0, "correlate": 92016.0 * c / 3, "texture": 149304.0 * c / 3}  # per tile
    every = sum(ops.values())
    kind = case["kind"]
    if kind == "convert":
        return {"bytes": fetch + clt, "flops": n * ops["convert"]}
    if kind == "correlate":
        return {"bytes": clt + corrs, "flops": n * ops["correlate"]}
    if kind == "rgba":
        return {"bytes": clt + 40.0 * n + image, "flops": n * ops["texture"]}
    if kind == "tiles":
        return {"bytes": clt + 4.0 * n + 1024.0 * n * _slices(case), "flops": n * ops["texture"]}
    if kind == "imclt":
        return {"bytes": 3072.0 * n + 12.0 * (W + 8) * (H + 8), "flops": n * 3 * 9728.0}
    if kind == "process":
        return {"bytes": fetch + corrs + image, "flops": n * every}
    if kind == "disparity":
        return {"bytes": corrs + n * 5400.0 + TX * TY * 5420.0 + 1.6e6,
                "flops": 2.0 * TX * TY * (1350 * 256 + 256 * 128 + 256)}
    return {"bytes": fetch + clt + corrs + image, "flops": n * every}  # frame, precision: the CLT is an output


# ---- the same in 64 bits -----------------------------------------------------------------------------------------


def _rind():
    """window sample -> transform index, and the signs of the cosine and sine branches"""
    idx = [n + 4 if n < 4 else 11 - n if n < 12 else n - 12 for n in range(16)]
    return idx, [1.0 if n < 4 else -1.0 for n in range(16)], [1.0 if n < 12 else -1.0 for n in range(16)]


def _hwin():
    return torch.tensor([math.sin(math.pi * (2 * n + 1) / 32) for n in range(16)], dtype=torch.float64, device="cuda")


def _lpf(which):
    s = (0.9, 0.9, 0.6, 0.4, 0.5, 0.9)[which]
    f = [1 + sum(2 * math.exp(-n * n / (2 * s)) * math.cos(math.pi * n * (2 * u + 1) / 16) for n in range(1, 8))
         for u in range(8)]
    f = torch.tensor(f, dtype=torch.float64, device="cuda") / f[0]
    return (torch.outer(f, f) * 1e8).round().div(1e8).float().double()


def _exact_convert(case, s):
    """The forward CLT of every camera, [tiles * 768] doubles; integer choices from the same 32-bit values"""
    W, H, mode = case["width"], case["height"], case["border"]
    TX, TY = _tiles(case)
    idx, sc, ss = _rind()
    idx = torch.tensor(idx, device="cuda")
    sign_c, sign_s = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (sc, ss))
    win = _hwin()
    quad = torch.cat([win[:8].flip(0), -win[:8]])
    c4, s4 = _mat(_dct4), _mat(_dst4)
    out = []
    for cam in range(4):
        clt = torch.zeros((TX * TY, 3, 4, 8, 8), dtype=torch.float64, device="cuda")
        image = s["images"][cam].reshape(-1)
        table, extra = s["kernels"][cam].reshape(-1, 4, 8, 8), s["extra"][cam].reshape(-1, 8)
        for n0 in range(0, s["tile"].numel(), 16384):
            part = slice(n0, n0 + 16384)
            tile, cx, cy = s["tile"][part], s["xy"][part, 2 * cam], s["xy"][part, 2 * cam + 1]
            kx = torch.round(cx / 16 + 1).long().clamp(0, s["KH"] - 1)
            ky = torch.round(cy / 16 + 1).long().clamp(0, s["KV"] - 1)
            kdx, kdy = (cx - 16 * kx) + 8, (cy - 16 * ky) + 8
            for color in range(3):
                at = (ky * s["KH"] + kx) * 3 + color
                e = extra[at]
                # on dyadic grids: exact in 32 bits in any order
                px = (cx - 8) - (e[:, 0] + e[:, 4] * kdx + e[:, 5] * kdy)
                py = (cy - 8) - (e[:, 1] + e[:, 6] * kdx + e[:, 7] * kdy)
                ix, iy = torch.floor(px + 0.5).long(), torch.floor(py + 0.5).long()
                ix, iy = torch.where(ix < 0, ix & 1, ix), torch.where(iy < 0, iy & 1, iy)
                far = (ix & (1 + W - 10)) if mode == 0 else (ix & 1) + W - 10
                ix, iy = torch.where(ix >= W - 8, far, ix), torch.where(iy >= H - 8, (iy & 1) + H - 10, iy)
                hx, hy = (ix - px).double(), (iy - py).double()
                turn = lambda h: win * (math.pi / 16 * h).cos()[:, None] + quad * (math.pi / 16 * h).sin()[:, None]  # noqa: E731,E501
                wh, wv = turn(hx), turn(hy) * sign_c
                whc, whs = wh * sign_c, wh * sign_s
                P = torch.zeros((tile.numel(), 8, 8), dtype=torch.float64, device="cuda")
                Q = torch.zeros_like(P)
                inside = (ix >= 0) & (ix < W - 16) & (iy >= 0) & (iy < H - 16)
                for phase in range(2 if color == 2 else 1):
                    colp = (ix & 1) ^ (1 ^ (color & 1) ^ (color >> 1) ^ phase)
                    rowp = (iy & 1) ^ ((color & 1) ^ phase)
                    two = 2 * torch.arange(8, device="cuda")
                    lr, lc = rowp[:, None] + two, colp[:, None] + two
                    row, col = iy[:, None] + lr, ix[:, None] + lc
                    if mode == 1:
                        row = torch.where(row < 0, row & 1, torch.where(row >= H, H - 2 + (row & 1), row))
                        col = torch.where(col < 0, col & 1, torch.where(col >= W, W - 2 + (col & 1), col))
                        a = row[:, :, None] * s["dstride"] + col[:, None, :]
                    else:
                        a = row[:, :, None] * s["dstride"] + col[:, None, :]
                        ec = 2 * (ix >> 1).clamp(0, H // 2 - 1) + (ix & 1)
                        er = 2 * ((iy >> 1)[:, None] + two // 2).clamp(0, W // 2 - 1) + (iy & 1)[:, None]
                        b = (rowp[:, None] + er)[:, :, None] * s["dstride"] + (ec[:, None] + lc)[:, None, :]
                        a = torch.where(inside[:, None, None], a, b.clamp(0, s["rows"] * s["dstride"] - 1))
                    pix = image[a].double()
                    d = pix * wv.gather(1, lr)[:, :, None]
                    put = idx[lr][:, :, None] * 8 + idx[lc][:, None, :]
                    for m, w in ((P, whc), (Q, whs)):
                        if m is P or color == 2:
                            m.view(-1, 64).scatter_add_(1, put.view(-1, 64),
                                                        (d * w.gather(1, lc)[:, None, :]).view(-1, 64))
                cc = c4 @ P @ c4.T
                if color == 2:
                    sc_ = c4 @ Q @ s4.T
                else:
                    sc_ = (1 - 2 * ((ix & 1) ^ (1 ^ color))).double()[:, None, None] * cc.flip(2)
                neg = (1 - 2 * ((ix & 1) ^ (iy & 1) ^ 1 ^ (color >> 1))).double()[:, None, None]
                cs_, ss_ = neg * sc_.flip(1, 2), neg * cc.flip(1, 2)
                k = table[at].double().unbind(1)
                q0 = cc * k[0] - sc_ * k[1] - cs_ * k[2] + ss_ * k[3]
                q1 = sc_ * k[0] + cc * k[1] - ss_ * k[2] - cs_ * k[3]
                q2 = cs_ * k[0] - ss_ * k[1] + cc * k[2] - sc_ * k[3]
                q3 = ss_ * k[0] + cs_ * k[1] + sc_ * k[2] + cc * k[3]
                odd = math.pi / 16 * (2 * torch.arange(8, device="cuda", dtype=torch.float64) + 1)
                ah, av = (hx[:, None] * odd)[:, None, :], (hy[:, None] * odd)[:, :, None]
                q0, q1 = q0 * ah.cos() - q1 * ah.sin(), q0 * ah.sin() + q1 * ah.cos()
                q2, q3 = q2 * ah.cos() - q3 * ah.sin(), q2 * ah.sin() + q3 * ah.cos()
                q0, q2 = q0 * av.cos() - q2 * av.sin(), q0 * av.sin() + q2 * av.cos()
                q1, q3 = q1 * av.cos() - q3 * av.sin(), q1 * av.sin() + q3 * av.cos()
                q = torch.stack([q0, q1, q2, q3], 1)
                if (case.get("lpf", 0) >> color) & 1:
                    q = q * _lpf(color)
                clt[tile, color] = q
        out.append(clt.reshape(-1))
    return out


def _exact_correlate(case, tile, clt):
    r, size = case["radius"], 2 * case["radius"] + 1
    out = torch.zeros((tile.numel(), 6, size, size), dtype=torch.float64, device="cuda")
    scales = SCALES
    clt = [c.reshape(-1, 3, 4, 64) for c in clt]
    m = (_mat(_dct2), _mat(_dst2))
    for n0 in range(0, tile.numel(), 8192):
        part = slice(n0, n0 + 8192)
        t = [c[tile[part]].double() for c in clt]
        for p, (i, j) in enumerate(PAIRS):
            acc = 0.0
            for color in range(case["colors"]):
                a, b = t[i][:, color].unbind(1), t[j][:, color].unbind(1)
                acc = acc + scales[color] * torch.stack([
                    a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3],
                    a[0] * b[1] - a[1] * b[0] + a[2] * b[3] - a[3] * b[2],
                    a[0] * b[2] - a[2] * b[0] + a[1] * b[3] - a[3] * b[1],
                    a[0] * b[3] + a[3] * b[0] - a[1] * b[2] - a[2] * b[1]], 1)
                if color == 1:
                    acc = acc * _lpf(4).reshape(64)
            acc = acc / torch.sqrt(FAT_ZERO * FAT_ZERO + (acc * acc).sum(1, keepdim=True)) * _lpf(5).reshape(64)
            q = acc.reshape(-1, 4, 8, 8)
            q = [m[k >> 1] @ q[:, k] @ m[k & 1].T for k in range(4)]
            # even and odd halves of the plane, then all four signs of (row, column)
            e = torch.zeros((2, 2, q[0].shape[0], 8, 8), dtype=torch.float64, device="cuda")
            e[0, 0], e[0, 1, :, :, 1:] = q[0], q[1][:, :, :7]
            e[1, 0, :, 1:], e[1, 1, :, 1:, 1:] = q[2][:, :7], q[3][:, :7, :7]
            y = torch.arange(-r, r + 1, device="cuda")
            sg = torch.where(y < 0, -1.0, 1.0).double()
            g = e[:, :, :, y.abs()][:, :, :, :, y.abs()]
            out[part, p] = 0.25 * (g[0, 0] + sg * g[0, 1] + sg[:, None] * (g[1, 0] + sg * g[1, 1]))
    return out.reshape(-1, size * size)


def _imclt(q):
    """[n, 4, 8, 8] -> [n, 16, 16]: inverse CLT, unfolded, without the window"""
    idx, sc, ss = _rind()
    c4, s4 = _mat(_dct4), _mat(_dst4)
    sign = [torch.tensor(v, dtype=torch.float64, device="cuda") for v in (sc, [1.0 if n < 12 else -1.0 for n in range(16)])]
    out = 0.0
    for k in range(4):
        y = (s4 if k >> 1 else c4) @ q[:, k] @ (s4 if k & 1 else c4).T
        out = out + sign[k >> 1][:, None] * sign[k & 1] * y[:, idx][:, :, idx]
    return out


def _exact_textures(case, tile, clt):
    """[n, colors + 1 + 4 + colors + 1, 16, 16]: colours, alpha, port weights, rms"""
    colors = case["colors"]
    win = _hwin()
    w2 = torch.outer(win, win)
    wnd2 = w2 * w2
    clt = [c.reshape(-1, 3, 4, 8, 8) for c in clt]
    chw = torch.tensor(WEIGHTS[:colors], dtype=torch.float64, device="cuda").view(1, -1, 1, 1)
    ks = 1 / (2 * DIFF_SIGMA * DIFF_SIGMA)
    out = []
    for n0 in range(0, tile.numel(), 8192):
        t = tile[n0:n0 + 8192]
        M = torch.stack([torch.stack([_imclt(clt[k][t, c].double() * _lpf(c if colors > 1 else 3)) * (w2 / 4)
                                      for c in range(colors)], 1) for k in range(4)])  # [cam, n, color, 16, 16]
        D = M
        if colors > 1:
            u = M / wnd2
            D = u.clone()
            orth = u[..., :-2, 1:-1] + u[..., 2:, 1:-1] + u[..., 1:-1, :-2] + u[..., 1:-1, 2:]
            diag = u[..., :-2, :-2] + u[..., :-2, 2:] + u[..., 2:, :-2] + u[..., 2:, 2:]
            mid = u[..., 1:-1, 1:-1]
            D[..., 1:-1, 1:-1] = 0.125 * orth + 0.5 * mid
            D[:, :, :2, 1:-1, 1:-1] = (0.0625 * diag + 0.125 * orth + 0.25 * mid)[:, :, :2]
            D = SCALE_SHOT * torch.where(D > MIN_SHOT, D.clamp_min(0).sqrt(), D / math.sqrt(MIN_SHOT)) * wnd2
        mse = ((D - D.mean(0)) ** 2).mean(0)
        N = D / wnd2
        w = torch.zeros((4,) + N.shape[1:2] + (16, 16), dtype=torch.float64, device="cuda")
        for i in range(4):
            for j in range(i + 1, 4):
                far = (PORTS[j][0] - PORTS[i][0]) ** 2 + (PORTS[j][1] - PORTS[i][1]) ** 2
                e = torch.exp(-ks / far * (chw * (N[i] - N[j]) ** 2).sum(1)) + 1e-4
                w[i] += e
                w[j] += e
        best = torch.sort(w, dim=0, descending=True, stable=True)
        p1, p2 = best[0][0], best[0][1]
        w1 = p1 / (p1 + p2)
        pick = lambda k: N.gather(0, best[1][k][None, :, None].expand(1, -1, colors, 16, 16))[0]  # noqa: E731
        avg = w1[:, None] * pick(0) + (1 - w1)[:, None] * pick(1)
        w = torch.exp(-ks * (chw * (N - avg) ** 2).sum(2)) + 1e-4
        worst = w.argmin(0, keepdim=True)
        wv = w.gather(0, worst)[0]
        a = (w.sum(0) - wv) / 3
        w = (w * (1 + wv * (a - wv) / (3 * a * a))).scatter(0, worst, (wv * wv / a)[None])
        ws = w.sum(0)
        rgb = ((w / ws)[:, :, None] * M).sum(0)
        out.append(torch.cat([rgb, (wnd2 * ws / 4)[:, None], w.transpose(0, 1), mse.sqrt(),
                              (chw * mse).sum(1, keepdim=True).sqrt()], 1))
    return torch.cat(out)


def _fade():
    """[16 neighbour masks, 16, 16]"""
    f = [0.5 * (1 - math.cos(math.pi * (i + 0.5) / 16)) for i in range(16)]
    out = torch.ones((16, 16, 16), dtype=torch.float64)
    for i in range(16):
        for j in range(16):
            v = {0: 0.0, 1: f[15 - i], 2: f[j], 4: f[i], 8: f[15 - j], 3: f[j] if j > 15 - i else f[15 - i],
                 6: f[j] if j > i else f[i], 9: f[15 - i] if j > i else f[15 - j],
                 12: f[i] if i > 15 - j else f[15 - j]}
            for k, x in v.items():
                out[k, i, j] = x
    return out.cuda()


def _exact_rgba(case, s, clt):
    TX, TY = _tiles(case)
    tile, colors = s["tile"], case["colors"]
    tx, ty = tile % TX, tile // TX
    there = torch.zeros((TY + 2, TX + 2), dtype=torch.bool, device="cuda")
    there[ty + 1, tx + 1] = True
    nbr = there[ty, tx + 1] * 1 + there[ty + 1, tx + 2] * 2 + there[ty + 2, tx + 1] * 4 + there[ty + 1, tx] * 8
    x0, y0 = int(tx.min()), int(ty.min())
    rows, cols = (int(ty.max()) - y0 + 2) * 8, (TX + 1) * 8
    t = _exact_textures(case, tile, clt)[:, :colors + 1]
    t = t * _fade()[nbr][:, None]
    image = torch.zeros(((TY + 1) * 8 * (colors + 1) * cols,), dtype=torch.float64, device="cuda")
    k = torch.arange(16, device="cuda")
    at = ((ty - y0)[:, None, None] * 8 + k[:, None]) * cols + (tx - x0)[:, None, None] * 8 + k
    for c in range(colors + 1):
        image.index_add_(0, (at + c * rows * cols).reshape(-1), t[:, c].reshape(-1))
    return image.reshape(-1, cols)


def _gelu(z):
    return 0.5 * z * (1 + torch.erf(z / math.sqrt(2)))


def _exact_train(case, seed):
    x, target, m, v = _train_inputs(case, seed)
    x, target = x.double(), target.double()
    p = {k: torch.from_numpy(a).cuda().double().requires_grad_() for k, a in _weights(seed).items()}
    h = _gelu(_gelu(x @ p["W1"] + p["b1"]) @ p["W2"] + p["b2"])
    o = h @ p["W3"] + p["b3"]
    s = o[:, 1].clamp(-12, 12)
    loss = (0.5 * torch.exp(-s) * (o[:, 0] - target) ** 2 + 0.5 * s).mean()
    loss.backward()
    t, new = ADAM_STEPS + 1, {}
    for k in p:
        g = p[k].grad
        mk = ADAM["beta1"] * m[k].double() + (1 - ADAM["beta1"]) * g
        vk = ADAM["beta2"] * v[k].double() + (1 - ADAM["beta2"]) * g * g
        step = mk / (1 - ADAM["beta1"] ** t) / ((vk / (1 - ADAM["beta2"] ** t)).sqrt() + ADAM["eps"])
        new[k] = p[k].detach() - ADAM["lr"] * step
    return {"loss": float(loss), "grads": {k: p[k].grad for k in p}, "params": new}


def _exact_disparity(case, seed):
    TX, TY = _tiles(case)
    tile, corrs = _corr_planes(case, seed)
    c = corrs.double().reshape(-1, 6, 15, 15)
    k = torch.arange(15, device="cuda")
    S = c[:, 0, 7, :] + c[:, 1, 7, :] + c[:, 2, :, 7] + c[:, 3, :, 7] + c[:, 4, k, k] + c[:, 5, 14 - k, k]
    top = S.argmax(1)
    a, b, d = (S.gather(1, (top + t).clamp(0, 14)[:, None])[:, 0] for t in (-1, 0, 1))
    den = a - 2 * b + d
    ok = (top > 0) & (top < 14) & (den < 0)
    off = torch.where(ok, (0.5 * (a - d) / torch.where(ok, den, 1.0)).clamp(-1, 1), 0.0)
    zeros = lambda *n: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    disp, strength, feat = zeros(TX * TY), zeros(TX * TY), zeros(TX * TY, disparity_net.TC_LDX)
    disp[tile], strength[tile] = top - 7 + off, torch.where(ok, b - 0.25 * (a - d) * off, b) / 6
    flat = c.reshape(-1, 1350)
    feat[tile, :1350] = flat / flat.abs().amax(1, keepdim=True)
    p = {n: torch.from_numpy(w).cuda().double() for n, w in _weights(seed).items()}
    out = torch.cat([_gelu(_gelu(f[:, :1350] @ p["W1"] + p["b1"]) @ p["W2"] + p["b2"]) @ p["W3"] + p["b3"]
                     for f in feat.split(8192)])
    return {"disp": disp, "strength": strength, "feat": feat, "out": out, "rho": disp + out[:, 0]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "disparity":
        return _exact_disparity(case, seed)
    if kind in ("correlate", "rgba", "tiles", "imclt"):
        s, clt = _clt(case, seed)
    else:
        s = _scene(case, seed)
        clt = _exact_convert(case, s)
    out = {}
    if kind in ("frame", "convert", "precision"):
        out["clt"] = clt
    if kind in ("frame", "correlate", "process", "precision"):
        out["corrs"] = _exact_correlate(case, s["tile"], clt)
    if kind in ("frame", "rgba", "process", "precision"):
        out["rgba"] = _exact_rgba(case, s, clt)
        out.update(counts=None, woi=None, tasks=None)
    if kind == "tiles":
        out["tiles"] = _exact_textures(case, s["tile"], clt)[:, :_slices(case)].contiguous()
    if kind == "imclt":
        W, H = case["width"], case["height"]
        TX, TY = _tiles(case)
        win = _hwin()
        cell = torch.outer(win, win) / 4
        planes = []
        for c in range(3):
            t = _imclt(clt[0].reshape(-1, 3, 4, 8, 8)[:, c].double()) * cell
            t = t.reshape(TY, TX, 16, 16)
            image = torch.zeros((H + 8, W + 8), dtype=torch.float64, device="cuda")
            for i in range(2):
                for j in range(2):
                    image[8 * i:8 * i + H, 8 * j:8 * j + W] += \
                        t[:, :, 8 * i:8 * i + 8, 8 * j:8 * j + 8].permute(0, 2, 1, 3).reshape(H, W)
            planes.append(image)
        out["rbg"] = torch.cat(planes)
    return out
