"""The one-call training step (tp_mlp_forward, tp_mlp_loss_backward,
tp_mlp_adam_set) and the tensor-core GEMM's roles at the edges of their tiles,
against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


# rows: one, the edges of the 128-row tile and of the head's 16 rows, K ranges of
# the weight gradients from none split to several chunks each
@pytest.mark.parametrize("rows", [1, 15, 17, 127, 128, 129, 300, 1025])
@pytest.mark.parametrize("weighted", [False, True])
def test_step_against_oracle(native, oracle, rows, weighted):
    """Outputs, loss and every gradient within 1e-5 (outputs, loss) and 1e-4
    (gradients) of FP64 relative to the largest magnitude, the bounds of the
    operation-by-operation step; the arrays' elements after Adam within 1e-6."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    rng = np.random.default_rng(rows)
    p = D.init_params(4)
    for k in p:
        if k.startswith("b"):
            p[k] = rng.normal(0, 0.1, p[k].shape).astype(np.float32)
    x = rng.normal(0, 0.3, (rows, D.N_IN)).astype(np.float32)
    t = rng.normal(0, 0.5, rows).astype(np.float32)
    w = (rng.random(rows) > 0.3).astype(np.float32)
    w[0] = 1.0
    net = D.DisparityMLP(p)
    for k in D.PARAMS:
        net.m[k].copy_(_dev(rng.normal(0, 1e-3, D.SHAPES[k])))
        net.v[k].copy_(_dev(rng.uniform(1e-5, 2e-5, D.SHAPES[k])))
    m0, v0 = ({k: d[k].cpu().numpy().astype(np.float64) for k in D.PARAMS} for d in (net.m, net.v))
    xd = _dev(x)
    out = net.forward(xd, rows).cpu().numpy()
    loss = net.loss_backward(xd, rows, _dev(t), weight=_dev(w) if weighted else None)
    net.step_count = 9
    net.adam_step(lr=1e-3)
    torch.cuda.synchronize()
    net.check()
    ref_out, _ = oracle.mlp_forward(p, x.astype(np.float64))
    ref_loss, ref_g = oracle.mlp_loss_and_grads(p, x.astype(np.float64), t.astype(np.float64), w if weighted else None)
    assert np.max(np.abs(out - ref_out)) / np.abs(ref_out).max() < 1e-5
    assert abs(loss - ref_loss) / max(abs(ref_loss), 1e-2) < 1e-5
    for k in D.PARAMS:
        g = net.g[k].cpu().numpy()
        assert np.max(np.abs(g - ref_g[k])) / np.abs(ref_g[k]).max() < 1e-4, k
        g = g.astype(np.float64)
        m, v = 0.9 * m0[k] + 0.1 * g, 0.999 * v0[k] + 0.001 * g * g
        want = p[k] - 1e-3 * (m / (1 - 0.9 ** 10)) / (np.sqrt(v / (1 - 0.999 ** 10)) + 1e-8)
        assert np.max(np.abs(net.p[k].cpu().numpy() - want)) < 1e-6, k


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 63, 31), (129, 65, 33), (128, 64, 160), (5, 130, 64)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad", [0, 1, 2])
def test_gemm_edges(native, M, N, K, ta, tb, pad):
    """Tile, chunk and stage-ring edges, and leading dimensions that allow four,
    two or one value a load, within 1e-5 of FP64; an infinity and a NaN (with
    the payload 0x7fffffff) reach the whole row they belong to and no other."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    rng = np.random.default_rng(M + N + K)
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)

    def put(x, trans):
        x = np.ascontiguousarray(x.T if trans else x)
        y = np.full((x.shape[0], x.shape[1] + pad), 7.0, np.float32)
        y[:, :x.shape[1]] = x
        return _dev(y), y.shape[1]

    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for bad in (None, np.inf, np.uint32(0x7fffffff).view(np.float32)):
        if bad is not None:
            a[0, K // 2] = bad
        A, lda = put(a, ta)
        B, ldb = put(b, tb)
        c = torch.zeros((M, N + pad), device="cuda")
        D.gemm(A, B, c, M, N, K, ta=ta, tb=tb, lda=lda, ldb=ldb, ldc=N + pad, tc=True, err=err)
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        got = c.cpu().numpy()
        assert np.all(got[:, N:] == 0)
        ref = a.astype(np.float64)[1 if bad is not None else 0:] @ b.astype(np.float64)
        rows = got[1 if bad is not None else 0:, :N]
        if ref.size:
            assert np.max(np.abs(rows - ref)) / np.abs(ref).max() < 1e-5
        if bad is not None:
            assert not np.any(np.isfinite(got[0, :N]))


def test_step_on_no_rows(native):
    """A step on an empty batch (tensors without elements have no address): loss
    0 and zero gradients, as a batch that happens to hold no tile gives."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    net = D.DisparityMLP(D.init_params(4))
    x, t = torch.randn((4, D.N_IN), device="cuda"), torch.randn(4, device="cuda")
    net.forward(x, 4)
    net.loss_backward(x, 4, t)
    none = torch.empty((0, D.N_IN), device="cuda")
    assert net.forward(none, 0).shape == (0, 2)
    assert net.loss_backward(none, 0, torch.empty(0, device="cuda")) == 0.0
    torch.cuda.synchronize()
    assert all(not bool(net.g[k].any()) for k in D.PARAMS)


@pytest.mark.parametrize("rows", [1, 17, 200, 224, 1025, 4096, 5000])
def test_step_repeats(native, rows):
    """The loss and the gradients of the biases and of the head repeat bit for
    bit, whatever the order blocks finish in; with up to 224 rows (no product
    splits its K) so does every gradient.  The buffers hold other values
    before each step."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, D.N_IN), generator=gen, device="cuda")
    t = torch.randn(rows, generator=gen, device="cuda")
    net = D.DisparityMLP(D.init_params(4))
    first = None
    for turn in range(30):
        for k in D.PARAMS:
            net.g[k].fill_(float(turn + 1))
        net.forward(x, rows)
        loss = net.loss_backward(x, rows, t)
        got = {k: net.g[k].clone() for k in D.PARAMS}
        if first is None:
            first = loss, got
        assert loss == first[0]
        for k in D.PARAMS:
            if rows <= 224 or k not in ("W1", "W2"):
                assert torch.equal(got[k], first[1][k]), (k, turn)


def test_step_memory_by_form(native):
    """The tensor-core step allocates no gradient of h1 and h2; the FP32 step
    of the same network does when it comes to it, and gives the same gradients."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    gen = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((300, D.N_IN), generator=gen, device="cuda")
    t = torch.randn(300, generator=gen, device="cuda")
    net = D.DisparityMLP(D.init_params(4))
    net.forward(x, 300)
    net.loss_backward(x, 300, t)
    floats = sum(v.numel() for v in net._ws.values() if isinstance(v, torch.Tensor))
    assert floats < 300 * (3 * D.N_H1 + 3 * D.N_H2 + 8) + 64
    got = {k: net.g[k].clone() for k in D.PARAMS}
    net.tc = False
    net.forward(x, 300)
    net.loss_backward(x, 300, t)
    for k in D.PARAMS:
        assert float((net.g[k] - got[k]).abs().max() / got[k].abs().max()) < 1e-4, k


@pytest.mark.parametrize("tc", [True, False])
@pytest.mark.parametrize("raw", [False, True])
def test_step_on_a_given_stream(native, tc, raw):
    """The loss is that of the step, which waits behind other work on the stream
    it was given (a torch stream or its handle)."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((100, D.N_IN), generator=gen, device="cuda")
    t = torch.randn(100, generator=gen, device="cuda")
    net = D.DisparityMLP(D.init_params(4), tc=tc)
    net.forward(x, 100)
    want = net.loss_backward(x, 100, t)
    torch.cuda.synchronize()
    for v in (net._ws["loss"], net._ws.get("loss_sum")):
        if v is not None:
            v.fill_(-1.0)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
    s = side.cuda_stream if raw else side
    net.forward(x, 100, stream=s)
    assert abs(net.loss_backward(x, 100, t, stream=s) - want) <= 1e-6 * abs(want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("rows", [115200, 131072])
def test_column_sums_of_long_batches(native, rows):
    """Batches on both sides of the rule that lays the parts of b1's gradient
    behind the head's, against FP64 sums of the step's own dz1, dz2 and dout
    (relative 1e-5 of the sum of magnitudes, as a sum of that many values in
    128-row parts stays far below)."""
    import torch
    from tile_processor_gpu_b200 import disparity_net as D
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, D.N_IN), generator=gen, device="cuda")
    t = torch.randn(rows, generator=gen, device="cuda")
    net = D.DisparityMLP(D.init_params(4))
    net.forward(x, rows)
    loss = net.loss_backward(x, rows, t)
    net.check()
    w = net._ws
    for k, v in (("b1", w["dz1"]), ("b2", w["dz2"]), ("b3", w["dout"])):
        v = v[:rows].double()
        assert float(((net.g[k].double() - v.sum(0)).abs() / v.abs().sum(0)).max()) < 1e-5, k
    want = float(w["loss"][:rows].double().sum()) / rows
    assert abs(loss - want) <= 1e-12 * abs(want)
    g3 = w["h2"][:rows].double().T @ w["dout"][:rows].double()
    assert float((net.g["W3"].double() - g3).abs().max() / g3.abs().max()) < 1e-5
    for k, a, b in (("W1", x, w["dz1"]), ("W2", w["h1"], w["dz2"])):
        ref = a[:rows].double().T @ b[:rows].double()
        assert float((net.g[k].double() - ref).abs().max() / ref.abs().max()) < 1e-5, k
