"""Networks with bf16 tiles that have convolutions or ReLUs keep one order of additions for every sum of a step: the sums against the same order
written out in numpy or asked for explicitly, to the bit, and every layer of a step at a large batch against 64 bits."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _ordered_colsum(d):
    """Slabs of 32 columns' rows; eight row lanes of four sums each, added up pairwise, then lane by lane, then slab by slab."""
    M, N = d.shape
    gx = -(-N // 32)
    n = max(1, min(-(-M // 128), -(-4 * 148 // gx), (1 << 21) // (gx * 32))) if gx <= 1024 else 1
    rows = -(-(-(-M // n)) // 8) * 8
    total, slabs = np.zeros(N, np.float32), -(-M // rows)
    for c in range(slabs):
        m0, m1 = c * rows, min(M, (c + 1) * rows)
        t = np.zeros(N, np.float32)
        for lane in range(8):
            a, m = np.zeros((4, N), np.float32), m0 + lane
            while m + 24 < m1:
                a += d[m:m + 32:8]
                m += 32
            for r in range(m, m1, 8):
                a[0] += d[r]
            t = t + ((a[0] + a[1]) + (a[2] + a[3]))
        if slabs == 1:
            return t
        total = total + t
    return total


@pytest.mark.parametrize("M,N", [(1, 1), (9, 8), (33, 10), (127, 33), (128, 32), (160, 40), (257, 128), (2048, 136), (5001, 16), (70000, 40), (512, 8192)])
def test_bias_sums_of_bf16_matrices(M, N):
    from oxidized_neural_orchestra_b200.ops import elementwise as ew

    torch.manual_seed(0)
    d = torch.zeros(M, -(-N // 8) * 8, device="cuda", dtype=torch.bfloat16)[:, :N]
    d.copy_(torch.randn(M, N))
    want = _ordered_colsum(d.float().cpu().numpy())
    base = torch.randn(N, device="cuda")
    for _ in range(2):      # the slab counters are left as they were found
        one, two = base.clone(), base.clone()
        ew.colsum(d, one)
        ew.colsum_jobs([(d, two, 0.0), (d, torch.empty_like(base), 0.0)])
        assert np.array_equal(one.cpu().numpy(), want) and np.array_equal(two.cpu().numpy(), want)
    acc = base.clone()
    ew.colsum(d, acc, beta=1.0)
    assert np.array_equal(acc.cpu().numpy(), base.cpu().numpy() + want)


@pytest.mark.parametrize("B,H,W,K,S,P,filters", [(3, 12, 12, 3, 1, 1, 32), (600, 6, 7, 3, 1, 1, 8), (2, 28, 28, 5, 1, 2, 6), (5, 20, 37, 5, 2, 0, 20),
                                                 (4, 9, 13, 3, 2, 1, 33), (601, 5, 5, 3, 1, 0, 5), (2, 17, 16, 3, 3, 1, 64)])
def test_one_channel_weight_gradient_of_bf16(B, H, W, K, S, P, filters):
    from oxidized_neural_orchestra_b200.ops import conv as cv

    torch.manual_seed(1)
    g = cv.geom(B, 1, H, W, K, S, P)
    OH, OW, F_ = g.OH, g.OW, filters
    x = torch.randn(B * H * W, 1, device="cuda").to(torch.bfloat16)
    dy = torch.zeros(B * OH * OW, -(-F_ // 16) * 16, device="cuda", dtype=torch.bfloat16)
    dy[:, :F_] = torch.randn(B * OH * OW, F_, device="cuda")
    gk, gb = torch.empty(F_ * K * K, device="cuda"), torch.empty(F_, device="cuda")
    cv.conv1_wgrad(g, F_, x, dy, gk, gb)
    xs = np.zeros((B, H + 2 * P + S, W + 2 * P + S), np.float32)
    xs[:, P:P + H, P:P + W] = x.float().cpu().numpy().reshape(B, H, W)
    ds = dy.float().cpu().numpy().reshape(B, OH, OW, -1)[..., :F_]
    nb, groups = min(B, 592), 4 if F_ % 4 == 0 else 1
    acc = np.zeros((nb, 8, groups, F_, K * K + 1), np.float32)      # products of two bf16 values are exact in f32
    for img in range(B):
        for oy in range(OH):
            for ox in range(OW):
                a, dv = acc[img % nb, oy % 8, ox % groups], ds[img, oy, ox]
                a[:, :-1] += dv[:, None] * xs[img, oy * S:oy * S + K, ox * S:ox * S + K].reshape(1, -1)
                a[:, -1] += dv
    v = acc[:, :, 0] if groups == 1 else (acc[:, :, 0] + acc[:, :, 1]) + (acc[:, :, 2] + acc[:, :, 3])
    part = np.zeros(v[:, 0].shape, np.float32)
    for w in range(8):
        part = part + v[:, w]
    lanes = np.zeros((32,) + part.shape[1:], np.float32)
    for b in range(nb):
        lanes[b % 32] += part[b]
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[np.arange(32) ^ o]
    assert np.array_equal(gk.cpu().numpy().reshape(F_, K * K), lanes[0][:, :-1])
    assert np.array_equal(gb.cpu().numpy(), lanes[0][:, -1])


LAYERS = [
    dict(kind="conv", input_dim=[1, 28, 28], kernel_dim=[32, 1, 3], stride=1, padding=1, act=("relu", 0.0)),
    dict(kind="conv", input_dim=[32, 28, 28], kernel_dim=[64, 32, 3], stride=2, padding=1, act=("relu", 0.0)),
    dict(kind="conv", input_dim=[64, 14, 14], kernel_dim=[64, 64, 3], stride=2, padding=1, act=("relu", 0.0)),
    dict(kind="dense", **{"in": 3136, "out": 128}, act=("relu", 0.0)),
    dict(kind="dense", **{"in": 128, "out": 10}, act=("softmax", 0.0)),
]


def _engine(B):
    from oxidized_neural_orchestra_b200.models.conv_engine import ConvNetEngine
    from oxidized_neural_orchestra_b200.models.engine import layer_param_count

    torch.manual_seed(2)
    n = sum(layer_param_count(l) for l in LAYERS)
    npad = (n + 15) // 16 * 16
    params, off = torch.zeros(npad, device="cuda"), 0
    for l in LAYERS:
        fan = l["in"] if l["kind"] == "dense" else l["kernel_dim"][1] * l["kernel_dim"][2] ** 2
        params[off:off + layer_param_count(l)] = torch.randn(layer_param_count(l), device="cuda") * (2.0 / fan) ** 0.5
        off += layer_param_count(l)
    grads = torch.zeros(npad, device="cuda")
    eng = ConvNetEngine(LAYERS, batch_size=B, tile_dtype="bf16", loss="cross_entropy", params=params, grads=grads,
                        params_bf16=params.to(torch.bfloat16))
    eng.refresh()
    x, y = torch.rand(B, 784, device="cuda"), F.one_hot(torch.randint(0, 10, (B,), device="cuda"), 10).float()
    eng.step(x, y, B)
    torch.cuda.synchronize()
    assert eng.status.item() == 0
    return eng, grads


@pytest.mark.parametrize("B", [40, 384])
def test_products_of_a_step_keep_their_order(B):
    from oxidized_neural_orchestra_b200.ops import conv as cv
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    eng, grads = _engine(B)
    de, kw = eng.dense, dict(status=eng.status, cluster=-1)
    sms, kb = torch.cuda.get_device_properties(0).multi_processor_count, 49      # k-blocks of 3136 values
    # the first dense layer: one chain of additions from 256 rows on, below that as many splits as fill the SMs
    again = torch.zeros_like(de.a[1])
    gemm(de.a[0][:B, :3136], de.w_k[0], b_mn_major=True, bias=de.b_view(0), act="relu", out_bf16=again,
         split_k=1 if B >= 256 else min(kb // 4, sms), **kw)
    assert torch.equal(again[:, :128], de.a[1][:, :128])
    gw = torch.zeros(3136, 128, device="cuda")
    gemm(de.a[0][:B, :3136], de.d[1][:B, :128], a_mn_major=True, b_mn_major=True, out=gw, split_k=1, **kw)
    assert torch.equal(gw, de.gw_view(0))
    for j, tiles in ((1, 3), (2, 5)):
        d = eng.front[j]
        M = B * d["OH"] * d["OW"]
        tmp, gk = torch.zeros_like(d["gk_tmp"]), torch.zeros(64 * d["ckk"], device="cuda")
        gemm(d["dy"][:M, :64], d["cols"][:M, :d["ckk"]], a_mn_major=True, b_mn_major=True, out=tmp[:, :d["ckk"]],
             split_k=min(-(-M // 64), -(-sms // tiles)), bn=128, **kw)
        cv.operand_grad_to_kernel(64, d["C"], 3, tmp[:, :d["ckk"]], gk)
        assert torch.equal(gk, grads[d["off"]:d["off"] + 64 * d["ckk"]])
    torch.cuda.synchronize()
    assert eng.status.item() == 0


def _rounded(got, want, mag, K):
    """``got`` is ``want`` rounded once to bf16 (8 significant bits: half a unit is at most 2^-8 of the value) after K / 8 f32 additions, each off by at most 2^-23 of the sum of magnitudes."""
    bound = 2.0 ** -8 * want.abs() * 1.01 + K / 8 * 2.0 ** -23 * mag + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


def test_every_layer_of_a_large_batch_against_64_bits():
    """Each stored activation, delta and gradient from the engine's own stored inputs of that layer."""
    B = 384
    eng, grads = _engine(B)
    de, f = eng.dense, eng.front
    img = lambda t, d, c: t[:, :c].double().view(B, d["OH"], d["OW"], c).permute(0, 3, 1, 2)
    for j in (1, 2):
        d, p = f[j], f[j - 1]
        k = d["kop"].double().view(64, 3, 3, d["C"]).permute(0, 3, 1, 2)
        x, b, M, ckk = img(p["y"], p, d["C"]), eng._kb_view(d).double(), B * d["OH"] * d["OW"], d["ckk"]
        z, mag = F.conv2d(x, k, b, 2, 1), F.conv2d(x.abs(), k.abs(), b.abs(), 2, 1)
        _rounded(img(d["y"], d, 64), torch.relu(z), mag, ckk)
        dy = d["dy"][:M, :64].double()
        # the input gradient, through the derivative below: columns of 64 f32 products, each rounded once to bf16 (to either side of where
        # it may have been before that), then folded in f32
        kop = d["kop"].double()
        exact, off = dy @ kop, 64 / 8 * 2.0 ** -23 * (dy.abs() @ kop.abs())
        fold = lambda c: F.fold(c.to(torch.bfloat16).double().view(B, -1, 9, d["C"]).permute(0, 3, 2, 1).reshape(B, ckk, -1), (d["H"], d["W"]), 3, stride=2, padding=1)
        on = (x > 0).double()
        lo, hi, mag = fold(exact - off) * on, fold(exact + off) * on, fold(exact.abs() + off) * on
        slack = 2.0 ** -8 * torch.maximum(lo.abs(), hi.abs()) * 1.01 + 4 * 2.0 ** -24 * mag + 1e-30
        got = img(p["dy"], p, d["C"])
        assert bool((got >= lo - slack).all()) and bool((got <= hi + slack).all())
        assert (exact - off).to(torch.bfloat16).eq((exact + off).to(torch.bfloat16)).double().mean() > 0.99
        c = d["cols"][:M, :ckk].double()
        gk, gm = dy.t() @ c, dy.abs().t() @ c.abs()
        got = grads[d["off"]:d["off"] + 64 * ckk].double().view(64, d["C"], 9).permute(0, 2, 1).reshape(64, ckk)
        assert bool(((got - gk).abs() <= M / 8 * 2.0 ** -23 * gm).all())
        gb = grads[d["off"] + 64 * ckk:d["off"] + d["n"]].double()
        assert bool(((gb - dy.sum(0)).abs() <= M * 2.0 ** -24 * dy.abs().sum(0)).all())
    d = f[0]
    x, dy = eng.xflat.double().view(B, 1, 28, 28), img(d["dy"], d, 32)
    k = eng._k_view(d).double().view(32, 1, 3, 3)
    b = eng._kb_view(d).double()
    _rounded(img(d["y"], d, 32), torch.relu(F.conv2d(x, k, b, 1, 1)), F.conv2d(x.abs(), k.abs(), b.abs(), 1, 1), 80)
    w = lambda a, c: torch.einsum("bktp,bfp->fkt", F.unfold(a, 3, padding=1).view(B, 1, 9, -1), c.reshape(B, 32, -1)).reshape(32, 9)
    assert bool(((grads[:288].double().view(32, 9) - w(x, dy)).abs() <= B * 784 * 2.0 ** -24 * w(x.abs(), dy.abs())).all())
    a0, a1 = de.a[0][:, :3136].double(), de.a[1][:, :128].double()
    w0, w1 = de.w_k[0].double(), de.w_k[1].double()
    _rounded(de.a[1][:, :128], torch.relu(a0 @ w0 + de.b_view(0).double()), a0.abs() @ w0.abs() + de.b_view(0).double().abs(), 3136)
    d1, d2 = de.d[1][:, :128].double(), de.d[2][:, :10].double()
    _rounded(de.d[1][:, :128], d2 @ w1.t() * (a1 > 0), d2.abs() @ w1.abs().t(), 16)
    _rounded(de.d[0][:, :3136], d1 @ w0.t(), d1.abs() @ w0.abs().t(), 128)
    assert bool(((de.gw_view(0).double() - a0.t() @ d1).abs() <= B / 8 * 2.0 ** -23 * (a0.abs().t() @ d1.abs())).all())


@pytest.mark.parametrize("act,kept", [("relu", True), ("tanh", False)])
@pytest.mark.parametrize("B", [27, 300])
def test_products_of_a_dense_step_keep_their_order(act, kept, B):
    """Unsplit from 256 rows on, below that split as the shape alone says; smooth activations are free to take any form."""
    from oxidized_neural_orchestra_b200.models.engine import GpuEngine
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    torch.manual_seed(4)
    n = 1200 * 640 + 640 + 640 * 16 + 16
    params, grads = torch.randn(n, device="cuda") * 0.03, torch.zeros(n, device="cuda")
    layers = [dict(kind="dense", **{"in": 1200, "out": 640}, act=(act, 0.0 if act == "relu" else 1.0)),
              dict(kind="dense", **{"in": 640, "out": 16}, act=("softmax", 0.0))]
    eng = GpuEngine(layers, batch_size=B, tile_dtype="bf16", loss="cross_entropy", params=params, grads=grads, params_bf16=params.to(torch.bfloat16))
    assert eng.fixed_order is kept
    eng.refresh()
    eng.step(torch.randn(B, 1200, device="cuda"), F.one_hot(torch.randint(0, 16, (B,), device="cuda"), 16).float(), B)
    sms, kb, tiles = torch.cuda.get_device_properties(0).multi_processor_count, 19, -(-B // 128) * 5
    kw, again = dict(status=eng.status, cluster=-1), torch.zeros_like(eng.a[1])
    gemm(eng.a[0][:B, :1200], eng.w_k[0], b_mn_major=True, bias=eng.b_view(0), act=act, act_param=layers[0]["act"][1], out_bf16=again,
         split_k=1 if B >= 256 else min(kb // 4, sms // tiles), **kw)
    gw = torch.zeros(1200, 640, device="cuda")
    gemm(eng.a[0][:B, :1200], eng.d[1][:B, :640], a_mn_major=True, b_mn_major=True, out=gw, split_k=1, **kw)
    torch.cuda.synchronize()
    assert eng.status.item() == 0
    if kept:
        assert torch.equal(again, eng.a[1]) and torch.equal(gw, eng.gw_view(0))
    else:
        assert (again.float() - eng.a[1].float()).abs().max().item() <= 2.0 ** -7
