"""K split over the CTAs of a cluster: every tile width and cluster size against the product in 64 bits, at the edges of tiles,
of the k-blocks and of the output's alignment; the automatic choice against the persistent kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mat(r, c, dt, pad=16):
    t = torch.zeros(r, (c + pad - 1) // pad * pad, device="cuda", dtype=dt)
    t[:, :c] = torch.randn(r, c, device="cuda")
    return t[:, :c]


def _sum_bound(K):
    # K / 8 additions into an f32 accumulator, each off by at most one unit in the last place of a partial sum below 4 K^0.5
    return K / 8 * 2.0 ** -23 * 4 * K ** 0.5


def _close(got, ref, K, dtype):
    # Products are exact for bf16. tf32 cuts each operand to 10 mantissa bits, towards zero: a product shrinks by a share e in
    # [0, 2^-9), so the sum shrinks by the mean share (at most 2^-9 of it) and spreads by 2^-9 / 12^0.5 * 2^0.5 * K^0.5, taken
    # five times over (a million values): 2^-10 * 4 * K^0.5.
    bound = _sum_bound(K) + 1e-5
    if dtype == torch.float32:
        bound = bound + 2.0 ** -9 * ref.abs() + 2.0 ** -10 * 4 * K ** 0.5
    assert bool(((got.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("bn,cluster", [(32, 1), (32, 2), (32, 4), (64, 1), (64, 2), (64, 8), (128, 1), (128, 2), (128, 4), (128, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 1, 257), (33, 129, 520), (130, 67, 1000), (200, 10, 4100)])
def test_cluster_forms(bn, cluster, dtype, shape):
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    M, N, K = shape
    if cluster > -(-K * (4 if dtype == torch.float32 else 2) // 128):
        pytest.skip("more CTAs than k-blocks")
    torch.manual_seed(0)
    a, b = _mat(M, K, dtype), _mat(N, K, dtype)
    bias, aux = torch.randn(N, device="cuda"), _mat(M, N, torch.float32)
    out, out_t, pre = _mat(M, N, torch.float32), _mat(N, M, torch.float32), _mat(M, N, torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = a.double() @ b.double().t()
    gemm(a, b, out=out, out_t=out_t, pre=pre, bias=bias, aux=aux, dact="tanh", dact_param=1.0, bn=bn, cluster=cluster, status=status)
    again = _mat(M, N, torch.float32)
    gemm(a, b, out=again, bias=bias, aux=aux, dact="tanh", dact_param=1.0, bn=bn, cluster=cluster, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(out, again) and torch.equal(out, out_t.t())
    _close(pre, ref + bias.double(), K, dtype)
    want = (ref + bias.double()) * (1 - aux.double() ** 2)
    bound = ((1 - aux.double() ** 2).abs().max() + 1).item()
    _close(out / bound, want / bound, K, dtype)
    if dtype == torch.bfloat16 and bn >= 64:          # MN-major operands, accumulation into the result, a row-padded 16-bit copy
        am, bm = _mat(K, M, dtype), _mat(K, N, dtype)
        gemm(am, bm, a_mn_major=True, b_mn_major=True, out=out, beta=2.0, bn=bn, cluster=cluster, status=status)
        torch.cuda.synchronize()
        assert status.item() == 0
        _close(out - 2.0 * again, am.double().t() @ bm.double(), K, dtype)


def test_cluster_refuses_what_it_cannot_run():
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    a, b, out = _mat(64, 64, torch.bfloat16), _mat(64, 64, torch.bfloat16), _mat(64, 64, torch.float32)
    for kw in (dict(bn=32, cluster=8), dict(bn=256, cluster=2), dict(bn=64, cluster=3), dict(bn=64, cluster=2), dict(bn=64)):
        with pytest.raises(RuntimeError):
            gemm(a, b, out=out, **kw)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(32, 128, 784), (32, 128, 10), (128, 10, 32), (200, 1001, 333), (342, 3136, 128), (513, 100, 2048), (1024, 10, 4096)])
def test_automatic_choice_agrees_with_the_persistent_kernel(dtype, shape):
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    M, N, K = shape
    torch.manual_seed(1)
    a, b = _mat(M, K, dtype), _mat(N, K, dtype)
    x, y = _mat(M, N, torch.float32), _mat(M, N, torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    gemm(a, b, out=x, act="sigmoid", act_param=1.0, status=status)
    gemm(a, b, out=y, act="sigmoid", act_param=1.0, cluster=-1, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0
    # the same products added in another order, through a slope of at most 1/4
    assert (x - y).abs().max().item() <= 2 * _sum_bound(K) / 4 + 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("shape", [(300, 60, 97), (257, 33, 64), (512, 260, 1024), (4000, 320, 128), (700, 1000, 600)])
def test_persistent_tiles_and_pairs_of_the_automatic_choice(dtype, a_mn, b_mn, shape):
    """64-column tiles (rows of 33 to 64), 128- and 256-column ones, single CTAs and pairs: derivative epilogue and plain result."""
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    M, N, K = shape
    torch.manual_seed(3)
    a = _mat(K, M, dtype) if a_mn else _mat(M, K, dtype)
    b = _mat(K, N, dtype) if b_mn else _mat(N, K, dtype)
    aux, bias, status = _mat(M, N, torch.float32), torch.randn(N, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    for pair in (0, -1, 1):
        out, out_t, plain = _mat(M, N, torch.float32), _mat(N, M, torch.float32), _mat(M, N, torch.float32)
        kw = dict(a_mn_major=a_mn, b_mn_major=b_mn, cluster=-1, split_k=1, pair=pair, status=status)
        gemm(a, b, out=plain, **kw)
        gemm(a, b, out=out, out_t=out_t, bias=bias, aux=aux, dact="sigmoid", dact_param=2.0, **kw)
        torch.cuda.synchronize()
        assert status.item() == 0 and torch.equal(out, out_t.t())
        _close(plain, ref, K, dtype)
        slope = aux.double() * (1 - aux.double() / 2)
        scale = slope.abs().max().item() + 1
        _close(out / scale, (ref + bias.double()) * slope / scale, K, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,mn", [((256, 256, 8192), False), ((384, 512, 6400), False), ((256, 1152, 9000), True), ((300, 700, 8200), True)])
def test_long_reductions_on_few_tiles_are_split(dtype, shape, mn):
    """What neither a cluster nor a pair of CTAs should run: the slabs of the two-pass form have been written."""
    from oxidized_neural_orchestra_b200.ops import gemm as G

    M, N, K = shape
    torch.manual_seed(4)
    a = _mat(K, M, dtype) if mn else _mat(M, K, dtype)
    b = _mat(K, N, dtype) if mn else _mat(N, K, dtype)
    ws, out, status = G._workspace(a.device, None), _mat(M, N, torch.float32), torch.zeros(1, dtype=torch.int32, device="cuda")
    ws[:M * N].fill_(float("nan"))
    G.gemm(a, b, a_mn_major=mn, b_mn_major=mn, out=out, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0 and not bool(ws[:M * N].isnan().any())
    _close(out, (a.double().t() if mn else a.double()) @ (b.double() if mn else b.double().t()), K, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(700, 1000, 600), (900, 60, 200), (513, 129, 70), (1300, 20, 40)])
@pytest.mark.parametrize("pair", [-1, 1])
def test_staged_epilogue_over_several_tiles_of_a_cta(dtype, shape, pair):
    """Stored activations are loaded ahead across the output tiles of a CTA: a few CTAs give the bits of one tile per CTA."""
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    M, N, K = shape
    torch.manual_seed(5)
    a, b, aux, bias = _mat(M, K, dtype), _mat(N, K, dtype), _mat(M, N, dtype), torch.randn(N, device="cuda")
    status, got = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for ctas in (0, 2, 6):
        out = _mat(M, N, torch.float32)
        gemm(a, b, out=out, bias=bias, aux=aux, dact="tanh", dact_param=1.0, cluster=-1, split_k=1, pair=pair, max_ctas=ctas, status=status)
        got.append(out)
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    slope = 1 - aux.double() ** 2
    scale = slope.abs().max().item() + 1
    _close(got[0] / scale, (a.double() @ b.double().t() + bias.double()) * slope / scale, K, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bn,cluster", [(32, 1), (32, 4), (64, 2), (64, 8), (128, 1), (128, 8)])
@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("shape", [(33, 129, 520), (130, 67, 1000), (200, 10, 4100)])
def test_cluster_forms_of_operands_as_they_are_stored(dtype, bn, cluster, a_mn, shape):
    """The forward pass of a small step has B MN-major, a weight gradient both; tf32 also with tiles of 32 columns."""
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    if dtype == torch.bfloat16 and bn == 32:
        pytest.skip("one MN-major box of bf16 is 64 wide")
    M, N, K = shape
    torch.manual_seed(6)
    a, b = (_mat(K, M, dtype) if a_mn else _mat(M, K, dtype)), _mat(K, N, dtype)
    out, status = _mat(M, N, torch.float32), torch.zeros(1, dtype=torch.int32, device="cuda")
    gemm(a, b, a_mn_major=a_mn, b_mn_major=True, out=out, bn=bn, cluster=cluster, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0
    _close(out, (a.double().t() if a_mn else a.double()) @ b.double(), K, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, True)])
@pytest.mark.parametrize("shape", [(32, 128, 784), (128, 10, 32), (200, 1001, 333), (342, 3136, 128), (3136, 128, 342), (513, 100, 2048)])
def test_automatic_choice_for_operands_as_they_are_stored(dtype, a_mn, b_mn, shape):
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    M, N, K = shape
    torch.manual_seed(7)
    a, b = (_mat(K, M, dtype) if a_mn else _mat(M, K, dtype)), (_mat(K, N, dtype) if b_mn else _mat(N, K, dtype))
    x, y, status = _mat(M, N, torch.float32), _mat(M, N, torch.float32), torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = dict(a_mn_major=a_mn, b_mn_major=b_mn, act="sigmoid", act_param=1.0, status=status)
    gemm(a, b, out=x, **kw)
    gemm(a, b, out=y, cluster=-1, **kw)
    torch.cuda.synchronize()
    assert status.item() == 0
    # the same products added in another order, through a slope of at most 1/4
    assert (x - y).abs().max().item() <= 2 * _sum_bound(K) / 4 + 1e-6
