"""Several small jobs in one launch, at the edges of tiles, slabs and of the job table: row jobs give the bits of the jobs one by one,
column sums are held against 64 bits (f32 matrices are cut into other slabs than one by one)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _m(r, c, dt=torch.float32, pad=16, off=0):
    t = torch.zeros(r, (c + pad - 1) // pad * pad + off, device="cuda", dtype=dt)
    t[:, :c + off] = torch.randn(r, c + off, device="cuda")
    return t[:, off:off + c]


@pytest.mark.parametrize("n", [1, 3, 12, 13])
def test_rows_jobs(n):
    from oxidized_neural_orchestra_b200.ops import elementwise as ew

    torch.manual_seed(0)
    shapes = [(1, 1), (33, 65), (64, 64), (256, 320), (300, 257), (257, 300), (1024, 64), (5, 2000)]
    idx = torch.randperm(300, device="cuda").to(torch.int32)
    jobs, again = [], []
    for k in range(n):
        R, W = shapes[k % len(shapes)]
        src = _m(max(R, 300), W)
        j = dict(src=src, n_rows=R, idx=idx if k % 3 == 2 and R <= 300 else None)
        outs = dict(dst=_m(R, W)) if k % 2 else dict(dst_bf16=_m(R, W, torch.bfloat16))
        if k % 4 < 2:
            outs["dst_t"] = _m(W, R)
        jobs.append(dict(j, **outs))
        again.append(dict(j, **{key: torch.zeros_like(v._base)[:, :v.shape[1]] for key, v in outs.items()}))
    zero = torch.full((1,), 3.0, dtype=torch.float64, device="cuda")
    assert ew.rows_jobs(jobs, zero=zero) == (n + 11) // 12
    for j in again:
        ew.rows(**j)
    torch.cuda.synchronize()
    assert zero.item() == 0.0
    for a, b in zip(jobs, again):
        for key in ("dst", "dst_bf16", "dst_t"):
            if key in a:
                assert torch.equal(a[key], b[key])


@pytest.mark.parametrize("n", [1, 5, 13])
def test_colsum_jobs(n):
    from oxidized_neural_orchestra_b200.ops import elementwise as ew

    torch.manual_seed(1)
    shapes = [(1, 1), (33, 10), (200, 1001), (5000, 16), (70000, 40), (512, 8192), (257, 33)]
    jobs, want = [], []
    for k in range(n):
        M, N = shapes[k % len(shapes)]
        d = _m(M, N, torch.bfloat16 if k % 2 else torch.float32, off=1 if k == 4 else 0)      # job 4: rows that are not aligned
        out, beta = torch.randn(N, device="cuda"), (2.0 if k % 3 == 0 else 0.0)
        want.append((beta * out.double() + d.double().sum(0), d.double().abs().sum(0)))
        jobs.append((d, out, beta))
    for _ in range(2):      # the slab counters are left as they were found
        outs = [o.clone() for _, o, _ in jobs]
        ew.colsum_jobs([(d, o, b) for (d, _, b), o in zip(jobs, outs)])
        torch.cuda.synchronize()
        for o, (ref, mag), (d, o0, b) in zip(outs, want, jobs):
            # f32 sums of at most M terms; a tree this shallow stays far below M roundings of the magnitude's sum
            assert bool(((o.double() - ref).abs() <= mag * 2.0 ** -24 * 64 + 1e-6 * (1 + b * o0.double().abs())).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(517, 333, 200), (64, 10, 32), (1000, 1001, 2100)])
@pytest.mark.parametrize("form", [0, -1])
def test_gemm_result_rows_anywhere(dtype, M, N, K, form):
    """A weight gradient inside a flat vector: rows of N values, N no multiple of four, at an odd offset."""
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    torch.manual_seed(2)
    a, b = _m(M, K, dtype), _m(N, K, dtype)
    flat = torch.full((M * N + 8,), 5.0, device="cuda")
    out = flat[3:3 + M * N].view(M, N)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    gemm(a, b, out=out, any_ld=True, cluster=form, status=status)
    once = out.clone()
    gemm(a, b, out=out, any_ld=True, beta=1.0, cluster=form, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0 and bool((flat[:3] == 5.0).all()) and bool((flat[3 + M * N:] == 5.0).all())
    ref = a.double() @ b.double().t()
    bound = K / 8 * 2.0 ** -23 * 4 * K ** 0.5 + 1e-5       # f32 accumulation, one unit of a partial sum below 4 K^0.5 each
    if dtype == torch.float32:                             # operands cut to 10 mantissa bits: the mean shrinkage and its spread
        bound = bound + 2.0 ** -9 * ref.abs() + 2.0 ** -10 * 4 * K ** 0.5
    assert bool(((once.double() - ref).abs() <= bound).all()) and bool(((out.double() - 2 * ref).abs() <= 2.1 * bound).all())
    if N % 4:
        with pytest.raises(RuntimeError):
            gemm(a, b, out=out, cluster=form)
