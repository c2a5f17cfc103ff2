"""A convolution's input gradient in one kernel: the same bits as the product and the fold as two, for every kind of window and ragged channel count."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B    C   H   W   F   K  S  P
SIZES = [(5, 32, 28, 28, 64, 3, 2, 1), (11, 64, 14, 14, 64, 3, 2, 1), (3, 6, 14, 14, 16, 5, 1, 0), (300, 17, 9, 11, 33, 3, 1, 1), (2, 8, 16, 16, 5, 3, 1, 1),
         (7, 37, 12, 10, 96, 5, 1, 2), (1, 4, 6, 6, 8, 3, 3, 0), (160, 9, 7, 7, 12, 2, 1, 0), (4, 20, 13, 17, 40, 4, 2, 1), (3, 3, 8, 8, 1, 1, 1, 0),
         (2, 16, 31, 29, 24, 5, 2, 2), (9, 1, 5, 5, 7, 5, 1, 4),
         # several images a unit with fewer in the last one, single pixels, units whose chunks are dealt out over a whole number of rounds
         (310, 32, 20, 20, 16, 3, 2, 1), (1000, 4, 1, 1, 8, 1, 1, 0), (200, 48, 16, 16, 8, 3, 1, 1), (501, 8, 6, 6, 12, 3, 1, 0)]


@pytest.mark.parametrize("B,C,H,W,F,K,S,P", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dact", [None, "relu", "tanh"])
def test_same_bits_as_product_and_fold(B, C, H, W, F, K, S, P, dtype, dact):
    from oxidized_neural_orchestra_b200.ops import conv as cv
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    up = lambda n: -(-n // 16) * 16
    torch.manual_seed(0)
    g = cv.geom(B, C, H, W, K, S, P)
    rows, ckk = B * g.OH * g.OW, C * K * K
    mk = lambda r, c: torch.nn.functional.pad(torch.randn(r, c, device="cuda"), (0, up(c) - c)).to(dtype)
    dy, kt, aux = mk(rows, F), mk(ckk, F), mk(B * H * W, C)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    dcols = torch.zeros(rows, up(ckk), device="cuda", dtype=dtype)
    out = {"out" if dtype == torch.float32 else "out_bf16": dcols[:, :ckk]}
    gemm(dy[:, :F], kt[:, :F], split_k=1, cluster=-1, status=status, **out)
    kw = dict(aux=aux, dact=dact, dact_param=0.1 if dact == "relu" else 1.0) if dact else {}
    want = torch.zeros(B * H * W, up(C), device="cuda", dtype=dtype)
    cv.col2im(g, dcols, want, **kw)
    assert cv.dgrad_fits(g, F, dy, kt, want, **({"aux": aux, "dact": dact} if dact else {}))
    store = torch.full((B * H * W + 4, up(C)), 3.0, device="cuda", dtype=dtype)
    got = store[2:-2]
    for _ in range(2):
        cv.dgrad(g, F, dy, kt, got, status=status, **kw)
        assert torch.equal(got[:, :C], want[:, :C])
    assert (store[:2] == 3.0).all() and (store[-2:] == 3.0).all() and status.item() == 0


def test_what_it_does_not_take():
    from oxidized_neural_orchestra_b200.ops import conv as cv

    t = lambda r, c: torch.zeros(r, c, device="cuda")
    assert not cv.dgrad_fits(cv.geom(1, 16, 28, 28, 3, 1, 1), 16, t(784, 16), t(144, 16), t(784, 16))       # more than 256 output pixels
    assert not cv.dgrad_fits(cv.geom(1, 16, 14, 14, 7, 1, 0), 16, t(64, 16), t(784, 16), t(196, 16))        # a 7 x 7 kernel
    assert not cv.dgrad_fits(cv.geom(1, 16, 14, 14, 3, 1, 1), 16, t(196, 16), t(144, 16), t(196, 18)[:, 2:])      # unaligned rows
    assert not cv.dgrad_fits(cv.geom(1, 16, 14, 14, 5, 1, 2), 600, t(196, 608), t(400, 608), t(196, 16))    # more filters than fit shared memory
