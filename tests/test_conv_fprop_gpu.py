"""Forward convolution in one kernel: columns and results with the same bits as im2col and the product."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B    C   H   W   F   K  S  P
SIZES = [(5, 32, 28, 28, 64, 3, 2, 1), (400, 32, 14, 14, 64, 3, 1, 1), (3, 8, 14, 14, 16, 5, 1, 0), (50, 16, 9, 11, 40, 3, 1, 1), (1, 8, 5, 5, 8, 3, 1, 0),
         (7, 40, 12, 10, 24, 5, 1, 2), (9, 64, 14, 14, 64, 3, 2, 1), (2, 8, 6, 6, 256, 3, 3, 0), (300, 64, 7, 7, 128, 1, 1, 0), (4, 24, 13, 17, 40, 4, 2, 1), (33, 16, 33, 31, 24, 2, 2, 0)]


@pytest.mark.parametrize("B,C,H,W,F,K,S,P", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act", [None, "relu", "tanh"])
def test_same_bits_as_im2col_and_product(B, C, H, W, F, K, S, P, dtype, act):
    from oxidized_neural_orchestra_b200.ops import conv as cv
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    up = lambda n: -(-n // 16) * 16
    torch.manual_seed(0)
    g = cv.geom(B, C, H, W, K, S, P)
    rows, ckk = B * g.OH * g.OW, C * K * K
    mk = lambda r, c: torch.nn.functional.pad(torch.randn(r, c, device="cuda"), (0, up(c) - c)).to(dtype)
    x, kop, bias = mk(B * H * W, C), mk(F, ckk), torch.randn(F, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cols, want = torch.zeros(rows, up(ckk), device="cuda", dtype=dtype), torch.zeros(rows, up(F), device="cuda", dtype=dtype)
    cv.im2col(g, x, cols)
    gemm(cols[:, :ckk], kop[:, :ckk], bias=bias, act=act, act_param=1.0, split_k=1, cluster=-1, status=status,
         **{"out" if dtype == torch.float32 else "out_bf16": want[:, :F]})
    store = torch.full((rows + 4, up(F)), 3.0, device="cuda", dtype=dtype)
    cstore = torch.full((rows + 4, up(ckk)), 3.0, device="cuda", dtype=dtype)
    got, gcols = store[2:-2], cstore[2:-2]
    assert cv.fprop_fits(g, F, x, kop, got, gcols)
    for with_cols in (True, False):
        got.fill_(3.0)
        cv.fprop(g, F, x, kop[:, :ckk], got, cols=gcols if with_cols else None, bias=bias, act=act, act_param=1.0, status=status)
        assert torch.equal(got[:, :F], want[:, :F]) and torch.equal(gcols[:, :ckk], cols[:, :ckk])
    assert all((t == 3.0).all() for t in (store[:2], store[-2:], cstore[:2], cstore[-2:], got[:, F:], gcols[:, ckk:])) and status.item() == 0


def test_what_it_does_not_take():
    from oxidized_neural_orchestra_b200.ops import conv as cv

    t = lambda r, c, d=torch.float32: torch.zeros(r, c, device="cuda", dtype=d)
    g = lambda c, k=3: cv.geom(2, c, 8, 8, k, 1, k // 2)
    assert cv.fprop_fits(g(8), 16, t(128, 16), t(16, 80), t(128, 16))
    assert not cv.fprop_fits(g(6), 16, t(128, 16), t(16, 64), t(128, 16))                   # channels that end inside a piece
    assert not cv.fprop_fits(g(8), 15, t(128, 16), t(15, 80), t(128, 16))                   # filters that do
    assert not cv.fprop_fits(g(8), 16, t(128, 18)[:, 2:], t(16, 80), t(128, 16))            # unaligned rows
    assert not cv.fprop_fits(g(64, 5), 96, t(128, 64), t(96, 1600), t(128, 96))             # a kernel tensor that does not fit shared memory
