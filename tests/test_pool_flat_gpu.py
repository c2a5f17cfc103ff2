"""A pooling layer and the change to flattened rows as one kernel: the same bits as the two kernels, forward and backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B    C   H   W   K  S  P
SIZES = [(64, 16, 8, 8, 2, 2, 0), (66, 20, 24, 24, 2, 2, 0), (592, 5, 6, 7, 3, 1, 1), (3, 8, 12, 10, 3, 2, 1), (64, 1, 9, 9, 2, 2, 0),
         (70, 12, 5, 5, 5, 5, 0), (2, 24, 4, 4, 1, 1, 0), (64, 7, 11, 13, 3, 3, 2)]


@pytest.mark.parametrize("B,C,H,W,K,S,P", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act,dact", [(None, "relu"), ("tanh", None), ("sigmoid", "gelu")])
def test_same_bits_as_two_kernels(B, C, H, W, K, S, P, dtype, act, dact):
    from oxidized_neural_orchestra_b200.ops import conv as cv

    up = lambda n: -(-n // 16) * 16
    torch.manual_seed(0)
    g = cv.geom(B, C, H, W, K, S, P)
    hw, rows = g.OH * g.OW, B * g.OH * g.OW
    assert cv.pool_flat_fits(g, dtype)
    new = lambda r, c, v=0.0: torch.full((r, up(c)), v, device="cuda", dtype=dtype)
    x = torch.randint(-3, 4, (B * H * W, up(C)), device="cuda").to(dtype)          # ties
    kw = dict(act=act, act_param=1.0)
    y, y1, arg, arg1 = new(rows, C), new(rows, C), *(torch.full((rows, C), 9, device="cuda", dtype=torch.int32) for _ in range(2))
    for pad in (0, 1):                                                             # rows that start at 16 bytes, and others
        flat, flat1 = (torch.full((B, up(C * hw) + pad), 7.0, device="cuda", dtype=dtype) for _ in range(2))
        cv.pool_fwd(g, x, y, arg, **kw)
        cv.nchw_flat(B, C, hw, True, y, flat)
        cv.pool_flat_fwd(g, x, y1, arg1, flat1, **kw)
        assert torch.equal(flat, flat1) and torch.equal(y, y1) and torch.equal(arg, arg1)
        d = torch.randn(B, up(C * hw) + pad, device="cuda").to(dtype)
        aux, dy = torch.randn(B * H * W, up(C), device="cuda").to(dtype), new(rows, C)
        dx, dx1 = new(B * H * W, C, 5.0), new(B * H * W, C, 5.0)
        bw = dict(act=act, act_param=1.0, aux=aux, dact=dact, dact_param=0.1)
        cv.nchw_flat(B, C, hw, False, dy, d)
        cv.pool_bwd(g, dy, y, arg, dx, **bw)
        cv.pool_flat_bwd(g, d, y1, arg1, dx1, **bw)
        assert torch.equal(dx, dx1)


def test_what_it_does_not_take():
    from oxidized_neural_orchestra_b200.ops import conv as cv

    assert not cv.pool_flat_fits(cv.geom(64, 64, 28, 28, 2, 2, 0), torch.float32)       # 50 KB of pooled values
    assert not cv.pool_flat_fits(cv.geom(593, 16, 8, 8, 2, 2, 0), torch.float32)        # more images than the separate kernels like
    assert not cv.pool_flat_fits(cv.geom(8, 16, 24, 24, 2, 2, 0), torch.float32)        # few images with many values
    assert not cv.pool_flat_fits(cv.geom(6, 6, 24, 24, 2, 1, 1), torch.bfloat16)        # channels that go one by one: seven rounds of a block
    assert not cv.pool_flat_fits(cv.geom(9, 40, 12, 12, 2, 1, 0), torch.float32)        # three rounds, windows that overlap
    assert cv.pool_flat_fits(cv.geom(9, 40, 12, 12, 2, 2, 0), torch.float32) and not cv.pool_flat_fits(cv.geom(155, 32, 31, 31, 2, 2, 0), torch.float32)
