"""The one-channel convolution where it takes another kernel: strides above 2, images too large for one tile, against 64 bits."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,W,K,S,P,filters", [(5, 28, 28, 3, 3, 1, 32), (3, 29, 31, 5, 4, 0, 20), (2, 64, 64, 5, 3, 2, 33), (601, 7, 9, 3, 5, 1, 6),
                                                 (300, 110, 110, 3, 1, 0, 8), (2, 220, 230, 3, 2, 1, 12), (1, 700, 40, 5, 1, 2, 4),
                                                 (1, 3, 2600, 3, 3, 1, 4), (2, 12, 1500, 5, 2, 2, 5)])
def test_forms(dtype, B, H, W, K, S, P, filters):
    from oxidized_neural_orchestra_b200.ops import conv as cv

    torch.manual_seed(0)
    g = cv.geom(B, 1, H, W, K, S, P)
    n = B * g.OH * g.OW
    x = torch.randn(B * H * W, 1, device="cuda").to(dtype)
    k, b = torch.randn(filters * K * K, device="cuda"), torch.randn(filters, device="cuda")
    ld = -(-filters // 16) * 16
    y, dy = torch.full((n, ld), 7.0, device="cuda", dtype=dtype), torch.zeros(n, ld, device="cuda", dtype=dtype)
    dy[:, :filters] = torch.randn(n, filters, device="cuda")
    gk, gb = torch.full_like(k, float("nan")), torch.full_like(b, float("nan"))
    cv.conv1_fwd(g, filters, x, k, b, y, act="relu")
    cv.conv1_wgrad(g, filters, x, dy, gk, gb)
    torch.cuda.synchronize()
    x4, k4 = x.double().view(B, 1, H, W), k.double().view(filters, 1, K, K)
    rows = lambda t: t.permute(0, 2, 3, 1).reshape(n, filters)
    want, mag = rows(torch.relu(F.conv2d(x4, k4, b.double(), S, P))), rows(F.conv2d(x4.abs(), k4.abs(), b.double().abs(), S, P))
    # K * K f32 additions, each off by at most 2^-24 of the sum of magnitudes; one rounding to bf16, at most 2^-8 of the value
    bound = K * K * 2.0 ** -24 * mag + (2.0 ** -8 * 1.01 * want if dtype == torch.bfloat16 else 0.0)
    assert bool(((y[:, :filters].double() - want).abs() <= bound).all()) and bool((y[:, filters:] == 7.0).all())
    cols = F.unfold(x4, K, padding=P, stride=S)                     # [B, K * K, pixels]
    d = dy[:, :filters].double().view(B, -1, filters)
    gw, gm = torch.einsum("bkp,bpf->fk", cols, d), torch.einsum("bkp,bpf->fk", cols.abs(), d.abs())
    # sums over n pixels in chains and trees: far fewer than n roundings reach one term, 2^-24 of the sum of magnitudes each
    assert bool(((gk.double().view(filters, -1) - gw).abs() <= min(n, 4096) * 2.0 ** -24 * gm).all())
    assert bool(((gb.double() - d.sum((0, 1))).abs() <= min(n, 4096) * 2.0 ** -24 * d.abs().sum((0, 1))).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W,K,S", [(29, 3, 1), (30, 5, 1), (28, 3, 2), (31, 5, 2), (31, 3, 3)])
def test_infinite_pixels_reach_only_the_taps_that_see_them(dtype, W, K, S):
    """Columns at the end of a row, which a group of pixels reaching past the row also loads."""
    from oxidized_neural_orchestra_b200.ops import conv as cv

    torch.manual_seed(2)
    B, H, filters = 3, 9, 8
    g = cv.geom(B, 1, H, W, K, S, 0)
    n = B * g.OH * g.OW
    for col in range(W - K - 2, W):
        x = torch.randn(B, H, W, device="cuda").to(dtype)
        x[1, 4, col] = torch.inf
        dy = torch.zeros(n, 16, device="cuda", dtype=dtype)
        dy[:, :filters] = torch.rand(n, filters, device="cuda") + 0.5
        gk, gb = torch.zeros(filters * K * K, device="cuda"), torch.zeros(filters, device="cuda")
        cv.conv1_wgrad(g, filters, x.view(-1, 1), dy, gk, gb)
        want = torch.einsum("bkp,bpf->fk", F.unfold(x.double().view(B, 1, H, W), K, stride=S), dy[:, :filters].double().view(B, -1, filters))
        assert torch.equal(gk.view(filters, -1).isinf(), want.isinf()) and not bool(gk.isnan().any()) and bool(gb.isfinite().all())
