"""Gathers and scatters around the convolution GEMMs against PyTorch: every piece width (C a multiple of 8, of 4, odd), strides,
paddings, ragged pixel counts, rows with padding, and the generic forms (transposed copies)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

GEOMS = [(3, 8, 9, 7, 3, 2, 1), (2, 32, 14, 14, 3, 2, 1), (5, 4, 6, 11, 3, 1, 1), (1, 20, 8, 8, 5, 1, 2), (2, 12, 13, 9, 5, 2, 0),
         (2, 5, 7, 7, 3, 2, 1), (3, 6, 9, 8, 5, 1, 0), (4, 64, 5, 5, 2, 2, 0), (70, 16, 3, 3, 3, 1, 1)]


def _padded(rows, c, ld, dt, fill=7.0):
    return torch.full((rows, ld), fill, device="cuda", dtype=dt)[:, :c]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("shape", GEOMS)
def test_im2col_and_col2im(dtype, transposed, shape):
    from oxidized_neural_orchestra_b200.ops import conv as CV

    B, C, H, W, K, S, P = shape
    g = CV.geom(*shape)
    torch.manual_seed(0)
    rows, ckk, npix = B * g.OH * g.OW, C * K * K, B * H * W
    x = _padded(npix, C, (C + 15) // 16 * 16, dtype)
    x.copy_(torch.randn(npix, C, device="cuda"))
    cols = _padded(rows, ckk, (ckk + 15) // 16 * 16, dtype)
    cols_t = torch.zeros(ckk, (rows + 15) // 16 * 16, device="cuda", dtype=dtype) if transposed else None
    CV.im2col(g, x, cols, cols_t)
    img = x.double().view(B, H, W, C).permute(0, 3, 1, 2)
    ref = F.unfold(img, K, padding=P, stride=S).view(B, C, K * K, -1).permute(0, 3, 2, 1).reshape(rows, ckk)   # (ky, kx, c)
    assert torch.equal(cols.double(), ref) and bool((cols._base[:, ckk:] == 7.0).all())
    if transposed:
        assert torch.equal(cols_t[:, :rows].double(), ref.t())

    d = _padded(rows, ckk, (ckk + 15) // 16 * 16, dtype)
    d.copy_(torch.randn(rows, ckk, device="cuda"))
    aux = _padded(npix, C, (C + 15) // 16 * 16, dtype)
    aux.copy_(torch.rand(npix, C, device="cuda") * 2 - 1)
    dx = _padded(npix, C, (C + 15) // 16 * 16, dtype)
    dx_t = torch.zeros(C, (npix + 15) // 16 * 16, device="cuda", dtype=dtype) if transposed else None
    CV.col2im(g, d, dx, dx_t, aux=aux, dact="tanh", dact_param=1.0)
    back = d.double().view(B, g.OH * g.OW, K * K, C).permute(0, 3, 2, 1).reshape(B, C * K * K, -1)
    want = F.fold(back, (H, W), K, padding=P, stride=S).permute(0, 2, 3, 1).reshape(npix, C) * (1 - aux.double() ** 2)
    # at most K * K f32 additions of N(0, 1) values, then one rounding to the tile type
    bound = K * K * 2.0 ** -23 * 4 * K + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22)
    assert bool(((dx.double() - want).abs() <= bound).all()) and bool((dx._base[:, C:] == 7.0).all())
    if transposed:
        assert torch.equal(dx_t[:, :npix].t(), dx)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(3, 6, 10, 8, 2, 2, 0), (2, 33, 7, 7, 3, 2, 1), (2, 4, 6, 6, 3, 1, 1), (4, 16, 9, 5, 2, 3, 0)])
def test_pooling_gradient_through_both_activations(dtype, shape):
    from oxidized_neural_orchestra_b200.ops import conv as CV

    B, C, H, W, K, S, P = shape
    g = CV.geom(*shape)
    torch.manual_seed(1)
    rows, npix, ld = B * g.OH * g.OW, B * H * W, (C + 15) // 16 * 16
    x = _padded(npix, C, ld, dtype)
    x.copy_(torch.randn(npix, C, device="cuda"))
    y, arg = _padded(rows, C, ld, dtype), torch.zeros(rows, C, device="cuda", dtype=torch.int32)
    CV.pool_fwd(g, x, y, arg, act="tanh", act_param=1.0)
    d = _padded(rows, C, ld, dtype)
    d.copy_(torch.randn(rows, C, device="cuda"))
    dx, dx_t = _padded(npix, C, ld, dtype), torch.zeros(C, (npix + 15) // 16 * 16, device="cuda", dtype=dtype)
    CV.pool_bwd(g, d, y, arg, dx, dx_t, act="tanh", act_param=1.0, aux=x, dact="sigmoid", dact_param=1.0)
    flow = d.double() * (1 - y.double() ** 2)
    want = torch.zeros(B, H * W, C, device="cuda", dtype=torch.float64)
    idx = arg.view(B, -1, C).long()
    want.scatter_add_(1, idx.clamp_min(0), torch.where(idx >= 0, flow.view(B, -1, C), torch.zeros_like(flow.view(B, -1, C))))
    want = want.view(npix, C) * x.double() * (1 - x.double())
    bound = 2.0 ** -18 + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18)
    assert bool(((dx.double() - want).abs() <= bound).all()) and bool((dx._base[:, C:] == 7.0).all())
    assert torch.equal(dx_t[:, :npix].t(), dx)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,C,HW", [(1, 1, 1), (3, 33, 31), (2, 64, 49), (5, 3, 784), (70000, 2, 3), (17, 64, 49), (300, 20, 144), (16, 12, 9), (33, 6, 7), (2000, 8, 16)])
def test_flattening_there_and_back(dtype, B, C, HW):
    from oxidized_neural_orchestra_b200.ops import conv as CV

    torch.manual_seed(2)
    img = _padded(B * HW, C, (C + 15) // 16 * 16, dtype)
    img.copy_(torch.randn(B * HW, C, device="cuda"))
    flat = _padded(B, C * HW, C * HW + 5, dtype)
    out_t = torch.zeros(C * HW, B, device="cuda", dtype=dtype)
    CV.nchw_flat(B, C, HW, True, img, flat, out_t)
    ref = img.reshape(B, HW, C).permute(0, 2, 1).reshape(B, C * HW)
    assert torch.equal(flat, ref) and torch.equal(out_t, ref.t()) and bool((flat._base[:, C * HW:] == 7.0).all())
    for ld in (C * HW + 5, (C * HW + 15) // 16 * 16):        # without the transposed copy; rows that are and are not aligned
        flat = _padded(B, C * HW, ld, dtype)
        CV.nchw_flat(B, C, HW, True, img, flat)
        assert torch.equal(flat, ref) and bool((flat._base[:, C * HW:] == 7.0).all())
        back = _padded(B * HW, C, (C + 15) // 16 * 16, dtype)
        CV.nchw_flat(B, C, HW, False, back, flat)
        assert torch.equal(back, img) and bool((back._base[:, C:] == 7.0).all())
        aux = _padded(B * HW, C, (C + 15) // 16 * 16, dtype)
        aux.copy_(torch.rand(B * HW, C, device="cuda"))
        CV.nchw_flat(B, C, HW, False, back, flat, aux=aux, dact="sigmoid", dact_param=1.0)
        want = img.double() * aux.double() * (1 - aux.double())
        # three f32 roundings, then one to the tile type
        assert bool(((back.double() - want).abs() <= want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) + 1e-6).all())
