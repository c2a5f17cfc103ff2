"""The loss kernel's forms (one value a lane, four, shared memory, memory) at their edges, and rows that are not ordinary numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
CLASSES = [1, 2, 32, 33, 64, 96, 100, 128, 129, 1000, 1023, 1024, 1025, 2500]


def _run(z, y, kind, softmax, eps=1.1920929e-07):
    from oxidized_neural_orchestra_b200.ops import elementwise as ew

    d, probs = torch.zeros_like(z), torch.zeros_like(z)
    db, ls = torch.zeros(z.shape, device="cuda", dtype=torch.bfloat16), torch.zeros(1, device="cuda", dtype=torch.float64)
    cor = torch.zeros(1, device="cuda", dtype=torch.int32)
    ew.loss_backward(z, y, kind=kind, softmax=softmax, loss_sum=ls, d=d, d_bf16=db, probs=probs, correct=cor, eps=eps)
    torch.cuda.synchronize()
    assert torch.equal(torch.nan_to_num(db.float()), torch.nan_to_num(d.to(torch.bfloat16).float()))
    return d, probs, ls.item(), cor.item()


def _ref(z, y, kind, softmax, eps=1.1920929e-07):
    z, y, n = z.double(), y.double(), z.numel()
    p = torch.softmax(z, 1) if softmax else z
    if kind == "cross_entropy":
        ps = p.clamp_min(eps)
        L, g = -(y * torch.log(ps)).sum() / n, -(y / ps) / n
    else:
        L, g = ((p - y) ** 2).sum() / n, 2 * (p - y) / n
    return (p * (g - (p * g).sum(1, keepdim=True)) if softmax else g), p, L.item()


@pytest.mark.parametrize("C", CLASSES)
@pytest.mark.parametrize("kind,softmax", [("cross_entropy", True), ("mse", True), ("mse", False), ("cross_entropy", False)])
@pytest.mark.parametrize("soft_labels", [False, True])
def test_forms_against_64_bits(C, kind, softmax, soft_labels):
    torch.manual_seed(C)
    B = 37
    z = torch.randn(B, C, device="cuda") * 3 if softmax else torch.rand(B, C, device="cuda") + 0.1
    y = torch.rand(B, C, device="cuda") if soft_labels else torch.eye(C, device="cuda")[torch.randint(0, C, (B,), device="cuda")]
    d, p, L, cor = _run(z, y, kind, softmax)
    rd, rp, rL = _ref(z, y, kind, softmax)
    # sums of C terms in f32, exponentials of arguments up to about 12 (12 units of 2^-24 each) and a handful of products
    tol = (64 + C / 32) * 2.0 ** -24
    assert (p.double() - rp).abs().max().item() <= tol * rp.abs().max().item()
    scale = rd.abs().max().item() + (1.0 / (B * C) if softmax else 0.0)     # (a row's terms cancel for C = 1)
    assert (d.double() - rd).abs().max().item() <= 4 * tol * scale
    assert abs(L - rL) <= 4 * tol * max(1.0, abs(rL)) and cor == (z.argmax(1) == y.argmax(1)).sum().item()


@pytest.mark.parametrize("C", [10, 33, 128, 129, 1024, 1025])
def test_rows_with_infinities_and_nan(C):
    torch.manual_seed(1)
    z = torch.randn(8, C, device="cuda")
    y = torch.eye(C, device="cuda")[torch.arange(8, device="cuda") % C]
    z[1, C - 1], z[2, 3], z[3, C - 2], z[5, 1:] = -torch.inf, torch.inf, torch.nan, -torch.inf
    z[4, :], z[6, :] = torch.finfo(torch.float32).min, torch.finfo(torch.float32).min
    z[6, 6] = 0.0
    d, p, _, _ = _run(z, y, "cross_entropy", True)
    rd, rp, _ = _ref(z, y, "cross_entropy", True)
    assert torch.equal(d.isnan(), rd.isnan()) and torch.equal(p.isnan(), rp.isnan())
    ok = ~rd.isnan().any(1)
    assert ok.tolist() == [True, True, False, False, True, True, True, True]
    assert (d.double() - rd)[ok].abs().max().item() <= 1e-5 * rd[ok].abs().max().item()
    # without a floor under the probability a class of probability zero takes the logarithm of zero, whatever its label
    assert _run(z[5:6], y[:1], "cross_entropy", True, eps=0.0)[0].isnan().all() and _ref(z[5:6], y[:1], "cross_entropy", True, 0.0)[0].isnan().all()
