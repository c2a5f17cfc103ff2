"""Small dense networks as two launches: against 64 bits and against the launches per layer, at the edges of rows, columns and reductions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layers(dims, act):
    acts = [(act, 1.0 if act != "relu" else 0.0)] * (len(dims) - 2)
    return [dict(kind="dense", **{"in": i, "out": o}, act=a) for i, o, a in zip(dims, dims[1:], acts + [("softmax", 0.0)])]


def _engine(layers, B, loss, params, grads, small, start=0):
    from oxidized_neural_orchestra_b200.models.engine import GpuEngine

    e = GpuEngine(layers, batch_size=B, tile_dtype="tf32", loss=loss, params=params, grads=grads)
    assert e.small == start
    if not small:
        e.small = None
    e.refresh()
    return e


def _reference(layers, params, x, y, loss):
    """Gradients and loss in 64 bits (the loss divides by batch x outputs)."""
    p = params.double().clone().requires_grad_()
    h, at = x.double(), 0
    for l in layers:
        i, o = l["in"], l["out"]
        h = h @ p[at:at + i * o].view(i, o) + p[at + i * o:at + i * o + o]
        at += i * o + o
        name = l["act"][0] if l["act"] else None
        h = {"tanh": torch.tanh, "sigmoid": torch.sigmoid, "relu": torch.relu, "gelu": torch.nn.functional.gelu, None: lambda v: v,
             "softmax": lambda v: v.softmax(1)}[name](h)
    value = -(y.double() * h.log()).sum() / h.numel() if loss == "cross_entropy" else ((h - y.double()) ** 2).sum() / h.numel()
    value.backward()
    return p.grad, value.item()


CASES = [([784, 128, 10], 32, "relu"), ([17, 5, 3], 1, "tanh"), ([33, 31, 30, 29, 28], 15, "sigmoid"), ([64, 100, 10], 193, "gelu"),
         ([100, 256, 200, 32], 192, "tanh"), ([517, 33, 3], 385, "tanh"), ([16, 16], 16, "tanh"), ([1, 1, 2], 700, "sigmoid"),
         ([129, 500, 7, 29], 17, "tanh"), ([784, 256, 10], 150, "tanh"), ([40, 48, 44, 36, 24, 20, 12], 33, "gelu"), ([200, 31, 10], 1024, "tanh"),
         # one layer: CTAs of a cluster with no row of the loss, with one and with two
         ([784, 10], 1, "tanh"), ([784, 10], 9, "tanh"), ([784, 10], 17, "tanh"), ([31, 32], 193, "tanh"), ([100, 7], 390, "tanh")]


# networks that do not fit as a whole: the layer from which on they do
TAILS = [([517, 1001, 233, 6], 200, "tanh", 2), ([3000, 100, 10], 256, "sigmoid", 1), ([900, 700, 61, 10], 33, "gelu", 2), ([2000, 250, 5], 31, "relu", 1),
         ([762, 68, 269, 10], 28, "gelu", 1), ([1500, 256, 100, 32], 384, "tanh", 1)]


@pytest.mark.parametrize("dims,B,act,start", [(*c, 0) for c in CASES] + TAILS, ids=lambda v: "x".join(map(str, v)) if isinstance(v, list) else str(v))
@pytest.mark.parametrize("loss", ["cross_entropy", "mse"])
def test_gradients_and_loss(dims, B, act, start, loss):
    layers = _layers(dims, act)
    if loss == "mse":
        layers[-1]["act"] = None if len(dims) % 2 else ("sigmoid", 1.0)
    n = sum((l["in"] + 1) * l["out"] for l in layers)
    torch.manual_seed(0)
    params = torch.randn(n, device="cuda") * (1.0 / max(dims[0], 16) ** 0.5)
    x = torch.rand(B, dims[0], device="cuda")
    y = torch.eye(dims[-1], device="cuda")[torch.randint(0, dims[-1], (B,), device="cuda")]
    want, value = _reference(layers, params, x, y, loss)
    got = []
    for small in (True, False):
        grads = torch.full((n,), 7.0, device="cuda")
        e = _engine(layers, B, loss, params, grads, small, start)
        for _ in range(2):
            e.step(x, y, B, zero_loss=True)
        assert abs(e.loss_sum.item() - value) < 2e-3 * abs(value) + 1e-9
        err = (grads.double() - want).norm() / want.norm()
        got.append((grads.clone(), err.item()))
        once = grads.clone()
        e.step(x, y, B, accumulate=True)            # adds to gradients and loss
        assert torch.allclose(grads, 2 * once, rtol=1e-5, atol=0) and abs(e.loss_sum.item() - 2 * value) < 4e-3 * abs(value) + 1e-9
    # both cut operands to 10 mantissa bits: the same errors up to the order of their sums (a ReLU within rounding of zero may flip)
    assert got[0][1] < 1.2 * got[1][1] + 1e-4, (got[0][1], got[1][1])
    assert torch.allclose(got[0][0], got[1][0], rtol=0, atol=(2e-4 if act != "relu" else 2e-2) * got[1][0].abs().max().item())


def test_fewer_rows_repeats_and_guards():
    """A short last batch; the same bits twice; nothing written past the gradients; rows that start between two vector loads."""
    layers, B = _layers([50, 37, 5], "tanh"), 48
    n = sum((l["in"] + 1) * l["out"] for l in layers)
    torch.manual_seed(1)
    params = torch.randn(n, device="cuda") * 0.2
    wide = torch.rand(B, 53, device="cuda")
    x, y = wide[:, 2:52], torch.eye(5, device="cuda")[torch.randint(0, 5, (B,), device="cuda")]
    store = torch.full((n + 64,), 7.0, device="cuda")
    e = _engine(layers, B, "cross_entropy", params, store[32:32 + n], True)
    seen = []
    for rows in (48, 47, 1, 48):
        e.step(x, y, rows, zero_loss=True)
        want, value = _reference(layers, params, x[:rows], y[:rows], "cross_entropy")
        assert (store[32:32 + n].double() - want).norm() < 3e-3 * want.norm() and abs(e.loss_sum.item() - value) < 2e-3 * value
        seen.append((store.clone(), e.loss_sum.item()))
    assert torch.equal(seen[0][0], seen[3][0]) and seen[0][1] == seen[3][1]
    assert (store[:32] == 7.0).all() and (store[32 + n:] == 7.0).all()


def test_rows_on_the_host_by_index_and_the_loss_there():
    layers, B = _layers([20, 16, 4], "tanh"), 24
    n = sum((l["in"] + 1) * l["out"] for l in layers)
    torch.manual_seed(2)
    params, grads = torch.randn(n, device="cuda") * 0.3, torch.zeros(n, device="cuda")
    x, y = torch.rand(100, 20), torch.eye(4)[torch.randint(0, 4, (100,))]
    idx = torch.randperm(100)[:B].to(torch.int32)
    want, value = _reference(layers, params, x[idx.long()].cuda(), y[idx.long()].cuda(), "cross_entropy")
    host = torch.zeros(1, dtype=torch.float64).pin_memory()
    e = _engine(layers, B, "cross_entropy", params, grads, True)
    e.set_report(host)
    for xs, ys, i in ((x.cuda(), y.cuda(), idx.cuda()), (x[idx.long()].pin_memory(), y[idx.long()].pin_memory(), None)):
        grads.zero_()
        host.zero_()
        e.step(xs, ys, B, idx=i, zero_loss=True)
        torch.cuda.synchronize()
        assert (grads.double() - want).norm() < 3e-3 * want.norm() and host.item() == e.loss_sum.item()
        assert abs(host.item() - value) < 2e-3 * value
