"""A batch in pinned host memory is a batch: every engine takes it like one on the GPU, also on a stream of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DENSE = [dict(kind="dense", **{"in": 70, "out": 40}, act=("tanh", 1.0)), dict(kind="dense", **{"in": 40, "out": 10}, act=("softmax", 0.0))]
CONV = [dict(kind="conv", input_dim=[1, 12, 12], kernel_dim=[6, 1, 3], stride=1, padding=1, act=("tanh", 1.0)),
        dict(kind="dense", **{"in": 864, "out": 10}, act=("softmax", 0.0))]
CHAIN = [dict(kind="dense", **{"in": 70, "out": 72}, act=("tanh", 1.0)),
         dict(kind="conv", input_dim=[2, 6, 6], kernel_dim=[4, 2, 3], stride=1, padding=1, act=("relu", 0.0)),
         dict(kind="dense", **{"in": 144, "out": 10}, act=("softmax", 0.0))]


@pytest.mark.parametrize("layers", [DENSE, CONV, CHAIN], ids=["dense", "conv", "chain"])
@pytest.mark.parametrize("tile", ["tf32", "bf16"])
@pytest.mark.parametrize("host", ["xy", "x", "y"])
def test_pinned_host_batch(layers, tile, host):
    from oxidized_neural_orchestra_b200.models.conv_engine import make_engine
    from oxidized_neural_orchestra_b200.models.engine import layer_param_count

    used = sum(layer_param_count(l) for l in layers)
    n = (used + 15) // 16 * 16
    torch.manual_seed(0)
    params, B = torch.randn(n, device="cuda") * 0.2, 20
    pb = params.to(torch.bfloat16) if tile == "bf16" else None
    xs = layers[0]["in"] if layers[0]["kind"] == "dense" else 144
    x, y = torch.rand(B, xs), torch.eye(10)[torch.randint(0, 10, (B,))]
    got = []
    for where in ("", host):
        grads = torch.zeros(n, device="cuda")
        eng = make_engine(layers, batch_size=B, tile_dtype=tile, loss="cross_entropy", params=params, grads=grads, params_bf16=pb)
        eng.loss_sum.fill_(3.0)
        bx, by = (t.pin_memory() if k in where else t.cuda() for k, t in (("x", x), ("y", y)))
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        eng.refresh(stream=st)
        eng.step(bx, by, B, stream=st, zero_loss=True)
        torch.cuda.synchronize()
        assert eng.status.item() == 0
        got.append((grads[:used].clone(), eng.loss_sum.item()))
    assert torch.equal(got[0][0], got[1][0]) and abs(got[0][1] - got[1][1]) <= 1e-12 * abs(got[0][1])


def test_batches_in_unpinned_host_memory_are_refused():
    from oxidized_neural_orchestra_b200.ops import elementwise as ew

    dst = torch.zeros(4, 16, device="cuda")
    with pytest.raises(RuntimeError):
        ew.rows_jobs([dict(src=torch.zeros(4, 16), dst=dst)])
