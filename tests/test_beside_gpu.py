"""Weight gradients on a second stream: the same bits as on one stream, eager and captured, for dense, conv and chained engines."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DENSE = [dict(kind="dense", **{"in": 70, "out": 200}, act=("tanh", 1.0)), dict(kind="dense", **{"in": 200, "out": 33}, act=("relu", 0.0)),
         dict(kind="dense", **{"in": 33, "out": 10}, act=("softmax", 0.0))]
CONV = [dict(kind="conv", input_dim=[1, 12, 12], kernel_dim=[6, 1, 5], stride=1, padding=2, act=("tanh", 1.0)),
        dict(kind="pool", input_dim=[6, 12, 12], filter_size=2, stride=2, padding=0, act=None),
        dict(kind="conv", input_dim=[6, 6, 6], kernel_dim=[16, 6, 3], stride=1, padding=0, act=("tanh", 1.0)),
        dict(kind="dense", **{"in": 256, "out": 40}, act=("tanh", 1.0)), dict(kind="dense", **{"in": 40, "out": 10}, act=("softmax", 0.0))]
CHAIN = [dict(kind="dense", **{"in": 70, "out": 72}, act=("tanh", 1.0)),
         dict(kind="conv", input_dim=[2, 6, 6], kernel_dim=[4, 2, 3], stride=1, padding=1, act=("relu", 0.0)),
         dict(kind="dense", **{"in": 144, "out": 10}, act=("softmax", 0.0))]


@pytest.mark.parametrize("layers", [DENSE, CONV, CHAIN], ids=["dense", "conv", "chain"])
@pytest.mark.parametrize("tile", ["tf32", "bf16"])
def test_same_gradients_on_one_and_two_streams(layers, tile):
    from oxidized_neural_orchestra_b200.models.conv_engine import make_engine
    from oxidized_neural_orchestra_b200.models.engine import layer_param_count

    n = (sum(layer_param_count(l) for l in layers) + 15) // 16 * 16
    torch.manual_seed(0)
    params, B = torch.randn(n, device="cuda") * 0.2, 48
    pb = params.to(torch.bfloat16) if tile == "bf16" else None
    xs = layers[0]["in"] if layers[0]["kind"] == "dense" else 144
    x, y = torch.rand(B, xs, device="cuda"), torch.eye(10, device="cuda")[torch.randint(0, 10, (B,), device="cuda")]
    got = []
    for side in (None, torch.cuda.Stream()):
        grads = torch.zeros(n, device="cuda")
        eng = make_engine(layers, batch_size=B, tile_dtype=tile, loss="cross_entropy", params=params, grads=grads, params_bf16=pb)
        eng.set_side(side)
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            eng.refresh(stream=st)
            eng.step(x, y, B, stream=st, zero_loss=True)
            eager = grads.clone()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                eng.step(x, y, B, stream=st, zero_loss=True)
            for _ in range(3):
                grads.fill_(9.0)
                graph.replay()
        torch.cuda.synchronize()
        used = sum(layer_param_count(l) for l in layers)
        assert eng.status.item() == 0 and torch.equal(eager[:used], grads[:used])
        got.append(grads[:used].clone())
    assert torch.equal(got[0], got[1])


def test_second_stream_has_a_workspace_of_its_own(monkeypatch):
    """Two streams may never share the library's static split-K buffer: whoever is given a second stream has slabs for it, also when the
    first step is captured; where they cannot be had the stream is refused."""
    from oxidized_neural_orchestra_b200.models.conv_engine import make_engine
    from oxidized_neural_orchestra_b200.models.engine import layer_param_count
    from oxidized_neural_orchestra_b200.ops import gemm as G

    monkeypatch.setattr(G, "_workspaces", {})
    n = (sum(layer_param_count(l) for l in CONV) + 15) // 16 * 16
    params, grads, side = torch.randn(n, device="cuda") * 0.2, torch.zeros(n, device="cuda"), torch.cuda.Stream()
    eng = make_engine(CONV, batch_size=48, tile_dtype="tf32", loss="cross_entropy", params=params, grads=grads)
    eng.set_side(side)
    assert [k[1] for k in G._workspaces] == [side.cuda_stream]
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st):
        with pytest.raises(RuntimeError):
            eng.set_side(torch.cuda.Stream())
        params.add_(0.0)        # (a capture that records nothing warns)
    assert eng.dense.side is side


def test_a_block_behind_convolutions_keeps_its_weight_gradients_beside(monkeypatch):
    """Every dense weight gradient of a chained network runs on the second stream: in all units something is below their first dense layer."""
    from oxidized_neural_orchestra_b200.models import engine as E
    from oxidized_neural_orchestra_b200.models.conv_engine import make_engine

    layers = CONV[:4] + [dict(kind="conv", input_dim=[10, 2, 2], kernel_dim=[4, 10, 1], stride=1, padding=0, act=("relu", 0.0)),
                         dict(kind="dense", **{"in": 16, "out": 12}, act=("tanh", 1.0)), dict(kind="dense", **{"in": 12, "out": 10}, act=("softmax", 0.0))]
    n = (sum(E.layer_param_count(l) for l in layers) + 15) // 16 * 16
    params, grads, side, seen = torch.randn(n, device="cuda") * 0.2, torch.zeros(n, device="cuda"), torch.cuda.Stream(), []
    eng = make_engine(layers, batch_size=48, tile_dtype="tf32", loss="cross_entropy", params=params, grads=grads)
    eng.set_side(side)
    eng.refresh()
    gemm = E.gemm

    def watched(a, b, **kw):
        if kw.get("a_mn_major"):
            seen.append(kw["stream"])
        return gemm(a, b, **kw)

    monkeypatch.setattr(E, "gemm", watched)
    eng.step(torch.rand(48, 144, device="cuda"), torch.eye(10, device="cuda")[torch.randint(0, 10, (48,), device="cuda")], 48, zero_loss=True)
    torch.cuda.synchronize()
    assert seen == [side] * 3 and eng.status.item() == 0
