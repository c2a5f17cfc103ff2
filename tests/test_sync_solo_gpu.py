"""The lone-rank form of the fused step (one rank, nobody to wait for) against the same update written in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["sgd", "momentum", "adam"])
@pytest.mark.parametrize("wire", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("ranges", [[(0, 4)], [(0, 2048), (4096, 4100), (8000, 8000 + 2052)], [(16, 5_000_003)]])
def test_solo_step_matches_reference(kind, wire, ranges):
    """Ranges of one group of four, exactly one block, a block and one group, an end inside a group; only they change."""
    from oxidized_neural_orchestra_b200.ops import _lib
    from oxidized_neural_orchestra_b200.parallel import sync as S

    torch.manual_seed(3)
    n = (ranges[-1][1] + 3) // 4 * 4 + 64
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[wire]
    p, m = torch.randn(n, device="cuda"), torch.randn(n, device="cuda") * 0.1
    v, g = torch.rand(n, device="cuda") * 0.01, (torch.randn(n, device="cuda")).to(dt)
    pb, copy = torch.zeros(n, device="cuda", dtype=torch.bfloat16), torch.zeros(n, device="cuda")
    pows, sumsq = torch.tensor([0.9, 0.999], device="cuda"), torch.zeros(1, device="cuda", dtype=torch.float64)
    want = {"p": p.double(), "m": m.double(), "v": v.double()}
    mask = torch.zeros(n, device="cuda", dtype=torch.bool)
    for b, e in ranges:
        mask[b:(e + 3) // 4 * 4] = True
    gd = g.double() / 3
    if kind == "sgd":
        new = {"p": want["p"] - 0.05 * gd}
    elif kind == "momentum":
        nm = 0.9 * want["m"] + gd
        new = {"m": nm, "p": want["p"] - 0.05 * nm}
    else:
        b1, b2 = (float(torch.tensor(x)) for x in (0.9, 0.999))        # the kernel's constants: 1 - b2 of the f32 value
        nm, nv = b1 * want["m"] + (1 - b1) * gd, b2 * want["v"] + (1 - b2) * gd * gd
        step = 0.05 * (1 - pows[1].double()).sqrt() / (1 - pows[0].double())
        new = {"m": nm, "v": nv, "p": want["p"] - step * nm / (nv.sqrt() + 1e-8)}
    for k, t in new.items():
        want[k] = torch.where(mask, t, want[k])
    s = _lib.OnoSync()
    S.fill_sync(s, nranks=1, rank=0, n=n, nblocks=4, algo=0, g_ptrs=[g.data_ptr()], p_f32_ptrs=[copy.data_ptr()],
                p_bf16_ptrs=[pb.data_ptr()], flag_ptrs=[0], worker_mask=1, member_mask=1, n_workers=3,
                opt=S.OptimizerCfg(kind=kind, lr=0.05, mu=0.9))
    S.fill_local(s.loc[0], p_master=p.data_ptr(), m=m.data_ptr(), v=v.data_ptr(), state_off=0, adam_pows=pows.data_ptr(), epoch=None,
                 ranges=ranges, sumsq=sumsq.data_ptr())
    s.g_dtype, s.zero_grad = {"f32": 0, "bf16": 1, "f16": 2}[wire], 1
    S.launch_sync(s)
    torch.cuda.synchronize()
    for k, t in (("p", p), ("m", m), ("v", v)):
        # a few roundings of values of order one, each 2^-24
        assert (t.double() - want[k]).abs().max().item() <= 1e-6 * max(1.0, want[k].abs().max().item()), k
    assert torch.equal(copy, torch.where(mask, p, torch.zeros_like(p))) and torch.equal(pb, copy.to(torch.bfloat16))
    assert torch.count_nonzero(g[mask]).item() == 0 and torch.count_nonzero(g[~mask]).item() > 0
    assert abs(sumsq.item() - (gd[mask] ** 2).sum().item()) <= 1e-5 * (gd[mask] ** 2).sum().item()
