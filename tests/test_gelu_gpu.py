"""GELU's derivative as the GEMM epilogues compute it, and derivatives from stored values at ragged edges in either type."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _slopes(z):
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    n = z.shape[1]
    out = torch.empty_like(z)
    gemm(torch.ones_like(z), torch.eye(n, device="cuda"), out=out, aux=z, dact="gelu")      # products with one are exact
    return out


@pytest.mark.parametrize("scale,bound", [(0.3, 4.0e-8), (1.0, 3.8e-8), (3.0, 3.8e-8)])
def test_derivative_against_64_bits(scale, bound):
    """``bound``: with erff and expf the errors were 3.82e-8, 3.94e-8 and 4.11e-8."""
    torch.manual_seed(0)
    z = torch.randn(2048, 64, device="cuda") * scale
    Z = z.double()
    want = torch.special.ndtr(Z) + Z * torch.exp(-Z * Z / 2) / math.sqrt(2 * math.pi)
    got = _slopes(z).double()
    assert (got - want).norm() / want.norm() < bound
    assert (got - want).abs().max() < 1.3e-7


def test_derivative_far_out():
    z = torch.tensor([[1e30, -1e30, 0.0, -0.0, 5e-30, 40.0, -40.0, float("nan")]], device="cuda")
    got = _slopes(z)[0]
    # (with a NaN among the stored values its own result alone is one)
    assert got[:7].tolist() == [1.0, 0.0, 0.5, 0.5, 0.5, 1.0, 0.0] and got[7].isnan()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,off", [(129, 257, 0), (300, 130, 0), (257, 999, 0), (128, 34, 0), (131, 66, 1)])
def test_stored_values_at_ragged_edges(dtype, M, N, off):
    """The persistent kernel fetches them a chunk ahead and unpacks them later; ``off``: rows that start between two vector loads."""
    from oxidized_neural_orchestra_b200.ops.gemm import gemm

    torch.manual_seed(1)
    K = 64
    a, b = torch.randn(M, K, device="cuda").to(dtype), torch.randn(N, K, device="cuda").to(dtype)
    ld = (N + 15) // 16 * 16
    aux = torch.randn(M, ld + 16, device="cuda").to(dtype)[:, off:off + N]
    out = torch.zeros(M, ld, device="cuda", dtype=dtype)[:, :N]
    gemm(a, b, **{"out" if dtype == torch.float32 else "out_bf16": out}, aux=aux, dact="sigmoid", act_param=0.0, dact_param=1.0, cluster=-1)
    s = aux.double()
    want = (a.double() @ b.double().t()) * s * (1 - s)
    # operands cut to 10 mantissa bits (tf32) or results rounded to 8 (bf16)
    assert (out.double() - want).norm() / want.norm() < (2e-3 if dtype == torch.float32 else 4e-3)
