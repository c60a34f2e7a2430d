"""The product of one bfloat16 row (csrc/row_gemm.cu) against float64, within the rounding bound of a float32 sum of K exact
products, (K + 8) 2^-24 |x| . |w|, and half an ulp (2^-8) where the result is bfloat16; at the edges of pieces, column groups
and the counts of warps that share a column."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -24


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def within(got, want, bound):
    half_ulp = 2.0 ** -8 * want.abs() if got.dtype == torch.bfloat16 else 0.0
    assert bool(((got.double() - want).abs() <= bound + half_ulp).all())


@pytest.mark.parametrize("N,K", [(1, 8), (3, 248), (4, 256), (130, 264), (1152, 896), (5000, 1032), (40000, 136), (64, 4872),
                                 (2048, 5632)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_against_float64(N, K, out_dtype):
    from tq_kv_b200 import kernels
    from tq_kv_b200.kernels import gemm
    w, bias = rnd(2 * N, K, seed=1).bfloat16(), rnd(2 * N, seed=2)
    x = rnd(3, K + 8).bfloat16()[1:2, 8:]
    y = x.double() @ w.double().T + bias.double()
    size = (x.double().abs() @ w.double().abs().T + bias.double().abs()) * ((K + 8) * U)
    out = torch.empty(1, N, dtype=out_dtype, device=DEV)
    gemm.row_gemm(x, w[:N], out, bias[:N])
    within(out, y[:, :N], size[:, :N])
    gemm.row_gemm(x, w, out, bias, swiglu=True)
    act, up = torch.nn.functional.silu(y[:, :N]), y[:, N:]
    within(out, act * up, 1.1 * size[:, :N] * up.abs() + act.abs() * size[:, N:] + 1.1 * size[:, :N] * size[:, N:]
           + 64 * U * (act * up).abs())
    if out_dtype == torch.float32:
        base = rnd(1, N, seed=4)
        out = base.clone()
        gemm.row_gemm(x, w[:N], out, bias[:N], accumulate=True)
        within(out, base.double() + y[:, :N], size[:, :N] + 2 * U * base.double().abs())
    else:
        gemm.row_gemm(x, w[:N], out, bias[:N], activation=kernels.elementwise.ACT_SQUARE_RELU)
        p = torch.relu(y[:, :N])
        within(out, p * p, 2 * p * size[:, :N] + size[:, :N] ** 2 + 4 * U * p * p)


@pytest.mark.parametrize("N,K,swiglu", [(10304, 1000, False), (3000, 4096, True), (40000, 264, False)])
def test_linear_gives_the_same_with_and_without(N, K, swiglu, monkeypatch):
    """kernels.linear of one row, given and after a pending norm, on this kernel and on the ones that ran before."""
    from tq_kv_b200 import kernels
    from tq_kv_b200.kernels import gemm
    w = (rnd(N * (2 if swiglu else 1), K, seed=1) * K ** -0.5).bfloat16()
    h, g = rnd(1, K, seed=2), rnd(K, seed=3)
    assert gemm._row_takes(1, w, swiglu)
    got = []
    for takes in (True, False):
        if not takes:
            monkeypatch.setattr(gemm, "_row_takes", lambda *a: False)
        for x in (h.bfloat16(), kernels.PendingNorm(h, g, 1e-6, torch.bfloat16)):
            got.append(kernels.linear(x, w, swiglu=swiglu, out_dtype=torch.float32))
    # given rows: sums in another order; after a norm the other kernels may round h * g instead of h / rms * g
    assert float((got[0] - got[2]).abs().max()) <= 1e-4 * float(got[2].abs().max())
    assert float((got[1] - got[3]).norm()) <= 6e-3 * float(got[3].norm())
