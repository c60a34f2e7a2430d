"""The many-row tcgen05 product where its tiles go in several bands of rows (more than 16 rows of 256 x 256 tiles): a last
band of one row of tiles, a whole one, a ragged one, every epilogue (GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [4097, 8192, 8192 + 3 * 256 + 5])
@pytest.mark.parametrize("N,K", [(520, 136), (1800, 64)])
def test_bands(M, N, K):
    from tq_kv_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).bfloat16() for n in (M, 2 * N))
    bias, base = torch.randn(N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
    y = x.double() @ w.double().T
    # float32 sums of K products of unit normals in any order: sqrt(K) of them, K 2^-24 each at the very most
    tol = K * math.sqrt(K) * 2.0 ** -24
    out = torch.full((M, N), 7.0, device="cuda")
    kernels.gemm_tc(x, w[:N], out, bias)
    assert float((out - (y[:, :N] + bias)).abs().max()) < tol
    out = base.clone()
    kernels.gemm_tc(x, w[:N], out, None, kernels.gemm.EPI_ACCUM)
    assert float((out - (y[:, :N] + base)).abs().max()) < tol
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    kernels.gemm_tc(x, w, out, None, kernels.gemm.EPI_SWIGLU)
    want = torch.nn.functional.silu(y[:, :N]) * y[:, N:]
    # a bfloat16 result: half a unit in its eighth bit, and the sums' error times the other factor
    assert bool(((out - want).abs() <= want.abs() * 2.0 ** -8 + tol * (1 + y.abs().max())).all())
    kernels.check_tc_status()


@pytest.mark.parametrize("M", [257, 300, 385])
@pytest.mark.parametrize("N,K", [(10304, 136), (3584, 1032)])
def test_rows_of_few_tiles(M, N, K):
    """Rows of two 256-row tiles on pairs of SMs and of three or four 128-row tiles on single ones: both forms, by size."""
    test_bands(M, N, K)
