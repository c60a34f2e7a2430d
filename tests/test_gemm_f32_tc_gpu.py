"""The float32 products on the tensor cores (csrc/gemm_f32_tc.cu): edges of tiles and steps, shares of K, all epilogues, no
further from 64 bits than the multiply-add tiles; and numbers that three bfloat16 parts do not hold (GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("M,N,K", [(1, 5, 4), (33, 256, 32), (128, 257, 36), (129, 130, 100), (300, 700, 4864), (130, 3000, 68)])
def test_plain(M, N, K):
    from tq_kv_b200.kernels import ACT_SQUARE_RELU, check_tc_status, gemm
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K + 8, device=DEV, generator=g)[:, 4:4 + K]
    w = torch.randn(N, K, device=DEV, generator=g) * K ** -0.5
    bias, base = torch.randn(N, device=DEV, generator=g), torch.randn(M, N, device=DEV, generator=g)
    want = x.double() @ w.double().T
    out = torch.full((M, N + 3), 7.0, device=DEV)              # rows that start off 16 bytes
    gemm.gemm_f32_tc(x, w, out[:, 1:1 + N])
    fma = torch.empty(M, N, device=DEV)
    gemm.gemm_f32(x, w, fma)
    err = _rel(out[:, 1:1 + N], want)
    # six exact products: what is left out is 2^-25 of the operands' sizes, a float32 result keeps 2^-25 of its own
    assert err <= max(1.05 * _rel(fma, want), 2.0 ** -23), (err, _rel(fma, want))
    assert bool((out[:, 0] == 7).all()) and bool((out[:, 1 + N:] == 7).all())
    out = base.clone()
    gemm.gemm_f32_tc(x, w, out, bias, accumulate=True)
    assert _rel(out, want + bias + base) <= 2.0 ** -22
    gemm.gemm_f32_tc(x, w, out, bias, activation=ACT_SQUARE_RELU)
    assert _rel(out, (want + bias).clamp(min=0) ** 2) <= 2.0 ** -20
    check_tc_status()


@pytest.mark.parametrize("M,N,K", [(40, 31, 8), (129, 128, 96), (300, 450, 900)])
@pytest.mark.parametrize("act", ["silu", "gelu"])
def test_gated(M, N, K, act):
    from tq_kv_b200.kernels import ACT_GELU_TANH, ACT_SILU, check_tc_status, gemm
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(2 * N, K, device=DEV, generator=g) * 2 * K ** -0.5
    bias = torch.randn(2 * N, device=DEV, generator=g)
    y = x.double() @ w.double().T + bias.double()
    f = torch.nn.functional.silu if act == "silu" else lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    want = f(y[:, :N]) * y[:, N:]
    out, fma = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    code = ACT_SILU if act == "silu" else ACT_GELU_TANH
    gemm.gemm_f32_tc(x, w, out, bias, swiglu=True, activation=code)
    gemm.gemm_f32(x, w, fma, bias, swiglu=True, activation=code)
    assert _rel(out, want) <= max(1.05 * _rel(fma, want), 2.0 ** -22)
    check_tc_status()


@pytest.mark.parametrize("K", [36, 2048])
@pytest.mark.parametrize("odd", [math.inf, -math.inf, math.nan, 3.3e38, 3.4028e38, 1.3e-38, 1.0e-42, 2.0 ** -115 * 1.1])
def test_numbers_that_three_parts_do_not_hold(K, odd):
    """Such a number makes what the multiply-add tiles make of it, and other rows and columns nothing else."""
    from tq_kv_b200.kernels import check_tc_status, gemm
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(150, K, device=DEV, generator=g), torch.randn(300, K, device=DEV, generator=g)
    x[7, K - 3], w[260, 1] = odd, odd
    if abs(odd) < 1:                                           # a row of nothing but such numbers
        x[9] *= odd
    out, fma = torch.empty(150, 300, device=DEV), torch.empty(150, 300, device=DEV)
    gemm.gemm_f32_tc(x, w, out)
    gemm.gemm_f32(x, w, fma)
    assert torch.equal(out.isnan(), fma.isnan()) and torch.equal(out.isinf(), fma.isinf())
    ok = fma.isfinite()
    assert torch.equal(out[~ok & ~fma.isnan()], fma[~ok & ~fma.isnan()])
    want = x.double() @ w.double().T
    for r in (7, 8, 9):                                        # each row by its own size
        fine = ok[r] & (want[r].abs() < 1e30)
        # float32 sums in two orders, and a unit of the smallest number where the results are about that small
        room = 1e-5 * float(want[r][fine].abs().max()) + 4 * 2.0 ** -149 if bool(fine.any()) else 0.0
        assert float((out[r] - fma[r])[fine].abs().max() if bool(fine.any()) else 0.0) <= room
    check_tc_status()


@pytest.mark.parametrize("rows,columns,gated,want", [(129, 5, False, True), (128, 1792, False, False), (128, 1793, False, True),
                                                     (33, 897, True, True), (32, 151936, False, False), (100, 896, True, False)])
def test_which_float32_products_come_here(rows, columns, gated, want):
    from tq_kv_b200.kernels import gemm
    assert gemm._f32_tc_takes(rows, columns, gated) is want
