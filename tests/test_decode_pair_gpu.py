"""The products of csrc/decode_pair_tc.cu where they can go wrong: rows of X around multiples of 16, bands whose last item is
ragged, K that is no multiple of 64, more items than SMs (two accumulators in turn); experts without rows, experts named twice
by a token (a second tile), experts without a gate (GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gated_error(x, w, bias, out, base, act):
    N = w.shape[0] // 2
    y = x.double() @ w.double().T + (0 if bias is None else bias.double())
    g, u = y[:, :N], y[:, N:]
    g = torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    want = g * u + (0 if base is None else base.double())
    # float32 sums of K products of numbers around one (2^-24 a sum of up to sqrt(K)), through a factor of a few; a bfloat16
    # result is rounded to 8 bits, its activation within a few float32 ulp
    room = 8 * math.sqrt(x.shape[1]) * 2.0 ** -24 * (1 + y.abs().max()) * (1 + u.abs())
    if out.dtype == torch.bfloat16:
        room = room + want.abs() * 2.0 ** -8
    return ((out.double() - want).abs() / room).max()


@pytest.mark.parametrize("M", [1, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(40, 64), (74, 200), (1000, 96), (5632, 2048), (19100, 72), (19100, 128)])
def test_gated(M, N, K):
    from tq_kv_b200 import kernels
    from tq_kv_b200.kernels import gemm
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    wide = torch.randn(M, K + 32, device=DEV, generator=g).bfloat16()
    x = wide[:, 8:8 + K]
    w = (torch.randn(2 * N, K, device=DEV, generator=g) * 2 / math.sqrt(K)).bfloat16()
    bias, base = torch.randn(2 * N, device=DEV, generator=g), torch.randn(M, N, device=DEV, generator=g)
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    gemm.decode_pair_tc(x, w, out)
    assert _gated_error(x, w, None, out, None, "silu") < 1
    out = base.clone()
    gemm.decode_pair_tc(x, w, out, bias, True, kernels.ACT_GELU_TANH)
    assert _gated_error(x, w, bias, out, base, "gelu") < 1
    out = torch.full((M, N + 3), 7.0, device=DEV)              # rows that start anywhere: entries stored one by one
    gemm.decode_pair_tc(x, w, out[:, 1:1 + N], bias)
    assert _gated_error(x, w, bias, out[:, 1:1 + N], None, "silu") < 1
    assert bool((out[:, 0] == 7).all()) and bool((out[:, 1 + N:] == 7).all())
    kernels.check_tc_status()


@pytest.mark.parametrize("T,E,top", [(1, 4, 2), (16, 8, 2), (17, 3, 3), (33, 40, 1), (64, 8, 2)])
@pytest.mark.parametrize("W,F,gated", [(72, 136, True), (256, 1000, True), (200, 264, False)])
def test_experts(T, E, top, W, F, gated):
    from tq_kv_b200 import kernels
    from tq_kv_b200.kernels import experts
    g = torch.Generator(device=DEV).manual_seed(T + E + W)
    x = torch.randn(T, W, device=DEV, generator=g).bfloat16()
    w_up = (torch.randn(E, (2 if gated else 1) * F, W, device=DEV, generator=g) * W ** -0.5).bfloat16()
    w_down = (torch.randn(E, W, F, device=DEV, generator=g) * F ** -0.5).bfloat16()
    live = max(1, E - 2)                                       # two experts get no rows
    choice = torch.stack([(torch.arange(top, device=DEV) + t) % live for t in range(T)]).int()
    choice[-1] = 0                                             # ... and one token names an expert `top` times
    y = torch.randn(T, W, device=DEV, generator=g)
    base = y.clone()
    assert T <= experts.FEW_TILE_ROWS
    kernels.routed_experts_tiles(x, w_up, w_down, choice, y, True, gated=gated)
    want = base.double()
    for t in range(T):
        for e in choice[t].tolist():
            h = w_up[e].double() @ x[t].double()
            h = torch.nn.functional.silu(h[:F]) * h[F:] if gated else h.clamp(min=0) ** 2
            want[t] += (w_down[e].double() @ h.bfloat16().double()) / top
    # the first product's result is rounded to bfloat16 (2^-9 of each entry, and the entries next to a boundary of rounding
    # may go either way: one unit of 2^-8), and a sum over F such entries carries sqrt(F) of them
    h_rms = (want - base).norm() / math.sqrt(want.numel())
    assert float((y - want).abs().max()) < 8 * 2.0 ** -8 * max(float(h_rms), 0.1)
    kernels.check_tc_status()


@pytest.mark.parametrize("rows,n,k,want", [(17, 64, 64, True), (9, 4864, 896, False), (9, 5632, 1024, True), (8, 5632, 2048, True),
                                           (8, 4864, 2048, False), (2, 64, 40, True)])
def test_which_gated_products_come_here(rows, n, k, want):
    from tq_kv_b200.kernels import gemm
    assert gemm._pair_takes(rows, torch.empty(2 * n, k, dtype=torch.bfloat16, device="meta")) is want
