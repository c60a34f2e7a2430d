"""The float32 products of csrc/gemm_f32.cu against float64, element by element within the rounding bound of a float32
sum of K products, (K + 4) 2^-24 (|x| . |w| + ...), at the edges of tiles, pieces and row counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -24


def rnd(*shape, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g).to(DEV)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 96, 300])
@pytest.mark.parametrize("N,K", [(1, 4), (5, 28), (64, 32), (128, 36), (129, 896), (203, 1000), (2049, 132), (16, 4864)])
def test_plain_accumulated_and_gated(M, N, K):
    from tq_kv_b200 import kernels
    x, w, bias = rnd(M, K + 8)[:, 4:4 + K], rnd(2 * N, K, seed=1), rnd(2 * N, seed=2)
    assert kernels.gemm._f32_ok(x, w, torch.empty(M, N, device=DEV))
    y = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T + bias.double().abs()
    out = torch.full((M, N + 3), 7.0, device=DEV)[:, :N]                # rows of an odd stride
    kernels.linear(x, w[:N], bias=bias[:N], out=out)
    assert bool(((out.double() - y[:, :N] - bias[:N].double()).abs() <= (K + 4) * U * size[:, :N]).all())
    base = rnd(M, N, seed=3)
    out = base.clone()
    kernels.linear(x, w[:N], out=out, accumulate=True)
    err = (out.double() - base.double() - y[:, :N]).abs()
    assert bool((err <= (K + 4) * U * (size[:, :N] + base.double().abs())).all())
    out = kernels.linear(x, w, bias=bias, swiglu=True)
    z = y + bias.double()
    act = torch.nn.functional.silu(z[:, :N])
    want = act * z[:, N:]
    # silu is 1.1-Lipschitz; its float32 evaluation and the product add a few roundings of the result
    bound = (K + 4) * U * (1.1 * size[:, :N] * z[:, N:].abs() + act.abs() * size[:, N:] + 1.1 * (K + 4) * U * size[:, :N] * size[:, N:]) + 16 * U * want.abs()
    assert bool(((out.double() - want).abs() <= bound).all())
    out = kernels.linear(x, w[:N], bias=bias[:N], activation=kernels.elementwise.ACT_SQUARE_RELU)
    p = torch.relu(z[:, :N])
    e = (K + 4) * U * size[:, :N]
    assert bool(((out.double() - p * p).abs() <= 2 * p * e + e * e + 4 * U * p * p).all())


@pytest.mark.parametrize("M", [2, 40])
def test_operands_that_the_kernels_refuse_run_on_the_general_ones(M):
    from tq_kv_b200 import kernels
    K, N = 130, 70
    x, w = rnd(M, K), rnd(N, K, seed=1)                                   # K is no multiple of 4
    shifted = rnd(M, K + 1)[:, 1:]                                        # rows that do not start on 16 bytes
    for a, b in ((x, w), (shifted[:, :128], w[:, :128].contiguous())):
        out = torch.empty(M, N, device=DEV)
        assert not kernels.gemm._f32_ok(a, b, out)
        kernels.linear(a, b, out=out)
        size = a.double().abs() @ b.double().abs().T
        assert bool(((out.double() - a.double() @ b.double().T).abs() <= (K + 4) * U * size).all())


def test_a_cut_along_k_gives_the_same_bits_twice():
    from tq_kv_b200 import kernels
    x, w = rnd(40, 4864), rnd(896, 4864, seed=1)                          # few tiles: K is shared by a cluster
    runs = [kernels.linear(x, w) for _ in range(3)]
    assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])


@pytest.mark.parametrize("M,N,K,dtype", [(1, 896, 896, torch.float32), (4, 2000, 512, torch.float32), (40, 896, 4864, torch.float32),
                                         (1, 10304, 2048, torch.bfloat16)])
def test_a_weight_that_the_kernel_in_front_writes(M, N, K, dtype):
    """Not a settled weight (the default): a norm kernel lets its successor start before it has written its rows."""
    from tq_kv_b200 import kernels
    x, g, w = rnd(M, K).to(dtype), torch.ones(K, device=DEV), torch.empty(N, K, dtype=dtype, device=DEV)
    for i in range(5):
        rows = rnd(N, K, seed=10 + i)
        torch.cuda.synchronize()
        kernels.rmsnorm(rows, g, 1e-6, w)
        out = kernels.linear(x, w, out_dtype=torch.float32)
        size = x.double().abs() @ w.double().abs().T
        assert bool(((out.double() - x.double() @ w.double().T).abs() <= (K + 8) * U * size).all())
        want = rows.double() * torch.rsqrt((rows.double() ** 2).mean(-1, keepdim=True) + 1e-6)
        assert float((w.double() - want).abs().max()) <= 0.02 * float(want.abs().max())


@pytest.mark.parametrize("swiglu", [False, True])
def test_more_columns_than_a_grid_has_tiles_for(swiglu):
    """The general kernels take them, as they did before."""
    from tq_kv_b200 import kernels
    N = 64 * 65535 + 1
    x, w = rnd(20, 4), rnd(1000, 4, seed=1).repeat(N // 500 + 1, 1)[:2 * N if swiglu else N]
    out = kernels.linear(x, w, swiglu=swiglu)
    z = x.double() @ w[:1000].double().T                                   # (the weight's rows repeat every 1,000)
    at = torch.tensor([0, 1, 999, 64 * 65535 - 1, N - 1], device=DEV)
    want = z[:, at % 1000]
    if swiglu:
        want = torch.nn.functional.silu(want) * z[:, (at + N) % 1000]
    assert float((out[:, at].double() - want).abs().max()) <= 64 * U * float(want.abs().max())
