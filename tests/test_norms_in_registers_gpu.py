"""Group norms and added norms with a row's part in registers (csrc/elementwise.cu): widths at the edges of the forms, every gate,
chosen rows, slices that start off 16 bytes (the general kernels), against float64 (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("gw,groups", [(4, 3), (64, 5), (128, 16), (132, 2), (256, 1), (260, 3), (512, 1), (516, 2), (1024, 2), (1028, 1),
                                       (2048, 1), (2052, 1), (4096, 1), (4100, 1), (130, 3)])
@pytest.mark.parametrize("mode", [None, 0, 1, 2])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_group_norm(gw, groups, mode, dtype):
    from tq_kv_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(gw + groups)
    T, W = 11, gw * groups
    for shift in (0, 1):                                       # 1: rows that start off 16 bytes
        x = torch.randn(T, W + 8, device=DEV, generator=g)[:, shift:shift + W]
        gate = torch.randn(T, W + 4, device=DEV, generator=g)[:, 4 - shift:4 - shift + W] if mode is not None else None
        w = torch.randn(W, device=DEV, generator=g)
        for rows in (None, torch.tensor([10, 0, 3], dtype=torch.int32, device=DEV)):
            out = torch.full((T if rows is None else 3, W), 7.0, device=DEV, dtype=dtype)
            kw = {} if mode is None else {"gate": gate, "gate_mode": mode}
            kernels.group_rmsnorm(x, w, 1e-5, out, groups=groups, rows=rows, **kw)
            v = x.double()
            if mode == 2:
                v = v * torch.nn.functional.silu(gate.double())
            v = v.reshape(T, groups, gw)
            y = (v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(T, W) * w.double()
            if mode == 0:
                y = y * torch.sigmoid(gate.double())
            if mode == 1:
                y = y * torch.nn.functional.silu(gate.double())
            if rows is not None:
                y = y[rows.long()]
            # a sum of gw squares in float32, a root, a quotient and a few products: some 2^-22 of each entry; bfloat16 keeps 2^-9
            room = y.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) + 1e-12
            assert bool(((out.double() - y).abs() <= room).all())


@pytest.mark.parametrize("W", [4, 1024, 1028, 2048, 2052, 4096, 4100, 130])
@pytest.mark.parametrize("n", [1, 2, 3])
def test_added_norms(W, n):
    from tq_kv_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(W + n)
    acc = torch.randn(7, W, device=DEV, generator=g)
    srcs = [(torch.randn(7, W, device=DEV, generator=g) * (k + 1), torch.randn(W, device=DEV, generator=g)) for k in range(n)]
    parts = [x.double() / (x.double().pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * w.double() for x, w in srcs]
    want = acc.double() + 0.5 * sum(parts)
    size = acc.double().abs() + 0.5 * sum(p.abs() for p in parts)
    kernels.add_normed(acc, srcs, 1e-6, 0.5)
    assert bool(((acc.double() - want).abs() <= size * 2.0 ** -20).all())
