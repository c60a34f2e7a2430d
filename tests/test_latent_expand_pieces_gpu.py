"""The heads' results from their latents (csrc/latent_attention.cu), whole heads a block and in pieces of 16 results: widths at the
pieces' edges, odd ranks, few and many tokens, every gate, against float64 (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("e", [1, 15, 16, 17, 35, 128])
@pytest.mark.parametrize("T,H", [(1, 2), (3, 16), (400, 3)])
@pytest.mark.parametrize("n,rp", [(33, 40), (512, 576)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_beside_float64(e, T, H, n, rp, dtype):
    from tq_kv_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(e + T + n)
    lat = torch.randn(T, H * rp, device=DEV, generator=g).to(dtype)
    uv = torch.randn(H * e, n, device=DEV, generator=g).to(dtype)
    lats = lat.double().reshape(T, H, rp)[..., :n]
    want = torch.einsum("thn,hen->the", lats, uv.double().reshape(H, e, n))
    size = torch.einsum("thn,hen->the", lats.abs(), uv.double().abs().reshape(H, e, n))
    for head_gate in (None, False, True):
        gate = None if head_gate is None else torch.randn(T, (H if head_gate else H * e) + 3, device=DEV, generator=g)[:, 3:]
        z = 1.0 if gate is None else torch.sigmoid(gate.double()).reshape(T, H, -1)
        out = torch.full((T, H * e), 7.0, device=DEV, dtype=dtype)
        kernels.latent_expand(lat, uv, out, heads=H, kv_rank=n, row_width=rp, value_dim=e, gate=gate, head_gate=bool(head_gate))
        # n / 32 additions a lane and five between lanes in float32, the gate, and the result's rounding
        room = (n / 32 + 8) * 2.0 ** -23 * size * z + (want * z).abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20)
        assert bool(((out.double().reshape(T, H, e) - want * z).abs() <= room + 1e-30).all())
