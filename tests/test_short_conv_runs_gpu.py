"""Convolutions of steps of several tokens in runs of eight (csrc/short_conv.cu): runs that span sequences, sequences shorter than
the taps, inputs from the state, vectors narrower than a warp's, unit length, and operands that the other kernel takes; against
float64, the state after the step included (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lens", [[2], [1, 7, 1], [8, 9], [30, 3, 1, 2, 17], [100]])
@pytest.mark.parametrize("C,regions", [(384, [(0, 128, 128, True, 0.25), (128, 128, 128, True, 1.0), (256, 128, 128, False, 1.0)]),
                                       (200, [(0, 200, 128, False, 1.0)]), (96, [(0, 64, 32, True, 2.0), (64, 32, 16, False, 1.0)]),
                                       (130, [(0, 130, 128, False, 1.0)])])
@pytest.mark.parametrize("K,with_bias", [(4, True), (4, False), (3, True)])
def test_beside_float64(lens, C, regions, K, with_bias):
    from tq_kv_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + C + K)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    T, B, H = sum(lens), len(lens), 3
    wide, w, bias = rnd(T, C + 12), rnd(C, K), rnd(C) if with_bias else None
    x = wide[:, 4:4 + C]
    state = rnd(B + 2, 40 + (K - 1) * C)
    before, slots = state.clone(), [B + 1 - b for b in range(B)]
    gate, beta, a_log, dt = rnd(T, H), rnd(T, H), rnd(H), rnd(H)
    out, scal = torch.full((T, C), 7.0, device=DEV), torch.empty(T, H, 4, device=DEV)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    kernels.short_conv(x, w, bias, out, state[:, 40:], tok_seq=i32([b for b, n in enumerate(lens) for _ in range(n)]), cu_seqlens=i32(cu),
                       slots=i32(slots), n_seqs=B, regions=regions, silu=True, single_tokens=False, unit_eps=1e-6, gate_raw=gate,
                       beta_raw=beta, a_log=a_log, dt_bias=dt, scalars=scal)
    for b, n in enumerate(lens):
        past = before[slots[b], 40:].reshape(K - 1, C)
        rows = torch.cat([past, x[cu[b]:cu[b + 1]]]).double()
        y = sum(rows[j:j + n] * w[:, j].double() for j in range(K)) + (bias.double() if with_bias else 0)
        y = torch.nn.functional.silu(y)
        for first, count, width, unit, scale in regions:
            if unit:
                v = y[:, first:first + count].reshape(n, -1, width)
                y[:, first:first + count] = (v * scale / (v.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()).reshape(n, count)
        # a sum of five terms around one, silu and a quotient in float32
        assert float((out[cu[b]:cu[b + 1]].double() - y).abs().max()) < 2e-6 * max(1.0, float(y.abs().max()))
        assert torch.equal(state[slots[b], 40:].reshape(K - 1, C), rows[n:].float())
    sp = torch.nn.functional.softplus(gate.double() + dt.double())
    assert float((scal[..., 0].double() - torch.exp(-torch.exp(a_log.double()) * sp)).abs().max()) < 1e-5
    assert float((scal[..., 1].double() - torch.sigmoid(beta.double())).abs().max()) < 1e-6
    untouched = [r for r in range(B + 2) if r not in slots]
    assert torch.equal(state[untouched], before[untouched]) and torch.equal(state[:, :40], before[:, :40])
