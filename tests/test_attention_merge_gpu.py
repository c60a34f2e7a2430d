"""The merge of the splits of an attention's keys (csrc/attention.cu) against float64: numbers of splits on both sides of
what a thread asks for ahead (8 for each group of threads), widths with one and several groups, splits without keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(hd, n_splits, starts, dtype, sink=None, shift=0, seed=0):
    """One token of each sequence over the general kernel in `n_splits`; (result, float64 reference)."""
    from tq_kv_b200 import kernels
    H, B, g = 3, len(starts), torch.Generator().manual_seed(seed + hd)
    width = max(s // 64 + 1 for s in starts)
    i32 = lambda x: torch.tensor(list(x), dtype=torch.int32, device=DEV)  # noqa: E731
    k, v = (torch.randn(B * width, 1, 64, hd, generator=g).to(dtype).to(DEV) for _ in range(2))
    q = torch.randn(B, H * hd, generator=g).to(dtype).to(DEV)
    table = i32(list(range(B * width))).reshape(B, width)
    out = torch.full((B * H * hd + shift,), float("nan"), dtype=dtype, device=DEV)[shift:].view(B, H * hd)
    scratch = torch.full((B * H * n_splits * (hd + 2),), float("nan"), device=DEV)
    kernels.attention_ext(q, out, n_heads=H, n_kv_heads=1, key_dim=hd, value_dim=hd, tok_pos=i32(starts), tok_seq=i32(range(B)),
                          cu_seqlens=i32(range(B + 1)), start_pos=i32(starts), scale=hd ** -0.5, k_pages=k, v_pages=v,
                          block_table=table, table_width=width, n_splits=n_splits, scratch=scratch, use_fast=False,
                          sink=False if sink is None else sink)
    want = torch.empty(B, H * hd, dtype=torch.float64, device=DEV)
    for b, p in enumerate(starts):
        kk, vv = (x[table[b].long()].reshape(-1, hd)[:p + 1].double() for x in (k, v))
        s = q[b].double().reshape(H, hd) @ kk.T * hd ** -0.5
        if sink is not None:
            s = torch.cat([s, sink.double().reshape(-1, 1)], 1)
        want[b] = (s.softmax(-1)[:, :p + 1] @ vv).reshape(-1)
    return out, want


def within(out, want, dtype):
    """float32: a few hundred roundings of sums of up to 5,000 terms of size 1; bfloat16: half an ulp beside that."""
    half_ulp = 2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0
    assert bool(((out.double() - want).abs() <= half_ulp + 2e-5).all())


@pytest.mark.parametrize("dtype,shift", [(torch.bfloat16, 1), (torch.float32, 1), (torch.float32, 2), (torch.bfloat16, 2)])
@pytest.mark.parametrize("hd", [64, 200])
def test_a_result_that_starts_between_two_pairs(hd, dtype, shift):
    out, want = run(hd, 3, [400, 5, 130], dtype, shift=shift)
    within(out, want, dtype)


@pytest.mark.parametrize("hd,n_splits", [(64, 64), (128, 64), (128, 65), (200, 33), (256, 32), (256, 33), (256, 64), (512, 16),
                                         (512, 17), (512, 40), (512, 64)])
@pytest.mark.parametrize("with_sink", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_more_splits_than_are_asked_for_ahead(hd, n_splits, with_sink, dtype):
    """Beside a long sequence whose splits all hold keys, short ones whose last splits hold none."""
    sink = torch.tensor([0.5, -1.0, 3.0], device=DEV) if with_sink else None
    out, want = run(hd, n_splits, [4500, 70, 0, 900], dtype, sink=sink)
    within(out, want, dtype)
