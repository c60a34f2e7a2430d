"""Decode attention over cached rows that are keys and values at once and wider than 128 entries (csrc/flash_decode.cu):
against float64 and beside the general kernel, whose float32 weights it keeps (three bfloat16 parts a weight).  The
result is rounded to bfloat16 once: half an ulp, up to 2^-8 of the value (8 significant bits); the scores and sums are float32 (their rounding,
about 1e-6 of a score, moves a weight by as much)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).to(DEV)


def case(hd, heads, starts, lens, seed, sharp=1.0):
    """Sequences that hold starts[b] rows and bring lens[b] more, on shuffled pages."""
    total = [s + n for s, n in zip(starts, lens)]
    width = max(-(-t // 64) for t in total)
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(len(starts) * width + 3, generator=g).to(torch.int32)
    table = perm[:len(starts) * width].reshape(len(starts), width).to(DEV)
    pages = rnd(len(perm), 1, 64, hd, seed=seed + 1)
    T = sum(lens)
    q = rnd(T, heads * hd, seed=seed + 2, scale=sharp)
    seqs = [b for b, n in enumerate(lens) for _ in range(n)]
    poss = [starts[b] + i for b, n in enumerate(lens) for i in range(n)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = i32([sum(lens[:b]) for b in range(len(lens) + 1)])
    return q, pages, table, width, i32(poss), i32(seqs), cu, i32(starts)


def exact(q, pages, table, poss, seqs, heads, hd, scale, window, sink):
    out = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for t, (p, b) in enumerate(zip(poss.tolist(), seqs.tolist())):
        rows = pages[table[b].long()].reshape(-1, hd)[:p + 1].double()
        s = q[t].double().reshape(heads, hd) @ rows.T * scale
        if window:
            s[:, :max(0, p - window + 1)] = -math.inf
        if sink is not None:
            s = torch.cat([s, sink.double().reshape(-1, 1)], 1)
        w = s.softmax(-1)[:, :p + 1]
        out[t] = (w @ rows).reshape(-1)
    return out


@pytest.mark.parametrize("hd", [192, 256])
@pytest.mark.parametrize("heads", [1, 5, 16, 24, 32])
@pytest.mark.parametrize("n_splits", [1, 3])
@pytest.mark.parametrize("window,with_sink", [(None, False), (70, True)])
def test_against_float64_and_the_general_kernel(hd, heads, n_splits, window, with_sink):
    from tq_kv_b200 import kernels
    starts, lens = [0, 15, 16, 63, 64, 127, 300, 1000], [1, 1, 2, 1, 3, 1, 20, 1]
    q, pages, table, width, poss, seqs, cu, st = case(hd, heads, starts, lens, seed=hd + heads, sharp=2.0)
    T, scale = q.shape[0], hd ** -0.5
    sink = torch.randn(heads, generator=torch.Generator().manual_seed(9)).to(DEV) if with_sink else None
    scratch = torch.empty(kernels.split_scratch_floats(T, heads, hd, n_splits) + 1, device=DEV)
    want = exact(q, pages, table, poss, seqs, heads, hd, scale, window, sink)
    common = dict(n_heads=heads, n_kv_heads=1, tok_pos=poss, tok_seq=seqs, cu_seqlens=cu, start_pos=st, window=window,
                  scale=scale, k_pages=pages, v_pages=pages, block_table=table, table_width=width, n_splits=n_splits,
                  scratch=scratch)
    got = {}
    for fast in (True, False):
        out = torch.full_like(q, float("nan"))
        if with_sink:
            kernels.attention_ext(q, out, key_dim=hd, value_dim=hd, sink=sink, use_fast=fast, **common)
        else:
            kernels.attention(q, out, head_dim=hd, use_flash=fast, **common)
        got[fast] = (out.double() - want).abs()
    # half an ulp of bfloat16, and 2e-5 for float32 scores of up to about 20 whose rounding enters the weights
    assert bool((got[True] <= 2.0 ** -8 * want.abs() + 2e-5).all())
    assert float(got[True].norm()) <= 1.02 * float(got[False].norm())     # no less exact than the general kernel


def test_a_weight_keeps_its_24_bits():
    """Two weights of about 0.71 that differ by 2^-12 of themselves, with values of 1 and -1: the mean is their small
    difference.  Weights of one bfloat16 part would be 20 times off, of two parts 1.2 % (computed on the CPU); of three the
    result's own rounding (2^-9) is what is left, and the exponential's, 1e-7 of the weights or 5e-4 of the difference."""
    from tq_kv_b200 import kernels
    hd = 256
    rows = torch.zeros(1, 1, 64, hd, device=DEV)
    rows[0, 0, :3, 0] = torch.tensor([3.125, 0.375, 0.375 - 2.0 ** -9])
    rows[0, 0, 1, 1], rows[0, 0, 2, 1] = 1.0, -1.0
    pages = rows.to(torch.bfloat16)
    assert torch.equal(pages.float(), rows)
    q = torch.zeros(1, hd, device=DEV, dtype=torch.bfloat16)
    q[0, 0] = 0.125
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    out = torch.empty_like(q)
    kernels.attention(q, out, n_heads=1, n_kv_heads=1, head_dim=hd, tok_pos=i32([2]), tok_seq=i32([0]), cu_seqlens=i32([0, 1]),
                      start_pos=i32([2]), window=None, scale=1.0, k_pages=pages, v_pages=pages, block_table=i32([[0]]),
                      table_width=1)
    r = pages[0, 0, :3].double()
    want = (0.125 * r[:, 0]).softmax(0) @ r
    assert float((out[0].double() - want).abs()[1]) <= 2.0 ** -8 * float(want[1].abs())


def common_args(hd, heads, q_pages, poss, seqs, cu, st, width, table):
    return dict(n_heads=heads, n_kv_heads=1, head_dim=hd, tok_pos=poss, tok_seq=seqs, cu_seqlens=cu, start_pos=st, window=None,
                k_pages=q_pages, v_pages=q_pages, block_table=table, table_width=width)


@pytest.mark.parametrize("hd", [192, 256])
def test_rows_that_the_kernel_in_front_writes(hd):
    """All cached rows, not the newest alone, come from a kernel that lets its successor start before it has written them."""
    from tq_kv_b200 import kernels
    q, pages, table, width, poss, seqs, cu, st = case(hd, 16, [3000] * 8, [1] * 8, seed=hd)
    scratch = torch.empty(kernels.split_scratch_floats(8, 16, hd, 6) + 1, device=DEV)
    g, flat = torch.ones(hd, device=DEV), pages.view(-1, hd)
    for i in range(5):
        rows = torch.randn(flat.shape, generator=torch.Generator().manual_seed(i)).to(DEV)
        out = torch.empty_like(q)
        torch.cuda.synchronize()
        kernels.rmsnorm(rows, g, 1e-6, flat)
        kernels.attention(q, out, n_splits=6, scratch=scratch, **common_args(hd, 16, pages, poss, seqs, cu, st, width, table))
        want = exact(q, pages, table, poss, seqs, 16, hd, hd ** -0.5, None, None)
        assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5).all())


@pytest.mark.parametrize("hd", [192, 256])
def test_a_query_off_the_16_byte_boundary(hd):
    """The general kernel takes it, as it did before these rows had a kernel of their own."""
    from tq_kv_b200 import kernels
    q, pages, table, width, poss, seqs, cu, st = case(hd, 5, [0, 70, 300], [1, 1, 1], seed=1)
    shifted = torch.empty(q.numel() + 1, dtype=q.dtype, device=DEV)[1:].view(q.shape).copy_(q)
    assert shifted.data_ptr() % 16 and shifted.is_contiguous()
    got, aligned = torch.empty_like(q), torch.empty_like(q)
    kw = common_args(hd, 5, pages, poss, seqs, cu, st, width, table)
    kernels.attention(shifted, got, **kw)
    kernels.attention(q, aligned, use_flash=False, **kw)
    assert torch.equal(got, aligned)
    ext = {k: v for k, v in kw.items() if k != "head_dim"}
    kernels.attention_ext(shifted, got, key_dim=hd, value_dim=hd, scale=hd ** -0.5, **ext)
    assert torch.equal(got, aligned)


@pytest.mark.parametrize("hd", [192, 256])
@pytest.mark.parametrize("n_splits", [1, 4])
@pytest.mark.parametrize("softcap", [None, 50.0])
def test_parts_that_leave_unmerged_come_from_the_general_kernel(hd, n_splits, softcap):
    """They are float32 results, and its sums are the more exact ones."""
    from tq_kv_b200 import kernels
    H = 16
    q, pages, table, width, poss, seqs, cu, st = case(hd, H, [3000, 500, 64, 40], [1] * 4, seed=hd)
    got = [kernels.attention_ext(q, None, n_heads=H, n_kv_heads=1, key_dim=hd, value_dim=hd, tok_pos=poss, tok_seq=seqs,
                                 cu_seqlens=cu, start_pos=st, scale=hd ** -0.5, softcap=softcap, k_pages=pages, v_pages=pages,
                                 block_table=table, table_width=width, n_splits=n_splits, unmerged=True, use_fast=fast)
           for fast in (True, False)]
    assert got[0][2] == got[1][2] == n_splits and torch.equal(got[0][1], got[1][1])
    full = got[0][1].reshape(4, H, n_splits, 2)[..., 1] > 0                # (a split without keys holds nothing)
    assert torch.equal(got[0][0].reshape(4, H, n_splits, hd)[full], got[1][0].reshape(4, H, n_splits, hd)[full])


@pytest.mark.parametrize("hd", [192, 256])
def test_a_cap_on_the_scores(hd):
    from tq_kv_b200 import kernels
    H, starts = 16, [700, 64]
    q, pages, table, width, poss, seqs, cu, st = case(hd, H, starts, [1] * 2, seed=hd, sharp=3.0)
    out = torch.empty_like(q)
    kernels.attention_ext(q, out, n_heads=H, n_kv_heads=1, key_dim=hd, value_dim=hd, tok_pos=poss, tok_seq=seqs, cu_seqlens=cu,
                          start_pos=st, scale=hd ** -0.5, softcap=20.0, k_pages=pages, v_pages=pages, block_table=table,
                          table_width=width)
    for t, p in enumerate(starts):
        rows = pages[table[t].long()].reshape(-1, hd)[:p + 1].double()
        want = ((20.0 * torch.tanh(q[t].double().reshape(H, hd) @ rows.T * hd ** -0.5 / 20.0)).softmax(-1) @ rows).reshape(-1)
        assert bool(((out[t].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5).all())
