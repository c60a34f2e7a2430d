"""Float32 prompt attention (csrc/prompt_attention_f32.cu) beside float64 and the general kernel: blocks of tokens that span
sequences, pieces of 32 keys and their remainders, windows, keys from pages and rings, one to 64 q heads a key head, values that
are no numbers (GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(lens, starts, nh, nkv, hd, window, paged, ring=0, odd=None, seed=0):
    from tq_kv_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(seed + sum(lens) + hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    T, B = sum(lens), len(lens)
    seq = [b for b, n in enumerate(lens) for _ in range(n)]
    pos = [s + i for n, s in zip(lens, starts) for i in range(n)]
    ends = [s + n for n, s in zip(lens, starts)]
    keys = [(rnd(e, nkv, hd), rnd(e, nkv, hd)) for e in ends]
    if odd is not None:
        keys[0][1][-1] = odd                                   # the last key's value: only its own row may see it
    q = rnd(T, nh * hd)
    kw = dict(n_heads=nh, n_kv_heads=nkv, head_dim=hd, tok_pos=i32(pos), tok_seq=i32(seq),
              cu_seqlens=i32([0] + torch.tensor(lens).cumsum(0).tolist()), start_pos=i32(starts), window=window)
    if paged:
        width = ring or -(-max(ends) // 64)
        pages = [torch.zeros(B * width, nkv, 64, hd, device=DEV) for _ in range(2)]
        table = torch.randperm(B * width, generator=torch.Generator().manual_seed(1)).int().reshape(B, width).to(DEV)
        for b, kv in enumerate(keys):
            js = torch.arange(max(0, ends[b] - width * 64) if ring else 0, ends[b], device=DEV)
            for p, x in zip(pages, kv):
                p[table[b][js // 64 % width].long(), :, js % 64] = x[js]
        kw |= dict(k_pages=pages[0], v_pages=pages[1], block_table=table, table_width=width, ring_pages=ring)
    else:
        kw |= dict(k_packed=torch.cat([k for k, _ in keys]).reshape(T, -1), v_packed=torch.cat([v for _, v in keys]).reshape(T, -1))
    out, general = torch.full_like(q, 7.0), torch.empty_like(q)
    kernels.attention(q, out, **kw)
    kernels.attention(q, general, use_flash=False, **kw)
    want = []
    for t in range(T):
        lo = max(0, pos[t] - window + 1) if window else 0
        k, v = (x[lo:pos[t] + 1].double().repeat_interleave(nh // nkv, 1) for x in keys[seq[t]])
        w = torch.einsum("hd,khd->hk", q[t].double().reshape(nh, hd), k) / math.sqrt(hd)
        want.append(torch.einsum("hk,khd->hd", w.softmax(-1), v).reshape(-1))
    return out, general, torch.stack(want)


@pytest.mark.parametrize("nh,nkv,hd", [(14, 2, 64), (4, 4, 128), (32, 2, 32), (64, 1, 96)])
@pytest.mark.parametrize("lens,starts,window,paged,ring", [
    ([2], [0], None, False, 0), ([33, 1, 65, 7], [0, 0, 0, 0], None, False, 0), ([150, 150], [0, 0], 40, False, 0),
    ([70, 3], [100, 0], None, True, 0), ([60, 30], [300, 31], 50, True, 2)])
def test_beside_float64_and_the_general_kernel(nh, nkv, hd, lens, starts, window, paged, ring):
    out, general, want = _run(lens, starts, nh, nkv, hd, window, paged, ring)
    err, err_general = (float((x.double() - want).norm() / want.norm()) for x in (out, general))
    # float32 sums of the same numbers in another order
    assert err <= max(1.5 * err_general, 4e-7), (err, err_general)


@pytest.mark.parametrize("odd", [math.inf, math.nan])
def test_a_value_that_is_no_number_stays_with_the_rows_that_see_it(odd):
    out, general, want = _run([40, 20], [0, 0], 14, 2, 64, None, False, odd=odd)
    assert torch.equal(out.isfinite(), general.isfinite()) and int((~out.isfinite()).any(-1).sum()) == 1
    ok = want.isfinite()
    assert float((out.double() - want)[ok].abs().max()) < 1e-5
