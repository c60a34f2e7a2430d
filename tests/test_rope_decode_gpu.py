"""The decode step's attention in one kernel (csrc/rope_decode.cu) beside float64 and the separate kernels: sequences of one
key, of a few, around chunks and pages, windows and rings, every number of splits, dims past the rotated ones, no bias, rows past
their sequence's new length, and which steps come here (GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _setup(lens, nh, nkv, hd, rot, ring=0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, width = len(lens), ring or -(-max(lens) // 64)
    pages = T * width + 3
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(seed))[:T * width].int().reshape(T, width).to(DEV).contiguous()
    ang = torch.rand(max(lens), rot // 2, device=DEV, generator=g) * 6
    return dict(qkv=rnd(T, (nh + 2 * nkv) * hd), bias=rnd((nh + 2 * nkv) * hd), cos=ang.cos(), sin=ang.sin(),
                k=rnd(pages, nkv, 64, hd).bfloat16(), v=rnd(pages, nkv, 64, hd).bfloat16(), table=table, width=width,
                pos=i32([n - 1 for n in lens]), seq=i32(list(range(T))), new=i32(lens), cu=i32(list(range(T + 1))))


def _wanted(s, nh, nkv, hd, rot, window, ring, bias, dtype=torch.bfloat16):
    """float64 from the step's row and the cache; q and the new key and value rounded as they are cached."""
    outs = []
    for t, pos in enumerate(s["pos"].tolist()):
        x = (s["qkv"][t] + (s["bias"] if bias else 0)).double().reshape(nh + 2 * nkv, hd)
        c, n = s["cos"][pos].double(), s["sin"][pos].double()
        h = x[:nh + nkv].clone()
        a, b = x[:nh + nkv, :rot // 2], x[:nh + nkv, rot // 2:rot]
        h[:, :rot // 2], h[:, rot // 2:rot] = a * c - b * n, a * n + b * c
        q, k_new, v_new = h[:nh].to(dtype).double(), h[nh:].to(dtype), x[nh + nkv:].to(dtype)
        lo = max(0, pos - window + 1) if window else 0
        js = torch.arange(lo, pos, device=DEV)
        lp = js // 64 % ring if ring else js // 64
        page = s["table"][t][lp].long()
        k = torch.cat([s["k"][page, :, js % 64], k_new[None]]).double()          # [keys, nkv, hd]
        v = torch.cat([s["v"][page, :, js % 64], v_new[None]]).double()
        rep = nh // nkv
        w = torch.einsum("hd,khd->hk", q, k.repeat_interleave(rep, 1)) / math.sqrt(hd)
        outs.append(torch.einsum("hk,khd->hd", w.softmax(-1), v.repeat_interleave(rep, 1)).reshape(-1))
    return torch.stack(outs)


@pytest.mark.parametrize("nh,nkv,hd,rot", [(14, 2, 64, 64), (28, 4, 64, 62), (4, 4, 32, 16), (16, 1, 32, 32)])
@pytest.mark.parametrize("lens,window,ring", [([1], None, 0), ([17, 2, 16, 33], None, 0), ([64, 65, 300, 1000, 129], None, 0),
                                              ([700, 30, 1], 100, 0), ([700, 130], 100, 3)])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
def test_beside_float64_and_the_separate_kernels(nh, nkv, hd, rot, lens, window, ring, splits):
    from tq_kv_b200 import kernels
    s = _setup(lens, nh, nkv, hd, rot, ring, seed=sum(lens) + hd)
    T, bias = len(lens), splits != 2
    common = dict(n_heads=nh, n_kv_heads=nkv, head_dim=hd)
    want = _wanted(s, nh, nkv, hd, rot, window, ring, bias)
    k0, v0 = s["k"].clone(), s["v"].clone()
    q = torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV)
    kernels.qkv_rope_cache(s["qkv"], s["bias"] if bias else None, s["cos"], s["sin"], s["pos"], s["seq"], s["new"], q, rotary_dim=rot,
                           k_pages=k0, v_pages=v0, block_table=s["table"], table_width=s["width"], ring_pages=ring, **common)
    row = s["qkv"].clone()
    out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    kernels.rope_decode(row, s["bias"] if bias else None, s["cos"], s["sin"], out, rotary_dim=rot, k_pages=s["k"], v_pages=s["v"],
                        block_table=s["table"], table_width=s["width"], ring_pages=ring, page_tokens=64, tok_pos=s["pos"],
                        tok_seq=s["seq"], new_lens=s["new"], window=window, n_splits=splits, clear_input=splits == 4, **common)
    # the new rows, and no others; the rotation's last bit (a product rounded before the sum, or not) may move a key's
    assert torch.equal(s["v"], v0) and float((s["k"].double() - k0.double()).abs().max()) <= 2.0 ** -8 * float(k0.abs().max())
    assert int((s["k"] != k0).sum()) <= 0.01 * T * nkv * hd + 1
    assert bool((row == 0).all()) if splits == 4 else torch.equal(row, s["qkv"])
    # weights are rounded to bfloat16 before they meet the values (2^-9 of a sum of values around one), and so is the result
    assert float((out.double() - want).abs().max()) < 2.0 ** -7 * float(want.abs().max()) + 2.0 ** -8


@pytest.mark.parametrize("nh,nkv,hd,rot", [(14, 2, 64, 64), (28, 2, 64, 62), (4, 4, 32, 16), (16, 1, 32, 32)])
@pytest.mark.parametrize("lens,window,ring", [([1], None, 0), ([33, 2, 32, 64], None, 0), ([65, 300, 1000], None, 0), ([700, 130], 100, 3)])
@pytest.mark.parametrize("splits", [1, 2, 8])
def test_float32_beside_float64_and_the_separate_kernels(nh, nkv, hd, rot, lens, window, ring, splits):
    from tq_kv_b200 import kernels
    s = _setup(lens, nh, nkv, hd, rot, ring, seed=sum(lens) + hd)
    s["k"], s["v"] = s["k"].float(), s["v"].float()
    T, bias = len(lens), s["bias"] if splits != 2 else None
    common = dict(n_heads=nh, n_kv_heads=nkv, head_dim=hd)
    cache = dict(block_table=s["table"], table_width=s["width"], ring_pages=ring)
    want = _wanted(s, nh, nkv, hd, rot, window, ring, bias is not None, torch.float32)
    k0, v0 = s["k"].clone(), s["v"].clone()
    q, apart, out = (torch.full((T, nh * hd), 7.0, device=DEV) for _ in range(3))
    kernels.qkv_rope_cache(s["qkv"], bias, s["cos"], s["sin"], s["pos"], s["seq"], s["new"], q, rotary_dim=rot, k_pages=k0, v_pages=v0,
                           **cache, **common)
    kernels.attention(q, apart, tok_pos=s["pos"], tok_seq=s["seq"], cu_seqlens=s["cu"], start_pos=s["pos"], window=window, k_pages=k0,
                      v_pages=v0, **cache, **common)
    kernels.rope_decode(s["qkv"], bias, s["cos"], s["sin"], out, rotary_dim=rot, k_pages=s["k"], v_pages=s["v"], page_tokens=64,
                        tok_pos=s["pos"], tok_seq=s["seq"], new_lens=s["new"], window=window, n_splits=splits, **cache, **common)
    assert torch.equal(s["v"], v0) and float((s["k"].double() - k0.double()).abs().max()) <= 2.0 ** -22 * float(k0.abs().max())
    err, err_apart = (float((x.double() - want).norm() / want.norm()) for x in (out, apart))
    assert err <= max(1.5 * err_apart, 4e-7), (err, err_apart)       # float32 sums of the same numbers in another order


def test_a_row_past_its_sequences_new_length_is_not_cached():
    from tq_kv_b200 import kernels
    s = _setup([40, 50], 4, 2, 64, 64)
    s["new"][1] = 49
    k, v = s["k"].clone(), s["v"].clone()
    out = torch.empty(2, 256, dtype=torch.bfloat16, device=DEV)
    kernels.rope_decode(s["qkv"], None, s["cos"], s["sin"], out, n_heads=4, n_kv_heads=2, head_dim=64, rotary_dim=64, k_pages=s["k"],
                        v_pages=s["v"], block_table=s["table"], table_width=s["width"], ring_pages=0, page_tokens=64,
                        tok_pos=s["pos"], tok_seq=s["seq"], new_lens=s["new"], window=None, n_splits=2)
    changed = (s["k"] != k).any(-1).any(1).nonzero().tolist()
    assert changed == [[int(s["table"][0, 0]), 39]] and int((s["v"] != v).any(-1).any(1).sum()) == 1


@pytest.mark.parametrize("T,nkv,hd,keys,want", [(1, 4, 64, 2048, 8), (8, 4, 64, 2048, 8), (16, 4, 32, 2048, 4), (64, 4, 64, 2048, 1),
                                                (1, 2, 64, 256, 1), (1, 2, 64, 300, 2), (1, 4, 64, 4160, 0), (64, 4, 64, 32768, 1),
                                                (1, 4, 128, 2048, 0)])
def test_splits(T, nkv, hd, keys, want):
    from tq_kv_b200 import kernels
    assert kernels.rope_decode_splits(T, nkv * 4, nkv, hd, keys, 64, 148) == want
