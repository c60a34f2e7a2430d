"""The matrix-state scans over steps of many tokens, on both sides of the line between the kernel that goes eight tokens at
a time (csrc/block_scan.cu) and the one that goes token by token (csrc/linear_scan.cu), against float64.  Bound: the sums
of a token are a few hundred float32 terms and the state fades or is overwritten, so errors stay a few 1e-7 of the largest
value; 2e-6 allows for the growth of undamped states."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def whatever_length(monkeypatch):
    """Short sequences too go through the kernel that goes eight at a time (as far as there are few columns)."""
    from tq_kv_b200.kernels import scan
    monkeypatch.setattr(scan, "_long_enough", lambda *a: True)


def i32(x):
    return torch.tensor(list(x), dtype=torch.int32, device=DEV)


def make(mode, lens, H, G, d, e, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    T = sum(lens)

    def rnd(*s):
        return torch.randn(*s, generator=g, device=DEV)

    p = {"q": rnd(T, G * d), "k": rnd(T, G * d), "v": rnd(T, H * e), "state": rnd(len(lens) + 2, H * d * e) * 0.3}
    if mode == "delta":
        p["a"], p["w"] = rnd(T, H * d), rnd(T, H * d) * 2
    elif mode == "decay":
        p["c"] = torch.linspace(0.5, 1.0, H, device=DEV)
    else:
        p["k"] = torch.nn.functional.normalize(p["k"].reshape(T, G, d), dim=-1).reshape(T, -1)
        p["s"] = torch.rand(T, H, 4, generator=g, device=DEV)
        p["s"][..., 0] = p["s"][..., 0] ** 0.2
        p["skip"] = rnd(H)
    return p


def exact(mode, p, lens, slots, H, G, d, e, eps=1e-6):
    T = sum(lens)
    q, k, v = (p[n].double() for n in "qkv")
    if mode == "decay":
        q, k, v = (torch.nn.functional.silu(x) for x in (q, k, v))
    q, k = (x.reshape(T, G, d).repeat_interleave(H // G, 1) for x in (q, k))
    v = v.reshape(T, H, e)
    out, state, t = torch.empty(T, H, e, dtype=torch.float64, device=DEV), p["state"].double().clone(), 0
    if mode == "delta":
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(p["w"].double())).reshape(T, H, d, 1)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + eps)
        na = -(torch.sigmoid(p["a"].double()).reshape(T, H, d) * u)
    for n, slot in zip(lens, slots):
        S = state[slot].reshape(H, d, e)
        for _ in range(n):
            if mode == "delta":
                r = (u[t].unsqueeze(1) @ S)
                S = w[t] * S + na[t].unsqueeze(-1) * r + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
            elif mode == "decay":
                S = p["c"].double().reshape(H, 1, 1) * S + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
            else:
                S = p["s"][t, :, 0].double().reshape(H, 1, 1) * S
                x = v[t] - (k[t].unsqueeze(1) @ S).squeeze(1) if mode == "gated_delta" else v[t]
                S = S + k[t].unsqueeze(-1) * (p["s"][t, :, 1].double().unsqueeze(-1) * x).unsqueeze(1)
            out[t] = (q[t].unsqueeze(1) @ S).squeeze(1)
            if mode == "gated":
                out[t] += p["skip"].double().unsqueeze(-1) * v[t]
            t += 1
        state[slot] = S.reshape(-1)
    return out.reshape(T, H * e), state


def run(mode, p, lens, slots, H, G, d, e, eps=1e-6):
    from tq_kv_b200 import kernels
    T, cu = sum(lens), [0]
    for n in lens:
        cu.append(cu[-1] + n)
    out, state = torch.full((T, H * e), float("nan"), device=DEV), p["state"].clone()
    if mode in ("delta", "decay"):
        cols = [p["q"], p["k"], p["v"]] + ([p["a"]] if mode == "delta" else [])
        kw = dict(decay_logit=p["w"].clone(), off_a=2 * H * d + H * e, unit_eps=eps) if mode == "delta" else dict(head_decay=p["c"], silu=True)
        kernels.linear_scan(torch.cat(cols, 1), state.reshape(-1, H, d, e), i32(cu), i32(slots), out, n_seqs=len(lens), heads=H,
                            key_dim=d, value_dim=e, off_q=0, off_k=H * d, off_v=2 * H * d, **kw)
    else:
        buf = torch.cat([p["q"], p["k"], p["v"]], 1)
        kernels.gated_scan(buf[:, :G * d], buf[:, G * d:2 * G * d], buf[:, 2 * G * d:], p["s"], state, i32(cu), i32(slots), out,
                           n_seqs=len(lens), heads=H, qk_heads=G, key_dim=d, value_dim=e, delta=mode == "gated_delta",
                           skip=p["skip"] if mode == "gated" else None)
    return out, state


MODES = ["delta", "decay", "gated", "gated_delta"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,d,e", [
    ([1, 7, 8, 9, 16, 17, 40], 2, 2, 32, 32), ([70], 4, 2, 128, 128), ([33, 2], 3, 1, 64, 40), ([20, 31], 2, 1, 100, 12),
    ([5, 64], 1, 1, 256, 20), ([9], 2, 2, 6, 132), ([25, 3], 32, 16, 128, 64),      # eight at a time, both forms
    ([9] * 20, 2, 1, 128, 128), ([3, 30] * 30, 4, 4, 40, 24)])                      # token by token
def test_against_float64(mode, lens, H, G, d, e):
    if mode == "delta":
        e = d
    if mode in ("delta", "decay"):
        G = H
    slots = list(range(len(lens) + 1, 1, -1))
    p = make(mode, lens, H, G, d, e, seed=d + e)
    out, state = run(mode, p, lens, slots, H, G, d, e)
    want, want_state = exact(mode, p, lens, slots, H, G, d, e)
    for got, ref in ((out, want), (state, want_state)):
        assert float((got.double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max())
    assert torch.equal(state[0], p["state"][0]) and torch.equal(state[1], p["state"][1])      # slots of no sequence


@pytest.mark.parametrize("mode", ["delta", "gated"])
def test_a_step_cut_into_pieces(mode):
    """More records than one piece takes: the state waits in its slot between the pieces."""
    from tq_kv_b200 import kernels
    H, d, lens = 16, 128, [2500, 700] if mode == "delta" else [3600, 2400]
    floats = kernels._lib.core().tq_scan_floats(1 if mode == "delta" else 2, sum(lens), 2, H, d, d)
    record = (4 if mode == "delta" else 2) * 8 * d + 2 * d + (16 if mode == "delta" else 8) * 8
    all_records = sum(-(-n // 8) for n in lens)
    assert floats * 4 <= 96 << 20 and floats < all_records * H * record          # two pieces
    assert floats // (H * record) < -(-lens[0] // 8)                              # the second sequence starts in the second
    p = make(mode, lens, H, H, d, d, seed=3)
    out, state = run(mode, p, lens, [1, 3], H, H, d, d)
    want, want_state = exact(mode, p, lens, [1, 3], H, H, d, d)
    for got, ref in ((out, want), (state, want_state)):
        assert float((got.double() - ref).abs().max()) <= 4e-6 * float(ref.abs().max())


@pytest.mark.parametrize("mode", MODES)
def test_a_token_changes_nothing_before_it(mode):
    """An infinite value in a later token of the same eight leaves the results before it as they are."""
    lens, H, d = [13], 2, 64
    p = make(mode, lens, H, H, d, d, seed=5)
    out, _ = run(mode, p, lens, [0], H, H, d, d)
    p["v"][5] = float("inf")
    spoiled, _ = run(mode, p, lens, [0], H, H, d, d)
    assert torch.equal(out[:5], spoiled[:5]) and not torch.isfinite(spoiled[5]).any()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 13])
def test_a_unit_key_without_a_floor(n):
    """unit_eps = 0: the tokens that fill a sequence's last eight have no key to divide by."""
    lens, H, d = [n, 20], 2, 64
    p = make("delta", lens, H, H, d, d, seed=n)
    out, state = run("delta", p, lens, [1, 3], H, H, d, d, eps=0.0)
    want, want_state = exact("delta", p, lens, [1, 3], H, H, d, d, eps=0.0)
    for got, ref in ((out, want), (state, want_state)):
        assert float((got.double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max())


@pytest.mark.parametrize("mode", ["delta", "gated_delta"])
def test_an_infinite_state_entry_meets_no_token_that_is_not_there(mode):
    """One token: the other entries of the column become infinite with the sign that their key's removal gives, none NaN."""
    H, d, lens = 2, 64, [1]
    p = make(mode, lens, H, H, d, d, seed=2)
    p["state"].reshape(-1, H, d, d)[1, 0, 5, 9] = float("inf")
    out, state = run(mode, p, lens, [1], H, H, d, d)
    want, want_state = exact(mode, p, lens, [1], H, H, d, d)
    fine = torch.isfinite(want_state)
    assert int((~fine).sum()) == d and int(torch.isnan(want_state).sum()) == 1
    assert torch.equal(torch.isnan(state), torch.isnan(want_state))
    assert torch.equal(state[~fine].nan_to_num(), want_state[~fine].float().nan_to_num())
    assert float((state.double() - want_state)[fine].abs().max()) <= 2e-6 * float(want_state[fine].abs().max())


def one_token(mode, p, state, H, d):
    """A token of each sequence through the kernel for one token; decays, steps and strengths of a half where not given."""
    from tq_kv_b200 import kernels
    T, n = p["q"].shape
    buf, out, cu, slots = torch.cat([p[x] for x in "qkva"], 1), torch.empty(T, n, device=DEV), i32(range(T + 1)), i32(range(T))
    scal = torch.full((T, H, 4), 0.5, device=DEV)
    common = dict(n_seqs=T, heads=H, key_dim=d, value_dim=d, single_tokens=True)
    qkv = (buf[:, :n], buf[:, n:2 * n], buf[:, 2 * n:3 * n])
    if mode in ("delta", "decay"):
        kw = dict(decay_logit=p["w"], off_a=3 * n) if mode == "delta" else dict(head_decay=torch.full((H,), 0.5, device=DEV))
        kernels.linear_scan(buf, state, cu, slots, out, off_q=0, off_k=n, off_v=2 * n, **common, **kw)
    elif mode == "channel_delta":
        kernels.channel_delta_scan(*qkv, torch.sigmoid(p["w"]), scal, state.reshape(T, -1), cu, slots, out, qk_heads=H, **common)
    else:
        kernels.gated_scan(*qkv, scal, state.reshape(T, -1), cu, slots, out, qk_heads=H, delta=mode == "gated_delta", **common)
    return state, out


@pytest.mark.parametrize("d", [6, 40, 100, 200])
@pytest.mark.parametrize("mode", MODES + ["channel_delta"])
@pytest.mark.parametrize("n", [1, 320])
def test_one_token_with_an_infinite_value(mode, d, n):
    """Key widths short of the kernel's: the keys that fill them up stay out of the sums (0 * inf is no 0)."""
    H, g = 2, torch.Generator(device=DEV).manual_seed(d)
    p = {x: torch.rand(n, H * d, generator=g, device=DEV) + 0.1 for x in "qkvaw"}
    p["v"][-1, 3] = float("inf")
    state, out = one_token(mode, p, torch.zeros(n, H, d, d, device=DEV), H, d)
    assert float(out[-1, 3]) == float("inf") and bool((state[-1, 0, :, 3] == float("inf")).all())
    assert int((~torch.isfinite(out)).sum()) == 1 and int((~torch.isfinite(state)).sum()) == d


@pytest.mark.parametrize("d,H,n", [(32, 2, 1), (32, 4, 200), (64, 2, 3), (64, 4, 80), (128, 2, 3), (128, 16, 8), (128, 8, 40), (256, 2, 2),
                                   (256, 4, 20), (6, 2, 2), (6, 4, 170), (40, 2, 2), (40, 4, 100), (100, 2, 2), (100, 8, 40), (200, 1, 3),
                                   (200, 4, 30)])
@pytest.mark.parametrize("mode", MODES + ["channel_delta"])
def test_one_token_against_float64(mode, d, H, n):
    """Whole and other widths, from a few blocks to more than four an SM."""
    g = torch.Generator(device=DEV).manual_seed(d + n)
    p = {x: torch.randn(n, H * d, generator=g, device=DEV) for x in "qkvaw"}
    p["k"] = torch.nn.functional.normalize(p["k"].reshape(n, H, d), dim=-1).reshape(n, -1)
    before = torch.randn(n, H, d, d, generator=g, device=DEV)
    state, out = one_token(mode, p, before.clone(), H, d)
    q, k, v, a, w = (p[x].double().reshape(n, H, d) for x in "qkvaw")
    S = before.double()
    if mode == "delta":
        w, u = torch.exp(-math.exp(-0.5) * torch.sigmoid(w)), k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S = w[..., None] * S - (torch.sigmoid(a) * u)[..., None] * (u[:, :, None] @ S) + k[..., None] * v[:, :, None]
    else:
        S = S * (torch.sigmoid(w)[..., None] if mode == "channel_delta" else 0.5)
        x = v if mode == "decay" else 0.5 * (v - (k[:, :, None] @ S)[:, :, 0] if "delta" in mode else v)
        S = S + k[..., None] * x[:, :, None]
    want = (q[:, :, None] @ S)[:, :, 0].reshape(n, -1)
    for got, ref in ((out, want), (state, S)):
        assert float((got.double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max())


@pytest.mark.parametrize("mode", MODES)
def test_no_less_exact_than_token_by_token(mode, monkeypatch):
    """The errors of both kernels against float64, in the norm.  Slow constant decays are the hardest: a rounding of their
    product over eight tokens is the same for each record and adds up over all that the state remembers."""
    from tq_kv_b200.kernels import scan
    lens, H, d = [803], 2, 128
    p = make(mode, lens, H, H, d, d, seed=7)
    if mode == "decay":
        p["c"] = torch.tensor([0.9, 0.996], device=DEV)
    want, want_state = exact(mode, p, lens, [0], H, H, d, d)
    errors = []
    for records in (scan._records, lambda *a: None):
        monkeypatch.setattr(scan, "_records", records)
        out, state = run(mode, p, lens, [0], H, H, d, d)
        errors.append([float((out.double() - want).norm() / want.norm()),
                       float((state[0].double() - want_state[0]).norm() / want_state[0].norm())])
    eight, one = errors
    assert eight[0] <= 1.1 * one[0] and eight[1] <= 1.1 * one[1], errors
