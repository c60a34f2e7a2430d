"""Matrix products: y = x · W^T with W stored [out, in].

`linear()` picks the kernel from the operands:
  * one row of bfloat16 and weights of middling size, or a head (`_row_takes`): the FMA
    row kernel of csrc/row_gemm.cu;
  * up to 16 rows of bfloat16 and small weights (decoding a small model; the
    limits are in `_tc_takes`): the weight-streaming mma.sync kernel of
    csrc/skinny_gemm.cu, which reads the weight once and fuses bias, SwiGLU
    gating and the float32 accumulation into the residual stream;
  * up to 64 rows of bfloat16 otherwise: the same job on tcgen05, TMA-fed
    (csrc/decode_pair_tc.cu for gated products, see `_pair_takes`; csrc/decode_gemm_tc.cu, with
    swapped operands, for the others);
  * up to 16 rows of anything else: the float32 row kernel of csrc/gemm.cu
    with the same epilogues;
  * many rows, bfloat16 × bfloat16: the TMA + tcgen05 kernels of
    csrc/gemm_tc.cu (pairs of SMs mostly, from 129 rows on) with the same fused epilogues; with USE_TCGEN05 off, the
    library matrix product (cuBLAS through torch.mm with float32 output), as
    the reference engine does for all its products
    (src/models/turbo_generic.rs:68-91 -> candle -> cuBLAS);
  * float32 operands and result (the float32 path): the FMA kernels of
    csrc/gemm_f32.cu with the same epilogues, for up to 8 rows and for more; many rows (`_f32_tc_takes`) on tcgen05
    with every number split exactly into three bfloat16 parts (csrc/gemm_f32_tc.cu);
  * everything else (mixed operands, rows that are not 16-byte aligned): the
    row kernel and the tiled FMA kernel of csrc/gemm.cu.  Never a
    reduced-precision mode.
"""
from __future__ import annotations

import os
from typing import Optional

import torch

from . import elementwise
from ._lib import (KernelError, check, check_tc_status, core, dtype_code, mark, need_contiguous, ptr, stream,
                   tc_status_word)

class PendingNorm:
    """An RMS norm that has not run yet: the float32 rows `h`, the norm's
    float32 weights and eps, and the dtype its result would have.  `linear()`
    takes it in place of activations and, where a decode kernel can, folds
    the norm into the product (the kernel reads h, multiplies with the
    weights while it builds its operand and scales its sums by each row's
    1 / sqrt(mean(h^2) + eps)); otherwise `materialize()` runs the norm's own
    kernel.  (src/models/turbo_generic.rs:41-51 is the norm.)"""

    def __init__(self, h: torch.Tensor, weight: torch.Tensor, eps: float, out_dtype: torch.dtype):
        self.h, self.weight, self.eps, self.out_dtype = h, weight, float(eps), out_dtype
        self._done: Optional[torch.Tensor] = None

    @property
    def shape(self):
        return self.h.shape

    @property
    def device(self):
        return self.h.device

    @property
    def dtype(self):
        return self.out_dtype

    def materialize(self) -> torch.Tensor:
        if self._done is None:
            out = torch.empty(self.h.shape, dtype=self.out_dtype, device=self.h.device)
            self._done = elementwise.rmsnorm(self.h, self.weight, self.eps, out)
            mark("norms")               # a recording timeline books the kernel under the norms, not the product
        return self._done


# Fold a pending norm into the decode products: True wherever a kernel can, False nowhere, "auto" where it was
# measured to pay (see _fused_norm).  TQ_FUSE_NORM=1 / 0 set True / False.
FUSE_NORM = {"1": True, "0": False}.get(os.environ.get("TQ_FUSE_NORM", ""), "auto")
FUSED_NORM_MAX_ROWS = 16
ROW_KERNEL_MAX_ROWS = 16
F32_ROW_KERNEL_MAX_ROWS = 8
SKINNY_MAX_ROWS = 64
# Weights from which a decode product of up to 16 rows runs on the tcgen05 kernel (see _tc_takes)
TC_DECODE_MIN_WEIGHT_BYTES = 24 << 20      # the product after a pending norm
TC_DECODE_MIN_GATED_BYTES = 64 << 20       # gated products
TC_DECODE_GATED_ROWS = 8                   # ... and from 9 rows on from this size
TC_DECODE_MIN_GATED_BYTES_ROWS = 40 << 20
TC_DECODE_MIN_ADDED_BYTES = 4 << 20        # float32 results of given rows, which leave as shares of K
TC_DECODE_ADDED_ROWS = 8                   # ... and these from 9 rows on at any size


def _tc_takes(rows: int, w: torch.Tensor, swiglu: bool, after_norm: bool, float32_out: bool) -> bool:
    """Which of the two decode kernels gets a bfloat16 product that both can run (gated: which one folds a pending norm
    in; without one `_pair_takes` decides): True for the TMA-fed
    tcgen05 kernel, False for the mma.sync one.  Over 16 rows always the former.  Below that by the weight's
    size, with limits that were measured (each product alone in a replayed graph, and the whole decode step
    of the 7B and 0.5B shapes): the product after a pending norm from 24 MB on (below it the mma.sync kernel
    with the norm folded in wins: 6 MB q|k|v 4.4 against 3.8 + a norm kernel); gated products from 64 MB on
    (55 MB at 8 rows: 12.8 against 14.3 us; 90 MB: 21.0 against 20.1), from 9 rows on from 40 MB (behind a norm
    kernel, at 9 / 16 rows: 17 MB 8.9 against 10.0 / 9.0 against 10.7, 34 MB 14.3 against 14.5 / 14.9 against 16.6,
    42 MB with K = 1,024 15.2 against 13.5 / 16.1 against 14.4, 46 MB 20.0 against 16.4 / 21.1 against 17.3); float32 results of rows that are
    given, which the tcgen05 kernel cuts into shares of K that meet in the L2, from 4 MB on and from 9 rows on
    at any size (9 MB with K = 4,864 at 8 rows: 6.1 against 4.5 us, at 16 rows 8.6 against 4.8; 5 MB with
    K = 1,536: 4.5 against 3.2; 1.6 MB at 8 rows: 2.9 against 2.7, a tie left where it was)."""
    if rows > ROW_KERNEL_MAX_ROWS or w.shape[1] % 32:
        return True
    size = w.numel() * 2
    if swiglu:
        return size >= (TC_DECODE_MIN_GATED_BYTES_ROWS if rows > TC_DECODE_GATED_ROWS else TC_DECODE_MIN_GATED_BYTES)
    if after_norm or not float32_out:
        return size >= TC_DECODE_MIN_WEIGHT_BYTES
    return size >= TC_DECODE_MIN_ADDED_BYTES or rows > TC_DECODE_ADDED_ROWS


ROW_GEMM_MIN_BYTES = 16 << 20              # one row: products from this size
ROW_GEMM_MIN_GATED_BYTES = 24 << 20        # (gated products from this one)
ROW_GEMM_MAX_BYTES = 64 << 20              # up to this, beyond it only ...
ROW_GEMM_HEAD_COLUMNS = 16384              # ... with so many columns


def _row_takes(rows: int, w: torch.Tensor, swiglu: bool) -> bool:
    """Which bfloat16 products of one row run on the FMA row kernel (csrc/row_gemm.cu), by the weight's size.  In replayed
    graphs of the same product with other weights, in us, the other kernel / here: 17 MB 8.2 / 4.8 (K = 2,048 and 1,024), 23
    MB 7.1 / 6.5, 25 MB 9.4 / 6.1, 33 MB 10.9 / 7.5 (K = 4,096) and 10.3 / 7.6 (K = 8,192), 35 MB 10.7 / 8.9, 52 MB 13.4 / 11.2;
    gated 46 MB 11.7 / 10.3, 50 MB 15.3 / 10.7, 55 MB 12.8 / 10.8, 59 MB 15.8 / 12.0, 63 MB 22.2 / 13.3; heads of 33 MB 9.0 /
    7.6, 77 MB 18.9 / 15.4, 272 MB 48.8 / 41.5.  Outside: 9 MB 4.2 / 4.4, gated 17 MB 5.0 / 5.4, 136 MB 23.9 / 23.6 (and in
    the 7B shape's step slower: its 3,584 long columns).  Whole passes of a prompt and 24 decoded tokens, in ms, without /
    with these: 7B 72.4 / 71.0, zodosun-2k 20.2 / 18.7, rirudra-2k 9.73 / 8.72.  With the norm made by the row kernel itself
    passes were slower (0.5B 15.9 -> 16.8 ms), two rows gain little (a head 49.1 / 46.5) or lose (26 MB 7.0 / 8.7)."""
    if rows != 1:
        return False
    size = w.numel() * 2
    if not swiglu and w.shape[0] >= ROW_GEMM_HEAD_COLUMNS:
        return size >= ROW_GEMM_MIN_BYTES
    return (ROW_GEMM_MIN_GATED_BYTES if swiglu else ROW_GEMM_MIN_BYTES) <= size <= ROW_GEMM_MAX_BYTES


PAIR_MIN_BYTES_ROWS = 20 << 20             # gated products of 9 to 16 rows: from this size
PAIR_MIN_BYTES = 40 << 20                  # ... of up to 8 rows


def _pair_takes(rows: int, w: torch.Tensor) -> bool:
    """Which gated bfloat16 products of given rows (a norm that is not folded in) run on csrc/decode_pair_tc.cu, by the
    weight's size: all of more than 16 rows, of 9 to 16 rows from 20 MB, of fewer from 40 MB; below, and where K is a multiple of
    32, the mma.sync kernel.  Behind a norm kernel, in replayed graphs with other weights, in us, before / here: 17 MB with
    K = 896 at 8 / 9 / 16 / 32 / 64 rows 6.6 / 8.8 / 9.0 / 11.9 / 14.7 against 9.0 / 9.0 / 9.2 / 9.4 / 10.1; 23 MB 8.7 / 13.1 / 13.7 /
    16.0 / 19.7 against 11.2 / 11.2 / 11.3 / 11.2 / 12.4; 46 MB with K = 2,048 15.7 / 16.3 / 17.1 / 18.1 / 21.1 against 13.5 / 13.5 / 13.7 /
    13.8 / 15.0; 55 MB 15.4 / 15.1 / 16.0 / 17.0 / 19.9 against 13.8 / 14.0 / 14.1 / 15.0 / 16.7; 100 MB 22.6 / 22.7 / 24.2 / 26.2 / 29.5
    against 20.7 / 20.8 / 21.3 / 22.2 / 24.0; 272 MB 44.7 / 44.9 / 46.0 / 47.8 / 52.3 against 45.6 / 45.9 / 46.7 / 48.3 / 51.8; 566 MB 91.6 /
    91.4 / 93.6 / 97.0 / 105.7 against 87.1 / 87.3 / 88.2 / 90.5 / 94.1."""
    size = w.numel() * 2
    if rows > ROW_KERNEL_MAX_ROWS or w.shape[1] % 32:
        return True
    return size >= (PAIR_MIN_BYTES_ROWS if rows > 8 else PAIR_MIN_BYTES)


def _gate(swiglu, activation) -> int:
    """The `swiglu` argument of the C functions: 0 for a plain product, ACT_SQUARE_RELU for a plain one with that
    activation on its result, else the gate's activation code."""
    return int(activation) if swiglu or activation == elementwise.ACT_SQUARE_RELU else 0


def skinny_gemm(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU):
    """bfloat16 x [M <= 64, K] times bfloat16 w [N, K]^T on the tensor cores,
    streaming w once (csrc/skinny_gemm.cu).  K must be a multiple of 32."""
    M, K = x.shape
    N = out.shape[1]
    check(core().tq_skinny_gemm(ptr(x), ptr(w), ptr(bias), ptr(out), dtype_code(out), M, N, K, x.stride(0),
                                w.stride(0), out.stride(0), int(accumulate), _gate(swiglu, activation), stream()),
          "skinny_gemm")
    return out


def row_gemm(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU, w_settled=False):
    """bfloat16 x [1, K] times bfloat16 w [N, K]^T on FMA units, streaming w once (csrc/row_gemm.cu); K a multiple of 8.
    `w_settled`: see `linear`."""
    check(core().tq_row_gemm(ptr(x), ptr(w), ptr(bias), ptr(out), dtype_code(out), out.shape[1], x.shape[1], w.stride(0),
                             int(accumulate), _gate(swiglu, activation), int(w_settled), stream()), "row_gemm")
    return out


# ---- tcgen05 + TMA product for many rows (csrc/gemm_tc.cu) -----------------------
USE_TCGEN05 = True                  # False: the library product (cuBLAS) takes the many-row bfloat16 case
EPI_STORE, EPI_ACCUM, EPI_SWIGLU, EPI_GELU, EPI_RELU2 = 0, 1, 2, 3, 4


def set_gemm_tc_mode(mode: int) -> None:
    """0: products of more than 128 rows run on pairs of SMs (tcgen05 cta_group::2, 256-row tiles) unless their
    last tiles' padding costs too much (csrc/gemm_tc.cu), smaller ones on single SMs; 1: single SMs always;
    2: pairs always.  The default is 0 (or TQ_GEMM_TC_MODE)."""
    if mode not in (0, 1, 2):
        raise KernelError(f"gemm_tc mode {mode}: 0, 1 or 2")
    core().tq_gemm_tc_mode(mode)


def gemm_tc(x, w, out, bias=None, epilogue=EPI_STORE):
    """out (=, +=) x · w^T on the tcgen05 tensor cores; with EPI_SWIGLU w holds
    gate rows then up rows and out = silu(gate) * up (EPI_GELU: the tanh form of gelu on the gate).  bfloat16 operands, K a
    multiple of 8, 16-byte aligned rows."""
    M, K = x.shape
    N = out.shape[1]
    check(core().tq_gemm_tc(ptr(x), ptr(w), ptr(bias), ptr(out), dtype_code(out), M, N, K, x.stride(0), w.stride(0),
                            out.stride(0), epilogue, ptr(tc_status_word(x.device)), stream()), "gemm_tc")
    return out


def decode_gemm_tc(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU):
    """bfloat16 x [M <= 64, K] times w [N, K]^T on the tcgen05 tensor cores
    with the operands swapped (csrc/decode_gemm_tc.cu): the weight streams once
    through TMA, K is split over a thread-block cluster where tiles are few.  Gated products: `decode_pair_tc`."""
    if swiglu:
        return decode_pair_tc(x, w, out, bias, accumulate, activation)
    M, K = x.shape
    N = out.shape[1]
    check(core().tq_decode_gemm_tc(ptr(x), ptr(w), ptr(bias), ptr(out), dtype_code(out), M, N, K, x.stride(0),
                                   w.stride(0), out.stride(0), int(accumulate), _gate(swiglu, activation),
                                   ptr(tc_status_word(x.device)), stream()), "decode_gemm_tc")
    return out


def decode_pair_tc(x, w, out, bias=None, accumulate=False, activation=elementwise.ACT_SILU):
    """out (=, +=) act(x · gate^T) * (x · up^T) for bfloat16 x [M <= 64, K] and w [2N, K] (gate rows, then up rows) on the tcgen05
    tensor cores, the columns cut so that every SM reads the same share of w once (csrc/decode_pair_tc.cu)."""
    M, K = x.shape
    check(core().tq_decode_pair_tc(ptr(x), ptr(w), ptr(bias), ptr(out), dtype_code(out), M, out.shape[1], K, x.stride(0),
                                   w.stride(0), out.stride(0), int(accumulate), int(activation),
                                   ptr(tc_status_word(x.device)), stream()), "decode_pair_tc")
    return out


def _fused_norm(x: "PendingNorm", w, out, bias, accumulate, swiglu, activation=elementwise.ACT_SILU) -> bool:
    """Runs out (=, +=) norm(h) . w^T with the norm folded into a decode product; False if none takes it."""
    h, g = x.h, x.weight
    M, K = h.shape
    if FUSE_NORM == "auto" and _row_takes(M, w, bool(swiglu)):
        return False                                                          # the FMA row kernel's case
    big = _tc_takes(M, w, bool(swiglu), True, out.dtype == torch.float32)     # the tcgen05 kernel's case
    # Measured inside whole decode steps: the tcgen05 kernel gains from the folded norm where it runs in its
    # cluster form anyway (gated products: 7B shape -0.8 % of a step) and loses where the norm costs it the
    # form with independent shares of K (float32 results: +8 %); the mma.sync kernel gains for plain products
    # (0.5B shape -1.5 %) and loses for gated ones, whose registers are scarce (+2 %).
    # (Gated products below 64 MB of 9 to 16 rows: 46 MB 18.0 with the fold, 15.6 and a norm kernel of 2 without.)
    if FUSE_NORM == "auto" and (big != bool(swiglu) or (swiglu and w.numel() * 2 < TC_DECODE_MIN_GATED_BYTES)):
        return False
    if not (FUSE_NORM and USE_TCGEN05 and x.out_dtype == torch.bfloat16 and w.dtype == torch.bfloat16
            and h.dtype == torch.float32 and g.dtype == torch.float32 and 0 < M <= FUSED_NORM_MAX_ROWS
            and h.stride(1) == 1 and h.stride(0) % 4 == 0 and h.data_ptr() % 16 == 0 and g.data_ptr() % 16 == 0
            and g.is_contiguous() and w.stride(0) % 8 == 0 and w.data_ptr() % 16 == 0 and K % 8 == 0
            and out.dtype in (torch.float32, torch.bfloat16) and (not accumulate or out.dtype == torch.float32)
            and (not swiglu or w.shape[0] % 2 == 0)):
        return False
    N = out.shape[1]
    args = (ptr(h), ptr(g), x.eps, ptr(w), ptr(bias), ptr(out), dtype_code(out), M, N, K, h.stride(0), w.stride(0),
            out.stride(0), int(accumulate), _gate(swiglu, activation))
    if big:
        check(core().tq_decode_gemm_tc_norm(*args, ptr(tc_status_word(h.device)), stream()), "decode_gemm_tc_norm")
    else:
        check(core().tq_skinny_gemm_norm(*args, stream()), "skinny_gemm_norm")
    return True


def product_adds_shares(rows: int, w: torch.Tensor, after_norm: bool = True) -> bool:
    """Whether linear() of `rows` bfloat16 rows (the result of a pending norm, or given rows) with `w` and a
    float32 result would run the decode product that cuts K into independent shares and adds them into the
    result (which it clears first, unless told to accumulate).  A caller that keeps a buffer of zeros can then
    ask for accumulation and save the clearing."""
    N, K = w.shape
    if not (USE_TCGEN05 and w.dtype == torch.bfloat16 and 0 < rows <= SKINNY_MAX_ROWS and K % 8 == 0
            and w.stride(0) % 8 == 0 and w.data_ptr() % 16 == 0):
        return False
    if _row_takes(rows, w, False):
        return False                                   # the FMA row kernel takes it
    if not _tc_takes(rows, w, False, after_norm, True):
        return False                                   # the mma.sync kernel takes it
    return bool(core().tq_decode_gemm_tc_adds_shares(N, K))


def _tc_ok(x, w, out, swiglu) -> bool:
    return (USE_TCGEN05 and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[1] % 8 == 0
            and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and (not swiglu or out.shape[1] % 2 == 0) and out.dtype in (torch.float32, torch.bfloat16)
            # the result leaves through TMA: 16-byte aligned base and row stride
            and out.data_ptr() % 16 == 0 and (out.stride(0) * out.element_size()) % 16 == 0)


def _skinny_ok(x, w) -> bool:
    K = x.shape[1]
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_MAX_ROWS
            and K % 32 == 0 and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def gemm_tiled(x, w, out, bias=None, accumulate=False):
    M, K = x.shape
    N = w.shape[0]
    check(core().tq_gemm_tiled(ptr(x), dtype_code(x), ptr(w), dtype_code(w), ptr(bias), ptr(out), dtype_code(out),
                               M, N, K, x.stride(0), w.stride(0), out.stride(0), int(accumulate), stream()),
          "gemm_tiled")
    return out


def gemv_rows(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU):
    M, K = x.shape
    N = out.shape[1]
    check(core().tq_gemv_rows(ptr(x), dtype_code(x), ptr(w), dtype_code(w), ptr(bias), ptr(out), dtype_code(out),
                              M, N, K, x.stride(0), w.stride(0), out.stride(0), int(accumulate),
                              _gate(swiglu, activation), stream()), "gemv_rows")
    return out


F32_TILE_MAX_COLUMNS = 64 * 65535          # column tiles of 64 gate and 64 up columns (128 of a plain product) in a grid


def _f32_ok(x, w, out) -> bool:
    """What csrc/gemm_f32.cu takes: float32 throughout, 16-byte pieces along K, rows that do not overlap, and with more
    rows than the row kernel's no more columns than a grid has tiles for."""
    K = x.shape[1]
    return ((x.shape[0] <= F32_ROW_KERNEL_MAX_ROWS or out.shape[1] <= F32_TILE_MAX_COLUMNS)
            and x.dtype == torch.float32 and w.dtype == torch.float32 and out.dtype == torch.float32 and K % 4 == 0
            and x.stride(0) % 4 == 0 and w.stride(0) % 4 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and (x.shape[0] == 1 or (x.stride(0) >= K and out.stride(0) >= out.shape[1])) and w.stride(0) >= K)


def _f32_tc_takes(rows: int, columns: int, gated: bool) -> bool:
    """Which float32 products run on csrc/gemm_f32_tc.cu (its error against 64 bits is no larger): of more than 128 rows all, of
    more than 32 those with at least 8 tiles of 256 columns (128 of a gated product).  In us, the FMA tiles / there: 300 rows,
    N = K = 896 18.8 / 15.6, N = 1,152 21.6 / 16.3; 100 rows, N = 896, K = 896 11.9 / 14.2 and K = 4,864 37 / 41, N = K = 2,048
    30.7 / 22.2; 64 rows, N = 1,152 12.0 / 13.4, N = K = 2,048 29.9 / 20.6, N = 8,224 56 / 35, N = 151,936 404 / 282; 32 rows, N = 8,224
    33.7 / 33.6, N = K = 2,048 17.6 / 19.6, N = 151,936 237 / 268."""
    return USE_TCGEN05 and (rows > 128 or (rows > 32 and columns > 7 * (128 if gated else 256)))


def gemm_f32_tc(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU, w_settled=False):
    """float32 x [M, K] times w [N, K]^T on the tcgen05 tensor cores, three exact bfloat16 parts a number
    (csrc/gemm_f32_tc.cu).  `w_settled`: see `linear`."""
    M, K = x.shape
    check(core().tq_gemm_f32_tc(ptr(x), ptr(w), ptr(bias), ptr(out), M, out.shape[1], K, x.stride(0), w.stride(0), out.stride(0),
                                int(accumulate), _gate(swiglu, activation), int(w_settled), ptr(tc_status_word(x.device)),
                                stream()), "gemm_f32_tc")
    return out


def gemm_f32(x, w, out, bias=None, accumulate=False, swiglu=False, activation=elementwise.ACT_SILU, w_settled=False):
    """float32 x [M, K] times w [N, K]^T on FMA units (csrc/gemm_f32.cu): up to 8 rows by the kernel that streams w
    once, more by tiles.  `w_settled`: see `linear`."""
    M, K = x.shape
    fn = core().tq_gemv_f32 if M <= F32_ROW_KERNEL_MAX_ROWS else core().tq_gemm_f32
    check(fn(ptr(x), ptr(w), ptr(bias), ptr(out), M, out.shape[1], K, x.stride(0), w.stride(0), out.stride(0),
             int(accumulate), _gate(swiglu, activation), int(w_settled), stream()), "gemm_f32")
    return out


def linear(x: torch.Tensor, w: torch.Tensor, *, bias: Optional[torch.Tensor] = None,
           out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
           accumulate: bool = False, swiglu: bool = False, activation: int = elementwise.ACT_SILU,
           w_settled: bool = False) -> torch.Tensor:
    """y = x · w^T (+ bias); with `swiglu`, w holds gate rows then up rows and
    y = act(x · gate^T) * (x · up^T), act being silu unless `activation` names another; without it and with
    `activation` ACT_SQUARE_RELU, y = max(x · w^T + bias, 0)^2 (not with `accumulate`); with `accumulate`, `out` (float32) gets
    y added to it.  x [M, K], w [N, K] (or [2N, K]); float32 accumulation
    throughout.

    `w_settled`: w was complete before the kernel in front of this product began, as a model's weights are.  The
    product may then start to read it while that kernel still runs; without it float32 products and the row kernel
    wait first.  The bfloat16 decode kernels (up to 64 rows) always read ahead: a bfloat16 w that a kernel of this
    package makes has to have another kernel behind it before its product."""
    pending = x if isinstance(x, PendingNorm) else None
    relu2 = activation == elementwise.ACT_SQUARE_RELU
    if relu2 and (swiglu or accumulate):
        raise KernelError("linear: the square of relu is an activation of plain products that are not accumulated")
    if len(x.shape) != 2 or w.dim() != 2 or x.shape[1] != w.shape[1]:
        raise KernelError(f"linear: shapes {tuple(x.shape)} and {tuple(w.shape)} do not multiply")
    if (pending is None and x.stride(1) != 1) or w.stride(1) != 1:
        raise KernelError("linear: operands must be contiguous along the inner dimension")
    M, K = x.shape
    rows_w = w.shape[0]
    if swiglu and rows_w % 2:
        raise KernelError("linear: a SwiGLU weight needs an even number of rows")
    N = rows_w // 2 if swiglu else rows_w
    if accumulate:
        if out is None or out.dtype != torch.float32:
            raise KernelError("linear: accumulate needs a float32 `out`")
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype or x.dtype, device=x.device)      # (a pending norm has both too)
    if tuple(out.shape) != (M, N) or out.stride(1) != 1:
        raise KernelError(f"linear: out has shape {tuple(out.shape)}, expected {(M, N)}")
    if bias is not None and (bias.dtype != torch.float32 or bias.shape[0] != rows_w):
        raise KernelError("linear: bias must be float32 with one entry per weight row")
    if M == 0:
        return out
    if pending is not None:
        if not relu2 and _fused_norm(pending, w, out, bias, accumulate, swiglu, activation):
            return out
        x = pending.materialize()

    if (_row_takes(M, w, bool(swiglu)) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and K % 8 == 0
            and w.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and out.dtype in (torch.float32, torch.bfloat16) and (not accumulate or out.dtype == torch.float32)):
        return row_gemm(x, w, out, bias, accumulate, swiglu, activation, w_settled)
    # decoding: a TMA-fed tcgen05 kernel or the mma.sync kernel (_pair_takes and _tc_takes say which, where both can)
    if (swiglu and USE_TCGEN05 and M <= SKINNY_MAX_ROWS and _tc_ok(x, w, out, swiglu)
            and (not accumulate or out.dtype == torch.float32) and (not _skinny_ok(x, w) or _pair_takes(M, w))):
        return decode_pair_tc(x, w, out, bias, accumulate, activation)
    if (not swiglu and USE_TCGEN05 and M <= SKINNY_MAX_ROWS and _tc_ok(x, w, out, swiglu)
            and (not accumulate or out.dtype == torch.float32) and not (relu2 and out.dtype != torch.bfloat16)
            and (not _skinny_ok(x, w)
                 or _tc_takes(M, w, False, pending is not None, out.dtype == torch.float32))):
        return decode_gemm_tc(x, w, out, bias, accumulate, False, activation)
    if _skinny_ok(x, w):
        return skinny_gemm(x, w, out, bias, accumulate, swiglu, activation)
    if _f32_ok(x, w, out):
        if _f32_tc_takes(M, N, bool(swiglu)):
            return gemm_f32_tc(x, w, out, bias, accumulate, swiglu, activation, w_settled)
        return gemm_f32(x, w, out, bias, accumulate, swiglu, activation, w_settled)
    if M <= ROW_KERNEL_MAX_ROWS:
        return gemv_rows(x, w, out, bias, accumulate, swiglu, activation)

    if (_tc_ok(x, w, out, swiglu) and (not accumulate or out.dtype == torch.float32)
            and not (relu2 and out.dtype != torch.bfloat16)):
        gated = EPI_GELU if activation == elementwise.ACT_GELU_TANH else EPI_SWIGLU
        plain = EPI_RELU2 if relu2 else (EPI_ACCUM if accumulate else EPI_STORE)
        return gemm_tc(x, w, out, bias, gated if swiglu else plain)

    if x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and bias is None:
        y = torch.mm(x, w.t(), out_dtype=torch.float32)          # library product, float32 out
        if swiglu:
            return elementwise.swiglu(y, out, activation)
        if relu2:
            return elementwise.square_relu(y, out)
        if accumulate:
            return elementwise.add_into(out, y)
        if out.dtype == torch.float32:
            out.copy_(y)
        else:
            out.copy_(y)
        return out

    if swiglu:
        y = torch.empty((M, rows_w), dtype=torch.float32, device=x.device)
        gemm_tiled(x, w, y, bias, False)
        return elementwise.swiglu(y, out, activation)
    if relu2:
        y = out if out.dtype == torch.float32 and out.is_contiguous() else torch.empty((M, N), dtype=torch.float32, device=x.device)
        gemm_tiled(x, w, y, bias, False)
        return elementwise.square_relu(y, out)
    return gemm_tiled(x, w, out, bias, accumulate)
