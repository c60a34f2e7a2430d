// The matrix-state recurrences of linear_scan.cu over steps of many tokens, eight tokens at a time.
//
// All four rules have the form (per head, S a d x e float32 state)
//
//   r_t = b_t^T S_{t-1},     S_t = diag(w_t) S_{t-1} + n_t r_t + x_t v_t,     o_t = S_t^T q_t  (+ skip v_t)
//
//   SCAN_DECAY         w = c_head,  x = k                              (no r)
//   SCAN_DELTA         w per channel, b = u = k / sqrt(|k|^2 + eps), n = -(a * u), x = k
//   SCAN_GATED         w = g_t,  x = dt_t k                            (no r)
//   SCAN_GATED_DELTA   w = g_t,  b = k,  n = -(beta_t g_t) k,  x = beta_t k
//
// Token by token that is a chain of dependent passes over the state.  For tokens 0 .. 7 with the state S before them,
// w_{a..b} the product of the decays of tokens a .. b (entry by entry; 1 if empty):
//
//   r_i = P_i^T S + sum_{j<i} F_ij v_j         P_i = w_{0..i-1} * b_i + sum_{j<i} A_ij P_j,   A_ij = b_i . (w_{j+1..i-1} * n_j)
//                                              F_ij = B_ij + sum_{j<m<i} A_im F_mj,          B_ij = b_i . (w_{j+1..i-1} * x_j)
//   o_i = Q_i^T S + sum_{j<=i} E_ij v_j        Q_i = w_{0..i} * q_i + sum_{j<=i} C_ij P_j,    C_ij = q_i . (w_{j+1..i} * n_j)
//                                              E_ij = D_ij + sum_{j<m<=i} C_im F_mj,         D_ij = q_i . (w_{j+1..i} * x_j)
//   S' = diag(w_{0..7}) S + sum_j N_j r_j + X_j v_j,      N_j = w_{j+1..7} * n_j,   X_j = w_{j+1..7} * x_j
//
// so that all 16 products with the state are independent of one another and the chain is one step in eight.  All float32.
// Decays enter as products: nothing overflows however fast a head fades.  Only the sums A to D of SCAN_DELTA, whose decays
// differ by channel, take the decays between two tokens as a quotient of two products; that is sound because eight of its
// decays are at least 0.008 (block_prepare), and is not for a decay per channel without such a bound.
//
// block_prepare   a block per (eight tokens, head), a thread a key channel, makes P, Q, N, X, the decays' product and the
//                 rows of F and E once for all columns, as one record; it also makes w, u and a * u from their logits
//                 and applies silu.
//                 The records of a step start at each sequence's first token; the last one of a sequence is filled up
//                 with tokens that change nothing (w = 1, all vectors 0).
// block_scan      a block owns some columns of one head of one sequence and walks the records in order, every thread 4
//                 keys (8 of rows over 128) x RC columns of the state in registers, the records three stages deep in shared memory
//                 (cp.async).  The sums over the KG lanes that share a column are made by trading halves of the values,
//                 so that each lane ends with the few sums that it completes (F v, E v) and hands on.
//
// Rounding.  Eight tokens' decays are one factor here, and a rounding of it that is the same for every record (a constant
// decay) would not average out over the tokens that a slow decay remembers: the factor is kept as hi + lo, and so are the
// products of decays that go into the vectors; the Gram sums are compensated.  But for the delta rule with a decay per
// channel the eight changes of the state are summed before they meet it.  Error of results / states against 64 bits, in
// 1e-7 of their norm, 1,200 tokens of 4 heads of 128 x 128, token by token -> here (without these): delta rule 0.99 / 0.68 ->
// 0.99 / 0.66 (1.34 / 0.71), one decay per token 1.02 / 0.76 -> 0.95 / 0.69 (1.28 / 0.94), with the delta rule 1.05 / 0.79
// -> 1.03 / 0.70 (1.38 / 1.04), constant decays of 0.875 to 0.996 0.82 / 2.78 -> 0.74 / 1.04 (6.44 / 7.63).
//
// What bounds it: the latency from one record to the next (the exchange over the lanes, the completed sums through shared
// memory and back: about 1.3 us, of which the 32 vectors' loads and products fill half).  Measured (one sequence of 3,000
// tokens, 16 heads of 128 x 128, launches included; before, token by token): delta rule 1,081 -> 600 us, one decay per token
// 718 -> 350, with the delta rule 899 -> 528, constant decay 708 -> 380.  A long step is cut into pieces of records that stay in the L2
// (SCAN_PIECE_BYTES): the state waits in its slot between them.
#include "common.cuh"
#include "scan_modes.cuh"

#define BS_TOKENS 8
#define BS_STAGES 3
#define BS_LDC 12                         // floats between the columns of v and r in shared memory
#define SCAN_PIECE_BYTES (96LL << 20)

__host__ __device__ constexpr int bs_record(int dp, bool delta) {
    return (delta ? 4 : 2) * BS_TOKENS * dp + 2 * dp + (delta ? 16 : 8) * BS_TOKENS;
}
// the first record of sequence b, whose first token is t0: leaves room for every sequence's part-filled last record
__device__ __forceinline__ int bs_first_record(int t0, int b) { return (t0 + (BS_TOKENS - 1) * b) / BS_TOKENS; }

__device__ __forceinline__ float bs_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float bs_silu(float z) { return z / (1.f + expf(-z)); }

// Sums and products kept as a float32 number and what its rounding left: hi + lo.
__device__ __forceinline__ float2 bs_minus(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ void bs_add(float2& hi, float2& lo, float2 x) {
    const float2 sum = __fadd2_rn(hi, x), part = bs_minus(sum, hi);
    lo = __fadd2_rn(lo, __fadd2_rn(bs_minus(hi, bs_minus(sum, part)), bs_minus(x, part)));
    hi = sum;
}
__device__ __forceinline__ void bs_times(float& hi, float& lo, float w) {
    const float product = __fmul_rn(hi, w);
    lo = fmaf(lo, w, fmaf(hi, w, -product));
    hi = product;
}

// Sums V values over N lanes (powers of two; `l`: the lane's place among them) by trading halves: afterwards a lane
// holds the full sums of values l * (V / N) .. in v[0 ..] (N > V: of value l / (N / V)).
template <int N, int V>
__device__ __forceinline__ void bs_trade_sums(float (&v)[V], int l) {
    int count = V;
#pragma unroll
    for (int off = N / 2; off > 0; off >>= 1) {
        if (count > 1) {
            count >>= 1;
            const bool high = l & off;
#pragma unroll
            for (int i = 0; i < V / 2; ++i)
                if (i < count) {
                    const float give = high ? v[i] : v[i + count], keep = high ? v[i + count] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        }
    }
}

// A block per (eight tokens, head), a thread per key channel (dp threads).  Everything is loaded once and stays in
// registers; the sums over the channels are products of small matrices in shared memory.  The decays between two tokens
// enter them as products where a token has one decay (GATED*, DECAY), and as a quotient of the products from the record's
// first token where it has one per channel (DELTA: eight of them are at least exp(-8 exp(-1/2)) = 0.008, so that the
// quotient costs a rounding and cannot overflow).
template <int MODE>
__global__ void block_prepare_kernel(ScanArgs a, int n_seqs, int rec0, float* rec) {
    constexpr bool DELTA = MODE == SCAN_DELTA || MODE == SCAN_GATED_DELTA;
    constexpr int TK = BS_TOKENS;
    // rows of the left and right factors: DELTA b | q against n | x, GATED_DELTA k | q against k, else q against k
    constexpr int LEFT = DELTA ? 16 : 8, RIGHT = MODE == SCAN_DELTA ? 16 : 8;
    extern __shared__ __align__(16) float sm[];
    const int dp = blockDim.x, ld = dp + 4;
    float* lf = sm;                                                      // [LEFT][ld]
    float* rt = lf + LEFT * ld;                                          // [RIGHT][ld]
    float* gram = rt + RIGHT * ld;                                       // [LEFT][RIGHT]
    float* mA = gram + LEFT * RIGHT;                                     // [8][8] each: A, B (below the diagonal), C, D
    float* norm = mA + 4 * TK * TK;                                      // [dp / 32][8] partial sums of squares
    float* sc = norm + 8 * TK;                                           // [8][2] decay, dt or beta
    const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    const int r = rec0 + blockIdx.x, h = blockIdx.y;
    pdl_wait();
    pdl_launch();
    int seq = -1;                                                        // whose record is it?
    for (int b0 = 0; b0 < n_seqs && seq < 0; b0 += 32) {
        const int s = b0 + lane;
        bool hit = false;
        if (s < n_seqs) {
            const int t0 = a.cu_seqlens[s], first = bs_first_record(t0, s);
            hit = r >= first && r < first + (a.cu_seqlens[s + 1] - t0 + TK - 1) / TK;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m) seq = b0 + __ffs(m) - 1;
    }
    if (seq < 0) return;                                                 // (the same answer in every warp)
    const int t0 = a.cu_seqlens[seq], t1 = a.cu_seqlens[seq + 1];
    const int t = t0 + (r - bs_first_record(t0, seq)) * TK, n = min(TK, t1 - t);
    float* out = rec + ((size_t)blockIdx.x * a.H + h) * bs_record(dp, DELTA);
    const int hq = h / a.qk_div;

    float q[TK], k[TK], w[TK], na[TK];                                   // na: DELTA only
#pragma unroll
    for (int j = 0; j < TK; ++j) {
        const bool here = i < a.d && j < n;
        const size_t row = (size_t)(t + j);
        q[j] = here ? a.q[row * a.ldp + hq * a.d + i] : 0.f;
        k[j] = here ? a.k[row * a.ldp + hq * a.d + i] : 0.f;
        if (MODE == SCAN_DELTA) {
            na[j] = here ? a.au[row * a.ldp + h * a.d + i] : 0.f;
            w[j] = here ? a.w[row * a.ldw + h * a.d + i] : 0.f;
        }
    }
    if (MODE >= SCAN_GATED && i < 2 * TK)
        sc[i] = (i >> 1) < n ? a.scal[((size_t)(t + (i >> 1)) * a.H + h) * 4 + (i & 1)] : ((i & 1) ? 0.f : 1.f);
    float b[TK];                                                         // DELTA: unit keys
    if (MODE == SCAN_DELTA) {
        float ss[TK];
#pragma unroll
        for (int j = 0; j < TK; ++j) ss[j] = k[j] * k[j];
        bs_trade_sums<32, TK>(ss, lane);                                 // four lanes hold the same sum
        if ((lane & 3) == 0) norm[warp * TK + (lane >> 2)] = ss[0];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < TK; ++j) {
            float sum = 0.f;
            for (int x = 0; x < dp / 32; ++x) sum += norm[x * TK + j];
            const bool here = i < a.d && j < n;
            b[j] = here ? k[j] * (1.f / sqrtf(sum + a.unit_eps)) : 0.f;   // (no token: no key to divide by, whatever unit_eps is)
            na[j] = here ? -(bs_sigmoid(na[j]) * b[j]) : 0.f;
            w[j] = here ? expf(-0.6065306597126334f * bs_sigmoid(w[j])) : 1.f;
        }
        float run = 1.f;
#pragma unroll
        for (int j = 0; j < TK; ++j) {
            lf[j * ld + i] = run * b[j];
            run *= w[j];
            lf[(TK + j) * ld + i] = run * q[j];
            const float back = 1.f / run;
            rt[j * ld + i] = na[j] * back;
            rt[(TK + j) * ld + i] = k[j] * back;
        }
    } else {
#pragma unroll
        for (int j = 0; j < TK; ++j) {
            if (MODE == SCAN_DECAY && a.silu) { q[j] = bs_silu(q[j]); k[j] = bs_silu(k[j]); }      // (silu(0) = 0)
            if (DELTA) lf[j * ld + i] = k[j];
            lf[((DELTA ? TK : 0) + j) * ld + i] = q[j];
            rt[j * ld + i] = k[j];
        }
    }
    __syncthreads();
    for (int p = i; p < LEFT * RIGHT; p += dp) {
        const float4* x = reinterpret_cast<const float4*>(lf + (p / RIGHT) * ld);
        const float4* y = reinterpret_cast<const float4*>(rt + (p % RIGHT) * ld);
        float2 s0 = make_float2(0.f, 0.f), s1 = s0, l0 = s0, l1 = s0;
#pragma unroll 2
        for (int c = 0; c < dp / 4; c += 4) {
            float4 u = x[c], v = y[c];
            float2 a0 = __fmul2_rn(make_float2(u.x, u.y), make_float2(v.x, v.y));
            float2 a1 = __fmul2_rn(make_float2(u.z, u.w), make_float2(v.z, v.w));
#pragma unroll
            for (int i = 1; i < 4; ++i) {
                u = x[c + i]; v = y[c + i];
                a0 = __ffma2_rn(make_float2(u.x, u.y), make_float2(v.x, v.y), a0);
                a1 = __ffma2_rn(make_float2(u.z, u.w), make_float2(v.z, v.w), a1);
            }
            bs_add(s0, l0, a0);
            bs_add(s1, l1, a1);
        }
        bs_add(s0, l0, s1);
        float2 t = make_float2(s0.x, 0.f), lo = make_float2((l0.x + l1.x) + (l0.y + l1.y), 0.f);
        bs_add(t, lo, make_float2(s0.y, 0.f));
        gram[p] = t.x + lo.x;
    }
    __syncthreads();
    // A, B, C, D: what token p's reading (A, B) or query (C, D) meets of token s's removal and write
    for (int p = i; p < TK * TK; p += dp) {
        const int row = p / TK, s = p % TK;
        if (MODE == SCAN_DELTA) {
            mA[p] = gram[row * RIGHT + s];
            mA[64 + p] = gram[row * RIGHT + TK + s];
            mA[128 + p] = gram[(TK + row) * RIGHT + s];
            mA[192 + p] = gram[(TK + row) * RIGHT + TK + s];
        } else {
            float fade = 1.f;                                            // decays of tokens s + 1 .. row - 1, then row
            for (int x = s + 1; x < row; ++x) fade *= MODE == SCAN_DECAY ? a.head_decay[h] : sc[2 * x];
            const float kk = DELTA ? gram[row * RIGHT + s] : 0.f, qk = gram[((DELTA ? TK : 0) + row) * RIGHT + s];
            const float write = MODE == SCAN_DECAY ? 1.f : sc[2 * s + 1];
            if (DELTA) {
                mA[p] = -(write * sc[2 * s]) * (fade * kk);
                mA[64 + p] = write * (fade * kk);
            }
            if (row > s) fade *= MODE == SCAN_DECAY ? a.head_decay[h] : sc[2 * row];
            if (DELTA) mA[128 + p] = -(write * sc[2 * s]) * (fade * qk);
            mA[192 + p] = write * (fade * qk);
        }
    }
    __syncthreads();
    const float *A = mA, *B = mA + 64, *C = mA + 128, *D = mA + 192;

    // the rows of F (r) and E (o): the last warp's lane j makes column j
    if (warp == dp / 32 - 1 && lane < TK) {
        float* rows = out + (DELTA ? 4 : 2) * TK * dp + 2 * dp;
        const int j = lane;
        float f[TK];
        if (DELTA) {
#pragma unroll
            for (int x = 0; x < TK; ++x) {
                float v = j < x ? B[x * TK + j] : 0.f;
#pragma unroll
                for (int m = 0; m < x; ++m)
                    if (m > j) v = fmaf(A[x * TK + m], f[m], v);
                f[x] = v;
                rows[x * TK + j] = v;
            }
        }
        const float skip = (MODE == SCAN_GATED && a.skip) ? a.skip[h] : 0.f;
#pragma unroll
        for (int x = 0; x < TK; ++x) {
            float v = j <= x ? D[x * TK + j] : 0.f;
            if (DELTA) {
#pragma unroll
                for (int m = 0; m <= x; ++m)
                    if (m > j) v = fmaf(C[x * TK + m], f[m], v);
            }
            if (j == x) v += skip;
            rows[((DELTA ? TK : 0) + x) * TK + j] = v;
        }
    }

    // the vectors: P, Q | N, X | the decays' product, and what its rounding left
    float* vq = out + (DELTA ? TK * dp : 0);
    float* vn = vq + TK * dp;
    float* vx = vn + (DELTA ? TK * dp : 0);
    float run = 1.f, run_lo = 0.f, p[TK];
#pragma unroll
    for (int j = 0; j < TK; ++j) {
        const float wj = MODE == SCAN_DELTA ? w[j] : (MODE == SCAN_DECAY ? (j < n ? a.head_decay[h] : 1.f) : sc[2 * j]);
        w[j] = wj;
        if (DELTA) {
            const float read = MODE == SCAN_DELTA ? b[j] : k[j];
            float v = fmaf(run, read, run_lo * read);
#pragma unroll
            for (int m = 0; m < j; ++m) v = fmaf(A[j * TK + m], p[m], v);
            p[j] = v;
            out[j * dp + i] = v;
        }
        bs_times(run, run_lo, wj);
        float y = fmaf(run, q[j], run_lo * q[j]);
        if (DELTA) {
#pragma unroll
            for (int m = 0; m <= j; ++m) y = fmaf(C[j * TK + m], p[m], y);
        }
        vq[j * dp + i] = y;
    }
    float tail = 1.f, tail_lo = 0.f;
#pragma unroll
    for (int j = TK - 1; j >= 0; --j) {
        float x = k[j], y = MODE == SCAN_DELTA ? na[j] : 0.f;
        if (MODE >= SCAN_GATED) x = sc[2 * j + 1] * k[j];
        if (MODE == SCAN_GATED_DELTA) y = -(sc[2 * j + 1] * sc[2 * j]) * k[j];
        if (DELTA) vn[j * dp + i] = fmaf(tail, y, tail_lo * y);
        vx[j * dp + i] = fmaf(tail, x, tail_lo * x);
        bs_times(tail, tail_lo, w[j]);
    }
    const float fade = run + run_lo;
    vx[TK * dp + i] = fade;
    vx[(TK + 1) * dp + i] = (run - fade) + run_lo;
}

__device__ __forceinline__ void bs_copy16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// APART: the eight tokens' changes of the state are summed before they meet it.
template <bool DELTA, bool APART, int KG, int RK, int THREADS, int RC>
__global__ void __launch_bounds__(THREADS) block_scan_kernel(ScanArgs a, int rec0, int rec1, int silu_v, const float* rec) {
    constexpr int TK = BS_TOKENS, DP = KG * RK, R4 = RK / 4, CT = THREADS / KG * RC, REC = bs_record(DP, DELTA);
    constexpr int ROWS = DELTA ? 16 : 8;                  // products with the state: r and o, or o
    constexpr int V = ROWS * RC;
    constexpr int PER = KG >= V ? 1 : V / KG, SAME = KG >= V ? KG / V : 1;      // sums of a lane; lanes with the same one
    constexpr int VE = (TK * CT + THREADS - 1) / THREADS; // entries of v that a thread fetches per record
    extern __shared__ __align__(16) float sm[];
    float* sv = sm + BS_STAGES * REC;                     // [2][CT][BS_LDC] values, column by column
    float* sr = sv + 2 * CT * BS_LDC;                     // [CT][BS_LDC] r
    float* so = sr + CT * BS_LDC;                         // [2][TK][CT] results
    const int b = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * CT;
    const int tid = threadIdx.x, kg = tid % KG, cg = tid / KG;
    const int d = a.d, e = a.e, colb = col0 + cg * RC;
    pdl_wait();
    pdl_launch();
    const int t0 = a.cu_seqlens[b], t1 = a.cu_seqlens[b + 1];
    const int first = bs_first_record(t0, b), count = (t1 - t0 + TK - 1) / TK;
    const int begin = max(first, rec0), end = min(first + count, rec1);
    if (begin >= end) return;
    const float* src = rec + ((size_t)(begin - rec0) * a.H + head) * REC;
    const int n_rec = end - begin, tb = t0 + (begin - first) * TK;

    auto stage_in = [&](int i) {
        if (i < n_rec) {
            const float* from = src + (size_t)i * a.H * REC;
            float* to = sm + (i % BS_STAGES) * REC;
            for (int p = tid; p < REC / 4; p += THREADS) bs_copy16(to + 4 * p, from + 4 * p);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float vreg[VE];
    auto fetch_v = [&](int i) {
#pragma unroll
        for (int x = 0; x < VE; ++x) {
            const int idx = tid + x * THREADS, j = idx / CT, c = idx % CT, t = tb + i * TK + j;
            vreg[x] = (idx < TK * CT && i < n_rec && t < t1 && col0 + c < e) ? a.v[(size_t)t * a.ldp + head * e + col0 + c] : 0.f;
        }
    };
    auto keep_v = [&](int i) {
        float* to = sv + (i & 1) * CT * BS_LDC;
#pragma unroll
        for (int x = 0; x < VE; ++x) {
            const int idx = tid + x * THREADS, j = idx / CT, c = idx % CT;
            if (idx < TK * CT) to[c * BS_LDC + j] = silu_v ? bs_silu(vreg[x]) : vreg[x];
        }
    };
#pragma unroll
    for (int i = 0; i < BS_STAGES - 1; ++i) stage_in(i);
    fetch_v(0);
    keep_v(0);
    fetch_v(1);

    float* st = a.state + (size_t)a.slots[b] * a.state_stride + (size_t)head * d * e;
    float2 S[2 * R4][RC];                                 // S[r][c]: keys 2r and 2r + 1 of this thread, column c
#pragma unroll
    for (int r = 0; r < RK; ++r) {
        const int key = ((r >> 2) * KG + kg) * 4 + (r & 3);
#pragma unroll
        for (int c = 0; c < RC; ++c) {
            const float x = (key < d && colb + c < e) ? st[(size_t)key * e + colb + c] : 0.f;
            if (r & 1) S[r >> 1][c].y = x; else S[r >> 1][c].x = x;
        }
    }
    auto write_out = [&](int i) {                         // the results of record i
        const float* from = so + (i & 1) * TK * CT;
        for (int idx = tid; idx < TK * CT; idx += THREADS) {
            const int j = idx / CT, c = idx % CT, t = tb + i * TK + j;
            if (t < t1 && col0 + c < e) a.out[(size_t)t * a.ldo + head * e + col0 + c] = from[idx];
        }
    };

    for (int i = 0; i < n_rec; ++i) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(BS_STAGES - 2) : "memory");
        __syncthreads();                                  // record i and its values are whole, record i - 1 is consumed
        stage_in(i + BS_STAGES - 1);
        keep_v(i + 1);
        fetch_v(i + 2);
        if (i > 0) write_out(i - 1);
        const int here = t1 - (tb + i * TK);              // tokens of this record (a count past TK is as good)
        const float* sc = sm + (i % BS_STAGES) * REC;
        const float4* pv = reinterpret_cast<const float4*>(sc) + kg;
        float val[V];
#pragma unroll
        for (int row = 0; row < ROWS; ++row) {
            float4 x[R4];
#pragma unroll
            for (int g = 0; g < R4; ++g) x[g] = pv[row * (DP / 4) + g * KG];
#pragma unroll
            for (int c = 0; c < RC; ++c) {
                float2 acc = __fmul2_rn(make_float2(x[0].x, x[0].y), S[0][c]);
                acc = __ffma2_rn(make_float2(x[0].z, x[0].w), S[1][c], acc);
#pragma unroll
                for (int g = 1; g < R4; ++g) {
                    acc = __ffma2_rn(make_float2(x[g].x, x[g].y), S[2 * g][c], acc);
                    acc = __ffma2_rn(make_float2(x[g].z, x[g].w), S[2 * g + 1][c], acc);
                }
                val[row * RC + c] = acc.x + acc.y;
            }
        }
        bs_trade_sums<KG, V>(val, kg);
        // this lane's sums get what the tokens before them in the record add
        const float* rows = sc + (DELTA ? 4 : 2) * TK * DP + 2 * DP;
        const float* vcol = sv + ((i & 1) * CT + cg * RC) * BS_LDC;
#pragma unroll
        for (int x = 0; x < PER; ++x) {
            const int idx = SAME > 1 ? kg / SAME : kg * PER + x, row = idx / RC, c = idx % RC;
            const int limit = (DELTA && row < TK) ? row : row - (DELTA ? TK : 0) + 1;
            float m[TK], u[TK];
            *reinterpret_cast<float4*>(m) = *reinterpret_cast<const float4*>(rows + row * TK);
            *reinterpret_cast<float4*>(m + 4) = *reinterpret_cast<const float4*>(rows + row * TK + 4);
            *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(vcol + c * BS_LDC);
            *reinterpret_cast<float4*>(u + 4) = *reinterpret_cast<const float4*>(vcol + c * BS_LDC + 4);
            float sum = val[x];
#pragma unroll
            for (int j = 0; j < TK; ++j)
                if (j < limit) sum = fmaf(m[j], u[j], sum);              // (a later token's value is not touched)
            if (DELTA && row < TK && row >= here) sum = 0.f;             // (no token: 0, and not 0 * an infinite state)
            if (SAME == 1 || kg % SAME == 0) {
                if (DELTA && row < TK) sr[(cg * RC + c) * BS_LDC + row] = sum;
                else so[((i & 1) * TK + row - (DELTA ? TK : 0)) * CT + cg * RC + c] = sum;
            }
        }
        __syncwarp();
        float2 change[2 * R4][RC];
        const float4* pf = pv + (DELTA ? 4 : 2) * TK * (DP / 4);
#pragma unroll
        for (int g = 0; g < R4; ++g) {
            const float4 hi = pf[g * KG], lo = pf[DP / 4 + g * KG];
#pragma unroll
            for (int c = 0; c < RC; ++c) {
                change[2 * g][c] = __fmul2_rn(make_float2(lo.x, lo.y), S[2 * g][c]);
                change[2 * g + 1][c] = __fmul2_rn(make_float2(lo.z, lo.w), S[2 * g + 1][c]);
                if (!APART) {
                    change[2 * g][c] = __ffma2_rn(make_float2(hi.x, hi.y), S[2 * g][c], change[2 * g][c]);
                    change[2 * g + 1][c] = __ffma2_rn(make_float2(hi.z, hi.w), S[2 * g + 1][c], change[2 * g + 1][c]);
                }
            }
        }
#pragma unroll
        for (int part = DELTA ? 0 : 1; part < 2; ++part) {               // N r, then X v
            const float4* pw = pv + ((DELTA ? 2 : 0) + part) * TK * (DP / 4);
            const float* from = part ? vcol : sr + cg * RC * BS_LDC;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float4 y[RC];
#pragma unroll
                for (int c = 0; c < RC; ++c) y[c] = *reinterpret_cast<const float4*>(from + c * BS_LDC + 4 * half);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float4 x[R4];
#pragma unroll
                    for (int g = 0; g < R4; ++g) x[g] = pw[(4 * half + j) * (DP / 4) + g * KG];
#pragma unroll
                    for (int c = 0; c < RC; ++c) {
                        const float z = j == 0 ? y[c].x : (j == 1 ? y[c].y : (j == 2 ? y[c].z : y[c].w));
                        const float2 zz = make_float2(z, z);
#pragma unroll
                        for (int g = 0; g < R4; ++g) {
                            change[2 * g][c] = __ffma2_rn(make_float2(x[g].x, x[g].y), zz, change[2 * g][c]);
                            change[2 * g + 1][c] = __ffma2_rn(make_float2(x[g].z, x[g].w), zz, change[2 * g + 1][c]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < R4; ++g) {
            const float4 hi = APART ? pf[g * KG] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < RC; ++c) {
                S[2 * g][c] = APART ? __ffma2_rn(make_float2(hi.x, hi.y), S[2 * g][c], change[2 * g][c]) : change[2 * g][c];
                S[2 * g + 1][c] = APART ? __ffma2_rn(make_float2(hi.z, hi.w), S[2 * g + 1][c], change[2 * g + 1][c])
                                        : change[2 * g + 1][c];
            }
        }
    }
    __syncthreads();
    write_out(n_rec - 1);
#pragma unroll
    for (int r = 0; r < RK; ++r) {
        const int key = ((r >> 2) * KG + kg) * 4 + (r & 3);
#pragma unroll
        for (int c = 0; c < RC; ++c)
            if (key < d && colb + c < e) st[(size_t)key * e + colb + c] = (r & 1) ? S[r >> 1][c].y : S[r >> 1][c].x;
    }
}

#define BS_SMEM_ALONE (116 * 1024)        // two such blocks do not fit the 228 KB of an SM
#define BS_SMEM_PAIR (78 * 1024)          // three do not

template <bool DELTA, bool APART, int KG, int RK, int THREADS, int RC>
static int launch_block_scan(const ScanArgs& a, int n_seqs, int rec0, int rec1, int silu_v, const float* rec, cudaStream_t stream) {
    constexpr int CT = THREADS / KG * RC, REC = bs_record(KG * RK, DELTA);
    size_t smem = ((size_t)BS_STAGES * REC + 3 * CT * BS_LDC + 2 * BS_TOKENS * CT) * sizeof(float);
    constexpr size_t most = ((size_t)BS_STAGES * REC + 3 * CT * BS_LDC + 2 * BS_TOKENS * CT) * sizeof(float) > BS_SMEM_ALONE
                                ? ((size_t)BS_STAGES * REC + 3 * CT * BS_LDC + 2 * BS_TOKENS * CT) * sizeof(float) : BS_SMEM_ALONE;
    static bool configured[64] = {false};                 // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(block_scan_kernel<DELTA, APART, KG, RK, THREADS, RC>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const dim3 grid(n_seqs, a.H, (a.e + CT - 1) / CT);
    // Blocks that start while the kernel before drains gather on the SMs that fall free first; with no more blocks than SMs
    // (twice as many) a block asks for more shared memory than half (a third of) an SM has.
    const long long blocks = (long long)grid.x * grid.y * grid.z;
    const size_t least = blocks <= tq_sm_count() ? BS_SMEM_ALONE : (blocks <= 2LL * tq_sm_count() ? BS_SMEM_PAIR : 0);
    if (smem < least) smem = least;
    return tq_launch_pdl(TQ_PDL_ELEMENTWISE, block_scan_kernel<DELTA, APART, KG, RK, THREADS, RC>, grid, dim3(THREADS), smem, stream, a, rec0,
                         rec1, silu_v, rec);
}

// Which form.  A thread holds four keys (eight of rows over 128), so that every load brings different entries to all 32
// lanes; a block of 128 threads with two columns each (8 columns of rows over 64, 16 and 32 of shorter ones) while there are
// at most two such blocks an SM, else of 256 threads with four each (32, 64 and 128 columns).  Measured with 128 x 128
// states, 3,000 tokens of one sequence, in us, before the sums were compensated (columns a block x threads; delta rule /
// one decay): 16 heads: 8 x 128 488 / 331, 16 x 256 490 / 346, 16 x 128 (eight keys a thread) 540 /
// 352; 32 heads: 8 x 128 763 / 487, 16 x 128 702 / 568, 32 x 256 707 / 447.
template <bool DELTA, bool APART, int DP>
static int pick_block_scan(const ScanArgs& a, int n_seqs, int rec0, int rec1, int silu_v, const float* rec, cudaStream_t stream) {
    constexpr int KG = DP >= 128 ? 32 : DP / 4;
#define TQ_FORM(T, RC) return launch_block_scan<DELTA, APART, KG, DP / KG, T, RC>(a, n_seqs, rec0, rec1, silu_v, rec, stream)
    const long long blocks = (long long)n_seqs * a.H * ((a.e + 128 / KG * 2 - 1) / (128 / KG * 2));
    if (blocks <= 2LL * tq_sm_count()) TQ_FORM(128, 2);
    TQ_FORM(256, 4);
#undef TQ_FORM
}

static int bs_padded_keys(int d) { return d <= 32 ? 32 : (d <= 64 ? 64 : (d <= 128 ? 128 : 256)); }

// Records of a step of n_tokens tokens of n_seqs sequences, and how many of them one piece takes.
static long long bs_records(int n_tokens, int n_seqs) { return ((long long)n_tokens + (BS_TOKENS - 1LL) * n_seqs) / BS_TOKENS + 1; }
static long long bs_piece(int mode, int n_tokens, int n_seqs, int H, int d) {
    const bool delta = mode == SCAN_DELTA || mode == SCAN_GATED_DELTA;
    const long long all = bs_records(n_tokens, n_seqs), bytes = (long long)H * bs_record(bs_padded_keys(d), delta) * 4;
    const long long most = SCAN_PIECE_BYTES / bytes > 1 ? SCAN_PIECE_BYTES / bytes : 1;
    const long long pieces = (all + most - 1) / most;
    return (all + pieces - 1) / pieces;
}

// The line between the two scans (and how long a step must be: kernels/scan.py).  Token by token, a step costs its longest sequence 210 to 350 ns a token however few
// columns (of the states of all heads and sequences) there are; with many columns both are bound by the SMs, and this one
// has its records to make as well.  Measured with 128 x 128 states, one at a time / eight at a time, in us: 3,000 tokens of
// 16 heads (2,048 columns) 1,083 / 584 (delta rule), 719 / 337 (one decay); of 32 heads (4,096 columns) 1,604 / 880, 983 /
// 471; four sequences of 250 tokens, 16 heads (8,192 columns): 158 / 200, 95 / 100.
long long block_scan_floats(int mode, int n_tokens, int n_seqs, int H, int d, int e) {
    if ((long long)n_seqs * H * e > 32LL * tq_sm_count()) return 0;
    const bool delta = mode == SCAN_DELTA || mode == SCAN_GATED_DELTA;
    return bs_piece(mode, n_tokens, n_seqs, H, d) * H * bs_record(bs_padded_keys(d), delta);
}

template <int MODE>
static int run_block_scan(const ScanArgs& a, int n_seqs, int n_tokens, float* rec, cudaStream_t stream) {
    constexpr bool DELTA = MODE == SCAN_DELTA || MODE == SCAN_GATED_DELTA;
    const int dp = bs_padded_keys(a.d), silu_v = MODE == SCAN_DECAY && a.silu;
    const long long all = bs_records(n_tokens, n_seqs), piece = bs_piece(MODE, n_tokens, n_seqs, a.H, a.d);
    for (long long r0 = 0; r0 < all; r0 += piece) {
        const long long r1 = r0 + piece < all ? r0 + piece : all;
        constexpr int LEFT = DELTA ? 16 : 8, RIGHT = MODE == SCAN_DELTA ? 16 : 8;
        const size_t smem = ((size_t)(LEFT + RIGHT) * (dp + 4) + LEFT * RIGHT + 4 * 64 + 64 + 16) * sizeof(float);
        int st = tq_launch_pdl(TQ_PDL_ELEMENTWISE, block_prepare_kernel<MODE>, dim3((unsigned)(r1 - r0), a.H), dim3(dp), smem, stream,
                               a, n_seqs, (int)r0, rec);
        if (st) return st;
        switch (dp) {
            case 32: st = pick_block_scan<DELTA, MODE != SCAN_DELTA, 32>(a, n_seqs, (int)r0, (int)r1, silu_v, rec, stream); break;
            case 64: st = pick_block_scan<DELTA, MODE != SCAN_DELTA, 64>(a, n_seqs, (int)r0, (int)r1, silu_v, rec, stream); break;
            case 128: st = pick_block_scan<DELTA, MODE != SCAN_DELTA, 128>(a, n_seqs, (int)r0, (int)r1, silu_v, rec, stream); break;
            default: st = pick_block_scan<DELTA, MODE != SCAN_DELTA, 256>(a, n_seqs, (int)r0, (int)r1, silu_v, rec, stream); break;
        }
        if (st) return st;
    }
    return 0;
}

int block_scan(int mode, const ScanArgs& a, int n_seqs, int n_tokens, float* rec, cudaStream_t stream) {
    switch (mode) {
        case SCAN_DECAY: return run_block_scan<SCAN_DECAY>(a, n_seqs, n_tokens, rec, stream);
        case SCAN_DELTA: return run_block_scan<SCAN_DELTA>(a, n_seqs, n_tokens, rec, stream);
        case SCAN_GATED: return run_block_scan<SCAN_GATED>(a, n_seqs, n_tokens, rec, stream);
        case SCAN_GATED_DELTA: return run_block_scan<SCAN_GATED_DELTA>(a, n_seqs, n_tokens, rec, stream);
        default: return (int)cudaErrorInvalidValue;
    }
}
