// Float32 products that gemm_f32_tc.cu does not take, on float32 fused multiply-adds:
// C[M,N] (=, +=) A[M,K] · W[N,K]^T (+ bias[N]), float32 operands and result, every sum in float32 (no reduced-precision mode).  Optional epilogues:
// W holding gate rows then up rows, C = act(gate) * up; or the square of relu.
//
// What bounds it: the 128 float32 lanes of an SM (about 72 TFLOP/s).  A block of 128 threads makes a tile of 64 x 128
// outputs (32 or 16 x 128 for few rows), 8 x 8 (4 or 2 x 8) a thread: 16 shared-memory loads of 16 bytes feed 128 packed
// multiply-adds, so the lanes and not the shared memory are the limit.  Tiles of both operands arrive by cp.async in
// their own layout (K inner), three stages of 32 columns deep; rows are 36 floats apart in shared memory, which puts
// eight neighbouring rows into different banks.  The packed multiply-adds take pairs along K (even and odd columns
// are summed apart and meet at the end), so nothing is transposed or duplicated.  Where tiles are fewer than the
// block slots, K is cut over a cluster of up to eight blocks; the partial tiles meet through distributed shared
// memory in the order of the ranks, so the result does not depend on timing.
//
// Measured (one B200, L2 flushed, in us; before: the 64 x 64 tiles of gemm.cu with 4 x 4 outputs a thread and loads of
// single floats): N = 151,936, K = 896: 300 rows 4,001 -> 1,820 (45 TFLOP/s), 2,000 rows 25,130 -> 11,340 (48); N = 896,
// K = 4,864: 300 rows 674 -> 104, 24 rows 751 -> 29; gated N = 5,632, K = 2,048: 300 rows 835 -> 319 (43 TFLOP/s).
// At 2,000 rows the lanes are 69 % busy, the shared-memory pipe 50 %, with two warps a scheduler (252 registers): what
// is left is latency that a third block would hide and its registers do not allow.
#include "common.cuh"

#include <cooperative_groups.h>

#define FT_THREADS 128
#define FT_BN 128
#define FT_BK 32
#define FT_LD 36                  // floats between rows of a stage
#define FT_STAGES 3
#define FT_OUT_LD 132             // floats between rows of the finished tile
#define FT_MAX_SPLIT 8

struct F32TileArgs {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc, accumulate, act, vec_out;
    int settled;              // W was complete before the kernel in front of this one began: read it before that one ends
};

__device__ __forceinline__ void ft_copy16(float* dst, const float* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(ok ? 16 : 0));
}

// Grid (row tiles * split, column tiles), clusters of `split` blocks along x.  GATED: a tile holds 64 gate and 64 up
// columns, the gate's column c of a warp's half beside the up column in the same thread.
template <int TM, bool GATED>
__global__ void __launch_bounds__(FT_THREADS, 2) f32_tile_kernel(const F32TileArgs a) {
    namespace cg = cooperative_groups;
    constexpr int BM = 8 * TM, STAGE = (BM + FT_BN) * FT_LD;
    extern __shared__ __align__(16) float sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 1, wn = warp & 1, tm = lane >> 3, tn = lane & 7;
    const int m0 = (blockIdx.x / split) * BM;
    const int n0 = blockIdx.y * (GATED ? FT_BN / 2 : FT_BN);
    const int steps = (a.K + FT_BK - 1) / FT_BK;
    const int s_begin = (int)((long long)steps * rank / split), s_end = (int)((long long)steps * (rank + 1) / split);
    const int n_steps = s_end - s_begin;

    // this thread's share of a stage: 16-byte pieces (row, piece) = (tid / 8 + 16 i, tid % 8)
    const int lr = tid >> 3, lk = (tid & 7) * 4;
    auto load_w = [&](int step) {
        float* dst = sm + (step % FT_STAGES) * STAGE + BM * FT_LD;
        const int k = (s_begin + step) * FT_BK + lk;
#pragma unroll
        for (int i = 0; i < FT_BN / 16; ++i) {
            const int r = lr + 16 * i;
            int n;
            bool ok;
            if (GATED) {                                     // rows of a warp's half: 32 of the gate, 32 of the up
                n = n0 + (r >> 6) * 32 + (r & 31);
                ok = n < a.N && k < a.K;
                n += ((r >> 5) & 1) * a.N;
            } else {
                n = n0 + r;
                ok = n < a.N && k < a.K;
            }
            ft_copy16(dst + r * FT_LD + lk, ok ? a.W + (size_t)n * a.ldw + k : a.W, ok);
        }
    };
    auto load_a = [&](int step) {
        float* dst = sm + (step % FT_STAGES) * STAGE;
        const int k = (s_begin + step) * FT_BK + lk;
#pragma unroll
        for (int i = 0; i < BM / 16; ++i) {
            const int r = lr + 16 * i, m = m0 + r;
            const bool ok = m < a.M && k < a.K;
            ft_copy16(dst + r * FT_LD + lk, ok ? a.A + (size_t)m * a.lda + k : a.A, ok);
        }
    };

    // weights do not depend on the kernel before: those of the first stages are asked for at once
    if (!a.settled) pdl_wait();
#pragma unroll
    for (int s = 0; s < FT_STAGES - 1; ++s)
        if (s < n_steps) load_w(s);
    pdl_wait();
    pdl_launch();
#pragma unroll
    for (int s = 0; s < FT_STAGES - 1; ++s) {
        if (s < n_steps) load_a(s);
        asm volatile("cp.async.commit_group;\n");
    }

    float2 acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);

    for (int step = 0; step < n_steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(FT_STAGES - 2));
        __syncthreads();                                     // the stage is whole, and the one before it is consumed
        if (step + FT_STAGES - 1 < n_steps) {
            load_w(step + FT_STAGES - 1);
            load_a(step + FT_STAGES - 1);
        }
        asm volatile("cp.async.commit_group;\n");
        const float* sa = sm + (step % FT_STAGES) * STAGE + (wm * 4 * TM + tm) * FT_LD;
        const float* sw = sm + (step % FT_STAGES) * STAGE + (BM + wn * 64 + tn) * FT_LD;
#pragma unroll
        for (int kc = 0; kc < FT_BK; kc += 4) {
            float4 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(sa + i * 4 * FT_LD + kc);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 wv = *reinterpret_cast<const float4*>(sw + j * 8 * FT_LD + kc);
#pragma unroll
                for (int i = 0; i < TM; ++i)
                    acc[i][j] = __ffma2_rn(make_float2(av[i].x, av[i].y), make_float2(wv.x, wv.y), acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
                    acc[i][j] = __ffma2_rn(make_float2(av[i].z, av[i].w), make_float2(wv.z, wv.w), acc[i][j]);
            }
        }
    }

    // the tile (or this rank's share of its sums) into shared memory, then the ranks' shares together
    asm volatile("cp.async.wait_group 0;\n");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            sm[(wm * 4 * TM + tm + 4 * i) * FT_OUT_LD + wn * 64 + tn + 8 * j] = acc[i][j].x + acc[i][j].y;
    if (split > 1) cluster.sync();
    else __syncthreads();

    constexpr int PIECES = GATED ? FT_BN / 8 : FT_BN / 4;    // 16-byte pieces of an output row
    for (int idx = rank * FT_THREADS + tid; idx < BM * PIECES; idx += split * FT_THREADS) {
        const int r = idx / PIECES, p = idx % PIECES, m = m0 + r, n = n0 + p * 4;
        if (m >= a.M || n >= a.N) continue;
        const int at = r * FT_OUT_LD + (GATED ? (p >> 3) * 64 + (p & 7) * 4 : p * 4);
        float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < split; ++s) {
            const float* part = split > 1 ? cluster.map_shared_rank(sm, s) : sm;
            const float4 x = *reinterpret_cast<const float4*>(part + at);
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            if (GATED) {
                const float4 y = *reinterpret_cast<const float4*>(part + at + 32);
                u[0] += y.x; u[1] += y.y; u[2] += y.z; u[3] += y.w;
            }
        }
        float* c = a.C + (size_t)m * a.ldc + n;
        float old[4] = {0.f, 0.f, 0.f, 0.f};
        const bool whole = a.vec_out && n + 4 <= a.N;
        if (a.accumulate) {
            if (whole) {
                const float4 x = *reinterpret_cast<const float4*>(c);
                old[0] = x.x; old[1] = x.y; old[2] = x.z; old[3] = x.w;
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (n + q < a.N) old[q] = c[q];
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool in = n + q < a.N;
            if (a.bias && in) {
                v[q] += a.bias[n + q];
                if (GATED) u[q] += a.bias[n + q + a.N];
            }
            if (GATED) v[q] = gated_act(v[q], a.act) * u[q];
            else if (a.act == TQ_ACT_SQUARE_RELU) v[q] = square_relu(v[q]);
            if (a.accumulate) v[q] += old[q];
        }
        if (whole) {
            *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (n + q < a.N) c[q] = v[q];
        }
    }
    if (split > 1) cluster.sync();                           // nobody leaves while its sums are being read
}

template <int TM, bool GATED>
static int launch_f32_tile(const F32TileArgs& a, int split, cudaStream_t stream) {
    constexpr int BM = 8 * TM;
    constexpr size_t smem = (size_t)FT_STAGES * (BM + FT_BN) * FT_LD * sizeof(float);
    static_assert(smem >= (size_t)BM * FT_OUT_LD * sizeof(float), "the finished tile reuses the stages");
    static bool configured[64] = {false};                    // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(f32_tile_kernel<TM, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int per = GATED ? FT_BN / 2 : FT_BN;
    const long long mt = (a.M + BM - 1) / BM, nt = (a.N + per - 1) / per;
    if (nt > 65535 || mt * split > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(mt * split), (unsigned)nt);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = tq_pdl_enabled(TQ_PDL_SKINNY) ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, f32_tile_kernel<TM, GATED>, a);
    if (e != cudaSuccess) return (int)e;
    return tq_launch_status();
}

// How many blocks share a tile's K: the count that makes (rounds of block slots) x (steps of a share + the pipeline's
// fill and the meeting of the shares, about 3 steps) least.
static int f32_tile_split(long long tiles, int steps) {
    const long long slots = 2LL * tq_sm_count();
    int best = 1;
    double least = 0;
    for (int s = 1; s <= FT_MAX_SPLIT && s <= steps; ++s) {
        const long long rounds = (tiles * s + slots - 1) / slots;
        const double t = (double)rounds * ((double)((steps + s - 1) / s) + 3.0);
        if (s == 1 || t < 0.97 * least) { best = s; least = t; }
    }
    return best;
}

// gate: 0 a plain product, TQ_ACT_SILU / TQ_ACT_GELU_TANH a gated one (W has 2 N rows), TQ_ACT_SQUARE_RELU a plain one
// with that activation.  K, lda and ldw are multiples of 4, A and W 16-byte aligned (other operands: tq_gemm_tiled).
// settled: no kernel that may still run when this one starts writes W (it was complete before the one in front began).
TQ_API int tq_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                       int ldc, int accumulate, int gate, int settled, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || lda % 4 || ldw % 4 || lda < K || ldw < K || ldc < N || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) ||
        gate < 0 || gate > TQ_ACT_SQUARE_RELU)
        return (int)cudaErrorInvalidValue;
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
    F32TileArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, gate,
                  (ldc % 4 == 0 && ((uintptr_t)C & 15) == 0) ? 1 : 0, settled};
    // tiles of 16 or 32 rows where tiles of 64 would be mostly padding (their threads do less work per load): N = 2,048,
    // K = 5,632 at 16 rows takes 41 us in tiles of 16 and 51 in tiles of 32
    const long long pad64 = (M + 63) / 64 * 64, pad32 = (M + 31) / 32 * 32;
    const int bm = M <= 16 ? 16 : (pad32 * 5 <= pad64 * 4 ? 32 : 64);
    const int per = gated ? FT_BN / 2 : FT_BN;
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + per - 1) / per);
    const int split = f32_tile_split(tiles, (K + FT_BK - 1) / FT_BK);
    if (bm == 16) return gated ? launch_f32_tile<2, true>(a, split, stream) : launch_f32_tile<2, false>(a, split, stream);
    if (gated) return bm == 32 ? launch_f32_tile<4, true>(a, split, stream) : launch_f32_tile<8, true>(a, split, stream);
    return bm == 32 ? launch_f32_tile<4, false>(a, split, stream) : launch_f32_tile<8, false>(a, split, stream);
}

// ---------------------------------------------------------------------------
// The same product for up to 8 rows (decoding in float32), bound by reading W once.  KW warps of a block make
// NC columns (rows of W): they take 128-column pieces of K in turn, so that a block's whole share of a small W is
// asked for at once (896 columns: one load per lane and row of W), for a settled W before the kernel waits for its
// predecessor, whose results it does not need for that; the next pieces are asked for while one is multiplied.  Every piece of A is read
// once per NC columns.  The lanes' sums meet by halving (31 shuffles for 32 sums instead of 160), the warps' in
// shared memory in the order of the warps.
// ---------------------------------------------------------------------------
#define FR_WARPS 8

struct F32RowsArgs {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc, accumulate, act, settled;
};

template <int MR, int NC, int KW, bool GATED>
__global__ void __launch_bounds__(FR_WARPS * 32) f32_rows_kernel(const F32RowsArgs a) {
    constexpr int V = MR * NC, OUT = GATED ? NC / 2 : NC, GROUPS = FR_WARPS / KW;
    __shared__ float red[FR_WARPS][V];
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % KW, group = (threadIdx.x >> 5) / KW;
    const int n0 = (blockIdx.x * GROUPS + group) * OUT;
    const int pieces = (a.K + 127) / 128;
    const float* wrow[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int n = min(n0 + (GATED ? c / 2 : c), a.N - 1);            // columns past the last repeat it, unused
        wrow[c] = a.W + (size_t)(n + (GATED && (c & 1) ? a.N : 0)) * a.ldw;
    }
    auto load = [&](int piece, float4 (&w)[NC]) {
        const int k = piece * 128 + lane * 4;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            w[c] = k < a.K ? *reinterpret_cast<const float4*>(wrow[c] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 w[NC], next[NC];
    if (!a.settled) pdl_wait();
    if (warp < pieces) load(warp, w);
    pdl_wait();
    pdl_launch();
    float2 acc[MR][NC];
#pragma unroll
    for (int r = 0; r < MR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[r][c] = make_float2(0.f, 0.f);
    for (int piece = warp; piece < pieces; piece += KW) {
        if (piece + KW < pieces) load(piece + KW, next);
        const int k = piece * 128 + lane * 4;
#pragma unroll
        for (int r = 0; r < MR; ++r) {
            const float4 x = (r < a.M && k < a.K) ? *reinterpret_cast<const float4*>(a.A + (size_t)r * a.lda + k)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                acc[r][c] = __ffma2_rn(make_float2(x.x, x.y), make_float2(w[c].x, w[c].y), acc[r][c]);
                acc[r][c] = __ffma2_rn(make_float2(x.z, x.w), make_float2(w[c].z, w[c].w), acc[r][c]);
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) w[c] = next[c];
    }
    // V sums over 32 lanes: each step halves the sums a lane holds (or, with one left, adds the lanes' copies)
    float v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = acc[i / NC][i % NC].x + acc[i / NC][i % NC].y;
    int held = 0;                                            // index of the sum in v[0]
#pragma unroll
    for (int off = 16, n = V; off > 0; off >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < V / 2; ++i)
                if (i < n) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], off);
            if (up) held += n;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        }
    }
    if (V >= 32 || (lane & (32 / (V < 32 ? V : 32) - 1)) == 0) red[group * KW + warp][held] = v[0];
    __syncthreads();
    for (int i = threadIdx.x; i < GROUPS * MR * OUT; i += FR_WARPS * 32) {
        const int r = i / (GROUPS * OUT), c = i % OUT, first = i / OUT % GROUPS * KW;
        const int n = blockIdx.x * GROUPS * OUT + i % (GROUPS * OUT);
        if (r >= a.M || n >= a.N) continue;
        const int at = r * NC + (GATED ? 2 * c : c);
        float y = 0.f, u = 0.f;
#pragma unroll
        for (int s = 0; s < KW; ++s) {
            y += red[first + s][at];
            if (GATED) u += red[first + s][at + 1];
        }
        if (a.bias) {
            y += a.bias[n];
            if (GATED) u += a.bias[n + a.N];
        }
        if (GATED) y = gated_act(y, a.act) * u;
        else if (a.act == TQ_ACT_SQUARE_RELU) y = square_relu(y);
        float* out = a.C + (size_t)r * a.ldc + n;
        *out = a.accumulate ? *out + y : y;
    }
}

template <int MR>
static int launch_f32_rows(const F32RowsArgs& a, bool gated, cudaStream_t stream) {
    const int out = gated ? 2 : 4;
    // Columns are plenty: a warp takes a whole row of W, and its sums meet once (N = 151,936, K = 896, 8 rows: 152 us
    // against 228 with eight warps a row).  Few: up to eight warps share a row, so that 32 warps an SM have work.
    const long long groups = (a.N + out - 1) / out;
    const long long want = 32LL * tq_sm_count();
#define TQ_ROWS(KW)                                                                                                     \
    do {                                                                                                                \
        const dim3 grid((unsigned)((groups + FR_WARPS / KW - 1) / (FR_WARPS / KW)));                                    \
        if (gated)                                                                                                      \
            return tq_launch_pdl(TQ_PDL_SKINNY, f32_rows_kernel<MR, 4, KW, true>, grid, dim3(FR_WARPS * 32), 0, stream, a); \
        return tq_launch_pdl(TQ_PDL_SKINNY, f32_rows_kernel<MR, 4, KW, false>, grid, dim3(FR_WARPS * 32), 0, stream, a); \
    } while (0)
    if (groups >= want) TQ_ROWS(1);
    if (groups * 2 >= want) TQ_ROWS(2);
    if (groups * 4 >= want) TQ_ROWS(4);
    TQ_ROWS(8);
#undef TQ_ROWS
}

// As tq_gemm_f32 for M <= 8 (from 9 rows on the tiles of 16 rows are faster or equal: 16 rows of N = 2,048, K = 5,632
// take 41 us there, and took 108 in a form of this kernel).
TQ_API int tq_gemv_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                       int ldc, int accumulate, int gate, int settled, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 8 || K <= 0 || K % 4 || lda % 4 || ldw % 4 || (M > 1 && (lda < K || ldc < N)) || ldw < K || ((uintptr_t)A & 15) ||
        ((uintptr_t)W & 15) || gate < 0 || gate > TQ_ACT_SQUARE_RELU)
        return (int)cudaErrorInvalidValue;
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
    const F32RowsArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, gate, settled};
    if (M == 1) return launch_f32_rows<1>(a, gated, stream);
    if (M == 2) return launch_f32_rows<2>(a, gated, stream);
    if (M <= 4) return launch_f32_rows<4>(a, gated, stream);
    return launch_f32_rows<8>(a, gated, stream);
}
