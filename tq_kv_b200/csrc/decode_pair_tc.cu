// Weight-streaming products of up to 64 rows on the tcgen05 tensor cores, cut to the GPU: gated products of a decode batch,
// and the products of routed experts that own a few rows each.
//   Y[m, n] = act(X[m] . W[n]) * (X[m] . W[n + second])          (gated)
//   Y[m, n] = X[m] . W[n], or the square of its relu             (plain)
//
// What bounds it is the reading of W, so every SM should read the same share of it, once.  A work item is two bands of `out`
// rows of W (gated: the gate rows and the up rows of the same outputs; plain: 2 * out neighbouring rows), `out` any multiple
// of 8 up to 128 that lets the items fill the SMs in the fewest equal rounds: 5,632 outputs are 141 items of 40, not 88 of 64.
// The bands are the "N" side of the instruction (2 * out <= 256), the up to 64 rows of X its "M" side of 128; the rows of X
// that are missing are whatever lies behind in shared memory, and only their own lanes of the accumulator, which nobody
// reads, depend on them.  (With W on the "M" side an item takes two instructions for every 16 of K, each about 80 cycles
// however few the rows of X: 46 MB, 32 rows 18 us.)
//
// One persistent block an SM: a ring of stages filled by one thread, which asks for 64 to 256 of K of all rows of a stage in
// one TMA load (at a load per band and 64 of K its instructions were the limit: 23 us), the first of W while the block still
// sets itself up and the kernel in front still runs; one thread that issues the instructions; four warps that lay the
// finished sums into shared memory and write them, two neighbouring outputs a thread (with a row of X a thread writing 16
// outputs at a time one warp did it all at 32 rows: 17 us), while the next item's accumulator fills.  46 MB, 32 rows, with the
// norm kernel in front: 13.8 us, of which 1.7 are the norm's and 7.2 the reading's at the copy bandwidth; before (64 outputs a
// block, decode_gemm_tc.cu) 18.1.
//
// The grouped form (experts) multiplies the tile t of X with the rows tile_b_row[t] .. of W (negative: no more tiles) for its
// first tile_rows[t] rows only.  8 experts of 2,048 x 2,816, two a token, 16 tokens, the whole layer's experts 75.0 -> 55.1 us
// (128-row tiles of gemm_tc.cu before), 64 tokens 74.3 -> 61.4; the reading takes 43.3.
//
// All waits on mbarriers are bounded (see gemm_tc.cu): a wait that runs out raises a bit in *status, the block still frees
// its tensor memory and returns.
#include <cuda.h>

#include "common.cuh"

#define DP_BK 64
#define DP_THREADS 192
#define DP_MAX_STAGES 12
#define DP_RING_BYTES (160 * 1024)
#define DP_TILE 64                       /* rows of X at most */
#define DP_WAIT_CYCLES (4000000000ll)

struct DecodePairArgs {
    const float* bias;
    void* Y;
    int M, N, K, ldy;
    int out;                             // rows of W in a band
    int second;                          // W row of an item's second band, counted from its first
    int chunks, items;                   // items per tile of X, and in all
    int acc_cols, tmem_cols;             // columns of an accumulator, and allocated
    int vec_out;                         // pairs of outputs may be stored together
    uint32_t sums_at;                    // where the finished sums lie in shared memory: behind the ring, or (one item a
                                         // block) over it
    int stages, chunks_k;                // stages of the ring, and how many times 64 of K a stage holds
    int x_tile;                          // rows of X in a stage (a multiple of 16), and of a tile of the grouped form
    int whole_k;                         // K is a multiple of 64 (else a stage holds 64 of K)
    const int *tile_b_row, *tile_rows;   // grouped form, else null
    int act, accumulate;
    int* status;
};

__device__ __forceinline__ uint32_t dp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool dp_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    for (uint32_t i = 1;; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((i & 255u) == 0 && clock64() - t0 > DP_WAIT_CYCLES) return false;
    }
}
__device__ __forceinline__ void dp_tma(uint32_t dst, const CUtensorMap* map, int c0, int row, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n"
        ::"r"(dst), "l"(map), "r"(c0), "r"(row), "r"(0), "r"(c3), "r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t dp_desc(uint32_t saddr) {      // K-major tile, 128-byte swizzle (see gemm_tc.cu)
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void dp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void dp_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// 32 lanes x 16 columns of tensor memory: 16 neighbouring columns of the thread's lane
__device__ __forceinline__ void dp_ld16(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}

// A block's shared memory: stages of [out rows | out rows | up to 64 rows of X] x 128 bytes, room for the rows that the
// last stage's instructions read past it, the barriers.
template <bool GATED, typename TO>
__global__ void __launch_bounds__(DP_THREADS, 1)
decode_pair_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const DecodePairArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * DP_MAX_STAGES + 4];
    __shared__ uint32_t tmem_slot, failed_flag;
    volatile uint32_t* failed = &failed_flag;
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full = bars, *empty = bars + DP_MAX_STAGES, *acc_full = bars + 2 * DP_MAX_STAGES, *acc_empty = acc_full + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stages = a.stages, CK = a.chunks_k, k_iters = (a.K + CK * DP_BK - 1) / (CK * DP_BK);
    const uint32_t band = (uint32_t)a.out * 128u, x_bytes = (uint32_t)a.x_tile * 128u;
    const uint32_t stage_bytes = (uint32_t)CK * (2 * band + x_bytes);

    // item w -> first row of W, first output, first row of X, live rows; false: there are no more items.  (The grouped
    // form's lists were written by a kernel that ended before the one in front of this began: they, and W, may be read
    // before pdl_wait().)
    auto item = [&](int w, int& b_row, int& n0, int& x_row, int& rows) {
        const int t = w / a.chunks;
        n0 = (w - t * a.chunks) * a.out * (GATED ? 1 : 2);
        b_row = n0;
        x_row = 0;
        rows = a.M;
        if (a.tile_b_row) {
            const int b = a.tile_b_row[t];
            if (b < 0) return false;
            b_row += b;
            x_row = t * a.x_tile;
            rows = a.tile_rows[t];
        }
        return true;
    };

    const uint32_t tiles_at = dp_smem(tiles), full_at = dp_smem(full), empty_at = dp_smem(empty);
    auto load_w = [&](int i, int b_row, uint32_t dst, uint32_t fb) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb), "r"(stage_bytes) : "memory");
        dp_tma(dst, &map_w, a.whole_k ? 0 : i * DP_BK, b_row, a.whole_k ? i * CK : 0, fb);
    };
    const int ahead = min(k_iters, stages);                // stages filled at once
    if (threadIdx.x == 32) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_x) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&empty[s])));
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&acc_full[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&acc_empty[b])));
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        // the first stages' rows of W, before the kernel in front has ended and while this block sets itself up
        int b_row, n0, x_row, rows;
        if (item(blockIdx.x, b_row, n0, x_row, rows))
            for (int i = 0; i < ahead; ++i) load_w(i, b_row, tiles_at + i * stage_bytes, full_at + i * 8);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(dp_smem(&tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    if (!(warp == 0 && lane == 0)) { pdl_wait(); pdl_launch(); }
    if (warp == 0 && lane == 0) {
        // ---- producer.  (One thread issues all of this: the stage's number, address and phase are kept, not computed.) ----
        uint32_t s = 0, phase = 1, at = tiles_at;          // phase of `empty` to wait for: a fresh barrier's waits for 1 pass
        auto next = [&]() {
            at += stage_bytes;
            if (++s == (uint32_t)stages) { s = 0; at = tiles_at; phase ^= 1; }
        };
        bool ok = true;
        pdl_wait();
        pdl_launch();
        for (int w = blockIdx.x; w < a.items && ok; w += gridDim.x) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            for (int i = 0; i < k_iters; ++i, next()) {
                const uint32_t fb = full_at + s * 8;
                if (w != (int)blockIdx.x || i >= ahead) {
                    if (!dp_wait(empty_at + s * 8, phase)) { *failed = 1; ok = false; break; }
                    load_w(i, b_row, at, fb);
                }
                dp_tma(at + CK * 2 * band, &map_x, a.whole_k ? 0 : i * DP_BK, x_row, a.whole_k ? i * CK : 0, fb);
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        uint32_t s = 0, phase = 0, at = tiles_at, local = 0;
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.out >> 2) << 17) | (8u << 24);
        bool ok = true;
        for (int w = blockIdx.x; w < a.items && ok; w += gridDim.x, ++local) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            const uint32_t buf = local & 1, d = tmem_base + buf * a.acc_cols;
            if (!dp_wait(dp_smem(&acc_empty[buf]), ((local >> 1) & 1) ^ 1)) { *failed = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int i = 0; i < k_iters; ++i) {
                if (!dp_wait(full_at + s * 8, phase)) { *failed = 1; ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                for (int c = 0; c < CK; ++c) {
                    const uint64_t w0 = dp_desc(at + c * 2 * band), x0 = dp_desc(at + CK * 2 * band + c * x_bytes);
#pragma unroll
                    for (int k = 0; k < DP_BK / 16; ++k)   // (16 of K are 32 bytes: 2 in the descriptor's units)
                        dp_mma(d, x0 + k * 2, w0 + k * 2, idesc, (i + c + k > 0) ? 1u : 0u);
                }
                dp_commit(empty_at + s * 8);
                at += stage_bytes;
                if (++s == (uint32_t)stages) { s = 0; at = tiles_at; phase ^= 1; }
            }
            if (ok) dp_commit(dp_smem(&acc_full[buf]));
        }
    } else if (warp >= 2) {
        // ---- epilogue: the sums to shared memory, a row of X a thread; then every thread two outputs at a time ----
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;                 // row of X = lane of tensor memory
        const int ld = a.acc_cols + 4;
        float* sums = reinterpret_cast<float*>(tiles + a.sums_at);
        uint32_t local = 0;
        for (int w = blockIdx.x; w < a.items; w += gridDim.x, ++local) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            const uint32_t buf = local & 1;
            // (a wait that runs out leaves the sums wrong and the flag raised; the warps stay together)
            if (!dp_wait(dp_smem(&acc_full[buf]), (local >> 1) & 1)) *failed = 1;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (quarter * 32 < rows) {
                const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * a.acc_cols;
                float* mine = sums + r * ld;
                for (int c = 0; c < a.acc_cols; c += 16) {
                    float v[16];
                    dp_ld16(t_row + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (r < rows)
#pragma unroll
                        for (int j = 0; j < 16; j += 4)
                            *reinterpret_cast<float4*>(mine + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
            if (threadIdx.x == 64) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(dp_smem(&acc_empty[buf])) : "memory");
            const int outs = GATED ? a.out : a.acc_cols, pairs = outs / 2;
            for (int idx = threadIdx.x - 64; idx < rows * pairs; idx += 128) {
                const int m = idx / pairs, c = (idx - m * pairs) * 2, n = n0 + c;
                if (n >= a.N) continue;
                const bool two = n + 1 < a.N;
                float2 v = *reinterpret_cast<const float2*>(sums + m * ld + c);
                if (a.bias) { v.x += a.bias[n]; if (two) v.y += a.bias[n + 1]; }
                if (GATED) {               // (a bfloat16 result keeps 8 bits: the fast exponential and division do)
                    float2 u = *reinterpret_cast<const float2*>(sums + m * ld + a.out + c);
                    if (a.bias) { u.x += a.bias[n + a.N]; if (two) u.y += a.bias[n + 1 + a.N]; }
                    v.x = (sizeof(TO) == 2 ? gated_act_fast(v.x, a.act) : gated_act(v.x, a.act)) * u.x;
                    v.y = (sizeof(TO) == 2 ? gated_act_fast(v.y, a.act) : gated_act(v.y, a.act)) * u.y;
                } else if (a.act == TQ_ACT_SQUARE_RELU) {
                    v.x = square_relu(v.x);
                    v.y = square_relu(v.y);
                }
                TO* y = reinterpret_cast<TO*>(a.Y) + (size_t)(x_row + m) * a.ldy + n;
                if (GATED && sizeof(TO) == 4 && a.accumulate) {
                    v.x += to_f32<TO>(y[0]);
                    if (two) v.y += to_f32<TO>(y[1]);
                }
                if (a.vec_out && two) {
                    store2_f32<TO>(y, v.x, v.y);
                } else {
                    y[0] = from_f32<TO>(v.x);
                    if (two) y[1] = from_f32<TO>(v.y);
                }
            }
            asm volatile("bar.sync 1, 128;\n" ::: "memory");        // the next item's sums may come
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && *failed && a.status) atomicOr(a.status, 2);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((uint32_t)a.tmem_cols) : "memory");
}

// A matrix of rows of K entries as [chunk of 64 of K][band][row][64 of K] (bands `second` rows apart), of which a box is
// chunks_k x bands x box_rows x 64: one TMA load brings a stage's share.  If K is no multiple of 64, the innermost extent is K
// (its end is filled with zeros) and a stage holds one chunk.
static int dp_make_map(CUtensorMap* map, const void* base, uint64_t rows, int K, uint64_t ld, int bands, uint64_t second,
                       int box_rows, int chunks_k, bool whole_k) {
    const cuuint64_t dims[4] = {(cuuint64_t)(whole_k ? DP_BK : K), rows, (cuuint64_t)bands, (cuuint64_t)(whole_k ? K / DP_BK : 1)};
    const cuuint64_t strides[3] = {ld * 2, second * ld * 2, DP_BK * 2};
    const cuuint32_t box[4] = {DP_BK, (cuuint32_t)box_rows, (cuuint32_t)bands, (cuuint32_t)chunks_k};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims,
                                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 1000 + (int)r;
}

// Rows of a band: the multiple of 8 up to 128 with which the busiest SM reads least, an item costing its two bands plus
// about 24 rows of K = 2,048 (filling the ring and writing the result: 1 us at an SM's share of the copy bandwidth).
static int dp_band(int tiles, int outputs_per_tile, int per_item, int K) {
    int best = 128;
    double least = 1e30;
    for (int out = 128; out >= 16; out -= 8) {
        const long long chunks = (outputs_per_tile + (long long)out * per_item - 1) / ((long long)out * per_item);
        const long long rounds = (chunks * tiles + tq_sm_count() - 1) / tq_sm_count();
        const double cost = (double)rounds * (2.0 * out * K + 24.0 * 2048.0);
        if (cost < least) { least = cost; best = out; }
    }
    return best;
}

template <bool GATED, typename TO>
static int launch_decode_pair(const void* X, long long x_rows, int ldx, const void* W, long long w_rows, int ldw,
                              DecodePairArgs a, int tiles, int live, cudaStream_t stream) {
    a.out = dp_band(live, a.N, GATED ? 1 : 2, a.K);
    a.chunks = (a.N + a.out * (GATED ? 1 : 2) - 1) / (a.out * (GATED ? 1 : 2));
    a.items = a.chunks * tiles;
    a.whole_k = a.K % DP_BK == 0;
    a.chunks_k = !a.whole_k || a.out > 80 ? 1 : (a.out > 32 ? 2 : 4);      // 10 to 32 KB of W a stage
    const int stage = a.chunks_k * (2 * a.out + a.x_tile) * 128;
    const int grid = a.items < tq_sm_count() ? a.items : tq_sm_count();
    const bool rounds = a.items > grid;
    const int sums = a.x_tile * (2 * a.out + 4) * 4, past = (128 - a.x_tile) * 128;
    constexpr int MOST = 220 * 1024;
    a.stages = DP_RING_BYTES / stage < DP_MAX_STAGES ? DP_RING_BYTES / stage : DP_MAX_STAGES;
    while (a.stages > 2 && a.stages * stage + past + (rounds ? sums : 0) + 1024 > MOST) --a.stages;
    const int ring = a.stages * stage + past;
    a.sums_at = rounds ? (uint32_t)ring : 0u;
    const int smem = (rounds ? ring + sums : (ring > sums ? ring : sums)) + 1024;
    a.acc_cols = 2 * a.out;
    a.tmem_cols = 32;
    while (a.tmem_cols < a.acc_cols * (rounds ? 2 : 1)) a.tmem_cols *= 2;
    a.vec_out = !(reinterpret_cast<uintptr_t>(a.Y) & (2 * sizeof(TO) - 1)) && a.ldy % 2 == 0;
    if (smem > MOST || a.stages < 2) return (int)cudaErrorInvalidValue;
    static bool configured[64] = {false};                    // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(decode_pair_tc_kernel<GATED, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    CUtensorMap mw, mx;
    // plain: one band of 2 * out rows
    int st = GATED ? dp_make_map(&mw, W, (uint64_t)(w_rows - a.second), a.K, (uint64_t)ldw, 2, (uint64_t)a.second, a.out,
                                 a.chunks_k, a.whole_k)
                   : dp_make_map(&mw, W, (uint64_t)w_rows, a.K, (uint64_t)ldw, 1, 1, 2 * a.out, a.chunks_k, a.whole_k);
    if (st) return st;
    st = dp_make_map(&mx, X, (uint64_t)x_rows, a.K, (uint64_t)ldx, 1, 1, a.x_tile, a.chunks_k, a.whole_k);
    if (st) return st;
    return tq_launch_pdl(TQ_PDL_DECODE_GEMM, decode_pair_tc_kernel<GATED, TO>, dim3(grid), dim3(DP_THREADS), smem, stream, mw,
                         mx, a);
}

static bool dp_operands_ok(const void* X, const void* W, int K, int ldx, int ldw) {
    return K > 0 && !(K & 7) && !(ldx & 7) && !(ldw & 7) && !(reinterpret_cast<uintptr_t>(X) & 15) &&
           !(reinterpret_cast<uintptr_t>(W) & 15);
}

// Gated product of up to 64 rows: X [M, K], W [2N, K] (gate rows, then up rows) bfloat16, rows of 16-byte pieces; Y [M, N]
// float32 or bfloat16 (accumulate: float32); bias [2N] float32 or null; act TQ_ACT_SILU or TQ_ACT_GELU_TANH.
TQ_API int tq_decode_pair_tc(const void* X, const void* W, const float* bias, void* Y, int y_dtype, int M, int N, int K, int ldx,
                             int ldw, int ldy, int accumulate, int act, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > DP_TILE || (accumulate && y_dtype != TQ_F32) || !dp_operands_ok(X, W, K, ldx, ldw) || (act != TQ_ACT_SILU && act != TQ_ACT_GELU_TANH))
        return (int)cudaErrorInvalidValue;
    DecodePairArgs a{bias, Y, M, N, K, ldy, 0, N, 0, 0, 0, 0, 0, 0, 0, 0, (M + 15) / 16 * 16, 0, nullptr, nullptr, act, accumulate, status};
    if (y_dtype == TQ_BF16) return launch_decode_pair<true, bf16>(X, M, ldx, W, 2ll * N, ldw, a, 1, 1, stream);
    if (y_dtype == TQ_F32) return launch_decode_pair<true, float>(X, M, ldx, W, 2ll * N, ldw, a, 1, 1, stream);
    return (int)cudaErrorInvalidValue;
}

// Many products in one launch: X [tiles * tile, K] (tile: 16, 32, 48 or 64 rows); tile t's first tile_rows[t] (at least 1) rows multiply with the N (gated: 2N)
// rows of W [w_rows, K] from row tile_b_row[t] on; the first negative entry ends the list, rows of Y of no live row stay as
// they are; the work is cut for `live` of them.  gate: TQ_ACT_SILU / TQ_ACT_GELU_TANH a gated product, TQ_ACT_SQUARE_RELU or 0 a plain one.  tile_b_row,
// tile_rows and W were complete before the kernel in front of this one began.
TQ_API int tq_decode_pair_tc_grouped(const void* X, const void* W, void* Y, int y_dtype, int tile, int tiles, int live, int N, int K, int ldx,
                                     int ldw, int ldy, int gate, int w_rows, const int* tile_b_row, const int* tile_rows,
                                     int* status, cudaStream_t stream) {
    if (tiles <= 0 || N <= 0) return 0;
    if (!dp_operands_ok(X, W, K, ldx, ldw) || w_rows <= 0 || live <= 0 || live > tiles || tile <= 0 || tile > DP_TILE || tile % 16 || !tile_b_row || !tile_rows ||
        gate < 0 || gate > TQ_ACT_SQUARE_RELU)
        return (int)cudaErrorInvalidValue;
    DecodePairArgs a{nullptr, Y, tile, N, K, ldy, 0, N, 0, 0, 0, 0, 0, 0, 0, 0, tile, 0, tile_b_row, tile_rows, gate, 0, status};
    const long long x_rows = (long long)tiles * tile;
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
#define TQ_DP(G, T) return launch_decode_pair<G, T>(X, x_rows, ldx, W, w_rows, ldw, a, tiles, live, stream)
    if (gated && y_dtype == TQ_BF16) TQ_DP(true, bf16);
    if (gated && y_dtype == TQ_F32) TQ_DP(true, float);
    if (!gated && y_dtype == TQ_BF16) TQ_DP(false, bf16);
    if (!gated && y_dtype == TQ_F32) TQ_DP(false, float);
#undef TQ_DP
    return (int)cudaErrorInvalidValue;
}
