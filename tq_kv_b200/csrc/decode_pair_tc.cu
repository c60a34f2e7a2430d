// Weight-streaming products of few rows on the tcgen05 tensor cores whose tiles are cut to the GPU: gated products of a
// decode batch, and the products of routed experts that own a few rows each.
//   Y[m, n] = act(X[m] . W[n]) * (X[m] . W[n + second])          (gated)
//   Y[m, n] = X[m] . W[n], or the square of its relu             (plain)
//
// Operands are swapped as in decode_gemm_tc.cu: rows of W are the "M" side of the instruction, the up to 64 rows of X its
// "N" side (a multiple of 16).  What bounds it is the reading of W, so every SM should read the same share of it, once.
// A work item is therefore two bands of `out` rows of W (gated: the gate rows and the up rows of the same outputs, so that a
// thread finds both factors in its own lane of tensor memory; plain: two neighbouring bands), `out` any multiple of 8 up to
// 128 that lets the items fill the SMs in the fewest equal rounds: 5,632 outputs are 141 items of 40, not 88 of 64.  The
// instruction always takes 128 rows; those past `out` are whatever lies behind in shared memory, and only their own lanes
// of the accumulator, which nobody reads, depend on them.  X is read from the L2 once per item: at 64 rows that is a
// quarter of W's bytes with out = 128, where two blocks an SM with half the rows each would read half.
//
// One persistent block an SM: warp 0 issues TMA loads into a ring of stages, warp 1 the instructions, warps 2 to 5 write
// one item's accumulators while the next item's fill the other pair.  The grouped form (experts) multiplies the 64-row
// tile t of X with the rows tile_b_row[t] .. of W (negative: no more tiles) for its first tile_rows[t] rows only.
//
// All waits on mbarriers are bounded (see gemm_tc.cu): a wait that runs out raises a bit in *status, the block still frees
// its tensor memory and returns.
#include <cuda.h>

#include "common.cuh"

#define DP_BK 64
#define DP_THREADS 192
#define DP_MAX_STAGES 12
#define DP_TILE 64                       /* rows of X: at most, and per tile of the grouped form */
#define DP_TMEM 256                      /* two pairs of accumulators of 64 columns */
#define DP_WAIT_CYCLES (4000000000ll)

struct DecodePairArgs {
    const float* bias;
    void* Y;
    int M, N, K, ldy;
    int out;                             // rows of W in a band
    int second;                          // W row of an item's second band, counted from its first
    int chunks, items;                   // items per tile of X, and in all
    int stages;
    const int *tile_b_row, *tile_rows;   // grouped form, else null
    int act;
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
__device__ __forceinline__ void dp_tma(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
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
    const int stages = a.stages, k_iters = (a.K + DP_BK - 1) / DP_BK;
    const uint32_t band = (uint32_t)a.out * 128u;
    const uint32_t stage_bytes = 2 * band + (a.tile_b_row ? DP_TILE : ((uint32_t)a.M + 15u) / 16u * 16u) * 128u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&empty[s])));
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(dp_smem(&acc_full[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(dp_smem(&acc_empty[b])));
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(dp_smem(&tmem_slot)), "r"((uint32_t)DP_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

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
            x_row = t * DP_TILE;
            rows = a.tile_rows[t];
        }
        return true;
    };

    if (!(warp == 0 && lane == 0)) { pdl_wait(); pdl_launch(); }
    if (warp == 0 && lane == 0) {
        // ---- producer: the first stages' bands of W before the kernel in front has ended, X after ----
        uint32_t it = 0;
        bool waited = false, ok = true;
        for (int w = blockIdx.x; w < a.items && ok; w += gridDim.x) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            const int boxes = (rows + 15) / 16;
            const uint32_t bytes = 2 * band + (uint32_t)boxes * 2048u;
            auto load_w = [&](int i, uint32_t at) {
                const uint32_t fb = dp_smem(&full[at % stages]), dst = dp_smem(tiles) + (at % stages) * stage_bytes;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb), "r"(bytes) : "memory");
                dp_tma(dst, &map_w, i * DP_BK, b_row, fb);
                dp_tma(dst + band, &map_w, i * DP_BK, b_row + a.second, fb);
            };
            auto load_x = [&](int i, uint32_t at) {
                const uint32_t fb = dp_smem(&full[at % stages]), dst = dp_smem(tiles) + (at % stages) * stage_bytes + 2 * band;
                for (int b = 0; b < boxes; ++b) dp_tma(dst + b * 2048, &map_x, i * DP_BK, x_row + 16 * b, fb);
            };
            int i = 0;
            if (!waited) {
                const int ahead = min(k_iters, stages);
                for (; i < ahead; ++i) load_w(i, i);
                pdl_wait();
                pdl_launch();
                waited = true;
                for (int j = 0; j < ahead; ++j) load_x(j, j);
                it = ahead;
            }
            for (; i < k_iters; ++i, ++it) {
                if (!dp_wait(dp_smem(&empty[it % stages]), ((it / stages) & 1) ^ 1)) { *failed = 1; ok = false; break; }
                load_w(i, it);
                load_x(i, it);
            }
        }
        if (!waited) { pdl_wait(); pdl_launch(); }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        uint32_t it = 0, local = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < a.items && ok; w += gridDim.x, ++local) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((rows + 15) / 16 * 2) << 17) | (8u << 24);
            const uint32_t buf = local & 1, d0 = tmem_base + buf * 128;
            if (!dp_wait(dp_smem(&acc_empty[buf]), ((local >> 1) & 1) ^ 1)) { *failed = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int i = 0; i < k_iters; ++i, ++it) {
                const uint32_t s = it % stages;
                if (!dp_wait(dp_smem(&full[s]), (it / stages) & 1)) { *failed = 1; ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t w_addr = dp_smem(tiles) + s * stage_bytes, x_addr = w_addr + 2 * band;
#pragma unroll
                for (int k = 0; k < DP_BK / 16; ++k) {
                    const uint32_t acc = (i > 0 || k > 0) ? 1u : 0u;
                    dp_mma(d0, dp_desc(w_addr + k * 32), dp_desc(x_addr + k * 32), idesc, acc);
                    dp_mma(d0 + 64, dp_desc(w_addr + band + k * 32), dp_desc(x_addr + k * 32), idesc, acc);
                }
                dp_commit(dp_smem(&empty[s]));
            }
            if (ok) dp_commit(dp_smem(&acc_full[buf]));
        }
    } else if (warp >= 2) {
        // ---- epilogue: a thread holds one output (plain: one of either band) of all rows of X ----
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;                 // row of the band = lane of tensor memory
        uint32_t local = 0;
        for (int w = blockIdx.x; w < a.items; w += gridDim.x, ++local) {
            int b_row, n0, x_row, rows;
            if (!item(w, b_row, n0, x_row, rows)) break;
            const uint32_t buf = local & 1;
            if (!dp_wait(dp_smem(&acc_full[buf]), (local >> 1) & 1)) { *failed = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (quarter * 32 < a.out) {
                const int c0 = n0 + r, c1 = c0 + a.out;    // (plain: the second band's output)
                const bool on0 = r < a.out && c0 < a.N, on1 = r < a.out && c1 < a.N;
                float b0 = 0.f, b1 = 0.f;
                if (a.bias) {
                    if (on0) b0 = a.bias[c0];
                    if (GATED ? on0 : on1) b1 = a.bias[GATED ? c0 + a.N : c1];
                }
                const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * 128;
                for (int m0 = 0; m0 < rows; m0 += 16) {
                    float v[16], u[16];
                    dp_ld16(t_row + m0, v);
                    dp_ld16(t_row + 64 + m0, u);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    TO* y = reinterpret_cast<TO*>(a.Y) + (size_t)(x_row + m0) * a.ldy;
#pragma unroll
                    for (int j = 0; j < 16; ++j, y += a.ldy) {
                        if (m0 + j >= rows) break;
                        float p = v[j] + b0, q = u[j] + b1;
                        if (GATED) {       // (a bfloat16 result keeps 8 bits: the fast exponential and division do)
                            p = (sizeof(TO) == 2 ? gated_act_fast(p, a.act) : gated_act(p, a.act)) * q;
                            if (on0) y[c0] = from_f32<TO>(p);
                        } else {
                            if (a.act == TQ_ACT_SQUARE_RELU) { p = square_relu(p); q = square_relu(q); }
                            if (on0) y[c0] = from_f32<TO>(p);
                            if (on1) y[c1] = from_f32<TO>(q);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(dp_smem(&acc_empty[buf])) : "memory");
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && *failed && a.status) atomicOr(a.status, 2);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((uint32_t)DP_TMEM) : "memory");
}

static int dp_make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {DP_BK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
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
                              DecodePairArgs a, int tiles, cudaStream_t stream) {
    a.out = dp_band(tiles, a.N, GATED ? 1 : 2, a.K);
    if (!GATED) a.second = a.out;
    a.chunks = (a.N + a.out * (GATED ? 1 : 2) - 1) / (a.out * (GATED ? 1 : 2));
    a.items = a.chunks * tiles;
    const int x_bytes = (a.tile_b_row ? DP_TILE : (a.M + 15) / 16 * 16) * 128;
    const int stage = 2 * a.out * 128 + x_bytes;
    static int budget = 0;
    if (!budget) { const char* e = getenv("TQ_DP_KB"); budget = (e ? atoi(e) : 168) * 1024; }
    a.stages = budget / stage;
    if (a.stages > DP_MAX_STAGES) a.stages = DP_MAX_STAGES;
    const int smem = a.stages * stage + (128 - a.out) * 128 + 1024;
    constexpr int MOST = 200 * 1024;
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
    int st = dp_make_map(&mw, W, (uint64_t)w_rows, (uint64_t)a.K, (uint64_t)ldw, (uint32_t)a.out);
    if (st) return st;
    st = dp_make_map(&mx, X, (uint64_t)x_rows, (uint64_t)a.K, (uint64_t)ldx, 16);
    if (st) return st;
    const int grid = a.items < tq_sm_count() ? a.items : tq_sm_count();
    return tq_launch_pdl(TQ_PDL_DECODE_GEMM, decode_pair_tc_kernel<GATED, TO>, dim3(grid), dim3(DP_THREADS), smem, stream, mw,
                         mx, a);
}

static bool dp_operands_ok(const void* X, const void* W, int K, int ldx, int ldw) {
    return K > 0 && !(K & 7) && !(ldx & 7) && !(ldw & 7) && !(reinterpret_cast<uintptr_t>(X) & 15) &&
           !(reinterpret_cast<uintptr_t>(W) & 15);
}

// Gated product of up to 64 rows: X [M, K], W [2N, K] (gate rows, then up rows) bfloat16, rows of 16-byte pieces; Y [M, N]
// float32 or bfloat16; bias [2N] float32 or null; act TQ_ACT_SILU or TQ_ACT_GELU_TANH.
TQ_API int tq_decode_pair_tc(const void* X, const void* W, const float* bias, void* Y, int y_dtype, int M, int N, int K, int ldx,
                             int ldw, int ldy, int act, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > DP_TILE || !dp_operands_ok(X, W, K, ldx, ldw) || (act != TQ_ACT_SILU && act != TQ_ACT_GELU_TANH))
        return (int)cudaErrorInvalidValue;
    DecodePairArgs a{bias, Y, M, N, K, ldy, 0, N, 0, 0, 0, nullptr, nullptr, act, status};
    if (y_dtype == TQ_BF16) return launch_decode_pair<true, bf16>(X, M, ldx, W, 2ll * N, ldw, a, 1, stream);
    if (y_dtype == TQ_F32) return launch_decode_pair<true, float>(X, M, ldx, W, 2ll * N, ldw, a, 1, stream);
    return (int)cudaErrorInvalidValue;
}

// Many products in one launch: X [tiles * 64, K]; tile t's first tile_rows[t] (1 .. 64) rows multiply with the N (gated: 2N)
// rows of W [w_rows, K] from row tile_b_row[t] on; the first negative entry ends the list, rows of Y of no live row stay as
// they are.  gate: TQ_ACT_SILU / TQ_ACT_GELU_TANH a gated product, TQ_ACT_SQUARE_RELU or 0 a plain one.  tile_b_row,
// tile_rows and W were complete before the kernel in front of this one began.
TQ_API int tq_decode_pair_tc_grouped(const void* X, const void* W, void* Y, int y_dtype, int tiles, int N, int K, int ldx,
                                     int ldw, int ldy, int gate, int w_rows, const int* tile_b_row, const int* tile_rows,
                                     int* status, cudaStream_t stream) {
    if (tiles <= 0 || N <= 0) return 0;
    if (!dp_operands_ok(X, W, K, ldx, ldw) || w_rows <= 0 || !tile_b_row || !tile_rows || gate < 0 || gate > TQ_ACT_SQUARE_RELU)
        return (int)cudaErrorInvalidValue;
    DecodePairArgs a{nullptr, Y, DP_TILE, N, K, ldy, 0, N, 0, 0, 0, tile_b_row, tile_rows, gate, status};
    const long long x_rows = (long long)tiles * DP_TILE;
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
#define TQ_DP(G, T) return launch_decode_pair<G, T>(X, x_rows, ldx, W, w_rows, ldw, a, tiles, stream)
    if (gated && y_dtype == TQ_BF16) TQ_DP(true, bf16);
    if (gated && y_dtype == TQ_F32) TQ_DP(true, float);
    if (!gated && y_dtype == TQ_BF16) TQ_DP(false, bf16);
    if (!gated && y_dtype == TQ_F32) TQ_DP(false, float);
#undef TQ_DP
    return (int)cudaErrorInvalidValue;
}
