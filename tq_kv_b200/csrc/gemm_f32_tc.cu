// The float32 products of many rows on the tcgen05 tensor cores, without giving up a bit of the operands:
// C[M,N] (=, +=) A[M,K] · W[N,K]^T (+ bias[N]), float32 operands and result; epilogues as in gemm_f32.cu.
//
// A float32 number is the sum of three bfloat16 numbers, x = x1 + x2 + x3: its first 8 bits, the next 8 rounded, and the rest.
// The split is exact.  A product is then the sum of six exact bfloat16 products,
//   x1 w3 + x3 w1 + x2 w2  +  x1 w2 + x2 w1  +  x1 w1,
// and what is left out, x2 w3 + x3 w2 + x3 w3, is below 2^-23 of the product, 2^-25 on average, and of either sign.  The tensor
// cores sum in float32, but cut off as they go: so an accumulator lives for 32 of K only, its small terms first, and the
// accumulators of the steps are added up in registers with float32 additions.  Error against 64 bits, 2-norm, the FMA tiles of
// gemm_f32.cu / here: K = 32 7.9e-8 / 6.4e-8, K = 100 9.1e-8 / 7.7e-8, K = 4,864 3.2e-7 / 1.2e-7, gated K = 896 4.0e-7 / 2.0e-7;
// all numbers positive, K = 4,864: 8.6e-8 / 7.7e-8.
//
// Numbers that the split does not give back (infinities, NaN, numbers whose third part is below bfloat16's smallest) leave
// low bits in the third part; a block that meets one computes its share again with float32 multiply-adds.
//
// A block makes a tile of 128 x 256 outputs.  Eight warps load the float32 rows of the next step, split those they have and
// write the six bfloat16 tiles of a step (64-byte rows, 64-byte swizzle) into one of two buffers; before a buffer is refilled
// they add the accumulator that came of it to their registers (32 lanes x 128 columns a warp), while the other buffer's
// instructions run.  A thread of a third warpgroup issues the instructions: the tensor pipe lets the issuing thread wait, and one
// of the eight warps that issued them was late with its own share each time.  Registers move from that warpgroup to the others.
// Where tiles are fewer than the SMs, K is cut over a cluster of up to eight blocks whose partial tiles meet through
// distributed shared memory in the order of the ranks: results do not depend on timing.
//
// Measured (weights not in the cache, us, gemm_f32.cu / here): gated N = 4,864, K = 896: 64 rows 38 / 25, 300 rows 141 / 57 (92
// TFLOP/s; the float32 lanes have 72), 700 rows 273 / 111; N = 896, K = 4,864, 300 rows 96 / 38; N = 151,936, K = 896, 300 rows
// 1,812 / 692; gated N = 5,632, K = 2,048, 700 rows 703 / 217.  A step of 32 of K takes 2,900 cycles, of which the instructions
// need 1,540; other forms that took as long or longer: 128 columns a tile on 8 warps (two blocks an SM) and on 16, steps of 64
// of K with 128-byte rows, two groups of warps in turn, four warps that split and eight that add.
//
// All waits on mbarriers are bounded (see gemm_tc.cu): a wait that runs out raises a bit in *status.
#include <cooperative_groups.h>

#include "common.cuh"

#define FS_BM 128
#define FS_BN 256
#define FS_BK 32
#define FS_WORKERS 256
#define FS_THREADS 384
#define FS_MAX_SPLIT 8
#define FS_WAIT_CYCLES (4000000000ll)

struct F32SplitArgs {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc, accumulate, act, vec_out;
    int settled;              // W was complete before the kernel in front of this one began: read it before that one ends
    int* status;
};

__device__ __forceinline__ uint32_t fs_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool fs_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    for (uint32_t i = 1;; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((i & 255u) == 0 && clock64() - t0 > FS_WAIT_CYCLES) return false;
    }
}
// Shared-memory descriptor of a K-major tile with rows of 64 bytes and 64-byte swizzle: groups of 8 rows (512 bytes) follow
// each other
__device__ __forceinline__ uint64_t fs_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ void fs_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// (an offset into the tile changes the low word only)
__device__ __forceinline__ uint64_t fs_step(uint64_t desc, uint32_t bytes) {
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;\n" : "=r"(lo), "=r"(hi) : "l"(desc));
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(desc) : "r"(lo + (bytes >> 4)), "r"(hi));
    return desc;
}
__device__ __forceinline__ void fs_ld16(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
// Two numbers -> their three parts, packed; `rest` gathers the bits of the third parts that bfloat16 would drop.  The first
// part is cut off, the second rounded: the third is then of either sign, and so are the products that are left out.
__device__ __forceinline__ void fs_split2(float2 x, uint32_t& p1, uint32_t& p2, uint32_t& p3, uint32_t& rest) {
    const float2 minus = make_float2(-1.f, -1.f);
    p1 = __byte_perm(__float_as_uint(x.x), __float_as_uint(x.y), 0x7632);
    x = __ffma2_rn(make_float2(__uint_as_float(__float_as_uint(x.x) & 0xffff0000u), __uint_as_float(__float_as_uint(x.y) & 0xffff0000u)),
                   minus, x);
    const __nv_bfloat162 h = __floats2bfloat162_rn(x.x, x.y);
    p2 = *reinterpret_cast<const uint32_t*>(&h);
    x = __ffma2_rn(make_float2(__uint_as_float(p2 << 16), __uint_as_float(p2 & 0xffff0000u)), minus, x);
    p3 = __byte_perm(__float_as_uint(x.x), __float_as_uint(x.y), 0x7632);
    rest |= __float_as_uint(x.x) | __float_as_uint(x.y);
}

// Grid (row tiles * split, column tiles), clusters of `split` blocks along x.  GATED: a tile holds BN / 2 gate and BN / 2 up
// rows of W, 32 and 32 in turn.
template <bool GATED>
__global__ void __launch_bounds__(FS_THREADS, 1) f32_split_kernel(const F32SplitArgs a) {
    namespace cg = cooperative_groups;
    constexpr int BN = FS_BN, A_PART = FS_BM * 64, B_PART = BN * 64, BUF = 3 * (A_PART + B_PART);
    constexpr int NA = FS_BM / 32, NB = BN / 32, COLS = BN / 2, OUT_LD = BN + 4;
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[2], done[2];
    __shared__ uint32_t tmem_slot, failed_flag, odd_flag;
    unsigned char* bufs = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    float* sm = reinterpret_cast<float*>(bufs);
    cg::cluster_group cluster = cg::this_cluster();
    const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = (blockIdx.x / split) * FS_BM;
    const int n0 = blockIdx.y * (GATED ? BN / 2 : BN);
    const int steps = (a.K + FS_BK - 1) / FS_BK;
    const int s_begin = (int)((long long)steps * rank / split), s_end = (int)((long long)steps * (rank + 1) / split);
    const int n_steps = s_end - s_begin;

    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(fs_smem(&full[b])), "r"(FS_WORKERS / 32));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(fs_smem(&done[b])));
        }
        failed_flag = 0;
        odd_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(fs_smem(&tmem_slot)), "r"((uint32_t)(2 * BN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    const int quarter = warp & 3, half = (warp >> 2) & 1;      // this warp's lanes and columns of the accumulators
    if (warp >= FS_WORKERS / 32) {
        // (40 and 224 registers: 128 x 40 + 256 x 224 are less than the 384 x 168 of the launch)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;\n");
        pdl_wait();
        pdl_launch();
        if (tid == FS_WORKERS) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (8u << 24);
            for (int s = 0; s < n_steps; ++s) {
                const int b = s & 1;
                if (!fs_wait(fs_smem(&full[b]), (s >> 1) & 1)) { failed_flag = 1; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t tile = fs_desc(fs_smem(bufs + b * BUF));
                constexpr int TA[6] = {0, 2, 1, 0, 1, 0}, TB[6] = {2, 0, 1, 1, 0, 0};  // the smallest terms first
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int k = 0; k < FS_BK / 16; ++k)
                        fs_mma(tmem_base + b * BN, fs_step(tile, TA[t] * A_PART + k * 32),
                               fs_step(tile, 3 * A_PART + TB[t] * B_PART + k * 32), idesc, (t > 0 || k > 0) ? 1u : 0u);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                             ::"r"(fs_smem(&done[b])) : "memory");
            }
        }
        __syncwarp();
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();                                     // the sums are made
        if (split > 1) cluster.sync();
        else __syncthreads();                                // ... and laid out
        if (split > 1) cluster.sync();
        else __syncthreads();                                // ... and read
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;\n");
    float acc[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
    bool in_time = true;                                     // (after a wait that ran out the rest runs without waiting)
    {
        // this thread's share of a step: 16-byte pieces (row, piece) = (tid / 8 + 32 i, tid % 8)
        const int lr = tid >> 3, piece = tid & 7;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 ra[NA], rb[NB];                               // of the next step
        // (which of them lie inside A and W, and where they start)
        uint32_t in_a = 0, in_w = 0;
#pragma unroll
        for (int i = 0; i < NA; ++i) in_a |= (uint32_t)(m0 + lr + 32 * i < a.M) << i;
#pragma unroll
        for (int i = 0; i < NB; ++i) in_w |= (uint32_t)(n0 + lr + (GATED ? (i >> 1) * 32 : i * 32) < a.N) << i;
        const float* pa = a.A + (size_t)(m0 + lr) * a.lda + (size_t)s_begin * FS_BK + piece * 4;
        const float* pw = a.W + (size_t)(n0 + lr) * a.ldw + (size_t)s_begin * FS_BK + piece * 4;
        const size_t lda32 = (size_t)a.lda * 32, ldw32 = (size_t)a.ldw * 32, to_up = GATED ? (size_t)a.N * a.ldw : 0;
        const int k_left = a.K - s_begin * FS_BK - piece * 4;                  // entries of K from this thread's first piece on
        auto load_w = [&](int step) {
            const bool in = step < n_steps && step * FS_BK < k_left;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                rb[i] = in && (in_w >> i & 1) ? *reinterpret_cast<const float4*>(pw + (GATED ? (i >> 1) * ldw32 + (i & 1) * to_up : i * ldw32) + step * FS_BK) : zero;
            }
        };
        auto load_a = [&](int step) {
            const bool in = step < n_steps && step * FS_BK < k_left;
#pragma unroll
            for (int i = 0; i < NA; ++i)
                ra[i] = in && (in_a >> i & 1) ? *reinterpret_cast<const float4*>(pa + i * lda32 + step * FS_BK) : zero;
        };
        uint32_t rest = 0;
        const uint32_t at = (uint32_t)lr * 64u + (uint32_t)(((piece >> 1) ^ ((lr >> 1) & 3)) << 4) + (uint32_t)(piece & 1) * 8u;
        auto put = [&](const float4& x, unsigned char* dst, int part) {
            uint2 p1, p2, p3;
            fs_split2(make_float2(x.x, x.y), p1.x, p2.x, p3.x, rest);
            fs_split2(make_float2(x.z, x.w), p1.y, p2.y, p3.y, rest);
            *reinterpret_cast<uint2*>(dst) = p1;
            *reinterpret_cast<uint2*>(dst + part) = p2;
            *reinterpret_cast<uint2*>(dst + 2 * part) = p3;
        };
        if (!a.settled) pdl_wait();
        load_w(0);
        pdl_wait();
        pdl_launch();
        load_a(0);
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * COLS;
        for (int s = 0; s < n_steps + 2; ++s) {
            const int b = s & 1;
            if (s >= 2) {                                    // the accumulator of the step before last; its buffer is free
                in_time = in_time && fs_wait(fs_smem(&done[b]), ((s - 2) >> 1) & 1);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    float v[16];
                    fs_ld16(t_row + b * BN + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
                }
            }
            if (s >= n_steps) continue;
            unsigned char* dst = bufs + b * BUF + at;
#pragma unroll
            for (int i = 0; i < NA; ++i) put(ra[i], dst + i * 2048, A_PART);
            load_a(s + 1);
#pragma unroll
            for (int i = 0; i < NB; ++i) put(rb[i], dst + 3 * A_PART + i * 2048, B_PART);
            load_w(s + 1);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(fs_smem(&full[b])) : "memory");
        }
        if (rest & 0xffffu) odd_flag = 1;
    }
    if (!in_time) failed_flag = 1;
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    {
        const int r = quarter * 32 + lane;
        if (odd_flag) {                                      // a number that the split does not give back: all again
            const int k_end = min(a.K, s_end * FS_BK);
            const float* x = a.A + (size_t)min(m0 + r, a.M - 1) * a.lda;
#pragma unroll 1
            for (int j0 = 0; j0 < COLS; j0 += 4) {
                const int c = half * COLS + j0;              // (four neighbouring columns: gate rows or up rows)
                const int n = n0 + (GATED ? (c >> 6) * 32 + (c & 31) : c), up = GATED && ((c >> 5) & 1) ? a.N : 0;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                for (int k = s_begin * FS_BK; k < k_end; k += 4) {
                    const float4 p = *reinterpret_cast<const float4*>(x + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 q = *reinterpret_cast<const float4*>(a.W + (size_t)(min(n + j, a.N - 1) + up) * a.ldw + k);
                        v[j] = fmaf(p.x, q.x, v[j]); v[j] = fmaf(p.y, q.y, v[j]);
                        v[j] = fmaf(p.z, q.z, v[j]); v[j] = fmaf(p.w, q.w, v[j]);
                    }
                }
                *reinterpret_cast<float4*>(sm + r * OUT_LD + c) = make_float4(v[0], v[1], v[2], v[3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < COLS; j += 4)
                *reinterpret_cast<float4*>(sm + r * OUT_LD + half * COLS + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
    }
    if (split > 1) cluster.sync();
    else __syncthreads();

    constexpr int PIECES = GATED ? BN / 8 : BN / 4;          // 16-byte pieces of an output row
    for (int idx = rank * FS_WORKERS + tid; idx < FS_BM * PIECES; idx += split * FS_WORKERS) {
        const int r = idx / PIECES, p = idx % PIECES, m = m0 + r, n = n0 + p * 4;
        if (m >= a.M || n >= a.N) continue;
        const int from = r * OUT_LD + (GATED ? (p >> 3) * 64 + (p & 7) * 4 : p * 4);
        float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < split; ++s) {
            const float* part = split > 1 ? cluster.map_shared_rank(sm, s) : sm;
            const float4 x = *reinterpret_cast<const float4*>(part + from);
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            if (GATED) {
                const float4 y = *reinterpret_cast<const float4*>(part + from + 32);
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
    else __syncthreads();
    if (tid == 0 && failed_flag && a.status) atomicOr(a.status, 2);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((uint32_t)(2 * BN)) : "memory");
}

template <bool GATED>
static int launch_f32_split(const F32SplitArgs& a, int split, cudaStream_t stream) {
    constexpr size_t smem = 2 * 3 * (FS_BM + FS_BN) * 64 + 1024;
    static_assert(smem >= (size_t)FS_BM * (FS_BN + 4) * sizeof(float) + 1024, "the finished tile reuses the buffers");
    static bool configured[64] = {false};                    // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(f32_split_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int per = GATED ? FS_BN / 2 : FS_BN;
    const long long mt = (a.M + FS_BM - 1) / FS_BM, nt = (a.N + per - 1) / per;
    if (nt > 65535 || mt * split > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(mt * split), (unsigned)nt);
    cfg.blockDim = dim3(FS_THREADS);
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, f32_split_kernel<GATED>, a);
    if (e != cudaSuccess) return (int)e;
    return tq_launch_status();
}

// How many blocks share a tile's K: the count that makes (rounds of SMs) x (steps of a share + the pipeline's fill and the
// meeting of the shares, about 4 steps) least.
static int f32_split_shares(long long tiles, int steps) {
    const long long slots = tq_sm_count();
    int best = 1;
    double least = 0;
    for (int s = 1; s <= FS_MAX_SPLIT && s <= steps; ++s) {
        const long long rounds = (tiles * s + slots - 1) / slots;
        const double t = (double)rounds * ((double)((steps + s - 1) / s) + 4.0);
        if (s == 1 || t < 0.97 * least) { best = s; least = t; }
    }
    return best;
}

// As tq_gemm_f32 (gemm_f32.cu), with the status word that the kernels' bounded waits report to.
TQ_API int tq_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                          int ldc, int accumulate, int gate, int settled, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || lda % 4 || ldw % 4 || lda < K || ldw < K || ldc < N || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) ||
        gate < 0 || gate > TQ_ACT_SQUARE_RELU)
        return (int)cudaErrorInvalidValue;
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
    F32SplitArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, gate,
                   (ldc % 4 == 0 && ((uintptr_t)C & 15) == 0) ? 1 : 0, settled, status};
    const int steps = (K + FS_BK - 1) / FS_BK;
    const long long mt = (M + FS_BM - 1) / FS_BM;
    const int per = gated ? FS_BN / 2 : FS_BN;
    const int split = f32_split_shares(mt * ((N + per - 1) / per), steps);
    return gated ? launch_f32_split<true>(a, split, stream) : launch_f32_split<false>(a, split, stream);
}
