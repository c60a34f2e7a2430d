// Matrix product of one row (decoding one sequence): Y[N] (=, +=) X[K] · W[N,K]^T, bfloat16 operands, float32
// multiply-adds (a product of two bfloat16 numbers is exact in float32) and float32 sums.  With one row the tensor cores
// have nothing to do: the product is the reading of W, and what counts is that as much of W as possible is on its way at
// any time, from the first instruction on.
//
// A group of KW warps makes NC = 4 neighbouring columns (rows of W; two gate and two up rows of a gated product).  A warp
// takes pieces of 256 entries of K (16 bytes a lane and row of W) in turn, two of them in registers; the first two are
// asked for before the kernel waits for its predecessor, if W is settled.  64 registers a thread keep four blocks of eight warps on an SM,
// so up to 128 KB an SM are in flight.  KW is the largest of 1, 2, 4, 8 with which all warps still run at once.  The lanes'
// sums meet by trading halves, the warps' in shared memory in warp order: no atomics, nothing to clear, and the result
// does not depend on timing.
//
// Measured in replayed graphs of the same product with other weights, in us, against the kernel that ran before
// (skinny_gemm.cu or decode_gemm_tc.cu): N = 2,048, K = 5,632 (23 MB) 7.1 -> 6.5; 3,584 x 3,584 (26 MB) 7.1 -> 6.4;
// 151,936 x 896 (272 MB) 48.8 -> 41.5, the copy bandwidth.  Which products come here: kernels/gemm.py.
#include "common.cuh"

#define RG_WARPS 8
#define RG_NC 4

struct RowGemmArgs {
    const bf16* X;
    const bf16* W;
    const float* bias;
    void* Y;
    int N, K, ldw, accumulate, act;
    int settled;              // W was complete before the kernel in front of this one began: read it before that one ends
};

__device__ __forceinline__ uint4 rg_load(const bf16* p) {
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void rg_widen(const uint4& v, float2 (&f)[4]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}

template <int KW, bool GATED, typename TO>
__global__ void __launch_bounds__(RG_WARPS * 32, 4) row_gemm_kernel(const RowGemmArgs a) {
    constexpr int OUT = GATED ? RG_NC / 2 : RG_NC, GROUPS = RG_WARPS / KW;
    __shared__ float red[RG_WARPS][RG_NC];
    const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) % KW, group = (threadIdx.x >> 5) / KW;
    const int n0 = (blockIdx.x * GROUPS + group) * OUT;
    const int pieces = (a.K + 255) / 256;
    const bf16* wrow[RG_NC];
#pragma unroll
    for (int c = 0; c < RG_NC; ++c) {
        const int n = min(n0 + (GATED ? c >> 1 : c), a.N - 1);           // columns past the last repeat it, unused
        wrow[c] = a.W + (size_t)(n + (GATED && (c & 1) ? a.N : 0)) * a.ldw + lane * 8;
    }
    auto load = [&](int piece, uint4 (&w)[RG_NC]) {
        const bool in = piece * 256 + lane * 8 < a.K;                    // (K is a multiple of 8; also false past the last piece)
#pragma unroll
        for (int c = 0; c < RG_NC; ++c) w[c] = in ? rg_load(wrow[c] + piece * 256) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 w0[RG_NC], w1[RG_NC];
    if (!a.settled) pdl_wait();
    load(part, w0);
    load(part + KW, w1);
    pdl_wait();
    pdl_launch();
    float2 acc[RG_NC];
#pragma unroll
    for (int c = 0; c < RG_NC; ++c) acc[c] = make_float2(0.f, 0.f);
    auto multiply = [&](int piece, const uint4 (&w)[RG_NC]) {
        const int k = piece * 256 + lane * 8;
        const uint4 x = k < a.K ? *reinterpret_cast<const uint4*>(a.X + k) : make_uint4(0u, 0u, 0u, 0u);
        float2 xf[4];
        rg_widen(x, xf);
#pragma unroll
        for (int c = 0; c < RG_NC; ++c) {
            float2 wf[4];
            rg_widen(w[c], wf);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[c] = __ffma2_rn(xf[e], wf[e], acc[c]);
        }
    };
    for (int piece = part; piece < pieces; piece += 2 * KW) {
        multiply(piece, w0);
        load(piece + 2 * KW, w0);
        multiply(piece + KW, w1);                                        // (past the last piece: zeros)
        load(piece + 3 * KW, w1);
    }
    // four sums over 32 lanes: two steps that halve the sums a lane holds, then the lanes with the same sum
    float v[RG_NC];
#pragma unroll
    for (int c = 0; c < RG_NC; ++c) v[c] = acc[c].x + acc[c].y;
    const bool high = lane & 16, odd = lane & 8;
    v[0] = (high ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, high ? v[0] : v[2], 16);
    v[1] = (high ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, high ? v[1] : v[3], 16);
    v[0] = (odd ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 8);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    if ((lane & 7) == 0) red[threadIdx.x >> 5][(high ? 2 : 0) + (odd ? 1 : 0)] = v[0];
    __syncthreads();
    const int n = blockIdx.x * GROUPS * OUT + threadIdx.x;
    if (threadIdx.x < GROUPS * OUT && n < a.N) {
        const int first = threadIdx.x / OUT * KW, at = (GATED ? 2 : 1) * (threadIdx.x % OUT);
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
        if (GATED)                 // (a bfloat16 result keeps 8 bits: the fast exponential and division do)
            y = (sizeof(TO) == 2 ? gated_act_fast(y, a.act) : gated_act(y, a.act)) * u;
        else if (a.act == TQ_ACT_SQUARE_RELU)
            y = square_relu(y);
        TO* out = reinterpret_cast<TO*>(a.Y) + n;
        if (a.accumulate) y += to_f32<TO>(*out);
        *out = from_f32<TO>(y);
    }
}

template <bool GATED, typename TO>
static int launch_row_gemm(const RowGemmArgs& a, cudaStream_t stream) {
    const int out = GATED ? RG_NC / 2 : RG_NC, pieces = (a.K + 255) / 256;
    const long long groups = (a.N + out - 1) / out, slots = 32LL * tq_sm_count();
#define TQ_RG(KW)                                                                                                  \
    return tq_launch_pdl(TQ_PDL_SKINNY, row_gemm_kernel<KW, GATED, TO>,                                            \
                         dim3((unsigned)((groups + RG_WARPS / KW - 1) / (RG_WARPS / KW))), dim3(RG_WARPS * 32), 0, \
                         stream, a)
    if (groups * 8 <= slots && pieces >= 8) TQ_RG(8);
    if (groups * 4 <= slots && pieces >= 4) TQ_RG(4);
    if (groups * 2 <= slots + slots / 16 && pieces >= 2) TQ_RG(2);
    TQ_RG(1);
#undef TQ_RG
}

// X [K] bf16, W [N, K] (or [2N, K] with a gate) bf16, Y [N] float32 or bf16.  K and ldw multiples of 8, 16-byte aligned
// bases.  gate: 0, TQ_ACT_SILU, TQ_ACT_GELU_TANH (gated), TQ_ACT_SQUARE_RELU (plain, on its result).
TQ_API int tq_row_gemm(const void* X, const void* W, const float* bias, void* Y, int y_dtype, int N, int K, int ldw,
                       int accumulate, int gate, int settled, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (K <= 0 || (K & 7) || (ldw & 7) || (reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) ||
        gate < 0 || gate > TQ_ACT_SQUARE_RELU || (y_dtype != TQ_F32 && y_dtype != TQ_BF16) ||
        (accumulate && (y_dtype != TQ_F32 || gate == TQ_ACT_SQUARE_RELU)))
        return (int)cudaErrorInvalidValue;
    const RowGemmArgs a{(const bf16*)X, (const bf16*)W, bias, Y, N, K, ldw, accumulate, gate, settled};
    const bool gated = gate == TQ_ACT_SILU || gate == TQ_ACT_GELU_TANH;
    if (y_dtype == TQ_F32) return gated ? launch_row_gemm<true, float>(a, stream) : launch_row_gemm<false, float>(a, stream);
    return gated ? launch_row_gemm<true, bf16>(a, stream) : launch_row_gemm<false, bf16>(a, stream);
}
