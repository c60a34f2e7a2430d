// Float32 attention of prompts: softmax(q k / sqrt(d)) v for steps in which some sequence brings several tokens, float32
// throughout (multiply-adds; the formulas are attention.cu's: src/models/turbo_generic.rs:1620-1631).
//
// A block takes up to 64 rows (32 where that leaves SMs without a block), a row being a (token, q head) pair of one key/value head, and walks their keys 32 at a time:
// keys and values of a piece lie in shared memory and serve all rows, where the general kernel reads them once per row with
// 32 lanes on 32 rows of the cache (its loads touch a line a lane, which bounds it).  16 x 16 threads: a thread makes 4 rows x 2
// keys of the scores (2 x 2) and 4 rows (2) x HD / 16 dims of the result; the 16 threads of a row trade maxima and sums by shuffles, so the
// weights need no barrier.  Tokens of a block that belong to several sequences are walked sequence by sequence.
// Bound by latency at the sizes it meets (a hundred blocks, a handful of pieces each).  Measured, two prompts of 150 tokens, 14
// heads on 2 of 64: general kernel 71 us a layer, with 64 rows a block 34, with 32 25.
#include "common.cuh"

#define PA_MOST_ROWS 64
#define PA_KEYS 32
#define PA_THREADS 256

struct PromptF32Args {
    const float *q, *k_packed, *v_packed, *k_pages, *v_pages;
    const int *block_table, *tok_pos, *tok_seq, *cu_seqlens, *start_pos;
    float* out;
    int table_width, ring_pages, page_tokens, window, n_tokens, nh, nkv, tile;      // tile: tokens of a block
    float scale;
};

template <int HD, int PA_ROWS>
__global__ void __launch_bounds__(PA_THREADS) prompt_attention_f32_kernel(const PromptF32Args a) {
    constexpr int LD = HD + 4, DV = HD / 16, RT = PA_ROWS / 16;               // floats between rows in shared memory; a thread's dims and rows
    extern __shared__ __align__(16) float sh[];
    float *qs = sh, *ks = qs + PA_ROWS * LD, *vs = ks + PA_KEYS * LD, *ps = vs + PA_KEYS * LD;      // ps: [64][33]
    __shared__ int seq_of[PA_ROWS], pos_of[PA_ROWS];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int g = blockIdx.y, t0 = blockIdx.x * a.tile, n_here = min(a.tile, a.n_tokens - t0);
    const int n_rep = a.nh / a.nkv, rows = n_here * n_rep;
    if (tid < PA_ROWS) {
        const int t = t0 + tid / n_rep;
        seq_of[tid] = tid < rows ? a.tok_seq[t] : -1;
        pos_of[tid] = tid < rows ? a.tok_pos[t] : 0;
    }
    for (int e = tid; e < PA_ROWS * (HD / 4); e += PA_THREADS) {
        const int r = e / (HD / 4), c = e % (HD / 4) * 4;
        const size_t from = ((size_t)(t0 + r / n_rep) * a.nh + g * n_rep + r % n_rep) * HD + c;
        *reinterpret_cast<float4*>(qs + r * LD + c) =
            r < rows ? *reinterpret_cast<const float4*>(a.q + from) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    float m[RT], l[RT], o[RT][DV];
    int seq[RT], pos[RT], low[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = ty * RT + i;
        seq[i] = seq_of[r];
        pos[i] = pos_of[r];
        low[i] = a.window > 0 && pos[i] - a.window + 1 > 0 ? pos[i] - a.window + 1 : 0;
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < DV; ++j) o[i][j] = 0.f;
    }
    for (int first = 0; first < n_here;) {                 // one sequence's tokens: first .. last
        const int b = seq_of[first * n_rep];
        int last = first;
        while (last + 1 < n_here && seq_of[(last + 1) * n_rep] == b) ++last;
        // the keys that any of them sees (positions grow along a sequence's tokens)
        const int p_lo = pos_of[first * n_rep], p_hi = pos_of[last * n_rep];
        const int lo = a.window > 0 && p_lo - a.window + 1 > 0 ? p_lo - a.window + 1 : 0;
        const int tok0 = a.k_packed ? a.cu_seqlens[b] - a.start_pos[b] : 0;
        for (int base = lo; base <= p_hi; base += PA_KEYS) {
            __syncthreads();                               // the piece before is used up
            bool odd = false;                              // a value that is no number or infinite: times 0 it would not vanish
            for (int e = tid; e < PA_KEYS * (HD / 4); e += PA_THREADS) {
                const int r = e / (HD / 4), c = e % (HD / 4) * 4, j = min(base + r, p_hi);
                size_t row;
                if (a.k_packed) {
                    row = (size_t)(tok0 + j) * a.nkv + g;
                } else {
                    int lp = j / a.page_tokens;
                    if (a.ring_pages > 0) lp %= a.ring_pages;
                    row = ((size_t)a.block_table[(size_t)b * a.table_width + lp] * a.nkv + g) * a.page_tokens + j % a.page_tokens;
                }
                *reinterpret_cast<float4*>(ks + r * LD + c) =
                    *reinterpret_cast<const float4*>((a.k_packed ? a.k_packed : a.k_pages) + row * HD + c);
                const float4 v = *reinterpret_cast<const float4*>((a.k_packed ? a.v_packed : a.v_pages) + row * HD + c);
                *reinterpret_cast<float4*>(vs + r * LD + c) = v;
                odd = odd || !(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))) < INFINITY) ||
                      isnan(v.x + v.y + v.z + v.w);
            }
            odd = __syncthreads_or(odd);
            float s[RT][2];
#pragma unroll
            for (int i = 0; i < RT; ++i) s[i][0] = s[i][1] = 0.f;
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                const float4 k0 = *reinterpret_cast<const float4*>(ks + tx * LD + d);
                const float4 k1 = *reinterpret_cast<const float4*>(ks + (tx + 16) * LD + d);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const float4 x = *reinterpret_cast<const float4*>(qs + (ty * RT + i) * LD + d);
                    s[i][0] = fmaf(x.x, k0.x, s[i][0]); s[i][0] = fmaf(x.y, k0.y, s[i][0]);
                    s[i][0] = fmaf(x.z, k0.z, s[i][0]); s[i][0] = fmaf(x.w, k0.w, s[i][0]);
                    s[i][1] = fmaf(x.x, k1.x, s[i][1]); s[i][1] = fmaf(x.y, k1.y, s[i][1]);
                    s[i][1] = fmaf(x.z, k1.z, s[i][1]); s[i][1] = fmaf(x.w, k1.w, s[i][1]);
                }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                float mx = -INFINITY;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int j = base + tx + 16 * u;
                    s[i][u] = seq[i] == b && j >= low[i] && j <= pos[i] ? s[i][u] * a.scale : -INFINITY;
                    mx = fmaxf(mx, s[i][u]);
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
                const float m_new = fmaxf(m[i], mx);
                const bool any = m_new > -INFINITY;        // (none yet: a row of another sequence, or before its window)
                const float corr = any ? expf(m[i] - m_new) : 1.f;
                float sum = 0.f;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float p = any ? expf(s[i][u] - m_new) : 0.f;
                    ps[(ty * RT + i) * (PA_KEYS + 1) + tx + 16 * u] = p;
                    sum += p;
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
                l[i] = l[i] * corr + sum;
                m[i] = m_new;
#pragma unroll
                for (int j = 0; j < DV; ++j) o[i][j] *= corr;
            }
            __syncwarp();                                  // a row's weights are written and read by one warp
            if (odd) {                                     // a row takes the keys that it sees and no others
                for (int j = 0; j < PA_KEYS; ++j)
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        if (seq[i] != b || base + j < low[i] || base + j > pos[i]) continue;
                        const float p = ps[(ty * RT + i) * (PA_KEYS + 1) + j];
#pragma unroll
                        for (int c = 0; c < DV; ++c) o[i][c] = fmaf(p, vs[j * LD + tx + 16 * c], o[i][c]);
                    }
                __syncwarp();
                continue;
            }
#pragma unroll 4
            for (int j = 0; j < PA_KEYS; ++j) {
                float p[RT];
#pragma unroll
                for (int i = 0; i < RT; ++i) p[i] = ps[(ty * RT + i) * (PA_KEYS + 1) + j];
#pragma unroll
                for (int c = 0; c < DV; ++c) {
                    const float v = vs[j * LD + tx + 16 * c];
#pragma unroll
                    for (int i = 0; i < RT; ++i) o[i][c] = fmaf(p[i], v, o[i][c]);
                }
            }
            __syncwarp();
        }
        first = last + 1;
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = ty * RT + i;
        if (r >= rows) continue;
        float* y = a.out + ((size_t)(t0 + r / n_rep) * a.nh + g * n_rep + r % n_rep) * HD;
        const float inv = 1.f / l[i];
#pragma unroll
        for (int c = 0; c < DV; ++c) y[tx + 16 * c] = o[i][c] * inv;
    }
}

template <int HD, int PA_ROWS>
static int launch_prompt_f32_rows(PromptF32Args a, cudaStream_t stream) {
    a.tile = PA_ROWS / (a.nh / a.nkv);
    constexpr size_t smem = ((PA_ROWS + 2 * PA_KEYS) * (HD + 4) + PA_ROWS * (PA_KEYS + 1)) * sizeof(float);
    static bool configured[64] = {false};                  // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(prompt_attention_f32_kernel<HD, PA_ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const dim3 grid((a.n_tokens + a.tile - 1) / a.tile, a.nkv);
    prompt_attention_f32_kernel<HD, PA_ROWS><<<grid, PA_THREADS, smem, stream>>>(a);
    return tq_launch_status();
}

template <int HD>
static int launch_prompt_f32(const PromptF32Args& a, cudaStream_t stream) {
    const int n_rep = a.nh / a.nkv;
    const long long blocks = (long long)(a.n_tokens + PA_MOST_ROWS / n_rep - 1) / (PA_MOST_ROWS / n_rep) * a.nkv;
    if (n_rep <= 32 && blocks < tq_sm_count()) return launch_prompt_f32_rows<HD, 32>(a, stream);
    return launch_prompt_f32_rows<HD, 64>(a, stream);
}

// As tq_attention (attention.cu) with one split, float32, heads of 32, 64, 96 or 128; the tokens of a sequence stand one behind
// the other, their positions growing by one.  Bases 16-byte aligned.  Returns cudaErrorNotSupported (801) for other shapes.
TQ_API int tq_prompt_attention_f32(const float* q, const float* k_packed, const float* v_packed, const float* k_pages,
                                   const float* v_pages, const int* block_table, int table_width, int ring_pages, int page_tokens,
                                   const int* tok_pos, const int* tok_seq, const int* cu_seqlens, const int* start_pos, int window,
                                   float scale, float* out, int n_tokens, int nh, int nkv, int hd, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (nkv <= 0 || nh % nkv || nh / nkv > PA_MOST_ROWS || nkv > 65535) return (int)cudaErrorNotSupported;
    const uintptr_t all = (uintptr_t)q | (uintptr_t)k_packed | (uintptr_t)v_packed | (uintptr_t)k_pages | (uintptr_t)v_pages;
    if (all & 15) return (int)cudaErrorNotSupported;
    if (k_packed ? !v_packed : (!k_pages || !v_pages || !block_table || page_tokens <= 0)) return (int)cudaErrorInvalidValue;
    const PromptF32Args a{q, k_packed, v_packed, k_pages, v_pages, block_table, tok_pos, tok_seq, cu_seqlens, start_pos, out,
                          table_width, ring_pages, page_tokens, window, n_tokens, nh, nkv, 0, scale};
    switch (hd) {
        case 32: return launch_prompt_f32<32>(a, stream);
        case 64: return launch_prompt_f32<64>(a, stream);
        case 96: return launch_prompt_f32<96>(a, stream);
        case 128: return launch_prompt_f32<128>(a, stream);
        default: return (int)cudaErrorNotSupported;
    }
}
