// Everything between the q|k|v product and the output product of a decode step's softmax attention, in one kernel: bias and
// rotary encoding of q and k, the new key and value into the cache, attention over the cached keys, the merge of the splits.
//
// A cluster of 1, 2, 4 or 8 blocks serves one (token, key/value head): the blocks split the cached keys, four warps a block
// as in flash_decode.cu (32-key chunks by cp.async, mma.sync, float32 online softmax), and meet through distributed
// shared memory in the order of the ranks, so results do not depend on timing.  The new key never makes the way through the
// cache: rank 0 turns it, writes it there for later steps and attends to it from shared memory.  Every key that is read from
// the cache is older than the step, so the first chunks are asked for before the product in front has ended.  A q|k|v buffer
// that a product adds its shares into is cleared here, by rank 0, once all blocks of the cluster have read it.
//
// What bounds it is latency: a step waits for the product, turns q, attends and meets.  The separate kernels (rotary, attention,
// merge) take 2.7 + 3.7 + 2.5 us a layer on the 0.5B shape with one sequence, this one 6.3, each without early starts; decode steps,
// us, separate / here: 1 sequence of 60 keys 609 / 546, of 4,000 621 / 610, of 8,000 638 / 683 (8 blocks are too few), 8 of 300
// 661 / 591, 8 of 4,000 731 / 688, 32 of 1,000 855 / 835, 64 of 300 914 / 886.  Heads of 128 (7B) gained nothing with one sequence
// (2,660 / 2,665) and lost with 8 (2,935 / 3,169): its blocks, let in while the product in front drains, crowd on the SMs that
// are free first.  So heads of up to 64 come here.
//
// Formulas: src/models/turbo_generic.rs:417-427 (rotation), :805-813 (bias), :1606-1631 (cache, attention).
#include <cooperative_groups.h>

#include "flash_decode.cuh"

#define RD_MAX_SPLITS 8

struct RopeDecodeArgs {
    float* qkv;                 // [T, (nh + 2 nkv) * hd]
    const float *bias, *cos_tab, *sin_tab;
    bf16 *k_pages, *v_pages;
    const int *block_table, *tok_pos, *tok_seq, *new_lens;
    bf16* out;                  // [T, nh * hd]
    int table_width, ring_pages, window, nh, nkv, rot, clear;
    float scale_log2;
};

template <int HD, int FD_CHUNK>
__global__ void __launch_bounds__(FD_WARPS * 32) rope_decode_kernel(const RopeDecodeArgs a) {
    namespace cg = cooperative_groups;
    constexpr int ROW = HD * 2 + 16;                       // bytes per key row in shared memory (padded)
    constexpr int TILE = FD_CHUNK * ROW;                   // one K or V chunk
    constexpr int WARP_BYTES = FD_STAGES * 2 * TILE;
    constexpr int KS = HD / 16, NT = HD / 8, PR = HD / 8, ST = FD_CHUNK / 8;
    constexpr int RS = HD + 2;                             // floats of a row of partial results: output, max, sum
    extern __shared__ __align__(16) unsigned char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int n_ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int t = blockIdx.z, g = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gid = lane >> 2, tid4 = lane & 3;
    const int n_rep = a.nh / a.nkv;
    unsigned char* q_sh = smem + FD_WARPS * WARP_BYTES;    // [16][ROW]
    bf16* new_kv = reinterpret_cast<bf16*>(q_sh + 16 * ROW);      // [2][HD]: the new key, the new value
    const int pos = a.tok_pos[t], b = a.tok_seq[t];
    // the cached keys lo_all .. pos - 1, counted from 0; [lo, hi): this block's
    const int lo_all = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int n_old = pos - lo_all;
    const int split_len = ((n_old + n_ranks - 1) / n_ranks + 15) & ~15;
    const int lo = min(n_old, rank * split_len), hi = min(n_old, lo + split_len);
    const int n_chunks = (hi - lo + FD_CHUNK - 1) / FD_CHUNK;
    unsigned char* my = smem + warp * WARP_BYTES;
    const int* table = a.block_table + (size_t)b * a.table_width;
    auto cache_row = [&](int j) {                          // offset of position j's row in the cache
        int lp = j / FD_PAGE;
        if (a.ring_pages > 0) lp %= a.ring_pages;
        return (((unsigned long long)table[lp] * a.nkv + g) * FD_PAGE + (j % FD_PAGE)) * HD;
    };
    // the copy of this warp's i-th chunk into stage i % FD_STAGES (see flash_decode.cu)
    auto issue = [&](int i) {
        const int chunk = warp + i * FD_WARPS;
        if (chunk < n_chunks) {
            const unsigned long long my_row = cache_row(lo_all + min(lo + chunk * FD_CHUNK + (lane & (FD_CHUNK - 1)), hi - 1));
            unsigned char* ks_ = my + (i % FD_STAGES) * 2 * TILE;
#pragma unroll
            for (int it = 0; it < FD_CHUNK * PR / 32; ++it) {
                const int p = lane + 32 * it, key = p / PR, c = p - key * PR;
                const unsigned long long row = __shfl_sync(0xffffffffu, my_row, key);
                fd_cp_async16(ks_ + key * ROW + c * 16, a.k_pages + row + c * 8);
                fd_cp_async16(ks_ + TILE + key * ROW + c * 16, a.v_pages + row + c * 8);
            }
        }
        fd_commit();
    };
#pragma unroll
    for (int i = 0; i < FD_STAGES - 1; ++i) issue(i);

    // ---- q (every block), the new key and value (rank 0) ----
    const int half = a.rot >> 1;
    const float *cs = a.cos_tab + (size_t)pos * half, *sn = a.sin_tab + (size_t)pos * half;
    const size_t width = (size_t)(a.nh + 2 * a.nkv) * HD;
    float* row = a.qkv + (size_t)t * width;
    const bool keep = rank == 0 && pos < a.new_lens[b];
    const unsigned long long new_row = keep ? cache_row(pos) : 0;
    // What a thread turns: pairs e = thread, thread + threads, ... of (head, pair), the q heads of the group and (rank 0) the key,
    // then the value's entries, PER at a time: what does not depend on the kernel in front is loaded before it ends, then all of
    // the row's entries at once (one after the other they took longer than the attention).
    constexpr int PER = 4;
    const int turned = (n_rep + (rank == 0 ? 1 : 0)) * (HD / 2), work = turned + (rank == 0 ? HD / 2 : 0);
    const float* bias = a.bias;
    bool waited = false;
    for (int e0 = threadIdx.x; e0 < work || !waited; e0 += PER * (FD_WARPS * 32)) {
        int at0[PER], at1[PER];                            // the two entries of the row
        float c[PER], s[PER], b0[PER], b1[PER], u0[PER], u1[PER];
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int e = e0 + p * (FD_WARPS * 32), r = e / (HD / 2), i = e - r * (HD / 2);
            const int head = r < n_rep ? g * n_rep + r : e < turned ? a.nh + g : a.nh + a.nkv + g;
            const bool turns = e < turned && i < half;
            const int d0 = e >= turned ? 2 * i : turns ? i : a.rot + 2 * (i - half);
            at0[p] = e < work ? head * HD + d0 : -1;
            at1[p] = at0[p] + (turns ? half : 1);
            c[p] = e < work && turns ? cs[i] : 1.f;
            s[p] = e < work && turns ? sn[i] : 0.f;
            b0[p] = e < work && bias ? bias[at0[p]] : 0.f;
            b1[p] = e < work && bias ? bias[at1[p]] : 0.f;
        }
        if (!waited) pdl_wait();
        waited = true;
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            u0[p] = at0[p] >= 0 ? row[at0[p]] : 0.f;
            u1[p] = at0[p] >= 0 ? row[at1[p]] : 0.f;
        }
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at0[p] < 0) continue;
            const int e = e0 + p * (FD_WARPS * 32), r = e / (HD / 2);
            const int d0 = at0[p] % HD, d1 = at1[p] % HD;
            const bool turns = e < turned && e - r * (HD / 2) < half;
            const float x0 = u0[p] + b0[p], x1 = u1[p] + b1[p];
            const bf16 y0 = __float2bfloat16_rn(turns ? fmaf(x0, c[p], -__fmul_rn(x1, s[p])) : x0), y1 = __float2bfloat16_rn(turns ? fmaf(x0, s[p], __fmul_rn(x1, c[p])) : x1);
            bf16* dst = r < n_rep ? reinterpret_cast<bf16*>(q_sh + r * ROW) : e < turned ? new_kv : new_kv + HD;
            dst[d0] = y0;
            dst[d1] = y1;
            if (keep && r >= n_rep) {
                bf16* page = (e < turned ? a.k_pages : a.v_pages) + new_row;
                page[d0] = y0;
                page[d1] = y1;
            }
        }
    }
    for (int e = threadIdx.x; e < (16 - n_rep) * PR; e += FD_WARPS * 32)      // rows of no head
        *reinterpret_cast<uint4*>(q_sh + (n_rep + e / PR) * ROW + (e % PR) * 16) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint32_t qf[KS][4];
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) fd_ldmatrix_x4(qf[ks], q_sh + (lane & 15) * ROW + (2 * ks + (lane >> 4)) * 16);

    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float o[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
    // one chunk: keys and values at ks_ and vs_, the first `live` of them count (at least one)
    auto attend = [&](const unsigned char* ks_, const unsigned char* vs_, int live) {
        float s[ST][4];
#pragma unroll
        for (int n = 0; n < ST; ++n) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f; }
        const int mat = lane >> 3, r8 = lane & 7;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int n = 0; n < ST; n += 2) {
                uint32_t kb[4];
                fd_ldmatrix_x4(kb, ks_ + ((n + (mat >> 1)) * 8 + r8) * ROW + (2 * ks + (mat & 1)) * 16);
                fd_mma(s[n], qf[ks], kb[0], kb[1]);
                fd_mma(s[n + 1], qf[ks], kb[2], kb[3]);
            }
        float corr[2], mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nt = 0; nt < ST; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float v = nt * 8 + 2 * tid4 + (e & 1) < live ? s[nt][e] * a.scale_log2 : -INFINITY;
                s[nt][e] = v;
                mx[e >> 1] = fmaxf(mx[e >> 1], v);
            }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            const float m_new = fmaxf(m_run[r], mx[r]);    // finite: the first key is always live
            corr[r] = exp2f(m_run[r] - m_new);
            m_run[r] = m_new;
        }
        float rs[2] = {0.f, 0.f};
#pragma unroll
        for (int nt = 0; nt < ST; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float p = exp2f(s[nt][e] - m_run[e >> 1]);
                s[nt][e] = p;
                rs[e >> 1] += p;
            }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            rs[r] += __shfl_xor_sync(0xffffffffu, rs[r], 1);
            rs[r] += __shfl_xor_sync(0xffffffffu, rs[r], 2);
            l_run[r] = l_run[r] * corr[r] + rs[r];
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            o[n][0] *= corr[0]; o[n][1] *= corr[0];
            o[n][2] *= corr[1]; o[n][3] *= corr[1];
        }
#pragma unroll
        for (int kk = 0; kk < FD_CHUNK / 16; ++kk) {
            uint32_t pf[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) pf[e] = fd_pack(s[2 * kk + (e >> 1)][2 * (e & 1)], s[2 * kk + (e >> 1)][2 * (e & 1) + 1]);
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t vb[4];
                fd_ldmatrix_x4_trans(vb, vs_ + (kk * 16 + (mat & 1) * 8 + r8) * ROW + (n + (mat >> 1)) * 16);
                fd_mma(o[n], pf, vb[0], vb[1]);
                fd_mma(o[n + 1], pf, vb[2], vb[3]);
            }
        }
    };
    const int my_chunks = n_chunks > warp ? (n_chunks - warp + FD_WARPS - 1) / FD_WARPS : 0;
    for (int i = 0; i < my_chunks; ++i) {
        issue(i + FD_STAGES - 1);
        fd_wait<FD_STAGES - 1>();                          // chunk i has landed
        __syncwarp();
        const unsigned char* ks_ = my + (i % FD_STAGES) * 2 * TILE;
        attend(ks_, ks_ + TILE, hi - (lo + (warp + i * FD_WARPS) * FD_CHUNK));
        __syncwarp();                                      // the stage may be overwritten by the next issue
    }
    fd_wait<0>();
    pdl_launch();                                          // the next kernel may ask for its weights while the blocks meet
    if (rank == 0 && warp == FD_WARPS - 1) {               // the new key: a chunk of its own, its other rows zero
        __syncwarp();
        for (int p = lane; p < 2 * FD_CHUNK * PR; p += 32) {
            const int which = p / (FD_CHUNK * PR), key = p / PR % FD_CHUNK, c = p % PR;
            *reinterpret_cast<uint4*>(my + which * TILE + key * ROW + c * 16) =
                key == 0 ? *reinterpret_cast<const uint4*>(new_kv + which * HD + c * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
        __syncwarp();
        attend(my, my + TILE, 1);
    }
    __syncthreads();

    // ---- the warps' results to shared memory: [warp][16 rows][HD + 2] (output, max, sum), then the block's: [n_rep][HD + 2] ----
    float* ms = reinterpret_cast<float*>(smem);
    float* part = ms + FD_WARPS * 16 * RS;
    float* mine = ms + (size_t)warp * 16 * RS;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int d = n * 8 + 2 * tid4;
        mine[gid * RS + d] = o[n][0];
        mine[gid * RS + d + 1] = o[n][1];
        mine[(gid + 8) * RS + d] = o[n][2];
        mine[(gid + 8) * RS + d + 1] = o[n][3];
    }
    if (tid4 == 0) {
        mine[gid * RS + HD] = m_run[0];
        mine[gid * RS + HD + 1] = l_run[0];
        mine[(gid + 8) * RS + HD] = m_run[1];
        mine[(gid + 8) * RS + HD + 1] = l_run[1];
    }
    __syncthreads();
    bf16* out = a.out + ((size_t)t * a.nh + (size_t)g * n_rep) * HD;
    for (int e = threadIdx.x; e < n_rep * HD; e += FD_WARPS * 32) {
        const int r = e / HD, d = e - r * HD;
        float m = -INFINITY, l = 0.f, v = 0.f;
#pragma unroll
        for (int w = 0; w < FD_WARPS; ++w) m = fmaxf(m, ms[(w * 16 + r) * RS + HD]);
#pragma unroll
        for (int w = 0; w < FD_WARPS; ++w) {
            const float* x = ms + (w * 16 + r) * RS;
            if (x[HD] > -INFINITY) {
                const float f = exp2f(x[HD] - m);
                l += x[HD + 1] * f;
                v += x[d] * f;
            }
        }
        if (n_ranks == 1) {
            out[e] = __float2bfloat16_rn(v / l);
        } else {
            part[r * RS + d] = v;
            if (d == 0) { part[r * RS + HD] = m; part[r * RS + HD + 1] = l; }
        }
    }
    if (n_ranks > 1) {
        cluster.sync();
        for (int e = rank * FD_WARPS * 32 + threadIdx.x; e < n_rep * HD; e += n_ranks * FD_WARPS * 32) {
            const int r = e / HD, d = e - r * HD;
            float pm[RD_MAX_SPLITS], pl[RD_MAX_SPLITS], pv[RD_MAX_SPLITS], m = -INFINITY, l = 0.f, v = 0.f;
#pragma unroll
            for (int p = 0; p < RD_MAX_SPLITS; ++p) {
                const float* x = p < n_ranks ? cluster.map_shared_rank(part, p) + r * RS : nullptr;
                pm[p] = x ? x[HD] : -INFINITY;
                pl[p] = x ? x[HD + 1] : 0.f;
                pv[p] = x ? x[d] : 0.f;
                m = fmaxf(m, pm[p]);
            }
#pragma unroll
            for (int p = 0; p < RD_MAX_SPLITS; ++p)
                if (pm[p] > -INFINITY) {
                    const float f = exp2f(pm[p] - m);
                    l += pl[p] * f;
                    v += pv[p] * f;
                }
            out[e] = __float2bfloat16_rn(v / l);
        }
    }
    if (a.clear && rank == 0) {                            // (all blocks of the cluster have read their q by now)
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int e = threadIdx.x; e < (n_rep + 2) * (HD / 4); e += FD_WARPS * 32) {
            const int r = e / (HD / 4), c = e - r * (HD / 4);
            const int head = r < n_rep ? g * n_rep + r : (r == n_rep ? a.nh + g : a.nh + a.nkv + g);
            *reinterpret_cast<float4*>(row + head * HD + c * 4) = zero;
        }
    }
    if (n_ranks > 1) cluster.sync();                       // nobody leaves while its results are being read
}

template <int HD>
static int launch_rope_decode(const RopeDecodeArgs& a, int n_tokens, int n_splits, cudaStream_t stream) {
    constexpr int ROW = HD * 2 + 16, FD_CHUNK = 32;
    constexpr size_t stages = (size_t)FD_WARPS * FD_STAGES * 2 * FD_CHUNK * ROW;
    constexpr size_t merge = (size_t)(FD_WARPS + 1) * 16 * (HD + 2) * sizeof(float);
    static_assert(stages >= merge, "the partial results reuse the stages");
    constexpr size_t smem = stages + 16 * ROW + 4 * HD;
    static bool configured[64] = {false};                  // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(rope_decode_kernel<HD, FD_CHUNK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_splits, a.nkv, n_tokens);
    cfg.blockDim = dim3(FD_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = tq_pdl_enabled(TQ_PDL_FLASH_DECODE) ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = n_splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, rope_decode_kernel<HD, FD_CHUNK>, a);
    if (e != cudaSuccess) return (int)e;
    return tq_launch_status();
}

// qkv [n_tokens, (nh + 2 nkv) * hd] float32 (16-byte aligned): every row is its sequence's only token of this step, and the
// kernels before this one in the stream that may still run write nothing that it reads but qkv.  Pages of 64 tokens; hd 32 or
// 64; at most 16 q heads a key/value head.  n_splits: 1, 2, 4 or 8 blocks for a token and head.  clear: qkv's rows are
// left zero.  Returns cudaErrorNotSupported (801) for shapes outside this kernel's reach.
TQ_API int tq_rope_decode(float* qkv, const float* bias, const float* cos_tab, const float* sin_tab, void* k_pages, void* v_pages,
                          const int* block_table, int table_width, int ring_pages, int page_tokens, const int* tok_pos,
                          const int* tok_seq, const int* new_lens, int window, float scale, void* out, int n_tokens, int nh,
                          int nkv, int hd, int rot, int n_splits, int clear, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (nkv <= 0 || nh % nkv || nh / nkv > 16 || page_tokens != FD_PAGE || nkv > 65535 || n_tokens > 65535 || rot < 2 || rot % 2 ||
        rot > hd || (reinterpret_cast<uintptr_t>(qkv) & 15))
        return (int)cudaErrorNotSupported;
    if (n_splits != 1 && n_splits != 2 && n_splits != 4 && n_splits != 8) return (int)cudaErrorInvalidValue;
    if (!k_pages || !v_pages || !block_table) return (int)cudaErrorInvalidValue;
    const RopeDecodeArgs a{qkv, bias, cos_tab, sin_tab, (bf16*)k_pages, (bf16*)v_pages, block_table, tok_pos, tok_seq, new_lens,
                           (bf16*)out, table_width, ring_pages, window, nh, nkv, rot, clear, scale * 1.4426950408889634f};
    switch (hd) {
        case 32: return launch_rope_decode<32>(a, n_tokens, n_splits, stream);
        case 64: return launch_rope_decode<64>(a, n_tokens, n_splits, stream);
        default: return (int)cudaErrorNotSupported;
    }
}

// ---- float32 ------------------------------------------------------------------------------------------------------
// The same in float32 throughout (multiply-adds; weights of the softmax included): pieces of 32 keys and values in shared
// memory, two stages, fetched by the whole block; a warp serves the q heads w, w + 8 of the group: a lane a key for the scores,
// a lane HD / 32 dims for the values.  The separate kernels (rotary, general attention, merge) took 3.2 + 13.9 + 2.5 us a layer for
// two sequences of 160 keys, 14 heads on 2 of 64; 6.4 here.
#define RF_KEYS 32
#define RF_THREADS 256

struct RopeDecodeF32Args {
    const float *qkv, *bias, *cos_tab, *sin_tab;
    float *k_pages, *v_pages;
    const int *block_table, *tok_pos, *tok_seq, *new_lens;
    float* out;
    int table_width, ring_pages, window, nh, nkv, rot;
    float scale;
};

template <int HD, int HPW>
__global__ void __launch_bounds__(RF_THREADS) rope_decode_f32_kernel(const RopeDecodeF32Args a) {
    namespace cg = cooperative_groups;
    constexpr int LD = HD + 4, TILE = RF_KEYS * LD, DV = HD / 32, RS = HD + 2;
    extern __shared__ __align__(16) float fsh[];
    float *stages = fsh, *qs = stages + 4 * TILE, *part = qs + 8 * HPW * LD;       // stages: [2][keys, values]
    cg::cluster_group cluster = cg::this_cluster();
    const int n_ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int t = blockIdx.z, g = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_rep = a.nh / a.nkv;
    const int pos = a.tok_pos[t], b = a.tok_seq[t];
    const int lo_all = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int n_old = pos - lo_all, split_len = (n_old + n_ranks - 1) / n_ranks;
    const int lo = min(n_old, rank * split_len), hi = min(n_old, lo + split_len);
    const int n_tiles = (hi - lo + RF_KEYS - 1) / RF_KEYS;
    const int* table = a.block_table + (size_t)b * a.table_width;
    auto cache_row = [&](int j) {
        int lp = j / FD_PAGE;
        if (a.ring_pages > 0) lp %= a.ring_pages;
        return (((unsigned long long)table[lp] * a.nkv + g) * FD_PAGE + (j % FD_PAGE)) * HD;
    };
    auto issue = [&](int i) {
        if (i < n_tiles) {
            float* dst = stages + (i & 1) * 2 * TILE;
            for (int e = threadIdx.x; e < RF_KEYS * (HD / 4); e += RF_THREADS) {
                const int key = e / (HD / 4), c = e % (HD / 4) * 4;
                const unsigned long long row = cache_row(lo_all + min(lo + i * RF_KEYS + key, hi - 1)) + c;
                fd_cp_async16(dst + key * LD + c, a.k_pages + row);
                fd_cp_async16(dst + TILE + key * LD + c, a.v_pages + row);
            }
        }
        fd_commit();
    };
    issue(0);
    const int half = a.rot >> 1;
    const float *cs = a.cos_tab + (size_t)pos * half, *sn = a.sin_tab + (size_t)pos * half;
    const float* row = a.qkv + (size_t)t * (a.nh + 2 * a.nkv) * HD;
    const bool keep = rank == 0 && pos < a.new_lens[b];
    const unsigned long long new_row = keep ? cache_row(pos) : 0;
    float* hold = part + 16 * RS;                          // rank 0: the new key, the new value
    // What a thread turns: pairs e = thread, thread + threads, ... of (head, pair), the q heads of the group and (rank 0) the key,
    // then the value's entries, PER at a time: what does not depend on the kernel in front is loaded before it ends, then all of
    // the row's entries at once (one after the other they took longer than the attention).
    constexpr int PER = 4;
    const int turned = (n_rep + (rank == 0 ? 1 : 0)) * (HD / 2), work = turned + (rank == 0 ? HD / 2 : 0);
    const float* bias = a.bias;
    bool waited = false;
    for (int e0 = threadIdx.x; e0 < work || !waited; e0 += PER * RF_THREADS) {
        int at0[PER], at1[PER];                            // the two entries of the row
        float c[PER], s[PER], b0[PER], b1[PER], u0[PER], u1[PER];
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int e = e0 + p * RF_THREADS, r = e / (HD / 2), i = e - r * (HD / 2);
            const int head = r < n_rep ? g * n_rep + r : e < turned ? a.nh + g : a.nh + a.nkv + g;
            const bool turns = e < turned && i < half;
            const int d0 = e >= turned ? 2 * i : turns ? i : a.rot + 2 * (i - half);
            at0[p] = e < work ? head * HD + d0 : -1;
            at1[p] = at0[p] + (turns ? half : 1);
            c[p] = e < work && turns ? cs[i] : 1.f;
            s[p] = e < work && turns ? sn[i] : 0.f;
            b0[p] = e < work && bias ? bias[at0[p]] : 0.f;
            b1[p] = e < work && bias ? bias[at1[p]] : 0.f;
        }
        if (!waited) pdl_wait();
        waited = true;
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            u0[p] = at0[p] >= 0 ? row[at0[p]] : 0.f;
            u1[p] = at0[p] >= 0 ? row[at1[p]] : 0.f;
        }
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at0[p] < 0) continue;
            const int e = e0 + p * RF_THREADS, r = e / (HD / 2);
            const int d0 = at0[p] % HD, d1 = at1[p] % HD;
            const bool turns = e < turned && e - r * (HD / 2) < half;
            const float x0 = u0[p] + b0[p], x1 = u1[p] + b1[p];
            const float y0 = (turns ? fmaf(x0, c[p], -__fmul_rn(x1, s[p])) : x0), y1 = (turns ? fmaf(x0, s[p], __fmul_rn(x1, c[p])) : x1);
            float* dst = r < n_rep ? qs + r * LD : e < turned ? hold : hold + HD;
            dst[d0] = y0;
            dst[d1] = y1;
            if (keep && r >= n_rep) {
                float* page = (e < turned ? a.k_pages : a.v_pages) + new_row;
                page[d0] = y0;
                page[d1] = y1;
            }
        }
    }
    float m[HPW], l[HPW], acc[HPW][DV];
#pragma unroll
    for (int h = 0; h < HPW; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int c = 0; c < DV; ++c) acc[h][c] = 0.f;
    }
    // keys and values at kt and vt (rows LD apart), the first `live` of them count (at least one)
    auto attend = [&](const float* kt, const float* vt, int live) {
#pragma unroll
        for (int h = 0; h < HPW; ++h) {
            const int r = warp + 8 * h;
            if (r >= n_rep) continue;
            float s = -INFINITY;
            if (lane < live) {
                float dot = 0.f;
#pragma unroll 8
                for (int d = 0; d < HD; d += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(qs + r * LD + d);
                    const float4 k = *reinterpret_cast<const float4*>(kt + lane * LD + d);
                    dot = fmaf(x.x, k.x, dot); dot = fmaf(x.y, k.y, dot);
                    dot = fmaf(x.z, k.z, dot); dot = fmaf(x.w, k.w, dot);
                }
                s = dot * a.scale;
            }
            const float m_new = fmaxf(m[h], warp_max(s));
            const float p = lane < live ? expf(s - m_new) : 0.f, corr = expf(m[h] - m_new);
            l[h] = l[h] * corr + warp_sum(p);
            m[h] = m_new;
#pragma unroll
            for (int c = 0; c < DV; ++c) acc[h][c] *= corr;
#pragma unroll 4
            for (int j = 0; j < live; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
                for (int c = 0; c < DV; ++c) acc[h][c] = fmaf(pj, vt[j * LD + lane + 32 * c], acc[h][c]);
            }
        }
    };
    for (int i = 0; i < n_tiles; ++i) {
        issue(i + 1);
        fd_wait<1>();
        __syncthreads();                                   // the piece (and at first q) is there for all
        const float* kt = stages + (i & 1) * 2 * TILE;
        attend(kt, kt + TILE, min(RF_KEYS, hi - lo - i * RF_KEYS));
        __syncthreads();                                   // the stage may be filled again
    }
    fd_wait<0>();
    pdl_launch();
    __syncthreads();
    if (rank == 0) attend(hold, hold + HD, 1);
#pragma unroll
    for (int h = 0; h < HPW; ++h) {
        const int r = warp + 8 * h;
        if (r >= n_rep) continue;
#pragma unroll
        for (int c = 0; c < DV; ++c) part[r * RS + lane + 32 * c] = acc[h][c];
        if (lane == 0) { part[r * RS + HD] = m[h]; part[r * RS + HD + 1] = l[h]; }
    }
    if (n_ranks > 1) cluster.sync();
    else __syncthreads();
    float* out = a.out + ((size_t)t * a.nh + (size_t)g * n_rep) * HD;
    for (int e = rank * RF_THREADS + threadIdx.x; e < n_rep * HD; e += n_ranks * RF_THREADS) {
        const int r = e / HD, d = e - r * HD;
        float pm[RD_MAX_SPLITS], pl[RD_MAX_SPLITS], pv[RD_MAX_SPLITS], top = -INFINITY, sum = 0.f, v = 0.f;
#pragma unroll
        for (int p = 0; p < RD_MAX_SPLITS; ++p) {
            const float* x = p < n_ranks ? (n_ranks > 1 ? cluster.map_shared_rank(part, p) : part) + r * RS : nullptr;
            pm[p] = x ? x[HD] : -INFINITY;
            pl[p] = x ? x[HD + 1] : 0.f;
            pv[p] = x ? x[d] : 0.f;
            top = fmaxf(top, pm[p]);
        }
#pragma unroll
        for (int p = 0; p < RD_MAX_SPLITS; ++p)
            if (pm[p] > -INFINITY) {
                const float f = expf(pm[p] - top);
                sum += pl[p] * f;
                v += pv[p] * f;
            }
        out[e] = v / sum;
    }
    if (n_ranks > 1) cluster.sync();                       // nobody leaves while its results are being read
}

template <int HD, int HPW>
static int launch_rope_decode_f32(const RopeDecodeF32Args& a, int n_tokens, int n_splits, cudaStream_t stream) {
    constexpr size_t smem = (4 * RF_KEYS * (HD + 4) + 8 * HPW * (HD + 4) + 16 * (HD + 2) + 2 * HD) * sizeof(float);
    static bool configured[64] = {false};                  // per device: the attribute belongs to its copy of the kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(rope_decode_f32_kernel<HD, HPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_splits, a.nkv, n_tokens);
    cfg.blockDim = dim3(RF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = tq_pdl_enabled(TQ_PDL_FLASH_DECODE) ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = n_splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, rope_decode_f32_kernel<HD, HPW>, a);
    if (e != cudaSuccess) return (int)e;
    return tq_launch_status();
}

// As tq_rope_decode with float32 pages and result; the rows of qkv stay as they are.
TQ_API int tq_rope_decode_f32(const float* qkv, const float* bias, const float* cos_tab, const float* sin_tab, float* k_pages,
                              float* v_pages, const int* block_table, int table_width, int ring_pages, int page_tokens,
                              const int* tok_pos, const int* tok_seq, const int* new_lens, int window, float scale, float* out,
                              int n_tokens, int nh, int nkv, int hd, int rot, int n_splits, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (nkv <= 0 || nh % nkv || nh / nkv > 16 || page_tokens != FD_PAGE || nkv > 65535 || n_tokens > 65535 || rot < 2 || rot % 2 ||
        rot > hd || ((reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages)) & 15))
        return (int)cudaErrorNotSupported;
    if (n_splits != 1 && n_splits != 2 && n_splits != 4 && n_splits != 8) return (int)cudaErrorInvalidValue;
    if (!k_pages || !v_pages || !block_table) return (int)cudaErrorInvalidValue;
    const RopeDecodeF32Args a{qkv, bias, cos_tab, sin_tab, k_pages, v_pages, block_table, tok_pos, tok_seq, new_lens, out,
                              table_width, ring_pages, window, nh, nkv, rot, scale};
#define TQ_RF(H) case H: return nh / nkv <= 8 ? launch_rope_decode_f32<H, 1>(a, n_tokens, n_splits, stream) : launch_rope_decode_f32<H, 2>(a, n_tokens, n_splits, stream)
    switch (hd) {
        TQ_RF(32);
        TQ_RF(64);
        default: return (int)cudaErrorNotSupported;
    }
#undef TQ_RF
}
