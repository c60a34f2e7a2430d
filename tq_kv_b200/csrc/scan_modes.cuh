// The rules and the arguments that linear_scan.cu (where they are described) and block_scan.cu share.
#pragma once
#include "common.cuh"

#define SCAN_DECAY 0
#define SCAN_DELTA 1
#define SCAN_GATED 2
#define SCAN_GATED_DELTA 3
#define SCAN_CHANNEL_DELTA 4

struct ScanArgs {
    const float* q;           // [T, ldp] query vectors, head h at columns h*d (the pointers are already offset)
    const float* k;           // keys, same layout
    const float* v;           // values, head h at columns h*e
    const float* au;          // SCAN_DELTA: minus removal rate times unit key (after scan_prepare)
    int ldp;                  // row stride of q, k, v, au (one projection buffer)
    const float* u;           // SCAN_DELTA: unit keys [T, ldu]
    int ldu;
    const float* w;           // SCAN_DELTA (after scan_prepare), SCAN_CHANNEL_DELTA: decay per key channel [T, ldw]
    int ldw;
    const float* head_decay;  // SCAN_DECAY: [H]
    float* state;             // [slots, H, d, e]
    const int* cu_seqlens;    // [B + 1] first token of each sequence in this step
    const int* slots;         // [B]
    float* out;               // [T, ldo], head h at columns h*e
    int ldo;
    int H, d, e;
    int chunk;                // tokens staged at a time
    int vec;                  // every vector starts on a 16-byte boundary and d, e are multiples of four
    int silu;                 // linear_step, SCAN_DECAY: q, k, v pass through silu (nothing was prepared)
    float unit_eps;           // linear_step, SCAN_DELTA: au and w hold the logits still (nothing was prepared)
    const float* scal;        // SCAN_GATED*: [T, H, 4] per token and head: decay, then step size or write strength
    const float* skip;        // SCAN_GATED: [H] or null, o += skip_head * v
    int qk_div;               // head h reads the q/k vectors of head h / qk_div
    size_t state_stride;      // floats from one slot's states to the next
};

// block_scan.cu: steps of many tokens of few sequences, eight tokens at a time.  `rec` is scratch of block_scan_floats(...)
// floats (0: linear_scan.cu's kernel is the faster one); au and w hold the logits still, q, k, v what silu has not seen.
long long block_scan_floats(int mode, int n_tokens, int n_seqs, int H, int d, int e);
int block_scan(int mode, const ScanArgs& a, int n_seqs, int n_tokens, float* rec, cudaStream_t stream);
