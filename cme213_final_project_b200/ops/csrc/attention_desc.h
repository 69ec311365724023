// The attention descriptor as plain C++, for the kernels' side (attention.h) and the compiled wrappers.  See attention.h.
#pragma once

struct CmeAttn {
    int nb, nh, T, HD;
    long long sb, sh, st;        // strides of Q / K / V / dQ / dK / dV
    long long osb, osh, ost;     // strides of O / dO
    int causal;
    float scale;                 // 1 / sqrt(HD)
    int dtype;                   // CME_BF16 or CME_F32
    const void* q; const void* k; const void* v;
    void* o;                     // forward output / backward input
    float* lse;                  // [nb*nh, T] log-sum-exp of scaled scores (saved by forward)
    // backward only
    const void* d_o; void* dq; void* dk; void* dv;
    float* delta;                // [nb*nh, T] scratch: rowsum(dO * O)
    float* dq_accum;             // fp32 scratch [nb*nh*T*HD] for the tcgen05 backward (may be null)
    void* ws; long long ws_bytes;    // scratch of attention_gemm_ws_bytes() for the batched-GEMM path (may be null)
    int* dq_sem;                 // [nb*nh * ceil(T / 128)] ints, zero before the first launch (the kernel leaves them zero);
                                 // needed by dq_mode 1 and 2
    int dq_mode;                 // how the tcgen05 backward completes dQ from the key blocks' parts:
                                 //   0  the launch clears dq_accum, the parts are added in arrival order, a second kernel
                                 //      scales and casts the sums
                                 //   1  the parts are added in a fixed order (bit-reproducible); key block 0 finishes
                                 //   2  arrival order; the CTA whose part comes last scales, casts and writes zeros back:
                                 //      dq_accum must be zero before the first launch and is zero after every launch
    int dq_accum_clean;          // dq_mode 0: non-zero = the caller has cleared dq_accum itself (e.g. on another stream,
                                 // ahead of time); the launch then skips its own clear
};

constexpr int CME_ATTN_FINISH_MAX_QBLOCKS = 64;      // dq_mode 2: query blocks (of 128 rows) per sequence

// The kernels that a call takes.
enum CmeAttnPath : int {
    CME_ATTN_PATH_SHORT = 0,     // one launch per direction, up to 64 tokens
    CME_ATTN_PATH_TC = 1,        // flash kernel on tcgen05; the backward adds up dQ in dq_accum
    CME_ATTN_PATH_GEMM = 2,      // batched products around row kernels, with `ws`
    CME_ATTN_PATH_SIMT = 3,
};
