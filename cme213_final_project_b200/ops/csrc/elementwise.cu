// Element-wise, bias / activation, column-sum, cast, scale and embedding kernels (bf16 or fp32 I/O).
//
// Counterparts in the reference: FINAL_CLEAN_CODE_/src/kernels/activations.cu:5-357 (ReLU fwd/bwd,
// residual add, bias + residual add, bias add, bias + ReLU, bias backward, fused ReLU-backward +
// bias-backward, scale, float<->half casts) and FINAL_CLEAN_CODE_/src/kernels/embedding.cu:4-79
// (token gather, scatter-add backward, positional add and its backward).  Differences by design:
// token gather and positional add are one kernel; column sums (bias gradients) are reduced in two
// deterministic stages instead of atomicAdd; everything moves 128 bits per thread where alignment allows.
#include "common.h"

namespace {

template <typename T> struct Vw;
template <> struct Vw<float> { static constexpr int N = 4; };
template <> struct Vw<__nv_bfloat16> { static constexpr int N = 8; };

template <typename T> __device__ __forceinline__ void ldv(const T* p, float* f);
template <> __device__ __forceinline__ void ldv<float>(const float* p, float* f) {
    float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void ldv<__nv_bfloat16>(const __nv_bfloat16* p, float* f) {
    unpack8(*reinterpret_cast<const Bf16x8*>(p), f);
}
template <typename T> __device__ __forceinline__ void unpack_words(const uint4& r, float* f);
template <> __device__ __forceinline__ void unpack_words<float>(const uint4& r, float* f) {
    f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w);
}
template <> __device__ __forceinline__ void unpack_words<__nv_bfloat16>(const uint4& r, float* f) { unpack8(r, f); }
template <typename T> __device__ __forceinline__ void stv(T* p, const float* f);
template <> __device__ __forceinline__ void stv<float>(float* p, const float* f) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
template <> __device__ __forceinline__ void stv<__nv_bfloat16>(__nv_bfloat16* p, const float* f) {
    *reinterpret_cast<Bf16x8*>(p) = pack8(f);
}

__device__ __forceinline__ float act_f(float v, int act) {
    return act == 1 ? fmaxf(v, 0.f) : act == 2 ? gelu_f(v) : v;
}
__device__ __forceinline__ float dact_f(float pre, int act) {
    return act == 1 ? (pre > 0.f ? 1.f : 0.f) : act == 2 ? dgelu_f(pre) : 1.f;
}

// out[m, n] = act(x[m, n] + bias[n]) + residual[m, n]; any of bias / residual / pre_out may be null.
// One thread per vector of the row-major [rows, cols] matrix; cols is a multiple of the vector width.
// The column comes from a 32-bit remainder (Index = unsigned) whenever the vectors can be counted in 31 bits.
template <typename T, typename Index>
__global__ void __launch_bounds__(256)
bias_act_res_kernel(const T* __restrict__ x, const T* __restrict__ bias, const T* __restrict__ res, T* __restrict__ pre_out,
                    T* __restrict__ out, Index nvec, int cols, int act) {
    constexpr int W = Vw<T>::N;
    const Index cvec = cols / W, step = (Index)gridDim.x * blockDim.x;
    for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += step) {
        const long long e = (long long)i * W;
        const int c = (int)(i % cvec) * W;
        float v[W];
        ldv<T>(x + e, v);
        if (bias) {
            float b[W];
            ldv<T>(bias + c, b);
#pragma unroll
            for (int j = 0; j < W; ++j) v[j] += b[j];
        }
        if (pre_out) stv<T>(pre_out + e, v);
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = act_f(v[j], act);
        if (res) {
            float r[W];
            ldv<T>(res + e, r);
#pragma unroll
            for (int j = 0; j < W; ++j) v[j] += r[j];
        }
        stv<T>(out + e, v);
    }
}
template <typename T>
__global__ void bias_act_res_scalar_kernel(const T* x, const T* bias, const T* res, T* pre_out, T* out, long long n,
                                           int cols, int act) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        float v = to_f32<T>(x[i]);
        if (bias) v += to_f32<T>(bias[i % cols]);
        if (pre_out) pre_out[i] = from_f32<T>(v);
        v = act_f(v, act);
        if (res) v += to_f32<T>(res[i]);
        out[i] = from_f32<T>(v);
    }
}

// g[m, n] = dout[m, n] * act'(pre[m, n])  (written if g != null)  and partial column sums of g.
// Block = 32 row-lanes x 8 column-lanes; each thread owns one vector of columns.
// grid = (ceil(cols / (8*W)), row_splits); partial is [row_splits][cols].
template <typename T>
__global__ void __launch_bounds__(256)
dact_colsum_kernel(const T* __restrict__ dout, const T* __restrict__ pre, T* __restrict__ g, float* __restrict__ partial,
                   int rows, int cols, int act) {
    constexpr int W = Vw<T>::N;
    __shared__ float sm[32][8 * W + 1];
    pdl_wait();
    const int cl = threadIdx.x & 7, rl = threadIdx.x >> 3;
    const int c0 = (blockIdx.x * 8 + cl) * W;
    float s[W];
#pragma unroll
    for (int j = 0; j < W; ++j) s[j] = 0.f;
    const int rows_per = cme_cdiv_dev(rows, (int)gridDim.y);
    const int r0 = blockIdx.y * rows_per, r1 = min(rows, r0 + rows_per);
    if (c0 < cols) {
        for (int r = r0 + rl; r < r1; r += 32) {
            const long long e = (long long)r * cols + c0;
            float d[W];
            ldv<T>(dout + e, d);
            if (pre) {
                float p[W];
                ldv<T>(pre + e, p);
#pragma unroll
                for (int j = 0; j < W; ++j) d[j] *= dact_f(p[j], act);
            }
            if (g) stv<T>(g + e, d);
#pragma unroll
            for (int j = 0; j < W; ++j) s[j] += d[j];
        }
    }
#pragma unroll
    for (int j = 0; j < W; ++j) sm[rl][cl * W + j] = s[j];
    __syncthreads();
    if (threadIdx.x < 8 * W) {
        float t = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) t += sm[r][threadIdx.x];
        const int c = blockIdx.x * 8 * W + threadIdx.x;
        if (c < cols) partial[(long long)blockIdx.y * cols + c] = t;
    }
}
// Scalar twin for column counts that are not a multiple of the vector width.
template <typename T>
__global__ void dact_colsum_scalar_kernel(const T* dout, const T* pre, T* g, float* partial, int rows, int cols,
                                          int act) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    const int rows_per = cme_cdiv_dev(rows, (int)gridDim.y);
    const int r0 = blockIdx.y * rows_per, r1 = min(rows, r0 + rows_per);
    float s = 0.f;
    for (int r = r0; r < r1; ++r) {
        const long long e = (long long)r * cols + c;
        float d = to_f32<T>(dout[e]);
        if (pre) d *= dact_f(to_f32<T>(pre[e]), act);
        if (g) g[e] = from_f32<T>(d);
        s += d;
    }
    partial[(long long)blockIdx.y * cols + c] = s;
}
template <typename T> __global__ void scale_kernel(T* x, long long n, float s) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = from_f32<T>(to_f32<T>(x[i]) * s);
}
template <typename TI, typename TO> __global__ void cast_kernel(const TI* x, TO* y, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = from_f32<TO>(to_f32<TI>(x[i]));
}
// out = a + b (element-wise)
template <typename T> __global__ void add_kernel(const T* a, const T* b, T* out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = from_f32<T>(to_f32<T>(a[i]) + to_f32<T>(b[i]));
}
// dx = dy where x > 0 else 0
template <typename T> __global__ void relu_bwd_kernel(const T* x, const T* dy, T* dx, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dx[i] = to_f32<T>(x[i]) > 0.f ? dy[i] : from_f32<T>(0.f);
}

// One xorshift round of (seed + i) -> uniform in [-scale, scale], evaluated in fp32.
template <typename T> __global__ void init_uniform_kernel(T* out, long long n, float scale, unsigned seed) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        unsigned s = seed + (unsigned)i;
        s ^= s << 13; s ^= s >> 17; s ^= s << 5;
        const float u = (float)(s & 0x7FFFFFFFu) / (float)0x7FFFFFFF;
        out[i] = from_f32<T>((u * 2.0f - 1.0f) * scale);
    }
}

// ---- embeddings -------------------------------------------------------------------------------
// out[bt, :] = tok[tokens[bt], :] + pos[bt % T, :], rows of whole 16-byte vectors.  A token has 2^lanes_log2 lanes, as many
// as its row has vectors, up to a warp: the row number, the id and the position are found once per row, not by a 64-bit
// division per vector (16 x 1024 tokens of 768 bf16 from L2: 6.1 us, 9.1 us with the division), and rows of 64 leave no lane without work (63 x 1024
// tokens: 9.8 us with a warp each, 3.3 us so).
template <typename T>
__global__ void __launch_bounds__(256)
embed_fwd_vec_kernel(const int* __restrict__ tokens, const T* __restrict__ tok, const T* __restrict__ pos,
                     T* __restrict__ out, int BT, int T_, int D, int V, int lanes_log2) {
    constexpr int W = Vw<T>::N;
    pdl_wait();
    const unsigned bt = blockIdx.x * (256u >> lanes_log2) + (threadIdx.x >> lanes_log2);
    if (bt >= (unsigned)BT) return;
    int id = tokens[bt];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    const T* pt = tok + (long long)id * D;
    const T* pp = pos + (long long)(bt % (unsigned)T_) * D;
    T* po = out + (long long)bt * D;
    const int lanes = 1 << lanes_log2;
#pragma unroll 4
    for (int c = (threadIdx.x & (lanes - 1)) * W; c < D; c += lanes * W) {
        float a[W], b[W];
        ldv<T>(pt + c, a);
        ldv<T>(pp + c, b);
#pragma unroll
        for (int j = 0; j < W; ++j) a[j] += b[j];
        stv<T>(po + c, a);
    }
}
template <typename T>
__global__ void embed_fwd_kernel(const int* __restrict__ tokens, const T* __restrict__ tok, const T* __restrict__ pos,
                                 T* __restrict__ out, int BT, int T_, int D, int V) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)BT * D;
         i += (long long)gridDim.x * blockDim.x) {
        const int bt = (int)(i / D), c = (int)(i % D);
        int id = tokens[bt];
        id = id < 0 ? 0 : (id >= V ? V - 1 : id);
        out[i] = from_f32<T>(to_f32<T>(tok[(long long)id * D + c]) + to_f32<T>(pos[(long long)(bt % T_) * D + c]));
    }
}
// dpos[t, c] (+)= sum_b dout[b*T + t, c]   (deterministic: one thread per (t, c), loop over b)
template <typename T>
__global__ void pos_bwd_kernel(const T* __restrict__ dout, T* __restrict__ dpos, int B, int T_, int D, int accumulate) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)T_ * D) return;
    float s = accumulate ? to_f32<T>(dpos[i]) : 0.f;
    for (int b = 0; b < B; ++b) s += to_f32<T>(dout[(long long)b * T_ * D + i]);
    dpos[i] = from_f32<T>(s);
}
// Same for rows of whole 16-byte vectors.  SPLIT: a block takes 32 vectors of the [T, D] table and splits the batch over its 8
// warps, whose sums are added in warp order (the scalar form walks the whole batch in every thread, 2 bytes a load): 64 x
// 256 x 384 bf16 4.2 -> 2.6 us, 63 x 1024 x 64 4.4 -> 2.4 us.  Else a thread has a vector and walks the batch.
template <typename T, bool SPLIT>
__global__ void __launch_bounds__(256)
pos_bwd_vec_kernel(const T* __restrict__ dout, T* __restrict__ dpos, int B, long long nvec, int accumulate) {
    constexpr int W = Vw<T>::N;
    __shared__ float part[SPLIT ? 8 : 1][W][32];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long v = SPLIT ? (long long)blockIdx.x * 32 + lane : (long long)blockIdx.x * 256 + threadIdx.x;
    const int per = SPLIT ? (B + 7) / 8 : B, b0 = SPLIT ? warp * per : 0, b1 = min(B, b0 + per);
    float s[W];
#pragma unroll
    for (int j = 0; j < W; ++j) s[j] = 0.f;
    if (v < nvec) {
        if (!SPLIT && accumulate) ldv<T>(dpos + v * W, s);
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
            float x[W];
            ldv<T>(dout + ((long long)b * nvec + v) * W, x);
#pragma unroll
            for (int j = 0; j < W; ++j) s[j] += x[j];
        }
    }
    if (SPLIT) {
#pragma unroll
        for (int j = 0; j < W; ++j) part[warp][j][lane] = s[j];
        __syncthreads();
        if (warp > 0 || v >= nvec) return;
#pragma unroll
        for (int j = 0; j < W; ++j) s[j] = 0.f;
        if (accumulate) ldv<T>(dpos + v * W, s);
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int w = 0; w < 8; ++w) s[j] += part[w][j][lane];
    }
    if (v < nvec) stv<T>(dpos + v * W, s);
}
// Small vocabularies: one block (8 warps) per vocabulary row.  Each warp scans its own contiguous eighth of the
// token list with ballots and sums the matching rows of dout in token order; the eight partial rows are then added
// in warp order.  Deterministic (no atomics) and the scan is 32 tokens per instruction.
//     dtok[v, :] (+)= sum_{bt : tokens[bt] == v} dout[bt, :]
template <typename T>
__global__ void __launch_bounds__(256)
tok_bwd_scan_kernel(const int* __restrict__ tokens, const T* __restrict__ dout, T* __restrict__ dtok, int BT, int D,
                    int accumulate) {
    extern __shared__ float part[];              // [8][D]
    const int v = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (BT + 7) / 8, t0 = warp * per, t1 = min(BT, t0 + per);
    for (int c0 = 0; c0 < D; c0 += 32 * 8) {     // 8 columns per lane per pass
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        for (int base = t0; base < t1; base += 32) {
            const int bt = base + lane;
            unsigned hit = __ballot_sync(0xffffffffu, bt < t1 && tokens[bt] == v);
            while (hit) {
                const int src = base + __ffs(hit) - 1;
                hit &= hit - 1;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = c0 + lane + 32 * j;
                    if (c < D) acc[j] += to_f32<T>(dout[(long long)src * D + c]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = c0 + lane + 32 * j;
            if (c < D) part[warp * D + c] = acc[j];
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        float s2 = accumulate ? to_f32<T>(dtok[(long long)v * D + c]) : 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s2 += part[w * D + c];
        dtok[(long long)v * D + c] = from_f32<T>(s2);
    }
}
// Token-table gradient by stripes of the vocabulary: block (stripe, chunk) owns the rows id = stripe, stripe + S, ... and
// one chunk of 32 16-byte vectors of columns.  It picks its tokens out of the list, sorts them by row in shared memory
// (counting sort, stable), then every row of the stripe is summed in fp32 in token order and written exactly once.
//     dtok[v, :] (+)= sum_{bt : tokens[bt] == v} dout[bt, :]
// Against a warp per token with bf16 atomics into a cleared table: no clearing pass, one rounding per element instead of
// one per token, the same bits every time, and no queue at the rows of frequent words.  Interleaved stripes spread those,
// whose ids are near one another, over the blocks.
// All of it is latency and bookkeeping, so there is one wave of blocks (two per SM while their shared memory fits, about
// 19000 tokens at 50304 x 768 bf16, then one: 32768 tokens 64 -> 54 us), the token list is read once (its few
// tokens of the stripe are kept in shared memory for the two passes of the sort), and loads are issued in batches: sixteen
// token ids per lane, eight tokens of a table row.  Rows without a token are stores only; the others are handed out to the
// 16 warps one by one; rows with many tokens are summed by the whole block in fixed shares (of a stripe with fewer rows than
// warps from nine tokens on: 2048 tokens, 65 x 128, 5.4 us, 8.9 us where a row of 64 is left to one warp).
constexpr int STRIPE_WARPS = 16, STRIPE_BATCH = 16, STRIPE_ENTRIES = 8, STRIPE_MAX_BT = 65535;
constexpr size_t STRIPE_SMEM = 200 * 1024;
constexpr size_t STRIPE_SMEM_TWO = 112 * 1024;           // 228 KB of an SM for two blocks and the 1 KB that each takes
constexpr int STRIPE_HOT = 64, STRIPE_HOT_FEW = 8;       // the block sums rows with more tokens: eight rounds of a warp's loads
                                                         // where the stripe has a row for every warp, else one
struct StripePlan {
    int S, R, chunks;            // stripes, rows per stripe (ceil), column chunks
    unsigned magic;              // ceil(2^32 / S): id / S == umulhi(id, magic) while V * S < 2^32
    int per, nhot;               // tokens per warp (a multiple of 32), room for rows summed by the block
    bool keep;                   // shared memory has room for the warps' lists
    size_t smem;
};
inline StripePlan stripe_plan(int BT, int D, int V, int W, int num_sms) {
    StripePlan p;
    p.chunks = cme_cdiv(D, 32 * W);
    p.per = (cme_cdiv(BT, STRIPE_WARPS) + 31) / 32 * 32;
    // One wave: two blocks per SM while two fit its shared memory, else one.
    for (int per_sm = 2; per_sm > 0; --per_sm) {
        const int s = num_sms * per_sm / p.chunks;
        p.S = s < 1 ? 1 : s < V ? s : V;
        p.R = cme_cdiv(V, p.S);
        p.magic = (unsigned)(((1ull << 32) + p.S - 1) / p.S);     // S == 1 wraps to 0: handled in the kernel
        p.nhot = p.R < STRIPE_WARPS ? p.R : BT / STRIPE_HOT + 1;
        // partial sums | counts [16][R] u16 (4-byte multiple) | starts [R + 1] i32 | hot rows i32 | rows with tokens i32 |
        // sorted positions [BT] u16 | the warps' positions [16][per] u16
        const size_t cnt = ((size_t)STRIPE_WARPS * p.R * 2 + 3) / 4 * 4;
        p.smem = (size_t)STRIPE_WARPS * 32 * W * 4 + cnt + ((size_t)p.R + 1) * 4 + (size_t)p.nhot * 4 + (size_t)p.R * 4 +
                 (size_t)BT * 2;
        const size_t lists = (size_t)STRIPE_WARPS * p.per * 2;
        p.keep = p.smem + lists <= STRIPE_SMEM;
        if (p.keep) p.smem += lists;
        if (p.smem <= STRIPE_SMEM_TWO || (long long)p.S * p.chunks <= num_sms) break;
    }
    return p;
}
template <typename T>
__global__ void __launch_bounds__(STRIPE_WARPS * 32, 2)
tok_bwd_stripe_kernel(const int* __restrict__ tokens, const T* __restrict__ dout, T* __restrict__ dtok, int BT, int D, int V,
                      const StripePlan plan, int accumulate) {
    constexpr int W = Vw<T>::N, NW = STRIPE_WARPS, NE = STRIPE_ENTRIES;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ int n_hot, n_used, next_used;
    const int S = plan.S, R = plan.R, per = plan.per;
    float* part = reinterpret_cast<float*>(sm_raw);                        // [NW][W][32]
    unsigned short* cnt = reinterpret_cast<unsigned short*>(part + NW * W * 32);   // [NW][R]
    int* start = reinterpret_cast<int*>(sm_raw + (size_t)NW * W * 32 * 4 + ((size_t)NW * R * 2 + 3) / 4 * 4);   // [R + 1]
    int* hot = start + R + 1;                                              // [nhot]
    int* used = hot + plan.nhot;                                           // [R] the other rows with tokens, any order
    unsigned short* sorted = reinterpret_cast<unsigned short*>(used + R);  // [BT]
    unsigned short* found = sorted + BT;                                   // [NW][per] positions of the stripe's tokens
    pdl_wait();
    const int stripe = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = (blockIdx.y * 32 + lane) * W;
    const bool in = c < D;
    for (int i = threadIdx.x; i < NW * R; i += NW * 32) cnt[i] = 0;
    if (threadIdx.x == 0) n_hot = n_used = next_used = 0;
    __syncthreads();
    const int t0 = warp * per, t1 = min(BT, t0 + per);
    unsigned short* wc = cnt + warp * R;
    unsigned short* wf = found + warp * per;
    // local row of a token id, or -1 if it is not of this stripe
    auto local = [&](int id) -> int {
        if (id < 0 || id >= V) return -1;
        const int q = S == 1 ? id : (int)__umulhi((unsigned)id, plan.magic);
        return id - q * S == stripe ? q : -1;
    };
    // the warp's tokens of this stripe, in order (without room for them, all its tokens)
    const bool keep = plan.keep;
    int nf = keep ? 0 : max(t1 - t0, 0);
    for (int base = t0; keep && base < t1; base += 32 * STRIPE_BATCH) {
        int id[STRIPE_BATCH];
#pragma unroll
        for (int k = 0; k < STRIPE_BATCH; ++k) id[k] = base + 32 * k + lane < t1 ? tokens[base + 32 * k + lane] : -1;
#pragma unroll
        for (int k = 0; k < STRIPE_BATCH; ++k) {
            const bool mine = local(id[k]) >= 0;
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            if (mine) wf[nf + __popc(m & ((1u << lane) - 1))] = (unsigned short)(base + 32 * k + lane);
            nf += __popc(m);
        }
    }
    __syncwarp();
    // pass 0 counts the warp's tokens per row; pass 1 puts their positions in order behind the earlier warps' ones
    for (int pass = 0; pass < 2; ++pass) {
        for (int base = 0; base < nf; base += 32) {
            const int pos = base + lane < nf ? (keep ? wf[base + lane] : t0 + base + lane) : -1;
            const int row = pos >= 0 ? local(tokens[pos]) : -1;
            if (!__any_sync(0xffffffffu, row >= 0)) continue;
            const unsigned same = __match_any_sync(0xffffffffu, row);
            const int before = __popc(same & ((1u << lane) - 1));
            if (row >= 0) {
                const int at = wc[row];
                if (pass) sorted[start[row] + at + before] = (unsigned short)pos;
            }
            __syncwarp();
            if (row >= 0 && before == 0) wc[row] = (unsigned short)(wc[row] + __popc(same));
            __syncwarp();
        }
        __syncthreads();
        if (pass) break;
        // each row's counts become the warps' offsets in the row; `start` the rows' lengths, then their first places
        const int hot_at = R >= NW ? STRIPE_HOT : STRIPE_HOT_FEW;
        for (int r = threadIdx.x; r < R; r += NW * 32) {
            int n = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const int k = cnt[w * R + r];
                cnt[w * R + r] = (unsigned short)n;
                n += k;
            }
            start[r] = n;
            if (n > hot_at) hot[atomicAdd(&n_hot, 1)] = r;
            else if (n > 0) used[atomicAdd(&n_used, 1)] = r;
        }
        __syncthreads();
        if (warp == 0) {
            int sum = 0;
            for (int r = lane; r < (R + 31) / 32 * 32; r += 32) {
                const int n = r < R ? start[r] : 0;
                int incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                if (r < R) start[r] = sum + incl - n;
                sum += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) start[R] = sum;
        }
        __syncthreads();
    }
    const T* src = dout + (in ? c : 0);                    // (lanes without columns read nothing)
    if (!accumulate && in) {                               // rows without a token
        float zero[W];
#pragma unroll
        for (int j = 0; j < W; ++j) zero[j] = 0.f;
        for (int r = warp; r < R; r += NW) {
            const long long id = (long long)r * S + stripe;
            if (id < V && start[r + 1] == start[r]) stv<T>(dtok + id * D + c, zero);
        }
    }
    // s += the rows dout[sorted[e0 .. e1)], NE loads in flight
    auto add_tokens = [&](float (&s)[W], int e0, int e1) {
        for (int e = e0; e < e1; e += NE) {
            uint4 raw[NE];
#pragma unroll
            for (int k = 0; k < NE; ++k)
                if (e + k < e1) raw[k] = *reinterpret_cast<const uint4*>(src + (long long)sorted[e + k] * D);
#pragma unroll
            for (int k = 0; k < NE; ++k) {
                if (e + k < e1) {
                    float x[W];
                    unpack_words<T>(raw[k], x);
#pragma unroll
                    for (int j = 0; j < W; ++j) s[j] += x[j];
                }
            }
        }
    };
    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&next_used, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= n_used) break;
        if (!in) continue;
        const int r = used[u];
        T* dst = dtok + ((long long)r * S + stripe) * D + c;
        float s[W];
#pragma unroll
        for (int j = 0; j < W; ++j) s[j] = 0.f;
        if (accumulate) ldv<T>(dst, s);
        add_tokens(s, start[r], start[r + 1]);
        stv<T>(dst, s);
    }
    const int nh = n_hot;
    for (int h = 0; h < nh; ++h) {
        const int r = hot[h], n0 = start[r], n = start[r + 1] - n0;
        T* dst = dtok + ((long long)r * S + stripe) * D + c;
        const int share = (n + NW - 1) / NW, e0 = min(n, warp * share), e1 = min(n, e0 + share);
        float s[W];
#pragma unroll
        for (int j = 0; j < W; ++j) s[j] = 0.f;
        if (in) add_tokens(s, n0 + e0, n0 + e1);
#pragma unroll
        for (int j = 0; j < W; ++j) part[(warp * W + j) * 32 + lane] = s[j];
        __syncthreads();
        if (warp < W) {                                    // warp j adds up column j of every lane's vector
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) t += part[(w * W + warp) * 32 + lane];
            part[warp * 32 + lane] = t;                    // (its own slots of warp 0's sums)
        }
        __syncthreads();
        if (warp == 0 && in) {
#pragma unroll
            for (int j = 0; j < W; ++j) s[j] = 0.f;
            if (accumulate) ldv<T>(dst, s);
#pragma unroll
            for (int j = 0; j < W; ++j) s[j] += part[j * 32 + lane];
            stv<T>(dst, s);
        }
        __syncthreads();
    }
}
// Large vocabularies: one warp per token, atomic adds into the (already initialised) table gradient.
__device__ __forceinline__ void atomic_add_t(float* p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_t(__nv_bfloat16* p, float v) { atomicAdd(p, __float2bfloat16_rn(v)); }
template <typename T>
__global__ void tok_bwd_atomic_kernel(const int* __restrict__ tokens, const T* __restrict__ dout, T* __restrict__ dtok,
                                      int BT, int D, int V) {
    const int bt = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (bt >= BT) return;
    const int id = tokens[bt];
    if (id < 0 || id >= V) return;
    if constexpr (sizeof(T) == 2) {
        if (D % 2 == 0) {
            for (int c = (threadIdx.x & 31) * 2; c < D; c += 64) {
                __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(dout + (long long)bt * D + c);
                atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtok + (long long)id * D + c), v);
            }
            return;
        }
    }
    for (int c = threadIdx.x & 31; c < D; c += 32)
        atomic_add_t(dtok + (long long)id * D + c, to_f32<T>(dout[(long long)bt * D + c]));
}

inline int grid_for(long long n, int block = 256, int cap = 148 * 16) {
    long long g = (n + block - 1) / block;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}
template <typename T> bool aligned16(const T* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T>
int bias_act_res_t(const void* x, const void* bias, const void* res, void* pre, void* out, long long rows, int cols,
                   int act, cudaStream_t st) {
    constexpr int W = Vw<T>::N;
    const long long n = rows * cols;
    const bool vec = cols % W == 0 && aligned16((const T*)x) && aligned16((const T*)out) &&
                     (!bias || aligned16((const T*)bias)) && (!res || aligned16((const T*)res)) &&
                     (!pre || aligned16((const T*)pre));
    if (vec && cme_index32(n / W))
        bias_act_res_kernel<T, unsigned><<<grid_for(n / W), 256, 0, st>>>((const T*)x, (const T*)bias, (const T*)res, (T*)pre,
                                                                           (T*)out, (unsigned)(n / W), cols, act);
    else if (vec)
        bias_act_res_kernel<T, unsigned long long><<<grid_for(n / W), 256, 0, st>>>(
            (const T*)x, (const T*)bias, (const T*)res, (T*)pre, (T*)out, (unsigned long long)(n / W), cols, act);
    else
        bias_act_res_scalar_kernel<T><<<grid_for(n), 256, 0, st>>>((const T*)x, (const T*)bias, (const T*)res,
                                                                    (T*)pre, (T*)out, n, cols, act);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// dbias[c] (+)= sum over the `slabs` rows of partial[slabs][cols], added in a fixed order: NG row groups per column, each
// of whose threads sums every NG-th row (four independent chains), then the groups' sums are added in shared memory.  The
// rows come from a GEMM epilogue that sums its stored output per 32-row slab, or from dact_colsum_kernel's row splits.
template <typename T, int NG>
__global__ void __launch_bounds__(NG == 1 ? 256 : NG * 32)
colsum_slabs_finalize_kernel(const float* __restrict__ partial, int slabs, int cols, T* dbias, int accumulate) {
    constexpr int NC = NG == 1 ? 256 : 32;         // columns per block
    __shared__ float sm[NG][33];
    pdl_wait();
    const int cx = threadIdx.x % NC, ry = threadIdx.x / NC;
    const int c = blockIdx.x * NC + cx;
    float s = 0.f;
    if (c < cols) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        int r = ry;
        if constexpr (NG == 32) {                  // many rows: rounds without a test per load
            for (; r + 3 * NG < slabs; r += 4 * NG) {
                s0 += partial[(long long)r * cols + c];
                s1 += partial[(long long)(r + NG) * cols + c];
                s2 += partial[(long long)(r + 2 * NG) * cols + c];
                s3 += partial[(long long)(r + 3 * NG) * cols + c];
            }
            for (; r < slabs; r += NG) s0 += partial[(long long)r * cols + c];
        } else {                                   // few: the last round's loads are in flight together too
            for (; r < slabs; r += 4 * NG) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = r + k * NG < slabs ? partial[(long long)(r + k * NG) * cols + c] : 0.f;
                s0 += v[0];
                s1 += v[1];
                s2 += v[2];
                s3 += v[3];
            }
        }
        s = (s0 + s1) + (s2 + s3);
    }
    if (NG > 1) {
        sm[ry][cx] = s;
        __syncthreads();
    }
    if (ry == 0 && c < cols) {
        float t = 0.f;
#pragma unroll
        for (int g = 0; g < NG; ++g) t += NG > 1 ? sm[g][cx] : s;
        dbias[c] = from_f32<T>(accumulate ? to_f32<T>(dbias[c]) + t : t);
    }
}
// The time is that of a thread's chain of loads while the blocks fit the chip: 32 groups where 8 need more than three rounds
// of loads (512 columns, us with 8 / 32 groups: 16 rows 1.3 / 1.5, 64 rows 1.5 / 1.7, 128 rows 1.7 / 1.6, 512 rows 3.6 / 2.6,
// 2048 rows 11 / 5.8).  Beyond 32768 columns the blocks come in several waves and fewer groups pay (50304 columns, 1 / 8 / 32
// groups: 16 rows 1.9 / 2.8 / 6.8, 512 rows 39 / 17 / 27, 2048 rows 159 / 74 / 93).
template <typename T>
int colsum_finish(const float* partial, int slabs, int cols, T* dbias, int accumulate, cudaStream_t st) {
    auto run = [&](auto kernel, int columns, int threads) -> int {
        CME_CUDA(cme_launch_dependent(kernel, dim3(cme_cdiv(cols, columns)), dim3(threads), 0, st, partial, slabs, cols, dbias,
                                      accumulate));
        CME_LAUNCH_CHECK();
        return CME_OK;
    };
    const bool wide = cols > 32768;
    if (wide && slabs <= 16) return run(colsum_slabs_finalize_kernel<T, 1>, 256, 256);
    if (wide || slabs <= 96) return run(colsum_slabs_finalize_kernel<T, 8>, 32, 256);
    return run(colsum_slabs_finalize_kernel<T, 32>, 32, 1024);
}

template <typename T>
int dact_colsum_t(const void* dout, const void* pre, void* g, void* dbias, float* scratch, int splits, int rows,
                  int cols, int act, int accumulate, cudaStream_t st) {
    constexpr int W = Vw<T>::N;
    const bool vec = cols % W == 0 && aligned16((const T*)dout) && (!pre || aligned16((const T*)pre)) &&
                     (!g || aligned16((const T*)g));
    if (vec) {
        dim3 grid(cme_cdiv(cols, 8 * W), splits);
        CME_CUDA(cme_launch_dependent(dact_colsum_kernel<T>, grid, dim3(256), 0, st, (const T*)dout, (const T*)pre, (T*)g,
                                      scratch, rows, cols, act));
    } else {
        dim3 grid(cme_cdiv(cols, 128), splits);
        dact_colsum_scalar_kernel<T><<<grid, 128, 0, st>>>((const T*)dout, (const T*)pre, (T*)g, scratch, rows, cols,
                                                            act);
    }
    CME_LAUNCH_CHECK();
    return dbias ? colsum_finish<T>(scratch, splits, cols, (T*)dbias, accumulate, st) : CME_OK;
}

}  // namespace

#define DISPATCH_T(dtype, expr_bf16, expr_f32) ((dtype) == CME_BF16 ? (expr_bf16) : (expr_f32))

// out = act(x + bias) + residual; pre_out receives x + bias.  act: 0 none, 1 relu, 2 gelu.
CME_API int cme_bias_act_residual(int dtype, const void* x, const void* bias, const void* residual, void* pre_out,
                                  void* out, long long rows, int cols, int act, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && cols > 0, CME_ERR_SHAPE, "bias_act_residual: empty input");
    return DISPATCH_T(dtype, bias_act_res_t<__nv_bfloat16>(x, bias, residual, pre_out, out, rows, cols, act, st),
                      bias_act_res_t<float>(x, bias, residual, pre_out, out, rows, cols, act, st));
}

// Row splits used by cme_dact_colsum for `rows`; scratch must hold splits * cols floats.
CME_API int cme_colsum_splits(int rows, int cols) {
    int col_blocks = cme_cdiv(cols, 64);
    int s = cme_cdiv(296, col_blocks);
    int max_s = cme_cdiv(rows, 64);
    if (s > max_s) s = max_s;
    return s < 1 ? 1 : s;
}

// g = dout * act'(pre) (pre, g optional) and dbias (+)= column sums of g.
CME_API int cme_dact_colsum(int dtype, const void* dout, const void* pre, void* g, void* dbias, float* scratch,
                            int rows, int cols, int act, int accumulate, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && cols > 0, CME_ERR_SHAPE, "dact_colsum: empty input");
    const int splits = cme_colsum_splits(rows, cols);
    return DISPATCH_T(dtype,
                      dact_colsum_t<__nv_bfloat16>(dout, pre, g, dbias, scratch, splits, rows, cols, act, accumulate, st),
                      dact_colsum_t<float>(dout, pre, g, dbias, scratch, splits, rows, cols, act, accumulate, st));
}

// dbias (+)= column sums of partial[slabs][cols] (the per-slab sums a GEMM epilogue left, gemm.h: colsum).
CME_API int cme_colsum_slabs_finalize(int dtype, const float* partial, int slabs, int cols, void* dbias, int accumulate,
                                      void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(slabs > 0 && cols > 0, CME_ERR_SHAPE, "colsum finalize: empty input");
    return DISPATCH_T(dtype, colsum_finish<__nv_bfloat16>(partial, slabs, cols, (__nv_bfloat16*)dbias, accumulate, st),
                      colsum_finish<float>(partial, slabs, cols, (float*)dbias, accumulate, st));
}

CME_API int cme_scale(int dtype, void* x, long long n, float s, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    if (dtype == CME_BF16) scale_kernel<__nv_bfloat16><<<grid_for(n), 256, 0, st>>>((__nv_bfloat16*)x, n, s);
    else scale_kernel<float><<<grid_for(n), 256, 0, st>>>((float*)x, n, s);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_cast(int src_dtype, const void* x, int dst_dtype, void* y, long long n, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    const int g = grid_for(n);
    if (src_dtype == CME_F32 && dst_dtype == CME_BF16)
        cast_kernel<float, __nv_bfloat16><<<g, 256, 0, st>>>((const float*)x, (__nv_bfloat16*)y, n);
    else if (src_dtype == CME_BF16 && dst_dtype == CME_F32)
        cast_kernel<__nv_bfloat16, float><<<g, 256, 0, st>>>((const __nv_bfloat16*)x, (float*)y, n);
    else if (src_dtype == CME_F32)
        cast_kernel<float, float><<<g, 256, 0, st>>>((const float*)x, (float*)y, n);
    else
        cast_kernel<__nv_bfloat16, __nv_bfloat16><<<g, 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_add(int dtype, const void* a, const void* b, void* out, long long n, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    if (dtype == CME_BF16)
        add_kernel<__nv_bfloat16><<<grid_for(n), 256, 0, st>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                                (__nv_bfloat16*)out, n);
    else add_kernel<float><<<grid_for(n), 256, 0, st>>>((const float*)a, (const float*)b, (float*)out, n);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_relu_bwd(int dtype, const void* x, const void* dy, void* dx, long long n, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    if (dtype == CME_BF16)
        relu_bwd_kernel<__nv_bfloat16><<<grid_for(n), 256, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)dy,
                                                                     (__nv_bfloat16*)dx, n);
    else relu_bwd_kernel<float><<<grid_for(n), 256, 0, st>>>((const float*)x, (const float*)dy, (float*)dx, n);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_init_uniform(int dtype, void* out, long long n, float scale, unsigned seed, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    if (dtype == CME_BF16) init_uniform_kernel<__nv_bfloat16><<<grid_for(n), 256, 0, st>>>((__nv_bfloat16*)out, n, scale, seed);
    else init_uniform_kernel<float><<<grid_for(n), 256, 0, st>>>((float*)out, n, scale, seed);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

namespace {

template <typename T>
int embed_fwd_t(const int* tokens, const void* tok, const void* pos, void* out, int BT, int T_, int D, int V, cudaStream_t st) {
    if (D % Vw<T>::N == 0 && aligned16((const T*)tok) && aligned16((const T*)pos) && aligned16((const T*)out)) {
        int lanes_log2 = 0;
        while (lanes_log2 < 5 && (Vw<T>::N << lanes_log2) < D) ++lanes_log2;
        CME_CUDA(cme_launch_dependent(embed_fwd_vec_kernel<T>, dim3(cme_cdiv(BT, 256 >> lanes_log2)), dim3(256), 0, st, tokens,
                                      (const T*)tok, (const T*)pos, (T*)out, BT, T_, D, V, lanes_log2));
    } else {
        embed_fwd_kernel<T><<<grid_for((long long)BT * D), 256, 0, st>>>(tokens, (const T*)tok, (const T*)pos, (T*)out, BT,
                                                                        T_, D, V);
    }
    CME_LAUNCH_CHECK();
    return CME_OK;
}

template <typename T>
int tok_bwd_t(const int* tokens, const void* dout, void* dtok, int BT, int D, int V, int accumulate, cudaStream_t st) {
    constexpr int W = Vw<T>::N;
    const bool scan = (long long)V * BT <= (1ll << 22) && D <= 1536;
    if (D % W == 0 && BT <= STRIPE_MAX_BT && aligned16((const T*)dout) && aligned16((const T*)dtok)) {
        int num_sms = 0;
        const int rc = cme_num_sms(&num_sms);
        if (rc) return rc;
        const StripePlan p = stripe_plan(BT, D, V, W, num_sms);
        // Stripes replace the block per vocabulary row wherever that would run (65 x 384 bf16, us rows / stripes: 16384 tokens
        // 64 / 11, 39000 152 / 22, three quarters of 16384 one id 707 / 97; lists of up to 512 tokens take 1 to 2 us more than its
        // 2.5 to 5, and 6 to 48 us less where half of them are one id).
        // On larger tables they replace the atomics for 16-bit types while the lists fit, because those round every sum
        // to 16 bits once per token (4.5e-3 off the exact sums instead of 1.8e-3) and in another order each time.  What that
        // costs or saves, token gradient alone, inputs from memory, us atomics with their clearing pass / stripes:
        //   50304 x 768   1024 tokens 22.6 / 19.7   16384 33.1 / 35.4   32768 50 / 54   three quarters of 16384 one id 150 / 160
        //   50304 x 256   4096 tokens 10.7 / 12.7   16384 14.6 / 20.8
        //   50304 x 64    4096 tokens  5.5 / 11.0   16384  6.9 / 19.0
        //   8192 x 512    4096 tokens 10.5 / 11.7   16384 16.6 / 20.4   three quarters of 16384 one id 128 / 154
        // Atomics keep fp32, whose sums they do not round to 16 bits, and longer lists, which every block would walk three
        // times (64512 tokens, 50304 x 768, with the position table: 128 / 267 us).
        const bool better = scan || (sizeof(T) == 2 && p.keep);
        if (better && (unsigned long long)V * p.S < (1ull << 32) && p.smem <= STRIPE_SMEM) {
            auto k = tok_bwd_stripe_kernel<T>;
            if (p.smem > 48 * 1024)
                CME_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STRIPE_SMEM));
            CME_CUDA(cme_launch_dependent(k, dim3(p.S, p.chunks), dim3(STRIPE_WARPS * 32), p.smem, st, tokens, (const T*)dout,
                                          (T*)dtok, BT, D, V, p, accumulate));
            CME_LAUNCH_CHECK();
            return CME_OK;
        }
    }
    if (scan) {
        const size_t sm = (size_t)8 * D * sizeof(float);
        CME_REQUIRE(sm <= 48 * 1024, CME_ERR_LIMIT, "embedding backward: hidden size %d too large for the scan path", D);
        tok_bwd_scan_kernel<T><<<V, 256, sm, st>>>(tokens, (const T*)dout, (T*)dtok, BT, D, accumulate);
    } else {
        if (!accumulate) CME_CUDA(cudaMemsetAsync(dtok, 0, (size_t)V * D * sizeof(T), st));
        tok_bwd_atomic_kernel<T><<<cme_cdiv(BT, 8), 256, 0, st>>>(tokens, (const T*)dout, (T*)dtok, BT, D, V);
    }
    CME_LAUNCH_CHECK();
    return CME_OK;
}

template <typename T>
int pos_bwd_t(const void* dout, void* dpos, int BT, int T_, int D, int accumulate, cudaStream_t st) {
    constexpr int W = Vw<T>::N;
    const long long n = (long long)T_ * D;
    if (D % W == 0 && aligned16((const T*)dout) && aligned16((const T*)dpos)) {
        // Whole blocks of vectors for two blocks an SM leave nothing to split while the batch is a thread's few loads
        // (1024 x 768 fp32, us split / whole: batch 1 4.8 / 1.6, 8 5.6 / 2.9, 16 7.0 / 4.2).
        const bool split = BT / T_ > 16 || n / W < 256 * 296;
        auto kernel = split ? pos_bwd_vec_kernel<T, true> : pos_bwd_vec_kernel<T, false>;
        CME_CUDA(cme_launch_dependent(kernel, dim3(cme_cdiv(n / W, split ? 32 : 256)), dim3(256), 0, st, (const T*)dout, (T*)dpos,
                                      BT / T_, n / W, accumulate));
    } else {
        pos_bwd_kernel<T><<<cme_cdiv(n, 256), 256, 0, st>>>((const T*)dout, (T*)dpos, BT / T_, T_, D, accumulate);
    }
    CME_LAUNCH_CHECK();
    return CME_OK;
}

}  // namespace

CME_API int cme_embedding_fwd(int dtype, const int* tokens, const void* tok, const void* pos, void* out, int BT, int T,
                              int D, int V, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(BT > 0 && D > 0 && T > 0, CME_ERR_SHAPE, "embedding: empty input");
    return DISPATCH_T(dtype, embed_fwd_t<__nv_bfloat16>(tokens, tok, pos, out, BT, T, D, V, st),
                      embed_fwd_t<float>(tokens, tok, pos, out, BT, T, D, V, st));
}

// dtok (+)= scatter of dout rows by token id; dpos (+)= sum over the batch.  With accumulate = 0 the outputs are
// overwritten.  The stripe kernel takes small vocabularies, and 16-bit tables of any size while a block's shared memory holds
// the token lists, where rows are whole 16-byte vectors and positions fit 16 bits; the rest: a block per vocabulary row for
// small vocabularies, else atomics into a table that is zero-filled first.
CME_API int cme_embedding_bwd(int dtype, const int* tokens, const void* dout, void* dtok, void* dpos, int BT, int T,
                              int D, int V, int accumulate, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(BT > 0 && D > 0 && T > 0 && BT % T == 0, CME_ERR_SHAPE, "embedding backward: bad shape");
    if (dtok) {
        const int rc = DISPATCH_T(dtype, tok_bwd_t<__nv_bfloat16>(tokens, dout, dtok, BT, D, V, accumulate, st),
                                  tok_bwd_t<float>(tokens, dout, dtok, BT, D, V, accumulate, st));
        if (rc) return rc;
    }
    if (dpos)
        return DISPATCH_T(dtype, pos_bwd_t<__nv_bfloat16>(dout, dpos, BT, T, D, accumulate, st),
                          pos_bwd_t<float>(dout, dpos, BT, T, D, accumulate, st));
    return CME_OK;
}

// ---------------------------------------------------------------------------------------------------
// Allocation-free variant of cme_dact_colsum (see noalloc.h for who it is for and the rules of use).
// ---------------------------------------------------------------------------------------------------
#include "noalloc.h"

#include <mutex>

// Scratch for the per-split partial column sums.  In host code this name is only a handle for the runtime
// (it is not a device address); the address kernels may use comes from cudaGetSymbolAddress below.
static __device__ __align__(256) float g_noalloc_scratch[CME_NOALLOC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device; looked up once per device.
int noalloc_scratch(float** out) {
    int dev = 0;
    CME_CUDA(cudaGetDevice(&dev));
    CME_REQUIRE(dev >= 0 && dev < kMaxDevices, CME_ERR_LIMIT, "noalloc: device index %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        float* p = nullptr;
        CME_CUDA(cudaGetSymbolAddress((void**)&p, g_noalloc_scratch));
        CME_REQUIRE(p != nullptr, CME_ERR_CUDA, "noalloc: cudaGetSymbolAddress returned a null address");
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return CME_OK;
}
}  // namespace

CME_API int cme_dact_colsum_noalloc(int dtype, const void* dout, const void* pre, void* g, void* dbias, int rows,
                                    int cols, int act, int accumulate, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && cols > 0, CME_ERR_SHAPE, "dact_colsum_noalloc: empty input");
    CME_REQUIRE(dtype == CME_F32 || dtype == CME_BF16, CME_ERR_SHAPE, "dact_colsum_noalloc: unknown dtype %d", dtype);
    const int splits = cme_colsum_splits(rows, cols);
    const long long need = (long long)splits * cols;
    CME_REQUIRE(need <= (long long)CME_NOALLOC_SCRATCH_FLOATS, CME_ERR_LIMIT,
                "dact_colsum_noalloc: %d rows x %d cols needs %lld scratch floats, the built-in scratch holds %d; "
                "use cme_dact_colsum with a caller-provided buffer",
                rows, cols, need, (int)CME_NOALLOC_SCRATCH_FLOATS);
    float* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    return DISPATCH_T(dtype,
                      dact_colsum_t<__nv_bfloat16>(dout, pre, g, dbias, scratch, splits, rows, cols, act, accumulate, st),
                      dact_colsum_t<float>(dout, pre, g, dbias, scratch, splits, rows, cols, act, accumulate, st));
}
