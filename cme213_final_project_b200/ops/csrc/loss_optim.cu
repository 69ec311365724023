// Fused softmax-cross-entropy (loss + gradient), global gradient norm, and Adam / AdamW on the flat arena.
//
// Reference counterparts: cross_entropy_kernel + reduce_sum_kernel + scale_device_scalar
// (FINAL_CLEAN_CODE_/src/kernels/activations.cu:438-531: one warp per row, loss summed with atomicAdd),
// norm_sq_kernel / clip_scale_kernel (:360-392) and adam_clipped_kernel
// (FINAL_CLEAN_CODE_/src/model/transformer.cu:598-636).  Here: one block per row with an online
// max / sum pass so a 50k-entry vocabulary row is read once for the statistics and once for the gradient,
// the mean loss and the squared norm are reduced in two fixed-order stages (bit-reproducible), and the
// optimizer reads its step counter, learning rate and the squared norm from device memory so that a
// captured CUDA graph of the step stays correct on every replay (the reference bakes the host-computed
// bias corrections into its captured launch).
#include "common.h"
#include <cuda_fp16.h>

namespace {

constexpr int CE_THREADS = 256;

// dlogits[r, :] = (softmax(logits[r, :]) - onehot(target)) * grad_scale; losses[r] = -log(p_target (+ eps)).
// In-place (dlogits == logits) is allowed: each element is read before it is written by the same thread.
template <typename T>
__global__ void __launch_bounds__(CE_THREADS)
cross_entropy_kernel(const T* __restrict__ logits, const int* __restrict__ targets, T* dlogits, float* __restrict__ losses,
                     int V, long long ld, float grad_scale, float prob_eps) {
    __shared__ float scratch[32];
    const long long off = (long long)blockIdx.x * ld;
    const T* row = logits + off;
    float m = -INFINITY, s = 0.f;
    for (int i = threadIdx.x; i < V; i += CE_THREADS) {
        const float x = to_f32<T>(row[i]);
        if (x > m) { s *= __expf(m - x); m = x; }
        s += __expf(x - m);
    }
    const float row_max = block_max(m, scratch);
    s *= __expf(m - row_max);               // m = -inf with s = 0 gives 0 * 0
    if (m == -INFINITY) s = 0.f;
    const float denom = block_sum(s, scratch);
    const float inv = 1.f / (denom + prob_eps);
    int tgt = targets[blockIdx.x];
    tgt = tgt < 0 ? 0 : (tgt >= V ? V - 1 : tgt);
    if (threadIdx.x == 0) {
        const float p = __expf(to_f32<T>(row[tgt]) - row_max) * inv;
        losses[blockIdx.x] = prob_eps > 0.f ? -logf(p + prob_eps) : -(to_f32<T>(row[tgt]) - row_max - logf(denom));
    }
    __syncthreads();                        // the target logit is read above before anyone overwrites it
    if (dlogits) {
        T* g = dlogits + off;
        for (int i = threadIdx.x; i < V; i += CE_THREADS) {
            float p = __expf(to_f32<T>(row[i]) - row_max) * inv;
            if (i == tgt) p -= 1.f;
            g[i] = from_f32<T>(p * grad_scale);
        }
    }
}


// bf16 rows whose length is a multiple of 8 and whose base is 16-byte aligned: 128-bit loads, the row is kept
// in shared memory between the statistics pass and the gradient pass when it fits (read once from DRAM).
constexpr int CEV_THREADS = 512;
__global__ void __launch_bounds__(CEV_THREADS)
cross_entropy_bf16_vec_kernel(const __nv_bfloat16* __restrict__ logits, const int* __restrict__ targets,
                              __nv_bfloat16* dlogits, float* __restrict__ losses, int V, long long ld,
                              float grad_scale, float prob_eps, int cache_row) {
    extern __shared__ uint4 srow[];
    __shared__ float scratch[32];
    const long long off = (long long)blockIdx.x * ld;
    const uint4* row = reinterpret_cast<const uint4*>(logits + off);
    const int nv = V / 8;
    float m = -INFINITY, s = 0.f;
    for (int i = threadIdx.x; i < nv; i += CEV_THREADS) {
        const uint4 u = row[i];
        if (cache_row) srow[i] = u;
        float x[8];
        unpack8(u, x);
        float mx = x[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) mx = fmaxf(mx, x[j]);
        if (mx > m) { s *= __expf(m - mx); m = mx; }
#pragma unroll
        for (int j = 0; j < 8; ++j) s += __expf(x[j] - m);
    }
    const float row_max = block_max(m, scratch);
    s = (m == -INFINITY) ? 0.f : s * __expf(m - row_max);
    const float denom = block_sum(s, scratch);
    const float inv = 1.f / (denom + prob_eps);
    int tgt = targets[blockIdx.x];
    tgt = tgt < 0 ? 0 : (tgt >= V ? V - 1 : tgt);
    if (threadIdx.x == 0) {
        const float xt = __bfloat162float(logits[off + tgt]);
        const float p = __expf(xt - row_max) * inv;
        losses[blockIdx.x] = prob_eps > 0.f ? -logf(p + prob_eps) : -(xt - row_max - logf(denom));
    }
    __syncthreads();
    if (dlogits) {
        uint4* g = reinterpret_cast<uint4*>(dlogits + off);
        for (int i = threadIdx.x; i < nv; i += CEV_THREADS) {
            float x[8];
            unpack8(cache_row ? srow[i] : row[i], x);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float p = __expf(x[j] - row_max) * inv;
                if (i * 8 + j == tgt) p -= 1.f;
                x[j] = p * grad_scale;
            }
            g[i] = pack8(x);
        }
    }
}

// Same contract, for rows of at most THREADS * NV 16-byte vectors: the row lives in registers from its single read to its single
// write.  Pass 1 finds the maximum, pass 2 evaluates exp(x - max) once per element and keeps it as fp16 in the registers that held
// the logits (values in (0, 1], 11 significant bits -- finer than the bf16 the gradient is stored in), pass 3 only scales.  One
// exponential per element instead of two: the kernel is otherwise bound by the special-function unit as much as by
// memory (100 K exponentials per row).
// A block's time is a chain of load, maximum, exponentials, sum and store with a barrier between each, so what counts is that all of
// its loads are on their way at once and that enough rows share an SM.  The loads are asm in a loop of their own: left to the
// compiler they alternate with the maxima (8192 x 50304: 311 us, 265 so, 6.2 TB/s).  NV is what the row needs: see ce_rows.
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_h2(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <int THREADS, int NV, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS)
cross_entropy_bf16_reg_kernel(const __nv_bfloat16* __restrict__ logits, const int* __restrict__ targets,
                              __nv_bfloat16* dlogits, float* __restrict__ losses, int V, long long ld,
                              float grad_scale, float prob_eps) {
    __shared__ float scratch[32];
    __shared__ int target;
    constexpr bool ONE = NV > 10;    // the target is in one thread's register only: with it in all, 64 don't hold a longer row
    pdl_wait();                      // (8192 x 50304: 280 us, 265 so; with shorter rows the other way round, 59 for 55 at 20000)
    int tgt = 0;
    if (!ONE || threadIdx.x == 0) tgt = targets[blockIdx.x];
    const long long off = (long long)blockIdx.x * ld;
    const uint4* row = reinterpret_cast<const uint4*>(logits + off);
    const int nv = V / 8;
    uint4 r[NV];
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + k * THREADS;
        if (i < nv)
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[k].x), "=r"(r[k].y), "=r"(r[k].z), "=r"(r[k].w)
                         : "l"(row + i));
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (threadIdx.x + k * THREADS < nv) {
            float x[8];
            unpack8(r[k], x);
#pragma unroll
            for (int j = 0; j < 8; ++j) m = fmaxf(m, x[j]);
        }
    }
    __shared__ float xt;
    tgt = tgt < 0 ? 0 : (tgt >= V ? V - 1 : tgt);
    if (threadIdx.x == 0) {          // read before the barriers: after them the row is overwritten in place
        xt = __bfloat162float(logits[off + tgt]);
        target = tgt;
    }
    const float row_max = block_max(m, scratch);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (threadIdx.x + k * THREADS < nv) {
            float x[8];
            unpack8(r[k], x);
#pragma unroll
            for (int j = 0; j < 8; ++j) { x[j] = __expf(x[j] - row_max); s += x[j]; }
            r[k] = make_uint4(pack_h2(x[0], x[1]), pack_h2(x[2], x[3]), pack_h2(x[4], x[5]), pack_h2(x[6], x[7]));
        }
    }
    const float denom = block_sum(s, scratch);
    const float inv = 1.f / (denom + prob_eps);
    if (threadIdx.x == 0) {
        const float p = __expf(xt - row_max) * inv;
        losses[blockIdx.x] = prob_eps > 0.f ? -logf(p + prob_eps) : -(xt - row_max - logf(denom));
    }
    if (dlogits) {
        uint4* g = reinterpret_cast<uint4*>(dlogits + off);
        const float sc = inv * grad_scale;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = threadIdx.x + k * THREADS;
            if (i < nv) {
                const float2 a = unpack_h2(r[k].x), b = unpack_h2(r[k].y), c = unpack_h2(r[k].z), d = unpack_h2(r[k].w);
                float x[8] = {a.x * sc, a.y * sc, b.x * sc, b.y * sc, c.x * sc, c.y * sc, d.x * sc, d.y * sc};
                const int t = (ONE ? target : tgt) - i * 8;
                if (t >= 0 && t < 8) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j == t) x[j] -= grad_scale;
                }
                g[i] = pack8(x);
            }
        }
    }
}

template <int THREADS, int NV, int BLOCKS>
cudaError_t ce_rows_launch(const __nv_bfloat16* logits, const int* targets, __nv_bfloat16* dlogits, float* losses, int rows, int V,
                           long long ld, float grad_scale, float prob_eps, cudaStream_t st) {
    return cme_launch_dependent(cross_entropy_bf16_reg_kernel<THREADS, NV, BLOCKS>, dim3(rows), dim3(THREADS), 0, st, logits, targets,
                                dlogits, losses, V, ld, grad_scale, prob_eps);
}
// By the length of the row: registers for it with the fewest idle threads, of the widths that a sweep of 28 forms left (rows x V, us
// with one form for all before, and now): 8192 x 2048 100 -> 14.5, 8192 x 4096 113 -> 25, 8192 x 8192 130 -> 43, 4096 x 12288
// 74 -> 35, 4096 x 20480 91 -> 56, 4096 x 28672 109 -> 83, 600 x 8192 13 -> 6.0.  Copy bandwidth would take 10, 20, 40, 30, 50, 71, 3.
constexpr int CER_MAX_V = 512 * 13 * 8;
cudaError_t ce_rows(const __nv_bfloat16* logits, const int* targets, __nv_bfloat16* dlogits, float* losses, int rows, int V,
                    long long ld, float grad_scale, float prob_eps, cudaStream_t st) {
#define CME_CER(T, NV, B) if (V <= T * NV * 8) return ce_rows_launch<T, NV, B>(logits, targets, dlogits, losses, rows, V, ld, grad_scale, prob_eps, st)
    CME_CER(64, 4, 16);
    CME_CER(128, 4, 12);
    CME_CER(128, 6, 10);
    CME_CER(128, 8, 10);
    CME_CER(256, 6, 5);
    CME_CER(256, 8, 5);
    CME_CER(256, 10, 4);
    CME_CER(256, 13, 4);
    CME_CER(512, 8, 2);
    CME_CER(512, 10, 2);
    CME_CER(512, 13, 2);
#undef CME_CER
    return cudaErrorInvalidValue;
}
// Rows of at most WARPS * 32 * NV elements of any length, alignment and type, held in registers from their one read to
// their one write: WARPS == 1 gives every warp a row (8 rows per block), else a block of WARPS warps shares one.
// Character vocabularies are a few elements per lane: what bounds them is the latency of one row's chain of load,
// maximum, exponentials, sum, store, so it is the number of rows in flight that counts -- a block per row leaves 191 of
// 256 threads of a 65-symbol row without work and pays four block-wide synchronisations per row.
// 16384 rows of 65 bf16 logits: 5.3 us, 27.8 us with a block per row.
// One exponential per element (the general kernel evaluates it once for the sum and again for the gradient).
template <typename T, int NV, int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 256 : WARPS * 32)
cross_entropy_short_kernel(const T* __restrict__ logits, const int* __restrict__ targets, T* dlogits,
                           float* __restrict__ losses, int rows, int V, long long ld, float grad_scale, float prob_eps) {
    __shared__ float scratch[32];
    constexpr int STEP = WARPS * 32;
    pdl_wait();
    const int lane = threadIdx.x % STEP;
    const int r = WARPS == 1 ? (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5) : (int)blockIdx.x;
    if (r >= rows) return;
    const T* row = logits + (long long)r * ld;
    int tgt = targets[r];
    tgt = tgt < 0 ? 0 : (tgt >= V ? V - 1 : tgt);
    float x[NV], m = -INFINITY;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = lane + i * STEP;
        x[i] = c < V ? to_f32<T>(row[c]) : -INFINITY;
        m = fmaxf(m, x[i]);
    }
    const float xt = to_f32<T>(row[tgt]);              // read before anyone overwrites it
    m = WARPS == 1 ? warp_max(m) : block_max(m, scratch);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (lane + i * STEP < V) { x[i] = __expf(x[i] - m); s += x[i]; }
    }
    s = WARPS == 1 ? warp_sum(s) : block_sum(s, scratch);
    const float inv = 1.f / (s + prob_eps);
    if (lane == 0) losses[r] = prob_eps > 0.f ? -logf(__expf(xt - m) * inv + prob_eps) : -(xt - m - logf(s));
    if (WARPS == 1) __syncwarp(); else __syncthreads();
    if (dlogits) {
        T* g = dlogits + (long long)r * ld;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = lane + i * STEP;
            if (c < V) g[c] = from_f32<T>((c == tgt ? x[i] * inv - 1.f : x[i] * inv) * grad_scale);
        }
    }
}

template <typename T, int NV, int WARPS>
cudaError_t ce_short_launch(const void* logits, const int* targets, void* dlogits, float* losses, int rows, int V,
                            long long ld, float grad_scale, float prob_eps, cudaStream_t st) {
    return cme_launch_dependent(cross_entropy_short_kernel<T, NV, WARPS>, dim3(WARPS == 1 ? cme_cdiv(rows, 8) : rows),
                                dim3(WARPS == 1 ? 256 : WARPS * 32), 0,
                                st, (const T*)logits, targets, (T*)dlogits, losses, rows, V, ld, grad_scale, prob_eps);
}
// One to four warps per row, so that a lane has at most 32 registers of it, and of these as few as the row fills: a second half of
// empty registers costs as much as a full one, eight warps wait for one another longer than four, and two of 12 or 16 registers are
// faster than one of 24 or 32 (bf16, us with 32 registers up to 1024, then 8 warps of 8 or 16, and so: 16384 x 620 22.9 and 14.6,
// x 1001 25.8 and 23.0, x 1250 51.8 and 26.8, x 2001 54.6 and 38.5, x 2500 85.3 and 50.3, 8192 x 4001 47.8 and 39.0; fp32 alike).
// Up to two rows per SM nothing overlaps a row's chain, and eight warps have the shorter one (128 x 2001 3.44 us, 4.02 with two
// warps; 296 x 4001 4.43 and 4.77; 400 x 1501 4.1 and 4.3, x 2500 4.7 and 4.1, 600 x 3001 6.3 and 5.3).
constexpr int CES_MAX_V = 4096;
template <typename T>
cudaError_t ce_short(const void* logits, const int* targets, void* dlogits, float* losses, int rows, int V, long long ld,
                     float grad_scale, float prob_eps, int sms, cudaStream_t st) {
#define CME_CES(NV, WARPS) ce_short_launch<T, NV, WARPS>(logits, targets, dlogits, losses, rows, V, ld, grad_scale, prob_eps, st)
    if (V <= 64) return CME_CES(2, 1);
    if (V <= 128) return CME_CES(4, 1);
    if (V <= 256) return CME_CES(8, 1);
    if (V <= 512) return CME_CES(16, 1);
    if (V <= 640) return CME_CES(20, 1);
    if (V <= 768) return CME_CES(12, 2);
    if (V <= 1024) return CME_CES(16, 2);
    if (rows <= 2 * sms) return V <= 2048 ? CME_CES(8, 8) : CME_CES(16, 8);
    if (V <= 1280) return CME_CES(20, 2);
    if (V <= 1536) return CME_CES(24, 2);
    if (V <= 2048) return CME_CES(32, 2);
    if (V <= 2560) return CME_CES(20, 4);
    if (V <= 3072) return CME_CES(24, 4);
    return CME_CES(32, 4);
#undef CME_CES
}

// out (+)= weight * sum(x[0..n)); single block, fixed order.  One block's time is its chain of loads, so each thread has
// four 16-byte loads in flight where x is aligned (16384 row losses: 2.3 us, 5.9 us with a 4-byte load per step).
__global__ void __launch_bounds__(1024) reduce_scalar_kernel(const float* __restrict__ x, int n, float weight, float* out,
                                                             int accumulate) {
    __shared__ float scratch[32];
    pdl_wait();
    float s = 0.f;
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4* v = reinterpret_cast<const float4*>(x);
        const int nv = n / 4, step = blockDim.x;
        done = nv * 4;
        for (int i = threadIdx.x; i < nv; i += 4 * step) {
            float4 u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) u[k] = i + k * step < nv ? v[i + k * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 4; ++k) s += (u[k].x + u[k].y) + (u[k].z + u[k].w);
        }
    }
    for (int i = done + threadIdx.x; i < n; i += blockDim.x) s += x[i];
    s = block_sum(s, scratch);
    if (threadIdx.x == 0) *out = (accumulate ? *out : 0.f) + s * weight;
}

constexpr int NORM_PARTIALS = 1024;

template <typename T>
__global__ void __launch_bounds__(256) normsq_partial_kernel(const T* __restrict__ g, long long n, float* partial, int* count) {
    __shared__ float scratch[32];
    if (count && blockIdx.x == 0 && threadIdx.x == 0) *count += 1;
    float s = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = to_f32<T>(g[i]);
        s += v * v;
    }
    s = block_sum(s, scratch);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Same over whole 16-byte words, four in flight per thread: with a 2-byte load per iteration the sum of 124 M bf16
// gradients waits for its loads (249 MB: 58 us, 86 us so).
template <typename T>
__global__ void __launch_bounds__(256) normsq_partial_vec_kernel(const T* __restrict__ grads, long long n, float* partial, int* count) {
    __shared__ float scratch[32];
    constexpr int W = 16 / sizeof(T);
    const uint4* g = reinterpret_cast<const uint4*>(grads);
    const long long nvec = n / W;
    pdl_wait();
    if (count && blockIdx.x == 0 && threadIdx.x == 0) *count += 1;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const long long step = (long long)gridDim.x * blockDim.x;
    auto add = [&](const uint4& u, float& t) {
        float x[W];
        if constexpr (sizeof(T) == 2) unpack8(u, x);
        else { x[0] = __uint_as_float(u.x); x[1] = __uint_as_float(u.y); x[2] = __uint_as_float(u.z); x[3] = __uint_as_float(u.w); }
#pragma unroll
        for (int j = 0; j < W; ++j) t = fmaf(x[j], x[j], t);
    };
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * step < nvec; i += 4 * step) {
        uint4 u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = g[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; ++k) add(u[k], s[k]);
    }
    for (; i < nvec; i += step) add(g[i], s[0]);
    if (blockIdx.x == 0 && threadIdx.x < (int)(n - nvec * W)) {          // what is left of the last word
        const float v = to_f32<T>(grads[nvec * W + threadIdx.x]);
        s[1] = fmaf(v, v, s[1]);
    }
    const float t = block_sum((s[0] + s[1]) + (s[2] + s[3]), scratch);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

__global__ void step_inc_kernel(int* step) {
    pdl_wait();
    *step += 1;
}

struct AdamArgs {
    float* master; __nv_bfloat16* compute; const void* grads; float* m; float* v;
    long long n;
    const int* step; const float* lr; const float* normsq;
    float beta1, beta2, eps, weight_decay, grad_scale, clip_norm;
    const long long* nodecay; int n_nodecay;      // sorted [start, end) pairs exempt from weight decay
    int n_norm; float* norm_out;                  // > 1: `normsq` holds that many partial sums; their total goes to norm_out
};

// The gradient's scale.  Partial sums of the squared norm are added by every block (1024 of them: a few loads from L2 and two
// barriers, against a kernel of its own in front of this one).
// `sq`: the first of them, or the squared norm itself.
__device__ __forceinline__ float adam_grad_scale(const AdamArgs& a, float sq, float* scratch) {
    if (!a.normsq || a.clip_norm <= 0.f) return a.grad_scale;
    if (a.n_norm > 1) {
        sq = 0.f;
        for (int i = threadIdx.x; i < a.n_norm; i += blockDim.x) sq += a.normsq[i];
        sq = block_sum(sq, scratch);
        if (a.norm_out && blockIdx.x == 0 && threadIdx.x == 0) *a.norm_out = sq;
    }
    const float norm = sqrtf(sq) * a.grad_scale;
    return norm > a.clip_norm ? a.grad_scale * (a.clip_norm / norm) : a.grad_scale;
}

// The first of `n` sorted no-decay ranges, from `lo` on, with end > i (n if there is none).
__device__ __forceinline__ int adam_range_at(const long long* ranges, int n, int lo, long long i) {
    int hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ranges[2 * mid + 1] > i) hi = mid; else lo = mid + 1;
    }
    return lo;
}
__device__ __forceinline__ bool adam_decays(const AdamArgs& a, long long i) {
    const int lo = adam_range_at(a.nodecay, a.n_nodecay, 0, i);
    return !(lo < a.n_nodecay && a.nodecay[2 * lo] <= i);
}

// m <- beta1 m + (1 - beta1) g,  v <- beta2 v + (1 - beta2) g^2.  The products with m and v, the larger terms, enter the
// sums unrounded; left to the compiler, one kernel rounded beta2 v first and its v was 3.8e-8 off 64 bits instead of 2.8e-8.
__device__ __forceinline__ void adam_moments(const AdamArgs& a, float g, float& m, float& v) {
    m = fmaf(a.beta1, m, (1.f - a.beta1) * g);
    v = fmaf(a.beta2, v, (1.f - a.beta2) * g * g);
}

template <typename TG>
__global__ void __launch_bounds__(256) adam_kernel(const AdamArgs a) {
    pdl_wait();
    const int t = *a.step;
    const float lr = *a.lr;
    const float bc1 = 1.f - powf(a.beta1, (float)t), bc2 = 1.f - powf(a.beta2, (float)t);
    __shared__ float scratch[32];
    const float gs = adam_grad_scale(a, a.normsq ? *a.normsq : 0.f, scratch);
    const TG* grads = reinterpret_cast<const TG*>(a.grads);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (long long)gridDim.x * blockDim.x) {
        const float g = to_f32<TG>(grads[i]) * gs;
        float mi = a.m[i], vi = a.v[i];
        adam_moments(a, g, mi, vi);
        a.m[i] = mi;
        a.v[i] = vi;
        float p = a.master[i];
        if (a.weight_decay > 0.f && adam_decays(a, i)) p *= 1.f - lr * a.weight_decay;
        p -= lr * (mi / bc1) / (sqrtf(vi / bc2) + a.eps);
        a.master[i] = p;
        if (a.compute) a.compute[i] = __float2bfloat16_rn(p);
    }
}


constexpr int ADAM_BLOCKS_PER_SM = 5;
constexpr int ADAM_LIST = 512;             // ranges that a block keeps in shared memory (8 KB); longer lists are read in place

// Four elements per thread and round (128-bit accesses on the fp32 state).  Requires 16-byte aligned arenas; the last n % 4
// elements and groups in which a no-decay range begins or ends are decided element by element.  RANGES: there is weight
// decay and a list of ranges.
// Bound by memory: 124 M elements with bf16 gradients, 3.49 GB: 519 us (6.7 TB/s; 523 with 150 ranges), 535 with the norm's partial sums
// to add up.  A block takes `rounds` x 256 consecutive groups, so that the blocks that run together, in their order, work on one window of
// each array; as 2368 blocks that stride through all of it the same loop took 558 us.  Five blocks an SM: four 536 us, six 538 (spills
// aside, more rows of DRAM open at once).
template <typename TG, bool RANGES>
__global__ void __launch_bounds__(256, ADAM_BLOCKS_PER_SM) adam_vec4_kernel(const AdamArgs a, const int rounds) {
    pdl_wait();
    const long long nv = a.n >> 2;
    const long long first = (long long)blockIdx.x * rounds * 256 + threadIdx.x;
    const long long end = first + (long long)rounds * 256 < nv ? first + (long long)rounds * 256 : nv;
    float4 m4, v4, p4;
    float g[4];
    auto load = [&](long long i) {
        const long long e = i << 2;
        m4 = *reinterpret_cast<const float4*>(a.m + e);
        v4 = *reinterpret_cast<const float4*>(a.v + e);
        p4 = *reinterpret_cast<const float4*>(a.master + e);
        if constexpr (sizeof(TG) == 2) {
            const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(a.grads) + e);
            float2 lo = bf2_to_f2(u.x), hi = bf2_to_f2(u.y);
            g[0] = lo.x; g[1] = lo.y; g[2] = hi.x; g[3] = hi.y;
        } else {
            const float4 u = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.grads) + e);
            g[0] = u.x; g[1] = u.y; g[2] = u.z; g[3] = u.w;
        }
    };
    // every load of the set-up is in flight before the first result is used, and with them those of the first round
    const int t = *a.step;
    const float lr = *a.lr;
    const float sq = a.normsq ? *a.normsq : 0.f;
    if (first < end) load(first);
    __shared__ float scratch[32], setup[2];
    if (threadIdx.x < 2) setup[threadIdx.x] = 1.f / (1.f - powf(threadIdx.x ? a.beta2 : a.beta1, (float)t));
    // The no-decay range at or after the element at hand stays in registers; where it is over, the next one is searched for
    // in a copy of the list in shared memory.  From global memory that is a chain of dependent loads: all of the list where
    // it was walked (150 ranges: 1 M elements 28 us, 16 M 113 us), seven loads a group where it was bisected (8.4 and 82 us).
    __shared__ long long list[RANGES ? 2 * ADAM_LIST : 1];
    const bool copied = a.n_nodecay <= ADAM_LIST;
    if (RANGES && copied)
        for (int k = threadIdx.x; k < 2 * a.n_nodecay; k += blockDim.x) list[k] = a.nodecay[k];
    __syncthreads();
    const float gs = adam_grad_scale(a, sq, scratch);
    const long long* ranges = copied ? list : a.nodecay;
    const float ibc1 = setup[0], ibc2 = setup[1];
    const float keep = a.weight_decay > 0.f ? 1.f - lr * a.weight_decay : 1.f;
    int seg = 0;
    long long seg_start = 0, seg_end = 0;
    for (long long i = first; i < end; i += 256) {
        const long long e = i << 2;
        if (i != first) load(i);
        float decay[4] = {keep, keep, keep, keep};
        if (RANGES) {
            auto advance = [&](long long to) {
                if (seg_end > to) return;
                seg = adam_range_at(ranges, a.n_nodecay, seg, to);
                seg_start = seg < a.n_nodecay ? ranges[2 * seg] : 0x7fffffffffffffffll;
                seg_end = seg < a.n_nodecay ? ranges[2 * seg + 1] : 0x7fffffffffffffffll;
            };
            advance(e);
            if (seg_start < e + 4) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    advance(e + j);                // (a range may end inside the group and another begin)
                    if (seg_start <= e + j) decay[j] = 1.f;
                }
            }
        }
        float* mp = &m4.x; float* vp = &v4.x; float* pp = &p4.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float gj = g[j] * gs;
            adam_moments(a, gj, mp[j], vp[j]);
            pp[j] = pp[j] * decay[j] - lr * (mp[j] * ibc1) / (sqrtf(vp[j] * ibc2) + a.eps);
        }
        *reinterpret_cast<float4*>(a.m + e) = m4;
        *reinterpret_cast<float4*>(a.v + e) = v4;
        *reinterpret_cast<float4*>(a.master + e) = p4;
        if (a.compute)
            *reinterpret_cast<uint2*>(a.compute + e) = make_uint2(f2_to_bf2(p4.x, p4.y), f2_to_bf2(p4.z, p4.w));
    }
    if (blockIdx.x == 0 && threadIdx.x < (int)(a.n & 3)) {
        const long long e = (nv << 2) + threadIdx.x;
        const float gj = to_f32<TG>(reinterpret_cast<const TG*>(a.grads)[e]) * gs;
        float mi = a.m[e], vi = a.v[e];
        adam_moments(a, gj, mi, vi);
        const float decay = RANGES && !adam_decays(a, e) ? 1.f : keep;
        const float p = a.master[e] * decay - lr * (mi * ibc1) / (sqrtf(vi * ibc2) + a.eps);
        a.m[e] = mi;
        a.v[e] = vi;
        a.master[e] = p;
        if (a.compute) a.compute[e] = __float2bfloat16_rn(p);
    }
}

}  // namespace

// *loss_out (+)= loss_weight * mean(losses).
CME_API int cme_loss_mean(const float* losses, int rows, float loss_weight, float* loss_out, int accumulate_loss, void* stream) {
    CME_REQUIRE(rows > 0, CME_ERR_SHAPE, "loss_mean: empty input");
    CME_CUDA(cme_launch_dependent(reduce_scalar_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, losses, rows,
                                  loss_weight / (float)rows, loss_out, accumulate_loss));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// Per-row loss and gradient, then *loss_out (+)= loss_weight * mean(losses).
// prob_eps > 0 selects the reference's form  -log(p + eps), p = e / (sum + eps);  0 the exact log-softmax.
CME_API int cme_cross_entropy(int dtype, const void* logits, const int* targets, void* dlogits, float* losses,
                              float* loss_out, int rows, int V, long long ld, float grad_scale, float prob_eps,
                              float loss_weight, int accumulate_loss, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && V > 0, CME_ERR_SHAPE, "cross_entropy: empty input");
    const bool vec = dtype == CME_BF16 && V % 8 == 0 && ld % 8 == 0 && V >= 2048 &&
                     (reinterpret_cast<uintptr_t>(logits) & 15) == 0 &&
                     (!dlogits || (reinterpret_cast<uintptr_t>(dlogits) & 15) == 0);
    if (vec && V <= CER_MAX_V) {
        CME_CUDA(ce_rows((const __nv_bfloat16*)logits, targets, (__nv_bfloat16*)dlogits, losses, rows, V, ld, grad_scale, prob_eps, st));
    } else if (vec) {
        const size_t row_bytes = (size_t)V * 2;
        const int cache = row_bytes <= 110 * 1024;          // two blocks per SM still fit
        static bool attr = false;
        if (!attr) {
            CME_CUDA(cudaFuncSetAttribute(cross_entropy_bf16_vec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          110 * 1024));
            attr = true;
        }
        cross_entropy_bf16_vec_kernel<<<rows, CEV_THREADS, cache ? row_bytes : 0, st>>>(
            (const __nv_bfloat16*)logits, targets, (__nv_bfloat16*)dlogits, losses, V, ld, grad_scale, prob_eps, cache);
    } else if (V <= CES_MAX_V) {
        int sms = 0;
        if (V > 1024) {
            const int rc = cme_num_sms(&sms);
            if (rc) return rc;
        }
        CME_CUDA(dtype == CME_BF16 ? ce_short<__nv_bfloat16>(logits, targets, dlogits, losses, rows, V, ld, grad_scale, prob_eps, sms, st)
                                   : ce_short<float>(logits, targets, dlogits, losses, rows, V, ld, grad_scale, prob_eps, sms, st));
    } else if (dtype == CME_BF16)
        cross_entropy_kernel<__nv_bfloat16><<<rows, CE_THREADS, 0, st>>>((const __nv_bfloat16*)logits, targets,
                                                                         (__nv_bfloat16*)dlogits, losses, V, ld,
                                                                         grad_scale, prob_eps);
    else
        cross_entropy_kernel<float><<<rows, CE_THREADS, 0, st>>>((const float*)logits, targets, (float*)dlogits, losses,
                                                                 V, ld, grad_scale, prob_eps);
    CME_LAUNCH_CHECK();
    return loss_out ? cme_loss_mean(losses, rows, loss_weight, loss_out, accumulate_loss, stream) : CME_OK;
}

// partial[0 .. 1024) = sums whose total is sum(g^2) over n elements; *step (or null) is incremented on the way.
CME_API int cme_grad_normsq_partials(int dtype, const void* g, long long n, float* partial, int* step, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const bool bf = dtype == CME_BF16;
    if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
        CME_CUDA(bf ? cme_launch_dependent(normsq_partial_vec_kernel<__nv_bfloat16>, dim3(NORM_PARTIALS), dim3(256), 0, st,
                                           (const __nv_bfloat16*)g, n, partial, step)
                    : cme_launch_dependent(normsq_partial_vec_kernel<float>, dim3(NORM_PARTIALS), dim3(256), 0, st, (const float*)g, n,
                                           partial, step));
    } else if (bf) {
        normsq_partial_kernel<__nv_bfloat16><<<NORM_PARTIALS, 256, 0, st>>>((const __nv_bfloat16*)g, n, partial, step);
    } else {
        normsq_partial_kernel<float><<<NORM_PARTIALS, 256, 0, st>>>((const float*)g, n, partial, step);
    }
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// *out = sum(g^2) over n elements; `partial` holds 1024 floats.
CME_API int cme_grad_normsq(int dtype, const void* g, long long n, float* partial, float* out, void* stream) {
    const int rc = cme_grad_normsq_partials(dtype, g, n, partial, nullptr, stream);
    if (rc) return rc;
    CME_CUDA(cme_launch_dependent(reduce_scalar_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, (const float*)partial,
                                  NORM_PARTIALS, 1.f, out, 0));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// Early loss read-back: bump the sequence number, write the loss and then the sequence number straight into
// pinned, device-mapped host memory.  A host thread that sees the new sequence number also sees the loss.
__global__ void publish_loss_kernel(const float* loss, int* seq, volatile float* host_loss, volatile int* host_seq) {
    const int s = *seq + 1;
    *seq = s;
    *host_loss = *loss;
    __threadfence_system();
    *host_seq = s;
    __threadfence_system();      // push the number out now: inside a CUDA graph nothing else flushes it before the end
}

// Device-side address of a pinned host allocation (once per buffer, outside stream capture).
CME_API int cme_host_device_ptr(void* host, void** dev) {
    CME_CUDA(cudaHostGetDevicePointer(dev, host, 0));
    return CME_OK;
}

CME_API int cme_publish_loss(const float* loss, int* seq, void* host_loss_dev, void* host_seq_dev, void* stream) {
    publish_loss_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(loss, seq, static_cast<volatile float*>(host_loss_dev),
                                                           static_cast<volatile int*>(host_seq_dev));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_step_inc(int* step, void* stream) {
    CME_CUDA(cme_launch_dependent(step_inc_kernel, dim3(1), dim3(1), 0, (cudaStream_t)stream, step));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// Adam / AdamW over [0, n).  `step` (already incremented), `lr` and `normsq` live in device memory.
// g_eff = grad * grad_scale * min(1, clip_norm / (sqrt(normsq) * grad_scale)); decoupled weight decay
// except inside the `nodecay` ranges; writes the fp32 master and, if given, its bf16 copy.
// n_norm > 1: `normsq` holds that many partial sums (cme_grad_normsq_partials: 1024); their total goes to norm_out (or null).
CME_API int cme_adam_partials(int grad_dtype, float* master, void* compute_bf16, const void* grads, float* m, float* v,
                              long long n, const int* step, const float* lr, const float* normsq, float beta1, float beta2,
                              float eps, float weight_decay, float grad_scale, float clip_norm, const long long* nodecay,
                              int n_nodecay, int n_norm, float* norm_out, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 0) return CME_OK;
    AdamArgs a{master, (__nv_bfloat16*)compute_bf16, grads, m, v, n, step, lr, normsq, beta1, beta2, eps,
               weight_decay, grad_scale, clip_norm, nodecay, n_nodecay, n_norm, norm_out};
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    auto al = [](const void* p, int b) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & (b - 1)) == 0; };
    bool vec = n >= 4 && al(master, 16) && al(m, 16) && al(v, 16) && al(compute_bf16, 8) &&
               al(grads, grad_dtype == CME_BF16 ? 8 : 16);
    if (vec) {
        // Rounds per block: its set-up (three scalars, two powers, the list of ranges, the norm's partial sums) takes as long as a round,
        // so the fewest that let all blocks run at once, five per SM, up to four; beyond that a second wave costs as much as it is full,
        // and three rounds are within 3 % of the best everywhere.  us with 1 / 2 / 3 / 4 / 8 rounds, bf16 gradients, no ranges or clipping:
        // 0.46 M elements 2.9 / 3.4 / 4.0 / 4.4 / 6.9, 1 M 4.8 / 4.6 / 5.0 / 5.3 / 7.1, 1.8 M 7.0 / 7.0 / 6.4 / 6.6 / 8.4, 2.5 M from memory
        // 10.3 / 9.6 / 10.3 / 9.4 / 11.8, 4 M 18.9 / 19.0 / 19.5 / 21.0 / 20.4, with ranges and the norm's partial sums 26.5 / 24.2 / 23.6 /
        // 25.6 / 23.3; 40 M with both 223 / 188 / 179 / 178 / 179.
        const long long groups = (n / 4 + 255) / 256;
        int sms = 0;
        const int rc = cme_num_sms(&sms);
        if (rc) return rc;
        const long long fit = (groups + ADAM_BLOCKS_PER_SM * sms - 1) / (ADAM_BLOCKS_PER_SM * sms);
        const int rounds = fit <= 4 ? (int)fit : 3;
        blocks = (groups + rounds - 1) / rounds;
        const bool ranges = weight_decay > 0.f && n_nodecay > 0;
        auto kernel = grad_dtype != CME_BF16 ? (ranges ? adam_vec4_kernel<float, true> : adam_vec4_kernel<float, false>)
                      : ranges               ? adam_vec4_kernel<__nv_bfloat16, true>
                                             : adam_vec4_kernel<__nv_bfloat16, false>;
        CME_CUDA(cme_launch_dependent(kernel, dim3((int)blocks), dim3(256), 0, st, a, rounds));
    } else {
        CME_CUDA(cme_launch_dependent(grad_dtype == CME_BF16 ? adam_kernel<__nv_bfloat16> : adam_kernel<float>,
                                      dim3((int)blocks), dim3(256), 0, st, a));
    }
    CME_LAUNCH_CHECK();
    return CME_OK;
}

CME_API int cme_adam(int grad_dtype, float* master, void* compute_bf16, const void* grads, float* m, float* v,
                     long long n, const int* step, const float* lr, const float* normsq, float beta1, float beta2,
                     float eps, float weight_decay, float grad_scale, float clip_norm, const long long* nodecay,
                     int n_nodecay, void* stream) {
    return cme_adam_partials(grad_dtype, master, compute_bf16, grads, m, v, n, step, lr, normsq, beta1, beta2, eps, weight_decay,
                             grad_scale, clip_norm, nodecay, n_nodecay, 1, nullptr, stream);
}
