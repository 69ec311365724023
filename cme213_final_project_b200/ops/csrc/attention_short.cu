// Fused attention for sequences of at most 64 tokens (the parity models, tiny-gpt's length), bf16, head size a multiple
// of 8 up to 128: one block per (batch, head) holds the whole problem in shared memory, one launch per direction.
//
// What bounds it is latency: 32 x 4 heads x 64 tokens x head size 128 is 0.94 GFLOP in both directions, 0.6 us of the
// chip, on 128 blocks.  So the products are warp-level mma.sync on fragments that stay in registers (scores to
// probabilities to the next product's operand without a trip through memory): a tcgen05 product would be a 128-row
// tile half empty, and each of the chain's steps would add a tensor-memory round trip and a barrier.
// Precision as in the paths it stands in for: scores, softmax, delta and all sums fp32, P and dS rounded to bf16 once.
// 32 x 4 heads x 64 tokens: head size 128 in 5.3 us forward and 7.5 us backward, where the batched products take 23.6 us in
// three launches and 44 us in seven; head size 32 5.7 and 6.7 us inside a training step.
#include "attention.h"

namespace {

constexpr int TS = 64;                     // tokens held by a block
constexpr int PP = TS + 8;                 // pitch of P and dS (elements): 8 rows start on 8 different 16-byte banks
constexpr int FWD_WARPS = 4, BWD_WARPS = 8;
template <int D> struct Tile { static constexpr int P = D + 8, ELEMS = TS * (D + 8); };

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s32(p)));
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s32(p)));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Operand addresses of a 16 x 16 block whose top left element is (r, c) of a tile with pitch P:
// A (row-major) or, transposed on load, A from [k][m]; B from [n][k], or, transposed on load, from [k][n].
__device__ __forceinline__ const __nv_bfloat16* at_a(const __nv_bfloat16* t, int P, int r, int c) {
    const int l = threadIdx.x & 31;
    return t + (r + (l & 15)) * P + c + (l >> 4) * 8;
}
__device__ __forceinline__ const __nv_bfloat16* at_b(const __nv_bfloat16* t, int P, int r, int c) {
    const int l = threadIdx.x & 31;
    return t + (r + (l & 7) + (l >> 4) * 8) * P + c + ((l >> 3) & 1) * 8;
}

// All rows of a [T, HD] operand into a [64][D] tile by asynchronous 16-byte copies, zeros beyond T and HD.
template <int D, int NT>
__device__ __forceinline__ void copy_tile(__nv_bfloat16* dst, const void* src, long long base, long long st, int T, int HD) {
#pragma unroll
    for (int k = 0; k < TS * (D / 8) / NT; ++k) {
        const int i = threadIdx.x + k * NT, r = i / (D / 8), c = (i % (D / 8)) * 8;
        const bool in = r < T && c < HD;
        const __nv_bfloat16* p = (const __nv_bfloat16*)src + base + (in ? (long long)r * st + c : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s32(dst + r * Tile<D>::P + c)), "l"(p),
                     "r"(in ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void copy_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A finished [64][D] tile to its rows in global memory, 16 bytes per thread.
template <int D, int NT>
__device__ __forceinline__ void store_tile(void* dst, const __nv_bfloat16* t, long long base, long long st, int T, int HD) {
#pragma unroll
    for (int k = 0; k < TS * (D / 8) / NT; ++k) {
        const int i = threadIdx.x + k * NT, r = i / (D / 8), c = (i % (D / 8)) * 8;
        if (r < T && c < HD)
            *reinterpret_cast<uint4*>((__nv_bfloat16*)dst + base + (long long)r * st + c) =
                *reinterpret_cast<const uint4*>(t + r * Tile<D>::P + c);
    }
}

__device__ __forceinline__ long long base_in(const CmeAttn& a, int bh) {
    return (long long)(bh / a.nh) * a.sb + (long long)(bh % a.nh) * a.sh;
}
__device__ __forceinline__ long long base_out(const CmeAttn& a, int bh) {
    return (long long)(bh / a.nh) * a.osb + (long long)(bh % a.nh) * a.osh;
}

// A warp owns 16 query rows; lane l holds columns 2 (l % 4), + 1 of each 8-column block of rows l / 4 and l / 4 + 8.
template <int D>
__global__ void __launch_bounds__(FWD_WARPS * 32) attn_short_fwd_kernel(const CmeAttn a, const bool normalise) {
    extern __shared__ __align__(16) __nv_bfloat16 smem[];
    constexpr int P = Tile<D>::P, NT = FWD_WARPS * 32;
    __nv_bfloat16* sQ = smem;
    __nv_bfloat16* sK = sQ + Tile<D>::ELEMS;
    __nv_bfloat16* sV = sK + Tile<D>::ELEMS;
    pdl_wait();
    const int bh = blockIdx.x, lane = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * 16;
    const long long base = base_in(a, bh);
    copy_tile<D, NT>(sQ, a.q, base, a.st, a.T, a.HD);
    copy_tile<D, NT>(sK, a.k, base, a.st, a.T, a.HD);
    copy_group();
    copy_tile<D, NT>(sV, a.v, base, a.st, a.T, a.HD);
    copy_group();
    copy_wait<1>();
    __syncthreads();
    float s[8][4] = {};
#pragma unroll
    for (int k = 0; k < D; k += 16) {
        uint32_t q[4];
        ldsm(q, at_a(sQ, P, r0, k));
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            uint32_t b[4];
            ldsm(b, at_b(sK, P, 16 * n, k));
            mma(s[2 * n], q, b[0], b[1]);
            mma(s[2 * n + 1], q, b[2], b[3]);
        }
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = r0 + (lane >> 2) + 8 * (e >> 1), col = 8 * n + 2 * (lane & 3) + (e & 1);
            s[n][e] = col < a.T && (!a.causal || col <= row) ? s[n][e] * a.scale : -INFINITY;
            m[e >> 1] = fmaxf(m[e >> 1], s[n][e]);
        }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 1));
        m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 2));
    }
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s[n][e] = m[e >> 1] == -INFINITY ? 0.f : __expf(s[n][e] - m[e >> 1]);
            l[e >> 1] += s[n][e];
        }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
    // row sums divide P (before it is rounded, like the batched products) or O (like the flash kernel)
    const float inv[2] = {l[0] > 0.f ? 1.f / l[0] : 0.f, l[1] > 0.f ? 1.f / l[1] : 0.f};
    if (normalise) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] *= inv[e >> 1];
    }
    copy_wait<0>();
    __syncthreads();
    float o[D / 8][4] = {};
#pragma unroll
    for (int k = 0; k < 4; ++k) {                  // 16 keys a step: the score layout is the A operand's layout
        const uint32_t p[4] = {f2_to_bf2(s[2 * k][0], s[2 * k][1]), f2_to_bf2(s[2 * k][2], s[2 * k][3]),
                               f2_to_bf2(s[2 * k + 1][0], s[2 * k + 1][1]), f2_to_bf2(s[2 * k + 1][2], s[2 * k + 1][3])};
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            uint32_t b[4];
            ldsm_t(b, at_a(sV, P, 16 * k, 16 * n));
            mma(o[2 * n], p, b[0], b[1]);
            mma(o[2 * n + 1], p, b[2], b[3]);
        }
    }
    const float on[2] = {normalise ? 1.f : inv[0], normalise ? 1.f : inv[1]};
#pragma unroll
    for (int n = 0; n < D / 8; ++n)                // the warp's own Q rows are free: stage O there
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<uint32_t*>(sQ + (r0 + (lane >> 2) + 8 * h) * P + 8 * n + 2 * (lane & 3)) =
                f2_to_bf2(o[n][2 * h] * on[h], o[n][2 * h + 1] * on[h]);
    if ((lane & 3) == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = r0 + (lane >> 2) + 8 * h;
            if (row < a.T) a.lse[(long long)bh * a.T + row] = m[h] + logf(l[h]);
        }
    }
    __syncthreads();
    store_tile<D, NT>(a.o, sQ, base_out(a, bh), a.ost, a.T, a.HD);
}

// Scores and dP in 16 x 32 blocks (4 row groups x 2 key halves), P and dS to shared memory, then each warp makes 16
// rows of half the columns of dQ, dV and dK.
template <int D>
__global__ void __launch_bounds__(BWD_WARPS * 32) attn_short_bwd_kernel(const CmeAttn a) {
    extern __shared__ __align__(16) __nv_bfloat16 smem[];
    constexpr int P = Tile<D>::P, NT = BWD_WARPS * 32;
    __nv_bfloat16* sQ = smem;
    __nv_bfloat16* sK = sQ + Tile<D>::ELEMS;
    __nv_bfloat16* sV = sK + Tile<D>::ELEMS;
    __nv_bfloat16* sO = sV + Tile<D>::ELEMS;       // dO
    __nv_bfloat16* sP = sO + Tile<D>::ELEMS;       // [64][PP]
    __nv_bfloat16* sS = sP + TS * PP;              // [64][PP]
    float* sDl = reinterpret_cast<float*>(sS + TS * PP);
    pdl_wait();
    const int bh = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = (warp & 3) * 16, half = warp >> 2;
    const long long base = base_in(a, bh), obase = base_out(a, bh);
    copy_tile<D, NT>(sQ, a.q, base, a.st, a.T, a.HD);
    copy_tile<D, NT>(sK, a.k, base, a.st, a.T, a.HD);
    copy_tile<D, NT>(sV, a.v, base, a.st, a.T, a.HD);
    copy_tile<D, NT>(sO, a.d_o, obase, a.ost, a.T, a.HD);
    copy_group();
    // delta = rowsum(dO * O): four threads per row, each a quarter of the row's 16-byte words, while the copies run
    {
        const int r = threadIdx.x >> 2;
        float d = 0.f;
        if (r < a.T) {
            const __nv_bfloat16* x = (const __nv_bfloat16*)a.d_o + obase + (long long)r * a.ost;
            const __nv_bfloat16* y = (const __nv_bfloat16*)a.o + obase + (long long)r * a.ost;
#pragma unroll
            for (int k = 0; k < D / 32; ++k) {
                const int c = ((threadIdx.x & 3) + 4 * k) * 8;
                if (c < a.HD) {
                    float u[8], w[8];
                    unpack8(*reinterpret_cast<const uint4*>(x + c), u);
                    unpack8(*reinterpret_cast<const uint4*>(y + c), w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) d = fmaf(u[j], w[j], d);
                }
            }
        }
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        if ((threadIdx.x & 3) == 0) sDl[r] = d;
    }
    float lse[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = r0 + (lane >> 2) + 8 * h;
        lse[h] = row < a.T ? a.lse[(long long)bh * a.T + row] : 0.f;
    }
    copy_wait<0>();
    __syncthreads();
    {
        float s[4][4] = {}, dp[4][4] = {};
#pragma unroll
        for (int k = 0; k < D; k += 16) {
            uint32_t q[4], d[4];
            ldsm(q, at_a(sQ, P, r0, k));
            ldsm(d, at_a(sO, P, r0, k));
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                uint32_t b[4];
                ldsm(b, at_b(sK, P, half * 32 + 16 * n, k));
                mma(s[2 * n], q, b[0], b[1]);
                mma(s[2 * n + 1], q, b[2], b[3]);
                ldsm(b, at_b(sV, P, half * 32 + 16 * n, k));
                mma(dp[2 * n], d, b[0], b[1]);
                mma(dp[2 * n + 1], d, b[2], b[3]);
            }
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = r0 + (lane >> 2) + 8 * h, col = half * 32 + 8 * n + 2 * (lane & 3);
                const float dl = sDl[row];
                float p[2], ds[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool ok = row < a.T && col + e < a.T && (!a.causal || col + e <= row);
                    p[e] = ok ? __expf(s[n][2 * h + e] * a.scale - lse[h]) : 0.f;
                    ds[e] = ok ? a.scale * p[e] * (dp[n][2 * h + e] - dl) : 0.f;
                }
                *reinterpret_cast<uint32_t*>(sP + row * PP + col) = f2_to_bf2(p[0], p[1]);
                *reinterpret_cast<uint32_t*>(sS + row * PP + col) = f2_to_bf2(ds[0], ds[1]);
            }
    }
    __syncthreads();
    constexpr int NB = D / 16;                     // 8-column blocks in half the columns
    float dq[NB][4] = {}, dv[NB][4] = {}, dk[NB][4] = {};
    const int n0 = half * (D / 2);
#pragma unroll
    for (int k = 0; k < TS; k += 16) {
        uint32_t pt[4], st[4], ds[4];
        {                                          // transposed: rows are keys r0 .., the sum runs over queries k ..
            uint32_t t[4];
            ldsm_t(t, at_a(sP, PP, k, r0));
            pt[0] = t[0]; pt[1] = t[2]; pt[2] = t[1]; pt[3] = t[3];
            ldsm_t(t, at_a(sS, PP, k, r0));
            st[0] = t[0]; st[1] = t[2]; st[2] = t[1]; st[3] = t[3];
        }
        ldsm(ds, at_a(sS, PP, r0, k));
#pragma unroll
        for (int n = 0; n < NB / 2; ++n) {
            uint32_t b[4];
            ldsm_t(b, at_a(sO, P, k, n0 + 16 * n));
            mma(dv[2 * n], pt, b[0], b[1]);
            mma(dv[2 * n + 1], pt, b[2], b[3]);
            ldsm_t(b, at_a(sQ, P, k, n0 + 16 * n));
            mma(dk[2 * n], st, b[0], b[1]);
            mma(dk[2 * n + 1], st, b[2], b[3]);
            ldsm_t(b, at_a(sK, P, k, n0 + 16 * n));
            mma(dq[2 * n], ds, b[0], b[1]);
            mma(dq[2 * n + 1], ds, b[2], b[3]);
        }
    }
    __syncthreads();                               // every operand has been read: the results take their places
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int at = (r0 + (lane >> 2) + 8 * h) * P + n0 + 8 * n + 2 * (lane & 3);
            *reinterpret_cast<uint32_t*>(sQ + at) = f2_to_bf2(dq[n][2 * h], dq[n][2 * h + 1]);
            *reinterpret_cast<uint32_t*>(sK + at) = f2_to_bf2(dk[n][2 * h], dk[n][2 * h + 1]);
            *reinterpret_cast<uint32_t*>(sV + at) = f2_to_bf2(dv[n][2 * h], dv[n][2 * h + 1]);
        }
    __syncthreads();
    store_tile<D, NT>(a.dq, sQ, base, a.st, a.T, a.HD);
    store_tile<D, NT>(a.dk, sK, base, a.st, a.T, a.HD);
    store_tile<D, NT>(a.dv, sV, base, a.st, a.T, a.HD);
}

template <int D, bool BWD> int launch(const CmeAttn* a, cudaStream_t st) {
    constexpr int smem = BWD ? 4 * Tile<D>::ELEMS * 2 + 2 * TS * PP * 2 + TS * 4 : 3 * Tile<D>::ELEMS * 2;
    auto run = [&](auto k, int warps, auto... more) -> int {
        if (smem > 48 * 1024) CME_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        CME_CUDA(cme_launch_dependent(k, dim3(a->nb * a->nh), dim3(warps * 32), (size_t)smem, st, *a, more...));
        CME_LAUNCH_CHECK();
        return CME_OK;
    };
    if constexpr (BWD) return run(attn_short_bwd_kernel<D>, BWD_WARPS);
    else return run(attn_short_fwd_kernel<D>, FWD_WARPS, attention_tc_supported(a) == 0);
}

}  // namespace

int attention_short_supported(const CmeAttn* a, int bwd) {
    if (a->dtype != CME_BF16 || a->T > TS || a->HD % 8 || a->HD > 128) return 0;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al16(a->q) || !al16(a->k) || !al16(a->v) || !al16(a->o)) return 0;
    if (bwd && (!al16(a->d_o) || !al16(a->dq) || !al16(a->dk) || !al16(a->dv))) return 0;
    return !((a->st | a->sh | a->sb | a->ost | a->osh | a->osb) & 7);
}
int attention_short_fwd(const CmeAttn* a, cudaStream_t st) {
    CME_REQUIRE(a->lse != nullptr, CME_ERR_SHAPE, "attention: lse buffer is required");
    return a->HD <= 32 ? launch<32, false>(a, st) : a->HD <= 64 ? launch<64, false>(a, st) : launch<128, false>(a, st);
}
int attention_short_bwd(const CmeAttn* a, cudaStream_t st) {
    CME_REQUIRE(a->lse && a->delta && a->d_o && a->dq && a->dk && a->dv, CME_ERR_SHAPE, "attention backward: missing buffer");
    return a->HD <= 32 ? launch<32, true>(a, st) : a->HD <= 64 ? launch<64, true>(a, st) : launch<128, true>(a, st);
}
