// CUDA-core attention, forward and backward, any head size up to 128, fp32 or bf16 I/O, fp32 math.
//
// This is the strict-precision / any-shape path (parity tests, head sizes the tensor-core kernel does not
// take).  The reference's production attention materialises scores, probabilities and their gradients as
// three [B*H, T, T] buffers around batched GEMMs (FINAL_CLEAN_CODE_/src/kernels/attention.cu:138-200,
// 253-328); its streaming kernel (:56-136) is forward-only and unused.  Here both directions stream
// key / query tiles through shared memory with an online softmax, keep only the log-sum-exp per row,
// and recompute probabilities in the backward pass, so nothing of size T x T touches global memory.
#include "attention.h"

namespace {

// What bounds these kernels is the fp32 multiply-add rate and, next to it, shared-memory reads: a 16-byte load per lane
// takes the SM's shared memory four clocks, in which its schedulers issue sixteen multiply-adds.  So every product is
// register-tiled.  In the forward the warps form groups of 16 rows x 2 halves -- of the streamed rows in the score products, of the
// head's columns in the others; a lane has 4 of the rows (ty + 4 i) and every eighth streamed row of its half (tx + 8 j), or VW
// consecutive columns in 8 VW.  In the backward four warps have a product (attn_bwd_kernel) and a lane 8 rows.  No load has a bank
// conflict, since a row's pitch is an odd number of 16-byte words.  Multiply-adds are packed pairs, fp32 tiles arrive by asynchronous
// copies, all that a group of warps needs at once; in the forward V's under the first product.
// The head size is padded with zeros to a multiple of 32 (template G = ceil(HD / 32)).
// 32 x 4 heads x 64 tokens x head size 128, fp32, forward + backward: 12.9 + 24.0 us; 18 + 31 with a warp for whole rows of the
// forward, single multiply-adds and tiles loaded through registers one after the other, 12.9 + 27.8 with eight warps on each of the
// backward's products (floor of both at the fp32 rate, 0.94 GFLOP at 74 TFLOP/s: 13 us).  64 query rows a block instead of 32 in the
// forward: 12.8 us, no different.
constexpr int CT = 64;               // rows streamed per step
constexpr int WR = 16;               // rows a warp of the forward owns
constexpr int LR = WR / 4;           // rows a lane has of them
constexpr int SP = CT + 4;           // pitch of the probability tiles
constexpr int MAX_HD = 128;
constexpr int BWD_ROWS = 64, BWD_THREADS = 256;
template <int G> struct Pitch { static constexpr int P = 32 * G + 4; };

__device__ __forceinline__ long long head_base(const CmeAttn& a, int bh) {
    return (long long)(bh / a.nh) * a.sb + (long long)(bh % a.nh) * a.sh;
}
__device__ __forceinline__ long long head_base_o(const CmeAttn& a, int bh) {
    return (long long)(bh / a.nh) * a.osb + (long long)(bh % a.nh) * a.osh;
}

template <typename T> __device__ __forceinline__ float4 ld4(const T* p);
template <> __device__ __forceinline__ float4 ld4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 ld4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 lo = bf2_to_f2(u.x), hi = bf2_to_f2(u.y);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
template <typename T> __device__ __forceinline__ void st4(T* p, const float* v);
template <> __device__ __forceinline__ void st4<float>(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <> __device__ __forceinline__ void st4<__nv_bfloat16>(__nv_bfloat16* p, const float* v) {
    *reinterpret_cast<uint2*>(p) = make_uint2(f2_to_bf2(v[0], v[1]), f2_to_bf2(v[2], v[3]));
}

// Rows [r0, r0 + NR) of a [T_, HD] operand to shared memory as fp32, zeros beyond T_ and HD.  `vec`: every
// row starts on a boundary of four elements and HD is a multiple of four.
template <typename T, int G, int NR, int NT>
__device__ __forceinline__ void load_rows(float* dst, const T* src, long long st, int r0, int T_, int HD, bool vec) {
    constexpr int N = NR * 8 * G / NT, U = N % 8 == 0 ? 8 : N % 6 == 0 ? 6 : N % 4 == 0 ? 4 : 2;
    static_assert(NR * 8 * G % NT == 0 && N % U == 0, "whole rounds");
    if (sizeof(T) == 2 && vec) {
        // U loads on their way before the first is used; with each under its branch and store, as below, they follow one another
        // (fp32 tiles come by asynchronous copies).  bf16 backward, 24 x 4 heads, head size 64, causal: 64 tokens 16.7 -> 13.6 us,
        // 96 tokens 54.1 -> 49.6; head size 128, 128 tokens 99 -> 82.
#pragma unroll 1
        for (int k0 = 0; k0 < N; k0 += U) {
            uint2 raw[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int i = threadIdx.x % NT + (k0 + k) * NT, r = i / (8 * G), c = (i % (8 * G)) * 4;
                const bool in = r0 + r < T_ && c < HD;
                raw[k] = *reinterpret_cast<const uint2*>(in ? src + (long long)(r0 + r) * st + c : src);
                if (!in) raw[k] = make_uint2(0u, 0u);
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int i = threadIdx.x % NT + (k0 + k) * NT, r = i / (8 * G), c = (i % (8 * G)) * 4;
                const float2 lo = bf2_to_f2(raw[k].x), hi = bf2_to_f2(raw[k].y);
                *reinterpret_cast<float4*>(dst + r * Pitch<G>::P + c) = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
        return;
    }
#pragma unroll 8
    for (int k = 0; k < NR * 8 * G / NT; ++k) {
        const int i = threadIdx.x % NT + k * NT, r = i / (8 * G), c = (i % (8 * G)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + r < T_ && c < HD) {
            const T* p = src + (long long)(r0 + r) * st + c;
            if (vec) {
                v = ld4<T>(p);
            } else {
                v.x = to_f32<T>(p[0]);
                if (c + 1 < HD) v.y = to_f32<T>(p[1]);
                if (c + 2 < HD) v.z = to_f32<T>(p[2]);
                if (c + 3 < HD) v.w = to_f32<T>(p[3]);
            }
        }
        *reinterpret_cast<float4*>(dst + r * Pitch<G>::P + c) = v;
    }
}

// The same as they are, fp32 in whole 16-byte words by asynchronous copies: all of a block's tiles are on their way at once,
// where the registers of a thread hold eight words (40 rounds of its loads for the forward's 80 KB and 128 threads).  Other
// types and alignments are loaded at once.  Complete after copies_wait by every thread and a barrier.
template <typename T, int G, int NR, int NT>
__device__ __forceinline__ void copy_rows(float* dst, const T* src, long long st, int r0, int T_, int HD, bool vec) {
    if (sizeof(T) == 4 && vec) {
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
        for (int k = 0; k < NR * 8 * G / NT; ++k) {
            const int i = threadIdx.x % NT + k * NT, r = i / (8 * G), c = (i % (8 * G)) * 4;
            const bool in = r0 + r < T_ && c < HD;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)(r * Pitch<G>::P + c) * 4u),
                         "l"(in ? src + (long long)(r0 + r) * st + c : src), "r"(in ? 16 : 0)
                         : "memory");
        }
    } else {
        load_rows<T, G, NR, NT>(dst, src, st, r0, T_, HD, vec);
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the last N committed groups of this thread have arrived.
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// s[i][j] = A[4 i] . B[8 j] over ND elements; A and B point at the lane's first rows.  Packed pairs: the even and the odd elements
// are summed apart, two multiply-adds per instruction, so that a scheduler with one or two warps has issue slots left for their
// loads.
template <int P, int ND, int NJ, int NI>
__device__ __forceinline__ void dot_tile(const float* A, const float* B, float (*s)[NJ]) {
    F32x2 t[NI][NJ];
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) t[i][j] = f2_splat(0.f);
#pragma unroll 2
    for (int d = 0; d < ND; d += 4) {
        float4 a[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) a[i] = *reinterpret_cast<const float4*>(A + 4 * i * P + d);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float4 b = *reinterpret_cast<const float4*>(B + 8 * j * P + d);
#pragma unroll
            for (int i = 0; i < NI; ++i)
                t[i][j] = f2_fma(f2_pack(a[i].z, a[i].w), f2_pack(b.z, b.w),
                                 f2_fma(f2_pack(a[i].x, a[i].y), f2_pack(b.x, b.y), t[i][j]));
        }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            float even, odd;
            f2_unpack(t[i][j], even, odd);
            s[i][j] = even + odd;
        }
    }
}

// VW consecutive columns from shared memory.
template <int VW> __device__ __forceinline__ void lds(const float* p, float* f);
template <> __device__ __forceinline__ void lds<4>(const float* p, float* f) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void lds<2>(const float* p, float* f) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    f[0] = v.x; f[1] = v.y;
}

// o[i][k] += w(i, j) * B[j][c0 + 8 VW k ...] over NJ streamed rows, c0 the lane's first column.  W: the weight tile, element
// (row, j) at row * WROW + j * WCOL, its first row being the lane's.
template <int G, int WROW, int WCOL, int NJ = CT, int NI, int NK, int VW>
__device__ __forceinline__ void weighted_rows(const float* W, const float* B, float (&o)[NI][NK][VW]) {
    constexpr int P = Pitch<G>::P;
#pragma unroll 2
    for (int j = 0; j < NJ; j += 4) {
        float w[NI][4];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            if (WCOL == 1) {
                lds<4>(W + 4 * i * WROW + j, w[i]);
            } else {
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) w[i][jj] = W[4 * i * WROW + (j + jj) * WCOL];
            }
        }
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                float b[VW];
                lds<VW>(B + (j + jj) * P + 8 * VW * k, b);
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int c = 0; c < VW; c += 2)
                        f2_unpack(f2_fma(f2_splat(w[i][jj]), f2_pack(b[c], b[c + 1]), f2_pack(o[i][k][c], o[i][k][c + 1])),
                                  o[i][k][c], o[i][k][c + 1]);
            }
        }
    }
}

// VW consecutive columns of an output row (the row is known to be inside the tensor).
template <typename T, int VW>
__device__ __forceinline__ void store_cols(T* row, int c, int HD, const float* v, float mul, bool vec) {
    float t[VW];
#pragma unroll
    for (int k = 0; k < VW; ++k) t[k] = v[k] * mul;
    if (VW == 4 && vec && c < HD) { st4<T>(row + c, t); return; }
#pragma unroll
    for (int k = 0; k < VW; ++k)
        if (c + k < HD) row[c + k] = from_f32<T>(t[k]);
}

// Blocks per SM that the registers have to leave room for: what shared memory takes (G = 1: five of seven, at 72 registers it spills).
// Left to itself the compiler gave the bf16 backward of two groups 162 registers and with them one block per SM for two (64 heads x 128
// tokens, head size 64: 51 us, 40 so), and the forwards of three and four groups fewer than there is room for.
template <int G, int NW> constexpr int fwd_blocks_per_sm() {
    return G == 1 ? (NW == 1 ? 8 : 5) : G == 2 ? (NW == 1 ? 5 : 4) : G == 3 ? 3 : 2;
}
template <typename T, int G, int NW>
__global__ void __launch_bounds__(NW * 64, fwd_blocks_per_sm<G, NW>()) attn_fwd_kernel(const CmeAttn a, const bool vec) {
    constexpr int P = Pitch<G>::P, RT = NW * WR, NT = NW * 64;
    // a lane's columns: VW at half * 16 G + tx * VW, then every 8 VW
    constexpr int VW = G % 2 == 0 ? 4 : 2, NK = 2 * G / VW;
    extern __shared__ __align__(16) float sm[];
    float* sQ = sm;                    // [RT][P]
    float* sK = sQ + RT * P;           // [CT][P]
    float* sV = sK + CT * P;           // [CT][P]
    float* sP = sV + CT * P;           // [RT][SP]
    __shared__ float sM[2][RT], sL[2][RT];     // the halves' row maxima and sums
    pdl_wait();
    const int bh = blockIdx.y, q0 = blockIdx.x * RT, HD = a.HD;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
    const int w0 = (warp % NW) * WR, half = warp / NW, c0 = half * 16 * G + tx * VW;
    const long long base = head_base(a, bh);
    copy_rows<T, G, RT, NT>(sQ, (const T*)a.q + base, a.st, q0, a.T, HD, vec);
    float m[LR], l[LR], o[LR][NK][VW];
#pragma unroll
    for (int i = 0; i < LR; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int g = 0; g < NK; ++g)
#pragma unroll
            for (int c = 0; c < VW; ++c) o[i][g][c] = 0.f;
    }
    const int kend = a.causal ? min(a.T, q0 + RT) : a.T;
    float* wP = sP + (w0 + ty) * SP;
    for (int k0 = 0; k0 < kend; k0 += CT) {
        __syncthreads();
        copy_rows<T, G, CT, NT>(sK, (const T*)a.k + base, a.st, k0, a.T, HD, vec);
        copies_commit();
        copy_rows<T, G, CT, NT>(sV, (const T*)a.v + base, a.st, k0, a.T, HD, vec);
        copies_commit();
        copies_wait<1>();
        __syncthreads();
        float s[LR][4];
        dot_tile<P, 32 * G, 4, LR>(sQ + (w0 + ty) * P, sK + (half * 32 + tx) * P, s);
#pragma unroll
        for (int i = 0; i < LR; ++i) {
            const int row = w0 + ty + 4 * i, q = q0 + row;
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = k0 + half * 32 + tx + 8 * j;
                s[i][j] = k < a.T && (!a.causal || k <= q) ? s[i][j] * a.scale : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            if (tx == 0) sM[half][row] = mx;
        }
        __syncthreads();                           // the other half of these rows' scores is another warp's
        float alpha[LR];
#pragma unroll
        for (int i = 0; i < LR; ++i) {
            const int row = w0 + ty + 4 * i;
            const float mnew = fmaxf(m[i], fmaxf(sM[0][row], sM[1][row]));
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = (mnew == -INFINITY) ? 0.f : __expf(s[i][j] - mnew);
                wP[4 * i * SP + half * 32 + tx + 8 * j] = p;
                sum += p;
            }
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (tx == 0) sL[half][row] = sum;
            alpha[i] = (m[i] == -INFINITY) ? 0.f : __expf(m[i] - mnew);
            m[i] = mnew;
        }
        copies_wait<0>();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < LR; ++i) {
            const int row = w0 + ty + 4 * i;
            l[i] = l[i] * alpha[i] + (sL[0][row] + sL[1][row]);
#pragma unroll
            for (int g = 0; g < NK; ++g)
#pragma unroll
                for (int c = 0; c < VW; ++c) o[i][g][c] *= alpha[i];
        }
        weighted_rows<G, SP, 1>(wP, sV + c0, o);
    }
#pragma unroll
    for (int i = 0; i < LR; ++i) {
        const int q = q0 + w0 + ty + 4 * i;
        if (q < a.T) {
            const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
            T* out = (T*)a.o + head_base_o(a, bh) + (long long)q * a.ost;
#pragma unroll
            for (int g = 0; g < NK; ++g) store_cols<T, VW>(out, c0 + 8 * VW * g, HD, o[i][g], inv, vec);
            if (half == 0 && tx == 0 && a.lse) a.lse[(long long)bh * a.T + q] = m[i] + logf(l[i]);
        }
    }
}

// delta[bh, t] = sum_d dO * O, bf16 of any head size (the CUDA-core backward makes its own).
__global__ void attn_delta_kernel(const CmeAttn a) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int rows = a.nb * a.nh * a.T;
    if (row >= rows) return;
    const int bh = row / a.T, t = row % a.T;
    const long long off = head_base_o(a, bh) + (long long)t * a.ost;
    float s = 0.f;
    for (int d = threadIdx.x & 31; d < a.HD; d += 32)
        s += __bfloat162float(((const __nv_bfloat16*)a.d_o)[off + d]) * __bfloat162float(((const __nv_bfloat16*)a.o)[off + d]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) a.delta[row] = s;
}
// bf16, head size 64, 16-byte aligned rows: 8 lanes per row (one 128-bit load of each operand per lane), two rows per
// lane so that four loads are in flight.  `clear`: 64 floats per row, set to zero in the same pass (the scratch the
// backward adds its parts of dQ to), which saves a clearing pass between this kernel and the backward: 16 x 12
// heads x 1024 tokens 12.7 us for both, 12.9 + 9.5 us as two passes.
__global__ void __launch_bounds__(256) attn_delta_hd64_kernel(const CmeAttn a, float* __restrict__ clear) {
    pdl_wait();
    const int rows = a.nb * a.nh * a.T, sub = threadIdx.x & 7;
    uint4 x[2], y[2];
    int row[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        row[k] = blockIdx.x * 64 + (threadIdx.x >> 3) + 32 * k;
        x[k] = y[k] = make_uint4(0, 0, 0, 0);
        if (row[k] < rows) {
            const int bh = row[k] / a.T, t = row[k] % a.T;
            const long long off = head_base_o(a, bh) + (long long)t * a.ost + sub * 8;
            x[k] = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.d_o + off);
            y[k] = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.o + off);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        float u[8], w[8], s = 0.f;
        unpack8(x[k], u);
        unpack8(y[k], w);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += u[i] * w[i];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if (row[k] < rows) {
            if (sub == 0) a.delta[row[k]] = s;
            if (clear) {
                float4* z = reinterpret_cast<float4*>(clear + (long long)row[k] * 64) + sub;
                z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
                z[8] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
}

// delta[r] = sum_d dO[r][d] * O[r][d] for the CT rows whose tiles are staged, one warp per row, four warps.
template <int G> __device__ __forceinline__ void delta_rows(float* dst, const float* sdO, const float* sO) {
    constexpr int NW = BWD_THREADS / 64;
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % NW;
#pragma unroll
    for (int k = 0; k < CT / NW; ++k) {
        const int r = warp + k * NW;
        float s = 0.f;
#pragma unroll
        for (int g = 0; g < G; ++g) s = fmaf(sdO[r * Pitch<G>::P + lane + 32 * g], sO[r * Pitch<G>::P + lane + 32 * g], s);
        s = warp_sum(s);
        if (lane == 0) dst[r] = s;
    }
}

// blockIdx.z == 0: the block owns 64 keys and streams queries:    dV = sum_i P_ij dO_i,  dK = scale * sum_i dS_ij Q_i.
//                  With one key block (T <= 64, ONE) it has all of dS as well and makes dQ too: five products instead of the
//                  seven of the split form.
// blockIdx.z == 1: the block owns 64 queries and streams keys:    dQ = scale * sum_j dS_ij K_j
// Both kinds run in one launch, and delta = rowsum(dO * O) is made from the staged rows instead of by a kernel before.
//
// The first four warps fetch Q and K, make P and then dV, the others fetch dO, V and O, make delta, dS and then dK: with four warps on
// a 64 x 64 product a lane has 8 rows of it where eight warps leave 4, and so loads 12 words for 32 results a step instead of 8 for 16.
// In dQ, a single product, they have half of the keys each.  A block that makes its scores once (ONE) and has the registers of a
// whole SM goes to 8 x 8, the elements of the heads split between two warps.  Shared memory's share of five products of width 128
// falls from 34800 clocks to 21200, next to 20500 of multiply-adds.  32 x 4 heads, fp32, us before and now: 64 tokens, head size 128
// 27.8 and 24.0, 64 18.0 and 14.5, 32 13.5 and 10.8; 128 tokens 142 and 120, 69.3 and 67.7, 46.0 and 41.7.
// O is staged as well, in the place of dS where its rows are no longer: loaded row by row into registers, under branches, it was a
// chain of memory round trips (as were the log-sum-exps, read where a score was finished).
template <int G> constexpr int bwd_tiles() { return 32 * G <= CT ? 4 : 5; }
__device__ __forceinline__ void half_sync(int half) { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); }
template <typename T, int G, bool ONE>
__global__ void __launch_bounds__(BWD_THREADS, G <= 2 ? 2 : 1) attn_bwd_kernel(const CmeAttn a, const bool vec) {
    constexpr int P = Pitch<G>::P, NT = BWD_THREADS / 2, RT = BWD_ROWS, NI = 8;
    constexpr int KS = ONE && G >= 3 ? 2 : 1;      // warps that share the elements of a score
    constexpr int NP = ONE || G >= 3 ? NI : 4;     // rows of a score product at a time: two blocks per SM leave 128 registers
    // delta after dP, whose product O's copies then run under; with one block per SM the other half would wait for it (24.9 us where
    // 24.0 are below)
    constexpr bool LATE = NP < NI;
    // a lane's columns: VW at part * 16 G + tx * VW, then every 8 VW
    constexpr int VW = G % 2 == 0 ? 4 : 2, NK = 2 * G / VW;
    static_assert(bwd_tiles<G>() == 5 || RT * P <= RT * SP, "O in the place of dS");
    static_assert(RT == CT && NT / 32 * 32 * 32 == RT * CT, "own and streamed tiles of one height, four warps on 32 x 32 each");
    static_assert(NT / 32 * 32 * NI * 4 <= RT * SP, "partial scores lie where the tile of P or dS will");
    static_assert(BWD_THREADS * 4 * NK * VW <= CT * P, "half of dQ lies in the tile of the streamed rows");
    extern __shared__ __align__(16) float sm[];
    float* sA = sm;                    // own rows       K | Q
    float* sB = sA + RT * P;           //                V | dO
    float* sC = sB + RT * P;           // streamed rows  Q | K
    float* sD = sC + CT * P;           //                dO | V
    float* sP = sD + CT * P;           // [RT][SP] P (own row, streamed row)
    float* sS = sP + RT * SP;          // [RT][SP] dS
    float* sDl = sS + RT * SP;         // [CT] delta of the queries in shared memory
    float* sL = sDl + CT;              // [CT] log-sum-exp of the same queries
    float* sO = bwd_tiles<G>() == 4 ? sS : sL + CT;        // O of the rows whose delta is made
    pdl_wait();
    const bool kv = ONE || blockIdx.z == 0;
    const int bh = blockIdx.y, r0 = blockIdx.x * RT, HD = a.HD;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
    const int half = warp >> 2, w0 = (warp & 1) * 32 + ty, part = (warp >> 1) & 1, c0 = part * 16 * G + tx * VW;
    const long long base = head_base(a, bh), obase = head_base_o(a, bh);
    const T* q = (const T*)a.q + base; const T* k = (const T*)a.k + base; const T* v = (const T*)a.v + base;
    const T* d_o = (const T*)a.d_o + obase; const T* o = (const T*)a.o + obase;
    const float* lse = a.lse + (long long)bh * a.T;
    float acc[NI][NK][VW];
    auto clear = [&] {
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int g = 0; g < NK; ++g)
#pragma unroll
                for (int c = 0; c < VW; ++c) acc[i][g][c] = 0.f;
    };
    if (!ONE) clear();
    // causal: queries see keys <= their index.  dQ blocks stop early; dK / dV blocks start late.
    const int s_begin = (kv && a.causal) ? r0 : 0;
    const int s_end = (!kv && a.causal) ? min(a.T, r0 + RT) : a.T;
    for (int s0 = s_begin; s0 < s_end; s0 += CT) {
        const bool first = ONE || s0 == s_begin;
        if (!first) __syncthreads();
        if (half == 0) {
            if (first) copy_rows<T, G, RT, NT>(sA, kv ? k : q, a.st, r0, a.T, HD, vec);
            copy_rows<T, G, CT, NT>(sC, kv ? q : k, a.st, s0, a.T, HD, vec);
            const int qi = (kv ? s0 : r0) + (int)threadIdx.x;
            if ((kv || first) && threadIdx.x < CT) sL[threadIdx.x] = qi < a.T ? lse[qi] : 0.f;
        } else {
            if (first) copy_rows<T, G, RT, NT>(sB, kv ? v : d_o, kv ? a.st : a.ost, r0, a.T, HD, vec);
            copy_rows<T, G, CT, NT>(sD, kv ? d_o : v, kv ? a.ost : a.st, s0, a.T, HD, vec);
            if (LATE) copies_commit();
            if (kv || first) copy_rows<T, G, CT, NT>(sO, o, a.ost, kv ? s0 : r0, a.T, HD, vec);
        }
        copies_commit();
        if (LATE && half) copies_wait<1>(); else copies_wait<0>();
        half_sync(half);
        if (!LATE && half && (kv || first)) delta_rows<G>(sDl, kv ? sD : sB, sO);
        // S or dP: rows w0 + 4 i, columns part * 32 + tx + 8 j
        const float* own = (half ? sB : sA) + w0 * P;
        const float* str = (half ? sD : sC) + tx * P;
        float s[NI][4];
        if (KS == 1) {
#pragma unroll
            for (int i = 0; i < NI; i += NP) dot_tile<P, 32 * G, 4, NP>(own + 4 * i * P, str + part * 32 * P, s + i);
        } else {
            float t[NI][8];                        // all 64 columns, half of the elements
            dot_tile<P, 16 * G, 8, NI>(own + part * 16 * G, str + part * 16 * G, t);
            float* mine = (half ? sS : sP) + (warp & 3) * (32 * NI * 4) + lane * 4;
            const float* other = (half ? sS : sP) + ((warp & 3) ^ 2) * (32 * NI * 4) + lane * 4;
#pragma unroll
            for (int i = 0; i < NI; ++i)
                *reinterpret_cast<float4*>(mine + i * 128) = part ? make_float4(t[i][0], t[i][1], t[i][2], t[i][3])
                                                                  : make_float4(t[i][4], t[i][5], t[i][6], t[i][7]);
            half_sync(half);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const float4 p = *reinterpret_cast<const float4*>(other + i * 128);
                s[i][0] = (part ? t[i][4] : t[i][0]) + p.x;
                s[i][1] = (part ? t[i][5] : t[i][1]) + p.y;
                s[i][2] = (part ? t[i][6] : t[i][2]) + p.z;
                s[i][3] = (part ? t[i][7] : t[i][3]) + p.w;
            }
            half_sync(half);                       // they have been read: P and dS go to the same place
        }
        if (LATE && half && (kv || first)) {
            copies_wait<0>();
            half_sync(half);
            delta_rows<G>(sDl, kv ? sD : sB, sO);
        }
        auto seen = [&](int row, int col) {
            const int qi = kv ? s0 + col : r0 + row, ki = kv ? r0 + row : s0 + col;
            return qi < a.T && ki < a.T && (!a.causal || ki <= qi);
        };
        if (half == 0) {
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = w0 + 4 * i, col = part * 32 + tx + 8 * j;
                    const float e = s[i][j] * a.scale - sL[kv ? col : row];
                    sP[row * SP + col] = __expf(seen(row, col) ? e : -INFINITY);
                }
        }
        __syncthreads();                           // P and, for dV, dO
        if (half) {
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = w0 + 4 * i, col = part * 32 + tx + 8 * j;
                    const float ds = sP[row * SP + col] * (s[i][j] - sDl[kv ? col : row]);
                    sS[row * SP + col] = seen(row, col) ? ds : 0.f;
                }
        }
        if (ONE) clear();
        if (!kv) {
            __syncthreads();
            weighted_rows<G, SP, 1, CT / 2>(sS + w0 * SP + half * (CT / 2), sC + half * (CT / 2) * P + c0, acc);      // dQ += dS K
        } else {
            if (half) half_sync(half);
            weighted_rows<G, SP, 1>((half ? sS : sP) + w0 * SP, (half ? sC : sD) + c0, acc);      // dV += P^T dO, dK += dS^T Q
        }
        if (ONE) break;
    }
    if (kv) {
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int r = r0 + w0 + 4 * i;
            if (r < a.T)
#pragma unroll
                for (int g = 0; g < NK; ++g)
                    store_cols<T, VW>((T*)(half ? a.dk : a.dv) + base + (long long)r * a.st, c0 + 8 * VW * g, HD, acc[i][g],
                                      half ? a.scale : 1.f, vec);
        }
        if (!ONE) return;
    }
    __syncthreads();                               // dS is complete, the streamed rows have been read
    if (ONE) {                                     // dQ_i = scale * sum_j dS_ij K_j: the tile read down its columns
        clear();
        weighted_rows<G, 1, SP, CT / 2>(sS + w0 + half * (CT / 2) * SP, sA + half * (CT / 2) * P + c0, acc);
    }
    // the halves' sums meet: each finishes four of a lane's rows
    float* give = sC + threadIdx.x * VW;
    const float* take = sC + (threadIdx.x ^ (BWD_THREADS / 2)) * VW;
#pragma unroll
    for (int i = 0; i < NI / 2; ++i)
#pragma unroll
        for (int g = 0; g < NK; ++g)
#pragma unroll
            for (int c = 0; c < VW; ++c) give[(i * NK + g) * BWD_THREADS * VW + c] = half ? acc[i][g][c] : acc[i + NI / 2][g][c];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NI / 2; ++i) {
        const int r = r0 + w0 + 4 * (i + (half ? NI / 2 : 0));
        if (r < a.T)
#pragma unroll
            for (int g = 0; g < NK; ++g) {
                float sum[VW];
#pragma unroll
                for (int c = 0; c < VW; ++c)
                    sum[c] = (half ? acc[i + NI / 2][g][c] : acc[i][g][c]) + take[(i * NK + g) * BWD_THREADS * VW + c];
                store_cols<T, VW>((T*)a.dq + base + (long long)r * a.st, c0 + 8 * VW * g, HD, sum, a.scale, vec);
            }
    }
}

// Rows of every operand start on a boundary of four elements (16 bytes of fp32, 8 of bf16) and HD is a multiple of
// four: vector loads and stores; anything else takes the scalar accesses of the same kernel.
bool rows_vectorisable(const CmeAttn* a, bool bwd) {
    const uintptr_t mask = a->dtype == CME_BF16 ? 7 : 15;
    uintptr_t p = reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) |
                  reinterpret_cast<uintptr_t>(a->v) | reinterpret_cast<uintptr_t>(a->o);
    if (bwd)
        p |= reinterpret_cast<uintptr_t>(a->d_o) | reinterpret_cast<uintptr_t>(a->dq) | reinterpret_cast<uintptr_t>(a->dk) |
             reinterpret_cast<uintptr_t>(a->dv);
    return !(p & mask) && a->HD % 4 == 0 &&
           !((a->sb | a->sh | a->st | a->osb | a->osh | a->ost) & 3);
}

template <typename K> int allow_smem(K kernel, size_t smem) {
    if (smem > 48 * 1024)
        CME_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return CME_OK;
}

template <typename T, int G, int NW> int fwd_launch(const CmeAttn* a, cudaStream_t st) {
    constexpr int P = Pitch<G>::P, RT = NW * WR;
    constexpr size_t smem = ((RT + 2 * CT) * P + RT * SP) * sizeof(float);
    auto k = attn_fwd_kernel<T, G, NW>;
    int rc = allow_smem(k, smem);
    if (rc) return rc;
    CME_CUDA(cme_launch_dependent(k, dim3(cme_cdiv(a->T, RT), a->nb * a->nh), dim3(NW * 64), smem, st, *a,
                                  rows_vectorisable(a, false)));
    CME_LAUNCH_CHECK();
    return CME_OK;
}
template <typename T, int G> int bwd_launch(const CmeAttn* a, cudaStream_t st) {
    constexpr int P = Pitch<G>::P, RT = BWD_ROWS;
    constexpr size_t smem = (bwd_tiles<G>() * RT * P + 2 * RT * SP + 2 * CT) * sizeof(float);
    static_assert(smem <= 227 * 1024, "one block's shared memory");
    auto k = a->T <= RT ? attn_bwd_kernel<T, G, true> : attn_bwd_kernel<T, G, false>;
    int rc = allow_smem(k, smem);
    if (rc) return rc;
    CME_CUDA(cme_launch_dependent(k, dim3(cme_cdiv(a->T, RT), a->nb * a->nh, a->T <= RT ? 1 : 2), dim3(BWD_THREADS), smem,
                                  st, *a, rows_vectorisable(a, true)));
    CME_LAUNCH_CHECK();
    return CME_OK;
}
template <typename T> int fwd_t(const CmeAttn* a, cudaStream_t st) {
    // 32 query rows per block; 16 where that leaves SMs without a block
    const bool few = (long long)cme_cdiv(a->T, 2 * WR) * a->nb * a->nh < 148;
    switch (cme_cdiv(a->HD, 32)) {
        case 1: return few ? fwd_launch<T, 1, 1>(a, st) : fwd_launch<T, 1, 2>(a, st);
        case 2: return few ? fwd_launch<T, 2, 1>(a, st) : fwd_launch<T, 2, 2>(a, st);
        case 3: return few ? fwd_launch<T, 3, 1>(a, st) : fwd_launch<T, 3, 2>(a, st);
        default: return few ? fwd_launch<T, 4, 1>(a, st) : fwd_launch<T, 4, 2>(a, st);
    }
}
template <typename T> int bwd_t(const CmeAttn* a, cudaStream_t st) {
    switch (cme_cdiv(a->HD, 32)) {
        case 1: return bwd_launch<T, 1>(a, st);
        case 2: return bwd_launch<T, 2>(a, st);
        case 3: return bwd_launch<T, 3>(a, st);
        default: return bwd_launch<T, 4>(a, st);
    }
}

int check(const CmeAttn* a, bool bwd) {
    CME_REQUIRE(a->nb > 0 && a->nh > 0 && a->T > 0 && a->HD > 0, CME_ERR_SHAPE, "attention: empty input");
    CME_REQUIRE(a->HD <= MAX_HD, CME_ERR_LIMIT, "attention: head size %d exceeds %d", a->HD, MAX_HD);
    CME_REQUIRE(a->lse != nullptr, CME_ERR_SHAPE, "attention: lse buffer is required");
    if (bwd) CME_REQUIRE(a->delta && a->d_o && a->dq && a->dk && a->dv, CME_ERR_SHAPE, "attention backward: missing buffer");
    return CME_OK;
}

}  // namespace

// delta[bh, t] = sum_d dO * O for the bf16 tensor-core backwards; `clear` (or null): fp32 scratch of 64 per row to zero.
int attention_delta_launch(const CmeAttn* a, cudaStream_t st, float* clear) {
    const int rows = a->nb * a->nh * a->T;
    const bool al = ((reinterpret_cast<uintptr_t>(a->d_o) | reinterpret_cast<uintptr_t>(a->o)) & 15) == 0 &&
                    a->ost % 8 == 0 && a->osh % 8 == 0 && a->osb % 8 == 0;
    if (a->HD == 64 && al) {
        CME_CUDA(cme_launch_dependent(attn_delta_hd64_kernel, dim3(cme_cdiv(rows, 64)), dim3(256), 0, st, *a, clear));
        CME_LAUNCH_CHECK();
        return CME_OK;
    }
    if (clear) CME_CUDA(cudaMemsetAsync(clear, 0, (size_t)rows * 64 * sizeof(float), st));
    attn_delta_kernel<<<cme_cdiv(rows, 8), 256, 0, st>>>(*a);
    CME_LAUNCH_CHECK();
    return CME_OK;
}

int attention_simt_fwd(const CmeAttn* a, cudaStream_t st) {
    int rc = check(a, false);
    if (rc) return rc;
    return a->dtype == CME_BF16 ? fwd_t<__nv_bfloat16>(a, st) : fwd_t<float>(a, st);
}
int attention_simt_bwd(const CmeAttn* a, cudaStream_t st) {
    int rc = check(a, true);
    if (rc) return rc;
    return a->dtype == CME_BF16 ? bwd_t<__nv_bfloat16>(a, st) : bwd_t<float>(a, st);
}

// The short-sequence kernel stands in for the two paths that round P to bf16 as it does; bf16 calls that neither takes
// (e.g. head size 32 in split layout) keep the fp32 probabilities of the SIMT kernel.  Up to 64 tokens because one
// block then holds the whole head; the flash kernel's 128-row tile is at least half padding there, and its backward is three
// launches.
int attention_takes_short(const CmeAttn* a, int bwd) {
    return attention_short_supported(a, bwd) && (attention_tc_supported(a) || attention_gemm_supported(a));
}

// backend: 0 auto (one-launch kernel up to 64 tokens, else fused tensor-core kernel, else batched-GEMM path, else SIMT),
//          1 fused tensor-core only, 2 SIMT only, 3 batched-GEMM path only
// The path of a call with that backend (CmeAttnPath).
CME_API int cme_attention_path(const CmeAttn* a, int backend, int bwd) {
    if (backend == 0 && attention_takes_short(a, bwd)) return CME_ATTN_PATH_SHORT;
    if ((backend == 0 || backend == 1) && attention_tc_supported(a)) return CME_ATTN_PATH_TC;
    if ((backend == 0 || backend == 3) && attention_gemm_supported(a)) return CME_ATTN_PATH_GEMM;
    return CME_ATTN_PATH_SIMT;
}
static int check_path(int backend, int path) {
    CME_REQUIRE(backend != 1 || path == CME_ATTN_PATH_TC, CME_ERR_SHAPE, "attention shape not supported by the tensor-core kernel");
    CME_REQUIRE(backend != 3 || path == CME_ATTN_PATH_GEMM, CME_ERR_SHAPE, "attention shape not supported by the batched-GEMM path");
    return CME_OK;
}
CME_API int cme_attention_fwd(const CmeAttn* a, int backend, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int path = cme_attention_path(a, backend, 0), rc = check_path(backend, path);
    if (rc) return rc;
    switch (path) {
        case CME_ATTN_PATH_SHORT: return attention_short_fwd(a, st);
        case CME_ATTN_PATH_TC: return attention_tc_fwd(a, st);
        case CME_ATTN_PATH_GEMM: return attention_gemm_fwd(a, st);
        default: return attention_simt_fwd(a, st);
    }
}
CME_API int cme_attention_bwd(const CmeAttn* a, int backend, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int path = cme_attention_path(a, backend, 1);
    int rc = check_path(backend, path);
    // the same calls are refused as without the one-launch kernel
    if (!rc && path == CME_ATTN_PATH_SHORT && attention_tc_supported(a)) rc = attention_tc_check_bwd(a);
    if (rc) return rc;
    switch (path) {
        case CME_ATTN_PATH_SHORT: return attention_short_bwd(a, st);
        case CME_ATTN_PATH_TC: return attention_tc_bwd(a, st);
        case CME_ATTN_PATH_GEMM: return attention_gemm_bwd(a, st);
        default: return attention_simt_bwd(a, st);
    }
}
CME_API long long cme_attention_gemm_ws_bytes(int nb, int T) { return attention_gemm_ws_bytes(nb, T); }
