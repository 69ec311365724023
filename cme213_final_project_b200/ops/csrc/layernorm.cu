// LayerNorm forward / backward with fused residual adds, bf16 or fp32 I/O, fp32 statistics.
//
// Covers the reference's five LayerNorm kernels (FINAL_CLEAN_CODE_/src/kernels/layernorm.cu:24-305):
// plain forward, forward saving mean / inverse std, fused residual + LayerNorm forward, backward dx with
// optional fused "gx += dx" residual-gradient add, and the column-wise d(gamma) / d(beta) reduction.
// The reference uses one block per row with a two-pass block reduction and a second kernel with one block
// per column for the weight gradients.  Here one warp owns a row (128-bit loads, shuffles only), and the
// backward kernel produces dx and per-block partial d(gamma)/d(beta) in a single pass over x and dy; a
// small second kernel sums the partials in a fixed order (no atomics, bit-reproducible).
#include "common.h"

namespace {

constexpr int LN_WARPS = 8;            // rows per block iteration
constexpr int LN_MAX_VEC = 4;          // 16-byte vectors per lane kept in registers (D <= 1024 bf16, 512 fp32)

template <typename T> struct VecOf;
template <> struct VecOf<float> { static constexpr int N = 4; };
template <> struct VecOf<__nv_bfloat16> { static constexpr int N = 8; };

template <typename T> __device__ __forceinline__ void load_vec(const T* p, float* f);
template <> __device__ __forceinline__ void load_vec<float>(const float* p, float* f) {
    float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16>(const __nv_bfloat16* p, float* f) {
    unpack8(*reinterpret_cast<const Bf16x8*>(p), f);
}
template <typename T> __device__ __forceinline__ void store_vec(T* p, const float* f);
template <> __device__ __forceinline__ void store_vec<float>(float* p, const float* f) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
template <> __device__ __forceinline__ void store_vec<__nv_bfloat16>(__nv_bfloat16* p, const float* f) {
    *reinterpret_cast<Bf16x8*>(p) = pack8(f);
}

template <typename T> __device__ __forceinline__ void unpack_raw(const uint4& r, float* f);
template <> __device__ __forceinline__ void unpack_raw<float>(const uint4& r, float* f) {
    f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w);
}
template <> __device__ __forceinline__ void unpack_raw<__nv_bfloat16>(const uint4& r, float* f) { unpack8(r, f); }

__device__ __forceinline__ void load_raw(uint4& r, const void* p) {
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
}

// Rows travel through a ring of shared-memory stages: all of its stages but one are ahead of the row a warp works on (three
// stages; two in the backward of four vectors per lane).  A lane copies exactly the 16-byte words it will read itself, so
// waiting for its own copies is all the synchronisation there is.  Registers alone keep one row in flight per warp, and the
// memory idle while its statistics are reduced.
constexpr int LN_STAGES = 3;
// Row numbers are unsigned: the row fetched ahead of the last ones may lie beyond the largest int.
constexpr unsigned row_ahead(unsigned row, unsigned step, int n) { return row + n * step; }
static_assert(row_ahead(0x7fffffffu, 2048 * LN_WARPS, LN_STAGES) > 0x7fffffffu, "no wrap around with up to 2048 blocks");
__device__ __forceinline__ void ring_copy(uint4* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ring_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The steps of a row on packed pairs: two elements per instruction, rounded like single ones.  The sums over a row are added one
// element after the other, because the order decides on their last bit and that, through ReLU and Adam, on a model's next step; even
// and odd elements apart are no faster (16384 x 768 bf16: forward 18.8 us for 19.1, backward 20.05 for 20.05).
template <int W> __device__ __forceinline__ void row_add(float (&x)[W], const float (&t)[W]) {
#pragma unroll
    for (int j = 0; j < W; j += 2) f2_unpack(f2_add(f2_pack(x[j], x[j + 1]), f2_pack(t[j], t[j + 1])), x[j], x[j + 1]);
}
template <int W> __device__ __forceinline__ void row_sum(float& sum, const float (&x)[W]) {
#pragma unroll
    for (int j = 0; j < W; ++j) sum += x[j];
}
template <int W> __device__ __forceinline__ void row_squares(float& sum, const float (&x)[W], F32x2 nmean) {
#pragma unroll
    for (int j = 0; j < W; j += 2) {
        float d0, d1;
        f2_unpack(f2_add(f2_pack(x[j], x[j + 1]), nmean), d0, d1);
        sum = fmaf(d1, d1, fmaf(d0, d0, sum));
    }
}
template <int W>
__device__ __forceinline__ void row_scale(float (&o)[W], const float (&x)[W], const float (&g)[W], const float (&bt)[W], F32x2 nmean,
                                          F32x2 rstd) {
#pragma unroll
    for (int j = 0; j < W; j += 2)
        f2_unpack(f2_fma(f2_mul(f2_add(f2_pack(x[j], x[j + 1]), nmean), rstd), f2_pack(g[j], g[j + 1]), f2_pack(bt[j], bt[j + 1])),
                  o[j], o[j + 1]);
}
// y = LN(a [+ b]) * gamma + beta; optionally writes r = a + b, mean and rstd.  fp32 rows of at most 32 * NV 16-byte vectors, one
// warp per row, the grid what is resident at once.
template <typename T, int NV>
__global__ void __launch_bounds__(LN_WARPS * 32, NV <= 3 ? 3 : 2)
ln_fwd_vec_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ r_out, const T* __restrict__ gamma,
                  const T* __restrict__ beta, T* __restrict__ y, float* __restrict__ mean_out,
                  float* __restrict__ rstd_out, int rows, int D, float eps) {
    constexpr int W = VecOf<T>::N, S = LN_STAGES;
    extern __shared__ uint4 ring[];                     // [LN_WARPS][S][1 or 2][NV][32]
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = D / W;
    const unsigned step = gridDim.x * LN_WARPS, n_rows = rows;
    const int stage = (b ? 2 : 1) * NV * 32;
    uint4* mine = ring + warp * S * stage + lane;
    auto fetch = [&](unsigned row, int s) {
        if (row < n_rows) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int v = lane + 32 * i;
                if (v < nvec) {
                    ring_copy(mine + s * stage + i * 32, a + (long long)row * D + v * W);
                    if (b) ring_copy(mine + s * stage + (NV + i) * 32, b + (long long)row * D + v * W);
                }
            }
        }
        ring_commit();
    };
    unsigned row = blockIdx.x * LN_WARPS + warp;
#pragma unroll
    for (int s = 0; s < S - 1; ++s) fetch(row_ahead(row, step, s), s);
    for (int s = 0; row < n_rows; row += step, s = s + 1 == S ? 0 : s + 1) {
        fetch(row_ahead(row, step, S - 1), s == 0 ? S - 1 : s - 1);
        ring_wait<S - 1>();
        const uint4* in = mine + s * stage;
        const long long off = (long long)row * D;
        float x[NV][W];
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = lane + 32 * i;
            if (v < nvec) {
                unpack_raw<T>(in[i * 32], x[i]);
                if (b) {
                    float t[W];
                    unpack_raw<T>(in[(NV + i) * 32], t);
                    row_add(x[i], t);
                    if (r_out) store_vec<T>(r_out + off + v * W, x[i]);
                }
                row_sum(sum, x[i]);
            }
        }
        const float mean = warp_sum(sum) / D;
        const F32x2 nmean = f2_splat(-mean);
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (lane + 32 * i < nvec) row_squares(q, x[i], nmean);
        }
        const float rstd = rsqrtf(warp_sum(q) / D + eps);
        const F32x2 rstd2 = f2_splat(rstd);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = lane + 32 * i;
            if (v < nvec) {
                float g[W], bt[W], o[W];
                load_vec<T>(gamma + v * W, g);
                load_vec<T>(beta + v * W, bt);
                row_scale(o, x[i], g, bt, nmean, rstd2);
                store_vec<T>(y + off + v * W, o);
            }
        }
        if (lane == 0) {
            if (mean_out) mean_out[row] = mean;
            if (rstd_out) rstd_out[row] = rstd;
        }
    }
}

// Same bits with one row per warp, from global memory to registers.  Bound by memory: bf16 16384 x 768 with the residual add and its
// sum stored (101 MB) 15.9 us, what a copy takes.  The loads of a bf16 row are asm ahead of all else: left to the compiler, which puts
// each under its sum and store, it took 17.6, and with the rows in a ring of asynchronous copies, as fp32 ones are, 18.7.  Four blocks
// an SM: with five or six forced the longest rows spill (16384 x 1024 22.3, 24.5 and 31.3).
template <typename T, int NV>
__global__ void __launch_bounds__(LN_WARPS * 32, sizeof(T) == 2 ? 4 : 0)      // 0: left to the compiler
ln_fwd_row_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ r_out, const T* __restrict__ gamma,
                  const T* __restrict__ beta, T* __restrict__ y, float* __restrict__ mean_out,
                  float* __restrict__ rstd_out, int rows, int D, float eps) {
    constexpr int W = VecOf<T>::N;
    pdl_wait();
    const int lane = threadIdx.x & 31, nvec = D / W;
    const int row = blockIdx.x * LN_WARPS + (threadIdx.x >> 5);
    if (row >= rows) return;
    const long long off = (long long)row * D;
    constexpr bool FIRST = sizeof(T) == 2;
    uint4 ra[NV], rb[NV];
    if (FIRST) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + 32 * i < nvec) {
                load_raw(ra[i], a + off + (lane + 32 * i) * W);
                if (b) load_raw(rb[i], b + off + (lane + 32 * i) * W);
            }
    }
    float x[NV][W];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = lane + 32 * i;
        if (v < nvec) {
            if (FIRST) unpack_raw<T>(ra[i], x[i]); else load_vec<T>(a + off + v * W, x[i]);
            if (b) {
                float t[W];
                if (FIRST) unpack_raw<T>(rb[i], t); else load_vec<T>(b + off + v * W, t);
                row_add(x[i], t);
                if (r_out) store_vec<T>(r_out + off + v * W, x[i]);
            }
            row_sum(s, x[i]);
        }
    }
    const float mean = warp_sum(s) / D;
    const F32x2 nmean = f2_splat(-mean);
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (lane + 32 * i < nvec) row_squares(q, x[i], nmean);
    }
    const float rstd = rsqrtf(warp_sum(q) / D + eps);
    const F32x2 rstd2 = f2_splat(rstd);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = lane + 32 * i;
        if (v < nvec) {
            float g[W], bt[W], o[W];
            load_vec<T>(gamma + v * W, g);
            load_vec<T>(beta + v * W, bt);
            row_scale(o, x[i], g, bt, nmean, rstd2);
            store_vec<T>(y + off + v * W, o);
        }
    }
    if (lane == 0) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
    }
}

// Same for rows that are not whole vectors or are too long for the registers.
template <typename T>
__global__ void __launch_bounds__(LN_WARPS * 32)
ln_fwd_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ r_out, const T* __restrict__ gamma,
              const T* __restrict__ beta, T* __restrict__ y, float* __restrict__ mean_out,
              float* __restrict__ rstd_out, int rows, int D, float eps) {
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * LN_WARPS + (threadIdx.x >> 5);
    if (row >= rows) return;
    const long long off = (long long)row * D;
    float s = 0.f;
    for (int c = lane; c < D; c += 32) {
        float v = to_f32<T>(a[off + c]);
        if (b) {
            v += to_f32<T>(b[off + c]);
            if (r_out) r_out[off + c] = from_f32<T>(v);
        }
        s += v;
    }
    const float mean = warp_sum(s) / D;
    const T* src = (b && r_out) ? r_out : a;
    float q = 0.f;
    for (int c = lane; c < D; c += 32) {
        float v = (b && !r_out) ? to_f32<T>(a[off + c]) + to_f32<T>(b[off + c]) : to_f32<T>(src[off + c]);
        const float d = v - mean;
        q += d * d;
    }
    const float rstd = rsqrtf(warp_sum(q) / D + eps);
    for (int c = lane; c < D; c += 32) {
        float v = (b && !r_out) ? to_f32<T>(a[off + c]) + to_f32<T>(b[off + c]) : to_f32<T>(src[off + c]);
        y[off + c] = from_f32<T>((v - mean) * rstd * to_f32<T>(gamma[c]) + to_f32<T>(beta[c]));
    }
    if (lane == 0) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
    }
}

// Backward for rows that fit NV 16-byte vectors per lane (D = W * 32 * NV at most).  One warp per row, grid-stride.
// Each lane owns fixed columns: both passes over a row (statistics, then dx) read it from the ring, and the lane's partial
// d(gamma) / d(beta) accumulate in registers over all rows of the warp; they reach the warp's shared-memory slice
// (slot (i*W + j)*32 + lane: conflict-free, in the ring's place) once at the end.  The grid is sized to what is
// resident at once, so every block runs the same number of rounds.  Bound by issue slots next to memory: 16384 x 768 bf16
// with a residual gradient (101 MB) takes 20.1 us on packed pairs, 21.2 us one element at a time, 24.4 us with the rows in
// registers instead of the ring.
template <typename T, int NV>
__global__ void __launch_bounds__(LN_WARPS * 32, NV == 1 ? 4 : 2)
ln_bwd_vec_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                  const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ dres,
                  T* __restrict__ dx, float* __restrict__ partial /*[gridDim.x][2][D]*/, int rows, int D) {
    constexpr int W = VecOf<T>::N, S = NV <= 3 ? LN_STAGES : 2;
    constexpr int SLOTS = NV * W * 32;
    extern __shared__ uint4 ring[];   // [LN_WARPS][S][3][NV][32] (x, dy, residual gradient); at the end [LN_WARPS][2][SLOTS] floats
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = D / W;
    const unsigned step = gridDim.x * LN_WARPS, n_rows = rows;
    const int stage = 3 * NV * 32;
    uint4* mine = ring + warp * S * stage + lane;
    auto fetch = [&](unsigned row, int s) {
        if (row < n_rows) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int v = lane + 32 * i;
                if (v < nvec) {
                    const long long at = (long long)row * D + v * W;
                    ring_copy(mine + s * stage + i * 32, x + at);
                    ring_copy(mine + s * stage + (NV + i) * 32, dy + at);
                    if (dres) ring_copy(mine + s * stage + (2 * NV + i) * 32, dres + at);
                }
            }
        }
        ring_commit();
    };
    F32x2 adg[NV][W / 2], adb[NV][W / 2];
    uint4 graw[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = lane + 32 * i;
        graw[i] = make_uint4(0, 0, 0, 0);
        if (v < nvec) graw[i] = *reinterpret_cast<const uint4*>(gamma + v * W);
#pragma unroll
        for (int j = 0; j < W / 2; ++j) adg[i][j] = adb[i][j] = f2_splat(0.f);
    }
    unsigned row = blockIdx.x * LN_WARPS + warp;
#pragma unroll
    for (int s = 0; s < S - 1; ++s) fetch(row_ahead(row, step, s), s);
    float mu_next = row < n_rows ? mean[row] : 0.f, rs_next = row < n_rows ? rstd[row] : 0.f;
    for (int s = 0; row < n_rows; row += step, s = s + 1 == S ? 0 : s + 1) {
        fetch(row_ahead(row, step, S - 1), s == 0 ? S - 1 : s - 1);
        const float mu = mu_next, rs = rs_next;
        if (row + step < n_rows) { mu_next = mean[row + step]; rs_next = rstd[row + step]; }
        ring_wait<S - 1>();
        const uint4* in = mine + s * stage;
        const long long off = (long long)row * D;
        const F32x2 nmu2 = f2_splat(-mu), rs2 = f2_splat(rs);
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (lane + 32 * i < nvec) {
                float xv[W], dv[W], g[W];
                unpack_raw<T>(in[i * 32], xv);
                unpack_raw<T>(in[(NV + i) * 32], dv);
                unpack_raw<T>(graw[i], g);
#pragma unroll
                for (int j = 0; j < W; j += 2) {
                    const F32x2 xh = f2_mul(f2_add(f2_pack(xv[j], xv[j + 1]), nmu2), rs2), dy2 = f2_pack(dv[j], dv[j + 1]);
                    const F32x2 d = f2_mul(dy2, f2_pack(g[j], g[j + 1]));
                    float d0, d1, x0, x1;
                    f2_unpack(d, d0, d1);
                    f2_unpack(xh, x0, x1);
                    s1 = s1 + d0 + d1;
                    s2 = fmaf(d1, x1, fmaf(d0, x0, s2));
                    adg[i][j / 2] = f2_fma(dy2, xh, adg[i][j / 2]);
                    adb[i][j / 2] = f2_add(adb[i][j / 2], dy2);
                }
            }
        }
        s1 = warp_sum(s1) / D;
        s2 = warp_sum(s2) / D;
        const F32x2 ns1 = f2_splat(-s1), ns2 = f2_splat(-s2);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = lane + 32 * i;
            if (v < nvec) {
                float xv[W], dv[W], g[W], o[W];
                unpack_raw<T>(in[i * 32], xv);
                unpack_raw<T>(in[(NV + i) * 32], dv);
                unpack_raw<T>(graw[i], g);
#pragma unroll
                for (int j = 0; j < W; j += 2) {
                    const F32x2 xh = f2_mul(f2_add(f2_pack(xv[j], xv[j + 1]), nmu2), rs2);
                    const F32x2 d = f2_mul(f2_pack(dv[j], dv[j + 1]), f2_pack(g[j], g[j + 1]));
                    f2_unpack(f2_mul(rs2, f2_add(f2_fma(xh, ns2, d), ns1)), o[j], o[j + 1]);
                }
                if (dres) {
                    float t[W];
                    unpack_raw<T>(in[(2 * NV + i) * 32], t);
                    row_add(o, t);
                }
                store_vec<T>(dx + off + v * W, o);
            }
        }
    }
    // the warp's partial sums go to its shared-memory slice once, after every warp's last row
    ring_wait<0>();
    __syncthreads();
    float* sm = reinterpret_cast<float*>(ring);
    float* wdg = sm + (size_t)warp * 2 * SLOTS;
    float* wdb = wdg + SLOTS;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
#pragma unroll
        for (int j = 0; j < W; j += 2) {
            f2_unpack(adg[i][j / 2], wdg[(i * W + j) * 32 + lane], wdg[(i * W + j + 1) * 32 + lane]);
            f2_unpack(adb[i][j / 2], wdb[(i * W + j) * 32 + lane], wdb[(i * W + j + 1) * 32 + lane]);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * D; c += blockDim.x) {
        const int which = c >= D, col = c - which * D;
        const int v = col / W, j = col % W;
        const int slot = ((v >> 5) * W + j) * 32 + (v & 31);
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < LN_WARPS; ++w) s += sm[(size_t)w * 2 * SLOTS + which * SLOTS + slot];
        partial[(long long)blockIdx.x * 2 * D + c] = s;
    }
}

// Fallback for row lengths the vector kernel does not take (not a multiple of the vector width, or too long):
// same arithmetic with scalar accesses, per-warp partial d(gamma) / d(beta) rows in shared memory.
template <typename T>
__global__ void __launch_bounds__(LN_WARPS * 32)
ln_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
              const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ dres,
              T* __restrict__ dx, float* __restrict__ partial /*[gridDim.x][2][D]*/, int rows, int D) {
    extern __shared__ float sm[];     // [LN_WARPS][2][D]
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = threadIdx.x; c < LN_WARPS * 2 * D; c += blockDim.x) sm[c] = 0.f;
    __syncthreads();
    for (int row = blockIdx.x * LN_WARPS + warp; row < rows; row += gridDim.x * LN_WARPS) {
        const long long off = (long long)row * D;
        const float mu = mean[row], rs = rstd[row];
        float s1 = 0.f, s2 = 0.f;
        for (int c = lane; c < D; c += 32) {
            const float xh = (to_f32<T>(x[off + c]) - mu) * rs;
            const float dv = to_f32<T>(dy[off + c]);
            const float d = dv * to_f32<T>(gamma[c]);
            s1 += d;
            s2 += d * xh;
            sm[(warp * 2 + 0) * D + c] += dv * xh;
            sm[(warp * 2 + 1) * D + c] += dv;
        }
        s1 = warp_sum(s1) / D;
        s2 = warp_sum(s2) / D;
        for (int c = lane; c < D; c += 32) {
            const float xh = (to_f32<T>(x[off + c]) - mu) * rs;
            const float d = to_f32<T>(dy[off + c]) * to_f32<T>(gamma[c]);
            float o = rs * (d - s1 - xh * s2);
            if (dres) o += to_f32<T>(dres[off + c]);
            dx[off + c] = from_f32<T>(o);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * D; c += blockDim.x) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < LN_WARPS; ++w) s += sm[w * 2 * D + c];
        partial[(long long)blockIdx.x * 2 * D + c] = s;
    }
}

// dgamma[c] (+)= sum_b partial[b][0][c];  dbeta[c] (+)= sum_b partial[b][1][c]
// Block (16 columns x NG block-groups): each thread sums every NG-th partial, then a fixed-order shared-memory reduction
// over the groups (deterministic).  The time is that of a thread's chain of loads, so it is kept to a handful.
template <typename T, int NG>
__global__ void __launch_bounds__(16 * NG)
ln_bwd_finalize_kernel(const float* __restrict__ partial, int nblocks, int D, T* dgamma, T* dbeta, int accumulate) {
    __shared__ float sm[NG][17];
    pdl_wait();
    const int cx = threadIdx.x & 15, ry = threadIdx.x >> 4;
    const int c = blockIdx.x * 16 + cx;
    float s = 0.f;
    if (c < 2 * D) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;      // independent chains: the loads of four blocks overlap
        int b = ry;
        if constexpr (NG == 64) {                          // many partials: rounds without a test per load
            for (; b + 3 * NG < nblocks; b += 4 * NG) {
                s0 += partial[(long long)b * 2 * D + c];
                s1 += partial[(long long)(b + NG) * 2 * D + c];
                s2 += partial[(long long)(b + 2 * NG) * 2 * D + c];
                s3 += partial[(long long)(b + 3 * NG) * 2 * D + c];
            }
            for (; b < nblocks; b += NG) s0 += partial[(long long)b * 2 * D + c];
        } else {                                           // few: the last round's loads are in flight together too
            for (; b < nblocks; b += 4 * NG) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = b + k * NG < nblocks ? partial[(long long)(b + k * NG) * 2 * D + c] : 0.f;
                s0 += v[0];
                s1 += v[1];
                s2 += v[2];
                s3 += v[3];
            }
        }
        s = (s0 + s1) + (s2 + s3);
    }
    sm[ry][cx] = s;
    __syncthreads();
    if (NG == 64) {
        if (ry < 4 && c < 2 * D) {                         // 64 groups -> 4
            float t = 0.f;
#pragma unroll
            for (int r = 0; r < NG / 4; ++r) t += sm[ry * (NG / 4) + r][cx];
            sm[ry * (NG / 4)][cx] = t;
        }
        __syncthreads();
    }
    if (ry == 0 && c < 2 * D) {
        float t = 0.f;
        if (NG == 64) {
            t = (sm[0][cx] + sm[NG / 4][cx]) + (sm[NG / 2][cx] + sm[3 * NG / 4][cx]);
        } else {
#pragma unroll
            for (int r = 0; r < NG; ++r) t += sm[r][cx];
        }
        T* dst = (c < D) ? dgamma + c : dbeta + (c - D);
        *dst = from_f32<T>(accumulate ? to_f32<T>(*dst) + t : t);
    }
}
template <typename T>
int ln_bwd_finalize(const float* partial, int nblocks, int D, T* dgamma, T* dbeta, int accumulate, cudaStream_t st) {
    // Blocks of 1024 threads cost more than they save while 16 groups read everything in two rounds (whole backward, 768
    // bf16 columns, us with 16 / 64 groups: 32 partials 5.6 / 5.8, 128 partials 5.9 / 6.3).
    const bool many = nblocks > 128;
    auto kernel = many ? ln_bwd_finalize_kernel<T, 64> : ln_bwd_finalize_kernel<T, 16>;
    CME_CUDA(cme_launch_dependent(kernel, dim3(cme_cdiv(2 * D, 16)), dim3(many ? 1024 : 256), 0, st, partial, nblocks, D, dgamma,
                                  dbeta, accumulate));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// Every operand (null ones aside) starts on a 16-byte boundary.
template <typename... P> bool aligned16(P... p) { return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0; }

// Blocks of `kernel` that are resident on the current device at once with `smem` bytes each.
template <typename K> int resident_blocks(K kernel, size_t smem, int* out) {
    int per_sm = 0, num_sms = 0;
    const int rc = cme_num_sms(&num_sms);
    if (rc) return rc;
    if (smem > 48 * 1024) CME_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CME_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, LN_WARPS * 32, smem));
    *out = num_sms * (per_sm > 0 ? per_sm : 1);
    return CME_OK;
}
// Blocks for `rows`: what is resident at once, evened out so that every block runs the same number of rounds.
inline int even_grid(int rows, int resident) {
    const int nb = cme_cdiv(rows, LN_WARPS);
    return nb > resident ? cme_cdiv(nb, cme_cdiv(nb, resident)) : nb;
}

template <typename T, int NV>
int ln_fwd_vec_launch(const T* a, const T* b, T* r, const T* g, const T* be, T* y, float* mean, float* rstd, int rows, int D,
                      float eps, cudaStream_t st) {
    // bf16 row by row whatever the size (with residual, us ring / row by row, from memory: 2048 x 768 3.7 / 3.5, 4096 x 768 6.6 / 5.8,
    // 8192 x 384 6.7 / 6.1, 16384 x 1024 25.0 / 22.3; from L2: 8192 x 1024 10.8 / 8.2, 65536 x 1024 98 / 82).  fp32 rows are twice as
    // many words a lane, and there the ring pays while the grid is a round or two (2048 x 512, residual, row by row / ring 4.5 / 4.4),
    // and from memory up to 90 MB.  Between the two more warps are worth more (8192 x 384 from L2 4.0 / 5.2), and beyond L2 as well
    // (65536 x 384, residual, 64 / 73).
    const double in_bytes = (double)rows * D * sizeof(T) * (b ? 2 : 1);
    if (sizeof(T) == 2 || (rows >= 8192 && (in_bytes <= 36e6 || in_bytes >= 90e6))) {
        CME_CUDA(cme_launch_dependent(ln_fwd_row_kernel<T, NV>, dim3(cme_cdiv(rows, LN_WARPS)), dim3(LN_WARPS * 32), 0, st, a, b,
                                      r, g, be, y, mean, rstd, rows, D, eps));
        CME_LAUNCH_CHECK();
        return CME_OK;
    }
    if constexpr (sizeof(T) == 4) {
        const size_t smem = (size_t)LN_WARPS * LN_STAGES * (b ? 2 : 1) * NV * 512;
        auto k = ln_fwd_vec_kernel<T, NV>;
        static int resident[2][CME_MAX_DEVICES];       // [residual][device]
        int dev = 0;
        CME_CUDA(cudaGetDevice(&dev));
        int& res = resident[b != nullptr][dev % CME_MAX_DEVICES];
        if (!res) {
            int n = 0;
            const int rc = resident_blocks(k, smem, &n);
            if (rc) return rc;
            res = n;
        }
        CME_CUDA(cme_launch_dependent(k, dim3(even_grid(rows, res)), dim3(LN_WARPS * 32), smem, st, a, b, r, g, be, y, mean, rstd,
                                      rows, D, eps));
        CME_LAUNCH_CHECK();
    }
    return CME_OK;
}

template <typename T>
int ln_fwd_t(const void* a, const void* b, void* r, const void* g, const void* be, void* y, float* mean, float* rstd,
             int rows, int D, float eps, cudaStream_t st) {
    constexpr int W = VecOf<T>::N;
    if (D % W == 0 && D / W <= 32 * LN_MAX_VEC && aligned16(a, b, r, g, be, y)) {
        const int nv = cme_cdiv(D / W, 32);
#define CME_LN_NV(N) ln_fwd_vec_launch<T, N>((const T*)a, (const T*)b, (T*)r, (const T*)g, (const T*)be, (T*)y, mean, rstd, \
                                             rows, D, eps, st)
        return nv == 1 ? CME_LN_NV(1) : nv == 2 ? CME_LN_NV(2) : nv == 3 ? CME_LN_NV(3) : CME_LN_NV(4);
#undef CME_LN_NV
    }
    CME_CUDA(cme_launch_dependent(ln_fwd_kernel<T>, dim3(cme_cdiv(rows, LN_WARPS)), dim3(LN_WARPS * 32), 0, st, (const T*)a,
                                  (const T*)b, (T*)r, (const T*)g, (const T*)be, (T*)y, mean, rstd, rows, D, eps));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

template <typename T, int NV>
int ln_bwd_vec_launch(const T* dy, const T* x, const T* g, const float* mean, const float* rstd, const T* dres, T* dx,
                      float* scratch, int max_blocks, int rows, int D, int* used_blocks, cudaStream_t st) {
    constexpr size_t ring = (size_t)LN_WARPS * (NV <= 3 ? LN_STAGES : 2) * 3 * NV * 512;
    constexpr size_t sums = (size_t)LN_WARPS * 2 * NV * VecOf<T>::N * 32 * sizeof(float);
    constexpr size_t smem = ring > sums ? ring : sums;
    auto k = ln_bwd_vec_kernel<T, NV>;
    static int resident[CME_MAX_DEVICES];
    int dev = 0;
    CME_CUDA(cudaGetDevice(&dev));
    int& res = resident[dev % CME_MAX_DEVICES];
    if (!res) {
        int n = 0;
        const int rc = resident_blocks(k, smem, &n);
        if (rc) return rc;
        res = n;
    }
    const int nb = even_grid(rows, res < max_blocks ? res : max_blocks);     // (the blocks' sums have room for max_blocks)
    CME_CUDA(cme_launch_dependent(k, dim3(nb), dim3(LN_WARPS * 32), smem, st, dy, x, g, mean, rstd, dres, dx, scratch, rows,
                                  D));
    *used_blocks = nb;
    return CME_OK;
}

template <typename T>
int ln_bwd_t(const void* dy, const void* x, const void* g, const float* mean, const float* rstd, const void* dres,
             void* dx, void* dgamma, void* dbeta, float* scratch, int nblocks, int rows, int D, int accumulate,
             cudaStream_t st, cudaStream_t fin_st = nullptr, cudaEvent_t fin_ev = nullptr) {
    constexpr int W = VecOf<T>::N;
    const bool vec = D % W == 0 && D / W <= 32 * LN_MAX_VEC && aligned16(dy, x, g, dres, dx);
    if (vec) {
        const int nv = cme_cdiv(D / W, 32);
        int rc;
#define CME_LN_NV(N) rc = ln_bwd_vec_launch<T, N>((const T*)dy, (const T*)x, (const T*)g, mean, rstd, (const T*)dres, \
                                                 (T*)dx, scratch, nblocks, rows, D, &nblocks, st)
        if (nv == 1) CME_LN_NV(1); else if (nv == 2) CME_LN_NV(2); else if (nv == 3) CME_LN_NV(3); else CME_LN_NV(4);
#undef CME_LN_NV
        if (rc) return rc;
    } else {
        const size_t smem = (size_t)LN_WARPS * 2 * D * sizeof(float);
        auto k = ln_bwd_kernel<T>;
        if (smem > 48 * 1024) CME_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        CME_CUDA(cme_launch_dependent(k, dim3(nblocks), dim3(LN_WARPS * 32), smem, st, (const T*)dy, (const T*)x,
                                      (const T*)g, mean, rstd, (const T*)dres, (T*)dx, scratch, rows, D));
    }
    CME_LAUNCH_CHECK();
    if (fin_st != nullptr && fin_st != st) {       // the weight gradients are finished on another stream
        CME_CUDA(cudaEventRecord(fin_ev, st));
        CME_CUDA(cudaStreamWaitEvent(fin_st, fin_ev, 0));
        st = fin_st;
    }
    return ln_bwd_finalize<T>(scratch, nblocks, D, (T*)dgamma, (T*)dbeta, accumulate, st);
}

}  // namespace

// y = LN(a + b); b, r_out, mean, rstd may be null.
CME_API int cme_layernorm_fwd(int dtype, const void* a, const void* b, void* r_out, const void* gamma,
                              const void* beta, void* y, float* mean, float* rstd, int rows, int D, float eps,
                              void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && D > 0, CME_ERR_SHAPE, "layernorm: empty input");
    return dtype == CME_BF16 ? ln_fwd_t<__nv_bfloat16>(a, b, r_out, gamma, beta, y, mean, rstd, rows, D, eps, st)
                             : ln_fwd_t<float>(a, b, r_out, gamma, beta, y, mean, rstd, rows, D, eps, st);
}

// Number of partial blocks the backward uses for `rows`; scratch must hold blocks * 2 * D floats.
CME_API int cme_layernorm_bwd_blocks(int rows) {
    int b = cme_cdiv(rows, LN_WARPS);
    return b < 592 ? b : 592;
}

// dx = LN'(dy) [+ dres]; dgamma/dbeta (+)= column sums.  `scratch`: cme_layernorm_bwd_blocks(rows)*2*D floats.
CME_API int cme_layernorm_bwd(int dtype, const void* dy, const void* x, const void* gamma, const float* mean,
                              const float* rstd, const void* dres, void* dx, void* dgamma, void* dbeta,
                              float* scratch, int rows, int D, int accumulate, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && D > 0, CME_ERR_SHAPE, "layernorm: empty input");
    CME_REQUIRE((size_t)LN_WARPS * 2 * D * 4 <= 200 * 1024, CME_ERR_LIMIT, "layernorm backward: D too large (%d)", D);
    const int nb = cme_layernorm_bwd_blocks(rows);
    return dtype == CME_BF16
               ? ln_bwd_t<__nv_bfloat16>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, nb, rows, D,
                                         accumulate, st)
               : ln_bwd_t<float>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, nb, rows, D, accumulate,
                                 st);
}

// Same, with the small kernel that sums the per-block partial d(gamma) / d(beta) on `fin_stream` (ordered after the main
// kernel through `fin_event`, a cudaEvent_t of the caller): nothing on `stream` needs those sums, so the chain of
// activation-gradient work on `stream` does not wait for them.  `scratch` must stay untouched until that kernel has run.
CME_API int cme_layernorm_bwd_split(int dtype, const void* dy, const void* x, const void* gamma, const float* mean,
                                    const float* rstd, const void* dres, void* dx, void* dgamma, void* dbeta,
                                    float* scratch, int rows, int D, int accumulate, void* stream, void* fin_stream,
                                    void* fin_event) {
    cudaStream_t st = (cudaStream_t)stream;
    CME_REQUIRE(rows > 0 && D > 0, CME_ERR_SHAPE, "layernorm: empty input");
    CME_REQUIRE((size_t)LN_WARPS * 2 * D * 4 <= 200 * 1024, CME_ERR_LIMIT, "layernorm backward: D too large (%d)", D);
    CME_REQUIRE(fin_stream == nullptr || fin_stream == stream || fin_event != nullptr, CME_ERR_SHAPE,
                "layernorm backward: a second stream needs an event");
    const int nb = cme_layernorm_bwd_blocks(rows);
    return dtype == CME_BF16
               ? ln_bwd_t<__nv_bfloat16>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, nb, rows, D,
                                         accumulate, st, (cudaStream_t)fin_stream, (cudaEvent_t)fin_event)
               : ln_bwd_t<float>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, nb, rows, D, accumulate,
                                 st, (cudaStream_t)fin_stream, (cudaEvent_t)fin_event);
}
