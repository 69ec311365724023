// Fused flash-style attention on the 5th-generation tensor cores (head size 64, bf16, causal or not, both
// head layouts): scores, probabilities (forward) and output partials live in TMEM, nothing of size T x T reaches
// global memory, only the per-row log-sum-exp is saved for backward.
//
// Replaces the reference's production attention -- two strided-batched GEMMs around an in-place softmax
// with P, dP and dS materialised as [B*H, T, T] buffers, and four more batched GEMMs plus a dS kernel in
// backward (FINAL_CLEAN_CODE_/src/kernels/attention.cu:138-200, 253-328).
//
// Forward, per CTA = one (batch, head) and 128 queries, 64 keys at a time; 4 softmax warps (thread = query row) + 1 warp whose
// lane 0 issues TMA loads and tcgen05.mma:
//     S_j = Q K_j^T (TMEM) -> registers -> online softmax with a lazily raised reference maximum
//     -> P_j (bf16 pairs) written over S_j with tcgen05.st -> O += P_j V_j with the A operand read from tensor memory (P
//     never passes through shared memory; TMEM accumulator, rescaled in place only when the reference maximum is raised)
// Backward, per CTA = one (batch, head) and 128 keys, looping over query blocks:
//     S, dP (TMEM)  ->  P, dS (bf16)  ->  dV += P^T dO_i,  dK += dS^T Q_i (TMEM accumulators),  dQ_i = dS K (TMEM).
//     dQ_i gets a part from every key block that sees query block i.  The parts are added to an fp32 scratch with
//     bulk reduce-adds in whatever order the CTAs arrive (fast; the last bits of dQ depend on the order), and
//     either (dq_mode 0, the default) the launch clears the scratch first and a small kernel scales and casts the
//     sums afterwards, or (dq_mode 2) a counter per tile tells the CTA whose part arrived last to do that itself --
//     a spare warp converts the tile and writes zeros back, so no clearing or conversion pass runs; the query
//     blocks are then walked downwards so that the finishing work spreads over the CTAs.  Still slower: every reduce-add
//     has to complete before its part is counted in, and one warp converts a 32 KB tile.  Deterministic form (dq_mode 1): the
//     highest key block stores its part, each lower one adds its own when the tile's counter says it is its turn,
//     and key block 0, whose turn is last, adds the sum to its part in registers, scales, casts and writes dQ --
//     bit-reproducible, no clearing or conversion pass, but the chain of turns makes CTAs wait for one another.  Whole backward in
//     modes 0 / 1 / 2: 16 x 12 heads x 1024 tokens 146 / 259 / 276 us causal, 227 / 473 / 369 all keys; 64 x 6 x 256 causal
//     48 / 69 / 98.
// Grids that fill the GPU take small CTAs, several to an SM; others, and the backward's modes 1 and 2, 128 x 128 blocks.
// Every mbarrier wait is bounded; on expiry the CTA flags the status word, frees TMEM and returns.
#include "attention.h"
#include "sm100_ptx.cuh"

#include <cuda.h>
#include <mutex>

using namespace sm100;

int* cme_attn_status_ptr();

namespace {

constexpr int HD = 64;
constexpr int BQ = 128;            // rows per tile (queries in forward, keys in backward)
constexpr int BKV = 128;           // streamed rows per step
constexpr int TILE_BYTES = 128 * HD * 2;        // 16 KB: 128 rows x 128 bytes
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
        : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(m)),
                 "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* m, const void* src, int c0, int c1, int c2) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(m)),
                 "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

// The largest of three in one instruction.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

// A descriptor whose start address is `bytes` further than that of `base` (the address field counts 16-byte
// units and never carries out of its 14 bits for shared-memory offsets), so the issuing thread spends one add
// per operand instead of re-encoding the descriptor for each of the ~30 MMAs of a block.
__device__ __forceinline__ uint64_t desc_add(uint64_t base, uint32_t bytes) { return base + (uint64_t)(bytes >> 4); }

// Swizzled position of 16-byte chunk `c` of row `r` inside a [rows x 128 B] tile.
__device__ __forceinline__ uint32_t swz(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

struct FwdParams {
    int T, nh, causal;
    float scale_log2;              // scale * log2(e)
    float* lse;
    int* status;
};

// ------------------------------------------------------------------------------------------------------
// Forward
// ------------------------------------------------------------------------------------------------------
// What bounds it: the chain MMA -> TMEM load -> softmax -> TMEM store -> MMA of a tile (no pipe is busy for half of the time).
// So a CTA is kept small enough for four on an SM: 128 queries, 64 keys at a time, P in the columns that its scores came
// from, 128 TMEM columns, 64 score registers per thread; every scheduler then has four softmax warps of independent chains,
// and a tile's start and end run under the others' work.  16 x 12 heads x 1024 tokens: causal 50.4 us, all keys 80.7 us.  Of the
// 2340 clocks of a block the exponentials take 512 at the least (MUFU), alone; four CTAs in their loops would keep it busy, but a CTA
// spends 5000 clocks starting and ending, so 2.75 are in their loops on average.
// S_{j+1} goes to the columns that P_j V_j reads its A operand from.  PTX orders two MMAs of a thread only if they accumulate in
// the same place, so S_{j+1} is issued once a barrier says that P_j V_j is complete.  Measured without that wait, when this form
// took 57 and 89 us: two CTAs with 128 keys at a time 70 us causal; three with S_{j+1} made under softmax_j 57 and 87 us; a quarter
// of the exponentials as a polynomial on the FMA pipe 58 and 91 us; the query tiles of a head side by side 73 us causal.
// shared: Q 16K | K[2] 16K | V[2] 16K | barriers      (P never passes through shared memory)
constexpr int FWD_BKV = 64;                // keys per step
constexpr int FWD_KV_BYTES = FWD_BKV * HD * 2;
constexpr int FWD_SMEM = TILE_BYTES + 4 * FWD_KV_BYTES + 128;
constexpr int FWD_THREADS = 160;
constexpr int FWD_CTAS_PER_SM = 4;
constexpr int FWD_TMEM_COLS = 128;         // S, then P (bf16 pairs, 32 columns): [0,64)  O accumulator: [64,128)
static_assert(FWD_CTAS_PER_SM * (FWD_SMEM + 1024) <= 228 * 1024, "the forward CTAs must fit one SM's shared memory");
static_assert(FWD_BKV + HD <= FWD_TMEM_COLS && FWD_CTAS_PER_SM * FWD_TMEM_COLS <= 512, "forward TMEM budget: S + O per CTA");
// log2 units: the running maximum is only raised when it grows by > 2^8.  The probability of the key that the reference belongs to
// is 1, which bf16 holds exactly, so the reference decides on the error too: settled after 64 keys the output is 2.055e-3 off its
// 64-bit values (16 x 12 heads x 1024, causal), after 128 keys 2.032e-3.  The rescale then is 1.2 us of the 59 (causal; 8 columns
// at a time 1.5).
constexpr float RESCALE_THRESHOLD = 8.f;

__global__ void __launch_bounds__(FWD_THREADS, FWD_CTAS_PER_SM)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                   const FwdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {             // swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, CME_ERR_SHAPE);
        return;
    }
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + TILE_BYTES;                            // 2 stages
    uint8_t* sV = sK + 2 * FWD_KV_BYTES;                      // 2 stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * FWD_KV_BYTES);
    uint64_t* q_full = bars;                  // 1
    uint64_t* k_full = bars + 1;              // [2]
    uint64_t* v_full = bars + 3;              // [2]
    uint64_t* s_full = bars + 5;              // phase j: S_j is ready and O is complete up to block j - 1
    uint64_t* p_ready = bars + 6;             // S_j read, P_j written over it, O rescaled (128 arrivals)
    uint64_t* p_free = bars + 7;              // P_j V_j complete: S_{j+1} may take the columns of P_j
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // the late (causal: heavy) query tiles of all heads first, so that the last wave is made of the light ones
    const int q0 = (gridDim.y - 1 - blockIdx.y) * BQ;
    const int bh = blockIdx.x, b = bh / p.nh, h = bh % p.nh;
    const int nkv = cme_cdiv_dev(p.causal ? min(q0 + BQ, p.T) : p.T, FWD_BKV);

    auto load_k = [&](int j) {
        mbar_arrive_expect_tx(&k_full[j & 1], FWD_KV_BYTES);
        tma_load_4d(sK + (j & 1) * FWD_KV_BYTES, &tmK, &k_full[j & 1], 0, j * FWD_BKV, h, b);
    };
    auto load_v = [&](int j) {
        mbar_arrive_expect_tx(&v_full[j & 1], FWD_KV_BYTES);
        tma_load_4d(sV + (j & 1) * FWD_KV_BYTES, &tmV, &v_full[j & 1], 0, j * FWD_BKV, h, b);
    };
    if (warp == 4 && elect_one()) {
        *abort_flag = 0;
        mbar_init(q_full, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1); }
        mbar_init(s_full, 1);
        mbar_init(p_ready, 128);
        mbar_init(p_free, 1);
        fence_barrier_init();
        pdl_wait();                                // the first loads run under the TMEM allocation
        mbar_arrive_expect_tx(q_full, TILE_BYTES);
        tma_load_4d(sQ, &tmQ, q_full, 0, q0, h, b);
        load_k(0);
        load_v(0);
        if (nkv > 1) { load_k(1); load_v(1); }
    }
    if (warp == 0) { tmem_alloc(tmem_slot, FWD_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_S = tmem_base, tmem_P = tmem_base, tmem_O = tmem_base + FWD_BKV;
    pdl_wait();        // barrier set-up and TMEM allocation above may overlap the tail of the previous kernel

    if (warp == 4) {
        if (elect_one()) {
            // ---------------- producer + MMA issuer (one thread) ----------------
            constexpr uint32_t idesc_s = make_idesc(1, false, false, BQ, FWD_BKV);   // Q K^T: both K-major
            constexpr uint32_t idesc_o = make_idesc(1, false, true, BQ, HD);         // P V: V is MN-major
            const uint64_t dQ_ = make_smem_desc(smem_u32(sQ), 0, 1024);
            const uint64_t dK0 = make_smem_desc(smem_u32(sK), 0, 1024);
            const uint64_t dV0 = make_smem_desc(smem_u32(sV), FWD_KV_BYTES, 1024);
            auto issue_s = [&](int j) {
                const uint64_t kd = desc_add(dK0, (j & 1) * FWD_KV_BYTES);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_S, desc_add(dQ_, k * 32), desc_add(kd, k * 32), idesc_s, k > 0);
                mma_commit(s_full);
            };
            bool ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(&k_full[0], 0, abort_flag);
            if (ok) { tc_fence_after(); issue_s(0); }
            for (int j = 0; j < nkv && ok; ++j) {
                if (!mbar_wait(p_ready, j & 1, abort_flag)) { ok = false; break; }
                if (!mbar_wait(&v_full[j & 1], (j >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t vd = desc_add(dV0, (j & 1) * FWD_KV_BYTES);
#pragma unroll
                for (int k = 0; k < FWD_BKV / 16; ++k)       // A = P from tensor memory: 16 keys = 8 columns per step
                    mma_f16_ts(tmem_O, tmem_P + k * 8, desc_add(vd, k * 2048), idesc_o, (j > 0 || k > 0));
                if (j + 1 < nkv) {
                    mma_commit(p_free);
                    // S_j has been read, so its MMAs and with them those of P_{j-1} V_{j-1} are complete: refill their tiles while
                    // the product just issued runs
                    if (j + 2 < nkv) load_k(j + 2);
                    if (j >= 1) load_v(j + 1);
                    if (!mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag) ||
                        !mbar_wait(p_free, j & 1, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    issue_s(j + 1);
                } else {
                    mma_commit(s_full);                      // phase nkv: O is complete
                }
            }
            if (!ok) for (int i = 0; i < 2000; ++i) __nanosleep(500);
        }
    } else {
        // ---------------- softmax warps: thread = query row ----------------
        const int row = warp * 32 + lane;                 // 0..127 == TMEM lane
        const int q = q0 + row;
        const uint32_t lane_addr = uint32_t(warp * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                 // reference maximum (log2 units) and running row sum
        bool ok = true;
        for (int j = 0; j < nkv; ++j) {
            if (!mbar_wait(s_full, j & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            uint32_t r[64];
            tmem_ld32(tmem_S + lane_addr, r);
            tmem_ld32(tmem_S + lane_addr + 32, r + 32);
            tmem_wait_ld();
            const int k0 = j * FWD_BKV;
            if ((k0 + FWD_BKV > p.T) || (p.causal && k0 + FWD_BKV - 1 > q0 + warp * 32)) {     // diagonal or ragged block
                // keys [0, lim) of this block are visible to this row: one compare and one select per score
                const int lim = min(p.T, p.causal ? q + 1 : p.T) - k0;
#pragma unroll
                for (int i = 0; i < 64; ++i) r[i] = i < lim ? r[i] : 0xff800000u;     // -inf
            }
            float mx4[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) mx4[c] = __uint_as_float(r[c]);
#pragma unroll
            for (int i = 4; i + 8 <= 64; i += 8) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    mx4[c] = max3(mx4[c], __uint_as_float(r[i + 2 * c]), __uint_as_float(r[i + 2 * c + 1]));
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(mx4[c], __uint_as_float(r[60 + c]));
            float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]);
            mx *= p.scale_log2;                            // scale > 0, so the maximum commutes with it
            // The reference is the maximum of the first 128 keys.  After them it is raised only when it would grow by more than
            // the threshold: the accumulated output then needs a rescale.
            const bool raise = j == 0 || mx > m_ref + (j == 1 ? 0.f : RESCALE_THRESHOLD);
            float alpha = 1.f;
            if (raise) {
                alpha = (m_ref == -INFINITY) ? 0.f : ex2_approx(m_ref - mx);
                m_ref = mx;
            }
            if (j > 0 && __any_sync(0xffffffffu, raise)) {
#pragma unroll 1
                for (int c = 0; c < HD / 16; ++c) {        // 16 columns at a time: the score row stays in registers
                    uint32_t o[16];
                    tmem_ld16(tmem_O + lane_addr + c * 16, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_st16(tmem_O + lane_addr + c * 16, o);
                }
                l *= alpha;
            }
            const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
            // scale-and-shift and the row sum on packed pairs (one instruction per two keys); four independent chains
            const F32x2 sc2 = f2_splat(p.scale_log2), nm2 = f2_splat(-m_use);
            F32x2 sum2[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) sum2[c] = f2_splat(0.f);
            // In passes over 32 keys, so that the 16 scale-and-shifts, then the 32 exponentials, then the sums and
            // stores are each a run of independent instructions (no exponential waits for its own operand or result)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float* x = reinterpret_cast<float*>(r + c * 32);
#pragma unroll
                for (int i = 0; i < 32; i += 2) f2_unpack(f2_fma(f2_pack(x[i], x[i + 1]), sc2, nm2), x[i], x[i + 1]);
#pragma unroll
                for (int i = 0; i < 32; ++i) x[i] = ex2_approx(x[i]);
#pragma unroll
                for (int i = 0; i < 32; i += 2) sum2[(i >> 1) & 3] = f2_add(sum2[(i >> 1) & 3], f2_pack(x[i], x[i + 1]));
                // 32 probabilities = 16 columns of bf16 pairs, straight into the A operand of the P V product
                uint32_t pw[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) pw[i] = f2_to_bf2(x[2 * i], x[2 * i + 1]);
                tmem_st16(tmem_P + lane_addr + c * 16, pw);
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(p_ready);
            float s0, s1;
            f2_unpack(f2_add(f2_add(sum2[0], sum2[1]), f2_add(sum2[2], sum2[3])), s0, s1);
            l += s0 + s1;
        }
        if (ok && mbar_wait(s_full, nkv & 1, abort_flag)) {
            tc_fence_after();
            const float inv = l > 0.f ? 1.f / l : 0.f;
            // stage this warp's 32 rows (every product is complete: the Q tile is free) and store them with one TMA
            uint8_t* stage = sQ + warp * 4096;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) {
                uint32_t t[32];
                tmem_ld32(tmem_O + lane_addr + c * 32, t);
                tmem_wait_ld();
                float* o = reinterpret_cast<float*>(t);
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] *= inv;
#pragma unroll
                for (int g = 0; g < 4; ++g) *reinterpret_cast<uint4*>(stage + swz(lane, c * 4 + g)) = pack8(o + g * 8);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                tma_store_4d(&tmO, stage, 0, q0 + warp * 32, h, b);
                tma_store_commit();
                tma_store_wait_read<0>();         // shared memory may go once the copy engine has read the tile
            }
            if (q < p.T) p.lse[(long long)bh * p.T + q] = (m_ref == -INFINITY) ? -INFINITY : (m_ref + log2f(l)) / LOG2E;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, CME_ERR_TIMEOUT);
    if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem_base, FWD_TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------
// Forward of grids that leave the small CTAs above without neighbours (fwd_wide)
// ------------------------------------------------------------------------------------------------------
// 128 keys per step in a CTA of which two fit an SM: S_j is copied to registers, the tensor core makes S_{j+1} while softmax_j runs, and P
// has columns of its own.  Alone on its SM, a CTA gets through its keys in 0.7 of the time that the small one takes.
// shared: Q 16K | K[3] 48K | V[3] 48K | barriers      (P never passes through shared memory)
constexpr int FWD_WIDE_STAGES = 3;           // a K / V tile is requested two blocks ahead of its use: its ~1200-clock
                                           // latency no longer delays the next S product
constexpr int FWD_WIDE_SMEM = (1 + 2 * FWD_WIDE_STAGES) * TILE_BYTES + 128;   // two CTAs per SM: 2 x (this + 1 KB) <= 228 KB
constexpr int FWD_WIDE_TMEM_COLS = 256;         // S: [0,128)  O accumulator: [128,192)  P (bf16 pairs): [192,256)
static_assert(2 * (FWD_WIDE_SMEM + 1024) <= 228 * 1024, "two forward CTAs must fit one SM's shared memory");
static_assert(128 + HD + BKV / 2 <= FWD_WIDE_TMEM_COLS && 2 * FWD_WIDE_TMEM_COLS <= 512,
              "forward TMEM budget: S + O + P per CTA, two CTAs per SM");

__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {             // swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, CME_ERR_SHAPE);
        return;
    }
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + TILE_BYTES;                            // FWD_WIDE_STAGES stages
    uint8_t* sV = sK + FWD_WIDE_STAGES * TILE_BYTES;            // FWD_WIDE_STAGES stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + FWD_WIDE_STAGES * TILE_BYTES);
    uint64_t* q_full = bars;                  // 1
    uint64_t* kv_full = bars + 1;             // [3]
    uint64_t* kv_empty = bars + 4;            // [3]
    uint64_t* s_full = bars + 7;              // S ready for softmax
    uint64_t* s_free = bars + 8;              // S copied to registers (128 arrivals): the next S may be issued
    uint64_t* p_ready = bars + 9;             // P written to tensor memory, O rescaled (128 arrivals)
    uint64_t* o_full = bars + 10;             // P V accumulated, P consumed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qt = gridDim.x - 1 - blockIdx.x;               // heavy (late) causal tiles first
    const int q0 = qt * BQ;
    const int bh = blockIdx.y, b = bh / p.nh, h = bh % p.nh;
    const int nkv = p.causal ? min((q0 + BQ + BKV - 1) / BKV, (p.T + BKV - 1) / BKV) : (p.T + BKV - 1) / BKV;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(q_full, 1);
        for (int s = 0; s < FWD_WIDE_STAGES; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
        mbar_init(s_full, 1);
        mbar_init(s_free, 128);
        mbar_init(p_ready, 128);
        mbar_init(o_full, 1);
        fence_barrier_init();
    }
    if (warp == 4) { tmem_alloc(tmem_slot, FWD_WIDE_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 128, tmem_P = tmem_base + 128 + HD;
    pdl_wait();        // barrier set-up and TMEM allocation above may overlap the tail of the previous kernel

    if (warp == 4) {
        if (elect_one()) {
            // ---------------- producer + MMA issuer (one thread) ----------------
            constexpr uint32_t idesc_s = make_idesc(1, false, false, 128, 128);   // Q K^T: both K-major
            constexpr uint32_t idesc_o = make_idesc(1, false, true, 128, HD);     // P V: V is MN-major
            bool ok = true;
            mbar_arrive_expect_tx(q_full, TILE_BYTES);
            tma_load_4d(sQ, &tmQ, q_full, 0, q0, h, b);
            auto load_kv = [&](int j) {
                const int st = j % FWD_WIDE_STAGES;
                mbar_arrive_expect_tx(&kv_full[st], 2 * TILE_BYTES);
                tma_load_4d(sK + st * TILE_BYTES, &tmK, &kv_full[st], 0, j * BKV, h, b);
                tma_load_4d(sV + st * TILE_BYTES, &tmV, &kv_full[st], 0, j * BKV, h, b);
            };
            const uint64_t dQ_ = make_smem_desc(smem_u32(sQ), 0, 1024);
            const uint64_t dK0 = make_smem_desc(smem_u32(sK), 0, 1024);
            const uint64_t dV0 = make_smem_desc(smem_u32(sV), TILE_BYTES, 1024);
            auto issue_s = [&](int j) {
                const uint64_t kd = desc_add(dK0, (j % FWD_WIDE_STAGES) * TILE_BYTES);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_S, desc_add(dQ_, k * 32), desc_add(kd, k * 32), idesc_s, k > 0);
                mma_commit(s_full);
            };
            for (int j = 0; j < FWD_WIDE_STAGES && j < nkv; ++j) load_kv(j);
            ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(&kv_full[0], 0, abort_flag);
            if (ok) { tc_fence_after(); issue_s(0); }
            for (int j = 0; j < nkv && ok; ++j) {
                const int st = j % FWD_WIDE_STAGES;
                if (j >= 1 && j + 2 < nkv) {
                    // the stage that block j - 1 used is refilled with block j + 2: its P V product was issued one
                    // block ago, so this wait does not hold anything up
                    if (!mbar_wait(&kv_empty[(j - 1) % FWD_WIDE_STAGES], ((j - 1) / FWD_WIDE_STAGES) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    load_kv(j + 2);
                }
                if (j + 1 < nkv) {
                    // S_j sits in registers now: the tensor core computes S_{j+1} while softmax_j runs
                    if (!mbar_wait(s_free, j & 1, abort_flag) ||
                        !mbar_wait(&kv_full[(j + 1) % FWD_WIDE_STAGES], ((j + 1) / FWD_WIDE_STAGES) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    issue_s(j + 1);
                }
                if (!mbar_wait(p_ready, j & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t vd = desc_add(dV0, st * TILE_BYTES);
#pragma unroll
                for (int k = 0; k < BKV / 16; ++k)       // A = P from tensor memory: 16 keys = 8 columns per step
                    mma_f16_ts(tmem_O, tmem_P + k * 8, desc_add(vd, k * 2048), idesc_o, (j > 0 || k > 0));
                mma_commit(o_full);
                mma_commit(&kv_empty[st]);
            }
            if (!ok) for (int i = 0; i < 2000; ++i) __nanosleep(500);
        }
    } else {
        // ---------------- softmax warps: thread = query row ----------------
        const int row = warp * 32 + lane;                 // 0..127 == TMEM lane
        const int q = q0 + row;
        const uint32_t lane_addr = uint32_t(warp * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                 // reference maximum (log2 units) and running row sum
        bool ok = true;
        for (int j = 0; j < nkv && ok; ++j) {
            if (!mbar_wait(s_full, j & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            uint32_t r[128];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(tmem_S + lane_addr + c * 32, r + c * 32);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(s_free);
            const int k0 = j * BKV;
            if ((k0 + BKV > p.T) || (p.causal && k0 + BKV - 1 > q0)) {        // diagonal or ragged block
                // keys [0, lim) of this block are visible to this row: one compare and one select per score
                const int lim = min(p.T, p.causal ? q + 1 : p.T) - k0;
#pragma unroll
                for (int i = 0; i < 128; ++i) r[i] = i < lim ? r[i] : 0xff800000u;     // -inf
            }
            // eight independent chains (a single one would be 128 dependent operations long)
            float mx8[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) mx8[c] = __uint_as_float(r[c]);
#pragma unroll
            for (int i = 8; i < 128; ++i) mx8[i & 7] = fmaxf(mx8[i & 7], __uint_as_float(r[i]));
            float mx = fmaxf(fmaxf(fmaxf(mx8[0], mx8[1]), fmaxf(mx8[2], mx8[3])),
                             fmaxf(fmaxf(mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])));
            mx *= p.scale_log2;                            // scale > 0, so the maximum commutes with it
            // Raise the reference maximum only when it would grow by more than the threshold: the accumulated
            // output then needs a rescale, which is rare after the first blocks.
            const bool raise = (j == 0) ? true : (mx > m_ref + RESCALE_THRESHOLD);
            float alpha = 1.f;
            if (raise) {
                alpha = (m_ref == -INFINITY) ? 0.f : ex2_approx(m_ref - mx);
                m_ref = mx;
            }
            if (j > 0) {
                // the previous P V product must be complete before P is overwritten or O is rescaled
                if (!mbar_wait(o_full, (j - 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                if (__any_sync(0xffffffffu, raise)) {
#pragma unroll 1
                    for (int c = 0; c < HD / 16; ++c) {       // 16 columns at a time: the score row stays in registers
                        uint32_t o[16];
                        tmem_ld16(tmem_O + lane_addr + c * 16, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st16(tmem_O + lane_addr + c * 16, o);
                    }
                    tmem_wait_st();
                }
                l *= alpha;
            }
            const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
            // scale-and-shift and the row sum on packed pairs (one instruction per two keys); four independent chains
            const F32x2 sc2 = f2_splat(p.scale_log2), nm2 = f2_splat(-m_use);
            F32x2 sum2[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) sum2[c] = f2_splat(0.f);
            // In passes over 32 keys, so that the 16 scale-and-shifts, then the 32 exponentials, then the sums and
            // stores are each a run of independent instructions (no exponential waits for its own operand or result)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float* x = reinterpret_cast<float*>(r + c * 32);
#pragma unroll
                for (int i = 0; i < 32; i += 2) f2_unpack(f2_fma(f2_pack(x[i], x[i + 1]), sc2, nm2), x[i], x[i + 1]);
#pragma unroll
                for (int i = 0; i < 32; ++i) x[i] = ex2_approx(x[i]);
#pragma unroll
                for (int i = 0; i < 32; i += 2) sum2[(i >> 1) & 3] = f2_add(sum2[(i >> 1) & 3], f2_pack(x[i], x[i + 1]));
                // 32 probabilities = 16 columns of bf16 pairs, straight into the A operand of the P V product
                uint32_t pw[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) pw[i] = f2_to_bf2(x[2 * i], x[2 * i + 1]);
                tmem_st16(tmem_P + lane_addr + c * 16, pw);
            }
            tmem_wait_st();
            {
                float s0, s1;
                f2_unpack(f2_add(f2_add(sum2[0], sum2[1]), f2_add(sum2[2], sum2[3])), s0, s1);
                l += s0 + s1;
            }
            tc_fence_before();
            mbar_arrive(p_ready);
        }
        if (ok && nkv > 0) {
            if (mbar_wait(o_full, (nkv - 1) & 1, abort_flag)) {
                tc_fence_after();
                float o[HD];
#pragma unroll
                for (int c = 0; c < HD / 32; ++c) {
                    uint32_t t[32];
                    tmem_ld32(tmem_O + lane_addr + c * 32, t);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[c * 32 + i] = __uint_as_float(t[i]);
                }
                const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
                for (int i = 0; i < HD; ++i) o[i] *= inv;
                // stage this warp's 32 rows (every product is complete and no load is in flight: the first K stage is
                // free) and store them with one TMA tile store
                uint8_t* stage = sK + warp * 4096;
#pragma unroll
                for (int g = 0; g < 8; ++g) *reinterpret_cast<uint4*>(stage + swz(lane, g)) = pack8(o + g * 8);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    tma_store_4d(&tmO, stage, 0, q0 + warp * 32, h, b);
                    tma_store_commit();
                    tma_store_wait_read<0>();         // shared memory may go once the copy engine has read the tile
                }
                if (q < p.T) p.lse[(long long)bh * p.T + q] = (m_ref == -INFINITY) ? -INFINITY : (m_ref + log2f(l)) / LOG2E;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, CME_ERR_TIMEOUT);
    if (warp == 4) { tc_fence_after(); tmem_dealloc(tmem_base, FWD_WIDE_TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------
// Backward
// ------------------------------------------------------------------------------------------------------
// CTA = one (batch, head) and 128 keys, walking over blocks of 64 queries; two CTAs per SM, so that the serial chain of one
// (MMA -> TMEM load -> arithmetic -> MMA), its start and its end run under the other's work.  The scores are computed
// transposed (thread = key row, columns = queries):
//     S^T = K Q_i^T,  dP^T = V dO_i^T (TMEM)  ->  P^T, dS^T (bf16)
//     dV += P^T dO_i,  dK += dS^T Q_i  with P^T and dS^T as A operands from TMEM, written over the scores they came from
//     dQ_i = dS K, whose A operand is the copy of dS^T in shared memory read transposed; its accumulator takes dP^T's place
// so P never passes through shared memory and 256 TMEM columns and 106 KB of shared memory are enough.
// The parts that the key blocks contribute to dQ_i are added to an fp32 scratch by bulk reduce-adds in arrival order; the
// launch clears the scratch beforehand and dq_convert_kernel scales and casts the sums.
// What bounds it: the chain of a block (two round trips to the tensor pipe, 3450 clocks, hidden by one other CTA only): 1500 from S^T
// to dS^T, the same until the next S^T.  The tensor pipe is busy for 41 % of the time, issue slots 31 %.
// 16 x 12 heads x 1024 tokens: causal 129 us, all keys 209 us (135 and 229 with dP^T made before S^T, arithmetic on the statistics as
// they are loaded, and reduce-adds awaited after each block).
// dS^T and the fp32 staging of the dQ that is made from it share a buffer, of which there are two: a block's tile is stored once
// the reduce-adds of two blocks ago have been read.
// shared: K 16K | V 16K | Q[3] 24K | dO[2] 16K | dS^T, then dQ staging [2] 32K | row statistics[2] 1K | barriers
constexpr int BWD_BQ = 64;                 // queries per step
constexpr int BWD_Q_BYTES = BWD_BQ * HD * 2;
constexpr int BWD_Q_STAGES = 3, BWD_DO_STAGES = 2;
constexpr int BWD_STAT_FLOATS = 2 * BWD_BQ;           // -log-sum-exp (log2 units) and -delta of a block's queries
constexpr int BWD_SMEM = 4 * TILE_BYTES + (BWD_Q_STAGES + BWD_DO_STAGES) * BWD_Q_BYTES + 2 * BWD_STAT_FLOATS * 4 + 192;
constexpr int BWD_MMA_WARP = 8;            // warps 0..7 compute, warp 8 issues TMA loads and MMA,
constexpr int BWD_STORE_WARP = 9;          // warp 9 issues the dQ reduce-adds
constexpr int BWD_THREADS = 10 * 32;
constexpr int BWD_TMEM_COLS = 256;         // S^T, then P^T and dS^T [0,64)   dP^T, then dQ [64,128)   dV [128,192)   dK [192,256)
static_assert(2 * (BWD_SMEM + 1024) <= 228 * 1024, "two backward CTAs must fit one SM's shared memory");
static_assert(2 * BWD_BQ + 2 * HD <= BWD_TMEM_COLS && 2 * BWD_TMEM_COLS <= 512, "backward TMEM budget, two CTAs per SM");

struct BwdParams {
    int T, nh, causal;
    float scale, scale_log2;
    const float* lse;
    const float* delta;
    __nv_bfloat16* dk; __nv_bfloat16* dv;
    long long sb, sh, st;          // strides of dK / dV
    int* status;
};

__global__ void __launch_bounds__(BWD_THREADS, 2)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmdQ, const BwdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, CME_ERR_SHAPE);
        return;
    }
    uint8_t* sK = smem;
    uint8_t* sV = sK + TILE_BYTES;
    uint8_t* sQ = sV + TILE_BYTES;
    uint8_t* sdO = sQ + BWD_Q_STAGES * BWD_Q_BYTES;
    uint8_t* sX = sdO + BWD_DO_STAGES * BWD_Q_BYTES;      // [2 buffers]: dS^T [128 keys][64 queries = 128 B], then
                                                          // dQ [2 column atoms][64 query rows][128 B]
    float* stats = reinterpret_cast<float*>(sX + 2 * TILE_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(stats + 2 * BWD_STAT_FLOATS);
    uint64_t* kv_full = bars;
    uint64_t* q_full = bars + 1;               // [3]
    uint64_t* do_full = bars + 4;              // [2]
    uint64_t* s_full = bars + 6;               // S^T of a query block is in TMEM
    uint64_t* dp_full = bars + 7;              // dP^T too
    uint64_t* p_ready = bars + 8;              // S^T, dP^T read; P^T, dS^T written; the next statistics stored (256 arrivals)
    uint64_t* dq_full = bars + 9;              // dQ of a query block complete
    uint64_t* dq_free = bars + 10;             // dQ in registers (256 arrivals): dP^T may overwrite it
    uint64_t* in_free = bars + 11;             // dV, dK accumulated: P^T and dS^T, the block's Q and dO tiles may be overwritten
    uint64_t* dqs_full = bars + 12;            // [2] dQ staging written (256 arrivals)
    uint64_t* dqs_free = bars + 14;            // [2] dQ staging read by the reduce-add
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // the key blocks that the most queries see (causal: the lowest) of all heads first
    const int k0 = blockIdx.y * BKV;
    const int bh = blockIdx.x, b = bh / p.nh, h = bh % p.nh;
    const int q_begin = p.causal ? k0 : 0;
    const int n_it = cme_cdiv_dev(p.T - q_begin, BWD_BQ);          // >= 1: k0 < T

    auto load_q = [&](int it) {
        const int s = it % BWD_Q_STAGES;
        mbar_arrive_expect_tx(&q_full[s], BWD_Q_BYTES);
        tma_load_4d(sQ + s * BWD_Q_BYTES, &tmQ, &q_full[s], 0, q_begin + it * BWD_BQ, h, b);
    };
    auto load_do = [&](int it) {
        const int s = it % BWD_DO_STAGES;
        mbar_arrive_expect_tx(&do_full[s], BWD_Q_BYTES);
        tma_load_4d(sdO + s * BWD_Q_BYTES, &tmdO, &do_full[s], 0, q_begin + it * BWD_BQ, h, b);
    };
    if (warp == BWD_MMA_WARP && elect_one()) {
        *abort_flag = 0;
        mbar_init(kv_full, 1);
        for (int s = 0; s < BWD_Q_STAGES; ++s) mbar_init(&q_full[s], 1);
        for (int s = 0; s < BWD_DO_STAGES; ++s) mbar_init(&do_full[s], 1);
        mbar_init(s_full, 1);
        mbar_init(dp_full, 1);
        mbar_init(p_ready, 256);
        mbar_init(dq_full, 1);
        mbar_init(dq_free, 256);
        mbar_init(in_free, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&dqs_full[s], 256); mbar_init(&dqs_free[s], 1); }
        fence_barrier_init();
        pdl_wait();                                // the first loads run under the TMEM allocation
        mbar_arrive_expect_tx(kv_full, 2 * TILE_BYTES);
        tma_load_4d(sK, &tmK, kv_full, 0, k0, h, b);
        load_q(0);
        tma_load_4d(sV, &tmV, kv_full, 0, k0, h, b);
        load_do(0);
        for (int it = 1; it < BWD_Q_STAGES && it < n_it; ++it) load_q(it);
        for (int it = 1; it < BWD_DO_STAGES && it < n_it; ++it) load_do(it);
    }
    if (warp == BWD_STORE_WARP) { tmem_alloc(tmem_slot, BWD_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_S = tmem_base, tmem_dP = tmem_base + BWD_BQ, tmem_dQ = tmem_dP, tmem_dV = tmem_base + 2 * BWD_BQ,
                   tmem_dK = tmem_dV + HD;
    pdl_wait();        // barrier set-up and TMEM allocation above may overlap the tail of the previous kernel

    if (warp == BWD_MMA_WARP) {
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc(1, false, false, BKV, BWD_BQ);    // K Q^T, V dO^T
            constexpr uint32_t idesc_t = make_idesc(1, false, true, BKV, HD);         // P^T dO, dS^T Q
            constexpr uint32_t idesc_q = make_idesc(1, true, true, BWD_BQ, HD);       // dS K (A read transposed)
            // descriptors are encoded once; per MMA only a byte offset is added
            const uint64_t kK = make_smem_desc(smem_u32(sK), 0, 1024), vK = make_smem_desc(smem_u32(sV), 0, 1024);
            const uint64_t kMN = make_smem_desc(smem_u32(sK), TILE_BYTES, 1024);
            const uint64_t qK0 = make_smem_desc(smem_u32(sQ), 0, 1024), oK0 = make_smem_desc(smem_u32(sdO), 0, 1024);
            const uint64_t qMN0 = make_smem_desc(smem_u32(sQ), BWD_Q_BYTES, 1024);
            const uint64_t oMN0 = make_smem_desc(smem_u32(sdO), BWD_Q_BYTES, 1024);
            const uint64_t sMN = make_smem_desc(smem_u32(sX), TILE_BYTES, 1024);
            auto issue_s = [&](int it) {
                const uint64_t qd = desc_add(qK0, (it % BWD_Q_STAGES) * BWD_Q_BYTES);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_S, desc_add(kK, k * 32), desc_add(qd, k * 32), idesc_s, k > 0);
            };
            auto issue_dp = [&](int it) {
                const uint64_t od = desc_add(oK0, (it % BWD_DO_STAGES) * BWD_Q_BYTES);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_dP, desc_add(vK, k * 32), desc_add(od, k * 32), idesc_s, k > 0);
            };
            bool ok = mbar_wait(kv_full, 0, abort_flag) && mbar_wait(&q_full[0], 0, abort_flag) &&
                      mbar_wait(&do_full[0], 0, abort_flag);
            if (ok) { tc_fence_after(); issue_s(0); mma_commit(s_full); issue_dp(0); mma_commit(dp_full); }
            for (int it = 0; it < n_it && ok; ++it) {
                if (!mbar_wait(p_ready, it & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t qd = desc_add(qMN0, (it % BWD_Q_STAGES) * BWD_Q_BYTES),
                               od = desc_add(oMN0, (it % BWD_DO_STAGES) * BWD_Q_BYTES), sd = desc_add(sMN, (it & 1) * TILE_BYTES);
                // dQ first: the warps read it out while the other products of this block run
#pragma unroll
                for (int k = 0; k < BKV / 16; ++k)        // reduction over the 128 keys of this CTA
                    mma_f16_ss(tmem_dQ, desc_add(sd, k * 2048), desc_add(kMN, k * 2048), idesc_q, k > 0);
                mma_commit(dq_full);
                const uint32_t acc = it > 0;
#pragma unroll
                for (int k = 0; k < BWD_BQ / 16; ++k)     // reduction over the 64 queries of this block
                    mma_f16_ts(tmem_dV, tmem_S + (k >> 1) * 32 + (k & 1) * 8, desc_add(od, k * 2048), idesc_t, acc | (k > 0));
#pragma unroll
                for (int k = 0; k < BWD_BQ / 16; ++k)
                    mma_f16_ts(tmem_dK, tmem_S + (k >> 1) * 32 + 16 + (k & 1) * 8, desc_add(qd, k * 2048), idesc_t, acc | (k > 0));
                mma_commit(in_free);
                if (it + 1 < n_it) {
                    // S^T takes the place of P^T and dS^T once a barrier says that the products above, which read them, are complete
                    // (PTX orders MMAs of a thread only if they accumulate in the same place): before the warps have dQ in
                    // registers, so that their exponentials run while dP^T, which takes its place, is made.
                    const int n = it + 1;
                    if (!mbar_wait(&q_full[n % BWD_Q_STAGES], (n / BWD_Q_STAGES) & 1, abort_flag) ||
                        !mbar_wait(in_free, it & 1, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    issue_s(n);
                    mma_commit(s_full);
                    if (!mbar_wait(&do_full[n % BWD_DO_STAGES], (n / BWD_DO_STAGES) & 1, abort_flag) ||
                        !mbar_wait(dq_free, it & 1, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    issue_dp(n);
                    mma_commit(dp_full);
                    if (it + BWD_DO_STAGES < n_it) load_do(it + BWD_DO_STAGES);
                    if (it + BWD_Q_STAGES < n_it) load_q(it + BWD_Q_STAGES);
                }
            }
            if (!ok) for (int i = 0; i < 2000; ++i) __nanosleep(500);
        }
    } else if (warp == BWD_STORE_WARP) {
        if (elect_one()) {
            for (int it = 0; it < n_it; ++it) {
                if (!mbar_wait(&dqs_full[it & 1], (it >> 1) & 1, abort_flag)) break;
                const int q0 = q_begin + it * BWD_BQ;
                const uint8_t* tile = sX + (it & 1) * TILE_BYTES;
                tma_reduce_add_3d(&tmdQ, tile, 0, q0, bh);
                tma_reduce_add_3d(&tmdQ, tile + TILE_BYTES / 2, 32, q0, bh);
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(&dqs_free[it & 1]);         // the buffer may be refilled; no shared memory is read after the last wait
            }
        }
    } else {
        // ---------------- gradient warps: warp w owns TMEM lanes 32 (w & 3).. (key rows) and the 32 queries (w >> 2) of a
        // block, so its P^T and dS^T go to columns that only it has read ----
        const int quarter = warp & 3, cg = warp >> 2;
        const int row = quarter * 32 + lane;            // TMEM lane: key row for S^T, dP^T, dV, dK
        const int key = k0 + row;
        const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
        const uint32_t tS = tmem_S + lane_addr + cg * 32;
        // -lse and -delta of a block's queries are read by all threads as columns: 128 threads bring them to shared memory,
        // one block ahead.  Queries beyond T get probability 2^-inf = 0.
        // The loaded value is not touched before it is stored: arithmetic on it here would wait for the load (800 clocks of every
        // block for these warps, and with them for all).
        const bool is_lse = threadIdx.x < BWD_BQ;
        const float* stat_src = (is_lse ? p.lse : p.delta) + (long long)bh * p.T;
        auto stat_q = [&](int it) { return q_begin + it * BWD_BQ + (int)(threadIdx.x & (BWD_BQ - 1)); };
        auto stat_load = [&](int it) { const int q = stat_q(it); return q < p.T ? stat_src[q] : 0.f; };
        auto stat_store = [&](int it, float v) {
            const float x = is_lse ? (stat_q(it) < p.T ? -v * LOG2E : -INFINITY) : -v;
            stats[(it & 1) * BWD_STAT_FLOATS + threadIdx.x] = x;
        };
        if (threadIdx.x < BWD_STAT_FLOATS) stat_store(0, stat_load(0));
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const F32x2 sc2 = f2_splat(p.scale_log2);
        bool ok = true;
        for (int it = 0; it < n_it; ++it) {
            const int q0 = q_begin + it * BWD_BQ;
            float next = 0.f;
            const bool fetch = it + 1 < n_it && threadIdx.x < BWD_STAT_FLOATS;
            if (fetch) next = stat_load(it + 1);
            // the statistics were stored before the previous block's arrivals on p_ready (a phase that is complete)
            if ((it > 0 && !mbar_wait(p_ready, (it - 1) & 1, abort_flag)) || !mbar_wait(s_full, it & 1, abort_flag)) {
                ok = false;
                break;
            }
            tc_fence_after();
            uint32_t rs[32], rd[32];
            tmem_ld32(tS, rs);
            tmem_wait_ld();
            if (q0 + BWD_BQ > p.T) {
                // the rows of Q beyond T are zeros, and 0 k is NaN where an element of the key is infinite: 0, so that the
                // statistics' -inf decides
                const int hi = p.T - q0 - cg * 32;
#pragma unroll
                for (int i = 0; i < 32; ++i) rs[i] = i < hi ? rs[i] : 0u;
            }
            const float4* st = reinterpret_cast<const float4*>(stats + (it & 1) * BWD_STAT_FLOATS + cg * 32);
            float* pr = reinterpret_cast<float*>(rs);
            // scale-and-shift, dP - delta and the product on packed pairs (one instruction per two queries)
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 nl = st[i / 4];
                f2_unpack(f2_fma(f2_pack(pr[i], pr[i + 1]), sc2, f2_pack(nl.x, nl.y)), pr[i], pr[i + 1]);
                f2_unpack(f2_fma(f2_pack(pr[i + 2], pr[i + 3]), sc2, f2_pack(nl.z, nl.w)), pr[i + 2], pr[i + 3]);
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) pr[i] = ex2_approx(pr[i]);
            if (k0 + BKV > p.T || (p.causal && q0 < k0 + BKV)) {
                // queries [lo, 32) of this thread's 32 see its key
                const int lo = (key < p.T ? (p.causal ? key - q0 : 0) : BWD_BQ) - cg * 32;
#pragma unroll
                for (int i = 0; i < 32; ++i) pr[i] = i >= lo ? pr[i] : 0.f;
            }
            if (!mbar_wait(dp_full, it & 1, abort_flag) ||
                (it >= 2 && !mbar_wait(&dqs_free[it & 1], ((it >> 1) - 1) & 1, abort_flag))) { ok = false; break; }
            tc_fence_after();
            tmem_ld32(tmem_dP + lane_addr + cg * 32, rd);
            tmem_wait_ld();
            uint8_t* tile = sX + (it & 1) * TILE_BYTES;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float* ds = reinterpret_cast<float*>(rd) + g * 8;
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    const float4 nd = st[(BWD_BQ + g * 8 + i) / 4];
                    f2_unpack(f2_add(f2_pack(ds[i], ds[i + 1]), f2_pack(nd.x, nd.y)), ds[i], ds[i + 1]);
                    f2_unpack(f2_add(f2_pack(ds[i + 2], ds[i + 3]), f2_pack(nd.z, nd.w)), ds[i + 2], ds[i + 3]);
                }
#pragma unroll
                for (int i = 0; i < 8; i += 2)
                    f2_unpack(f2_mul(f2_pack(pr[g * 8 + i], pr[g * 8 + i + 1]), f2_pack(ds[i], ds[i + 1])), ds[i], ds[i + 1]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {           // the packed pairs take the registers of the scores they came from
                    rs[g * 4 + i] = f2_to_bf2(pr[g * 8 + 2 * i], pr[g * 8 + 2 * i + 1]);
                    rd[g * 4 + i] = f2_to_bf2(ds[2 * i], ds[2 * i + 1]);
                }
                *reinterpret_cast<uint4*>(tile + swz(row, cg * 4 + g)) =
                    make_uint4(rd[g * 4], rd[g * 4 + 1], rd[g * 4 + 2], rd[g * 4 + 3]);
            }
            tmem_st16(tS, rs);
            tmem_st16(tS + 16, rd);
            if (fetch) stat_store(it + 1, next);
            tmem_wait_st();
            tc_fence_before();
            fence_proxy_async();                        // dS^T
            mbar_arrive(p_ready);
            // dQ: 64 query rows in lanes 0..15 of each quarter; this warp takes 16 rows x 32 columns to the staging tile
            // (swizzled for TMA), from where the store warp adds it to the global scratch
            if (!mbar_wait(dq_full, it & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            uint32_t t[32];
            tmem_ld32(tmem_dQ + lane_addr + cg * 32, t);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(dq_free);
            if (lane < 16) {                            // dS^T has been read by the product that made dQ
                uint8_t* atom = tile + cg * (TILE_BYTES / 2);
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    *reinterpret_cast<uint4*>(atom + swz(quarter * 16 + lane, g)) =
                        make_uint4(t[4 * g], t[4 * g + 1], t[4 * g + 2], t[4 * g + 3]);
            }
            fence_proxy_async();
            mbar_arrive(&dqs_full[it & 1]);
        }
        // dV, dK of this key block: this warp's 32 columns (64 bytes = two full sectors per row) straight from registers
        if (ok && mbar_wait(in_free, (n_it - 1) & 1, abort_flag)) {
            tc_fence_after();
            const long long off = (long long)b * p.sb + (long long)h * p.sh + (long long)key * p.st + cg * 32;
            uint32_t t[32];
            tmem_ld32(tmem_dV + lane_addr + cg * 32, t);
            tmem_wait_ld();
            if (key < p.T) {
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    *reinterpret_cast<uint4*>(p.dv + off + g * 8) = pack8(reinterpret_cast<const float*>(t) + g * 8);
            }
            tmem_ld32(tmem_dK + lane_addr + cg * 32, t);
            tmem_wait_ld();
            if (key < p.T) {
                float* v = reinterpret_cast<float*>(t);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] *= p.scale;
#pragma unroll
                for (int g = 0; g < 4; ++g) *reinterpret_cast<uint4*>(p.dk + off + g * 8) = pack8(v + g * 8);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, CME_ERR_TIMEOUT);
    if (warp == BWD_STORE_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, BWD_TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------
// Backward with 128 x 128 blocks and one CTA per SM: where dQ is finished inside the kernel (dq_mode 1 and 2), and for grids that leave
// the small CTAs above without neighbours (bwd_wide)
// ------------------------------------------------------------------------------------------------------
struct BwdWideParams {
    int T, nh, causal;
    float scale, scale_log2;
    const float* lse;
    const float* delta;
    float* dq_accum;               // fp32 [nb*nh, T, HD] scratch for the partial sums of dQ
    __nv_bfloat16* dk; __nv_bfloat16* dv;
    long long sb, sh, st;          // strides of dQ / dK / dV
    int* status;
    int* dq_sem;                   // [nb*nh, query blocks] contribution counters (zero between launches); null in mode 0
    __nv_bfloat16* dq;             // final dQ (modes 1 and 2)
    int dq_mode;                   // 0: unordered adds into a scratch the launch cleared, converted by dq_convert_kernel
                                   // 1: ordered adds, key block 0 finishes   2: unordered adds, the last part's CTA finishes
};

// Bounded wait until *sem >= want (acquire).  Lane 0 of the calling warp polls; the warp then synchronises.
__device__ __forceinline__ bool sem_wait_warp(const int* sem, int want, volatile int* abort_flag) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) {
        uint32_t i = 0;
        for (;; ++i) {
            int v;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(sem) : "memory");
            if (v >= want) break;
            if ((i & 255u) == 255u && *abort_flag) { ok = false; break; }
            if (i >= (1u << 22)) { *abort_flag = 1; ok = false; break; }
            __nanosleep(32);
        }
    }
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    return ok;
}

// shared: K 16K | V 16K | Q[2] 32K | dO[2] 32K | P 32K | dS[2] 64K | dQ staging (fp32) 32K | barriers   (one CTA per SM)
constexpr int BWD_WIDE_SMEM = 14 * TILE_BYTES + 512;     // tiles | barriers, flags and the finishing warp's ring
constexpr int BWD_WIDE_MMA_WARP = 16;           // warps 0..15 compute, warp 16 issues TMA loads and MMA,
constexpr int BWD_WIDE_STORE_WARP = 17;         // warp 17 issues the dQ reduce-stores
constexpr int BWD_WIDE_CONVERT_WARP = 18;        // warp 18 (mode 2) converts the dQ tiles whose last part this CTA added
constexpr int BWD_WIDE_THREADS = 19 * 32;
constexpr int FIN_RING = CME_ATTN_FINISH_MAX_QBLOCKS;   // a CTA hands over at most one tile per query block
constexpr int BWD_WIDE_TMEM_COLS = 512;     // S [0,128) dP [128,256) dV [256,320) dK [320,384) dQ [384,448)
static_assert(12 * 8 + 4 + 4 + 4 + FIN_RING * 4 <= 512, "barriers, flags and ring exceed their block");
static_assert(BWD_WIDE_SMEM <= 227 * 1024, "backward shared-memory carve-up exceeds what one CTA may have");
static_assert(2 * 128 + 3 * HD <= BWD_WIDE_TMEM_COLS, "backward TMEM budget: S, dP, dV, dK, dQ");

__global__ void __launch_bounds__(BWD_WIDE_THREADS, 1)
attn_bwd_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmdQ, const BwdWideParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, CME_ERR_SHAPE);
        return;
    }
    uint8_t* sK = smem;
    uint8_t* sV = sK + TILE_BYTES;
    uint8_t* sQ = sV + TILE_BYTES;             // 2 stages
    uint8_t* sdO = sQ + 2 * TILE_BYTES;        // 2 stages
    uint8_t* sP = sdO + 2 * TILE_BYTES;        // [2 key atoms][128 query rows][128 B]; free again once dV's MMAs ran
    uint8_t* sdS = sP + 2 * TILE_BYTES;        // 2 buffers, same layout
    uint8_t* sdQ = sdS + 4 * TILE_BYTES;       // fp32 dQ staging: [2 column atoms][128 query rows][128 B]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sdQ + 2 * TILE_BYTES);
    uint64_t* kv_full = bars;
    uint64_t* q_full = bars + 1;               // [2]
    uint64_t* q_empty = bars + 3;              // [2]
    uint64_t* s_full = bars + 5;               // S and dP of a query block are in TMEM
    uint64_t* p_ready = bars + 6;              // P, dS written; S, dP, previous dQ consumed (512 arrivals)
    uint64_t* dq_full = bars + 7;              // dV, dK accumulated and dQ of a query block complete
    uint64_t* p_free = bars + 8;               // dV's MMAs of a block have read P
    uint64_t* dqs_full = bars + 9;             // dQ staging written (512 arrivals)
    uint64_t* dqs_free = bars + 10;            // dQ staging read by the reduce-store
    uint64_t* s_free = bars + 11;              // S and dP of a query block are in registers (512 arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* fin_count = abort_flag + 1;  // tiles handed to the finishing warp so far; -1 - n once the store warp
                                               // has ended after n tiles
    volatile int* fin_ring = abort_flag + 2;   // [FIN_RING] query-block indices

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // Ordered form: higher key blocks are dispatched first, so a CTA only ever waits for the dQ parts of key blocks
    // above its own, which are then resident or finished.  Unordered form: the key blocks with the most query blocks
    // (the lowest) first.
    const int nkb = gridDim.x;
    const bool ordered = p.dq_mode == 1, finish_last = p.dq_mode == 2;
    const int kb = ordered ? nkb - 1 - (int)blockIdx.x : (int)blockIdx.x, k0 = kb * BKV;
    const int bh = blockIdx.y, b = bh / p.nh, h = bh % p.nh;
    const int nq = (p.T + BQ - 1) / BQ;
    // first key block to contribute to query block qi (the highest one that sees it); key block kb's turn comes when
    // first_kb(qi) - kb parts are in, key block 0 finishes the tile
    auto first_kb = [&](int qi) { return p.causal ? min(qi, nkb - 1) : nkb - 1; };
    const int i_begin = p.causal ? kb : 0;     // query blocks that see this key block
    const int n_it = nq - i_begin;
    // Query block of iteration `it`.  Mode 2 walks them downwards: the key blocks of a head start together, so all of
    // them then reach a query tile in the same iteration and whichever comes last finishes it -- the finishing work
    // spreads over the CTAs instead of queueing up on key block 0, which is the last arrival of every tile when all
    // walk upwards.
    auto qblock = [&](int it) { return finish_last ? nq - 1 - it : i_begin + it; };

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        *fin_count = 0;
        mbar_init(kv_full, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
        mbar_init(s_full, 1);
        mbar_init(p_ready, 512);
        mbar_init(dq_full, 1);
        mbar_init(p_free, 1);
        mbar_init(dqs_full, 512);
        mbar_init(dqs_free, 1);
        mbar_init(s_free, 512);
        fence_barrier_init();
    }
    if (warp == BWD_WIDE_MMA_WARP) { tmem_alloc(tmem_slot, BWD_WIDE_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_S = tmem_base, tmem_dP = tmem_base + 128, tmem_dV = tmem_base + 256,
                   tmem_dK = tmem_base + 320, tmem_dQ = tmem_base + 384;

    if (warp == BWD_WIDE_MMA_WARP) {
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc(1, false, false, 128, 128);    // Q K^T, dO V^T
            constexpr uint32_t idesc_t = make_idesc(1, true, true, 128, HD);       // P^T dO, dS^T Q (A read transposed)
            constexpr uint32_t idesc_q = make_idesc(1, false, true, 128, HD);      // dS K
            bool ok = true;
            mbar_arrive_expect_tx(kv_full, 2 * TILE_BYTES);
            tma_load_4d(sK, &tmK, kv_full, 0, k0, h, b);
            tma_load_4d(sV, &tmV, kv_full, 0, k0, h, b);
            auto load_q = [&](int it) {
                const int st = it & 1;
                mbar_arrive_expect_tx(&q_full[st], 2 * TILE_BYTES);
                tma_load_4d(sQ + st * TILE_BYTES, &tmQ, &q_full[st], 0, qblock(it) * BQ, h, b);
                tma_load_4d(sdO + st * TILE_BYTES, &tmdO, &q_full[st], 0, qblock(it) * BQ, h, b);
            };
            // descriptors are encoded once; per MMA only a byte offset is added
            const uint64_t kK = make_smem_desc(smem_u32(sK), 0, 1024), vK = make_smem_desc(smem_u32(sV), 0, 1024);
            const uint64_t kMN = make_smem_desc(smem_u32(sK), TILE_BYTES, 1024);
            // stage / buffer 1 of each ring lies a fixed distance after stage 0, so its descriptor is base + offset
            const uint64_t qK0 = make_smem_desc(smem_u32(sQ), 0, 1024), oK0 = make_smem_desc(smem_u32(sdO), 0, 1024);
            const uint64_t qMN0 = make_smem_desc(smem_u32(sQ), TILE_BYTES, 1024);
            const uint64_t oMN0 = make_smem_desc(smem_u32(sdO), TILE_BYTES, 1024);
            const uint64_t pMN0 = make_smem_desc(smem_u32(sP), TILE_BYTES, 1024);
            const uint64_t sMN0 = make_smem_desc(smem_u32(sdS), TILE_BYTES, 1024);
            const uint64_t sK0 = make_smem_desc(smem_u32(sdS), 0, 1024);
            auto issue_s = [&](int it) {
                const uint64_t qd = desc_add(qK0, (it & 1) * TILE_BYTES), od = desc_add(oK0, (it & 1) * TILE_BYTES);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_S, desc_add(qd, k * 32), desc_add(kK, k * 32), idesc_s, k > 0);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    mma_f16_ss(tmem_dP, desc_add(od, k * 32), desc_add(vK, k * 32), idesc_s, k > 0);
                mma_commit(s_full);
            };
            if (n_it > 0) load_q(0);
            if (n_it > 1) load_q(1);
            ok = mbar_wait(kv_full, 0, abort_flag);
            if (ok && n_it > 0) {
                ok = mbar_wait(&q_full[0], 0, abort_flag);
                if (ok) { tc_fence_after(); issue_s(0); }
            }
            for (int it = 0; it < n_it && ok; ++it) {
                const int st = it & 1;
                if (it + 1 < n_it) {
                    // The next block's S and dP are issued as soon as this block's have been read out of TMEM (the
                    // gradient warps signal that right after their loads), so they are computed while the warps
                    // do this block's arithmetic instead of after it.
                    if (!mbar_wait(s_free, it & 1, abort_flag)) { ok = false; break; }
                    if (!mbar_wait(&q_full[(it + 1) & 1], ((it + 1) >> 1) & 1, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    issue_s(it + 1);
                }
                if (!mbar_wait(p_ready, it & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t pd = pMN0, sd = desc_add(sMN0, st * 2 * TILE_BYTES),
                               sk = desc_add(sK0, st * 2 * TILE_BYTES), qd = desc_add(qMN0, st * TILE_BYTES),
                               od = desc_add(oMN0, st * TILE_BYTES);
                const uint32_t acc = it > 0;
#pragma unroll
                for (int k = 0; k < BQ / 16; ++k)        // dV first: P is single-buffered and is released right after
                    mma_f16_ss(tmem_dV, desc_add(pd, k * 2048), desc_add(od, k * 2048), idesc_t, acc | (k > 0));
                mma_commit(p_free);
#pragma unroll
                for (int k = 0; k < BQ / 16; ++k)        // reduction over the 128 queries of this block
                    mma_f16_ss(tmem_dK, desc_add(sd, k * 2048), desc_add(qd, k * 2048), idesc_t, acc | (k > 0));
#pragma unroll
                for (int k = 0; k < BKV / 16; ++k)       // reduction over the 128 keys of this CTA
                    mma_f16_ss(tmem_dQ, desc_add(sk, (k >> 2) * TILE_BYTES + (k & 3) * 32), desc_add(kMN, k * 2048),
                               idesc_q, k > 0);
                mma_commit(dq_full);
                mma_commit(&q_empty[st]);
                if (it + 2 < n_it) {
                    if (!mbar_wait(&q_empty[st], (it >> 1) & 1, abort_flag)) { ok = false; break; }
                    load_q(it + 2);
                }
            }
            if (!ok) for (int i = 0; i < 2000; ++i) __nanosleep(500);
        }
    } else if (warp == BWD_WIDE_STORE_WARP) {
        // ---------------- dQ store issuer: moves each staged 128 x 64 fp32 tile into the global scratch.  Ordered form:
        // when it is this key block's turn -- a plain tile store if it is the first part, else a bulk reduce-add --
        // and the tile's counter is raised once the write has completed.  Key block 0 does not come through here.
        if (!(ordered && kb == 0) && elect_one()) {
            for (int f = 0; f < n_it; ++f) {
                if (!mbar_wait(dqs_full, f & 1, abort_flag)) break;
                const int qi = qblock(f), q0 = qi * BQ;
                int* sem = ordered ? p.dq_sem + (long long)bh * nq + qi : nullptr;
                const int turn = ordered ? first_kb(qi) - kb : 1;
                if (ordered) {
                    bool mine = false;
                    for (uint32_t i = 0; i < (1u << 22); ++i) {
                        int v;
                        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(sem) : "memory");
                        if (v >= turn) { mine = true; break; }
                        if ((i & 255u) == 255u && *abort_flag) break;
                        __nanosleep(32);
                    }
                    if (!mine) { *abort_flag = 1; break; }
                }
                if (turn == 0) {
                    tma_store_3d(&tmdQ, sdQ, 0, q0, bh);
                    tma_store_3d(&tmdQ, sdQ + TILE_BYTES, 32, q0, bh);
                } else {
                    tma_reduce_add_3d(&tmdQ, sdQ, 0, q0, bh);
                    tma_reduce_add_3d(&tmdQ, sdQ + TILE_BYTES, 32, q0, bh);
                }
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(dqs_free);                  // the staging tile may be refilled
                if (ordered) {
                    tma_store_wait<0>();                // the tile is in global memory
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                    __threadfence();
                    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(sem), "r"(turn + 1) : "memory");
                } else if (finish_last) {
                    // count this part in once the adds have been performed; whoever brings the count to the number of
                    // key blocks that see the tile hands it to the finishing warp
                    tma_store_wait<0>();
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                    __threadfence();
                    int before;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;"
                                 : "=r"(before) : "l"(p.dq_sem + (long long)bh * nq + qi) : "memory");
                    if (before + 1 == first_kb(qi) + 1) {
                        const int n = *fin_count;
                        fin_ring[n % FIN_RING] = qi;
                        __threadfence_block();
                        *fin_count = n + 1;
                    }
                }
            }
            tma_store_wait<0>();
            if (finish_last) { __threadfence_block(); *fin_count = -1 - *fin_count; }
        }
    } else if (warp == BWD_WIDE_CONVERT_WARP) {
        // ---------------- finishing warp (mode 2): every part of a handed-over tile is in the scratch; scale and cast the
        // sums to dQ, and leave zeros behind for the next launch.  A tile is 128 x 64 fp32 = 32 KB of contiguous scratch.
        if (finish_last && n_it > 0) {
            int taken = 0;
            bool ok = true;
            for (uint32_t spin = 0; ok;) {
                const int c = *fin_count;
                const int avail = c >= 0 ? c : -1 - c;
                if (taken == avail) {
                    if (c < 0) break;                                   // the store warp has ended and nothing is left
                    if ((++spin & 255u) == 0 && *abort_flag) break;
                    if (spin >= (1u << 24)) { *abort_flag = 1; break; }
                    __nanosleep(200);
                    continue;
                }
                spin = 0;
                __threadfence_block();
                const int qi = fin_ring[taken % FIN_RING];
                ++taken;
                __threadfence();
                asm volatile("fence.proxy.async.global;" ::: "memory");
                const int q0 = qi * BQ;
                const int rows_here = min(BQ, p.T - q0);
                float4* tile = reinterpret_cast<float4*>(p.dq_accum + ((long long)bh * p.T + q0) * HD);
                __nv_bfloat16* dst0 = p.dq + (long long)b * p.sb + (long long)h * p.sh + (long long)q0 * p.st;
                const int n4 = rows_here * (HD / 4);                    // float4 elements of the tile
#pragma unroll 1
                for (int base = 0; base < n4; base += 32 * 8) {
                    float4 v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int i = base + j * 32 + lane;
                        v[j] = i < n4 ? __ldcg(tile + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int i = base + j * 32 + lane;
                        if (i < n4) {
                            const int r = i / (HD / 4), c4 = i % (HD / 4);
                            __nv_bfloat162 lo = __floats2bfloat162_rn(v[j].x * p.scale, v[j].y * p.scale);
                            __nv_bfloat162 hi = __floats2bfloat162_rn(v[j].z * p.scale, v[j].w * p.scale);
                            uint2 out;
                            out.x = *reinterpret_cast<uint32_t*>(&lo);
                            out.y = *reinterpret_cast<uint32_t*>(&hi);
                            *reinterpret_cast<uint2*>(dst0 + (long long)r * p.st + c4 * 4) = out;
                            __stcg(tile + i, make_float4(0.f, 0.f, 0.f, 0.f));
                        }
                    }
                }
                if (lane == 0) p.dq_sem[(long long)bh * nq + qi] = 0;  // nobody else touches it before the next launch
            }
        }
    } else {
        // ---------------- gradient warps: 16 warps; warp w owns TMEM lanes 32*(w&3).. (query rows) and the
        // 32-column group (w>>2) of every S / dP tile, so each scheduler has four warps to hide latency with ----
        const int quarter = warp & 3, cg = warp >> 2;
        const int row = quarter * 32 + lane;            // TMEM lane: query row for S, dP, dQ; key row for dV, dK
        const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
        bool ok = true;
        // dQ of a finished query block: this warp's 16 columns go to the fp32 staging tile (swizzled for TMA); the
        // store warp then adds the tile into the global accumulator with one bulk reduce per 32-column half
        // `signal`: false leaves the proxy fence and the arrival on dqs_full to the caller, who then covers the P / dS
        // stores of the current block and this staging write with one fence
        const bool finisher = ordered && kb == 0;       // this CTA completes dQ of every query block it sees
        auto flush_dq = [&](int f, bool signal) -> bool {
            if (!mbar_wait(dq_full, f & 1, abort_flag)) return false;
            tc_fence_after();
            uint32_t t[16];
            tmem_ld16(tmem_dQ + lane_addr + cg * 16, t);
            tmem_wait_ld();
            if (finisher) {
                // every other key block's part of this query block is in the scratch tile (their counters say so):
                // add it to this thread's 16 columns, scale, cast, store dQ
                const int qi = qblock(f), need = first_kb(qi);
                const int qrow = qi * BQ + row;
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(t[i]);
                if (need > 0) {
                    if (!sem_wait_warp(p.dq_sem + (long long)bh * nq + qi, need, abort_flag)) return false;
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                    if (qrow < p.T) {
                        const float4* src = reinterpret_cast<const float4*>(p.dq_accum + ((long long)bh * p.T + qrow) * HD + cg * 16);
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const float4 a = __ldcg(src + g);
                            v[4 * g] += a.x; v[4 * g + 1] += a.y; v[4 * g + 2] += a.z; v[4 * g + 3] += a.w;
                        }
                    }
                }
                if (qrow < p.T) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] *= p.scale;
                    __nv_bfloat16* dst = p.dq + (long long)b * p.sb + (long long)h * p.sh + (long long)qrow * p.st + cg * 16;
                    *reinterpret_cast<uint4*>(dst) = pack8(v);
                    *reinterpret_cast<uint4*>(dst + 8) = pack8(v + 8);
                }
                return true;
            }
            if (f > 0 && !mbar_wait(dqs_free, (f - 1) & 1, abort_flag)) return false;
            uint8_t* atom = sdQ + (cg >> 1) * TILE_BYTES;
#pragma unroll
            for (int g = 0; g < 4; ++g)
                *reinterpret_cast<uint4*>(atom + swz(row, (cg & 1) * 4 + g)) =
                    make_uint4(t[4 * g], t[4 * g + 1], t[4 * g + 2], t[4 * g + 3]);
            if (signal) {
                fence_proxy_async();
                mbar_arrive(dqs_full);
            }
            return true;
        };
        // row statistics of a query block are fetched one block ahead: their global-memory latency must not sit
        // between the arrival of S and the first exponential
        auto row_stats = [&](int it2, float& l2, float& d2) {
            const int qc2 = min(qblock(it2) * BQ + row, p.T - 1);
            l2 = p.lse[(long long)bh * p.T + qc2];       // used untouched a block later, so that nothing waits for it here
            d2 = p.delta[(long long)bh * p.T + qc2];
        };
        float lse2_n = 0.f, dl_n = 0.f;
        if (n_it > 0) row_stats(0, lse2_n, dl_n);
        for (int it = 0; it < n_it && ok; ++it) {
            const int qi0 = qblock(it) * BQ;
            const int q = qi0 + row;
            const float lse2 = lse2_n * LOG2E, dl = dl_n;
            if (it + 1 < n_it) row_stats(it + 1, lse2_n, dl_n);
            uint8_t* bufP = sP;
            uint8_t* bufS = sdS + (it & 1) * 2 * TILE_BYTES;
            if (!mbar_wait(s_full, it & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const bool need_mask = (qi0 + BQ > p.T) || (k0 + BKV > p.T) || (p.causal && qi0 < k0 + BKV);
            uint32_t rs[32], rd[32];
            tmem_ld32(tmem_S + lane_addr + cg * 32, rs);
            tmem_ld32(tmem_dP + lane_addr + cg * 32, rd);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(s_free);                        // S and dP may be overwritten by the next block's products
            if (it > 0 && !mbar_wait(p_free, (it - 1) & 1, abort_flag)) { ok = false; break; }
            // scale-and-shift, dP - delta and the product on packed pairs (one instruction per two keys)
            const F32x2 sc2 = f2_splat(p.scale_log2), nl2 = f2_splat(-lse2), nd2 = f2_splat(-dl);
            const int lim = (q < p.T ? min(p.T, p.causal ? q + 1 : p.T) : 0) - (k0 + cg * 32);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float pr[8], ds[8];
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    float a0, a1;
                    f2_unpack(f2_fma(f2_pack(__uint_as_float(rs[g * 8 + i]), __uint_as_float(rs[g * 8 + i + 1])), sc2, nl2),
                              a0, a1);
                    float pv0 = ex2_approx(a0), pv1 = ex2_approx(a1);
                    if (need_mask) {        // this thread's keys [0, lim) of the 32 are visible to its row
                        pv0 = g * 8 + i < lim ? pv0 : 0.f;
                        pv1 = g * 8 + i + 1 < lim ? pv1 : 0.f;
                    }
                    pr[i] = pv0;
                    pr[i + 1] = pv1;
                    f2_unpack(f2_mul(f2_pack(pv0, pv1),
                                     f2_add(f2_pack(__uint_as_float(rd[g * 8 + i]), __uint_as_float(rd[g * 8 + i + 1])), nd2)),
                              ds[i], ds[i + 1]);
                }
                const uint32_t off = (cg >> 1) * TILE_BYTES + swz(row, (cg & 1) * 4 + g);
                *reinterpret_cast<uint4*>(bufP + off) = pack8(pr);
                *reinterpret_cast<uint4*>(bufS + off) = pack8(ds);
            }
            // the previous block's dQ is read here, after this block's arithmetic, so that its MMAs had the whole
            // time of that arithmetic to finish
            if (it > 0 && !flush_dq(it - 1, false)) { ok = false; break; }
            tc_fence_before();
            fence_proxy_async();                        // one fence for P, dS and the dQ staging tile
            if (it > 0 && !finisher) mbar_arrive(dqs_full);
            mbar_arrive(p_ready);
        }
        if (ok && n_it > 0) ok = flush_dq(n_it - 1, true);
        // dK, dV of this key block (all MMAs are complete: the last dq_full wait covered them); this warp stores its
        // 16 columns (32 bytes = one full sector per row) straight from registers
        if (ok) {
            const int key = k0 + row;
            const long long off = (long long)b * p.sb + (long long)h * p.sh + (long long)key * p.st + cg * 16;
            uint32_t t[16];
            float v[16];
            if (n_it > 0) { tmem_ld16(tmem_dV + lane_addr + cg * 16, t); tmem_wait_ld(); }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = n_it > 0 ? __uint_as_float(t[i]) : 0.f;
            if (key < p.T) {
                *reinterpret_cast<uint4*>(p.dv + off) = pack8(v);
                *reinterpret_cast<uint4*>(p.dv + off + 8) = pack8(v + 8);
            }
            if (n_it > 0) { tmem_ld16(tmem_dK + lane_addr + cg * 16, t); tmem_wait_ld(); }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = n_it > 0 ? __uint_as_float(t[i]) * p.scale : 0.f;
            if (key < p.T) {
                *reinterpret_cast<uint4*>(p.dk + off) = pack8(v);
                *reinterpret_cast<uint4*>(p.dk + off + 8) = pack8(v + 8);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    // every warp of the finishing CTA is past its waits and no other CTA touches these counters again: back to zero
    // for the next launch
    if (ordered && kb == 0 && (int)threadIdx.x < n_it) p.dq_sem[(long long)bh * nq + i_begin + threadIdx.x] = 0;
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, CME_ERR_TIMEOUT);
    if (warp == BWD_WIDE_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, BWD_WIDE_TMEM_COLS); }
}

// dq[b, h, t, :] = scale * acc[b * nh + h, t, :] (bf16, strided destination).  One thread per 8 elements, one (batch, head)
// per grid row, so that no index needs a division by the sequence length (50 + 25 MB: 10.3 us, 18.4 us with divisions).
__global__ void __launch_bounds__(256)
dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int T, int nh, long long sb, long long sh,
                  long long st, float scale) {
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x, t = i >> 3, c = (i & 7) * 8, bh = blockIdx.y;
    if (t >= T) return;
    const float4* src = reinterpret_cast<const float4*>(acc + ((long long)bh * T + t) * HD + c);
    const float4 u = __ldcs(src), v = __ldcs(src + 1);
    const float f[8] = {u.x * scale, u.y * scale, u.z * scale, u.w * scale, v.x * scale, v.y * scale, v.z * scale, v.w * scale};
    *reinterpret_cast<uint4*>(dq + (long long)(bh / nh) * sb + (long long)(bh % nh) * sh + (long long)t * st + c) = pack8(f);
}

// ------------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encoder() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

// bf16 map over (d, t, h, b) with box (64, rows, 1, 1) and 128-byte swizzle.
int make_map4(CUtensorMap* out, const void* base, int T, int nh, int nb, long long st, long long sh, long long sb,
              int rows) {
    EncodeTiledFn enc = encoder();
    CME_REQUIRE(enc != nullptr, CME_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[4] = {(cuuint64_t)HD, (cuuint64_t)T, (cuuint64_t)nh, (cuuint64_t)nb};
    cuuint64_t strides[3] = {(cuuint64_t)st * 2, (cuuint64_t)(nh > 1 ? sh : HD) * 2,
                             (cuuint64_t)(nb > 1 ? sb : (long long)T * st) * 2};
    cuuint32_t box[4] = {(cuuint32_t)HD, (cuuint32_t)rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CME_REQUIRE(r == CUDA_SUCCESS, CME_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed (%d) T=%d nh=%d nb=%d st=%lld",
                (int)r, T, nh, nb, st);
    return CME_OK;
}

// fp32 map over the dQ accumulator [nbh, T, 64]: box (32 columns = 128 bytes, rows, 1), 128-byte swizzle.
int make_map_dq(CUtensorMap* out, const void* base, int T, int nbh, int rows) {
    EncodeTiledFn enc = encoder();
    CME_REQUIRE(enc != nullptr, CME_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[3] = {(cuuint64_t)HD, (cuuint64_t)T, (cuuint64_t)nbh};
    cuuint64_t strides[2] = {(cuuint64_t)HD * 4, (cuuint64_t)T * HD * 4};
    cuuint32_t box[3] = {32, (cuuint32_t)rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CME_REQUIRE(r == CUDA_SUCCESS, CME_ERR_CUDA, "attention: dQ tensor map failed (%d)", (int)r);
    return CME_OK;
}

}  // namespace

// Status word of the attention kernels on the current device (null if the device state cannot be set up).
int* cme_attn_status_ptr() {
    CmeDeviceState* ds;
    return cme_device_state(&ds) ? nullptr : ds->status + CME_STATUS_ATTENTION;
}

int attention_tc_supported(const CmeAttn* a) {
    if (a->dtype != CME_BF16 || a->HD != HD) return 0;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al16(a->q) || !al16(a->k) || !al16(a->v) || !al16(a->o)) return 0;
    if (a->st % 8 || a->ost % 8 || (a->nh > 1 && (a->sh % 8 || a->osh % 8)) || (a->nb > 1 && (a->sb % 8 || a->osb % 8)))
        return 0;
    return 1;
}

// Which kernel a call takes, by how it fills the SMs.  ctas: 128-row tiles of all heads; the small CTAs share an SM by four (forward)
// or two (backward), the wide ones by two or one.  Times in us, wide / small, heads x tokens.
//
// Forward.  Up to two tiles per SM the small CTAs run without enough neighbours: 16 x 1024 13.1 / 19.2 causal, 24 x 582 9.9 / 13.3,
// 192 x 128 6.3 / 6.8, 128 x 256 8.2 / 8.2 (with 129 to 192 tokens up to one: 64 x 192 6.9 / 6.7, 96 x 192 7.9 / 7.0).  Beyond, causal
// calls take the small ones (192 x 256 12.1 / 9.8, 96 x 1024 36.3 / 29.2) but for long sequences just beyond.  With all keys both do a
// full GPU's work at one rate, and the last wave decides: to six tiles per SM the wide ones (64 x 1024 32.5 / 33.6, 80 x 1024 41.3 / 43.7;
// 192 x 582 42.7 / 38.0), then where that of the small ones would be a quarter full.
// The lines were drawn before the small CTAs issued their products faster; near them the small ones are ahead by now (where the
// wide ones run: causal 48 x 1024 22.6 / 20.8; all keys 96 x 1024 48.1 / 47.5, 160 x 1024 71.9 / 68.9).  They have not been drawn anew:
// which kernel runs shows in the last bits of the results.
bool fwd_wide(long long ctas, int T, bool causal, int sms) {
    if (T > 128 && T <= 192) return ctas <= sms;
    if (ctas <= 2ll * sms) return true;
    if (causal) return (T > 512 && 5 * ctas <= 13ll * sms) || (T > 768 && ctas <= 3ll * sms);
    const long long last = ctas % (4ll * sms);
    return (T > 512 && ctas <= 6ll * sms) || (T > 768 && ctas > 8ll * sms && last > 0 && last <= sms);
}
// Backward.  One tile per SM: 16 x 1024 20.9 / 28.4, 24 x 582 15.2 / 19.4, 64 x 256 10.1 / 10.7, 128 x 128 8.2 / 7.9.  Two per SM: the
// small ones (96 x 256 16.9 / 12.6, all keys 24 x 1024 40.9 / 36.6), causal not beyond 448 tokens.  With all keys and an odd number the
// small ones' last wave is half empty (48 x 1024 61.8 / 63.0, 64 x 582 42.7 / 42.2; 192 x 192 26.0 / 19.0).  Else the small ones (causal
// 48 x 1024 47.6 / 38.8, 96 x 1024 83.5 / 65.5; all keys 96 x 1024 125 / 106, 128 x 1024 149 / 138).  These lines, too, are older than
// the faster small CTAs (causal 32 x 1024 36.5 / 31.9, 48 x 582 25.8 / 21.6; all keys 192 x 256 28.3 / 22.8, 80 x 1024 103 / 97, 128 x 582
// 72.5 / 65.2) and stay.
bool bwd_wide(long long ctas, int T, bool causal, int sms) {
    const long long waves = (ctas + sms - 1) / sms;
    if (causal) return waves <= 1 || (waves == 2 && T > 448);
    return waves <= 1 || (waves == 3 && T > 192) || (waves == 5 && T > 512);
}
CME_API int cme_attention_tc_wide(int heads, int T, int causal, int bwd, int num_sms) {
    const long long ctas = (long long)heads * cme_cdiv(T, BQ);
    return bwd ? bwd_wide(ctas, T, causal != 0, num_sms) : fwd_wide(ctas, T, causal != 0, num_sms);
}

int attention_tc_fwd(const CmeAttn* a, cudaStream_t st) {
    CME_REQUIRE(attention_tc_supported(a), CME_ERR_SHAPE, "attention: shape not supported by the tensor-core kernel");
    CME_REQUIRE(a->lse != nullptr, CME_ERR_SHAPE, "attention: lse buffer is required");
    int* const g_attn_status = cme_attn_status_ptr();
    CME_REQUIRE(g_attn_status != nullptr, CME_ERR_CUDA, "attention: device state unavailable");
    CUtensorMap mq, mk, mv, mo;
    int rc, sms;
    if ((rc = cme_num_sms(&sms))) return rc;
    const bool wide = cme_attention_tc_wide(a->nb * a->nh, a->T, a->causal, 0, sms) != 0;
    const int krows = wide ? BKV : FWD_BKV;
    if ((rc = make_map4(&mq, a->q, a->T, a->nh, a->nb, a->st, a->sh, a->sb, 128))) return rc;
    if ((rc = make_map4(&mk, a->k, a->T, a->nh, a->nb, a->st, a->sh, a->sb, krows))) return rc;
    if ((rc = make_map4(&mv, a->v, a->T, a->nh, a->nb, a->st, a->sh, a->sb, krows))) return rc;
    if ((rc = make_map4(&mo, a->o, a->T, a->nh, a->nb, a->ost, a->osh, a->osb, 32))) return rc;
    static bool attr[CME_MAX_DEVICES] = {};               // function attributes are per device
    int dev = 0;
    CME_CUDA(cudaGetDevice(&dev));
    if (!attr[dev % CME_MAX_DEVICES]) {
        CME_CUDA(cudaFuncSetAttribute(attn_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM));
        CME_CUDA(cudaFuncSetAttribute(attn_fwd_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_WIDE_SMEM));
        attr[dev % CME_MAX_DEVICES] = true;
    }
    FwdParams p{a->T, a->nh, a->causal, a->scale * LOG2E, a->lse, g_attn_status};
    const int tiles = cme_cdiv(a->T, BQ), heads = a->nb * a->nh;
    if (wide)
        CME_CUDA(cme_launch_dependent(attn_fwd_wide_kernel, dim3(tiles, heads), dim3(FWD_THREADS), (size_t)FWD_WIDE_SMEM, st, mq, mk,
                                      mv, mo, p));
    else
        CME_CUDA(cme_launch_dependent(attn_fwd_tc_kernel, dim3(heads, tiles), dim3(FWD_THREADS), (size_t)FWD_SMEM, st, mq, mk, mv, mo,
                                      p));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

int attention_delta_launch(const CmeAttn* a, cudaStream_t st, float* clear = nullptr);

int attention_tc_check_bwd(const CmeAttn* a) {
    CME_REQUIRE(attention_tc_supported(a), CME_ERR_SHAPE, "attention: shape not supported by the tensor-core kernel");
    CME_REQUIRE(a->lse && a->delta && a->dq_accum && a->d_o && a->dq && a->dk && a->dv, CME_ERR_SHAPE,
                "attention backward: missing buffer");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    CME_REQUIRE(al16(a->d_o) && al16(a->dq) && al16(a->dk) && al16(a->dv) && al16(a->dq_accum), CME_ERR_SHAPE,
                "attention backward: gradient buffers must be 16-byte aligned");
    CME_REQUIRE(a->dq_mode >= 0 && a->dq_mode <= 2 && (a->dq_mode == 0 || a->dq_sem != nullptr), CME_ERR_SHAPE,
                "attention backward: dq_mode 1 and 2 need the counter array");
    CME_REQUIRE(a->dq_mode != 2 || cme_cdiv(a->T, BQ) <= CME_ATTN_FINISH_MAX_QBLOCKS, CME_ERR_LIMIT,
                "attention backward: dq_mode 2 handles up to %d query blocks", CME_ATTN_FINISH_MAX_QBLOCKS);
    return CME_OK;
}

int attention_tc_bwd(const CmeAttn* a, cudaStream_t st) {
    int rc = attention_tc_check_bwd(a);
    if (rc) return rc;
    int* const g_attn_status = cme_attn_status_ptr();
    CME_REQUIRE(g_attn_status != nullptr, CME_ERR_CUDA, "attention: device state unavailable");
    // delta, and in the same pass over the rows the zeros that the dQ parts are added to
    if ((rc = attention_delta_launch(a, st, a->dq_mode == 0 && !a->dq_accum_clean ? a->dq_accum : nullptr))) return rc;
    CUtensorMap mq, mk, mv, mdo, mdq;
    int sms;
    if ((rc = cme_num_sms(&sms))) return rc;
    const bool finish = a->dq_mode != 0;           // dQ is completed inside the kernel
    const bool wide = finish || cme_attention_tc_wide(a->nb * a->nh, a->T, a->causal, 1, sms) != 0;
    const int qrows = wide ? BQ : BWD_BQ;
    if ((rc = make_map4(&mq, a->q, a->T, a->nh, a->nb, a->st, a->sh, a->sb, qrows))) return rc;
    if ((rc = make_map4(&mk, a->k, a->T, a->nh, a->nb, a->st, a->sh, a->sb, 128))) return rc;
    if ((rc = make_map4(&mv, a->v, a->T, a->nh, a->nb, a->st, a->sh, a->sb, 128))) return rc;
    if ((rc = make_map4(&mdo, a->d_o, a->T, a->nh, a->nb, a->ost, a->osh, a->osb, qrows))) return rc;
    if ((rc = make_map_dq(&mdq, a->dq_accum, a->T, a->nb * a->nh, qrows))) return rc;
    static bool attr[CME_MAX_DEVICES] = {};               // function attributes are per device
    int dev = 0;
    CME_CUDA(cudaGetDevice(&dev));
    if (!attr[dev % CME_MAX_DEVICES]) {
        CME_CUDA(cudaFuncSetAttribute(attn_bwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM));
        CME_CUDA(cudaFuncSetAttribute(attn_bwd_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_WIDE_SMEM));
        attr[dev % CME_MAX_DEVICES] = true;
    }
    if (wide) {
        BwdWideParams p{a->T, a->nh, a->causal, a->scale, a->scale * LOG2E, a->lse, a->delta, a->dq_accum,
                        (__nv_bfloat16*)a->dk, (__nv_bfloat16*)a->dv, a->sb, a->sh, a->st, g_attn_status, a->dq_sem,
                        (__nv_bfloat16*)a->dq, a->dq_mode};
        dim3 grid(cme_cdiv(a->T, BKV), a->nb * a->nh);
        attn_bwd_wide_kernel<<<grid, BWD_WIDE_THREADS, BWD_WIDE_SMEM, st>>>(mq, mk, mv, mdo, mdq, p);
        CME_LAUNCH_CHECK();
        if (finish) return CME_OK;
    } else {
        BwdParams p{a->T, a->nh, a->causal, a->scale, a->scale * LOG2E, a->lse, a->delta, (__nv_bfloat16*)a->dk,
                    (__nv_bfloat16*)a->dv, a->sb, a->sh, a->st, g_attn_status};
        CME_CUDA(cme_launch_dependent(attn_bwd_tc_kernel, dim3(a->nb * a->nh, cme_cdiv(a->T, BKV)), dim3(BWD_THREADS),
                                      (size_t)BWD_SMEM, st, mq, mk, mv, mdo, mdq, p));
        CME_LAUNCH_CHECK();
    }
    CME_CUDA(cme_launch_dependent(dq_convert_kernel, dim3(cme_cdiv(a->T, 32), a->nb * a->nh), dim3(256), 0, st,
                                  (const float*)a->dq_accum, (__nv_bfloat16*)a->dq, a->T, a->nh, a->sb, a->sh, a->st,
                                  a->scale));
    CME_LAUNCH_CHECK();
    return CME_OK;
}

// Reads and clears the attention status word (non-zero: a bounded wait ran out).
CME_API int cme_attention_check_status(int* host_out) {
    return cme_check_status_word(CME_STATUS_ATTENTION, host_out);
}
