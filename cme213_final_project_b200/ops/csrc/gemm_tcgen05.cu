// Host side of the tcgen05 GEMM: tile / split-K planning, tensor maps, dispatch to the kernel instantiation that
// matches the layout and the fused epilogue, split-K reduction kernels and the status word.  The kernel itself is in
// gemm_tcgen05_kernel.cuh; its instantiations live in gemm_tc_inst_*.cu.
#include "gemm_tcgen05_kernel.cuh"

#include <dlfcn.h>
#include <mutex>

using namespace gemm_tc;

// Instantiated elsewhere (one line per launcher; each covers the four operand layouts).
#define CME_GEMM_TC_EXTERN(BN, SIMPLE, PAIR, SPEC)                                                                  \
    extern template int gemm_tc::launch_bn<BN, SIMPLE, PAIR, SPEC>(bool, bool, const CUtensorMap&, const CUtensorMap&, \
                                                                   const CUtensorMap&, const CUtensorMap&,             \
                                                                   const CUtensorMap&, const EpiParams&, int, cudaStream_t);
#include "gemm_tc_inst_list.h"
#undef CME_GEMM_TC_EXTERN

namespace {

// Sums split-K partials in a fixed order and applies the accumulate flag:  C (+)= sum_s P[s].
__global__ void splitk_reduce_kernel(const float* __restrict__ P, int splits, long long per_split, void* Cout,
                                     int c_f32, int accumulate, int M, int N, long long ldc, long long strideC,
                                     int batch) {
    const long long total = (long long)batch * M * N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int k = 0; k < splits; ++k) s += P[k * per_split + i];
        const long long b = i / ((long long)M * N), rem = i % ((long long)M * N);
        const long long off = b * strideC + (rem / N) * ldc + (rem % N);
        if (c_f32) {
            float* C = reinterpret_cast<float*>(Cout);
            C[off] = accumulate ? C[off] + s : s;
        } else {
            __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(Cout);
            C[off] = __float2bfloat16_rn(accumulate ? __bfloat162float(C[off]) + s : s);
        }
    }
}

// Same, four consecutive columns per thread: 16-byte reads of every partial.  The partials' rows are N4 float4 long, which
// may be padding beyond N; `vec`: C takes four columns at once (N, ldc, strideC multiples of 4, C aligned).  The index is
// split with one 32-bit division (Index = unsigned, whenever the partials of one split fit): with 64-bit divisions the
// kernel is bound by them, not by memory (two partials of 3072 x 768 4.8 us, 10.9 us with those; four of 2048 x 512 3.8 and
// 9.0 us).
template <typename Index>
__global__ void __launch_bounds__(256)
splitk_reduce_vec4_kernel(const float4* __restrict__ P, int splits, long long per_split4, void* Cout, int c_f32, int accumulate,
                          int M, int N, int N4, long long ldc, long long strideC, int batch, int vec) {
    pdl_wait();
    const Index total = (Index)batch * M * N4, step = (Index)gridDim.x * blockDim.x;
    for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
        float4 s = P[i];
        int k = 1;
        for (; k + 4 <= splits; k += 4) {          // four loads in flight, added in order
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = P[(k + j) * per_split4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) { s.x += v[j].x; s.y += v[j].y; s.z += v[j].z; s.w += v[j].w; }
        }
        for (; k < splits; ++k) {
            const float4 v = P[k * per_split4 + i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        Index r = i / N4, b = 0;
        const int c = (int)(i - r * N4) * 4;
        if (batch > 1) { b = r / M; r -= b * M; }
        const long long off = (long long)b * strideC + (long long)r * ldc + c;
        if (!vec) {
            const float t[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (c + j < N) {
                    if (c_f32) {
                        float* C = reinterpret_cast<float*>(Cout) + off + j;
                        *C = accumulate ? *C + t[j] : t[j];
                    } else {
                        __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(Cout) + off + j;
                        *C = __float2bfloat16_rn(accumulate ? __bfloat162float(*C) + t[j] : t[j]);
                    }
                }
            }
        } else if (c_f32) {
            float4* C = reinterpret_cast<float4*>(reinterpret_cast<float*>(Cout) + off);
            if (accumulate) { const float4 o = *C; s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w; }
            *C = s;
        } else {
            uint2* C = reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(Cout) + off);
            if (accumulate) {
                const uint2 o = *C;
                const float2 a = bf2_to_f2(o.x), d = bf2_to_f2(o.y);
                s.x += a.x; s.y += a.y; s.z += d.x; s.w += d.y;
            }
            *C = make_uint2(f2_to_bf2(s.x, s.y), f2_to_bf2(s.z, s.w));
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encoder() {
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

// 3-D tensor map: dims (inner, rows, batch), 128-byte swizzle, box (128 bytes of inner, box_rows, 1).
int make_tmap(CUtensorMap* out, const void* base, long long inner, long long rows, long long ld, long long batch,
              long long batch_stride, int box_rows, bool f32 = false, bool round_tf32 = false,
              bool mn_major = false) {
    EncodeTiledFn enc = get_encoder();
    CME_REQUIRE(enc != nullptr, CME_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const int es = f32 ? 4 : 2;
    cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)(batch > 0 ? batch : 1)};
    cuuint64_t strides[2] = {(cuuint64_t)ld * es, (cuuint64_t)(batch_stride > 0 ? batch_stride : ld * rows) * es};
    cuuint32_t box[3] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    // operands of a tf32 product are rounded to tf32 (to nearest) by the copy engine on their way into shared
    // memory; the tensor core would otherwise just drop the low mantissa bits, a one-sided error
    const CUtensorMapDataType dt = !f32 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                        : round_tf32 ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    CUresult r = enc(out, dt, 3,
                     const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     round_tf32 && mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CME_REQUIRE(r == CUDA_SUCCESS, CME_ERR_CUDA,
                "cuTensorMapEncodeTiled failed (%d): inner=%lld rows=%lld ld=%lld batch=%lld bstride=%lld box_rows=%d",
                (int)r, inner, rows, ld, batch, batch_stride, box_rows);
    return CME_OK;
}

// How many CTA pairs of the pair kernel can be resident at once (the persistent grid must not exceed it: a pair
// that is not resident would only start when another has finished all of its tiles).
int query_max_pairs(int num_sms) {
    auto kern = gemm_tc_kernel<256, false, false, true, true, -1>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<256, true, true>::SMEM_BYTES) !=
        cudaSuccess) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * num_sms);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = Cfg<256, true, true>::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}

}  // namespace

static int gemm_tcgen05_run(const CmeGemm* g, cudaStream_t stream, bool sum3);

CME_API int cme_gemm_status_word(int** out) {
    CmeDeviceState* ds;
    int rc = cme_device_state(&ds);
    if (rc) return rc;
    *out = ds->status + CME_STATUS_GEMM;
    return CME_OK;
}

// How the operands of a product lie in memory, as far as the time of their loads depends on it.
struct OperandLayout {
    bool a_mn, b_mn;               // stored along M / N instead of along K
    long long a_pitch, b_pitch;    // bytes from row to row
};

// Tile shape and K splits for a product: the smallest estimated time.  Pure host arithmetic.
//   force_bn: 0 = choose; 64 / 128 / 256 = tile width on one CTA; 512 / 384 = the 256 x 256 / 256 x 192 tile on a CTA pair
//   force_splits: 0 = choose.  Split-K needs the plain epilogue, a workspace for the fp32 partials and at least
//   four 64-deep k-blocks per split.
// The estimate, in us: a start that depends on the tile (launch, first loads, last stores), then for every wave of tiles a time per
// tile and one per 128-byte k-block.  A k-block takes what its tile needs alone (issuing its MMAs, or the tensor pipe's rate), or as
// long as L2 takes to deliver the k-blocks of all SMs that load: 22 TB/s.  Rows that do not start on 128-byte lines cost up to 1.4
// times that, on odd 16-byte pieces twice.  Constants: least squares over 33000 products (1400 shapes of 128-50304 x 128-50304 x
// 128-50304, every tile, 1-16 splits).  The plan is then 0.75 % slower than the best one on average (2.5-3 % with the constants
// from before the k-blocks got faster), at most 1.2 times.
static void plan_tiles(int M, int N, int K, int batch, bool plain_epi, long long workspace_bytes, int num_sms,
                       int max_pairs, int force_bn, int force_splits, int* bn_out, bool* pair_out, int* splits_out,
                       const OperandLayout& at, int bk = 64, double* us_out = nullptr) {
    const int num_kb = cme_cdiv(K, bk);
    int bn = force_bn, splits = force_splits;
    bool pair = false;
    if (bn == 512 || bn == 384) { bn /= 2; pair = true; }
    if (!bn || !splits) {
        struct Tile { int bn; bool pair; double kblock[2], unit[2], start[2]; };          // [bf16, tf32]
        static const Tile tiles[5] = {{256, true, {0.268, 0.279}, {1.01, 1.31}, {3.58, 4.01}},
                                      {256, false, {0.305, 0.305}, {0.98, 1.57}, {3.18, 3.21}},
                                      {128, false, {0.190, 0.182}, {0.42, 0.56}, {2.96, 3.37}},
                                      {64, false, {0.147, 0.151}, {0.22, 0.33}, {2.75, 3.05}},
                                      {192, true, {0.232, 0.0}, {0.80, 0.0}, {3.39, 0.0}}};
        const int t32 = bk == 32;
        const double l2_bytes = t32 ? 21.5e6 : 22.2e6;       // per us, all SMs together
        // shares of the operands whose rows leave the 128-byte lines (along K, along M / N) or the 32-byte sectors, and what they
        // add to the time of a k-block alone (k) and to that of L2 (l)
        static const double line_k[2][2] = {{0.21, 0.40}, {0.21, 0.07}}, line_l[2][2] = {{0.17, 0.165}, {0.255, 0.11}};
        static const double sector_l[2] = {0.82, 0.20};
        double best = 1e30;
        int best_bn = 128, best_s = 1;
        bool best_pair = false;
        for (int i = 0; i < 5; ++i) {
            const Tile& t = tiles[i];
            const bool pr = t.pair;
            if (t.bn == 192 && t32) continue;
            if (pr && (max_pairs <= 0 || M <= BM)) continue;
            if (force_bn && force_bn != (pr ? 2 : 1) * t.bn) continue;
            if (t.bn > 64 && N <= t.bn / 2) continue;                // tile mostly padding
            const long long count = (long long)cme_cdiv(M, pr ? 2 * BM : BM) * cme_cdiv(N, t.bn) * batch;
            const int slots = pr ? max_pairs : num_sms;
            // bytes that an SM loads per k-block (half of a 192-column tile stored along N arrives as two groups of 64)
            const double a_bytes = BM * BK_BYTES;
            const double b_bytes = BK_BYTES * (!pr ? t.bn : t.bn == 192 && !at.b_mn ? 96 : 128);
            double more_k = 1.0, more_l = 1.0;
            auto operand = [&](bool mn, long long pitch, double share) {
                if (pitch % 128) { more_k += share * line_k[t32][mn]; more_l += share * line_l[t32][mn]; }
                if (pitch % 32) more_l += share * sector_l[t32];
            };
            operand(at.a_mn, at.a_pitch, a_bytes / (a_bytes + b_bytes));
            operand(at.b_mn, at.b_pitch, b_bytes / (a_bytes + b_bytes));
            const double alone = t.kblock[t32] * more_k * (t32 ? 1.0 + 0.034 * ((int)at.a_mn + (int)at.b_mn) : 1.0);
            for (int s = 1; s <= 16; ++s) {
                if (force_splits && s != force_splits) continue;
                if (s > 1 && (!plain_epi || num_kb / s < 4 || (long long)s * batch * M * N * 4 > workspace_bytes)) break;
                const int kb = cme_cdiv(num_kb, s), parts = cme_cdiv(num_kb, kb);
                const long long units = count * parts;
                const double waves = (double)((units + slots - 1) / slots);
                const double loading = (double)(units < slots ? units : slots) * (pr ? 2 : 1);
                const double shared = (a_bytes + b_bytes) * more_l * loading / l2_bytes;
                double est = t.start[t32] + waves * (kb * (alone > shared ? alone : shared) + t.unit[t32]);
                // the reduction's launch, the partials written and read
                if (parts > 1) est += (t32 ? 1.65 : 2.17) + (double)parts * M * N * batch * (t32 ? 5.5e-7 : 5.9e-7);
                if (est < best) { best = est; best_bn = t.bn; best_s = s; best_pair = pr; }
            }
        }
        if (!bn) { bn = best_bn; pair = best_pair; }
        if (!splits) splits = best_s;
        if (us_out) *us_out = best;
    }
    *bn_out = bn; *pair_out = pair; *splits_out = splits;
}

// K splits of the engine's bf16 products.  A training step keeps the order of its sums from one version to the next: Adam's first steps
// divide each gradient by its own size, so one result that rounds the other way can turn a step of a parameter round, and a run from
// the same seed ends 3 % elsewhere (parity model of width 512, 45 x 64 tokens, the splits of plan_tiles).  So the number is that of the
// estimate that the engine has always had, with k-blocks at their former pace; the tile's width, which changes no sum, comes from
// plan_tiles.  us a step with these splits / with the plan's: char-gpt 2114 / 2115, GPT-2 small 15240 / 15180, width 512 over 45 x 64
// tokens 212 / 201 (512 x 512 x 2048 takes 8 splits where 4 are planned).
static int kept_splits(int M, int N, int K, int batch, bool plain_epi, long long workspace_bytes, int num_sms, int max_pairs) {
    const int num_kb = cme_cdiv(K, 64);
    static const struct { int bn; bool pair; double per_step; } tiles[4] = {{256, true, 136.0}, {256, false, 168.0},
                                                                            {128, false, 138.0}, {64, false, 140.0}};
    double best = 1e30;
    int best_s = 1;
    for (const auto& t : tiles) {
        if ((t.pair && (max_pairs <= 0 || M <= BM)) || (t.bn > 64 && N <= t.bn / 2)) continue;
        const long long count = (long long)cme_cdiv(M, t.pair ? 2 * BM : BM) * cme_cdiv(N, t.bn) * batch;
        const int slots = t.pair ? max_pairs : num_sms;
        for (int s = 1; s <= 16; ++s) {
            if (s > 1 && (!plain_epi || num_kb / s < 4 || (long long)s * batch * M * N * 4 > workspace_bytes)) break;
            const double waves = (double)((count * s + slots - 1) / slots), kb = (double)cme_cdiv(num_kb, s);
            double est = waves * ((kb + 2.0) * 4.0 * t.per_step + 6.0 * 4.0 * t.bn / 2.0) + (t.pair ? 2000.0 : 0.0);
            if (s > 1) est += 6000.0 + (double)s * M * N * batch / num_sms / 16.0;
            if (est < best) { best = est; best_s = s; }
        }
    }
    return best_s;
}

static int pairs_of(CmeDeviceState* ds) {
    if (ds->max_pairs < 0) {
        const char* e = getenv("CME213_GEMM_PAIR");
        ds->max_pairs = (e && e[0] == '0') ? 0 : query_max_pairs(ds->num_sms);
    }
    return ds->max_pairs;
}

// The same for a product's descriptor on the current device; 0: planned as any other.
int gemm_kept_splits(const CmeGemm* g) {
    CmeDeviceState* ds;
    if (g->ab_dtype != CME_BF16 || cme_device_state(&ds)) return 0;
    const bool plain_epi = !g->bias && !g->residual && !g->aux_out && !g->act && !g->dact;
    return kept_splits(g->M, g->N, g->K, g->batch, plain_epi, g->workspace ? g->workspace_bytes : 0, ds->num_sms, pairs_of(ds));
}

// ... and without a device.
CME_API int cme_gemm_kept_splits(int M, int N, int K, int batch, int plain_epilogue, long long workspace_bytes, int num_sms,
                                 int max_pairs) {
    return kept_splits(M, N, K, batch, plain_epilogue != 0, workspace_bytes, num_sms, max_pairs);
}

// The plan the launcher would choose for operands stored along K, without a device: `num_sms` SMs, `max_pairs` co-resident CTA
// pairs (0 = no cluster launches).  out = {tile width, pair (0/1), splits}.
CME_API int cme_gemm_plan(int M, int N, int K, int batch, int plain_epilogue, long long workspace_bytes, int num_sms,
                          int max_pairs, int force_bn, int force_splits, int* out) {
    CME_REQUIRE(M > 0 && N > 0 && K > 0 && batch > 0 && num_sms > 0, CME_ERR_SHAPE, "gemm plan: empty problem");
    int bn = 0, splits = 0;
    bool pair = false;
    plan_tiles(M, N, K, batch, plain_epilogue != 0, workspace_bytes, num_sms, max_pairs, force_bn, force_splits, &bn,
               &pair, &splits, {false, false, K * 2ll, K * 2ll});
    out[0] = bn; out[1] = pair ? 1 : 0; out[2] = splits;
    return CME_OK;
}

// The same for a plain tf32 product with `mn_operands` operands (0, 1, 2) stored along M or N.
CME_API int cme_gemm_plan_tf32(int M, int N, int K, int mn_operands, long long workspace_bytes, int num_sms, int max_pairs,
                               int* out) {
    CME_REQUIRE(M > 0 && N > 0 && K > 0 && num_sms > 0, CME_ERR_SHAPE, "gemm plan: empty problem");
    bool pair = false;
    const bool a_mn = mn_operands > 1, b_mn = mn_operands > 0;
    plan_tiles(M, N, K, 1, true, workspace_bytes, num_sms, max_pairs, 0, 0, &out[0], &pair, &out[2],
               {a_mn, b_mn, (a_mn ? M : K) * 4ll, (b_mn ? N : K) * 4ll}, 32);
    out[1] = pair ? 1 : 0;
    return CME_OK;
}

int gemm_tcgen05_supported(const CmeGemm* g) {
    const bool tf32 = g->ab_dtype == CME_F32;
    // fp32 operands run as tf32, and only where the caller allows the reduced input precision: plain products
    // (fp32 output, optionally accumulated), rows of C addressable in 16-byte units
    if (tf32 && (!g->allow_tf32 || g->c_dtype != CME_F32 || g->bias || g->residual || g->aux_out || g->aux_in ||
                 g->act || g->dact || g->N % 4 || g->ldc % 4 || (g->batch > 1 && g->strideC % 4)))
        return 0;
    // Which fp32 products run as tf32 shows in their results, so without the caller's word for all of them (allow_tf32 = 2) the
    // line lies where it always lay: with an operand stored along M or N, K is a multiple of four and those operands take up
    // to half of the workspace (a K-major copy of each had to fit there once).  The others keep all 24 bits of their inputs on
    // the CUDA cores: as tf32 the weight gradients of a 9749 x 152 x 608 feed-forward block are 1.3 and 1.4 times as far from
    // 64-bit sums, and 20 times as fast (8192 x 512 x 2048: 39 us for 788).
    if (tf32 && g->allow_tf32 < 2 && (g->a_trans || !g->b_trans)) {
        const long long na = g->a_trans ? (long long)(g->strideA ? g->batch : 1) * g->M * g->K : 0;
        const long long nb = !g->b_trans ? (long long)(g->strideB ? g->batch : 1) * g->N * g->K : 0;
        if (g->K % 4 || !g->workspace || (na + nb) * 4 + 512 > g->workspace_bytes / 2) return 0;
    }
    // the tf32 variants only store: an accumulating product adds its fp32 result from the workspace
    if (tf32 && g->accumulate && (!g->workspace || (long long)g->batch * g->M * g->N * 4 > g->workspace_bytes)) return 0;
    if (!tf32 && g->ab_dtype != CME_BF16) return 0;
    if (g->M <= 0 || g->N <= 0 || g->K <= 0 || g->batch <= 0) return 0;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al16(g->A) || !al16(g->B) || !al16(g->C)) return 0;
    const int unit = tf32 ? 4 : 8;                           // elements per 16 bytes
    if (g->lda % unit || g->ldb % unit || g->strideA % unit || g->strideB % unit) return 0;
    // Extents need not be multiples of the 16-byte unit: row pitches are (checked above), and a box that reaches
    // past an extent reads zeros.  Degenerate extents go to the SIMT kernel.
    const long long innerA = g->a_trans ? g->M : g->K, innerB = g->b_trans ? g->K : g->N;
    if (innerA < unit || innerB < unit) return 0;
    if (g->c_dtype == CME_F32 && (g->act || g->dact || g->residual || g->aux_out)) return 0;
    return 1;
}

// Whether cme_gemm_sum3 has three products made by one launch: where that is the shorter way. Its 64-wide tiles pass over the k-blocks of all three,
// against three launches with the tiles that suit one (parity-h128, 2048 x 128 x 128: 5.1 us for 12.9; 16384 x 512 x 512 planned as
// three).
CME_API int cme_gemm_sum3_planned(const CmeGemm* g) {
    if (g->batch != CHAIN || g->ab_dtype != CME_BF16 || g->c_dtype != CME_BF16 || !g->strideA || !g->strideB || g->bias || g->residual ||
        g->aux_out || g->aux_in || g->act || g->dact || g->accumulate || g->force_bn || g->force_splits > 1 || g->ldc % 8 ||
        !gemm_tcgen05_supported(g))
        return 0;
    CmeDeviceState* ds;
    if (cme_device_state(&ds)) return 0;
    int bn = 0, splits = 0;
    bool pair = false;
    double one = 0.0, three = 0.0;
    const OperandLayout at = {g->a_trans != 0, g->b_trans == 0, g->lda * 2, g->ldb * 2};
    plan_tiles(g->M, g->N, g->K, 1, false, 0, ds->num_sms, pairs_of(ds), 0, 0, &bn, &pair, &splits, at, 64, &one);
    bn = 64; splits = 0;
    plan_tiles(g->M, g->N, cme_cdiv(g->K, 64) * 64 * CHAIN, 1, false, 0, ds->num_sms, 0, 64, 0, &bn, &pair, &splits, at, 64, &three);
    return three < CHAIN * one;
}

int gemm_tcgen05_launch(const CmeGemm* g, cudaStream_t stream) { return gemm_tcgen05_run(g, stream, false); }

// sum3: batch entry 0, + 1 and + 2 go to the same C, which is rounded after each.
static int gemm_tcgen05_run(const CmeGemm* g, cudaStream_t stream, bool sum3) {
    CME_REQUIRE(gemm_tcgen05_supported(g), CME_ERR_SHAPE, "gemm shape/alignment not supported by the tcgen05 kernel");
    CmeDeviceState* ds;
    {
        int rc0 = cme_device_state(&ds);
        if (rc0) return rc0;
    }
    const int g_num_sms = ds->num_sms, g_max_pairs = pairs_of(ds);
    int* const g_status = ds->status + CME_STATUS_GEMM;
    const bool tf32 = g->ab_dtype == CME_F32;
    const int BK = tf32 ? 32 : 64;                            // K elements per 128-byte k-block
    int tiles_m = cme_cdiv(g->M, BM);
    const int num_kb = cme_cdiv(g->K, BK);
    const bool plain_epi = !g->bias && !g->residual && !g->aux_out && !g->act && !g->dact;
    int bn = 0, splits = 0;
    bool pair = false;
    const int batch = sum3 ? 1 : g->batch;
    if (sum3) { bn = 64; splits = 1; }
    else plan_tiles(g->M, g->N, g->K, g->batch, plain_epi, g->workspace ? g->workspace_bytes : 0, g_num_sms, g_max_pairs,
               g->force_bn, g->force_splits, &bn, &pair, &splits,
               {g->a_trans != 0, g->b_trans == 0, g->lda * (tf32 ? 4 : 2), g->ldb * (tf32 ? 4 : 2)}, BK);
    // A tf32 product that accumulates into C goes through the fp32 workspace like a split-K product (one "split"
    // is then added to C by the reduction kernel): the tf32 kernel variants only store.
    const bool via_ws = splits > 1 || (tf32 && g->accumulate);
    if (tf32 && g->accumulate)
        CME_REQUIRE(g->workspace && (long long)splits * g->batch * g->M * g->N * 4 <= g->workspace_bytes, CME_ERR_LIMIT,
                    "tf32 accumulate needs an fp32 workspace of M x N");
    CME_REQUIRE(bn == 64 || bn == 128 || bn == 256 || (bn == 192 && pair && !tf32), CME_ERR_SHAPE,
                "tile width must be 64, 128, 256, 512 (pair) or, in bf16, 384 (pair, 192 columns)");
    CME_REQUIRE(!pair || g_max_pairs > 0, CME_ERR_SHAPE, "CTA-pair tiles are not available on this device");
    if (pair) tiles_m = cme_cdiv(g->M, 2 * BM);
    static const bool trace = getenv("CME213_GEMM_TRACE") != nullptr;
    if (trace)
        fprintf(stderr, "[gemm] M=%d N=%d K=%d batch=%d at=%d bt=%d -> bn=%d pair=%d splits=%d\n", g->M, g->N, g->K,
                g->batch, g->a_trans, g->b_trans, bn, (int)pair, splits);
    const int tiles_n = cme_cdiv(g->N, bn);
    const long long tiles = (long long)tiles_m * tiles_n * batch;
    if (splits > 1) {
        CME_REQUIRE(plain_epi, CME_ERR_SHAPE, "split-K supports only the plain / accumulate epilogue");
        CME_REQUIRE(g->workspace && (long long)splits * g->batch * g->M * g->N * 4 <= g->workspace_bytes,
                    CME_ERR_LIMIT, "split-K workspace too small");
    }
    int kb_per = cme_cdiv(num_kb, splits);
    splits = cme_cdiv(num_kb, kb_per);

    CUtensorMap ta, tb;
    int rc;
    // A: K-major -> map (K, M), box (64, 128); MN-major -> map (M, K), box (64, 64)
    if (!g->a_trans) rc = make_tmap(&ta, g->A, g->K, g->M, g->lda, g->strideA ? g->batch : 1, g->strideA, BM, tf32, tf32);
    else             rc = make_tmap(&ta, g->A, g->M, g->K, g->lda, g->strideA ? g->batch : 1, g->strideA, BK, tf32, tf32, true);
    if (rc) return rc;
    // B: stored [N, K] (b_trans) is K-major -> map (K, N), box (64, bn); stored [K, N] -> map (N, K), box (64, 64)
    if (g->b_trans) rc = make_tmap(&tb, g->B, g->K, g->N, g->ldb, g->strideB ? g->batch : 1, g->strideB,
                                   pair ? bn / 2 : bn, tf32, tf32);
    else            rc = make_tmap(&tb, g->B, g->N, g->K, g->ldb, g->strideB ? g->batch : 1, g->strideB, BK, tf32, tf32, true);
    if (rc) return rc;

    EpiParams ep{};
    ep.M = g->M; ep.N = g->N; ep.K = g->K; ep.batch = batch;
    ep.tiles_m = tiles_m; ep.tiles_n = tiles_n; ep.splits = splits; ep.kb_per_split = kb_per; ep.num_kb = num_kb;
    ep.a_batched = g->strideA != 0 && g->batch > 1; ep.b_batched = g->strideB != 0 && g->batch > 1;
    {
        // Tile order by estimated DRAM traffic.  The CTAs that run together walk K at about the same pace, so the
        // operand they share is fetched once per wave of tiles from DRAM and served to the others from L2; the
        // operand they do not share is needed again a wave later and comes from DRAM again unless it stays in L2
        // (taken as half of its 126 MB).  So the order that shares the operand too large for L2 wins.
        const int es = tf32 ? 4 : 2;
        const double a_bytes = (double)g->M * g->K * es, b_bytes = (double)g->N * g->K * es, l2 = 63.0e6;
        const double slots = pair ? (double)g_max_pairs : (double)g_num_sms;
        const double waves = (double)tiles_m * tiles_n / slots > 1.0 ? (double)tiles_m * tiles_n / slots : 1.0;
        const double ra = waves < tiles_n ? waves : tiles_n, rb = waves < tiles_m ? waves : tiles_m;
        const double m_fast = a_bytes * (a_bytes > l2 ? ra : 1.0) + b_bytes;         // B stripe shared, A rows distinct
        const double n_fast = b_bytes * (b_bytes > l2 ? rb : 1.0) + a_bytes;         // A rows shared
        static const char* force = getenv("CME213_GEMM_NFAST");
        // At equal traffic a large A is walked row by row too: all of its tiles of a row run together, so each wave fetches its own
        // part of A.  The other way the first wave fetches all of it and the later ones wait for nothing (16384 x 384 x 1536 bf16
        // 20.0 -> 18.2 us, 16384 x 768 x 2304 tf32 96.6 -> 83; 592 products: 0.9 % faster on average, the worst 1.08 times slower;
        // from 16 MB on instead of 4, 0.6 %).
        const bool tie = n_fast == m_fast && a_bytes > b_bytes && a_bytes > 4e6;
        ep.n_fast = force ? (force[0] == '1') : ((n_fast < m_fast || tie) && tiles_n > 1);
        // the stored derivative is written once by forward and read once by backward, a layer's worth of other work
        // apart: keep it from displacing what the neighbouring kernels re-read (CME213_GEMM_STREAM_AUX=0: off)
        static const bool stream_aux = !(getenv("CME213_GEMM_STREAM_AUX") && getenv("CME213_GEMM_STREAM_AUX")[0] == '0');
        ep.stream_aux = (stream_aux && g->aux_deriv && (g->act == CME_ACT_GELU || g->dact == CME_ACT_GELU)) ? 1 : 0;
    }
    ep.status = g_status;
    ep.div_fast.set(ep.n_fast ? tiles_n : tiles_m);
    ep.div_mn.set(tiles_m * tiles_n);
    ep.div_batch.set(batch);
    // Partial rows are padded to whole 16-byte words where the workspace has room: they then leave by TMA stores and are
    // read back four columns at a time also when N is odd, like the 65-column output head's weight gradient.
    const int n_pad = (g->N + 3) / 4 * 4;
    const int ldw = (long long)splits * g->batch * g->M * n_pad * 4 <= g->workspace_bytes &&
                            (reinterpret_cast<uintptr_t>(g->workspace) & 15) == 0 ? n_pad : g->N;
    if (via_ws) {
        ep.C = g->workspace; ep.ldc = ldw; ep.strideC = (long long)g->M * ldw; ep.c_f32 = 1;
    } else {
        ep.C = g->C; ep.ldc = g->ldc; ep.strideC = g->strideC; ep.c_f32 = g->c_dtype == CME_F32;
        ep.bias = reinterpret_cast<const __nv_bfloat16*>(g->bias);
        ep.residual = g->residual; ep.ldres = g->ldres;
        ep.aux_out = g->aux_out; ep.aux_in = g->aux_in; ep.ldaux = g->ldaux;
        ep.act = g->act; ep.dact = g->dact; ep.accumulate = g->accumulate;
        ep.aux_deriv = (g->aux_deriv && (g->act == CME_ACT_GELU || g->dact == CME_ACT_GELU)) ? 1 : 0;
    }
    if (g->colsum_slabs) *g->colsum_slabs = 0;
    // Outputs through shared-memory staging + TMA tile stores when rows are 16-byte addressable.
    CUtensorMap tc = ta, tx = ta, ti = ta;
    {
        const int es = ep.c_f32 ? 4 : 2;
        auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
        const long long nb = (long long)splits * batch;
        bool ok = al16(ep.C) && (ep.ldc * es) % 16 == 0 && (nb == 1 || (ep.strideC * es) % 16 == 0);
        if (ep.aux_out) ok = ok && al16(ep.aux_out) && (ep.ldaux * 2) % 16 == 0;
        if (ok) {
            rc = make_tmap(&tc, ep.C, g->N, g->M, ep.ldc, nb, nb > 1 ? ep.strideC : 0, 32, ep.c_f32 != 0);
            if (rc) return rc;
            if (ep.aux_out) {
                rc = make_tmap(&tx, ep.aux_out, g->N, g->M, ep.ldaux, g->batch, g->batch > 1 ? ep.strideC : 0, 32);
                if (rc) return rc;
            }
            ep.tma_store = 1;
            // The operand the fused epilogue reads per output element comes in by TMA, chunk by chunk, ahead of use.
            if (!ep.c_f32) {
                const void* ib = nullptr;
                long long ild = 0;
                int kind = 0;
                if (ep.dact) { ib = ep.aux_in; ild = ep.ldaux; kind = 1; }
                else if (ep.residual) { ib = ep.residual; ild = ep.ldres; kind = 2; }
                else if (ep.accumulate) { ib = ep.C; ild = ep.ldc; kind = 3; }
                if (kind && al16(ib) && (ild * 2) % 16 == 0 && (g->batch == 1 || (ep.strideC * 2) % 16 == 0)) {
                    rc = make_tmap(&ti, ib, g->N, g->M, ild, g->batch, g->batch > 1 ? ep.strideC : 0, 32);
                    if (rc) return rc;
                    ep.in_kind = kind;
                }
                ep.aux_ring = ep.aux_out && !ep.in_kind;
            }
        }
    }
    const long long total = tiles * splits;
    const int grid = pair ? 2 * (int)(total < g_max_pairs ? total : g_max_pairs)
                          : (int)(total < g_num_sms ? total : g_num_sms);
    const bool a_mn = g->a_trans != 0, b_mn = g->b_trans == 0;
    const bool simple = !sum3 && ep.tma_store && !ep.c_f32 && !ep.bias && !ep.residual && !ep.aux_out && !ep.aux_in &&
                        !ep.act && !ep.dact && !ep.accumulate;
    int spec = -1, spec_colsum = -1;
    CME_REQUIRE(!sum3 || ep.tma_store, CME_ERR_SHAPE, "sum of three products: output rows are not 16-byte addressable");
    if (sum3) {
        spec = SPEC_SUM3;
    } else if (!simple) {
        if (ep.tma_store && !ep.c_f32) {
            spec = spec_pack(ep.bias != nullptr, ep.act, ep.dact, ep.residual != nullptr, ep.accumulate != 0,
                             ep.aux_out != nullptr, ep.in_kind, ep.aux_ring != 0, ep.aux_deriv != 0, false);
            // column sums ride in the variants whose input arrives through the ring (one output buffer per chunk)
            if (g->colsum && g->colsum_slabs && splits == 1 && g->batch == 1 && ep.in_kind == 1 && ep.dact)
                spec_colsum = spec | (1 << 13);
        } else if (ep.tma_store && ep.c_f32 && !ep.accumulate) {
            spec = tf32 ? SPEC_TF32 : SPEC_F32;
        }
    }
    CME_REQUIRE(!tf32 || spec == SPEC_TF32, CME_ERR_SHAPE, "tf32 product: output rows are not 16-byte addressable");
    // the instantiation with this tile, pairing and compile-time epilogue (first with the column sums, if asked
    // for); else the run-time epilogue of that tile
    rc = -1;
    for (int attempt = 0; attempt < 3 && rc == -1; ++attempt) {
        const int want = attempt == 0 ? spec_colsum : attempt == 1 ? spec : -1;
        if (attempt == 0 && want < 0) continue;
        ep.colsum = attempt == 0 ? g->colsum : nullptr;
#define CME_GEMM_TC_EXTERN(BN, SIMPLE, PAIR, SPEC)                                              \
    if (rc == -1 && bn == BN && simple == SIMPLE && pair == PAIR && want == SPEC)               \
        rc = launch_bn<BN, SIMPLE, PAIR, SPEC>(a_mn, b_mn, ta, tb, tc, tx, ti, ep, grid, stream);
#include "gemm_tc_inst_list.h"
#undef CME_GEMM_TC_EXTERN
        if (rc == CME_OK && attempt == 0) *g->colsum_slabs = cme_cdiv(g->M, 32);
    }
    CME_REQUIRE(rc != -1, CME_ERR_SHAPE, "gemm: no kernel instantiation for tile %d pair %d", bn, (int)pair);
    if (rc) return rc;
    if (via_ws) {
        const long long per = (long long)g->batch * g->M * ldw;
        const bool f32 = g->c_dtype == CME_F32;
        const bool vec = g->N % 4 == 0 && g->ldc % 4 == 0 && (g->batch == 1 || g->strideC % 4 == 0) &&
                         (reinterpret_cast<uintptr_t>(g->C) & (f32 ? 15 : 7)) == 0;
        if (ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(g->workspace) & 15) == 0) {
            const long long per4 = per / 4;
            const int blocks = (int)((per4 + 255) / 256 < 8 * g_num_sms ? (per4 + 255) / 256 : 8 * g_num_sms);
            auto kernel = cme_index32(per4) ? splitk_reduce_vec4_kernel<unsigned>
                                            : splitk_reduce_vec4_kernel<unsigned long long>;
            CME_CUDA(cme_launch_dependent(kernel, dim3(blocks), dim3(256), 0, stream,
                                          reinterpret_cast<const float4*>(g->workspace), splits, per4, g->C, (int)f32,
                                          g->accumulate, g->M, g->N, ldw / 4, g->ldc, g->strideC, g->batch, (int)vec));
        } else {
            const int blocks = (int)((per + 255) / 256 < 4096 ? (per + 255) / 256 : 4096);
            splitk_reduce_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const float*>(g->workspace), splits, per,
                                                             g->C, f32, g->accumulate, g->M, g->N, g->ldc, g->strideC,
                                                             g->batch);
        }
        CME_LAUNCH_CHECK();
    }
    return CME_OK;
}

// C = round(round(A0 B0) + A1 B1) + A2 B2, rounded: three products that accumulate into C in bf16, in one launch where
// that is planned.  g->batch = 3, strideA and strideB lead from one to the next, strideC is not used.
CME_API int cme_gemm_sum3(const CmeGemm* g, int backend, void* stream) {
    if (backend != 2 && cme_gemm_sum3_planned(g)) return gemm_tcgen05_run(g, reinterpret_cast<cudaStream_t>(stream), true);
    CmeGemm one = *g;
    one.batch = 1; one.strideA = one.strideB = one.strideC = 0;
    const long long es = g->ab_dtype == CME_F32 ? 4 : 2;
    for (int i = 0; i < CHAIN; ++i) {
        one.A = (const char*)g->A + i * g->strideA * es;
        one.B = (const char*)g->B + i * g->strideB * es;
        one.accumulate = i > 0 || g->accumulate;
        const int rc = cme_gemm(&one, backend, stream);
        if (rc) return rc;
    }
    return CME_OK;
}

// Reads and clears the device status word (0 = every bounded wait completed).
CME_API int cme_gemm_check_status(int* host_out) { return cme_check_status_word(CME_STATUS_GEMM, host_out); }
