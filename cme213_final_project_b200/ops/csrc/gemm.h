// GEMM interface shared by the tcgen05 kernel, the SIMT fallback and the engine.
//
// One descriptor covers every GEMM site of the reference (FINAL_CLEAN_CODE_/include/kernels.h:6-60:
// gemm_tiled / _AT / _BT, their `_acc` twins, split-K, strided-batched NN / TN / NT) and the epilogues it
// runs as separate kernels (bias+ReLU, bias+residual, ReLU-backward; activations.cu:84-199).
#pragma once
#include "common.h"
#include "gemm_desc.h"

enum CmeAct : int { CME_ACT_NONE = 0, CME_ACT_RELU = 1, CME_ACT_GELU = 2 };

// C[b] (+)= epilogue(A[b] * B[b]);   row-major storage everywhere.
//   a_trans = 0: A stored [M, K] (lda = row stride);  1: A stored [K, M]
//   b_trans = 0: B stored [K, N] (ldb = row stride);  1: B stored [N, K]
//   batch strides are in elements; 0 means the operand is shared by all batches.
// Epilogue, in this order:  acc += bias[n];  aux_out[m,n] = acc (pre-activation, optional);
//   acc = act(acc);  acc *= act'(aux_in[m,n]) (dact);  acc += residual[m,n];  acc += C_old (accumulate).
// aux_deriv != 0 changes what the auxiliary tensor holds: the forward product stores act'(pre-activation) in
//   aux_out instead of the pre-activation (one tanh serves GELU and its derivative), and the backward product
//   multiplies by aux_in as it is -- the derivative is evaluated once, in forward, instead of once more per
//   backward element.  (For ReLU the derivative is the sign of the activation; aux_deriv is ignored.)
// colsum != null asks for column sums of the stored C (a bias gradient when C is the gradient of a pre-activation):
//   the kernel writes one fp32 row of partial sums per 32 rows of C, [ceil(M / 32)][N], and *colsum_slabs receives
//   the number of such rows -- or 0 when the kernel that ran cannot produce them (the caller then sums C itself).
//   cme_colsum_slabs_finalize adds the rows up in a fixed order.
// (struct CmeGemm: gemm_desc.h)

int gemm_tcgen05_supported(const CmeGemm* g);
int gemm_tcgen05_launch(const CmeGemm* g, cudaStream_t stream);
int gemm_kept_splits(const CmeGemm* g);
extern "C" int cme_gemm(const CmeGemm* g, int backend, void* stream);
extern "C" int cme_gemm_sum3(const CmeGemm* g, int backend, void* stream);     // see gemm_tcgen05.cu
int gemm_simt_launch(const CmeGemm* g, cudaStream_t stream);
