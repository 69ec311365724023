// Attention interface shared by the SIMT kernels, the tcgen05 kernels and the engine.
//
// One layout descriptor serves both head layouts of the framework:
//   * "flat": the reference's reinterpretation of the row-major [B*T, D] projection as [B*H, T, HD]
//     (FINAL_CLEAN_CODE_/src/model/transformer.cu:71-75,352-356) -> nb = B*H, nh = 1, batch stride T*HD,
//     row stride HD;
//   * "split": the standard [B, T, H, HD] split -> nb = B, nh = H, batch stride T*D, head stride HD,
//     row stride D.
// Element (b, h, t, d) of Q / K / V / dQ / dK / dV lives at  b*sb + h*sh + t*st + d;  O and dO have their own
// strides (osb, osh, ost), because a fused [B*T, 3D] projection buffer has a different row pitch than O.
#pragma once
#include "common.h"
#include "attention_desc.h"

int attention_simt_fwd(const CmeAttn* a, cudaStream_t st);
int attention_simt_bwd(const CmeAttn* a, cudaStream_t st);
int attention_short_supported(const CmeAttn* a, int bwd);
int attention_short_fwd(const CmeAttn* a, cudaStream_t st);
int attention_short_bwd(const CmeAttn* a, cudaStream_t st);
// Whether backend 0 runs the one-launch kernel for short sequences (no dQ scratch then).
int attention_takes_short(const CmeAttn* a, int bwd);
int attention_gemm_supported(const CmeAttn* a);
int attention_gemm_fwd(const CmeAttn* a, cudaStream_t st);
int attention_gemm_bwd(const CmeAttn* a, cudaStream_t st);
long long attention_gemm_ws_bytes(int nb, int T);
int attention_tc_supported(const CmeAttn* a);
int attention_tc_fwd(const CmeAttn* a, cudaStream_t st);
int attention_tc_bwd(const CmeAttn* a, cudaStream_t st);
int attention_tc_check_bwd(const CmeAttn* a);            // what attention_tc_bwd refuses
