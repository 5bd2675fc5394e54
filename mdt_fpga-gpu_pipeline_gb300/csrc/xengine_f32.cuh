// xengine_f32.cuh -- host-visible pieces of the FP32 X-engines.
#pragma once
#include "mdt_common.cuh"

namespace mdt {

// V_c = alpha X_c X_c^H + beta V_c on X[k*ld + e] (blocked 0) or on blocks of 8
// samples X[(k/8)*ld + e*8 + k%8] (blocked 1; 16-byte aligned, the last block
// zero-padded).
mdt_status xengine_herm_f32(int ne, long nbatch, int nsp, const float2 *X,
                            const float2 *const *Xptrs, long ld, long xstride, float2 *V,
                            float2 *const *Vptrs, long ldv, long vstride, float2 alpha,
                            float2 beta, bool beta_zero, cudaStream_t stream, int blocked);
// Its form on the SIMT cores (any number of spectra).
mdt_status xengine_simt_f32(int ne, long nbatch, int nsp, const float2 *X,
                            const float2 *const *Xptrs, long ld, long xstride, float2 *V,
                            float2 *const *Vptrs, long ldv, long vstride, float2 alpha,
                            float2 beta, bool beta_zero, cudaStream_t stream, int blocked);


}  // namespace mdt
