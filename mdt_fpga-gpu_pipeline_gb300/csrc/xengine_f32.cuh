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

// V_rr of an element whose visibilities the tensor-core form leaves to
// xengine_simt_redo, or the first value of a 64 x 64 tile below the diagonal that it leaves
// whole.  Its own results are finite.
__device__ __forceinline__ float2 xf_mark()
{
    return make_float2(__uint_as_float(0x7fc01234u), __uint_as_float(0x7fc05678u));
}
__device__ __forceinline__ bool xf_is_mark(float2 v)
{
    return __float_as_uint(v.x) == 0x7fc01234u && __float_as_uint(v.y) == 0x7fc05678u;
}
// The marked elements' and tiles' visibilities, or all of them, on the SIMT cores with
// sums in two levels.
mdt_status xengine_simt_redo(int ne, long nbatch, int nsp, const float2 *X, const float2 *const *Xptrs,
                             long ld, long xstride, float2 *V, float2 *const *Vptrs, long ldv,
                             long vstride, float2 alpha, float2 beta, bool beta_zero, bool all,
                             cudaStream_t stream, int blocked);

}  // namespace mdt
