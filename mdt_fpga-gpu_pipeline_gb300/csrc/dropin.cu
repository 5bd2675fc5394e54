// dropin.cu -- the reference's three __global__ kernels with their exact
// signatures (reference MDT_device_functions.h:44-46), so that a caller that
// launches them with <<<grid, block, 0, stream>>> links against this library
// unchanged; plus C-ABI launchers and the library's error plumbing.
//
// Semantics follow the reference kernels (MDT_device_functions.cu), with two
// deliberate differences that only widen what works:
//  * every kernel walks its index space with grid-stride loops, so any grid
//    that covers the reference's implied sizes produces the same result
//    (NE and Nspectra are still taken from gridDim exactly as the reference
//    kernels take them);
//  * ReorderFOutput stages full 32x32 tiles with whatever block shape it is
//    given; the reference loads only blockDim.x channels of each tile
//    (:193,197) and writes 32, which is wrong for its documented NE < 32
//    geometry (:175).
#include <math.h>
#include <mutex>
#include <stdio.h>
#include <unordered_map>

#include "MDT_device_functions.h"
#include "mdt_common.cuh"

namespace mdt {

static thread_local std::string g_last_error;

void set_error(const std::string &msg) { g_last_error = msg; }

mdt_status invalid(const std::string &msg)
{
    set_error(msg);
    return MDT_ERR_INVALID_VALUE;
}

mdt_status cuda_status(cudaError_t err, const char *what)
{
    if (err == cudaSuccess) return MDT_SUCCESS;
    set_error(std::string(what) + ": " + cudaGetErrorName(err) + " (" + cudaGetErrorString(err) +
              ")");
    return MDT_ERR_CUDA;
}

int sm_count()
{
    static std::mutex mu;
    static std::unordered_map<int, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        n = 148;
    cache[dev] = n;
    return n;
}

}  // namespace mdt

// ----------------------------------------------------------------- kernels

// nvcc gives __global__ host stubs hidden visibility by default; the drop-in
// kernels are part of the library's interface, so their stubs are exported.
#define MDT_KERNEL_EXPORT __attribute__((visibility("default")))

// Minimum 4-term Blackman-Harris windowed sinc (reference :52-88), with the
// reference's float argument conventions; sinpif/cospif are CUDA's.
__global__ MDT_KERNEL_EXPORT void PFB_Window_min4term_BH(int Nchannels, int Ntaps, float *Window)
{
    const long total = (long)Ntaps * Nchannels;
    const long step = (long)gridDim.x * blockDim.x;
    for (long idx = threadIdx.x + (long)blockIdx.x * blockDim.x; idx < total; idx += step) {
        float arg = (idx - 0.5f * Ntaps * Nchannels) / Nchannels;
        float sinc = (arg == 0.0f) ? 1.0f : sinpif(arg) / (3.14159265358979323846f * arg);
        float x = 2.0f * idx / (Ntaps * Nchannels);
        float bh = 0.35875f - 0.48829f * cospif(x) + 0.14128f * cospif(2.0f * x) -
                   0.01168f * cospif(3.0f * x);
        Window[idx] = sinc * bh;
    }
}

namespace mdt {

// nspec spectra of one (element, channel).  Sample j feeds spectrum j - i at
// tap i; its sum is in slot (j - i) % NT and complete at tap NT - 1.  Sums of
// spectra before the first or past the last one are formed and not stored.
template <int NT>
__device__ __forceinline__ void pps_run(int nch, int nspec, const float2 *in, const float *w,
                                        float2 *out, long stride_spec)
{
    constexpr int U = 8;  // samples per batch of loads
    float re[NT], im[NT], wr[NT];
#pragma unroll
    for (int i = 0; i < NT; i++) {
        re[i] = im[i] = 0.0f;
        wr[i] = __ldg(w + (long)i * nch);
    }
    const int total = nspec + NT - 1;
    for (int j0 = 0; j0 < total; j0 += U, in += U * stride_spec) {
        float2 x[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            x[u] = j0 + u < total ? __ldg(in + u * stride_spec) : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
            for (int i = NT - 1; i >= 0; i--) {
                const int k = (u - i + 2 * U) % NT;
                re[k] = __fmaf_rn(wr[i], x[u].x, i ? re[k] : 0.0f);
                im[k] = __fmaf_rn(wr[i], x[u].y, i ? im[k] : 0.0f);
                if (i == NT - 1) {
                    const int r = j0 + u - i;
                    if (r >= 0 && r < nspec) out[r * stride_spec] = make_float2(re[k], im[k]);
                }
            }
        }
    }
}

// The launcher's form for 4 and 8 taps: run-long runs of consecutive spectra of
// an element, each sample and window value of a run read once, the sums of the
// NT spectra that a sample feeds in registers; each output is the same fmaf
// chain.  One output per thread reads every sample Ntaps times through L2.
// Bound by HBM (16 bytes a sample): NE=38, Nch=1024, Ntaps=8, Nsp=1024 takes
// 95 us (6.7 TB/s), one output per thread 245 us.  The same runs on the
// caller's grid, where all but every 32nd block end at once, took 194 us: a
// block of 1024 threads takes half a microsecond to come and go.
constexpr int PPS_THREADS = 256;
template <int NT>
__global__ void __launch_bounds__(PPS_THREADS, 4)
    pps_runs_kernel(int nch, int nsp, int run, const float *__restrict__ w,
                    const float2 *__restrict__ in, float2 *__restrict__ out)
{
    const int c = blockIdx.x * PPS_THREADS + threadIdx.x, s0 = blockIdx.y * run;
    if (c >= nch) return;
    const long stride_spec = (long)gridDim.z * nch;
    const long at = s0 * stride_spec + (long)blockIdx.z * nch + c;
    pps_run<NT>(nch, min(run, nsp - s0), in + at, w + c, out + at, stride_spec);
}

}  // namespace mdt

// Polyphase structure (reference :113-161):
//   out[s][e][c] = sum_{i<Ntaps} W[i*Nch + c] * in[s+i][e][c]
// accumulated with fmaf in increasing i from zero (bit-exact with the
// reference).  NE = gridDim.z, spectrum s = blockIdx.y, element e = blockIdx.z.
__global__ MDT_KERNEL_EXPORT void PpS_Batch(int Nchannels, int Ntaps, float *Window, cuComplex *InSignal,
                          cufftComplex *PolyStruct)
{
    const long stride_spec = (long)gridDim.z * Nchannels;
    const long base = (long)blockIdx.y * stride_spec + (long)blockIdx.z * Nchannels;
    const float2 *__restrict__ in = reinterpret_cast<const float2 *>(InSignal) + base;
    const float *__restrict__ w = Window;
    float2 *__restrict__ out = reinterpret_cast<float2 *>(PolyStruct) + base;
    const int step = gridDim.x * blockDim.x;
    for (int c = threadIdx.x + blockIdx.x * blockDim.x; c < Nchannels; c += step) {
        float re = 0.0f, im = 0.0f;
        const float2 *p = in + c;
        const float *wp = w + c;
#pragma unroll 8
        for (int i = 0; i < Ntaps; i++) {
            float2 x = __ldg(p + (long)i * stride_spec);
            float wi = __ldg(wp + (long)i * Nchannels);
            re = __fmaf_rn(wi, x.x, re);
            im = __fmaf_rn(wi, x.y, im);
        }
        out[c] = make_float2(re, im);
    }
}

namespace mdt {

// Tile of the corner turn (see ReorderFOutput below) and threads of the
// launcher's blocks: four per SM, each with a 32 KB tile in flight.
constexpr int RF_T = 64, RF_THREADS = 512;

// NTHR: threads of the block (0: nthr, known at run time only).  VEC 2: two
// channels per 16-byte load (Nch even, F 16-byte aligned).
template <int NTHR, int VEC>
__device__ __forceinline__ void reorder_tile(float2 (*tile)[RF_T + 1], const float2 *__restrict__ F,
                                             float2 *__restrict__ X, long rows, int nch, long r0,
                                             int c0, int tid, int nthr)
{
    const int step = NTHR ? NTHR : nthr;
    const int nr = (int)min((long)RF_T, rows - r0), nc = min(RF_T, nch - c0);
    constexpr int CV = RF_T / VEC;
    const float2 *src = F + r0 * nch + c0;
#pragma unroll
    for (int k = tid; k < RF_T * CV; k += step) {
        const int lr = k / CV, lc = (k % CV) * VEC;
        if (lr < nr && lc < nc) {
            if constexpr (VEC == 2) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(src + (long)lr * nch + lc));
                tile[lr][lc] = make_float2(v.x, v.y);
                tile[lr][lc + 1] = make_float2(v.z, v.w);
            } else {
                tile[lr][lc] = __ldg(src + (long)lr * nch + lc);
            }
        }
    }
    __syncthreads();
    float2 *dst = X + (long)c0 * rows + r0;
#pragma unroll
    for (int k = tid; k < RF_T * RF_T; k += step) {
        const int lc = k / RF_T, lr = k % RF_T;
        if (lr < nr && lc < nc) dst[(long)lc * rows + lr] = tile[lr][lc];
    }
}

__global__ void __launch_bounds__(RF_THREADS, 4)
    reorder_kernel(long rows, int nch, const float2 *__restrict__ F, float2 *__restrict__ X)
{
    __shared__ float2 tile[RF_T][RF_T + 1];
    const long r0 = (long)blockIdx.x * RF_T;
    const int c0 = blockIdx.y * RF_T;
    if (nch % 2 == 0 && ((size_t)F & 15) == 0)
        reorder_tile<RF_THREADS, 2>(tile, F, X, rows, nch, r0, c0, threadIdx.x, RF_THREADS);
    else
        reorder_tile<RF_THREADS, 1>(tile, F, X, rows, nch, r0, c0, threadIdx.x, RF_THREADS);
}

}  // namespace mdt

// Corner turn (reference :183-208):  X[(c*Nsp + s)*NE + e] = F[(s*NE + e)*Nch + c]
// with Nsp = gridDim.z.  With r = s*NE + e this is the plain transpose of
// [Nsp*NE][Nch] into [Nch][Nsp*NE], which the blocks walk in RF_T x RF_T
// tiles through shared memory, whatever the grid and block shape.  Bound by
// HBM: flat rows leave no part of a tile empty when NE is not a multiple of
// the tile, and 64 x 64 tiles keep 32 KB a block in flight.  The reference's
// grid has a block per 32 x 32 (element, channel) tile of a spectrum, most of
// which find no tile left; starting and ending them then takes half of the
// kernel's time, so the launcher below starts its own grid.  NE=38, Nch=1024,
// Nsp=1024: 94.5 us by the launcher (6.8 TB/s), 222 us on the reference's grid
// and 354 us there with a 32 x 32 tile of one spectrum per block.
__global__ MDT_KERNEL_EXPORT void __launch_bounds__(1024, 2)
    ReorderFOutput(int NpolsxNelements, int Nchannels, cufftComplex *FOutput, cuComplex *XInput)
{
    using mdt::RF_T;
    __shared__ float2 tile[RF_T][RF_T + 1];
    // few instructions before a block without a tile ends: most blocks have none
    const unsigned long long rows = (unsigned long long)gridDim.z * (unsigned)NpolsxNelements;
    const unsigned nct = ((unsigned)Nchannels + RF_T - 1) / RF_T;
    const unsigned long long ntiles = (rows + RF_T - 1) / RF_T * nct;
    const unsigned long long nxy = (unsigned long long)gridDim.x * gridDim.y;
    unsigned long long t = nxy * blockIdx.z + (unsigned long long)gridDim.x * blockIdx.y + blockIdx.x;
    if (t >= ntiles) return;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    const float2 *F = reinterpret_cast<const float2 *>(FOutput);
    float2 *X = reinterpret_cast<float2 *>(XInput);
    const bool v2 = Nchannels % 2 == 0 && ((size_t)F & 15) == 0;
    for (; t < ntiles; t += nxy * gridDim.z) {
        // 32-bit division wherever the tile index fits
        const long rt = t >> 32 ? (long)(t / nct) : (long)((unsigned)t / nct);
        const long r0 = rt * RF_T;
        const int c0 = (int)((long)t - rt * nct) * RF_T;
        if (nthr == 1024 && v2)
            mdt::reorder_tile<1024, 2>(tile, F, X, (long)rows, Nchannels, r0, c0, tid, nthr);
        else
            mdt::reorder_tile<0, 1>(tile, F, X, (long)rows, Nchannels, r0, c0, tid, nthr);
        __syncthreads();
    }
}

// Hamming windowed sinc (no reference counterpart; see mdt_fx.h):
// evaluated in double per coefficient and rounded once to float.
__global__ void mdt_window_hamming_sinc_kernel(int nch, int ntaps, float *w)
{
    const long L = (long)ntaps * nch;
    for (long n = threadIdx.x + (long)blockIdx.x * blockDim.x; n < L;
         n += (long)gridDim.x * blockDim.x) {
        double t = ((double)n - 0.5 * (double)L) / (double)nch;
        double sinc = (t == 0.0) ? 1.0 : sinpi(t) / (3.141592653589793238462643383279502884 * t);
        double hw = 0.54 - 0.46 * cospi(2.0 * (double)n / (double)L);
        w[n] = (float)(sinc * hw);
    }
}

// ------------------------------------------------------------------- C ABI

// Whether <<<(gx, gy, gz), (bx, by, bz)>>> is a valid launch.
static bool launchable(unsigned gx, unsigned gy, unsigned gz, unsigned bx, unsigned by, unsigned bz)
{
    return gx >= 1 && gx <= 0x7fffffffu && gy >= 1 && gy <= 65535 && gz >= 1 && gz <= 65535 &&
           bx >= 1 && bx <= 1024 && by >= 1 && by <= 1024 && bz >= 1 && bz <= 64 &&
           (unsigned long long)bx * by * bz <= 1024;
}

extern "C" {

MDT_API int mdt_version(void) { return 1000; }

MDT_API const char *mdt_last_error(void) { return mdt::g_last_error.c_str(); }

MDT_API mdt_status mdt_launch_PFB_Window_min4term_BH(unsigned gx, unsigned gy, unsigned gz,
                                                     unsigned bx, unsigned by, unsigned bz,
                                                     cudaStream_t stream, int nchannels,
                                                     int ntaps, float *window)
{
    if (!window || nchannels <= 0 || ntaps <= 0) return mdt::invalid("window: bad arguments");
    PFB_Window_min4term_BH<<<dim3(gx, gy, gz), dim3(bx, by, bz), 0, stream>>>(nchannels, ntaps,
                                                                           window);
    return mdt::launch_status("PFB_Window_min4term_BH");
}

MDT_API mdt_status mdt_launch_PpS_Batch(unsigned gx, unsigned gy, unsigned gz, unsigned bx,
                                        unsigned by, unsigned bz, cudaStream_t stream,
                                        int nchannels, int ntaps, float *window, void *insignal,
                                        void *polystruct)
{
    if (!window || !insignal || !polystruct || nchannels <= 0 || ntaps <= 0)
        return mdt::invalid("PpS_Batch: bad arguments");
    // runs of 32 to 8 spectra, as long as leaves eight blocks per SM; fewer
    // outputs, other tap counts and grids that cannot be launched take the
    // drop-in kernel on the caller's grid
    for (unsigned run = 32; launchable(gx, gy, gz, bx, by, bz) && (ntaps == 4 || ntaps == 8) && run >= 8;
         run /= 2) {
        const dim3 grid((unsigned)mdt::cdiv(nchannels, mdt::PPS_THREADS), (unsigned)mdt::cdiv(gy, run), gz);
        if ((long)grid.x * grid.y * grid.z < 8L * mdt::sm_count()) continue;
        auto kern = ntaps == 4 ? mdt::pps_runs_kernel<4> : mdt::pps_runs_kernel<8>;
        kern<<<grid, mdt::PPS_THREADS, 0, stream>>>(nchannels, (int)gy, (int)run, window,
                                               (const float2 *)insignal, (float2 *)polystruct);
        return mdt::launch_status("pps_runs_kernel");
    }
    PpS_Batch<<<dim3(gx, gy, gz), dim3(bx, by, bz), 0, stream>>>(
        nchannels, ntaps, window, (cuComplex *)insignal, (cufftComplex *)polystruct);
    return mdt::launch_status("PpS_Batch");
}

MDT_API mdt_status mdt_launch_ReorderFOutput(unsigned gx, unsigned gy, unsigned gz, unsigned bx,
                                             unsigned by, unsigned bz, cudaStream_t stream,
                                             int npolsxnelements, int nchannels, void *foutput,
                                             void *xinput)
{
    if (!foutput || !xinput || npolsxnelements <= 0 || nchannels <= 0)
        return mdt::invalid("ReorderFOutput: bad arguments");
    const long rows = (long)gz * npolsxnelements;
    const dim3 grid((unsigned)mdt::cdiv(rows, mdt::RF_T), (unsigned)mdt::cdiv(nchannels, mdt::RF_T));
    if (launchable(gx, gy, gz, bx, by, bz) && grid.y <= 65535 && mdt::cdiv(rows, mdt::RF_T) <= 0x7fffffffL) {
        mdt::reorder_kernel<<<grid, mdt::RF_THREADS, 0, stream>>>(rows, nchannels, (const float2 *)foutput,
                                                        (float2 *)xinput);
        return mdt::launch_status("reorder_kernel");
    }
    ReorderFOutput<<<dim3(gx, gy, gz), dim3(bx, by, bz), 0, stream>>>(
        npolsxnelements, nchannels, (cufftComplex *)foutput, (cuComplex *)xinput);
    return mdt::launch_status("ReorderFOutput");
}

MDT_API mdt_status mdt_window_hamming_sinc(int nchannels, int ntaps, float *window,
                                           cudaStream_t stream)
{
    if (!window || nchannels <= 0 || ntaps <= 0) return mdt::invalid("window: bad arguments");
    long L = (long)nchannels * ntaps;
    int blocks = (int)mdt::cdiv(L, 256);
    mdt_window_hamming_sinc_kernel<<<blocks, 256, 0, stream>>>(nchannels, ntaps, window);
    return mdt::launch_status("window_hamming_sinc");
}

}  // extern "C"
