// fft.cu -- batched C2C FFT on the shared-memory Stockham core
// (fft_core.cuh) and the cuFFT subset the reference client calls
// (cufftPlan1d / cufftSetStream / cufftExecC2C / cufftDestroy /
// cufftGetVersion, reference MDT_OneStation_client.cu:441-446,622-630,1105).
#include <cufft.h>
#include "mdt_cufft_cublas_shim.h"  // checks the exported signatures

#include <map>
#include <mutex>
#include <vector>

#include "fft_core.cuh"

namespace mdt {

// ------------------------------------------------------------ twiddles
const float2 *fft_twiddles(int n, mdt_status *st)
{
    static std::mutex mu;
    static std::map<std::pair<int, int>, float2 *> tables;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto key = std::make_pair(dev, n);
    auto it = tables.find(key);
    if (it != tables.end()) {
        *st = MDT_SUCCESS;
        return it->second;
    }
    std::vector<float2> h(n);
    for (int k = 0; k < n; k++) {
        double a = -2.0 * 3.141592653589793238462643383279502884 * (double)k / (double)n;
        h[k] = make_float2((float)cos(a), (float)sin(a));
    }
    float2 *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(float2) * n);
    if (e != cudaSuccess) {
        *st = cuda_status(e, "twiddle table alloc");
        return nullptr;
    }
    e = cudaMemcpy(d, h.data(), sizeof(float2) * n, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        *st = cuda_status(e, "twiddle table copy");
        return nullptr;
    }
    tables[key] = d;
    *st = MDT_SUCCESS;
    return d;
}

// ------------------------------------------------------------ kernel
template <int N>
struct RowsCfg {
    static constexpr int TPR = fft::Shape<N>::TPR;
    static constexpr int ROWS = (256 / TPR) < 1 ? 1 : 256 / TPR;
    static constexpr int THREADS = ROWS * TPR;
    static constexpr size_t SMEM = sizeof(float2) * fft::Shape<N>::PADN * ROWS;
};

template <int N>
__global__ void __launch_bounds__(RowsCfg<N>::THREADS)
    fft_rows_kernel(const float2 *in, float2 *out, long rows, const float2 *__restrict__ tw,
                    int inverse)
{
    using C = RowsCfg<N>;
    extern __shared__ float2 smem2[];
    const int lrow = threadIdx.x / C::TPR;
    const int t = threadIdx.x - lrow * C::TPR;
    const long row = (long)blockIdx.x * C::ROWS + lrow;
    const bool valid = row < rows;
    float2 *sx = smem2 + (size_t)lrow * fft::Shape<N>::PADN;
    const float2 *src = in + (valid ? row : 0) * (long)N;
    float2 *dst = out + (valid ? row : 0) * (long)N;
    auto load = [&](int i) -> float2 {
        float2 v = valid ? src[i] : make_float2(0.f, 0.f);
        return inverse ? cconj(v) : v;
    };
    auto store = [&](int i, float2 v) {
        if (valid) dst[i] = inverse ? cconj(v) : v;
    };
    fft::transform_row<N, C::TPR, true, true>(sx, t, tw, load, store);
}

template <int N>
static mdt_status launch_rows(const float2 *in, float2 *out, long rows, int inverse,
                              cudaStream_t stream)
{
    using C = RowsCfg<N>;
    mdt_status st;
    const float2 *tw = fft_twiddles(N, &st);
    if (!tw) return st;
    if (C::SMEM > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fft_rows_kernel<N>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)C::SMEM);
        if (e != cudaSuccess) return cuda_status(e, "fft smem attribute");
    }
    long blocks = cdiv(rows, C::ROWS);
    if (blocks > 0x7fffffffL) return invalid("fft: too many rows");
    fft_rows_kernel<N><<<(unsigned)blocks, C::THREADS, C::SMEM, stream>>>(in, out, rows, tw,
                                                                        inverse);
    return launch_status("fft_rows_kernel");
}

mdt_status fft_c2c(const void *in, void *out, long rows, int n, int direction,
                   cudaStream_t stream)
{
    if (!in || !out || rows < 0) return invalid("fft: bad pointers or rows");
    if (direction != -1 && direction != 1) return invalid("fft: direction must be -1 or +1");
    if (rows == 0) return MDT_SUCCESS;
    const float2 *i2 = (const float2 *)in;
    float2 *o2 = (float2 *)out;
    int inv = direction == 1;
    switch (n) {
        case 2: return launch_rows<2>(i2, o2, rows, inv, stream);
        case 4: return launch_rows<4>(i2, o2, rows, inv, stream);
        case 8: return launch_rows<8>(i2, o2, rows, inv, stream);
        case 16: return launch_rows<16>(i2, o2, rows, inv, stream);
        case 32: return launch_rows<32>(i2, o2, rows, inv, stream);
        case 64: return launch_rows<64>(i2, o2, rows, inv, stream);
        case 128: return launch_rows<128>(i2, o2, rows, inv, stream);
        case 256: return launch_rows<256>(i2, o2, rows, inv, stream);
        case 512: return launch_rows<512>(i2, o2, rows, inv, stream);
        case 1024: return launch_rows<1024>(i2, o2, rows, inv, stream);
        case 2048: return launch_rows<2048>(i2, o2, rows, inv, stream);
        case 4096: return launch_rows<4096>(i2, o2, rows, inv, stream);
        case 8192: return launch_rows<8192>(i2, o2, rows, inv, stream);
        case 16384: return launch_rows<16384>(i2, o2, rows, inv, stream);
        default: break;
    }
    set_error("fft: n must be a power of two in [2, 16384]");
    return MDT_ERR_NOT_SUPPORTED;
}

// ------------------------------------------------------------ reorder adjoint and inverse
// dP[row][k] = inverse FFT over c of conj(g[c][row % NE]) dY[c][row], rows = Nsp * NE: the
// adjoint of gains, corner turn and FFT in one pass.  A block takes up to 8 rows: it reads 64
// contiguous bytes of each channel into the rows' shared memory and stores the last FFT pass
// straight to dP.  Bound by HBM (16 bytes a value) and by the latency of its loads: NE=64,
// Nch=512, Nsp=2048 240 us; mdt_gain_adjoint's dF (212) and then mdt_fft_c2c (169) write and
// read the values once more.  Nch 2048, Nsp=512 381 us and 408; from 4096 channels on a block
// has too few rows for whole sectors (467 and 457) and the two calls stay.
template <int N>
struct TurnCfg {
    static constexpr int TPR = N < 256 ? N / 8 : N / 16;
    static constexpr int ROWS = 1024 / TPR < 8 ? 1024 / TPR : 8;
    static constexpr int THREADS = ROWS * TPR;
    static constexpr int RSTRIDE = fft::Shape<N>::PADN + 2;  // rows in different banks
    static constexpr size_t SMEM = sizeof(float2) * (size_t)RSTRIDE * ROWS;
};

template <int N>
__global__ void __launch_bounds__(TurnCfg<N>::THREADS, 1024 / TurnCfg<N>::THREADS)
    reorder_adjoint_ifft_kernel(int ne, long rows, const float2 *__restrict__ dY,
                                const float2 *__restrict__ g, float2 *__restrict__ dP,
                                const float2 *__restrict__ tw)
{
    using C = TurnCfg<N>;
    extern __shared__ float2 smem2[];
    const long row0 = (long)blockIdx.x * C::ROWS;
    {
        const int r = threadIdx.x % C::ROWS;  // a thread's values are all of one row
        const bool valid = row0 + r < rows;
        const long row = valid ? row0 + r : 0;
        const float2 *src = dY + row, *gr = g + row % ne;
#pragma unroll 8
        for (int c = threadIdx.x / C::ROWS; c < N; c += C::TPR) {
            const float2 v = cmul(cconj(__ldg(gr + (long)c * ne)), __ldg(src + (long)c * rows));
            smem2[r * C::RSTRIDE + fft::pad(c)] = valid ? cconj(v) : make_float2(0.f, 0.f);
        }
    }
    __syncthreads();
    const int lrow = threadIdx.x / C::TPR, t = threadIdx.x - lrow * C::TPR;
    const bool valid = row0 + lrow < rows;
    float2 *dst = dP + (valid ? row0 + lrow : 0) * N;
    auto none_load = [](int) { return make_float2(0.f, 0.f); };
    auto store = [&](int i, float2 v) {
        if (valid) dst[i] = cconj(v);
    };
    fft::transform_row<N, C::TPR, false, true>(smem2 + (size_t)lrow * C::RSTRIDE, t, tw, none_load, store);
}

template <int N>
static mdt_status launch_turn(int ne, long rows, const float2 *dY, const float2 *g, float2 *dP,
                              cudaStream_t stream)
{
    using C = TurnCfg<N>;
    mdt_status st;
    const float2 *tw = fft_twiddles(N, &st);
    if (!tw) return st;
    cudaError_t e = cudaFuncSetAttribute(reorder_adjoint_ifft_kernel<N>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return cuda_status(e, "reorder_adjoint_ifft smem attribute");
    const long blocks = cdiv(rows, C::ROWS);
    if (blocks > 0x7fffffffL) return invalid("reorder_adjoint_ifft: too many rows");
    reorder_adjoint_ifft_kernel<N><<<(unsigned)blocks, C::THREADS, C::SMEM, stream>>>(ne, rows, dY, g,
                                                                                     dP, tw);
    return launch_status("reorder_adjoint_ifft_kernel");
}

// ------------------------------------------------------------ cuFFT subset
struct ShimPlan {
    int n = 0;
    long batch = 0;
    cudaStream_t stream = 0;
};
static std::mutex g_plan_mu;
static std::map<int, ShimPlan> g_plans;
static int g_next_plan = 1;

}  // namespace mdt

extern "C" {

MDT_API mdt_status mdt_fft_c2c(const void *in, void *out, long rows, int n, int direction,
                               cudaStream_t stream)
{
    return mdt::fft_c2c(in, out, rows, n, direction, stream);
}

MDT_API mdt_status mdt_reorder_adjoint_ifft(int ne, int nch, int nsp, const void *dY,
                                            const void *gains, void *dP, cudaStream_t stream)
{
    if (!dY || !gains || !dP || dY == dP || ne < 1 || nsp < 1)
        return mdt::invalid("reorder_adjoint_ifft: bad arguments");
    const long rows = (long)nsp * ne;
    const float2 *y = (const float2 *)dY, *g = (const float2 *)gains;
    float2 *p = (float2 *)dP;
    switch (nch) {
        case 32: return mdt::launch_turn<32>(ne, rows, y, g, p, stream);
        case 64: return mdt::launch_turn<64>(ne, rows, y, g, p, stream);
        case 128: return mdt::launch_turn<128>(ne, rows, y, g, p, stream);
        case 256: return mdt::launch_turn<256>(ne, rows, y, g, p, stream);
        case 512: return mdt::launch_turn<512>(ne, rows, y, g, p, stream);
        case 1024: return mdt::launch_turn<1024>(ne, rows, y, g, p, stream);
        case 2048: return mdt::launch_turn<2048>(ne, rows, y, g, p, stream);
        default: break;
    }
    return mdt::invalid("reorder_adjoint_ifft: Nch must be a power of two in [32, 2048]");
}

// cufftPlan1d(&plan, Nch, CUFFT_C2C, Nspectra*Npols*Nelements)
// (reference MDT_OneStation_client.cu:622).  Supported: C2C, nx = 2^k in
// [2, 16384], batch >= 1.  The plan allocates nothing per batch; the
// twiddle table for nx is created here, outside any stream capture.
cufftResult CUFFTAPI cufftPlan1d(cufftHandle *plan, int nx, cufftType type, int batch)
{
    if (!plan) return CUFFT_INVALID_VALUE;
    if (type != CUFFT_C2C) return CUFFT_NOT_SUPPORTED;
    if (batch < 1) return CUFFT_INVALID_VALUE;
    if (!mdt::is_pow2(nx) || nx < 2 || nx > 16384) return CUFFT_INVALID_SIZE;
    mdt_status st;
    if (!mdt::fft_twiddles(nx, &st)) return CUFFT_ALLOC_FAILED;
    std::lock_guard<std::mutex> lk(mdt::g_plan_mu);
    int h = mdt::g_next_plan++;
    mdt::ShimPlan p;
    p.n = nx;
    p.batch = batch;
    mdt::g_plans[h] = p;
    *plan = h;
    return CUFFT_SUCCESS;
}

// cufftSetStream (reference :630)
cufftResult CUFFTAPI cufftSetStream(cufftHandle plan, cudaStream_t stream)
{
    std::lock_guard<std::mutex> lk(mdt::g_plan_mu);
    auto it = mdt::g_plans.find(plan);
    if (it == mdt::g_plans.end()) return CUFFT_INVALID_PLAN;
    it->second.stream = stream;
    return CUFFT_SUCCESS;
}

// cufftExecC2C(plan, d_FOutput, d_FOutput, CUFFT_FORWARD) (reference :1105);
// in place or out of place, forward or inverse, unnormalised.
cufftResult CUFFTAPI cufftExecC2C(cufftHandle plan, cufftComplex *idata, cufftComplex *odata,
                                  int direction)
{
    mdt::ShimPlan p;
    {
        std::lock_guard<std::mutex> lk(mdt::g_plan_mu);
        auto it = mdt::g_plans.find(plan);
        if (it == mdt::g_plans.end()) return CUFFT_INVALID_PLAN;
        p = it->second;
    }
    if (!idata || !odata) return CUFFT_INVALID_VALUE;
    if (direction != CUFFT_FORWARD && direction != CUFFT_INVERSE) return CUFFT_INVALID_VALUE;
    mdt_status st = mdt::fft_c2c(idata, odata, p.batch, p.n, direction, p.stream);
    if (st == MDT_SUCCESS) return CUFFT_SUCCESS;
    if (st == MDT_ERR_NOT_SUPPORTED) return CUFFT_NOT_SUPPORTED;
    if (st == MDT_ERR_INVALID_VALUE) return CUFFT_INVALID_VALUE;
    return CUFFT_EXEC_FAILED;
}

cufftResult CUFFTAPI cufftDestroy(cufftHandle plan)
{
    std::lock_guard<std::mutex> lk(mdt::g_plan_mu);
    auto it = mdt::g_plans.find(plan);
    if (it == mdt::g_plans.end()) return CUFFT_INVALID_PLAN;
    mdt::g_plans.erase(it);
    return CUFFT_SUCCESS;
}

// Reports this library's version code (mdt_version), not a cuFFT release:
// the reference only prints it (MDT_OneStation_client.cu:443,446).
cufftResult CUFFTAPI cufftGetVersion(int *version)
{
    if (!version) return CUFFT_INVALID_VALUE;
    *version = mdt_version();
    return CUFFT_SUCCESS;
}

}  // extern "C"
