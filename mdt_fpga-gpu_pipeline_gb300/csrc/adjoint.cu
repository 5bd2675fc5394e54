// adjoint.cu -- hand-written adjoint kernels of the FX path, for gradients
// through the correlator (gain calibration, PFB tap optimisation).
//
// Gradients follow the convention of PyTorch for complex tensors: for a real
// loss L and complex z, grad(z) = dL/dRe(z) + i dL/dIm(z) = 2 dL/dconj(z).
//
// * X-engine: V_c = Y_c Y_c^H / Nsp (Y_c = NE x Nsp, stored Y[c][s][e]).
//   grad(Y_c) = (G_c + G_c^H) Y_c / Nsp with G = grad(V) in the visibility
//   layout (column-major per channel: G[c][q*NE + r] = G_rq).
// * F-engine: X = DFT(P), P[s][e][k] = sum_i W[i][k] in[s+i][e][k] with real
//   taps W.  grad(P) = DFT^H grad(X) (the unnormalised inverse FFT, done with
//   mdt_fft_c2c direction +1) and
//   grad(W)[i][k] = sum_{s,e} Re(grad(P)[s][e][k] * conj(in[s+i][e][k])).
#include <algorithm>
#include <type_traits>

#include "mdt_common.cuh"

namespace mdt {

// Compensated dot products: hi + lo accumulates sum a*b with every rounding
// error of the products and of the sum carried along in lo (Dot2 of Ogita,
// Rump and Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26,
// 2005), which is as accurate as a sum in twice the working precision (2^-48).
// The GPU's FP64 rate is a hundredth of its FP32 rate: sums kept in double
// held the two gradient kernels below on the FP64 pipe.  Infinities and NaN
// leave NaN in lo, and the error of a product below 2^-102 is no longer an FP32
// number (that of a sum of 2^-80 and above does not miss it).  settled() is false
// in both cases, and the kernels repeat the thread's sums in double, unless SumAny
// finds that every product is zero.
struct Sum2 {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float a, float b)
    {
        const float p = __fmul_rn(a, b);
        const float e = __fmaf_rn(a, b, -p);
        const float s = __fadd_rn(hi, p);
        const float v = __fsub_rn(s, hi);
        const float d = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, v)), __fsub_rn(p, v));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(e, d));
    }
    __device__ __forceinline__ bool settled() const
    {
        const float v = fabsf(hi + lo);
        return v >= 0x1p-80f && v < __int_as_float(0x7f800000);
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
struct SumAny {
    bool any = false;
    __device__ __forceinline__ void add(float a, float b)
    {
        any = any || (a != 0.0f && b != 0.0f) || !isfinite(a) || !isfinite(b);
    }
    __device__ __forceinline__ bool settled() const { return !any; }
    __device__ __forceinline__ double value() const { return 0.0; }
};
struct SumD {
    double v = 0.0;
    __device__ __forceinline__ void add(float a, float b) { v += (double)a * (double)b; }
    __device__ __forceinline__ bool settled() const { return true; }
    __device__ __forceinline__ double value() const { return v; }
};

// VEC consecutive complex64 values (VEC 2: 16-byte aligned).
template <int VEC>
__device__ __forceinline__ void load_c64(const float2 *p, float2 (&v)[VEC])
{
    if constexpr (VEC == 2) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = make_float2(t.x, t.y);
        v[1] = make_float2(t.z, t.w);
    } else {
        v[0] = __ldg(p);
    }
}

// Y[c][s][e] = g[c][e] * X[c][s][e] (complex gains on the F-engine output).
// Bound by HBM (16 bytes a value).  A block covers AG_ITEMS vectors of VEC
// elements per thread, a block's width apart, so that the element index is
// one division per thread and then steps without one, and every access is 16
// bytes wide (VEC 2: NE even and 16-byte buffers; otherwise one value).
// NE=64, Nch=512, Nsp=2048: 157 us (6.8 TB/s); one value and two 64-bit
// divisions per thread took 277 us.
constexpr int AG_THREADS = 256, AG_ITEMS = 4;
template <int VEC>
__global__ void __launch_bounds__(AG_THREADS)
    apply_gains_kernel(int nch, int ne, long per, int step, const float2 *__restrict__ X,
                       const float2 *__restrict__ g, float2 *__restrict__ Y)
{
    // per = Nsp * NE / VEC vectors of a channel; step = AG_THREADS * VEC mod NE
    const long i0 = (long)blockIdx.x * (AG_THREADS * AG_ITEMS) + threadIdx.x;
    if (i0 >= per) return;
    const int e0 = (int)((i0 * VEC) % ne);
    for (int c = blockIdx.y; c < nch; c += gridDim.y) {
        const float2 *xc = X + (long)c * per * VEC, *gc = g + (long)c * ne;
        float2 *yc = Y + (long)c * per * VEC;
        int e = e0;
#pragma unroll
        for (int k = 0; k < AG_ITEMS; k++) {
            const long i = i0 + k * AG_THREADS;
            if (i < per) {
                float2 x[VEC], gv[VEC];
                load_c64<VEC>(xc + i * VEC, x);
                load_c64<VEC>(gc + e, gv);
                if constexpr (VEC == 2) {
                    const float2 a = cmul(gv[0], x[0]), b = cmul(gv[1], x[1]);
                    *reinterpret_cast<float4 *>(yc + i * 2) = make_float4(a.x, a.y, b.x, b.y);
                } else {
                    yc[i] = cmul(gv[0], x[0]);
                }
            }
            e += step;
            if (e >= ne) e -= ne;
        }
    }
}

// dg[c][e] = sum_s dY[c][s][e] * conj(X[c][s][e]).  32 vectors of VEC (c, e)
// pairs per block, GG_PH spectrum phases per pair (compensated FP32 sums),
// combined in double in a fixed order.  Bound by HBM (16 bytes a value); four
// blocks of eight warps per SM keep enough 16-byte loads in flight (two blocks
// of sixteen: 320 us).  NE=64, Nch=512, Nsp=2048: 172 us (6.2 TB/s); sums in
// double took 1284 us.
constexpr int GG_PH = 8;
template <int VEC, class Sum>
__device__ __forceinline__ bool gain_sums(int ne, int nsp, int ph, const float2 *dY,
                                          const float2 *X, double (&re)[VEC], double (&im)[VEC])
{
    Sum ar[VEC], ai[VEC];
#pragma unroll 4
    for (int s = ph; s < nsp; s += GG_PH) {
        float2 a[VEC], b[VEC];
        load_c64<VEC>(dY + (long)s * ne, a);
        load_c64<VEC>(X + (long)s * ne, b);
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            ar[v].add(a[v].x, b[v].x);
            ar[v].add(a[v].y, b[v].y);
            ai[v].add(a[v].y, b[v].x);
            ai[v].add(-a[v].x, b[v].y);
        }
    }
    bool ok = true;
#pragma unroll
    for (int v = 0; v < VEC; v++) {
        ok = ok && ar[v].settled() && ai[v].settled();
        re[v] = ar[v].value();
        im[v] = ai[v].value();
    }
    return ok;
}

template <int VEC>
__global__ void __launch_bounds__(32 * GG_PH, 4)
    gain_grad_kernel(int ne, int nch, int nsp, const float2 *__restrict__ dY,
                     const float2 *__restrict__ X, float2 *__restrict__ dg)
{
    __shared__ double sre[GG_PH][32 * VEC + 1], sim[GG_PH][32 * VEC + 1];
    const int ev = ne / VEC;
    const long j = (long)blockIdx.x * 32 + threadIdx.x;
    const int ph = threadIdx.y;
    const bool in = j < (long)nch * ev;
    double re[VEC] = {}, im[VEC] = {};
    if (in) {
        const long c = j / ev, e = (j - c * ev) * VEC;
        const long base = c * nsp * (long)ne + e;
        if (!gain_sums<VEC, Sum2>(ne, nsp, ph, dY + base, X + base, re, im) &&
            !gain_sums<VEC, SumAny>(ne, nsp, ph, dY + base, X + base, re, im))
            gain_sums<VEC, SumD>(ne, nsp, ph, dY + base, X + base, re, im);
    }
#pragma unroll
    for (int v = 0; v < VEC; v++) {
        sre[ph][threadIdx.x * VEC + v] = re[v];
        sim[ph][threadIdx.x * VEC + v] = im[v];
    }
    __syncthreads();
    if (ph == 0 && in) {
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            for (int p = 1; p < GG_PH; p++) {
                re[v] += sre[p][threadIdx.x * VEC + v];
                im[v] += sim[p][threadIdx.x * VEC + v];
            }
            dg[j * VEC + v] = make_float2((float)re[v], (float)im[v]);
        }
    }
}

// Adjoint of the gains and of the channel-major reorder:
// dF[s][e][c] = conj(g[c][e]) * dY[c][s][e] -- a FA_T x FA_T tiled transpose
// of (channel) x (spectrum, element) rows.  Bound by HBM (16 bytes a value):
// eight independent loads per thread, the element index formed once per
// thread and row half.  NE=64, Nch=512, Nsp=2048: 210 us (5.1 TB/s), with
// 32 x 32 tiles and a 64-bit division per value 233 us.
template <int FA_T>
__global__ void __launch_bounds__(8 * FA_T)
    fout_adjoint_kernel(int ne, int nch, long rows, const float2 *__restrict__ dY,
                        const float2 *__restrict__ g, float2 *__restrict__ dF)
{
    __shared__ float2 t[FA_T][FA_T + 1];
    const long r0 = (long)blockIdx.x * FA_T;
    const int c0 = blockIdx.y * FA_T, lane = threadIdx.x, warp = threadIdx.y;
#pragma unroll
    for (int h = 0; h < FA_T / 32; h++) {
        const long r = r0 + 32 * h + lane;
        const int e = (int)(r % ne);
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const int c = c0 + warp + FA_T / 4 * y;
            if (c < nch && r < rows) {
                const float2 gv = g ? __ldg(g + (long)c * ne + e) : make_float2(1.f, 0.f);
                t[warp + FA_T / 4 * y][32 * h + lane] = cmul(cconj(gv), __ldg(dY + (long)c * rows + r));
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int y = 0; y < 4; y++) {
        const long r = r0 + warp + FA_T / 4 * y;
        if (r >= rows) continue;
#pragma unroll
        for (int h = 0; h < FA_T / 32; h++) {
            const int c = c0 + 32 * h + lane;
            if (c < nch) dF[r * nch + c] = t[32 * h + lane][warp + FA_T / 4 * y];
        }
    }
}

// dY[c][s][r] = scale * sum_q (G_rq + conj(G_qr)) Y[c][s][q].  A block takes R
// elements r of one channel and `tiles` tiles of S spectra; a thread holds SP spectra x
// 4 elements, summed over q in increasing order with the multiply-adds of a complex
// product in turn, two lanes of an f32x2 fma each.  Chunks of R elements q of
// H = G + G^H and of Y go through shared memory (H stays there over the block's
// spectra when one chunk holds all of it).  With 8 spectra a thread it is bound by the
// FP32 pipe: per pair of q a warp issues 128 packed fmas against 16 shared-memory
// wavefronts (one output per thread and 16 x 16 tiles: two 8-byte loads per four fmas).
// NE=64, Nch=512, Nsp=2048: 0.95 ms (36 TFLOP/s, 47 % of the FP32 rate), 2.44 before.
constexpr int XA_THREADS = 128;
template <int R, int SP>
struct XaCfg {
    static constexpr int TX = R / 4, TY = XA_THREADS / TX;  // threads over elements, spectra
    static constexpr int S = SP * TY;
    static constexpr int YS = R + 2;  // float2 per staged row of Y (16-byte rows, skewed banks)
    static constexpr size_t SMEM = sizeof(float2) * ((size_t)R * R + (size_t)S * YS);
};

template <int R, int SP>
__global__ void __launch_bounds__(XA_THREADS, 4)
    xengine_adjoint_kernel(int ne, int nsp, int tiles, const float2 *__restrict__ G,
                           const float2 *__restrict__ Y, float2 *__restrict__ dY, float scale)
{
    using C = XaCfg<R, SP>;
    extern __shared__ float4 xa_smem[];
    float2 *sh = reinterpret_cast<float2 *>(xa_smem);  // [q][r]
    float2 *sy = sh + R * R;                           // [s][q], YS per row
    const int c = blockIdx.z, r0 = blockIdx.x * R, tid = threadIdx.x;
    const float2 *Gc = G + (long)c * ne * ne;
    const float2 *Yc = Y + (long)c * nsp * ne;
    float2 *dYc = dY + (long)c * nsp * ne;
    // elements 2 tr + {0, 1, R/2, R/2 + 1}, spectra ts + TY i
    const int tr = tid % C::TX, ts = tid / C::TX;
    const int nchunk = (ne + R - 1) / R;
    // H[q0 + q][r0 + r] = G_rq + conj(G_qr), zero past NE
    auto load_h = [&](int q0) {
        for (int i = tid; i < R * R; i += XA_THREADS) {
            const int q = i / R, r = i % R;
            float2 h = make_float2(0.f, 0.f);
            if (r0 + r < ne && q0 + q < ne) h = __ldg(Gc + (long)(q0 + q) * ne + r0 + r);  // G_rq
            sh[i] = h;
        }
        __syncthreads();
        for (int i = tid; i < R * R; i += XA_THREADS) {
            const int r = i / R, q = i % R;
            if (r0 + r < ne && q0 + q < ne) {
                const float2 b = __ldg(Gc + (long)(r0 + r) * ne + q0 + q);  // G_qr
                float2 &h = sh[q * R + r];
                h = make_float2(h.x + b.x, h.y - b.y);
            }
        }
    };
    auto load_y = [&](int s0, int q0) {
#pragma unroll 8
        for (int i = tid; i < C::S * R; i += XA_THREADS) {
            const int s = i / R, q = i % R;
            sy[s * C::YS + q] = s0 + s < nsp && q0 + q < ne
                                    ? __ldg(Yc + (long)(s0 + s) * ne + q0 + q)
                                    : make_float2(0.f, 0.f);
        }
    };
    if (nchunk == 1) load_h(0);
    for (int t = 0; t < tiles; t++) {
        const int s0 = (blockIdx.y * tiles + t) * C::S;
        if (s0 >= nsp) break;
        float2 acc[SP][4];
#pragma unroll
        for (int i = 0; i < SP; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.f, 0.f);
        for (int k = 0; k < nchunk; k++) {
            __syncthreads();  // the staged chunks have been read
            if (nchunk > 1) load_h(k * R);
            load_y(s0, k * R);
            __syncthreads();
            const int nq = min(R, (ne - k * R + 1) & ~1);
#pragma unroll 2
            for (int q = 0; q < nq; q += 2) {
                float4 h[2][2];
#pragma unroll
                for (int u = 0; u < 2; u++)
#pragma unroll
                    for (int v = 0; v < 2; v++)
                        h[u][v] = *reinterpret_cast<const float4 *>(sh + (q + u) * R + R / 2 * v + 2 * tr);
#pragma unroll
                for (int i = 0; i < SP; i++) {
                    const float4 y4 = *reinterpret_cast<const float4 *>(sy + (ts + C::TY * i) * C::YS + q);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const float2 y = u ? make_float2(y4.z, y4.w) : make_float2(y4.x, y4.y);
                        const float2 yx = make_float2(y.y, y.x);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float4 hh = h[u][j >> 1];
                            const float2 g = j & 1 ? make_float2(hh.z, hh.w) : make_float2(hh.x, hh.y);
                            // (h.x y.x, h.x y.y), then (-h.y y.y, h.y y.x)
                            acc[i][j] = __ffma2_rn(make_float2(g.x, g.x), y, acc[i][j]);
                            acc[i][j] = __ffma2_rn(make_float2(-g.y, g.y), yx, acc[i][j]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < SP; i++) {
            const int s = s0 + ts + C::TY * i;
            if (s >= nsp) continue;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = r0 + R / 2 * (j >> 1) + 2 * tr + (j & 1);
                if (r < ne)
                    dYc[(long)s * ne + r] = make_float2(acc[i][j].x * scale, acc[i][j].y * scale);
            }
        }
    }
}

template <int R, int SP>
static mdt_status xengine_adjoint_launch(int ne, int nch, int nsp, const float2 *G, const float2 *Y,
                                         float2 *dY, float scale, cudaStream_t stream)
{
    using C = XaCfg<R, SP>;
    // up to four tiles to a block (they share its H) while that leaves four blocks an SM
    const long gx = cdiv(ne, R), all = cdiv(nsp, C::S);
    const int tiles = (int)std::max<long>(1, std::min<long>(4, gx * all * nch / (4L * sm_count())));
    cudaError_t e = cudaFuncSetAttribute(xengine_adjoint_kernel<R, SP>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return cuda_status(e, "xengine_adjoint_f32 smem attribute");
    const dim3 grid((unsigned)gx, (unsigned)cdiv(all, tiles), (unsigned)nch);
    xengine_adjoint_kernel<R, SP><<<grid, XA_THREADS, C::SMEM, stream>>>(ne, nsp, tiles, G, Y, dY,
                                                                         scale);
    return launch_status("xengine_adjoint_kernel");
}

// The tile by the elements and spectra that it would leave empty.  Up to 16 elements
// 16 x 64 spectra (NE=12, Nch=512, Nsp=1000: 40 us; 32 x 128 68, 64 x 64 143).  Up to 32
// spectra 32 x 32 (NE=64, Nsp=30: 31 us; 32 x 128 69, 64 x 64 50), and up to 64 for up to
// 32 elements.  Otherwise 32 x 128 (NE=28, Nsp=1000: 129 us, 64 x 64 249; NE=96 1175
// and 1715, NE=192 4437 and 5078), but for 33 to 64 elements, whose H one 64 x 64 tile
// keeps (NE=64, Nsp=1000: 502 us, 32 x 128 541), and for too few spectra (NE=128,
// Nsp=60: 168 and 262).
static mdt_status xengine_adjoint(int ne, int nch, int nsp, const float2 *G, const float2 *Y,
                                  float2 *dY, float scale, cudaStream_t stream)
{
    if (ne <= 16) return xengine_adjoint_launch<16, 2>(ne, nch, nsp, G, Y, dY, scale, stream);
    if (nsp <= (ne <= 32 ? 64 : 32))
        return xengine_adjoint_launch<32, 2>(ne, nch, nsp, G, Y, dY, scale, stream);
    if (ne > 32 && (ne <= 64 || nsp <= 64))
        return xengine_adjoint_launch<64, 8>(ne, nch, nsp, G, Y, dY, scale, stream);
    return xengine_adjoint_launch<32, 8>(ne, nch, nsp, G, Y, dY, scale, stream);
}

// Partial tap gradients: split p of the (spectrum, element) rows.
// part[p][i][k] = sum over the split's rows (s, e) of
//                 Re(gP[s][e][k] * conj(in[s+i][e][k])), accumulated in double.
__global__ void pfb_tap_grad_partial_kernel(int nch, int ntaps, int ne, int nsp, int nsplit,
                                            const float2 *__restrict__ gP,
                                            const char2 *__restrict__ iq,
                                            double *__restrict__ part)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    const int p = blockIdx.z;
    if (k >= nch) return;
    const long rows = (long)nsp * ne;
    const long r0 = rows * p / nsplit, r1 = rows * (p + 1) / nsplit;
    double acc = 0.0;
    for (long row = r0; row < r1; row++) {
        const long s = row / ne, e = row - s * ne;
        const float2 g = gP[row * nch + k];
        const char2 x = iq[((s + i) * ne + e) * nch + k];
        acc += (double)g.x * (double)x.x + (double)g.y * (double)x.y;
    }
    part[((long)p * ntaps + i) * nch + k] = acc;
}

// NT = 4 or 8 taps at once: part[p][i][k] as above.  A thread owns VEC
// channels and walks runs of `len` spectra of one element, so that every
// gradient value and (but for the NT-1 spectra of a run's lead-in) every
// sample is read once; the samples of the NT taps rotate through registers.
// The runs are dealt to the TG_PH warps of a block and to the splits in turn;
// each thread's sums are compensated FP32, combined in double in a fixed
// order.  Bound by the FP32 pipe (10 operations a product; 145 us at NE=64,
// Nch=512, 4 taps, Nsp=2048) and by latency: 265 us there, 3328 us with sums
// in double.  With 8 taps 455 us (522 with a test on each spectrum of a run).
constexpr int TG_PH = 16, TG_RUN = 32;  // warps, longest run

template <int VEC>
__device__ __forceinline__ void load_iq(const char2 *p, float (&re)[VEC], float (&im)[VEC])
{
    if constexpr (VEC == 2) {
        const char4 t = __ldg(reinterpret_cast<const char4 *>(p));
        re[0] = (float)t.x;
        im[0] = (float)t.y;
        re[1] = (float)t.z;
        im[1] = (float)t.w;
    } else {
        const char2 t = __ldg(p);
        re[0] = (float)t.x;
        im[0] = (float)t.y;
    }
}

template <int NT, int VEC, class Sum>
__device__ __forceinline__ bool tap_sums(int nch, int ne, int nsp, int len, int k, long first, long stride,
                                         const float2 *__restrict__ gP,
                                         const char2 *__restrict__ iq, double (&out)[NT][VEC])
{
    Sum acc[NT][VEC];
    const long nruns = (long)ne * ((nsp + len - 1) / len);
    const long spec = (long)ne * nch;
    for (long t = first; t < nruns; t += stride) {
        const int run = (int)(t / ne), e = (int)(t - (long)run * ne);
        const int s0 = run * len, s1 = min(nsp, s0 + len);
        const float2 *g = gP + (long)s0 * spec + (long)e * nch + k;
        const char2 *x = iq + (long)s0 * spec + (long)e * nch + k;
        float xr[NT][VEC], xi[NT][VEC];  // spectrum s in slot (s - s0) % NT
#pragma unroll
        for (int i = 0; i < NT - 1; i++) load_iq<VEC>(x + i * spec, xr[i], xi[i]);
        // NT spectra from s on; without a test on each, their loads are all issued ahead
        auto group = [&](int s, auto full) {
#pragma unroll
            for (int u = 0; u < NT; u++) {
                if (decltype(full)::value || s + u < s1) {
                    float2 gv[VEC];
                    load_c64<VEC>(g + (long)(s + u - s0) * spec, gv);
                    load_iq<VEC>(x + (long)(s + u - s0 + NT - 1) * spec, xr[(u + NT - 1) % NT],
                                 xi[(u + NT - 1) % NT]);
#pragma unroll
                    for (int i = 0; i < NT; i++)
#pragma unroll
                        for (int v = 0; v < VEC; v++) {
                            acc[i][v].add(gv[v].x, xr[(u + i) % NT][v]);
                            acc[i][v].add(gv[v].y, xi[(u + i) % NT][v]);
                        }
                }
            }
        };
        int s = s0;
        for (; s + NT <= s1; s += NT) group(s, std::true_type());
        if (s < s1) group(s, std::false_type());
    }
    bool ok = true;
#pragma unroll
    for (int i = 0; i < NT; i++)
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            ok = ok && acc[i][v].settled();
            out[i][v] = acc[i][v].value();
        }
    return ok;
}

template <int NT, int VEC>
__global__ void __launch_bounds__(32 * TG_PH, NT * VEC <= 8 ? 2 : 1)
    pfb_tap_grad_all_kernel(int nch, int ne, int nsp, int len, int nsplit,
                            const float2 *__restrict__ gP, const char2 *__restrict__ iq, double *__restrict__ part)
{
    __shared__ double red[TG_PH][32 * VEC];
    const int k = (blockIdx.x * 32 + threadIdx.x) * VEC;
    const int ph = threadIdx.y, p = blockIdx.y;
    const long first = (long)p * TG_PH + ph, stride = (long)nsplit * TG_PH;
    double sum[NT][VEC] = {};
    if (k < nch && !tap_sums<NT, VEC, Sum2>(nch, ne, nsp, len, k, first, stride, gP, iq, sum) &&
        !tap_sums<NT, VEC, SumAny>(nch, ne, nsp, len, k, first, stride, gP, iq, sum))
        tap_sums<NT, VEC, SumD>(nch, ne, nsp, len, k, first, stride, gP, iq, sum);
    const int tid = ph * 32 + threadIdx.x;
#pragma unroll
    for (int i = 0; i < NT; i++) {
#pragma unroll
        for (int v = 0; v < VEC; v++) red[ph][threadIdx.x * VEC + v] = sum[i][v];
        __syncthreads();
        const int kk = blockIdx.x * 32 * VEC + tid;
        if (tid < 32 * VEC && kk < nch) {
            double acc = red[0][tid];
            for (int q = 1; q < TG_PH; q++) acc += red[q][tid];
            part[((long)p * NT + i) * nch + kk] = acc;
        }
        __syncthreads();
    }
}

// gW[i][k] = sum_p part[p][i][k] (deterministic): eight interleaved partial
// sums of 32 outputs per block, added in a fixed order.
__global__ void __launch_bounds__(256)
    pfb_tap_grad_reduce_kernel(int n, int nsplit, const double *__restrict__ part,
                               float *__restrict__ gW)
{
    __shared__ double red[8][32];
    const int j = blockIdx.x * 32 + threadIdx.x;
    double acc = 0.0;
    if (j < n)
        for (int p = threadIdx.y; p < nsplit; p += 8) acc += part[(long)p * n + j];
    red[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && j < n) {
        for (int q = 1; q < 8; q++) acc += red[q][threadIdx.x];
        gW[j] = (float)acc;
    }
}

}  // namespace mdt

extern "C" {

MDT_API mdt_status mdt_xengine_adjoint_f32(int ne, int nch, int nsp, const void *G, const void *Y,
                                           void *dY, float scale, cudaStream_t stream)
{
    if (!G || !Y || !dY || ne < 1 || nch < 1 || nsp < 1 || nch > 65535)
        return mdt::invalid("xengine_adjoint_f32: bad arguments");
    if (mdt::cdiv(nsp, 16) > 65535) return mdt::invalid("xengine_adjoint_f32: Nsp too large");
    return mdt::xengine_adjoint(ne, nch, nsp, (const float2 *)G, (const float2 *)Y, (float2 *)dY,
                                scale, stream);
}

MDT_API mdt_status mdt_apply_gains(int ne, int nch, int nsp, const void *X, const void *gains,
                                   void *Y, cudaStream_t stream)
{
    if (!X || !gains || !Y || ne < 1 || nch < 1 || nsp < 1)
        return mdt::invalid("apply_gains: bad arguments");
    // 16-byte vectors need an even NE (every row and gain pair then starts on one)
    const bool v2 = ne % 2 == 0 && (((uintptr_t)X | (uintptr_t)gains | (uintptr_t)Y) & 15) == 0;
    const int vec = v2 ? 2 : 1;
    const long per = (long)nsp * ne / vec;
    const dim3 grid((unsigned)mdt::cdiv(per, mdt::AG_THREADS * mdt::AG_ITEMS),
                    (unsigned)std::min(nch, 65535));
    const int step = mdt::AG_THREADS * vec % ne;
    if (v2)
        mdt::apply_gains_kernel<2><<<grid, mdt::AG_THREADS, 0, stream>>>(
            nch, ne, per, step, (const float2 *)X, (const float2 *)gains, (float2 *)Y);
    else
        mdt::apply_gains_kernel<1><<<grid, mdt::AG_THREADS, 0, stream>>>(
            nch, ne, per, step, (const float2 *)X, (const float2 *)gains, (float2 *)Y);
    return mdt::launch_status("apply_gains_kernel");
}

MDT_API mdt_status mdt_gain_adjoint(int ne, int nch, int nsp, const void *dY, const void *X,
                                    const void *gains, void *dgains, void *dF,
                                    cudaStream_t stream)
{
    if (!dY || ne < 1 || nch < 1 || nsp < 1 || nch > 65535 * 32)
        return mdt::invalid("gain_adjoint: bad arguments");
    if (dgains) {
        if (!X) return mdt::invalid("gain_adjoint: X is needed for the gain gradient");
        // 16-byte loads need an even NE (every row then starts on one)
        const bool v2 = ne % 2 == 0 && (((uintptr_t)dY | (uintptr_t)X) & 15) == 0;
        const dim3 block(32, mdt::GG_PH);
        const unsigned blocks = (unsigned)mdt::cdiv((long)nch * (ne / (v2 ? 2 : 1)), 32);
        if (v2)
            mdt::gain_grad_kernel<2><<<blocks, block, 0, stream>>>(
                ne, nch, nsp, (const float2 *)dY, (const float2 *)X, (float2 *)dgains);
        else
            mdt::gain_grad_kernel<1><<<blocks, block, 0, stream>>>(
                ne, nch, nsp, (const float2 *)dY, (const float2 *)X, (float2 *)dgains);
        mdt_status st = mdt::launch_status("gain_grad_kernel");
        if (st != MDT_SUCCESS) return st;
    }
    if (dF) {
        const long rows = (long)nsp * ne;
        // tiles of 32 where those of 64 would leave SMs without a pair of blocks
        auto launch = [&](auto kern, int t) {
            const dim3 grid((unsigned)mdt::cdiv(rows, t), (unsigned)mdt::cdiv(nch, t));
            kern<<<grid, dim3(32, t / 4), 0, stream>>>(ne, nch, rows, (const float2 *)dY,
                                                       (const float2 *)gains, (float2 *)dF);
        };
        if (mdt::cdiv(rows, 64) * mdt::cdiv(nch, 64) < 2L * mdt::sm_count())
            launch(mdt::fout_adjoint_kernel<32>, 32);
        else
            launch(mdt::fout_adjoint_kernel<64>, 64);
        return mdt::launch_status("fout_adjoint_kernel");
    }
    return MDT_SUCCESS;
}

MDT_API mdt_status mdt_pfb_tap_grad(int ne, int nch, int ntaps, int nsp, const void *gradP,
                                    const int8_t *iq, float *gradW, void *workspace,
                                    size_t workspace_bytes, cudaStream_t stream)
{
    if (!gradP || !iq || !gradW || !workspace || ne < 1 || nch < 1 || ntaps < 1 || nsp < 1 ||
        ntaps > 65535)
        return mdt::invalid("pfb_tap_grad: bad arguments");
    const long n = (long)ntaps * nch;
    int nsplit = (int)std::min<long>(64, std::max<long>(1, workspace_bytes / (sizeof(double) * n)));
    if (nsplit < 1 || workspace_bytes < sizeof(double) * n)
        return mdt::invalid("pfb_tap_grad: workspace must hold Ntaps*Nch doubles");
    mdt_status st;
    if (ntaps == 4 || ntaps == 8) {
        // two channels per thread (16-byte gradients, 4-byte samples) where Nch is
        // even and the buffers are aligned for it
        const bool v2 = nch % 2 == 0 && ((uintptr_t)gradP & 15) == 0 && ((uintptr_t)iq & 3) == 0;
        // two blocks of 16 warps fit an SM: as many splits as fill the GPU once
        // (64 splits, 1.7 waves at Nch 512: 296 us against 265)
        const long once = 2L * mdt::sm_count() / mdt::cdiv(nch, 32 * (v2 ? 2 : 1));
        // shorter runs where those of 32 spectra are too few for the warps of a wave
        // (NE=28, Nch=512, Nsp=30: 14 us, with runs of 32 25 us)
        int len = mdt::TG_RUN;
        while (len > 8 && ne * mdt::cdiv(nsp, len) < once * mdt::TG_PH) len /= 2;
        const long runs = ne * mdt::cdiv(nsp, len);
        nsplit = (int)std::max<long>(1, std::min<long>(std::min<long>(nsplit, once),
                                                       mdt::cdiv(runs, mdt::TG_PH)));
        auto launch = [&](auto kern, int vec) {
            const dim3 grid((unsigned)mdt::cdiv(nch, 32 * vec), (unsigned)nsplit);
            kern<<<grid, dim3(32, mdt::TG_PH), 0, stream>>>(
                nch, ne, nsp, len, nsplit, (const float2 *)gradP, (const char2 *)iq, (double *)workspace);
        };
        if (ntaps == 4) {
            if (v2) launch(mdt::pfb_tap_grad_all_kernel<4, 2>, 2);
            else launch(mdt::pfb_tap_grad_all_kernel<4, 1>, 1);
        } else {
            if (v2) launch(mdt::pfb_tap_grad_all_kernel<8, 2>, 2);
            else launch(mdt::pfb_tap_grad_all_kernel<8, 1>, 1);
        }
        st = mdt::launch_status("pfb_tap_grad_all_kernel");
    } else {
        dim3 grid((unsigned)mdt::cdiv(nch, 128), (unsigned)ntaps, (unsigned)nsplit);
        mdt::pfb_tap_grad_partial_kernel<<<grid, 128, 0, stream>>>(
            nch, ntaps, ne, nsp, nsplit, (const float2 *)gradP, (const char2 *)iq,
            (double *)workspace);
        st = mdt::launch_status("pfb_tap_grad_partial_kernel");
    }
    if (st != MDT_SUCCESS) return st;
    mdt::pfb_tap_grad_reduce_kernel<<<(unsigned)mdt::cdiv(n, 32), dim3(32, 8), 0, stream>>>(
        (int)n, nsplit, (const double *)workspace, gradW);
    return mdt::launch_status("pfb_tap_grad_reduce_kernel");
}

}  // extern "C"
