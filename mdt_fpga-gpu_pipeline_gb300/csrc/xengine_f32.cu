// xengine_f32.cu -- FP32 Hermitian X-engine on the tensor cores: per channel c
//   V_c = alpha * X_c X_c^H
// on the lower triangle, mirrored; the reference's cublasCgemmBatched call
// (OP_N, OP_C, A == B, alpha = 1/Nspectra, beta = 0;
// MDT_OneStation_client.cu:1128, :656-660, :683-686).
//
// Arithmetic.  Over a stage of 64 spectra an element's samples are scaled by a
// power of two that brings the largest component to [1024, 2048) and split into
// an integer h and the rest l in f16: x s = h + l, |l| <= 1/2, which keeps 23
// bits below the largest component.  A product of two samples is
//   (x s)(y t) = h h' + (h l' + l h' + l l'),
// exact f16 products all.  The h h' sum is kept apart from the others: it is a
// sum of integers, exact in FP32 below 2^24.  That matters because the tensor
// core truncates when it adds to its accumulator: sums with fractions lose half a
// unit per step, always towards zero (f16 pairs split by value: autocorrelations
// 2.3e-7 low after 64 spectra).  Noise reaches 2^23 to 2^25 (autocorrelations 0.3e-7
// low), a tone of constant amplitude 2^28: its autocorrelations come out 0.7e-7 to
// 1.5e-7 low, with an error of 1.1e-7 (SIMT kernel: 0.6e-7 at 10 inputs, 1.6e-7 to
// 6e-7 at 40).  Half the scale ends that (0.2e-7), but costs products of unlike
// elements a bit (noise, 1000 spectra: 3.3e-7 for 1.8e-7; SIMT 2.2e-7).  The stage's sums go to FP32 registers, XF_FLUSH
// stages at a time and then to a second level, so that a visibility of 1000
// spectra is rounded about ten times, not a thousand times.
// Relative error of V against 64-bit sums of the same FP32 samples (normal
// noise), here and by FP32 multiply-adds in spectrum order (the SIMT kernel):
//   NE=10, Nsp=1000: 5.8e-8, 9.2e-8;   NE=40, Nsp=512: 7.1e-8, 2.4e-7;
//   NE=40, Nsp=4096: 6.0e-8, 6.2e-7;   NE=256, Nsp=2048: 7.9e-8, 8.8e-7.
//
// Where it does not hold.  The rest is rounded on the grid of the largest component, so
// samples far below it lose bits that FP32 would keep; if the other element is zero where
// the large ones are (a burst in one element, spectra lost in the other), nothing makes up
// for it: a spectrum of 64 that is 2^10 above the others cost 5e-6 of such a visibility,
// 2^16 2e-5.  So on the diagonal tiles the kernel counts for each element and stage the
// spectra with a component within 2^-4 (at most 2^-5) of the largest; where a quarter or
// more are below, or the largest is outside [2^-48, 2^48] or not finite, it leaves a mark
// for the element (xf_mark), and xengine_simt_redo forms all its visibilities by FP32
// multiply-adds.  Two elements that pass share half the spectra of every stage well above
// the grid.  (Normal noise fails less than once in 10^9 stages; an element that is zero
// throughout a stage passes, its products are exact.)  Infinities and NaN appear as those
// multiply-adds give them.  A block whose waits gave up (each is bounded) leaves its whole
// tile to them.
//
// Layout of the products: re and im of an element are separate rows of one real
// operand Z (2 nb rows, nb = elements rounded up to 8), and D = Z Z^T holds
//   Re V_rq = D[re r][re q] + D[im r][im q],  Im V_rq = D[im r][re q] - D[re r][im q],
// four real products per pair and no product formed twice.  M = 128 rows are 64
// elements of one channel, or, so that small arrays fill the instruction and
// share its latency, 32 elements of two channels or 16 of four (the products
// between channels are ignored).  Larger arrays are cut into 64 x 64 tiles.
//
// A block per SM: sixteen converting warps and an issuing one (issuing an MMA
// holds the thread until the queue takes it).  Per stage a converting thread
// loads eight samples of one element per operand, converts them into words of
// the K-major 128-byte-swizzled operand, and adds the sums of an earlier stage from
// tensor memory to its registers.  Two operand stages and two accumulator sets
// alternate: while the tensor core works on stage k + 1, the warps drain stage k
// and write stage k + 2 over its operands.
//
// What bounds it: an M = 128, K = 16 MMA takes 63 cycles for any N up to 128, so the
// sixteen of a stage take 1000 of the 3150 cycles that a stage takes at 40 inputs and of
// the 4600 at 256; the rest is the warps' chain of tensor-memory reads, conversion and
// sample loads, one after the other.  The count takes 50 to 150 cycles of a stage, the
// search for marks 2 us (a plan's X-engine without them: NE=10, Nch=1024, Nsp=1000 56 us,
// with them 59; NE=32, Nsp=4096 392 and 430; NE=40, Nch=2048, Nsp=4096 1.34 and 1.39 ms;
// NE=256, Nch=1024, Nsp=2048 4.97 and 4.93).  Against the SIMT kernel, Nch=1024, Nsp=1000:
// NE=10 59 us, 68; NE=20 112, 104; NE=32 127, 171; NE=40 203, 229; NE=64 253, 563; NE=65
// 683, 839; NE=128 0.78 ms, 1.85; NE=256 2.71, 6.35.
#include <cuda_fp16.h>

#include <algorithm>

#include "tc_ptx.cuh"
#include "xengine_f32.cuh"

namespace mdt {

constexpr int XF_WARPS = 16;  // converting warps, then the issuing one
// With 128 rows a channel the issuing warp has three more without work beside it, since
// registers are shared out by warpgroups: of the XF_REGS a thread at the launch the
// converting ones take XF_REGS_CONV, the others keep XF_REGS_REST, the same 61,440 in all.
constexpr int XF_REGS = 96, XF_REGS_CONV = 104, XF_REGS_REST = 64;
constexpr int xf_threads(int slot) { return 32 * (XF_WARPS + (slot == 128 ? 4 : 1)); }
static_assert(XF_REGS_CONV * 32 * XF_WARPS + XF_REGS_REST * 32 * 4 <= XF_REGS * xf_threads(128), "register split");
constexpr int XF_K = 64;                          // spectra per stage
constexpr int XF_PLANE = 128 * 128;               // 128 rows of 64 f16
constexpr int XF_OPERAND = 2 * XF_PLANE;          // h, l
constexpr int XF_AHEAD = 3;                       // stages between L2 prefetch and load
constexpr int XF_FLUSH = 8;                       // stages per first-level sum
// Spectra from which the tensor cores are used.  Shorter sums round little in FP32
// multiply-adds (NE=10: 6.7e-8 at 64 spectra, 8.6e-8 at 250), there the split is no closer
// to the 64-bit sums, and there is little time to gain.  At the line, Nch=1024, 256 and 400
// spectra, here and by the SIMT kernel:  NE=3 23 and 31 us, 18 and 25;  NE=16 25 and 33, 26
// and 37;  NE=20 41 and 55, 33 and 48;  NE=33 68 and 100, 64 and 97;  NE=64 94 and 130, 153
// and 238;  NE=129 494 and 713, 601 and 931.  Up to 24 inputs the SIMT kernel is the faster
// up to some 600 spectra, but rounds more (400 spectra: NE=3 5.3e-8 here, 7.1e-8; NE=20
// 6.3e-8, 7.9e-8; NE=33 7.0e-8, 2.3e-7), so the line is the same for all.
constexpr int XF_MIN_SPECTRA = 256;
// A stage of an element is uneven if, of its spectra, a quarter or more have no component
// of XF_SIG or above in the scale that brings the largest one to [1024, 2048), or if that
// one is outside [2^-XF_EXP, 2^XF_EXP] (whose products are far from FP32's limits).
constexpr float XF_SIG = 64.0f;
constexpr int XF_EXP = 48;
constexpr int XF_DS = 129;                        // floats per row of the exchanged sums
constexpr size_t XF_D_BYTES = (size_t)128 * XF_DS * sizeof(float);
constexpr size_t xf_smem(bool off)
{
    return 1024 + (size_t)2 * (off ? 2 : 1) * XF_OPERAND + XF_D_BYTES;
}

struct XfArgs {
    int ne, nsp, npairs;
    int nb;                      // operand rows of re (and of im) per channel
    const float2 *X;             // base (when Xptrs == nullptr)
    const float2 *const *Xptrs;  // per-channel operand pointers (cuBLAS shim)
    long ld, xstride;
    float2 *V;
    float2 *const *Vptrs;
    long ldv, vstride;
    float2 alpha;
    long nbatch;
};

// Two floats as packed f16 (a in the low half), round to nearest even.
__device__ __forceinline__ uint32_t f16x2(float2 v)
{
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
    return r;
}

// The largest of three values; NaN if one of them is.
__device__ __forceinline__ float max_nan(float a, float b, float c)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Counts the spectra that have a component of XF_SIG or above, two at a time (re, im:
// their integers as f16 pairs), from 1024 in the low half and 0 in the high one.
__device__ __forceinline__ void count_significant(__half2 &n, uint32_t re, uint32_t im)
{
    const __half2 a = __habs2(*reinterpret_cast<const __half2 *>(&re));
    const __half2 b = __habs2(*reinterpret_cast<const __half2 *>(&im));
    n = __hadd2(n, __hge2(__hmax2(a, b), __float2half2_rn(XF_SIG)));
}

__device__ __forceinline__ int lane_significant(__half2 n)
{
    // 1024 + the lane's count, as f16: the low digits of its bits
    return __half_as_ushort(__hadd(__low2half(n), __high2half(n))) & 15;
}

// Of the eight lanes that hold an element (all lanes of the warp): a byte for each element.
__device__ __forceinline__ int total_significant(__half2 n)
{
    const int at = threadIdx.x & 24;
    return __reduce_add_sync(0xffffffffu, (uint32_t)lane_significant(n) << at) >> at & 255;
}

// OFF: the grid holds tiles below the diagonal (NE > 64), with an operand of
// their own for the columns.  SLOT: rows of M per channel (128, 64 or 32).
// BLOCKED: operand X[(k/8)*ld + e*8 + k%8] (blocks of 8 spectra, the last one
// zero-padded), else X[k*ld + e].
template <bool OFF, int SLOT, bool BLOCKED>
__global__ void __launch_bounds__(xf_threads(SLOT), 1) xengine_f32_kernel(const XfArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t bars[4];  // full[2] (operands written), done[2] (products complete)
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ bool s_uneven[64];  // elements of a diagonal tile: in one of their stages
    __shared__ __align__(16) float s_inv[4][2][64];  // [stage % 4][operand][element]: 1 / scale
    constexpr int NSLOT = 128 / SLOT, EB = SLOT / 2;  // channels, and elements per channel
    constexpr int STAGE = (OFF ? 2 : 1) * XF_OPERAND;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;

    const long ch0 = OFF ? blockIdx.x / a.npairs : (long)blockIdx.x * NSLOT;
    int I = 0, J = 0;
    if constexpr (OFF) {
        const int p = (int)(blockIdx.x - ch0 * a.npairs);  // p = I (I + 1) / 2 + J
        I = (int)((sqrtf(8.0f * p + 1.0f) - 1.0f) * 0.5f);
        while ((I + 1) * (I + 2) / 2 <= p) I++;
        while (I * (I + 1) / 2 > p) I--;
        J = p - I * (I + 1) / 2;
    }
    const bool sep = OFF && I != J;  // columns have their own operand
    const int r0 = I * 64, q0 = J * 64;
    const int nr = min(EB, a.ne - r0), nq = min(EB, a.ne - q0);
    const int nb = OFF ? 64 : a.nb;
    // Stages of 64 spectra, but the first two share what is left (32 or more each): a short
    // one has too few for the count of significant spectra (of 16 normally distributed ones,
    // one in 10^5 has four small ones; with a last stage of 16 of 400 spectra, some channel
    // nearly always went to xengine_simt_redo, 152 us for 105 at NE=38, Nch=1024).
    const int nstage = (a.nsp + XF_K - 1) / XF_K;              // four or more (XF_MIN_SPECTRA)
    const int two = 2 * XF_K - (nstage * XF_K - a.nsp) / 8 * 8;  // of the first two together
    const int first = (two / 2 + 7) / 8 * 8;                   // of the first

    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(tc::smem_u32(&bars[i]), XF_WARPS);
            tc::mbar_init(tc::smem_u32(&bars[2 + i]), 1);
        }
        s_fail = 0;
        tc::fence_mbar_init();
    }
    if (warp == XF_WARPS) {
        tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
        tc::tmem_relinquish();
        tc::fence_before_sync();
    }
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp >= XF_WARPS) {
        if constexpr (SLOT == 128) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(XF_REGS_REST));
        if (warp == XF_WARPS && lane == 0) {
            // ---------------- MMA issuer: h h' to columns 0..127 of the stage's set,
            // the products with l to columns 128..255
            const int N = (NSLOT - 1) * SLOT + 2 * nb;
            const uint32_t id = tc::idesc_f16(N, 0, 0);
            bool ok = true;
            for (int k = 0; k < nstage && ok; k++) {
                const int s = k & 1;
                ok = tc::mbar_wait(tc::smem_u32(&bars[s]), (k >> 1) & 1);
                if (!ok) break;
                tc::fence_after_sync();
                const uint32_t sa = tc::smem_u32(smem + (size_t)s * STAGE);
                const uint64_t ad = tc::sw128_kmajor_desc(sa);
                const uint64_t bd = tc::sw128_kmajor_desc(sep ? sa + XF_OPERAND : sa);
                const uint32_t d = tmem + (uint32_t)(s * 256);
                constexpr uint64_t L = XF_PLANE >> 4;
#pragma unroll
                for (int j = 0; j < 4; j++) {  // 16 spectra each
                    tc::mma_f16(d, ad + 2 * j, bd + 2 * j, id, j > 0);
                    tc::mma_f16(d + 128, ad + L + 2 * j, bd + L + 2 * j, id, j > 0);
                    tc::mma_f16(d + 128, ad + 2 * j, bd + L + 2 * j, id, 1);
                    tc::mma_f16(d + 128, ad + L + 2 * j, bd + 2 * j, id, 1);
                }
                tc::mma_commit(tc::smem_u32(&bars[2 + s]));
            }
            if (!ok) atomicExch(&s_fail, 1);
        }
        __syncwarp();
    } else {
        if constexpr (SLOT == 128) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(XF_REGS_CONV));
        // ---------------- converting warps.  A thread takes element e of channel
        // slot g and the spectra 8 (4 sg + i) + 2 p + {0, 1}, i < 4, of a stage: in
        // the blocked layout four lanes (p) read 64 contiguous bytes, and a warp's
        // 4-byte stores fall in 32 banks.
        const int p = lane & 3, sg = (lane >> 2) & 1, el = warp * 4 + (lane >> 3);
        const int e = el % EB, g = el / EB;
        const bool liveA = ch0 + g < a.nbatch && e < nr, liveB = sep && e < nq;
        const long ch = min(ch0 + g, a.nbatch - 1);
        const float2 *Xc = a.Xptrs ? a.Xptrs[ch] : a.X + ch * a.xstride;
        const float2 *xa = Xc + (BLOCKED ? (long)(r0 + e) * 8 : (long)(r0 + e));
        const float2 *xb = Xc + (BLOCKED ? (long)(q0 + e) * 8 : (long)(q0 + e));
        float2 re[4], im[4];  // the two spectra of run i
        // spectra s0 .. s0 + 63, but none from s1 on
        auto load = [&](const float2 *x, bool live, int s0, int s1) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int s = s0 + 8 * (4 * sg + i);
                if constexpr (BLOCKED) {
                    const float4 v = live && s < s1
                                         ? __ldg(reinterpret_cast<const float4 *>(x + (long)(s >> 3) * a.ld) + p)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
                    re[i] = make_float2(v.x, v.z);
                    im[i] = make_float2(v.y, v.w);
                } else {
                    const int s2 = s + 2 * p;
                    const float2 u = live && s2 < s1 ? __ldg(x + (long)s2 * a.ld) : make_float2(0.f, 0.f);
                    const float2 v = live && s2 + 1 < s1 ? __ldg(x + (long)(s2 + 1) * a.ld)
                                                         : make_float2(0.f, 0.f);
                    re[i] = make_float2(u.x, v.x);
                    im[i] = make_float2(u.y, v.y);
                }
            }
            // into L2, XF_AHEAD stages further on
            if constexpr (BLOCKED) {
                const int s = s0 + XF_AHEAD * XF_K + 8 * (4 * sg + p);
                if (live && s < a.nsp && !(e & 1))
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (long)(s >> 3) * a.ld));
            } else {
                const int s = s0 + XF_AHEAD * XF_K + 8 * (4 * sg + p) + 2 * (e & 3);
                if (live && s < a.nsp) {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (long)s * a.ld));
                    if (s + 1 < a.nsp)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (long)(s + 1) * a.ld));
                }
            }
        };
        // writes the operand rows; on a diagonal tile the lane's count of significant spectra
        auto convert = [&](int k, int op, bool live) {
            // the eight lanes of an element agree on the scale
            float m = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                m = max_nan(m, fabsf(re[i].x), fabsf(re[i].y));
                m = max_nan(m, fabsf(im[i].x), fabsf(im[i].y));
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) m = max_nan(m, m, __shfl_xor_sync(0xffffffffu, m, o));
            // scale 2^(10 - exponent of m); at most 2^126, so that its inverse is normal
            const int bs = min(127 + 10 + 127 - (int)(__float_as_uint(m) >> 23), 253);
            const float sc = __uint_as_float((uint32_t)bs << 23);
            if ((lane & 7) == 0) s_inv[k & 3][op][el] = __uint_as_float((uint32_t)(254 - bs) << 23);
            const __half2 none = __floats2half2_rn(1024.f, 0.f), all = __floats2half2_rn(1024.f + 8.f, 0.f);
            if (!live) return all;  // rows without an element feed sums that are never read
            const float2 sc2 = make_float2(sc, sc);
            const float2 big = make_float2(12582912.0f, 12582912.0f);  // 1.5 * 2^23: rounds to integers
            const float2 nbig = make_float2(-12582912.0f, -12582912.0f);
            uint8_t *st = smem + (size_t)(k & 1) * STAGE + (size_t)op * XF_OPERAND;
            __half2 nsig = none;
            uint32_t hre[4];
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int row = g * SLOT + c * nb + e;
                uint8_t *w = st + row * 128 + 4 * p;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 x = c ? im[i] : re[i];
                    const float2 h = __fadd2_rn(__ffma2_rn(x, sc2, big), nbig);
                    const float2 l = __ffma2_rn(x, sc2, make_float2(-h.x, -h.y));
                    const int at = ((4 * sg + i) ^ (row & 7)) << 4;
                    const uint32_t h16 = f16x2(h);
                    *reinterpret_cast<uint32_t *>(w + at) = h16;
                    *reinterpret_cast<uint32_t *>(w + at + XF_PLANE) = f16x2(l);
                    if (c == 0)
                        hre[i] = h16;
                    else if (!sep)
                        count_significant(nsig, hre[i], h16);
                }
            }
            if (m == 0.0f) return all;
            return m >= 1.0f / (1ll << XF_EXP) && m <= (float)(1ll << XF_EXP) ? nsig : none;
        };
        bool uneven = false;
        auto check = [&](int n, __half2 nsig) {  // n: spectra of the stage
            if (!sep) {
                // a quarter of 64 spectra are two or more of some lane's eight, which few warps
                // have (asking first gains 6 us of 399 at NE=20, Nsp=4096, but costs 20 of 1376
                // with OFF at NE=129, Nch=512, Nsp=2048)
                if (OFF || n < XF_K || __any_sync(0xffffffffu, lane_significant(nsig) <= 6)) {
                    const int sig = total_significant(nsig);  // by all lanes
                    uneven |= sig < n - (n - 1) / 4;
                }
            }
        };
        auto arrive = [&](int k) {  // operands of stage k written, sums of stage k - 2 read
            tc::fence_proxy_async();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(tc::smem_u32(&bars[k & 1]));
        };
        // this thread's sums: row (warp & 3) * 32 + lane, columns col0 .. col0 + nb / 2, of
        // the channel slot that the row belongs to
        const int quarter = warp & 3, cg = warp >> 2;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int slot = quarter * 32 / SLOT, q_el = (cg & 1) * (nb / 2);
        const int col0 = slot * SLOT + (cg >> 1) * nb + q_el;
        int r_el = quarter * 32 + lane - slot * SLOT;  // element of the row
        r_el = r_el >= nb ? r_el - nb : r_el;
        r_el = min(r_el, EB - 1);
        constexpr int NC = EB / 4;  // pairs of columns
        float2 acc[NC];
#pragma unroll
        for (int i = 0; i < NC; i++) acc[i] = make_float2(0.f, 0.f);
        // second-level sums, after the operands: each thread its own entries until the end
        float *D = reinterpret_cast<float *>(smem + 2 * STAGE);
        float *drow = D + (quarter * 32 + lane) * XF_DS + col0;
        auto flush = [&](bool first) {
#pragma unroll
            for (int j = 0; j < NC; j++)
                if (2 * j < nb / 2) {
                    drow[2 * j] = first ? acc[j].x : drow[2 * j] + acc[j].x;
                    drow[2 * j + 1] = first ? acc[j].y : drow[2 * j + 1] + acc[j].y;
                    acc[j] = make_float2(0.f, 0.f);
                }
        };
        auto drain = [&](int k) {
            const uint32_t d = tmem + (uint32_t)((k & 1) * 256) + lane_off + (uint32_t)col0;
            const float sr = s_inv[k & 3][0][slot * EB + r_el];
            const float2 sr2 = make_float2(sr, sr);
            const float *sq = &s_inv[k & 3][sep ? 1 : 0][slot * EB + q_el];
#pragma unroll
            for (int c = 0; c < 2 * NC; c += 8) {
                if (c >= nb / 2) break;  // uniform
                uint32_t v[8], w[8];
                tc::tmem_ld8(d + c, v);
                tc::tmem_ld8(d + 128 + c, w);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 t = __fadd2_rn(
                        make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])),
                        make_float2(__uint_as_float(w[2 * j]), __uint_as_float(w[2 * j + 1])));
                    const float2 f = __fmul2_rn(sr2, *reinterpret_cast<const float2 *>(sq + c + 2 * j));
                    acc[c / 2 + j] = __ffma2_rn(t, f, acc[c / 2 + j]);
                }
            }
        };
        bool ok = true;
        for (int k = 0; k < 2; k++) {
            const int s0 = k ? first : 0, s1 = k ? two : first;
            load(xa, liveA, s0, s1);
            const __half2 nsig = convert(k, 0, liveA);
            if (sep) {
                load(xb, liveB, s0, s1);
                convert(k, 1, liveB);
            }
            arrive(k);
            check(s1 - s0, nsig);
        }
        load(xa, liveA, two, a.nsp);
        for (int k = 0; k < nstage; k++) {
            const int s = k & 1;
            // the products are complete; all warps' scales of the stage are written
            ok = ok && tc::mbar_wait(tc::smem_u32(&bars[2 + s]), (k >> 1) & 1) &&
                 tc::mbar_wait(tc::smem_u32(&bars[s]), (k >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::fence_after_sync();
            const bool more = k + 2 < nstage;
            drain(k);
            __half2 nsig;
            if (more) {
                nsig = convert(k + 2, 0, liveA);
                if (sep) load(xb, liveB, two + k * XF_K, a.nsp);
            }
            if (k % XF_FLUSH == XF_FLUSH - 1) flush(k < XF_FLUSH);
            if (more) {
                if (sep) convert(k + 2, 1, liveB);
                arrive(k + 2);
                if (k + 3 < nstage) load(xa, liveA, two + (k + 1) * XF_K, a.nsp);
                check(min(XF_K, a.nsp - two - k * XF_K), nsig);
            }
        }
        if (!ok && lane == 0) atomicExch(&s_fail, 1);
        tc::fence_before_sync();
        flush(nstage < XF_FLUSH);
        if ((lane & 7) == 0) s_uneven[el] = uneven;
        tc::named_barrier(1, 32 * XF_WARPS);
        const bool fail = s_fail != 0;
        auto put = [&](float2 *Vc, long at, float2 v) {
            Vc[at] = make_float2(a.alpha.x * v.x - a.alpha.y * v.y, a.alpha.x * v.y + a.alpha.y * v.x);
        };
        for (int sl = 0; sl < NSLOT; sl++) {
            const long c = ch0 + sl;
            if (c >= a.nbatch) break;
            float2 *Vc = a.Vptrs ? a.Vptrs[c] : a.V + c * a.vstride;
            const float *Ds = D + sl * SLOT * XF_DS + sl * SLOT;
            auto at = [&](int r, int q) { return Ds[r * XF_DS + q]; };
            // sum over the spectra for row r, column q of the tile (r >= q on the diagonal)
            auto product = [&](int r, int q) {
                return make_float2(at(r, q) + at(nb + r, nb + q), at(nb + r, q) - at(r, nb + q));
            };
            if (!sep) {  // the tile's square, the upper half as conjugates
                for (int i = tid; i < nr * nr; i += 32 * XF_WARPS) {
                    const int q = i / nr, r = i - q * nr;
                    float2 v = product(max(r, q), min(r, q));
                    if (r == q) v.y = 0.f;  // autocorrelations are real
                    if (r < q) v.y = -v.y;
                    put(Vc, (long)(q0 + q) * a.ldv + r0 + r, v);
                    if (r == q && (fail || s_uneven[sl * EB + r])) Vc[(long)(q0 + q) * a.ldv + r0 + r] = xf_mark();
                }
            } else {
                for (int i = tid; i < nr * 64; i += 32 * XF_WARPS) {
                    const int q = i / nr, r = i - q * nr;
                    put(Vc, (long)(q0 + q) * a.ldv + r0 + r, product(r, q));
                    if (i == 0 && fail) Vc[(long)q0 * a.ldv + r0] = xf_mark();
                }
                for (int i = tid; i < nr * 64; i += 32 * XF_WARPS) {
                    const int r = i >> 6, q = i & 63;
                    const float2 v = product(r, q);
                    put(Vc, (long)(r0 + r) * a.ldv + q0 + q, make_float2(v.x, -v.y));
                }
            }
        }
    }
    __syncthreads();
    if (warp == XF_WARPS) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 512);
    }
}

// Whether a launch has the registers that the converting warps take: setmaxnreg waits
// for ever where it has not.
static bool split_fits(void (*kern)(const XfArgs))
{
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess && (fa.numRegs + 7) / 8 * 8 >= XF_REGS;
}

mdt_status xengine_herm_f32(int ne, long nbatch, int nsp, const float2 *X,
                            const float2 *const *Xptrs, long ld, long xstride, float2 *V,
                            float2 *const *Vptrs, long ldv, long vstride, float2 alpha,
                            float2 beta, bool beta_zero, cudaStream_t stream, int blocked)
{
    if (ne <= 0 || nbatch <= 0) return MDT_SUCCESS;
    // blocked: complex64 between 8-sample blocks; read as 16-byte vectors
    if (blocked && ld == 0) ld = (long)ne * 8;
    const bool vectors = !blocked || (((uintptr_t)X & 15) == 0 && !Xptrs && ld % 2 == 0 && xstride % 2 == 0);
    if (nsp < XF_MIN_SPECTRA || !vectors || ne > (1 << 20))
        return xengine_simt_f32(ne, nbatch, nsp, X, Xptrs, ld, xstride, V, Vptrs, ldv, vstride, alpha,
                                beta, beta_zero, stream, blocked);
    // what a visibility was before cannot be added again to one that is formed twice
    if (!beta_zero)
        return xengine_simt_redo(ne, nbatch, nsp, X, Xptrs, ld, xstride, V, Vptrs, ldv, vstride, alpha,
                                 beta, false, true, stream, blocked);
    XfArgs a;
    a.ne = ne;
    a.nsp = nsp;
    a.npairs = (int)(cdiv(ne, 64) * (cdiv(ne, 64) + 1) / 2);
    a.nb = (ne + 7) / 8 * 8;
    a.X = X;
    a.Xptrs = Xptrs;
    a.ld = ld;
    a.xstride = xstride;
    a.V = V;
    a.Vptrs = Vptrs;
    a.ldv = ldv;
    a.vstride = vstride;
    a.alpha = alpha;
    a.nbatch = nbatch;
    auto launch = [&](auto kern, bool off, int slot, long blocks) -> mdt_status {
        if (blocks > 0x7fffffffL) return invalid("xengine: grid too large");
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)xf_smem(off));
        if (e != cudaSuccess) return cuda_status(e, "xengine smem attribute");
        if (slot == 128 && !split_fits(kern)) return invalid("xengine: compiled with too few registers to split");
        kern<<<(unsigned)blocks, xf_threads(slot), xf_smem(off), stream>>>(a);
        const mdt_status st = launch_status("xengine_f32_kernel");
        if (st != MDT_SUCCESS) return st;
        return xengine_simt_redo(ne, nbatch, nsp, X, Xptrs, ld, xstride, V, Vptrs, ldv, vstride, alpha,
                                 make_float2(0.f, 0.f), true, false, stream, blocked);
    };
    if (ne > 64)
        return blocked ? launch(xengine_f32_kernel<true, 128, true>, true, 128, nbatch * a.npairs)
                       : launch(xengine_f32_kernel<true, 128, false>, true, 128, nbatch * a.npairs);
    if (ne > 32)
        return blocked ? launch(xengine_f32_kernel<false, 128, true>, false, 128, nbatch)
                       : launch(xengine_f32_kernel<false, 128, false>, false, 128, nbatch);
    if (ne > 16)
        return blocked ? launch(xengine_f32_kernel<false, 64, true>, false, 64, cdiv(nbatch, 2))
                       : launch(xengine_f32_kernel<false, 64, false>, false, 64, cdiv(nbatch, 2));
    return blocked ? launch(xengine_f32_kernel<false, 32, true>, false, 32, cdiv(nbatch, 4))
                   : launch(xengine_f32_kernel<false, 32, false>, false, 32, cdiv(nbatch, 4));
}

}  // namespace mdt
