// depack.cu -- GPU depacketiser: SNAP packets -> [spectrum][element][channel]
// samples, with packet-gap detection.
//
// Replaces the host loop of the reference client's rank 1
// (MDT_OneStation_client.cu:846-907).  A packet is `words_header` 32-bit
// header words -- [0] station, [1] SNAP board, [2] packet counter -- then
// `sper_element` samples for each of InputsPerSNAP[snap] inputs, sample-major
// (payload sample (i, j) = input j of sample i).  Element-sample index of
// sample i is counter * sper_element + i; its spectrum is index / Nch and its
// channel index % Nch.  Element = station * inputs_per_station +
// sum_{k < snap} InputsPerSNAP[k] + j.
//
// Samples are either the reference's int32 fixed point (two words, re and im,
// scaled by 2^-19 into complex64) or int8 I/Q pairs (two bytes, copied to the
// int8 I/Q layout of the fused path).  The int32 conversion follows the
// reference bit for bit, including its mapping of 0x80000000 to +4096.0
// (the reference negates 2^32 - w through an int, which wraps for w = 2^31).
//
// The output window is element-samples [sample0, sample0 + nspectra * Nch)
// (sample0 a multiple of Nch); packets outside it are counted and skipped.
// Arrivals are counted per (station, SNAP, packet slot) in `seen`; the finish
// step zero-fills the samples of slots that never arrived, counts them, and
// clears `seen` for the next window.
#include <algorithm>

#include "mdt_common.cuh"

namespace mdt {

struct DepackGeom {
    int hdr_words, sper, ips, nsnap, nstation, bits;
    long pkt_bytes;
    int ne, nch, nspectra;
    long long sample0, c0;  // first packet counter touching the window
    long nslots;
    int snap_off[MDT_MAX_SNAPS + 1];
    int snap_n[MDT_MAX_SNAPS];
};

__device__ __forceinline__ float fixed19_to_float(uint32_t w)
{
    // reference: w >= 2^31 -> -2^-19 * (int)(2^32 - w), else 2^-19 * (int)w,
    // both in double, then rounded to float.
    if (w == 0x80000000u) return 4096.0f;
    return __int2float_rn((int)w) * 1.9073486328125e-06f;
}

__global__ void depacketise_kernel(DepackGeom g, const unsigned char *__restrict__ pkts,
                                   void *__restrict__ out, unsigned int *__restrict__ seen,
                                   mdt_depack_stats *__restrict__ stats)
{
    const unsigned char *p = pkts + (long)blockIdx.x * g.pkt_bytes;
    const uint32_t *hdr = (const uint32_t *)p;
    const uint32_t station = hdr[0], snap = hdr[1], counter = hdr[2];
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        int ok = 1;
        if (snap >= (uint32_t)g.nsnap || station >= (uint32_t)g.nstation ||
            (long)station * g.ips + g.snap_off[snap] + g.snap_n[snap] > g.ne) {
            atomicAdd(&stats->bad, 1ull);
            ok = 0;
        } else {
            const long long slot = (long long)counter - g.c0;
            if (slot < 0 || slot >= g.nslots) {
                atomicAdd(&stats->outside, 1ull);
                ok = 0;
            } else {
                const unsigned int prev =
                    atomicAdd(&seen[((long)station * g.nsnap + snap) * g.nslots + slot], 1u);
                if (prev) atomicAdd(&stats->duplicate, 1ull);
                atomicAdd(&stats->accepted, 1ull);
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) return;
    const int nin = g.snap_n[snap];
    const long elem0 = (long)station * g.ips + g.snap_off[snap];
    const long long first = (long long)counter * g.sper - g.sample0;
    const long long wlen = (long long)g.nspectra * g.nch;
    const int total = g.sper * nin;
    // consecutive threads take consecutive samples of one input, so the
    // stores run along channels
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int j = idx / g.sper, i = idx - j * g.sper;
        const long long s = first + i;
        if (s < 0 || s >= wlen) continue;
        const long long spec = s / g.nch;
        const int chan = (int)(s - spec * g.nch);
        const long o = ((long)spec * g.ne + elem0 + j) * g.nch + chan;
        if (g.bits == 32) {
            const uint32_t *w = hdr + g.hdr_words + 2 * (i * nin + j);
            ((float2 *)out)[o] = make_float2(fixed19_to_float(w[0]), fixed19_to_float(w[1]));
        } else {
            const char2 *w = (const char2 *)(p + 4 * g.hdr_words) + (i * nin + j);
            ((char2 *)out)[o] = *w;
        }
    }
}

// The same for packets whose 32-sample runs fit a warp's staging buffer: one
// warp per packet, `turns` packets per warp, four apart.  Payload words are copied
// contiguously (WB = 16 bytes where the packets' alignment allows it, else 4)
// into one of the warp's two buffers with cp.async, the next packet's before
// this one's header is looked at, and written with the lanes along the samples
// of one input, i.e. along channels.  The counters are summed per block and
// added once (one atomic per packet on the same counter serialises in L2).
// Bound by HBM: 8 + 8 (int32) or 2 + 2 (int8) bytes a sample.  38 inputs, 1024
// channels and spectra, 28 samples a packet, int32: 123 us (5.2 TB/s) against
// 205 us with a block per packet and strided 8-byte reads; without the second
// buffer 141 us.
constexpr int DP_WARPS = 4;
constexpr int DP_BUF = 4096;  // bytes of a staging buffer

template <int WB>
__device__ __forceinline__ void copy_words(unsigned char *dst, const unsigned char *src, int words,
                                           int lane)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int w = lane; w < words; w += 32)
        if constexpr (WB == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * w),
                         "l"(src + 16 * w)
                         : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * w),
                         "l"(src + 4 * w)
                         : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int WB>
__global__ void __launch_bounds__(32 * DP_WARPS)
    depacketise_warp_kernel(DepackGeom g, int maxn, int turns, const unsigned char *__restrict__ pkts,
                            int npackets, void *__restrict__ out, unsigned int *__restrict__ seen,
                            mdt_depack_stats *__restrict__ stats)
{
    __shared__ __align__(16) unsigned char sbuf[DP_WARPS][2][DP_BUF];
    __shared__ unsigned int s_cnt[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 4) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const int per = g.bits == 32 ? 8 : 2;  // bytes of a sample
    const long long wlen = (long long)g.nspectra * g.nch;
    // the first run of a packet, sized for the widest SNAP (inside the packet
    // whatever its SNAP is: packet_bytes holds the widest payload)
    const int lead = (min(32, g.sper) * maxn * per + WB - 1) / WB;
    const long pk0 = (long)blockIdx.x * (turns * DP_WARPS) + warp;
    const unsigned char *pay = pkts + 4 * g.hdr_words;
    if (pk0 < npackets) copy_words<WB>(sbuf[warp][0], pay + pk0 * g.pkt_bytes, lead, lane);
    for (int m = 0; m < turns; m++) {
        const long pk = pk0 + (long)m * DP_WARPS;
        if (pk >= npackets) break;
        unsigned char *buf = sbuf[warp][m & 1];
        // the packet after this one (an empty group when there is none)
        const bool more = m + 1 < turns && pk + DP_WARPS < npackets;
        copy_words<WB>(sbuf[warp][(m + 1) & 1], pay + (pk + DP_WARPS) * g.pkt_bytes,
                       more ? lead : 0, lane);
        const uint32_t *hdr = (const uint32_t *)(pkts + pk * g.pkt_bytes);
        const uint32_t station = __ldg(hdr), snap = __ldg(hdr + 1), counter = __ldg(hdr + 2);
        const long long slot = (long long)counter - g.c0;
        // this packet's copy has landed, also where the packet is then rejected: the
        // next iteration issues a copy into the same buffer, and copies of different
        // groups may land in any order
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (snap >= (uint32_t)g.nsnap || station >= (uint32_t)g.nstation ||
            (long)station * g.ips + g.snap_off[snap] + g.snap_n[snap] > g.ne) {
            if (lane == 0) atomicAdd(&s_cnt[2], 1u);
            continue;
        }
        if (slot < 0 || slot >= g.nslots) {
            if (lane == 0) atomicAdd(&s_cnt[1], 1u);
            continue;
        }
        if (lane == 0) {
            const unsigned int prev =
                atomicAdd(&seen[((long)station * g.nsnap + snap) * g.nslots + slot], 1u);
            if (prev) atomicAdd(&s_cnt[3], 1u);
            atomicAdd(&s_cnt[0], 1u);
        }
        const int nin = g.snap_n[snap];
        const long elem0 = (long)station * g.ips + g.snap_off[snap];
        const long long first = (long long)counter * g.sper - g.sample0;
        for (int i0 = 0; i0 < g.sper; i0 += 32) {
            // samples i0 .. i0 + 31 of every input are contiguous; a run starts
            // on a multiple of 32 samples, so on a 16-byte boundary of the payload
            const int ns = min(32, g.sper - i0);
            if (i0) {
                copy_words<WB>(buf, pay + pk * g.pkt_bytes + (long)i0 * nin * per,
                               (ns * nin * per + WB - 1) / WB, lane);
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncwarp();
            const long long s = first + i0 + lane;
            if (lane < ns && s >= 0 && s < wlen) {
                // 32-bit division wherever the window's sample index fits
                const long spec = wlen >> 32 ? (long)(s / g.nch)
                                             : (long)((unsigned)s / (unsigned)g.nch);
                const long o = (spec * g.ne + elem0) * g.nch + (long)(s - (long long)spec * g.nch);
                if (g.bits == 32) {
                    const uint2 *v = (const uint2 *)buf + lane * nin;
                    float2 *dst = (float2 *)out + o;
#pragma unroll 2
                    for (int j = 0; j < nin; j++, dst += g.nch)
                        *dst = make_float2(fixed19_to_float(v[j].x), fixed19_to_float(v[j].y));
                } else {
                    const char2 *v = (const char2 *)buf + lane * nin;
                    char2 *dst = (char2 *)out + o;
#pragma unroll 2
                    for (int j = 0; j < nin; j++, dst += g.nch) *dst = v[j];
                }
            }
            __syncwarp();
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 4 && s_cnt[threadIdx.x]) {
        unsigned long long *c = threadIdx.x == 0   ? &stats->accepted
                                : threadIdx.x == 1 ? &stats->outside
                                : threadIdx.x == 2 ? &stats->bad
                                                   : &stats->duplicate;
        atomicAdd(c, (unsigned long long)s_cnt[threadIdx.x]);
    }
}

// One thread per (station, SNAP, slot) looks for slots that never arrived and
// clears the arrival counts; its warp then zero-fills the missing slots it
// found one after another, all lanes on one slot (lanes along the samples):
// one slot per thread left the kernel waiting for its slowest thread (15 us
// against 3.4 with 0.1 % of the packets lost).
__global__ void depack_finish_kernel(DepackGeom g, void *__restrict__ out,
                                     unsigned int *__restrict__ seen,
                                     mdt_depack_stats *__restrict__ stats)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long ngrp = (long)g.nstation * g.nsnap;
    bool miss = false;
    if (t < ngrp * g.nslots) {
        const long grp = t / g.nslots;
        const int station = (int)(grp / g.nsnap), snap = (int)(grp - (long)station * g.nsnap);
        const unsigned int n = seen[t];
        if (n) seen[t] = 0;
        miss = !n && g.snap_n[snap] > 0 &&
               (long)station * g.ips + g.snap_off[snap] + g.snap_n[snap] <= g.ne;
    }
    unsigned int todo = __ballot_sync(0xffffffffu, miss);
    if (!todo) return;
    const int lane = threadIdx.x & 31;
    if (lane == 0) atomicAdd(&stats->missing, (unsigned long long)__popc(todo));
    const long long wlen = (long long)g.nspectra * g.nch;
    for (; todo; todo &= todo - 1) {
        const long tm = t - lane + (__ffs(todo) - 1);
        const long grp = tm / g.nslots, slot = tm - grp * g.nslots;
        const int station = (int)(grp / g.nsnap), snap = (int)(grp - (long)station * g.nsnap);
        const long elem0 = (long)station * g.ips + g.snap_off[snap];
        const int nin = g.snap_n[snap];
        const long long first = (g.c0 + slot) * g.sper - g.sample0;
        for (int i = lane; i < g.sper; i += 32) {
            const long long s = first + i;
            if (s < 0 || s >= wlen) continue;
            const long long spec = s / g.nch;
            const long o = ((long)spec * g.ne + elem0) * g.nch + (long)(s - spec * g.nch);
            for (int j = 0; j < nin; j++) {
                if (g.bits == 32)
                    ((float2 *)out)[o + (long)j * g.nch] = make_float2(0.f, 0.f);
                else
                    ((char2 *)out)[o + (long)j * g.nch] = make_char2(0, 0);
            }
        }
    }
}

static mdt_status make_geom(const mdt_packet_format *f, int ne, int nch, long long sample0,
                            int nspectra, DepackGeom *g)
{
    if (!f) return invalid("depacketise: null packet format");
    if (f->words_header < 3 || f->sper_element < 1 || f->inputs_per_station < 1 ||
        f->nsnap < 1 || f->nsnap > MDT_MAX_SNAPS || (f->sample_bits != 32 && f->sample_bits != 8))
        return invalid("depacketise: bad packet format");
    if (ne < 1 || nch < 1 || nspectra < 1 || sample0 < 0 || sample0 % nch)
        return invalid("depacketise: bad window (sample0 must be a multiple of Nch)");
    g->hdr_words = f->words_header;
    g->sper = f->sper_element;
    g->ips = f->inputs_per_station;
    g->nsnap = f->nsnap;
    g->bits = f->sample_bits;
    int off = 0, maxn = 0;
    for (int k = 0; k < f->nsnap; k++) {
        if (f->inputs_per_snap[k] < 0) return invalid("depacketise: negative inputs_per_snap");
        g->snap_off[k] = off;
        g->snap_n[k] = f->inputs_per_snap[k];
        off += f->inputs_per_snap[k];
        maxn = std::max(maxn, f->inputs_per_snap[k]);
    }
    g->snap_off[f->nsnap] = off;
    if (off > f->inputs_per_station) return invalid("depacketise: SNAP inputs exceed a station");
    const long need = 4L * f->words_header +
                      (long)f->sper_element * maxn * (f->sample_bits == 32 ? 8 : 2);
    g->pkt_bytes = f->packet_bytes;
    if (g->pkt_bytes < need || g->pkt_bytes % 4)
        return invalid("depacketise: packet_bytes smaller than the largest packet or not a "
                       "multiple of 4");
    g->ne = ne;
    g->nch = nch;
    g->nspectra = nspectra;
    g->sample0 = sample0;
    g->nstation = (int)cdiv(ne, f->inputs_per_station);
    const long long end = sample0 + (long long)nspectra * nch;
    g->c0 = sample0 / f->sper_element;
    g->nslots = (long)((end + f->sper_element - 1) / f->sper_element - g->c0);
    return MDT_SUCCESS;
}

}  // namespace mdt

extern "C" {

MDT_API mdt_status mdt_depacketise_seen_words(const mdt_packet_format *fmt, int ne, int nch,
                                              long long sample0, int nspectra, size_t *words)
{
    mdt::DepackGeom g;
    mdt_status st = mdt::make_geom(fmt, ne, nch, sample0, nspectra, &g);
    if (st != MDT_SUCCESS) return st;
    if (!words) return mdt::invalid("depacketise_seen_words: null output");
    *words = (size_t)g.nstation * g.nsnap * g.nslots;
    return MDT_SUCCESS;
}

MDT_API mdt_status mdt_depacketise(const mdt_packet_format *fmt, const void *packets, int npackets,
                                   int ne, int nch, long long sample0, int nspectra, void *out,
                                   unsigned int *seen, mdt_depack_stats *stats,
                                   cudaStream_t stream)
{
    mdt::DepackGeom g;
    mdt_status st = mdt::make_geom(fmt, ne, nch, sample0, nspectra, &g);
    if (st != MDT_SUCCESS) return st;
    if (npackets < 0 || (npackets && !packets) || !out || !seen || !stats)
        return mdt::invalid("depacketise: bad buffers");
    if (npackets == 0) return MDT_SUCCESS;
    if (((uintptr_t)packets & 3) || ((uintptr_t)out & (fmt->sample_bits == 32 ? 7 : 1)))
        return mdt::invalid("depacketise: misaligned packets or output");
    // A warp per packet while 32 samples of the widest SNAP fit its staging
    // buffer (16 inputs of int32, 64 of int8); wider SNAPs take a block per packet.
    int maxn = 0;
    for (int k = 0; k < fmt->nsnap; k++) maxn = std::max(maxn, fmt->inputs_per_snap[k]);
    if ((long)maxn * 32 * (fmt->sample_bits == 32 ? 8 : 2) <= mdt::DP_BUF) {
        // As many packets per warp, up to eight, as fill the GPU with six blocks an SM: a
        // warp takes its packets one after the other (588 packets of int32, eight each: 13.3
        // us, one each 3.3; 9364, eight 14.1, two 10.3).
        const int turns = (int)std::max<long>(1, std::min<long>(8, npackets / (6L * mdt::DP_WARPS * mdt::sm_count())));
        const unsigned blocks = (unsigned)mdt::cdiv(npackets, mdt::DP_WARPS * turns);
        // 16-byte reads where every payload starts on a 16-byte boundary and the
        // packet stride keeps the last read inside the packet
        const bool wide = (((uintptr_t)packets | (uintptr_t)fmt->packet_bytes |
                            (uintptr_t)(4L * fmt->words_header)) & 15) == 0;
        if (wide)
            mdt::depacketise_warp_kernel<16><<<blocks, 32 * mdt::DP_WARPS, 0, stream>>>(
                g, maxn, turns, (const unsigned char *)packets, npackets, out, seen, stats);
        else
            mdt::depacketise_warp_kernel<4><<<blocks, 32 * mdt::DP_WARPS, 0, stream>>>(
                g, maxn, turns, (const unsigned char *)packets, npackets, out, seen, stats);
        return mdt::launch_status("depacketise_warp_kernel");
    }
    mdt::depacketise_kernel<<<(unsigned)npackets, 128, 0, stream>>>(
        g, (const unsigned char *)packets, out, seen, stats);
    return mdt::launch_status("depacketise_kernel");
}

MDT_API mdt_status mdt_depacketise_finish(const mdt_packet_format *fmt, int ne, int nch,
                                          long long sample0, int nspectra, void *out,
                                          unsigned int *seen, mdt_depack_stats *stats,
                                          cudaStream_t stream)
{
    mdt::DepackGeom g;
    mdt_status st = mdt::make_geom(fmt, ne, nch, sample0, nspectra, &g);
    if (st != MDT_SUCCESS) return st;
    if (!out || !seen || !stats) return mdt::invalid("depacketise_finish: bad buffers");
    const long n = (long)g.nstation * g.nsnap * g.nslots;
    mdt::depack_finish_kernel<<<(unsigned)mdt::cdiv(n, 128), 128, 0, stream>>>(g, out, seen,
                                                                              stats);
    return mdt::launch_status("depack_finish_kernel");
}

}  // extern "C"
