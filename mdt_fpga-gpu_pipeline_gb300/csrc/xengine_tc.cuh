// xengine_tc.cuh -- host-visible pieces of the tensor-core X-engine shared
// with the batch driver (batch.cu): tile and work descriptors.
#pragma once
#include "mdt_common.cuh"

namespace mdt {

struct TcTile {
    int16_t r0, q0, n, a_sep;  // row-tile start, column-chunk start, chunk width, A loaded apart
};

// One job of a batched X-engine launch.
struct XJob {
    const uint8_t *X;  // X16 operand of the job
    long chunk_bytes;  // stride between 32-spectrum chunks: Nch * NEp * 128
    long chan_bytes;   // stride between channels: NEp * 128
    int ne, nep, nkc;
    float alpha;       // 1 / (Nsp * scale^2)
    float2 *V;         // visibilities [nch][ne*ne]
};

// One work entry of a batched X-engine launch: a tile of one channel of one job.
struct XWork {
    int job, ch;
    int grouped;  // the tile holds the rows of several channels from ch on (tc_group)
    TcTile tile;
};

constexpr int TCB_MAXW = 128;  // widest column chunk of the batched X-engine

// Lower-triangle tiles (row tiles of 128, column chunks of <= maxw) for NE
// elements padded to nep rows; returns the count or -1 if more than 160.
int make_tiles(int ne, int nep, int maxw, TcTile *tiles);
// Channels whose rows one tile takes together (1, 2, 4 or 8), by the padded rows and
// the blocks or work entries that there are at one channel each and an SM holds.
int tc_group(int nep, long blocks, int per_sm);
int x16_padded_rows(int ne);
int x16_chunks(int nsp);
mdt_status xengine_tc_batched(const XJob *jobs, const XWork *work, int nwork, int *err,
                              cudaStream_t stream);

}  // namespace mdt
