// Device work list of the uneven-batch kernel (uneven.cu), built by the planner (plan.cpp).

#pragma once

#include "pass_desc.hpp"

#include <cuda_runtime.h>

namespace crdfft
{

struct SmoothSched;

enum UnevenKind : int
{
    kUnevenSmall = 0, // up to `lines` whole transforms of one length, at offsets line_off[line_table + a]
    kUnevenCol = 1,   // columns q0 .. q0+lines-1 of one long transform -> its workspace region (+ four-step twiddle)
    kUnevenRow = 2,   // rows of one long transform's workspace region -> the output (waits for its COL items)
};

struct UnevenItem
{
    int kind;
    int sched;       // index into the schedule table (the item's line length)
    int lines;       // lines of the item
    int lpc;         // lines of its tile (a power of two for COL and ROW)
    int sl, sp;      // the tile's places (smooth_line.cuh)
    int first, last; // Lanes::across of the stages (the middle ones run as the first)
    int line_table;  // SMALL: first index into line_off; else -1
    int transform;   // COL/ROW: index of the long transform (completion counter)
    int need;        // ROW: COL items of that transform
    int q0;          // COL: first column (four-step twiddle row)
    int pad;
    const void* ftw_hi; // COL: W_n^{16 (q>>4) k1} at hi[(q>>4) n1 + k1]; else null
    const void* ftw_lo; //      W_n^{(q&15) k1} at lo[16 k1 + (q&15)]
    long long in_base, in_ldist, in_estride;
    long long out_base, out_ldist, out_estride;
};

struct UnevenDesc
{
    const UnevenItem* items;
    const SmoothSched* scheds; // one per line length
    const long long* line_off;
    int* started;   // CTAs started, and behind it done (both zeroed before a launch with long transforms)
    int* done;      // COL items finished, per long transform
    int* err;
    int nitems;
    int ntransforms;
    int spin_limit;
    int conj;       // inverse: conjugate in and out
    float scale;
};

constexpr int kUnevenTile = 4096; // the longest line of an item, and the points of a tile of several
constexpr int kUnevenLines = 64; // lines of an item
// CTAs the device holds at once at this much shared memory, or 0 on an error.
int uneven_resident(int smem_bytes);
cudaError_t launch_uneven(const UnevenDesc& u, int smem_bytes, const void* in, void* out, void* scratch,
                          cudaStream_t stream);

} // namespace crdfft
