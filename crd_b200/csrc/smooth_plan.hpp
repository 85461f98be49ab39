// Host side of the run-time-schedule lines (smooth_line.cuh): the radix schedule of a 7-smooth length and the index
// constants of its stages. Plain integer arithmetic.

#pragma once

#include <vector>

namespace crdfft
{

struct PassDesc;
struct SmoothSched;
namespace smooth
{
struct Tile;
}

// The radices of a 7-smooth n in execution order; false when n has another prime factor or needs too many stages.
// arith: the schedule's cost by the rule that picked it (instructions a point).
bool smooth_radices(long long n, std::vector<int>& out, double* arith = nullptr);
// The stages' index constants; tw: the stage-ordered twiddle table of these radices (device memory).
bool smooth_sched(int n, const int* radix, int nstages, const void* tw, SmoothSched* s);
// Whether a schedule holds a radix above 16 (the wide build of the kernels).
bool smooth_wide(const int* radix, int nstages);

// The schedule and the tile of a line pass at `lpc` lines a CTA, for kernels that run its tiles themselves.
bool smooth_tile(const PassDesc& d, int lpc, SmoothSched* s, smooth::Tile* t);

} // namespace crdfft
