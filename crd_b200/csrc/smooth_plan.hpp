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
// arith: the schedule's cost by the rule that picked it (instructions a point). wide_cost: what a radix above 16 costs
// the whole line, by the resident warps its registers leave (720 points 8.10.9 67.6 us a 256 MiB batch, 240 16.15 49.5
// against 12.20 59.2, but 3000 12.10.25 78.8 against 10.10.6.5 97.0, a stage more).
constexpr double kSmoothWideCost = 1.12;
bool smooth_radices(long long n, std::vector<int>& out, double* arith = nullptr, double wide_cost = kSmoothWideCost);
// The stages' index constants; tw: the stage-ordered twiddle table of these radices (device memory).
bool smooth_sched(int n, const int* radix, int nstages, const void* tw, SmoothSched* s);
// Whether a schedule holds a radix above 16 (the wide build of the kernels).
bool smooth_wide(const int* radix, int nstages);

// Threads of a CTA of `lpc` lines with this much shared memory and registers a thread, in a launch of `grid` CTAs.
int smooth_threads(const SmoothSched& s, int lpc, int smem_bytes, int regs, long long grid);
// The schedule and the tile of a line pass at `lpc` lines a CTA, for kernels that run its tiles themselves.
bool smooth_tile(const PassDesc& d, int lpc, SmoothSched* s, smooth::Tile* t);

} // namespace crdfft
