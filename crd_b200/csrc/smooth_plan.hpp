// Host side of the run-time-schedule lines (smooth_line.cuh): the radix schedule of a 7-smooth length and the index
// constants of its stages. Plain integer arithmetic.

#pragma once

#include <vector>

namespace crdfft
{

struct SmoothSched;

// The radices of a 7-smooth n in execution order; false when n has another prime factor or needs too many stages.
bool smooth_radices(long long n, std::vector<int>& out);
// The stages' index constants; tw: the stage-ordered twiddle table of these radices (device memory).
bool smooth_sched(int n, const int* radix, int nstages, const void* tw, SmoothSched* s);
// Whether a schedule holds a radix above 16 (the wide build of the kernels).
bool smooth_wide(const int* radix, int nstages);

} // namespace crdfft
