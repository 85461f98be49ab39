// The line-FFT pass of every 7-smooth length without a compile-time schedule (240, 1000, 3000, 6144 ..): the tile code
// of smooth_line.cuh between the pass's global line maps, with the conjugations, scale and four-step twiddle of the
// pass in the first and last stage's accesses.

#include "index.cuh"
#include "kernels.hpp"
#include "pass_desc.hpp"
#include "smem_limit.hpp"
#include "smooth_line.cuh"
#include "smooth_plan.hpp"

#include <algorithm>
#include <atomic>
#include <map>

namespace crdfft
{

namespace
{

// Arithmetic of one radix's butterfly a point (FP32 instructions), and what a stage costs besides (shared-memory
// round trip, addresses, twiddle).
struct RadixCost
{
    int R;
    double per_point;
};
constexpr RadixCost kRadices[] = {{2, 2.0},   {3, 4.7},   {4, 4.0},   {5, 7.6},   {6, 6.7},   {7, 9.4},
                                  {8, 6.5},   {9, 12.0},  {10, 9.6},  {12, 8.7},  {14, 11.4}, {15, 12.3},
                                  {16, 10.5}, {18, 14.0}, {20, 11.6}, {21, 14.1}, {24, 11.7}, {25, 19.0}};
constexpr double kStageCost = 14.0;     // a point: shared-memory round trip, twiddle
constexpr double kButterflyCost = 25.0; // a butterfly: its indices and addresses

struct Best
{
    double cost = 1e30;
    int R = 0;
};

// Cheapest product of radices up to `top` for n.
double cheapest(long long n, int top, std::map<long long, Best>& memo)
{
    if (n == 1)
        return 0.0;
    auto it = memo.find(n);
    if (it != memo.end())
        return it->second.cost;
    Best b;
    for (const RadixCost& r : kRadices)
        if (r.R <= top && n % r.R == 0)
        {
            const double c = cheapest(n / r.R, top, memo) + kStageCost + kButterflyCost / r.R + r.per_point;
            if (c < b.cost)
                b = Best{c, r.R};
        }
    memo[n] = b;
    return b.cost;
}

} // namespace

bool smooth_wide(const int* radix, int nstages)
{
    for (int i = 0; i < nstages; ++i)
        if (radix[i] > 16)
            return true;
    return false;
}

bool smooth_radices(long long n, std::vector<int>& out, double* arith, double wide_cost)
{
    struct Schedule
    {
        std::vector<int> radices;
        double cost = 0.0;
    };
    thread_local std::map<std::pair<long long, double>, Schedule> memo; // a few hundred line lengths
    out.clear();
    if (n < 1)
        return false;
    auto it = memo.find({n, wide_cost});
    if (it == memo.end())
    {
        Schedule s;
        std::map<long long, Best> narrow, wide;
        const double cn = cheapest(n, 16, narrow), cw = wide_cost * cheapest(n, 25, wide);
        std::map<long long, Best>& pick = cw < cn ? wide : narrow;
        s.cost = std::min(cn, cw);
        if (n == 1)
            s.radices.push_back(1);
        for (long long m = n; m > 1;)
        {
            const Best& b = pick[m];
            if (b.R == 0)
                return false;
            s.radices.push_back(b.R);
            m /= b.R;
        }
        // Largest first (most loads in flight a thread, and the last stage's runs n / Rs in global memory are long),
        // the smallest in the middle: 60 as 12.5 51.6 us against 4.15 62.6, 5000 as 25.10.20 83.2 against 10.20.25
        // 89.1.
        std::sort(s.radices.rbegin(), s.radices.rend());
        if (s.radices.size() > 2)
            std::swap(s.radices[1], s.radices.back());
        if (n > 65535)
        {
            out = s.radices;
            if (arith != nullptr)
                *arith = s.cost;
            return out.size() <= static_cast<size_t>(kSmoothStages);
        }
        it = memo.emplace(std::make_pair(n, wide_cost), s).first;
    }
    out = it->second.radices;
    if (arith != nullptr)
        *arith = it->second.cost;
    return out.size() <= static_cast<size_t>(kSmoothStages);
}

bool smooth_sched(int n, const int* radix, int nstages, const void* tw, SmoothSched* out)
{
    if (nstages < 1 || nstages > kSmoothStages || n > 65535)
        return false;
    SmoothSched s{};
    s.n = n;
    s.ns = nstages;
    s.tw = tw;
    auto magic = [](int d) { return d <= 1 ? 0u : 0xFFFFFFFFu / static_cast<unsigned>(d) + 1u; };
    const int R1 = radix[0];
    const int n1 = n / R1;
    s.p1 = nstages > 1 ? n1 | 1 : n1;
    s.m1 = magic(R1);
    int L = 1, off = 0;
    for (int i = 0; i < nstages; ++i)
    {
        SmoothStage& t = s.st[i];
        t.R = radix[i];
        t.L = L;
        t.N = n / t.R;
        t.ni = n / (L * t.R);
        t.C = i == 0 ? t.N : t.N / R1;
        t.tw = off;
        t.mN = magic(t.N);
        t.mC = magic(t.C);
        t.mni = magic(t.ni);
        if (L > 1)
            off += (t.R - 1) * L;
        L *= t.R;
    }
    if (L != n)
        return false;
    *out = s;
    return true;
}

namespace smooth
{
namespace
{

template <int EPI, bool WIDE>
__global__ void __maxnreg__(WIDE ? 96 : EPI == 2 ? 72 : 64)
    smooth_line_kernel(const PassDesc d, const SmoothSched s, const Tile t, const float2* gin, float2* gout)
{
    pass_tile<EPI, WIDE>(d, s, t, gin, gout, blockIdx.x, d.lines);
}

int log2_exact(int v)
{
    int l = 0;
    while ((1 << l) < v)
        ++l;
    return (1 << l) == v ? l : -1;
}

// The tile of a pass at `lpc` lines a CTA: layout and thread maps.
Tile tile_of(const PassDesc& d, const SmoothSched& s, int lpc)
{
    Tile t{};
    t.lpc = lpc;
    const int places = s.st[0].R * s.p1;
    const int lg = log2_exact(lpc);
    const bool in_across = lg > 0 && d.in.estride != 1 && d.in.ldist == 1 && d.lines_per_group > 1;
    const bool out_across = lg > 0 && d.out.estride != 1 && d.out.ldist == 1 && d.lines_per_group > 1;
    // Lines interleaved when the first stage runs across them (8 bytes apart, as they arrive); else one line after
    // another, an odd number of places apart, so that a last stage across the lines meets no bank twice.
    t.sp = in_across ? lpc : 1;
    t.sl = in_across ? 1 : places | 1;
    t.first = in_across ? lg : -1;
    t.mid = in_across ? lg : -1;
    t.last = out_across ? lg : -1;
    t.flat = d.lines_per_group >= lpc ? 1 : 0;
    return t;
}

int tile_bytes(const SmoothSched& s, int lpc) { return s.ns == 1 ? 0 : lpc * (s.st[0].R * s.p1 | 1) * 8; }

} // namespace
} // namespace smooth

bool smooth_line_supported(const PassDesc& d)
{
    SmoothSched s;
    return smooth_sched(d.n, d.radix, d.nstages, d.tw, &s);
}

int smooth_line_smem(const PassDesc& d, int lpc)
{
    SmoothSched s;
    return smooth_sched(d.n, d.radix, d.nstages, d.tw, &s) ? smooth::tile_bytes(s, lpc) : 0;
}

bool smooth_tile(const PassDesc& d, int lpc, SmoothSched* s, smooth::Tile* t)
{
    if (!smooth_sched(d.n, d.radix, d.nstages, d.tw, s) || lpc < 1 || static_cast<long long>(lpc) * d.n > 65535)
        return false;
    *t = smooth::tile_of(d, *s, lpc);
    return true;
}

// Threads of a tile: as many as the registers allow the CTAs an SM holds, whether shared memory or the grid sets their
// number, 128 to 512 and no more than the tile has butterflies for (1000-point lines along: 128 threads 68.8 us, 320
// 71.5; eight interleaved, three CTAs an SM: 320 threads 89.1 us, 416 93.2, two CTAs).
int smooth_threads(const SmoothSched& s, int lpc, int smem_bytes, int regs, long long grid)
{
    const long long fill = (grid + 147) / 148; // CTAs an SM that the grid has
    const int ctas = static_cast<int>(std::clamp(227LL * 1024 / (smem_bytes + 1024), 1LL, std::max(1LL, fill)));
    int most = 0;
    for (int i = 0; i < s.ns; ++i)
        most = std::max(most, (lpc * s.st[i].N + 31) / 32 * 32);
    return std::min(std::clamp(65536 / regs / ctas / 32 * 32, 128, 512), most);
}

// Lines a CTA: along the lines, tiles of about 2200 points (many CTAs an SM hide each other's phases: 1000-point lines
// 2 a CTA 68.8 us, 8 74.8); across them, runs of 64 bytes or more as long as a tile fits (2400 points 8 a CTA 110 us, 4
// 114; 360 points 32 a CTA 66.3, 8 71.5). A pass of fewer tiles than SMs takes shorter ones, one an SM: its time is then
// that of one tile, whose threads do less each (3000 points x 33: 8 a CTA 17.9 us, one 8.3; x 256: 17.0, two 10.2).
int smooth_line_lpc(const PassDesc& d, PassMap map)
{
    const bool across = map == PassMap::Col || (d.out.estride != 1 && d.out.ldist == 1 && d.lines_per_group > 1);
    int lpc = 1;
    if (across)
    {
        lpc = d.n <= 400 ? 32 : d.n <= 560 ? 16 : d.n <= 3000 ? 8 : d.n <= 6000 ? 4 : 2;
        while (lpc < 128 && lpc * d.n < 1500)
            lpc *= 2;
        while (lpc > 1 && d.lines <= 148LL * (lpc / 2))
            lpc /= 2;
    }
    else
        lpc = std::max(1, 2200 / d.n);
    return std::min(lpc, 256);
}

cudaError_t launch_smooth_line(const PassDesc& d, int lpc, const void* in, void* out, cudaStream_t stream)
{
    SmoothSched s;
    if (!smooth_sched(d.n, d.radix, d.nstages, d.tw, &s) || lpc < 1 || static_cast<long long>(lpc) * d.n > 65535)
        return cudaErrorInvalidConfiguration;
    const long long groups = (d.lines + lpc - 1) / lpc;
    if (groups <= 0)
        return cudaSuccess;
    const int smem = smooth::tile_bytes(s, lpc);
    if (groups > 0x7fffffffLL || smem > 227 * 1024)
        return cudaErrorInvalidConfiguration;
    const int epi = d.ftw_M != 0 ? 2 : (d.conj_in != 0 || d.conj_out != 0 || d.scale != 1.0f) ? 1 : 0;
    const bool wide = smooth_wide(d.radix, d.nstages);
    const int regs = wide ? 96 : epi == 2 ? 72 : 64; // the kernels' __maxnreg__
    using Fn = void (*)(const PassDesc, const SmoothSched, const smooth::Tile, const float2*, float2*);
    const Fn fns[2][3] = {{smooth::smooth_line_kernel<0, false>, smooth::smooth_line_kernel<1, false>,
                           smooth::smooth_line_kernel<2, false>},
                          {smooth::smooth_line_kernel<0, true>, smooth::smooth_line_kernel<1, true>,
                           smooth::smooth_line_kernel<2, true>}};
    const Fn fn = fns[wide ? 1 : 0][epi];
    if (const cudaError_t e = allow_smem(fn, smem); e != cudaSuccess)
        return e;
    fn<<<static_cast<unsigned>(groups), smooth_threads(s, lpc, smem, regs, groups), smem, stream>>>(
        d, s, smooth::tile_of(d, s, lpc), static_cast<const float2*>(in), static_cast<float2*>(out));
    return cudaGetLastError();
}

} // namespace crdfft
