#pragma once

// Lines of any 7-smooth length in shared memory, the radix schedule read at run time: the tile code of the kernels
// that have no compile-time schedule for their length (smooth_line.cu).
//
// The transform is decimation in time, in place. An element of a line is a mixed-radix number of its digits
// j1 j2 .. js (j1 most significant, radices R1 .. Rs); stage i replaces digit j_i by the frequency digit k_i:
//     v_r = y[.. r ..] * W_{L R}^{r k},  k = k1 + R1 k2 + ..  over the digits done so far (L = R1 .. R_{i-1})
//     y[.. k_i ..] = DFT_R(v)
// so a butterfly writes the places it read. What that buys over the self-sorting form: one buffer a line and no
// barrier between a stage's reads and its writes, so a thread takes its butterflies one after another and holds one
// of them in registers; one barrier a stage; and the same twiddle table (its k index is the digits done so far). The
// reordering costs nothing: stage 1 reads elements b + r n/R1 from global memory and the last stage writes elements
// b + r n/Rs to it, so those are the only global accesses and an s-stage line makes s - 1 round trips through shared
// memory. Threads run along a line's elements or across the lines of the tile, separately for the first and the last
// stage, whichever is unit-stride in global memory: a transposed store needs no extra round trip.
//
// Places: element e of line l is at l * sl + (e + (e / n1) pad) * sp, n1 = n / R1: the R1 blocks of the last stage's
// strided reads start on odd multiples of the bank width.

#include "codelets.cuh"
#include "index.cuh"
#include "pass_desc.hpp"

#include <cuda_runtime.h>

#include <cstdint>

namespace crdfft
{

constexpr int kSmoothStages = 8;

// One stage of a schedule, with the multiply-high constants ceil(2^32 / d) of the divisions its index needs (exact for
// dividends below 2^16 and divisors below 2^16).
struct SmoothStage
{
    int R;
    int N;        // butterflies a line: n / R
    int L;        // product of the radices before
    int ni;       // places between a butterfly's elements: n / (L R)
    int C;        // butterflies a block of n1 places (middle stages): N / R1
    int tw;       // the stage's twiddles in the table
    unsigned mN;  // / N
    unsigned mC;  // / C
    unsigned mni; // / ni
};

struct SmoothSched
{
    int n;
    int ns;
    int p1;      // places a block of n1 = n / R1 elements takes (odd for two stages or more)
    unsigned m1; // / R1
    const void* tw; // float2, stage-ordered: W_{LR}^{rk} at tw + (r - 1) L + k
    SmoothStage st[kSmoothStages];
};

namespace smooth
{

// A tile of a line pass: lines a CTA, the places' strides, the thread map of each stage.
struct Tile
{
    int lpc;
    int sl, sp;
    int first, mid, last; // Lanes::across of each stage
    int flat;             // every tile's lines lie in one address group, or wrap into the next one at most once
};

namespace
{

__device__ __forceinline__ int mdiv(int a, unsigned m) { return m == 0u ? a : static_cast<int>(__umulhi(static_cast<unsigned>(a), m)); }

// How a stage's (line, butterfly) pairs go over the threads: consecutive threads along a line's butterflies, or across
// the lines of the tile (a power of two of them).
struct Lanes
{
    int across; // log2 of the tile's lines, or -1: along the line
};

__device__ __forceinline__ void place(const Lanes& ln, int idx, const SmoothStage& s, int& l, int& b)
{
    if (ln.across >= 0)
    {
        l = idx & ((1 << ln.across) - 1);
        b = idx >> ln.across;
    }
    else
    {
        l = mdiv(idx, s.mN);
        b = idx - l * s.N;
    }
}

// A middle stage's butterfly b: block k1 first, then the digits k2 .. k_{i-1} (most significant first), then the place
// j within the block that the stage splits. Returns the first element's place; k: the twiddle column.
__device__ __forceinline__ int mid_place(const SmoothSched& s, int i, int b, int& k)
{
    const SmoothStage& t = s.st[i];
    const int k1 = mdiv(b, t.mC);
    const int rest = b - k1 * t.C;
    if (i == 1)
    {
        k = k1;
        return k1 * s.p1 + rest;
    }
    const int q = mdiv(rest, t.mni);
    const int j = rest - q * t.ni;
    if (i == 2)
        k = k1 + s.st[0].R * q;
    else
    {
        // q = (k2 R3 + k3) R4 + ..: reverse its digits
        int qq = q, w = t.L, acc = 0;
        for (int a = i - 1; a >= 1; --a)
        {
            const int R = s.st[a].R;
            w /= R;
            const int d = qq % R;
            qq /= R;
            acc += d * w;
        }
        k = k1 + acc;
    }
    return k1 * s.p1 + q * (t.ni * t.R) + j;
}

// The last stage's butterfly b = k1 + R1 (k2 + R2 (..)): the place of its first element.
__device__ __forceinline__ int last_place(const SmoothSched& s, int b)
{
    if (s.ns == 2)
        return b * s.p1;
    int q = mdiv(b, s.m1);
    int p = (b - q * s.st[0].R) * s.p1;
    if (s.ns == 3)
        return p + q * s.st[1].ni;
    for (int a = 1; a < s.ns - 1; ++a)
    {
        const int R = s.st[a].R;
        const int t = q / R;
        p += (q - t * R) * s.st[a].ni;
        q = t;
    }
    return p;
}

template <int R> __device__ __forceinline__ void twiddle(float2* v, const float2* tw, int L, int k)
{
#pragma unroll
    for (int r = 1; r < R; ++r)
        v[r] = cmul(v[r], __ldg(tw + (r - 1) * L + k));
}

// Stage 1: global memory (io.get) to shared memory, or to global memory when it is the only stage.
template <int R, class IO>
__device__ __forceinline__ void first_stage(const SmoothSched& s, const Lanes& ln, float2* sm, int sl, int sp, int lpc,
                                            int lines, const IO& io)
{
    const SmoothStage& t = s.st[0];
    const int total = lpc * t.N;
    const int step = s.p1 * sp;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        float2 v[R];
        io.template get<R>(v, l, b, t.N);
        Dft<R>::run(v);
        if (s.ns == 1)
            io.template put<R>(v, l, b, t.N);
        else
        {
            float2* p = sm + l * sl + b * sp;
#pragma unroll
            for (int r = 0; r < R; ++r)
                p[r * step] = v[r];
        }
    }
}

template <int R>
__device__ __forceinline__ void mid_stage(const SmoothSched& s, int i, const Lanes& ln, float2* sm, int sl, int sp,
                                          int lpc, int lines)
{
    const SmoothStage& t = s.st[i];
    const int total = lpc * t.N;
    const int step = t.ni * sp;
    const float2* tw = static_cast<const float2*>(s.tw) + t.tw;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b, k;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        float2* p = sm + l * sl + mid_place(s, i, b, k) * sp;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = p[r * step];
        twiddle<R>(v, tw, t.L, k);
        Dft<R>::run(v);
#pragma unroll
        for (int r = 0; r < R; ++r)
            p[r * step] = v[r];
    }
}

// The last of two or more stages: shared memory to global memory (io.put).
template <int R, class IO>
__device__ __forceinline__ void last_stage(const SmoothSched& s, const Lanes& ln, const float2* sm, int sl, int sp,
                                           int lpc, int lines, const IO& io)
{
    const SmoothStage& t = s.st[s.ns - 1];
    const int total = lpc * t.N;
    const float2* tw = static_cast<const float2*>(s.tw) + t.tw;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        // two stages: the last one's elements are n1 = Rs consecutive places of a block
        const float2* p = sm + l * sl + last_place(s, b) * sp;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = p[r * sp];
        twiddle<R>(v, tw, t.L, b);
        Dft<R>::run(v);
        io.template put<R>(v, l, b, t.N);
    }
}

// Every radix a schedule may hold, WIDE: with those above 16 (their butterflies need more registers than four
// 256-thread CTAs an SM leave).
template <bool WIDE, class F> __device__ __forceinline__ void with_radix(int R, F&& f)
{
    switch (R)
    {
        case 1: f.template operator()<1>(); break; // a line of one element: the copy with its scale
        case 2: f.template operator()<2>(); break;
        case 3: f.template operator()<3>(); break;
        case 4: f.template operator()<4>(); break;
        case 5: f.template operator()<5>(); break;
        case 6: f.template operator()<6>(); break;
        case 7: f.template operator()<7>(); break;
        case 8: f.template operator()<8>(); break;
        case 9: f.template operator()<9>(); break;
        case 10: f.template operator()<10>(); break;
        case 12: f.template operator()<12>(); break;
        case 14: f.template operator()<14>(); break;
        case 15: f.template operator()<15>(); break;
        case 16: f.template operator()<16>(); break;
        default:
            if constexpr (WIDE)
            {
                switch (R)
                {
                    case 18: f.template operator()<18>(); break;
                    case 20: f.template operator()<20>(); break;
                    case 21: f.template operator()<21>(); break;
                    case 24: f.template operator()<24>(); break;
                    default: f.template operator()<25>(); break;
                }
            }
            break;
    }
}

// A whole tile: `lines` of at most lpc lines, every thread of the CTA.
template <bool WIDE, class IO>
__device__ __forceinline__ void run_tile(const SmoothSched& s, float2* sm, int sl, int sp, int lpc, int lines,
                                         const Lanes& first, const Lanes& mid, const Lanes& last, const IO& io)
{
    with_radix<WIDE>(s.st[0].R, [&]<int R>() { first_stage<R>(s, first, sm, sl, sp, lpc, lines, io); });
    for (int i = 1; i < s.ns - 1; ++i)
    {
        __syncthreads();
        with_radix<WIDE>(s.st[i].R, [&]<int R>() { mid_stage<R>(s, i, mid, sm, sl, sp, lpc, lines); });
    }
    if (s.ns > 1)
    {
        __syncthreads();
        with_radix<WIDE>(s.st[s.ns - 1].R, [&]<int R>() { last_stage<R>(s, last, sm, sl, sp, lpc, lines, io); });
    }
}

// ---- convolution: transform, filter, transform back ------------------------------------------------------------------
//
// y = conj(DFT(conj(DFT(x) H))). After the forward stages the frequency digits sit at their places, k1 most
// significant; a stage of the second transform takes digit k_i of place i back to the output digit j_i, last stage
// first, so it reads and writes the places of the forward stage and ends in the order the input had:
//     v = DFT_R(conj(..)), then v_j *= W_{L R}^{j k}  (the forward stage's twiddles, after the butterfly)
// The last forward stage and the first one back share their places: one round trip, the filter applied in registers.

// The last stage of two or more, the filter (io.filter on the frequencies b + r N), and its way back.
template <int R, class IO>
__device__ __forceinline__ void turn_stage(const SmoothSched& s, const Lanes& ln, float2* sm, int sl, int sp, int lpc,
                                           int lines, const IO& io)
{
    const SmoothStage& t = s.st[s.ns - 1];
    const int total = lpc * t.N;
    const float2* tw = static_cast<const float2*>(s.tw) + t.tw;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        float2* p = sm + l * sl + last_place(s, b) * sp;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = p[r * sp];
        twiddle<R>(v, tw, t.L, b);
        Dft<R>::run(v);
        io.template filter<R>(v, l, b, t.N);
        Dft<R>::run(v);
        twiddle<R>(v, tw, t.L, b);
#pragma unroll
        for (int r = 0; r < R; ++r)
            p[r * sp] = v[r];
    }
}

template <int R>
__device__ __forceinline__ void mid_back(const SmoothSched& s, int i, const Lanes& ln, float2* sm, int sl, int sp,
                                         int lpc, int lines)
{
    const SmoothStage& t = s.st[i];
    const int total = lpc * t.N;
    const int step = t.ni * sp;
    const float2* tw = static_cast<const float2*>(s.tw) + t.tw;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b, k;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        float2* p = sm + l * sl + mid_place(s, i, b, k) * sp;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = p[r * step];
        Dft<R>::run(v);
        twiddle<R>(v, tw, t.L, k);
#pragma unroll
        for (int r = 0; r < R; ++r)
            p[r * step] = v[r];
    }
}

template <int R, class IO>
__device__ __forceinline__ void first_back(const SmoothSched& s, const Lanes& ln, const float2* sm, int sl, int sp,
                                           int lpc, int lines, const IO& io)
{
    const SmoothStage& t = s.st[0];
    const int total = lpc * t.N;
    const int step = s.p1 * sp;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x)
    {
        int l, b;
        place(ln, idx, t, l, b);
        if (l >= lines)
            continue;
        const float2* p = sm + l * sl + b * sp;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = p[r * step];
        Dft<R>::run(v);
        io.template put<R>(v, l, b, t.N);
    }
}

// A whole tile of a schedule of two or more stages, every thread of the CTA, threads along the lines.
template <bool WIDE, class IO>
__device__ __forceinline__ void run_conv_tile(const SmoothSched& s, float2* sm, int sl, int sp, int lpc, int lines,
                                              const Lanes& ln, const IO& io)
{
    with_radix<WIDE>(s.st[0].R, [&]<int R>() { first_stage<R>(s, ln, sm, sl, sp, lpc, lines, io); });
    for (int i = 1; i < s.ns - 1; ++i)
    {
        __syncthreads();
        with_radix<WIDE>(s.st[i].R, [&]<int R>() { mid_stage<R>(s, i, ln, sm, sl, sp, lpc, lines); });
    }
    __syncthreads();
    with_radix<WIDE>(s.st[s.ns - 1].R, [&]<int R>() { turn_stage<R>(s, ln, sm, sl, sp, lpc, lines, io); });
    for (int i = s.ns - 2; i >= 1; --i)
    {
        __syncthreads();
        with_radix<WIDE>(s.st[i].R, [&]<int R>() { mid_back<R>(s, i, ln, sm, sl, sp, lpc, lines); });
    }
    __syncthreads();
    with_radix<WIDE>(s.st[0].R, [&]<int R>() { first_back<R>(s, ln, sm, sl, sp, lpc, lines, io); });
}

// ---- a line pass (pass_desc.hpp) as the tile's input and output ---------------------------------------------------

// EPI: 0 plain, 1 conjugations and scale, 2 also the four-step twiddle.
template <int EPI> struct LineIO
{
    const PassDesc& d;
    const float2* gin;
    float2* gout;
    long long line0, g0, q0;
    int flat;
    float in_im, out_re, out_im;

    __device__ __forceinline__ void where(int l, long long& g, long long& q) const
    {
        if (d.lines_per_group == 1)
        {
            g = line0 + l;
            q = 0;
        }
        else if (flat)
        {
            const bool wrap = q0 + l >= d.lines_per_group;
            g = wrap ? g0 + 1 : g0;
            q = wrap ? q0 + l - d.lines_per_group : q0 + l;
        }
        else
        {
            g = idiv(line0 + l, d.lines_per_group);
            q = line0 + l - g * d.lines_per_group;
        }
    }
    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        long long g, q;
        where(l, g, q);
        const float2* p = gin + g * d.in.gdist + q * d.in.ldist + static_cast<long long>(b) * d.in.estride;
        const long long step = static_cast<long long>(N) * d.in.estride;
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            v[r] = __ldcs(p);
            p += step;
        }
        if constexpr (EPI > 0)
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r].y *= in_im;
        }
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        long long g, q;
        where(l, g, q);
        float2* p = gout + g * d.out.gdist + q * d.out.ldist + static_cast<long long>(b) * d.out.estride;
        const long long step = static_cast<long long>(N) * d.out.estride;
        if constexpr (EPI == 2)
        {
            const int qi = static_cast<int>(idiv(q, d.ftw_div));
            const float2* th = static_cast<const float2*>(d.ftw_hi) + (qi >> 4) * d.n + b;
            const float2* tl = static_cast<const float2*>(d.ftw_lo) + b * 16 + (qi & 15);
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r] = cmul(v[r], cmul(__ldg(th + r * N), __ldg(tl + r * N * 16)));
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            if constexpr (EPI > 0)
                v[r] = make_float2(v[r].x * out_re, v[r].y * out_im);
            __stcs(p, v[r]);
            p += step;
        }
    }
};

// Tile `blk` of a pass of `nlines` lines: lines [blk * lpc, blk * lpc + lpc).
template <int EPI, bool WIDE>
__device__ __forceinline__ void pass_tile(const PassDesc& d, const SmoothSched& s, const Tile& t, const float2* gin,
                                          float2* gout, long long blk, long long nlines)
{
    extern __shared__ float2 sm[];
    const long long line0 = blk * t.lpc;
    const long long left = nlines - line0;
    const int lines = left < t.lpc ? static_cast<int>(left) : t.lpc;
    const long long g0 = idiv(line0, d.lines_per_group);
    const LineIO<EPI> io{d,      gin,
                         gout,   line0,
                         g0,     line0 - g0 * d.lines_per_group,
                         t.flat, d.conj_in ? -1.0f : 1.0f,
                         d.scale, d.conj_out ? -d.scale : d.scale};
    run_tile<WIDE>(s, sm, t.sl, t.sp, t.lpc, lines, Lanes{t.first}, Lanes{t.mid}, Lanes{t.last}, io);
    if (d.discard_in && s.ns > 1 && d.in.estride == 1 && d.in.ldist == d.n && d.in.gdist == d.lines_per_group * d.n)
    {
        // A dead input (a four-step intermediate in L2; the barriers since the first stage end this CTA's reads of
        // it): drop the 128-byte lines that lie wholly in the tile, whose rows are consecutive in memory, so that L2
        // does not write them back. A line shared with the next tile stays: that CTA may not have read it yet.
        const uintptr_t lo = reinterpret_cast<uintptr_t>(gin + line0 * d.n);
        const uintptr_t hi = lo + static_cast<uintptr_t>(lines) * d.n * 8;
        for (uintptr_t p = ((lo + 127) & ~static_cast<uintptr_t>(127)) + threadIdx.x * 128; p + 128 <= hi;
             p += blockDim.x * 128)
            asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
    }
}

} // namespace
} // namespace smooth
} // namespace crdfft
