// Bluestein's chirp-z transform of lengths with a prime factor above 7, on the run-time-schedule tiles (smooth_line.cuh):
// with chirp_k = exp(+iπ k²/n), X_k = conj(chirp_k) sum_j (x_j conj(chirp_j)) chirp_{k-j}, a circular convolution of a
// 7-smooth length m >= 2n - 1 (include/crd/hesap/fft/bluestein.hpp:87-136, which pads to a power of two).
//
//   m <= kChirpLine   one launch: the chirp product in the first stage's loads, the convolution in shared memory, the
//                     chirp product in the last stage's stores. 8 bytes a point in, 8 out.
//   longer            three launches over m = n1 n2: columns (chirp and zero padding in the loads, four-step twiddle),
//                     rows (transform, filter, transform back in place, twiddle), columns (chirp in the stores). The
//                     convolution needs no transposes: the rows' second transform runs on the order the first left.
//                     The padded sequences stay in L2 (waves of a few tens of MB).
//
// Ten and more launches over m = 2^k before (pad, two transforms of two passes and two waves each, product, chirp):
// 10007 points x 251, m = 32768, 226 us; bound then by the launches' ramps and by L2. Now 92 us, bound by latency at 19
// to 24 warps an SM (39-43 % issue) and by instruction fetch.

#include "kernels.hpp"
#include "pass_desc.hpp"
#include "smem_limit.hpp"
#include "smooth_line.cuh"
#include "smooth_plan.hpp"

#include <algorithm>

namespace crdfft
{
namespace smooth
{
namespace
{

__device__ __forceinline__ float2 chirp_in(const ChirpDesc& p, float2 x, float2 c)
{
    if (p.conj)
        x.y = -x.y;
    return make_float2(x.x * c.x + x.y * c.y, x.y * c.x - x.x * c.y);
}

// The convolution's value arrives conjugated (y = conj(DFT(..))).
__device__ __forceinline__ float2 chirp_out(const ChirpDesc& p, float2 v, float2 c)
{
    const float re = (v.x * c.x - v.y * c.y) * p.scale;
    const float im = (-v.y * c.x - v.x * c.y) * p.scale;
    return make_float2(re, p.conj ? -im : im);
}

// W_m^{q k1} from the four-step tables.
__device__ __forceinline__ float2 split_twiddle(const ChirpDesc& p, int q, int k1)
{
    return cmul(__ldg(static_cast<const float2*>(p.hi) + (q >> 4) * static_cast<int>(p.n1) + k1),
                __ldg(static_cast<const float2*>(p.lo) + k1 * 16 + (q & 15)));
}

// One CTA a line of m points: line l of the tile is transform line0 + l.
struct LineChirpIO
{
    const ChirpDesc& p;
    const float2* x;
    float2* out;
    long long line0;
    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        const float2* src = x + (line0 + l) * p.idist;
        const float2* ch = static_cast<const float2*>(p.chirp);
        const int n = static_cast<int>(p.n);
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            const int e = b + r * N;
            v[r] = e < n ? chirp_in(p, __ldcs(src + e), __ldg(ch + e)) : make_float2(0.f, 0.f);
        }
    }
    template <int R> __device__ __forceinline__ void filter(float2* v, int, int b, int N) const
    {
        const float2* h = static_cast<const float2*>(p.bfft) + b;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = cconj(cmul(v[r], __ldg(h + r * N)));
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        float2* dst = out + (line0 + l) * p.odist;
        const float2* ch = static_cast<const float2*>(p.chirp);
        const int n = static_cast<int>(p.n);
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            const int e = b + r * N;
            if (e < n)
                __stcs(dst + e, chirp_out(p, v[r], __ldg(ch + e)));
        }
    }
};

// Column q of a transform (lines of the pass: q fastest, then transforms): elements j1 n2 + q, the frequencies k1.
struct Column
{
    long long t;
    int q;
};
__device__ __forceinline__ Column column_of(const ChirpDesc& p, long long t0, int q0, int l)
{
    const int n2 = static_cast<int>(p.n2);
    Column c{t0, q0 + l};
    while (c.q >= n2) // a tile past the end of a transform's columns (short rows: past several)
    {
        c.q -= n2;
        ++c.t;
    }
    return c;
}

struct ColsInIO
{
    const ChirpDesc& p;
    const float2* x;
    float2* w;
    long long t0;
    int q0;
    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        const Column c = column_of(p, t0, q0, l);
        const int n2 = static_cast<int>(p.n2);
        const long long e0 = static_cast<long long>(b) * n2 + c.q;
        const long long step = static_cast<long long>(N) * n2;
        const float2* src = x + c.t * p.idist;
        const float2* ch = static_cast<const float2*>(p.chirp);
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            const long long e = e0 + r * step;
            v[r] = e < p.n ? chirp_in(p, __ldcs(src + e), __ldg(ch + e)) : make_float2(0.f, 0.f);
        }
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        const Column c = column_of(p, t0, q0, l);
        const long long step = static_cast<long long>(N) * p.n2;
        float2* dst = w + c.t * p.m + static_cast<long long>(b) * p.n2 + c.q;
#pragma unroll
        for (int r = 0; r < R; ++r)
            dst[r * step] = cmul(v[r], split_twiddle(p, c.q, b + r * N));
    }
};

struct RowsIO
{
    const ChirpDesc& p;
    float2* w;
    long long line0; // transform * n1 + k1
    int k0;          // line0 mod n1
    __device__ __forceinline__ int row(int l) const
    {
        int k1 = k0 + l;
        while (k1 >= static_cast<int>(p.n1))
            k1 -= static_cast<int>(p.n1);
        return k1;
    }
    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        const float2* src = w + (line0 + l) * p.n2 + b;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = src[r * N];
    }
    template <int R> __device__ __forceinline__ void filter(float2* v, int l, int b, int N) const
    {
        const float2* h = static_cast<const float2*>(p.bfft) + row(l) * p.n2 + b;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = cconj(cmul(v[r], __ldg(h + r * N)));
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        const int k1 = row(l);
        float2* dst = w + (line0 + l) * p.n2 + b;
#pragma unroll
        for (int r = 0; r < R; ++r)
            dst[r * N] = cmul(v[r], split_twiddle(p, b + r * N, k1));
    }
};

struct ColsOutIO
{
    const ChirpDesc& p;
    const float2* w;
    float2* out;
    long long t0;
    int q0;
    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        const Column c = column_of(p, t0, q0, l);
        const long long step = static_cast<long long>(N) * p.n2;
        const float2* src = w + c.t * p.m + static_cast<long long>(b) * p.n2 + c.q;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = __ldcs(src + r * step);
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        const Column c = column_of(p, t0, q0, l);
        const int n2 = static_cast<int>(p.n2);
        const long long e0 = static_cast<long long>(b) * n2 + c.q;
        const long long step = static_cast<long long>(N) * n2;
        float2* dst = out + c.t * p.odist;
        const float2* ch = static_cast<const float2*>(p.chirp);
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            const long long e = e0 + r * step;
            if (e < p.n)
                __stcs(dst + e, chirp_out(p, v[r], __ldg(ch + e)));
        }
    }
};

// Lines of the launch, lines a CTA and places of the tile.
struct Launch
{
    long long lines;
    int lpc;
    int sl, sp;
    int across;
};

enum class Pass : int
{
    Line,
    ColsIn,
    Rows,
    ColsOut
};

template <Pass PASS, bool WIDE>
__global__ void __maxnreg__(WIDE ? 128 : 80)
    chirp_kernel(const ChirpDesc p, const SmoothSched s, const Launch g, const float2* in, float2* out)
{
    extern __shared__ float2 sm[];
    const long long line0 = static_cast<long long>(blockIdx.x) * g.lpc;
    const long long left = g.lines - line0;
    const int lines = left < g.lpc ? static_cast<int>(left) : g.lpc;
    const Lanes ln{g.across};
    if constexpr (PASS == Pass::Line)
        run_conv_tile<WIDE>(s, sm, g.sl, g.sp, g.lpc, lines, ln, LineChirpIO{p, in, out, line0});
    else if constexpr (PASS == Pass::Rows)
    {
        const int k0 = static_cast<int>(line0 - idiv(line0, p.n1) * p.n1);
        run_conv_tile<WIDE>(s, sm, g.sl, g.sp, g.lpc, lines, ln, RowsIO{p, out, line0, k0});
    }
    else
    {
        const long long t0 = idiv(line0, p.n2);
        const int q0 = static_cast<int>(line0 - t0 * p.n2);
        if constexpr (PASS == Pass::ColsIn)
            run_tile<WIDE>(s, sm, g.sl, g.sp, g.lpc, lines, ln, ln, ln, ColsInIO{p, in, out, t0, q0});
        else
            run_tile<WIDE>(s, sm, g.sl, g.sp, g.lpc, lines, ln, ln, ln, ColsOutIO{p, in, out, t0, q0});
    }
}

template <Pass PASS>
cudaError_t launch(const ChirpDesc& p, long long len, const void* tw, long long lines, const void* in, void* out,
                   cudaStream_t stream)
{
    std::vector<int> rad;
    SmoothSched s;
    if (!chirp_radices(len, rad) ||
        !smooth_sched(static_cast<int>(len), rad.data(), static_cast<int>(rad.size()), tw, &s))
        return cudaErrorInvalidConfiguration;
    constexpr bool cols = PASS == Pass::ColsIn || PASS == Pass::ColsOut;
    const int places = s.st[0].R * s.p1;
    Launch g{};
    g.lines = lines;
    g.lpc = 1;
    g.across = -1;
    if (cols)
    {
        g.lpc = len <= 400 ? 32 : len <= 560 ? 16 : len <= 3000 ? 8 : len <= 6000 ? 4 : len <= 12000 ? 2 : 1;
        while (g.lpc < 64 && g.lpc * len < 1500)
            g.lpc *= 2;
        while ((1 << (g.across + 1)) <= g.lpc)
            ++g.across;
    }
    else
        g.lpc = std::max(1, static_cast<int>(2200 / len));
    if (PASS == Pass::Rows && g.lpc > 2)
        g.lpc = (g.lpc + 3) / 4 * 4;
    g.sl = cols ? 1 : places | 1;
    g.sp = cols ? g.lpc : 1;
    const long long grid = (lines + g.lpc - 1) / g.lpc;
    const int smem = g.lpc * (places | 1) * 8;
    if (grid < 1)
        return cudaSuccess;
    if (grid > 0x7fffffffLL || smem > 227 * 1024 || g.lpc * len > 65535)
        return cudaErrorInvalidConfiguration;
    const bool wide = smooth_wide(rad.data(), static_cast<int>(rad.size()));
    const auto fn = wide ? chirp_kernel<PASS, true> : chirp_kernel<PASS, false>;
    if (const cudaError_t e = allow_smem(fn, smem); e != cudaSuccess)
        return e;
    // Full column tiles take up to 256 threads, the most that leave the fewest idle in the stages' last rounds: fewer,
    // larger CTAs, since warps of one CTA are in the same stage and share its instructions (128-point columns, 32 a
    // tile: 10007 x 251 in 90.3 us with 256, 95.8 with 128; 168 points in 60 us with 160 or 192, 70 with 256).
    int threads = smooth_threads(s, g.lpc, smem, wide ? 128 : 80, grid);
    if (cols && g.lpc * len >= 4000)
    {
        double top = 0.0;
        for (int nt = threads; nt <= 256; nt += 32)
        {
            double slots = 0.0;
            for (int i = 0; i < s.ns; ++i)
                slots += static_cast<double>((g.lpc * s.st[i].N + nt - 1) / nt * nt) * s.st[i].R;
            if (1.0 / slots >= top)
            {
                top = 1.0 / slots;
                threads = nt;
            }
        }
    }
    fn<<<static_cast<unsigned>(grid), threads, smem, stream>>>(
        p, s, g, static_cast<const float2*>(in), static_cast<float2*>(out));
    return cudaGetLastError();
}

__global__ void chirp_gather_kernel(const float2* x, float2* w, long long n, long long dist, long long total)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        const long long t = idiv(i, n);
        w[i] = x[t * dist + (i - t * n)];
    }
}

} // namespace
} // namespace smooth

// The line schedules, with a single radix split in two: the convolution turns around in a stage after the first.
bool chirp_radices(long long m, std::vector<int>& out, double* arith)
{
    // (the turning stage holds its butterfly, twiddles and filter at once: radices above 16 cost 128 registers, and
    // 8000 points 10.10.10.8 64.1 us a 600-line batch, 20.20.20 76.8)
    if (m < 4 || m > 16384 || !smooth_radices(m, out, arith, 1.35))
        return false;
    if (out.size() == 1)
    {
        const int R = out[0];
        for (int a = 2; a * a <= R; ++a)
            if (R % a == 0)
                out = {R / a, a};
    }
    return out.size() >= 2;
}

cudaError_t launch_chirp_gather(const ChirpDesc& p, const void* x, void* w, cudaStream_t stream)
{
    const long long total = p.n * p.batch;
    const long long blocks = std::min((total + 255) / 256, 148LL * 8);
    smooth::chirp_gather_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        static_cast<const float2*>(x), static_cast<float2*>(w), p.n, p.idist, total);
    return cudaGetLastError();
}

cudaError_t launch_chirp_line(const ChirpDesc& p, const void* x, void* out, cudaStream_t stream)
{
    return smooth::launch<smooth::Pass::Line>(p, p.m, p.tw1, p.batch, x, out, stream);
}

cudaError_t launch_chirp_cols_in(const ChirpDesc& p, const void* x, void* w, cudaStream_t stream)
{
    return smooth::launch<smooth::Pass::ColsIn>(p, p.n1, p.tw1, p.batch * p.n2, x, w, stream);
}

cudaError_t launch_chirp_rows(const ChirpDesc& p, void* w, cudaStream_t stream)
{
    return smooth::launch<smooth::Pass::Rows>(p, p.n2, p.tw2, p.batch * p.n1, w, w, stream);
}

cudaError_t launch_chirp_cols_out(const ChirpDesc& p, const void* w, void* out, cudaStream_t stream)
{
    return smooth::launch<smooth::Pass::ColsOut>(p, p.n1, p.tw1, p.batch * p.n2, w, out, stream);
}

} // namespace crdfft
