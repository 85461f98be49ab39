// Welch's average for the power-of-two segment lengths 256 .. 8192, two segments a complex transform: with
// z = s1 + i s2 and Z = FFT(z), |S1[k]|^2 + |S2[k]|^2 = (|Z[k]|^2 + |Z[N-k]|^2) / 2, so the sum over segments needs
// neither the pairs' recombination nor any store of a spectrum: each thread adds |Z|^2 of the outputs its last stage
// leaves in registers, over all the pairs its line takes, and the frequencies k and N - k meet once at the end.
//
// One line of T = N / R1 threads a pair (a warp for 1024 points, so that its exchanges need no CTA barrier); a CTA
// takes `ppc` consecutive pairs of one signal and writes one row of sums, in a fixed order.
//
// The segment-by-segment kernel (spectral.cu) with a half-length real transform issues 104 instructions a complex point,
// its shared-memory pipe 74 % busy, and leaves a row of sums every few segments for the second launch to add: 606 us for
// 64 signals x 2^21 samples at 1024. Here 48 instructions a point, 74 % of the issue slots (what bounds it now), and a
// few dozen rows a signal: 238 us.

#include "codelets.cuh"
#include "index.cuh"
#include "kernels.hpp"
#include "smem_limit.hpp"

#include <algorithm>
#include <vector>

namespace crdfft
{
namespace
{

template <int R1, int R2, int R3> struct Shape
{
    static constexpr int N = R1 * R2 * R3;
    static constexpr int n1 = N / R1;
    static constexpr int T = n1;                       // threads a line: one first-stage butterfly each
    static constexpr int p1 = n1 | 1;                  // places a block of n1 takes (odd: the last stage's stride)
    static constexpr int Rs = R3 == 1 ? R2 : R3;       // the last radix
    static constexpr int Bs = N / Rs / T;              // last-stage butterflies a thread
    static constexpr int B2 = R3 == 1 ? 0 : N / R2 / T;
    static constexpr int threads = T <= 32 ? 128 : T;
    static constexpr int lines = threads / T;
    static constexpr int places = R1 * p1;
};

template <bool WARP> __device__ __forceinline__ void line_sync()
{
    if constexpr (WARP)
        __syncwarp();
    else
        __syncthreads();
}

template <int R> __device__ __forceinline__ void twiddle(float2* v, const float2* tw, int L, int k)
{
#pragma unroll
    for (int r = 1; r < R; ++r)
        v[r] = cmul(v[r], __ldg(tw + (r - 1) * L + k));
}

template <int R1, int R2, int R3>
__global__ void __launch_bounds__(Shape<R1, R2, R3>::threads, 512 / Shape<R1, R2, R3>::threads)
    welch_pair_kernel(const SpectralDesc sd, const float* __restrict__ x, float* __restrict__ part)
{
    using S = Shape<R1, R2, R3>;
    constexpr int N = S::N, n1 = S::n1, T = S::T, Rs = S::Rs, Bs = S::Bs;
    constexpr bool warp = T <= 32;
    extern __shared__ float2 sm[];
    __shared__ float2 s_sum[S::threads / 32];
    const int tid = threadIdx.x;
    const int ll = tid / T;
    const int jt = tid - ll * T;
    float2* line = sm + ll * S::places;
    const long long g = idiv(blockIdx.x, sd.ntiles);
    const int c = static_cast<int>(blockIdx.x - g * sd.ntiles);
    const float* sig = x + g * sd.nsamples;
    const float2* tw = static_cast<const float2*>(sd.pair_tw);
    const long long npairs = (sd.nseg + 1) / 2;
    const long long first = static_cast<long long>(c) * sd.ppc;
    const int mine = static_cast<int>(npairs - first < sd.ppc ? npairs - first : sd.ppc);

    float acc[Bs][Rs];
#pragma unroll
    for (int b = 0; b < Bs; ++b)
#pragma unroll
        for (int r = 0; r < Rs; ++r)
            acc[b][r] = 0.0f;

    // every line runs the same number of rounds (warps and barriers stay whole); a line past its last pair adds zeros
    for (int i0 = 0; i0 < mine; i0 += S::lines)
    {
        const int i = i0 + ll;
        const bool on = i < mine;
        const long long s0 = 2 * (first + (on ? i : 0));
        const bool two = on && s0 + 1 < sd.nseg;
        const float* xa = sig + s0 * sd.hop + jt;
        const float* xb = xa + (two ? sd.hop : 0);
        float2 v[R1];
        float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < R1; ++r)
        {
            v[r] = make_float2(on ? __ldg(xa + r * n1) : 0.0f, two ? __ldg(xb + r * n1) : 0.0f);
            sum = cadd(sum, v[r]);
        }
        if (sd.detrend)
        {
#pragma unroll
            for (int m = (warp ? T : 32) / 2; m >= 1; m >>= 1)
            {
                sum.x += __shfl_xor_sync(0xffffffffu, sum.x, m);
                sum.y += __shfl_xor_sync(0xffffffffu, sum.y, m);
            }
            if constexpr (!warp)
            {
                if ((tid & 31) == 0)
                    s_sum[tid / 32] = sum;
                __syncthreads();
                sum = s_sum[0];
#pragma unroll
                for (int w = 1; w < T / 32; ++w)
                    sum = cadd(sum, s_sum[w]);
            }
            const float2 mean = cscale(sum, 1.0f / static_cast<float>(N));
#pragma unroll
            for (int r = 0; r < R1; ++r)
                v[r] = csub(v[r], mean);
        }
#pragma unroll
        for (int r = 0; r < R1; ++r)
            v[r] = cscale(v[r], __ldg(sd.win + jt + r * n1));
        Dft<R1>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r)
            line[r * S::p1 + jt] = v[r];
        line_sync<warp>();
        if constexpr (R3 != 1)
        {
#pragma unroll
            for (int b = 0; b < S::B2; ++b)
            {
                const int j = jt + b * T;
                const int k1 = j / (n1 / R2);
                float2* p = line + k1 * S::p1 + (j - k1 * (n1 / R2));
                float2 u[R2];
#pragma unroll
                for (int r = 0; r < R2; ++r)
                    u[r] = p[r * R3];
                twiddle<R2>(u, tw, R1, k1);
                Dft<R2>::run(u);
#pragma unroll
                for (int r = 0; r < R2; ++r)
                    p[r * R3] = u[r];
            }
            line_sync<warp>();
        }
        constexpr int L = N / Rs;
        const float2* twl = tw + (R3 == 1 ? 0 : (R2 - 1) * R1);
#pragma unroll
        for (int b = 0; b < Bs; ++b)
        {
            const int j = jt + b * T;
            const float2* p = R3 == 1 ? line + j * S::p1 : line + (j % R1) * S::p1 + (j / R1) * R3;
            float2 u[Rs];
#pragma unroll
            for (int r = 0; r < Rs; ++r)
                u[r] = p[r];
            twiddle<Rs>(u, twl, L, j);
            Dft<Rs>::run(u);
            if (on)
            {
#pragma unroll
                for (int r = 0; r < Rs; ++r)
                    acc[b][r] = fmaf(u[r].x, u[r].x, fmaf(u[r].y, u[r].y, acc[b][r]));
            }
        }
        line_sync<warp>(); // the line is read: the next pair may overwrite it (and the sums)
    }

    __syncthreads();
    float* mine_f = reinterpret_cast<float*>(line); // N sums of this line, natural order
#pragma unroll
    for (int b = 0; b < Bs; ++b)
#pragma unroll
        for (int r = 0; r < Rs; ++r)
            mine_f[jt + b * T + r * (N / Rs)] = acc[b][r];
    __syncthreads();
    constexpr int nfreq = N / 2 + 1;
    float* dst = part + static_cast<long long>(blockIdx.x) * nfreq;
    for (int k = tid; k < nfreq; k += S::threads)
    {
        float a = 0.0f;
        for (int l = 0; l < S::lines; ++l)
        {
            const float* f = reinterpret_cast<const float*>(sm + l * S::places);
            a += (k == 0 || k == N / 2) ? f[k] : f[k] + f[N - k]; // doubled off DC and Nyquist, halved by the identity
        }
        dst[k] = sd.scale * a;
    }
}

using PairFn = void (*)(const SpectralDesc, const float*, float*);
struct Pair
{
    int n;
    PairFn fn;
    int threads, lines, smem;
    int radix[3];
};

template <int R1, int R2, int R3> Pair make()
{
    using S = Shape<R1, R2, R3>;
    return Pair{S::N, welch_pair_kernel<R1, R2, R3>, S::threads, S::lines, S::lines * S::places * 8, {R1, R2, R3}};
}

const Pair* find(int nperseg)
{
    static const Pair table[] = {make<16, 16, 1>(), make<32, 16, 1>(),  make<32, 32, 1>(),
                                 make<16, 16, 8>(), make<16, 16, 16>(), make<32, 16, 16>()};
    for (const Pair& p : table)
        if (p.n == nperseg)
            return &p;
    return nullptr;
}

} // namespace

bool welch_pair_shape(int nperseg, long long count, long long nseg, std::vector<int>* radices, int* ntiles, int* ppc)
{
    const Pair* p = find(nperseg);
    if (p == nullptr)
        return false;
    radices->clear();
    for (int r : p->radix)
        if (r > 1)
            radices->push_back(r);
    // About three rounds of the CTAs the device holds (512 threads an SM), each a whole number of rounds of its lines.
    const long long npairs = (nseg + 1) / 2;
    const long long want = std::max(1LL, 3LL * 148 * (512 / p->threads) / count);
    long long each = (npairs + want - 1) / want;
    each = (each + p->lines - 1) / p->lines * p->lines;
    *ppc = static_cast<int>(std::min(each, 1LL << 30));
    *ntiles = static_cast<int>((npairs + *ppc - 1) / *ppc);
    return true;
}

cudaError_t launch_welch_pair(const SpectralDesc& sd, const void* x, void* part, cudaStream_t stream)
{
    const Pair* p = find(sd.nperseg);
    if (p == nullptr || sd.ppc < 1)
        return cudaErrorInvalidConfiguration;
    const long long blocks = sd.count * sd.ntiles;
    if (blocks <= 0)
        return cudaSuccess;
    if (blocks > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    if (const cudaError_t e = allow_smem(p->fn, p->smem); e != cudaSuccess)
        return e;
    p->fn<<<static_cast<unsigned>(blocks), p->threads, p->smem, stream>>>(sd, static_cast<const float*>(x),
                                                                          static_cast<float*>(part));
    return cudaGetLastError();
}

} // namespace crdfft
