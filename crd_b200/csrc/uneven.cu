// Uneven batch: thousands of independent complex transforms of different 7-smooth lengths, each at its own offset
// in a packed buffer, in one persistent launch. The reference runs such a batch as a loop of per-size plans over
// crd-jobs ranges (include/crd/hesap/fft/detail/batch_arms.hpp:59-77, one plan per job); here one kernel walks a
// device work list:
//
//   SMALL  up to `lines` transforms of one length n <= 4096, one CTA, all stages in shared memory
//   COL    a tile of adjacent columns of one long transform (n = n1 n2 > 4096): length-n1 DFTs, four-step twiddle,
//          written to the transform's region of the workspace
//   ROW    a tile of rows of that transform's workspace region: length-n2 DFTs, transposed store to the output
//
// Each item is a tile of the run-time-schedule lines (smooth_line.cuh), up to 4096 points: about 35 KB of shared memory
// and 256 threads at 80 registers, three CTAs an SM, so that one item's loads, stages and stores overlap the others'
// (20,000 transforms: 1.85 ms; 128 threads and five CTAs 1.96, tiles of 8192 points 1.85 but 60 transforms 25 us
// instead of 17). CTAs (as many as fit on the GPU at once, G of them) take items in list order, CTA c the items c, c + G,
// ...; the next item's descriptor, schedule and line offsets come into shared memory while the current one is transformed.
//
// While COL items of other transforms remain, a transform's ROW items follow its last COL item by more than G items, so
// those are nearly always done when it starts, and near enough that the intermediate is still in L2 (whose lines the ROW
// item drops after reading); the last transforms' ROW items follow the SMALL ones, however few, and may have to wait.
// A wait on its transform's completion counter always ends: the earliest unfinished item of the list is the next one of
// its CTA (the CTA's earlier items are earlier in the list), and what it waits for is earlier still. That needs every CTA
// of the grid resident at once, whatever other streams run: a list with waits is launched cooperatively, which costs 2 us,
// or, where every CTA has one item, each takes the next of the list by a counter as it starts: what it waits for has
// started before it. (Every item claimed so needs no residency either, but the 20,000 transforms then take 2.08 ms with
// one claim ahead of the work and 2.17 with two.) The wait is bounded anyway (spin_limit polls): one that runs out sets
// the plan's status word and skips the item.
//
// Two asynchronously filled 32 KB slots and out-of-place stages before: 215 instructions a point and pass, two CTAs an
// SM, every intermediate through HBM, 3.63 ms. Now 95 instructions; bound by latency (42 % issue, the barriers of two or
// three short stages an item first among the stalls).

#include "kernels.hpp"
#include "smem_limit.hpp"
#include "smooth_line.cuh"
#include "uneven.hpp"

namespace crdfft
{
namespace smooth
{
namespace
{

constexpr int kThreads = 256;

struct ItemIO
{
    const UnevenItem& it;
    const long long* off; // SMALL: the lines' offsets
    const float2* src;
    float2* dst;
    const float2* fh;
    const float2* fl;
    int n;
    float in_im, out_re, out_im;
    bool cached; // the input never changes during the launch (not the workspace)

    template <int R> __device__ __forceinline__ void get(float2* v, int l, int b, int N) const
    {
        const long long o = it.kind == kUnevenSmall ? off[l] : it.in_base + l * it.in_ldist;
        const float2* p = src + o + b * it.in_estride;
        const long long step = N * it.in_estride;
        if (cached)
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r] = __ldcs(p + r * step);
        }
        else
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r] = __ldcg(p + r * step);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r].y *= in_im;
    }
    template <int R> __device__ __forceinline__ void put(float2* v, int l, int b, int N) const
    {
        const long long o = it.kind == kUnevenSmall ? off[l] : it.out_base + l * it.out_ldist;
        float2* p = dst + o + b * it.out_estride;
        const long long step = N * it.out_estride;
        if (fh != nullptr)
        {
            const int q = it.q0 + l; // column of the long transform
            const float2* th = fh + (q >> 4) * n + b;
            const float2* tl = fl + b * 16 + (q & 15);
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r] = cmul(v[r], cmul(__ldg(th + r * N), __ldg(tl + r * N * 16)));
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            p[r * step] = make_float2(v[r].x * out_re, v[r].y * out_im);
    }
};

template <class T> __device__ __forceinline__ void copy_words(T* dst, const T* src, int tid)
{
    static_assert(sizeof(T) % 4 == 0);
    const int* s = reinterpret_cast<const int*>(src);
    int* d = reinterpret_cast<int*>(dst);
    for (int i = tid; i < static_cast<int>(sizeof(T) / 4); i += kThreads)
        d[i] = __ldg(s + i);
}

__global__ void __launch_bounds__(kThreads, 3)
    uneven_kernel(const UnevenDesc u, const float2* gin, float2* gout, float2* scratch)
{
    extern __shared__ float2 sm[];
    __shared__ UnevenItem s_it[2];
    __shared__ SmoothSched s_sc[2];
    __shared__ long long s_off[2][kUnevenLines];
    __shared__ int s_go;
    __shared__ int s_claim;
    const int tid = threadIdx.x;
    const int G = gridDim.x;
    const float in_im = u.conj ? -1.0f : 1.0f;
    const float out_im = u.conj ? -u.scale : u.scale;

    // An item whose descriptor is in slot k: its schedule and, for whole transforms, its lines' offsets.
    auto fetch_rest = [&](int k) {
        const UnevenItem& it = s_it[k];
        copy_words(&s_sc[k], u.scheds + it.sched, tid);
        if (it.kind == kUnevenSmall)
            for (int a = tid; a < it.lines; a += kThreads)
                s_off[k][a] = __ldg(u.line_off + it.line_table + a);
    };
    // Thread 0: whether item slot k may run; a ROW item waits for its COL items.
    auto ready = [&](int k) {
        const UnevenItem& it = s_it[k];
        if (it.kind != kUnevenRow)
            return 1;
        const volatile int* done = u.done + it.transform;
        for (int i = 0; *done < it.need; ++i)
        {
            if (i > u.spin_limit)
            {
                atomicOr(u.err, 1);
                return 0;
            }
            __nanosleep(64);
        }
        __threadfence(); // acquire: the COL items' workspace writes are visible past the next barrier
        return 1;
    };

    int idx = blockIdx.x;
    if (u.started != nullptr)
    {
        if (tid == 0)
            s_claim = atomicAdd(u.started, 1);
        __syncthreads();
        idx = s_claim;
    }
    if (idx >= u.nitems)
        return;
    copy_words(&s_it[0], u.items + idx, tid);
    __syncthreads();
    fetch_rest(0);
    if (tid == 0)
        s_go = ready(0);
    __syncthreads();
    for (int k = 0; idx < u.nitems; k ^= 1)
    {
        const UnevenItem& it = s_it[k];
        const SmoothSched& s = s_sc[k];
        const bool more = idx + G < u.nitems;
        if (more)
            copy_words(&s_it[k ^ 1], u.items + idx + G, tid);
        const bool go = s_go != 0;
        const bool first_pass = it.kind != kUnevenRow, last_pass = it.kind != kUnevenCol;
        const ItemIO io{it,
                        s_off[k],
                        first_pass ? gin : scratch,
                        last_pass ? gout : scratch,
                        static_cast<const float2*>(it.ftw_hi),
                        static_cast<const float2*>(it.ftw_lo),
                        s.n,
                        first_pass ? in_im : 1.0f,
                        last_pass ? u.scale : 1.0f,
                        last_pass ? out_im : 1.0f,
                        first_pass};
        const Lanes first{it.first}, last{it.last};
        if (go)
            with_radix<false>(s.st[0].R, [&]<int R>() { first_stage<R>(s, first, sm, it.sl, it.sp, it.lpc, it.lines, io); });
        __syncthreads(); // this item's loads are done and its tile filled; the next item's descriptor is here
        if (more)
            fetch_rest(k ^ 1);
        if (go)
        {
            for (int i = 1; i < s.ns - 1; ++i)
            {
                with_radix<false>(s.st[i].R, [&]<int R>() { mid_stage<R>(s, i, first, sm, it.sl, it.sp, it.lpc, it.lines); });
                __syncthreads();
            }
            if (s.ns > 1)
                with_radix<false>(s.st[s.ns - 1].R,
                                  [&]<int R>() { last_stage<R>(s, last, sm, it.sl, it.sp, it.lpc, it.lines, io); });
            if (it.kind == kUnevenRow)
            {
                // the rows are read: drop the 128-byte lines of the workspace that lie wholly in them
                const uintptr_t lo = reinterpret_cast<uintptr_t>(scratch + it.in_base);
                const uintptr_t hi = lo + static_cast<uintptr_t>(it.lines) * s.n * 8;
                for (uintptr_t p = ((lo + 127) & ~static_cast<uintptr_t>(127)) + tid * 128; p + 128 <= hi;
                     p += kThreads * 128)
                    asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
            }
        }
        __syncthreads(); // the tile is free, every store of the item issued
        if (tid == 0)
        {
            if (it.kind == kUnevenCol)
            {
                __threadfence(); // release: the CTA's workspace writes before the item's count
                atomicAdd(u.done + it.transform, 1);
            }
            if (more)
                s_go = ready(k ^ 1); // after the count: the next item may wait for this one
        }
        __syncthreads(); // this slot is free
        idx += G;
    }
}

} // namespace
} // namespace smooth

int uneven_resident(int smem_bytes)
{
    if (allow_smem(smooth::uneven_kernel, smem_bytes) != cudaSuccess)
        return 0;
    int per_sm = 0, dev = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, smooth::uneven_kernel, smooth::kThreads, smem_bytes) !=
            cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return per_sm * sms;
}

cudaError_t launch_uneven(const UnevenDesc& u0, int smem_bytes, const void* in, void* out, void* scratch,
                          cudaStream_t stream)
{
    UnevenDesc u = u0;
    int grid = uneven_resident(smem_bytes);
    if (grid < 1)
        return cudaErrorInvalidConfiguration;
    if (grid > u.nitems)
        grid = u.nitems;
    if (grid < 1)
        return cudaSuccess;
    if (u.ntransforms > 0)
    {
        const cudaError_t e = cudaMemsetAsync(u.started, 0, sizeof(int) * (1 + u.ntransforms), stream);
        if (e != cudaSuccess)
            return e;
    }
    const bool waits = u.ntransforms > 0;
    if (!waits || grid < u.nitems)
        u.started = nullptr;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(smooth::kThreads, 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = waits && u.started == nullptr ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, smooth::uneven_kernel, u, static_cast<const float2*>(in), static_cast<float2*>(out),
                              static_cast<float2*>(scratch));
}

} // namespace crdfft
