// The dynamic shared memory a kernel may be launched with. cudaFuncSetAttribute sets the limit for the whole process:
// a launcher that sets it to its own launch's size can lower it between another thread's call and that thread's launch
// of the same kernel at a larger size, which then fails. Here a kernel's limit only ever rises.

#pragma once

#include <algorithm>
#include <mutex>
#include <unordered_map>

namespace crdfft
{

class SmemLimits
{
public:
    // Calls set(limit) with the largest size asked for `fn` so far, `bytes` among them; a size that is refused is not
    // remembered. Returns set's result (0: done).
    template <class Set> auto raise(const void* fn, int bytes, Set&& set) -> decltype(set(bytes))
    {
        std::lock_guard<std::mutex> lk(mu_);
        auto it = most_.find(fn);
        const int want = it == most_.end() ? bytes : std::max(it->second, bytes);
        const auto e = set(want);
        if (static_cast<int>(e) == 0)
            most_[fn] = want;
        return e;
    }

private:
    std::mutex mu_;
    std::unordered_map<const void*, int> most_; // one entry a kernel of the library
};

#ifdef __CUDACC__
// Lets `fn` be launched with `bytes` of dynamic shared memory (48 KB need no asking).
template <class Fn> cudaError_t allow_smem(Fn* fn, int bytes)
{
    static SmemLimits limits; // of the kernels of this type; each kernel's launches all come through here
    if (bytes <= 48 * 1024)
        return cudaSuccess;
    return limits.raise(reinterpret_cast<const void*>(fn), bytes, [&](int limit) {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    });
}
#endif

} // namespace crdfft
