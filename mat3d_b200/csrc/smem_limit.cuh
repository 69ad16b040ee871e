// smem_limit.cuh -- the dynamic shared memory limit of a kernel.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

namespace m3d {

// Let a kernel use all dynamic shared memory left next to its static arrays
// (227 KB per block on sm_100 in total).
// Done once per kernel and device; safe to call from several host threads: the
// lock is held until the limit is set, so that whoever returns may launch.
inline std::mutex g_attr_mu;
inline std::set<std::pair<int, const void*>> g_attr_done;
template <class K>
void allow_smem(K kernel) {
    int dev = 0;
    cudaGetDevice(&dev);
    const void* const fn = (const void*)kernel;
    const auto key = std::make_pair(dev, fn);
    std::lock_guard<std::mutex> lk(g_attr_mu);
    if (g_attr_done.count(key)) return;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, fn) == cudaSuccess) {
        const int maxdyn = 227 * 1024 - (int)a.sharedSizeBytes;
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, maxdyn);
    }
    (void)cudaGetLastError();  // an unsupported request must not surface at the next launch check
    g_attr_done.insert(key);
}

}  // namespace m3d
