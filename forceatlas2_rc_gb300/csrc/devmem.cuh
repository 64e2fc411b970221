// devmem.cuh -- device buffers of a session, released together.
#pragma once

#include <cuda_runtime.h>
#include <utility>
#include <vector>

namespace fa2cu {

struct DevMem {
    std::vector<void *> ptrs;
    double bytes = 0.0;
    bool failed = false;
    cudaError_t err = cudaSuccess;
    // With a pool: stream-ordered allocations on `s` from `pool` (no device
    // synchronisation on allocation or release). Dry: count bytes only.
    cudaMemPool_t pool = nullptr;
    cudaStream_t s = nullptr;
    bool dry = false;
    // planned(): one allocation from which get() takes the buffers
    static constexpr size_t ALIGN = 256;
    char *slab = nullptr;
    size_t slab_size = 0, slab_used = 0;

    void *raw(size_t b)
    {
        void *p = nullptr;
        err = pool ? cudaMallocFromPoolAsync(&p, b, pool, s) : cudaMalloc(&p, b);
        if (err != cudaSuccess) {
            failed = true;
            return nullptr;
        }
        ptrs.push_back(p);
        return p;
    }
    template <class T> T *get(size_t count)
    {
        if (failed) return nullptr;
        const size_t b = (count > 0 ? count : 1) * sizeof(T);
        const size_t room = (b + ALIGN - 1) / ALIGN * ALIGN;
        if (dry) {
            bytes += (double) b;
            slab_size += room;
            return nullptr;
        }
        void *p;
        if (room <= slab_size - slab_used) {
            p = slab + slab_used;
            slab_used += room;
        } else {
            p = raw(b);
            if (!p) return nullptr;
        }
        bytes += (double) b;
        return (T *) p;
    }
    // Runs `take` (a sequence of get()) twice: to count, then to hand out
    // parts of one allocation of that size. (A layout has about 35 buffers, at
    // a few microseconds for each cudaMalloc and cudaFree.)
    template <class F> void planned(F take)
    {
        if (dry || failed) return take();
        DevMem was;
        std::swap(was.slab, slab);
        std::swap(was.slab_size, slab_size);
        std::swap(was.slab_used, slab_used);
        const double before = bytes;
        dry = true;
        take();
        dry = false;
        bytes = before;
        slab = (char *) raw(slab_size);
        if (!slab) slab_size = 0;
        take();
    }
    void release()
    {
        for (void *p : ptrs) {
            if (pool)
                cudaFreeAsync(p, s);
            else
                cudaFree(p);
        }
        ptrs.clear();
        slab = nullptr;
        slab_size = slab_used = 0;
    }
};

} // namespace fa2cu
