// kept_allocs.h -- device memory of a state that a context builds again and again.
//
// cudaMalloc and cudaFree wait for the device and map memory: the dozen of a tracer's or a charge
// solver's state took 1-2 ms of every lbgpu_mp_init / lbgpu_pnp_init.  A state built over an older
// one of the same context takes its buffers where the sizes agree; what is left of the old state is
// freed before the call returns.  Memory goes back with the state (lbgpu_mp_release, the context).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <utility>
#include <vector>

namespace lbg {

class KeptAllocs {
public:
    // a buffer of that size: one of the older state, or new
    cudaError_t get(void **p, size_t bytes)
    {
        for (size_t k = 0; k < spare_.size(); ++k)
            if (spare_[k].second == bytes) {
                *p = spare_[k].first;
                live_.push_back(spare_[k]);
                spare_.erase(spare_.begin() + (long)k);
                return cudaSuccess;
            }
        cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation && !spare_.empty()) {   // give the older state's back first
            cudaGetLastError();
            drop_spare();
            e = cudaMalloc(p, bytes);
        }
        if (e == cudaSuccess) live_.emplace_back(*p, bytes);
        return e;
    }
    // the buffers of an older state, whose work is on the stream that the new one uses
    void take(KeptAllocs &old)
    {
        spare_ = std::move(old.live_);
        old.live_.clear();
    }
    // frees what the new state did not take, however its construction ends
    struct SpareGuard {
        KeptAllocs &a;
        ~SpareGuard() { a.drop_spare(); }
    };
    void drop_spare()
    {
        for (auto &a : spare_) cudaFree(a.first);
        spare_.clear();
    }
    void free_all()
    {
        drop_spare();
        for (auto &a : live_) cudaFree(a.first);
        live_.clear();
    }

private:
    std::vector<std::pair<void *, size_t>> live_, spare_;
};

}  // namespace lbg
