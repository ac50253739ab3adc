// Streams that the shading stage forks from the wavefront's stream and joins to it again.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdint>

namespace bf200 {

constexpr uint32_t kShadeBranches = 3U;
struct ShadeBranches {
    cudaStream_t stream[kShadeBranches];
    cudaEvent_t fork, join[kShadeBranches];
};

// Runs body(on), which queues work on `stream` and on the branches on[k] (on `stream` itself without
// branches), behind `stream` and before what `stream` runs next. When any step fails, the branches have
// nothing left in flight on return: what they hold may use the caller's buffers, and the caller then waits
// for `stream` alone.
template <class Body>
cudaError_t fork_join(const ShadeBranches* branches, cudaStream_t stream, Body&& body) {
    cudaStream_t on[kShadeBranches] = {stream, stream, stream};
    if (branches == nullptr) {
        return body(on);
    }
    cudaError_t e = cudaEventRecord(branches->fork, stream);
    for (uint32_t k = 0; k < kShadeBranches && e == cudaSuccess; ++k) {
        on[k] = branches->stream[k];
        e = cudaStreamWaitEvent(on[k], branches->fork, 0);
    }
    if (e == cudaSuccess) {
        e = body(on);
    }
    for (uint32_t k = 0; k < kShadeBranches && e == cudaSuccess; ++k) {
        e = cudaEventRecord(branches->join[k], on[k]);
        if (e == cudaSuccess) {
            e = cudaStreamWaitEvent(stream, branches->join[k], 0);
        }
    }
    if (e != cudaSuccess) {
        for (cudaStream_t branch : branches->stream) {
            cudaStreamSynchronize(branch);
        }
    }
    return e;
}

}  // namespace bf200
