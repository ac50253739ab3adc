// fork_join over a fake of the CUDA runtime's stream and event calls: call number `fail` fails (0: none),
// and every stream keeps the work that nobody has waited for.
#include <cstdint>
#include <map>
#include <set>

#include "bf200_branches.h"

namespace {
int calls = 0, fail = 0;
int next_work = 0;
std::map<void*, std::set<int>> in_flight;  // per stream: work that its synchronisation would wait for
std::map<void*, std::set<int>> recorded;   // per event
std::set<int> finished;

cudaError_t step() { return ++calls == fail ? cudaErrorLaunchFailure : cudaSuccess; }

template <class T>
T handle(uintptr_t v) {
    return reinterpret_cast<T>(v);
}
}  // namespace

extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t event, cudaStream_t stream) {
    if (const cudaError_t e = step(); e != cudaSuccess) {
        return e;
    }
    recorded[event] = in_flight[stream];
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t stream, cudaEvent_t event, unsigned int) {
    if (const cudaError_t e = step(); e != cudaSuccess) {
        return e;
    }
    in_flight[stream].insert(recorded[event].begin(), recorded[event].end());
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t stream) {
    finished.insert(in_flight[stream].begin(), in_flight[stream].end());
    return cudaSuccess;
}

// The stage with its `failing`-th call failing, then the caller's synchronisation of the main stream. Returns
// the work that is still in flight, or -1 when an error is lost; *made: the calls that were made.
int run_fork_join(int failing, int with_branches, int* made) {
    calls = next_work = 0;
    fail = failing;
    in_flight.clear();
    recorded.clear();
    finished.clear();
    bf200::ShadeBranches b{};
    for (uint32_t k = 0; k < bf200::kShadeBranches; ++k) {
        b.stream[k] = handle<cudaStream_t>(16U + k);
        b.join[k] = handle<cudaEvent_t>(32U + k);
    }
    b.fork = handle<cudaEvent_t>(48U);
    const auto stream = handle<cudaStream_t>(1U);
    in_flight[stream].insert(next_work++);  // what the branches must run behind
    bool behind = true;
    const cudaError_t e =
        bf200::fork_join(with_branches != 0 ? &b : nullptr, stream, [&](const cudaStream_t(&on)[bf200::kShadeBranches]) {
            cudaError_t launched = cudaSuccess;
            for (cudaStream_t s : {stream, on[0], on[1], on[2]}) {  // one launch each, until one fails
                behind = behind && in_flight[s].count(0) == 1U;
                if (launched == cudaSuccess) {
                    launched = step();
                    if (launched == cudaSuccess) {
                        in_flight[s].insert(next_work++);
                    }
                }
            }
            return launched;
        });
    *made = calls;
    if (!behind || (e == cudaSuccess) != (failing == 0 || failing > calls)) {
        return -1;
    }
    cudaStreamSynchronize(stream);
    return next_work - static_cast<int>(finished.size());
}
}
