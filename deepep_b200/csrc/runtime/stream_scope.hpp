// What the stream-control arguments of a call ask for: the stream its kernels run on, what they wait for and who waits
// for them. Shared by the drivers of the multi-rank and of the one-rank kernels.
#pragma once

#include <cstdlib>

#include "runtime.hpp"
#include "tensors.hpp"

namespace ep {

inline bool env_flag(const char* name) {
    const char* v = std::getenv(name);
    return v != nullptr && v[0] != '\0' && v[0] != '0';
}

inline at::TensorOptions opts(at::ScalarType dtype, int device) {
    return at::TensorOptions().dtype(dtype).device(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
}

// Everything the stream-control arguments ask for before the first launch.
struct StreamScope {
    at::cuda::CUDAStream compute, comm;     // `comm`: where the kernels of the call go
    Runtime& runtime;
    bool switched = false;
    // `may_stay`: a call that hands back nothing asynchronous and waits for nothing but the caller's stream may run on
    // that stream itself. That is the same order of work without the four event calls of the round trip over the
    // communication stream (about 5 us of host time and a few microseconds between dependent kernels on the GPU).
    StreamScope(const StreamControl& sc, Runtime& rt, bool may_stay = false)
        : compute(at::cuda::getCurrentCUDAStream()), comm(rt.comm_stream()), runtime(rt) {
        if (may_stay && !sc.async_with_compute_stream && !sc.allocate_on_comm_stream && !sc.previous_event.has_value()) {
            comm = compute;
            rt.order_behind_last_call(comm, compute);
            return;
        }
        if (sc.allocate_on_comm_stream) {
            at::cuda::setCurrentCUDAStream(comm);
            switched = true;
        }
        if (sc.previous_event.has_value()) sc.previous_event->stream_wait(comm);
        else stream_wait(comm, compute);
        rt.order_behind_last_call(comm, sc.previous_event.has_value() ? comm : compute);
    }
    // Either hands back an event (async) or makes the compute stream wait for the comm stream.
    std::optional<EventHandle> finish(const StreamControl& sc, const std::vector<at::Tensor>& tensors) {
        std::optional<EventHandle> event;
        if (sc.async_with_compute_stream) {
            event = EventHandle(comm);
            // EP_AVOID_RECORD_STREAM=1: the event keeps the tensors alive instead (the caller holds the event until it
            // has waited on it); record_stream delays the reuse of a block by the caching allocator in a way that is
            // hard to predict (csrc/elastic/buffer.hpp:556-584 of the reference offers the same switch).
            static const bool avoid_record_stream = env_flag("EP_AVOID_RECORD_STREAM");
            for (const auto& t : tensors) {
                if (!t.defined() || !t.is_cuda()) continue;
                if (avoid_record_stream) {
                    event->keep_alive.push_back(t);
                    continue;
                }
                // (views of the heap are not owned by the caching allocator; record_stream ignores them)
                t.record_stream(comm);
                if (sc.allocate_on_comm_stream) t.record_stream(compute);
            }
        } else if (comm != compute) {
            stream_wait(compute, comm);
        }
        if (switched) at::cuda::setCurrentCUDAStream(compute);
        if (sc.async_with_compute_stream) runtime.call_ended(comm, std::nullopt);
        else runtime.call_ended(comm, compute);
        return event;
    }
};

}  // namespace ep
