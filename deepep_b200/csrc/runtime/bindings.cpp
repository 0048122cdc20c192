// Python bindings of the native runtime (module deepep_b200._C).
//
// Parity: csrc/python_api.cpp:22-39 and the pybind blocks at csrc/elastic/buffer.hpp:1346-1380,
// csrc/legacy/buffer.hpp:1751-1792 of the reference.
#include <pybind11/stl.h>
#include <torch/extension.h>

#include "py_tuples.hpp"
#include "runtime.hpp"
#include "tensors.hpp"

namespace py = pybind11;
using namespace ep;

namespace {

// A call of one rank arrives as one tuple and its results leave as one tuple: filling an argument block and reading a
// result block attribute by attribute from Python cost about 15 us per call, which bounded small calls. The orders are
// those of ElasticBuffer._dispatch_call / _dispatch_result / _combine_call.
DispatchArgs dispatch_args(PyObject* call) {
    const TupleReader t(call, 24);
    DispatchArgs a;
    a.x = t.tensor(0);
    a.sf = t.maybe_tensor(1);
    a.topk_idx = t.maybe_tensor(2);
    a.topk_weights = t.maybe_tensor(3);
    a.cumulative_stats = t.maybe_tensor(4);
    a.num_experts = t.integer(5);
    a.num_max_tokens = t.integer(6);
    a.expert_alignment = t.integer(7);
    a.num_sms = t.integer(8);
    a.quant_mode = t.integer(9);
    a.do_expand = t.flag(10);
    a.do_zero_padding = t.flag(11);
    a.do_cpu_sync = t.flag(12);
    a.zero_copy = t.flag(13);
    a.num_worst_tokens = t.integer(14);
    a.col_major_sf = t.flag(15);
    a.copy_topk_idx = t.flag(16);
    a.sc.previous_event = t.event(17);
    a.sc.previous_event_before_epilogue = t.event(18);
    a.sc.async_with_compute_stream = t.flag(19);
    a.sc.allocate_on_comm_stream = t.flag(20);
    a.mask_weights = t.flag(22);
    a.defer_counts = t.flag(23);
    if (!t.none(21)) {        // the routing of an earlier dispatch
        const TupleReader h(t.item(21), 8);
        a.cached = true;
        a.h_token_slot = h.maybe_tensor(0);
        a.h_pair_row = h.maybe_tensor(1);
        a.h_psum_rank = h.maybe_tensor(2);
        a.h_psum_expert = h.maybe_tensor(3);
        a.h_num_unaligned = h.maybe_tensor(4);
        a.h_recv_src_metadata = h.maybe_tensor(5);
        a.h_num_recv_tokens = h.integer(6);
        a.h_num_expanded_tokens = h.integer(7);
    }
    return a;
}

py::list dispatch_calls(const std::vector<std::shared_ptr<Runtime>>& rts, const py::list& calls) {
    std::vector<DispatchArgs> args;
    for (const auto& c : calls) args.push_back(dispatch_args(c.ptr()));
    std::vector<DispatchResult> res;
    {
        // The drivers may block on the host for a long time (the wait for the received counts): they run without the GIL
        // so that Python threads of this process -- the heartbeat of the failure detector among them -- keep running.
        py::gil_scoped_release release;
        res = Runtime::dispatch(rts, args);
    }
    py::list out;
    for (size_t v = 0; v < res.size(); ++v) {
        DispatchResult& r = res[v];
        std::optional<at::Tensor> per_expert;
        if (!args[v].cached) per_expert = first_rows(r.psum_expert, r.psum_expert.size(0) - 1);    // the last word is the number of expanded rows
        TupleWriter t(19);
        t.put(r.recv_x).put(r.recv_sf).put(r.recv_topk_idx).put(r.recv_topk_weights).put(r.token_slot).put(r.pair_row).put(r.psum_rank).put(r.psum_expert)
            .put(per_expert).put(r.num_unaligned).put(r.recv_src_metadata).put(r.count_matrix).put(r.topk_idx).put(r.num_recv_tokens)
            .put(r.num_expanded_tokens).put(r.num_sms).put(r.num_recv_tokens_per_expert_list).put(r.event).put(r.counts_pending);
        out.append(t.take());
    }
    return out;
}

py::list combine_calls(const std::vector<std::shared_ptr<Runtime>>& rts, const py::list& calls) {
    std::vector<CombineArgs> args;
    for (const auto& c : calls) {
        const TupleReader t(c.ptr(), 20);
        CombineArgs a;
        a.x = t.tensor(0);
        a.topk_weights = t.maybe_tensor(1);
        a.bias0 = t.maybe_tensor(2);
        a.bias1 = t.maybe_tensor(3);
        a.recv_src_metadata = t.tensor(4);
        a.topk_idx = t.tensor(5);
        a.psum_rank = t.tensor(6);
        a.dst_slot = t.maybe_tensor(7);
        a.count_matrix = t.maybe_tensor(8);
        a.num_experts = t.integer(9);
        a.num_max_tokens = t.integer(10);
        a.num_sms = t.integer(11);
        a.do_expand = t.flag(12);
        a.weighted = t.flag(13);
        a.allow_multiple_reduction = t.flag(14);
        a.fuse_reduce = t.integer(15);
        a.sc.previous_event = t.event(16);
        a.sc.previous_event_before_epilogue = t.event(17);
        a.sc.async_with_compute_stream = t.flag(18);
        a.sc.allocate_on_comm_stream = t.flag(19);
        args.push_back(std::move(a));
    }
    std::vector<CombineResult> res;
    {
        py::gil_scoped_release release;
        res = Runtime::combine(rts, args);
    }
    py::list out;
    for (auto& r : res) {
        TupleWriter t(3);
        t.put(r.combined_x).put(r.combined_topk_weights).put(r.event);
        out.append(t.take());
    }
    return out;
}

}  // namespace

void register_extra_bindings(py::module_& m);   // low latency, AGRS, PP, ops (other translation units)

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.doc() = "B200-native expert-parallel communication runtime";

    py::register_exception<EPException>(m, "EPException");
    static py::exception<EPTimeoutError> timeout_exc(m, "EPTimeoutError");
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const EPTimeoutError& e) {
            timeout_exc(e.what());
        }
    });

    m.attr("MAX_RANKS") = kMaxRanks;
    m.attr("MAX_EXPERTS") = kMaxExperts;
    m.attr("MAX_LOCAL_EXPERTS") = kMaxLocalExperts;
    m.attr("MAX_TOPK") = kMaxTopk;
    m.attr("MAX_VRANKS") = kMaxVRanks;
    m.attr("HEAP_ALIGNMENT") = static_cast<int64_t>(kHeapAlignment);
    m.attr("CONTROL_BYTES") = static_cast<int64_t>(kCtlBytes);


    py::class_<EventHandle>(m, "EventHandle")
        .def(py::init<>())
        .def("record_again", &EventHandle::record_again)
        .def("current_stream_wait", &EventHandle::current_stream_wait);

    py::class_<Runtime, std::shared_ptr<Runtime>>(m, "Runtime")
        .def(py::init<int, int, int64_t, double, double, int64_t>(), py::arg("rank"), py::arg("num_ranks"), py::arg("num_bytes"),
             py::arg("gpu_timeout_secs") = 100.0, py::arg("cpu_timeout_secs") = 300.0, py::arg("num_cpu_bytes") = 0)
        .def("finish_export", &Runtime::finish_export)
        .def("heap_is_vmm", &Runtime::heap_is_vmm)
        .def_static("heap_backend_is_vmm", &Runtime::heap_backend_is_vmm)
        .def("destroy", &Runtime::destroy)
        .def("export_handle", [](const Runtime& rt) { return py::bytes(rt.export_handle()); })
        .def("open_peers", [](Runtime& rt, const std::vector<py::bytes>& handles) {
            std::vector<std::string> raw;
            for (const auto& h : handles) raw.push_back(static_cast<std::string>(h));
            rt.open_peers(raw);
        })
        .def_static("connect_local", &Runtime::connect_local)
        .def("status", &Runtime::status)
        .def("check_status", &Runtime::check_status)
        .def("clear_status", &Runtime::clear_status)
        .def("set_gpu_timeout", &Runtime::set_gpu_timeout)
        .def("enable_profiling", &Runtime::enable_profiling)
        .def("num_kernel_launches", &Runtime::num_kernel_launches)
        .def("last_timings", &Runtime::last_timings)
        .def("last_dispatch_phases", &Runtime::last_dispatch_phases)
        .def("last_timeline", &Runtime::last_timeline)
        .def("rank", &Runtime::rank)
        .def("num_ranks", &Runtime::num_ranks)
        .def("num_bytes", &Runtime::num_bytes)
        .def("num_device_sms", &Runtime::num_device_sms)
        .def("heap_tensor", &Runtime::heap_tensor)
        .def("comm_stream_ptr", [](const Runtime& rt) { return reinterpret_cast<uintptr_t>(rt.comm_stream().stream()); })
        .def("comm_stream_id", [](const Runtime& rt) {
            const auto s = rt.comm_stream();
            return std::make_tuple(static_cast<int64_t>(s.id()), static_cast<int64_t>(s.device_index()),
                                   static_cast<int64_t>(s.device_type()));
        })
        // (may synchronise a stream: without the GIL, see dispatch_calls)
        .def_static("barrier", &Runtime::barrier, py::arg("runtimes"), py::arg("use_comm_stream") = true, py::arg("with_cpu_sync") = false,
                    py::call_guard<py::gil_scoped_release>())
        .def("take_counts", &Runtime::take_counts, py::call_guard<py::gil_scoped_release>())
        .def_static("dispatch", &dispatch_calls)
        .def_static("combine", &combine_calls)
        .def_static("ht_buffer_size", &Runtime::ht_buffer_size);

    // A host-side wait of the given length without the GIL: what a driver does while it spins on the received counts
    // or synchronises a stream. Lets a CPU test check that Python threads (the heartbeat) keep running meanwhile.
    m.def("debug_blocking_host_wait", [](double seconds) {
        const auto end = std::chrono::steady_clock::now() + std::chrono::duration<double>(seconds);
        volatile uint64_t spins = 0;
        while (std::chrono::steady_clock::now() < end) ++spins;
        return static_cast<uint64_t>(spins);
    }, py::call_guard<py::gil_scoped_release>());

    register_extra_bindings(m);
}
