// Python bindings (torch extension module fast_b200._C): symmetric heap, status blocks, and the
// launchers of every sm_100a kernel. Takes the place of the reference's TORCH_LIBRARY class
// flash_comm_t (nvidia/alltoall_nvshmem.cpp:390-662) and pybind module flash_t
// (amd/flash.cpp:650-666); the user-facing API built on top lives in fast_b200/parallel.
#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <algorithm>
#include <memory>

#include "py_types.h"

namespace py = pybind11;
using namespace fastb;
using namespace fastb_py;

namespace {


// ---- a2a program ----------------------------------------------------------------------------------
struct A2AProgramPy {
  torch::Tensor program_dev;     // the work list, then the expected rail bytes from rail_off on
  int64_t rail_off = 0;
  int n_items = 0, num_stages = 0;
  bool has_waits = false;  // some item waits for bytes another item of a peer's (or this) launch forwards
  unsigned long long expect_output = 0, expect_balance = 0;
  int64_t total_bytes = 0, largest_item = 0;
  int64_t input_bytes = 0, output_bytes = 0;  // what the rank's input and output hold (set by the owner, checked by the group launch)
  // The list goes up in order on the stream that is current when the schedule is made, `home`; launches may be on any stream.
  c10::cuda::CUDAStream home;
  mutable at::cuda::CUDAEvent upload;
  mutable bool uploaded = false;   // the upload was seen complete: launches have nothing to wait for any more

  // items: int64[k, 10] as produced by Plan.lower(); expect_rail: list of bytes per stage.
  A2AProgramPy(torch::Tensor items, const std::vector<int64_t>& expect_rail, int64_t exp_out, int64_t exp_bal, int device)
      : home(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device))) {
    TORCH_CHECK(items.dim() == 2 && items.size(1) == 10 && items.dtype() == torch::kInt64 && items.is_cpu(), "items must be CPU int64[k, 10]");
    TORCH_CHECK(static_cast<int>(expect_rail.size()) <= kSigMaxStages, "too many stages for the signal block");
    c10::cuda::CUDAGuard g(static_cast<c10::DeviceIndex>(device));
    // Captured, the upload would be read again at every replay from host memory that is somebody else's by then.
    TORCH_CHECK(!capturing(), "a schedule cannot be made while its stream is being captured: make it before the capture");
    n_items = static_cast<int>(items.size(0));
    num_stages = static_cast<int>(expect_rail.size());
    expect_output = static_cast<unsigned long long>(exp_out);
    expect_balance = static_cast<unsigned long long>(exp_bal);
    // Work list and expected rail bytes go up in one copy from pinned memory, in stream order: nothing here waits for the GPU.
    const int64_t list_bytes = std::max<int64_t>(n_items, 1) * static_cast<int64_t>(sizeof(A2AWork)), all_bytes = list_bytes + std::max(num_stages, 1) * 8;
    const auto u8 = torch::TensorOptions().dtype(torch::kUInt8);
    auto host = torch::empty({all_bytes}, u8.pinned_memory(true));   // given back once the copy is done, see below
    A2AWork* w = reinterpret_cast<A2AWork*>(host.data_ptr());
    auto it = items.contiguous();
    const int64_t* q = it.data_ptr<int64_t>();
    int64_t total = 0, largest = 0, waits = 0;   // locals: stores through w could alias the members
    for (int i = 0, n = n_items; i < n; ++i, q += 10) {
      A2AWork x;
      x.src_off = q[0]; x.dst_off = q[1]; x.bytes = q[2]; x.dst_rank = static_cast<int>(q[3]);
      x.src_buf = static_cast<unsigned char>(q[4]); x.dst_buf = static_cast<unsigned char>(q[5]);
      x.wait_kind = static_cast<unsigned char>(q[6]); x.signal_kind = static_cast<unsigned char>(q[7]);
      x.stage = static_cast<int>(q[8]); x.wait_stage = static_cast<int>(q[9]); x.pad_ = 0;
      total += q[2];
      largest = std::max(largest, q[2]);
      waits |= q[6];
      w[i] = x;
    }
    total_bytes = total; largest_item = largest; has_waits = waits != 0;
    std::copy(expect_rail.begin(), expect_rail.end(), reinterpret_cast<int64_t*>(host.data_ptr<uint8_t>() + list_bytes));
    program_dev = torch::empty({all_bytes}, u8.device(torch::kCUDA, device));
    // The copy itself, and the note that the host block is in use until it is done: what Tensor::copy_ does, without its dispatch.
    cuda_check(cudaMemcpyAsync(program_dev.data_ptr(), host.data_ptr(), static_cast<size_t>(all_bytes), cudaMemcpyHostToDevice, home.stream()), "work list upload");
    at::getHostAllocator(at::kCUDA)->record_event(host.data_ptr(), host.storage().data_ptr().get_context(), home.unwrap());
    upload.record(home);
    rail_off = list_bytes;
  }

  static bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

  // Called before a launch on `stream` (the current one; `captured`: it is being captured): the launch comes after the upload, and
  // the list's memory is not given to anybody else before the launch has ended, also when the schedule is dropped earlier. On the
  // stream of the upload itself both hold as they are.
  void ready_on(c10::cuda::CUDAStream stream, bool captured) const {
    if (!uploaded && (captured || stream != home)) {
      c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);   // a capture elsewhere does not mind the query
      if (upload.query()) uploaded = true;
      else if (captured) { upload.synchronize(); uploaded = true; }   // a captured launch cannot wait for an event from outside of its graph
      else upload.block(stream);
    }
    if (stream != home) c10::cuda::CUDACachingAllocator::recordStream(program_dev.storage().data_ptr(), stream);
  }

  A2ARankArgs args(const HeapPy& heap, std::array<int64_t, 4> src_ptrs, std::array<int64_t, 4> dst_offs, int64_t sig_off,
                   uint64_t epoch, const StatusPy& st, uint64_t timeout_ns, int64_t stamps_ptr = 0) const {
    A2ARankArgs a{};
    a.items = reinterpret_cast<const A2AWork*>(program_dev.data_ptr());
    a.n_items = n_items; a.rank = heap.h->rank(); a.world = heap.h->world(); a.num_stages = num_stages;
    // Slices of 128 KiB (two passes of the copy loop: 512 threads x 8 x 16 bytes each), at most 16 per item.
    a.slice_bytes = std::max<int64_t>(128 << 10, (largest_item / 16 + 0xFFFF) & ~int64_t{0xFFFF});
    a.split = static_cast<int>(std::max<int64_t>(1, (largest_item + a.slice_bytes - 1) / a.slice_bytes));
    a.peer_table = heap.h->device_peer_table();
    for (int i = 0; i < 4; ++i) { a.src_base[i] = reinterpret_cast<const unsigned char*>(src_ptrs[i]); a.dst_heap_off[i] = dst_offs[i]; }
    a.sig_heap_off = sig_off; a.epoch = epoch; a.expect_output = expect_output; a.expect_balance = expect_balance;
    a.expect_rail = reinterpret_cast<const unsigned long long*>(program_dev.data_ptr<uint8_t>() + rail_off);
    a.status = st.d; a.timeout_ns = timeout_ns;
    a.phase_stamps = reinterpret_cast<unsigned long long*>(stamps_ptr);
    return a;
  }
};

void a2a_launch(const A2AProgramPy& p, const HeapPy& heap, std::array<int64_t, 4> src_ptrs, std::array<int64_t, 4> dst_offs,
                int64_t sig_off, uint64_t epoch, const StatusPy& st, uint64_t timeout_ns, int ctas, int threads, int64_t stamps_ptr, bool bulk) {
  TORCH_CHECK(heap.h->world() <= kSigMaxWorld, "world larger than the signal block supports");
  A2ARankArgs a = p.args(heap, src_ptrs, dst_offs, sig_off, epoch, st, timeout_ns, stamps_ptr);
  a.bulk = bulk ? 1 : 0;
  p.ready_on(c10::cuda::getCurrentCUDAStream(), !p.uploaded && A2AProgramPy::capturing());
  cuda_check(launch_a2a_push(a, ctas, threads, cur_stream(), p.has_waits), "a2a_push launch");
}

// One cooperative launch that runs every virtual rank of an in-process group. Outputs lie in the ranks' heaps at one common
// offset (else nothing is launched and the answer is false: the caller stages them); the checks of sizes are made here, so
// that a small collective is not paid for in interpreter time. stage_offs: heap offsets of the balance and rail areas.
// The ranks' heaps and status blocks are handed over once; the status blocks, which kernels write to, live as long as the group, the heaps
// are not kept alive (a closed communicator lets go of its slab).
struct A2AGroupPy {
  std::vector<std::weak_ptr<SymmHeap>> heaps;
  std::vector<std::shared_ptr<StatusPy>> statuses;
  A2AGroupPy(const std::vector<const HeapPy*>& hs, std::vector<std::shared_ptr<StatusPy>> sts) : statuses(std::move(sts)) {
    TORCH_CHECK(hs.size() == statuses.size(), "one heap and one status block per virtual rank");
    for (const HeapPy* h : hs) heaps.push_back(h->h);
  }
};
bool a2a_launch_group(const A2AGroupPy& group, const std::vector<const A2AProgramPy*>& progs, const std::vector<torch::Tensor>& outs, const std::vector<torch::Tensor>& ins,
                      std::array<int64_t, 2> stage_offs, int64_t sig_off, uint64_t epoch, uint64_t timeout_ns, int ctas, int threads) {
  const size_t n = progs.size();
  const std::vector<std::shared_ptr<StatusPy>>& sts = group.statuses;
  std::array<HeapPy, kSigMaxWorld> locked{};
  std::array<const HeapPy*, kSigMaxWorld> heaps{};
  TORCH_CHECK(n <= group.heaps.size() && n <= static_cast<size_t>(kSigMaxWorld), "one entry per virtual rank");
  for (size_t r = 0; r < n; ++r) {
    locked[r].h = group.heaps[r].lock();
    if (!locked[r].h) throw std::runtime_error("communicator is closed");
    heaps[r] = &locked[r];
  }
  TORCH_CHECK(n >= 1 && group.heaps.size() == n && outs.size() == n && ins.size() == n,
              "one entry per virtual rank");
  std::array<int64_t, 4> dst{0, 0, stage_offs[0], stage_offs[1]};
  std::array<A2ARankArgs, kSigMaxWorld> host;
  int most = 1;
  for (size_t r = 0; r < n; ++r) {
    const int64_t base = reinterpret_cast<int64_t>(heaps[r]->h->local_base());
    const int64_t out = reinterpret_cast<int64_t>(outs[r].data_ptr()), out_bytes = static_cast<int64_t>(outs[r].nbytes());
    if (out < base || out + out_bytes > base + static_cast<int64_t>(heaps[r]->h->bytes())) return false;
    if (r == 0) dst[1] = out - base;
    if (static_cast<int64_t>(ins[r].nbytes()) < progs[r]->input_bytes) throw py::value_error("input smaller than the schedule needs");
    if (out_bytes < progs[r]->output_bytes) throw py::value_error("output smaller than the schedule needs");
    if (out - base != dst[1]) throw std::runtime_error("virtual ranks disagree on symmetric offsets; allocate in the same order on every rank");
    most = std::max(most, progs[r]->n_items);
  }
  for (size_t r = 0; r < n; ++r) {
    const int64_t base = reinterpret_cast<int64_t>(heaps[r]->h->local_base());
    host[r] = progs[r]->args(*heaps[r], {reinterpret_cast<int64_t>(ins[r].data_ptr()), 0, base + dst[2], base + dst[3]}, dst, sig_off, epoch, *sts[r], timeout_ns);
  }
  const auto stream = c10::cuda::getCurrentCUDAStream();
  const bool captured = std::any_of(progs.begin(), progs.end(), [](const A2AProgramPy* p) { return !p->uploaded; }) && A2AProgramPy::capturing();
  for (const A2AProgramPy* p : progs) p->ready_on(stream, captured);
  // A rank with a handful of work items needs a handful of CTAs (every launched CTA takes a turn at the exit counter).
  cuda_check(launch_a2a_push_group(host.data(), static_cast<int>(n), std::min(ctas, most), threads, cur_stream()), "a2a_push group launch");
  return true;
}

}  // namespace

void bind_moe(py::module_& m);  // defined in moe_bindings.cpp

PYBIND11_MODULE(_C, m) {
  m.doc() = "fast_b200 native runtime and sm_100a kernels";
  m.attr("SIG_WORDS") = kSigWords;

  py::class_<HeapPy>(m, "SymmHeap")
      .def(py::init([](int rank, int world, int64_t bytes, int device) {
        c10::cuda::CUDAGuard g(device);
        return HeapPy{std::make_shared<SymmHeap>(rank, world, static_cast<size_t>(bytes)), device};
      }))
      .def_static("create_local_group", [](int world, int64_t bytes, int device) {
        c10::cuda::CUDAGuard g(device);
        std::vector<HeapPy> out;
        for (SymmHeap* h : SymmHeap::create_local_group(world, static_cast<size_t>(bytes))) out.push_back(HeapPy{std::shared_ptr<SymmHeap>(h), device});
        return out;
      })
      .def_static("create_device_group", [](std::vector<int> devices, int64_t bytes) {
        std::vector<HeapPy> out;
        auto hs = SymmHeap::create_device_group(devices, static_cast<size_t>(bytes));
        for (size_t r = 0; r < hs.size(); ++r) out.push_back(HeapPy{std::shared_ptr<SymmHeap>(hs[r]), devices[r]});
        return out;
      })
      .def("ipc_handle", [](const HeapPy& h) { return py::bytes(h.h->ipc_handle()); })
      .def("open_peers", [](HeapPy& h, std::vector<std::string> handles) { c10::cuda::CUDAGuard g(h.device); h.h->open_peers(handles); })
      .def("close_peers", [](HeapPy& h) { c10::cuda::CUDAGuard g(h.device); h.h->close_peers(); })
      .def("alloc", [](HeapPy& h, int64_t bytes) { return static_cast<int64_t>(h.h->alloc(static_cast<size_t>(bytes))); })
      .def("free", [](HeapPy& h, int64_t off) { h.h->free(static_cast<size_t>(off)); })
      .def("tensor", &HeapPy::tensor)
      .def("base_ptr", [](const HeapPy& h, int r) { return reinterpret_cast<int64_t>(h.h->peer_base(r)); })
      .def("table_ptr", [](const HeapPy& h) { return reinterpret_cast<int64_t>(h.h->device_peer_table()); })
      .def_property_readonly("rank", [](const HeapPy& h) { return h.h->rank(); })
      .def_property_readonly("world", [](const HeapPy& h) { return h.h->world(); })
      .def_property_readonly("bytes", [](const HeapPy& h) { return static_cast<int64_t>(h.h->bytes()); })
      .def_property_readonly("in_use", [](const HeapPy& h) { return static_cast<int64_t>(h.h->in_use()); });

  py::class_<StatusPy, std::shared_ptr<StatusPy>>(m, "StatusBlock")
      .def(py::init<>())
      .def("read", &StatusPy::read)
      .def("clear", &StatusPy::clear)
      .def("ptr", [](const StatusPy& s) { return reinterpret_cast<int64_t>(s.d); });

  py::class_<A2AProgramPy>(m, "A2AProgram")
      .def(py::init<torch::Tensor, std::vector<int64_t>, int64_t, int64_t, int>())
      .def_readwrite("input_bytes", &A2AProgramPy::input_bytes)
      .def_readwrite("output_bytes", &A2AProgramPy::output_bytes)
      .def_readonly("n_items", &A2AProgramPy::n_items)
      .def_readonly("num_stages", &A2AProgramPy::num_stages)
      .def_readonly("has_waits", &A2AProgramPy::has_waits)
      .def_readonly("total_bytes", &A2AProgramPy::total_bytes);

  m.def("a2a_launch", &a2a_launch, py::arg("program"), py::arg("heap"), py::arg("src_ptrs"), py::arg("dst_offs"), py::arg("sig_off"), py::arg("epoch"),
        py::arg("status"), py::arg("timeout_ns"), py::arg("ctas"), py::arg("threads"), py::arg("stamps_ptr") = 0, py::arg("bulk") = false);
  m.attr("PHASE_STAMP_WORDS") = kPhaseStampWords;
  m.attr("SIG_MAX_WORLD") = kSigMaxWorld;
  py::class_<A2AGroupPy>(m, "A2AGroup").def(py::init<const std::vector<const HeapPy*>&, std::vector<std::shared_ptr<StatusPy>>>());
  m.def("a2a_launch_group", &a2a_launch_group);
  m.def("wait_probe", [](int64_t flag_ptr, uint64_t want, const StatusPy& st, uint64_t timeout_ns) {
    cuda_check(launch_wait_probe(reinterpret_cast<const unsigned long long*>(flag_ptr), want, st.d, timeout_ns, cur_stream()), "wait_probe");
  });
  m.def("launch_count", &launch_count);
  bind_moe(m);
}
