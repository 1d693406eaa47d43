// C ABI: tb200_reduce, tb200_version, tb200_sm_arch, tb200_workspace_status, tb200_workspace_watch, tb200_workspace_read.
#include "abi_common.cuh"
#include "thrust_b200/reduce.cuh"
#include <vector>

using namespace tb200_abi;

TB200_API int tb200_version(void) { return 100; }
TB200_API int tb200_sm_arch(void) { return 100; }

namespace {

// Pinned memory of a host thread: the block that an announced call's kernels write to (host_report), and room for copies of headers (a
// read-back into pageable memory is staged by the driver first).  A block whose call was never read may still be written to: it is
// retired, not used again, and freed with the thread once the device is idle.  When RETIRED_MAX blocks have gone that way the
// thread's calls are no longer announced.
struct pinned_headers {
  static constexpr size_t RETIRED_MAX = 16;
  struct retired_block { tb200::ws_header* p; int device; };
  tb200::ws_header* report = nullptr;
  tb200::ws_header* staging = nullptr;
  int device = 0;                    // on which the announced call's kernels run
  std::vector<retired_block> retired;

  static tb200::ws_header* get(tb200::ws_header*& p) {
    void* q = nullptr;
    if (!p && cudaHostAlloc(&q, sizeof(tb200::ws_header), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) p = static_cast<tb200::ws_header*>(q);
    else if (!p) cudaGetLastError();
    return p;
  }
  // The block for reports: kernels reach it under its host address (one address space of host and devices; without that there is no block).
  tb200::ws_header* report_block() {
    if (report || !get(report)) return report;
    void* mapped = nullptr;
    if (cudaHostGetDevicePointer(&mapped, report, 0) != cudaSuccess || mapped != report) { cudaGetLastError(); cudaFreeHost(report); report = nullptr; }
    return report;
  }
  void retire() { retired.push_back({report, device}); report = nullptr; }
  ~pinned_headers() {
    if (tb200::thread_report().bytes) retire();
    if (staging) cudaFreeHost(staging);
    if (report) cudaFreeHost(report);
    int current = 0;
    if (retired.empty() || cudaGetDevice(&current) != cudaSuccess) return;
    for (const retired_block& b : retired)
      if (cudaSetDevice(b.device) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess) cudaFreeHost(b.p);
    cudaSetDevice(current);
  }
};
thread_local pinned_headers pinned;

// The announcement ends; a block that kernels may still write to is put aside.
void end_announcement() {
  tb200::host_report& r = tb200::thread_report();
  if (r.bytes) pinned.retire();
  r = tb200::host_report();
}

// What the announced call has left in the block, once the stream is idle, as part of the header that was read to h_dst
void overlay_report(void* h_dst, size_t bytes) {
  const tb200::host_report& r = tb200::thread_report();
  if (bytes >= sizeof(unsigned) && r.block->error != tb200::ERR_NONE) memcpy(h_dst, &r.block->error, sizeof(unsigned));
}

}  // namespace

void tb200_abi::call_begins(const void*) {
  tb200::host_report& r = tb200::thread_report();
  if (r.begun) end_announcement();
  else r.begun = true;
}

TB200_API int tb200_workspace_status(const void* d_ws, tb200_stream_t stream, unsigned* h_status) {
  if (!d_ws || !h_status) return ERR_INVALID;
  cudaError_t e = cudaMemcpyAsync(h_status, d_ws, sizeof(unsigned), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  const tb200::host_report& r = tb200::thread_report();
  if (e == cudaSuccess && r.bytes && r.ws == d_ws) overlay_report(h_status, sizeof(unsigned));
  return (int)e;
}

TB200_API int tb200_workspace_watch(const void* d_ws) {
  end_announcement();
  if (!d_ws || pinned.retired.size() >= pinned_headers::RETIRED_MAX || cudaGetDevice(&pinned.device) != cudaSuccess) return 0;
  tb200::ws_header* const block = pinned.report_block();
  if (!block) return 0;
  memset(block, 0, sizeof(*block));
#ifdef TB200_TEST_HOOKS
  block->flags = tb200::test_hook_flags() & 3u;
#endif
  tb200::host_report& r = tb200::thread_report();
  r.ws = d_ws;
  r.block = block;
  return 0;
}

TB200_API int tb200_workspace_read(const void* d_ws, size_t bytes, void* h_dst, tb200_stream_t stream) {
  if (!d_ws || !h_dst || bytes > sizeof(tb200::ws_header)) return ERR_INVALID;
  tb200::host_report& r = tb200::thread_report();
  const bool announced = r.bytes && r.ws == d_ws;
  const void* from = announced ? r.block : nullptr;
  cudaError_t e = cudaSuccess;
  if (!announced || bytes > r.bytes) {           // more than the announced call's kernels leave in the block
    from = pinned_headers::get(pinned.staging);
    e = cudaMemcpyAsync(from ? pinned.staging : h_dst, d_ws, bytes, cudaMemcpyDeviceToHost, stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess && from) memcpy(h_dst, from, bytes);
  if (r.ws != d_ws) return (int)e;               // another workspace's announcement stands
  if (e != cudaSuccess) { end_announcement(); return (int)e; }
  if (announced) {
    overlay_report(h_dst, bytes);
    // a later look at the workspace finds an error there too
    if (r.block->error != tb200::ERR_NONE && cudaMemcpyAsync(const_cast<void*>(d_ws), r.block, sizeof(unsigned), cudaMemcpyHostToDevice, stream) == cudaSuccess)
      e = cudaStreamSynchronize(stream);
  }
  r = tb200::host_report();
  return (int)e;
}

namespace {

template <class In, class Acc>
int reduce_typed(const void* d_in, size_t n, int op, const void* h_init, void* d_out, void* d_ws, size_t* ws_bytes, cudaStream_t stream) {
  int rc;
  if (workspace_gate(d_ws, ws_bytes, tb200::reduce_workspace_bytes<Acc>(), rc)) return rc;
  if (!h_init || !d_out || (n && !d_in)) return ERR_INVALID;
  Acc init; memcpy(&init, h_init, sizeof(Acc));
  return by_op(op, [&](auto o) {
    return (int)tb200::reduce_async(static_cast<const In*>(d_in), n, init, o, static_cast<Acc*>(d_out), d_ws, stream);
  });
}

}  // namespace

TB200_API int tb200_reduce(const void* d_in, size_t n, int in_t, int acc_t, int op, const void* h_init, void* d_out, void* d_ws,
                           size_t* ws_bytes, tb200_stream_t stream) {
#define CASE(ti, In, ta, Acc) \
  if (in_t == ti && acc_t == ta) return reduce_typed<In, Acc>(d_in, n, op, h_init, d_out, d_ws, ws_bytes, stream);
  CASE(TB200_I8, int8_t, TB200_I32, int32_t) CASE(TB200_I8, int8_t, TB200_I64, long long)
  CASE(TB200_I16, int16_t, TB200_I32, int32_t) CASE(TB200_I16, int16_t, TB200_I64, long long)
  CASE(TB200_I32, int32_t, TB200_I32, int32_t) CASE(TB200_I32, int32_t, TB200_I64, long long)
  CASE(TB200_U8, uint8_t, TB200_U32, uint32_t) CASE(TB200_U8, uint8_t, TB200_U64, unsigned long long)
  CASE(TB200_U16, uint16_t, TB200_U32, uint32_t) CASE(TB200_U16, uint16_t, TB200_U64, unsigned long long)
  CASE(TB200_U32, uint32_t, TB200_U32, uint32_t) CASE(TB200_U32, uint32_t, TB200_U64, unsigned long long)
  CASE(TB200_I64, long long, TB200_I64, long long) CASE(TB200_U64, unsigned long long, TB200_U64, unsigned long long)
  CASE(TB200_F32, float, TB200_F32, float) CASE(TB200_F32, float, TB200_F64, double)
  CASE(TB200_F64, double, TB200_F64, double)
#undef CASE
  return ERR_UNSUPPORTED;
}
