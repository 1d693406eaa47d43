// C ABI: tb200_reduce, tb200_version, tb200_sm_arch, tb200_workspace_status, tb200_workspace_watch, tb200_workspace_read.
#include "abi_common.cuh"
#include "thrust_b200/reduce.cuh"
#include <vector>

using namespace tb200_abi;

TB200_API int tb200_version(void) { return 100; }
TB200_API int tb200_sm_arch(void) { return 100; }

TB200_API int tb200_workspace_status(const void* d_ws, tb200_stream_t stream, unsigned* h_status) {
  if (!d_ws || !h_status) return ERR_INVALID;
  cudaError_t e = cudaMemcpyAsync(h_status, d_ws, sizeof(unsigned), cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return (int)e;
  return (int)cudaStreamSynchronize(stream);
}

namespace {

// One pinned header's worth per host thread, which kernels can write to (host_report) and copies can land in: a read-back into
// pageable memory is staged by the driver first.  give_up(): the block of a call that failed half-way may still be written to by what it
// did launch; it is not used again and freed with the thread.
struct pinned_header {
  tb200::ws_header* p = nullptr;
  std::vector<void*> old;
  tb200::ws_header* get() {
    void* q = nullptr;
    if (!p && cudaHostAlloc(&q, sizeof(tb200::ws_header), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) p = static_cast<tb200::ws_header*>(q);
    else if (!p) cudaGetLastError();
    return p;
  }
  void give_up() { old.push_back(p); p = nullptr; }
  ~pinned_header() { if (p) cudaFreeHost(p); for (void* q : old) cudaFreeHost(q); }
};
thread_local pinned_header pinned;

}  // namespace

TB200_API int tb200_workspace_watch(const void* d_ws) {
  tb200::host_report& r = tb200::thread_report();
  if (r.served) pinned.give_up();            // watched and launched, but never read
  r = tb200::host_report();
  if (!d_ws) return 0;
  tb200::ws_header* const block = pinned.get();
  void* mapped = nullptr;
  // (where the device sees the block at another address than the host, calls report through their workspaces)
  if (!block || cudaHostGetDevicePointer(&mapped, block, 0) != cudaSuccess || mapped != block) { cudaGetLastError(); return 0; }
  memset(block, 0, sizeof(*block));
#ifdef TB200_TEST_HOOKS
  block->flags = tb200::test_hook_flags() & 3u;
#endif
  r.ws = d_ws;
  r.block = block;
  return 0;
}

TB200_API int tb200_workspace_read(const void* d_ws, size_t bytes, void* h_dst, tb200_stream_t stream) {
  if (!d_ws || !h_dst || bytes > sizeof(tb200::ws_header)) return ERR_INVALID;
  tb200::host_report& r = tb200::thread_report();
  const bool there = r.served && r.ws == d_ws;   // the watched call's kernels write what is asked for to the block
  void* const via = pinned.get();
  cudaError_t e = there ? cudaSuccess : cudaMemcpyAsync(via ? via : h_dst, d_ws, bytes, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess && via) memcpy(h_dst, via, bytes);
  if (e != cudaSuccess && r.served) pinned.give_up();
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
