// Single-pass device-wide reduction for sm_100a.
//
// Small inputs: one launch of one cluster, whose CTAs store their totals into the first one's shared memory; nothing to clear.  A call
// and the wait for it: 1000 int32 9.8 us against 12.5 with partials, ticket and clearing launch, 65 k 11.5 against 13.0, 131 k
// 11.8 against 13.4.  reduce_cluster says where it ends.  Larger inputs:
// One launch: a grid sized to the SM count streams the input with 16-byte evict-first loads
// (four in flight per thread), folds it with warp shuffles, and the last CTA to finish (found
// with an atomic ticket) folds the per-CTA partials and `init` into the result.  Replaces the
// two-kernel cub::DispatchReduce call of thrust/system/cuda/detail/reduce.h:946-983.
// Like that path it needs an associative and commutative operator.
#pragma once
#include "cluster.cuh"
#include "common.cuh"

namespace tb200 {

constexpr int REDUCE_BLOCK = 256;
constexpr int REDUCE_UNROLL = 4;
constexpr int REDUCE_UNROLL_GENERIC = 16;
constexpr int REDUCE_CTAS_PER_SM = 4;
constexpr int REDUCE_MAX_GRID = 4096;

template <class AccT, class Op>
__device__ __forceinline__ opt<AccT> block_reduce_opt(opt<AccT> x, Op op, opt<AccT>* smem /*[32]*/) {
  const int lane = lane_id(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  x = warp_reduce_opt(x, op);
  if (lane == 0) smem[warp] = x;
  __syncthreads();
  opt<AccT> r; r.has = false;
  if (warp == 0) {
    if (lane < nwarps) r = smem[lane];
    r = warp_reduce_opt(r, op);
  }
  return r;  // valid in thread 0
}

// Up to how many vectors (or items behind an iterator) one cluster of up to 16 CTAs does it, without partials, ticket and the launch that
// clears them, and how many of them a thread takes: one where a step may cost something (an iterator that computes or gathers, a caller's
// operator), which is what the grid gives it too; as many as are read at a time where it is an addition or a comparison, up to 512 KB.
// A transform of 2000 dependent multiply-adds, a call and the wait for it, here / when 16 items a thread and 512 KB went for all: 4000 items
// 15 us / 77, 65 k 18 / 78, 131 k 23 / 145; item & 7 behind an iterator 65 k 13.6 / 11.5 (the grid then clears its header first).
template <class AccT, class Op, int VEC> struct reduce_cluster {
  static constexpr bool SHORT_STEP = VEC > 0 && std::is_arithmetic<AccT>::value &&
                                     (std::is_same<Op, plus_op>::value || std::is_same<Op, min_op>::value || std::is_same<Op, max_op>::value);
  static constexpr size_t MOST = SHORT_STEP ? ((size_t)1 << 19) / sizeof(vec16) : (size_t)CLUSTER_MAX_CTAS * REDUCE_BLOCK;
  static constexpr int ROWS = SHORT_STEP ? (int)(MOST / (CLUSTER_MAX_CTAS * REDUCE_BLOCK)) : 1;   // what a thread takes at most
  static_assert((size_t)ROWS * CLUSTER_MAX_CTAS * REDUCE_BLOCK == MOST, "whole rows");
  static constexpr size_t PER_CTA = (size_t)REDUCE_BLOCK * (SHORT_STEP ? REDUCE_UNROLL : 1);
};

// In = element type read from memory (or an iterator's value), AccT = accumulator.
// VEC = elements per 16-byte load when `in` is a 16-byte-aligned pointer to a 1/2/4/8-byte type,
// 0 for the generic path (any random-access iterator, one element per load).
template <class InIt, class AccT, class Op, int VEC>
__global__ void __launch_bounds__(REDUCE_BLOCK)
reduce_kernel(InIt in, size_t n, AccT init, Op op, AccT* partials, unsigned* partial_has,
              ws_header* hdr, AccT* out, AccT* rep_out, bool one_cluster) {
  using Cluster = reduce_cluster<AccT, Op, VEC>;
  if (one_cluster && gridDim.x > 1) cluster_arrive_started();
  TB200_SHARED_ARRAY(opt<AccT>, smem, 32);
  __shared__ bool is_last;
  const size_t tid = (size_t)blockIdx.x * REDUCE_BLOCK + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * REDUCE_BLOCK;
  opt<AccT> acc; acc.has = false;

  if constexpr (VEC > 0) {
    using In = typename std::remove_cv<typename std::remove_pointer<InIt>::type>::type;
    const size_t nvec = n / VEC;
    const vec16* vin = reinterpret_cast<const vec16*>(in);
    size_t v = tid;
    if constexpr (Cluster::ROWS > 1) {
      // Every vector a thread takes is in flight, and their sums are added up as a tree, which is what the grid's CTAs make of them.  Root mean
      // square of the relative error of uniform 4-byte floats, here / one after the other: 19 k 4.1e-8 / 5.7e-8, 60 k 3.2e-8 / 5.7e-8, 131 k
      // 4.3e-8 / 5.9e-8; a call and the wait 11.6 us / 11.9 at 131 k.
      if (one_cluster) {
        vec16 r[Cluster::ROWS];
        opt<AccT> row[Cluster::ROWS];
#pragma unroll
        for (int u = 0; u < Cluster::ROWS; ++u) {
          row[u].has = v + u * stride < nvec;
          if (row[u].has) r[u] = load_stream16(vin + v + u * stride);
        }
#pragma unroll
        for (int u = 0; u < Cluster::ROWS; ++u) {
          if (!row[u].has) continue;
          const In* e = reinterpret_cast<const In*>(&r[u]);
          AccT t = (AccT)e[0];
#pragma unroll
          for (int k = 1; k < VEC; ++k) t = op(t, (AccT)e[k]);
          row[u].v = t;
        }
#pragma unroll
        for (int d = 1; d < Cluster::ROWS; d <<= 1) {
#pragma unroll
          for (int u = 0; u + d < Cluster::ROWS; u += 2 * d) row[u].append_opt(row[u + d], op);
        }
        acc = row[0];
        v = nvec;
      }
    }
    for (; v + (REDUCE_UNROLL - 1) * stride < nvec; v += REDUCE_UNROLL * stride) {
      vec16 r[REDUCE_UNROLL];
#pragma unroll
      for (int u = 0; u < REDUCE_UNROLL; ++u) r[u] = load_stream16(vin + v + u * stride);
#pragma unroll
      for (int u = 0; u < REDUCE_UNROLL; ++u) {
        const In* e = reinterpret_cast<const In*>(&r[u]);
        AccT t = (AccT)e[0];
#pragma unroll
        for (int k = 1; k < VEC; ++k) t = op(t, (AccT)e[k]);
        acc.append(t, op);
      }
    }
    for (; v < nvec; v += stride) {
      vec16 r = load_stream16(vin + v);
      const In* e = reinterpret_cast<const In*>(&r);
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc.append((AccT)e[k], op);
    }
    // ragged tail (fewer than VEC elements)
    size_t t = nvec * VEC + tid;
    if (t < n) acc.append((AccT)in[t], op);
  } else {
    // one element per load: sixteen of them in flight per thread keep as many bytes on their way as
    // the four 16-byte loads of the vector path (a transform_iterator over 4-byte items, say)
    constexpr int U = REDUCE_UNROLL_GENERIC;
    size_t i = tid;
    for (; i + (U - 1) * stride < n; i += U * stride) {
      AccT r[U];
#pragma unroll
      for (int u = 0; u < U; ++u) r[u] = (AccT)in[i + u * stride];
      AccT t = r[0];
#pragma unroll
      for (int u = 1; u < U; ++u) t = op(t, r[u]);
      acc.append(t, op);
    }
    for (; i < n; i += stride) acc.append((AccT)in[i], op);
  }

  if constexpr (cluster_storable<AccT>::value) {
    if (one_cluster) {   // a header that nobody has cleared (`out` may lie behind its first fields); the CTAs' totals travel to the first one
      __shared__ __align__(16) unsigned char totals_raw[CLUSTER_MAX_CTAS * sizeof(AccT)];
      __shared__ unsigned has_total[CLUSTER_MAX_CTAS];
      AccT* const totals = reinterpret_cast<AccT*>(totals_raw);
      if (blockIdx.x == 0 && threadIdx.x < sizeof(ws_header) / 4) reinterpret_cast<unsigned*>(hdr)[threadIdx.x] = 0;
      opt<AccT> all = block_reduce_opt(acc, op, smem);
      if (gridDim.x > 1) {
        cluster_wait_started();
        if (threadIdx.x == 0) {
          if (all.has) cluster_store(cluster_addr(smem_addr(totals + blockIdx.x), 0), all.v);
          cluster_store(cluster_addr(smem_addr(has_total + blockIdx.x), 0), (unsigned)all.has);
        }
        cluster_barrier();
        all.has = false;
        if (blockIdx.x == 0 && threadIdx.x < 32) {
          if (threadIdx.x < gridDim.x && has_total[threadIdx.x]) { all.v = totals[threadIdx.x]; all.has = true; }
          all = warp_reduce_opt(all, op);
        }
      }
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const AccT result = all.has ? op(init, all.v) : init;
        *out = result;
        if (rep_out) *rep_out = result;
      }
      return;
    }
  }
  opt<AccT> blk = block_reduce_opt(acc, op, smem);
  if (threadIdx.x == 0) {
    if (blk.has) partials[blockIdx.x] = blk.v;
    partial_has[blockIdx.x] = blk.has;
    __threadfence();
    unsigned t = atomicAdd(&hdr->ticket, 1u);
    is_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  opt<AccT> f; f.has = false;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += REDUCE_BLOCK) {
    if (__ldcg(partial_has + b)) f.append(load_cg_any(partials + b), op);
  }
  __syncthreads();
  f = block_reduce_opt(f, op, smem);
  if (threadIdx.x == 0) {
    const AccT result = f.has ? op(init, f.v) : init;
    *out = result;
    if (rep_out) *rep_out = result;
    hdr->ticket = 0;
  }
}

inline int reduce_grid(size_t work_items /* vectors or elements */) {
  const device_info& di = current_device_info();
  size_t want = (work_items + REDUCE_BLOCK - 1) / REDUCE_BLOCK;
  size_t cap = (size_t)di.sm_count * REDUCE_CTAS_PER_SM;
  if (cap > REDUCE_MAX_GRID) cap = REDUCE_MAX_GRID;
  if (want < 1) want = 1;
  return (int)(want < cap ? want : cap);
}

template <class AccT> size_t reduce_workspace_bytes() {
  return sizeof(ws_header) + align_up(REDUCE_MAX_GRID * sizeof(AccT), 256) + align_up(REDUCE_MAX_GRID * 4, 256) +
         align_up(sizeof(AccT), 256);
}

// Launches the reduction on `stream`; the result lands in *d_out (device memory).  No sync.
// `ws` must hold reduce_workspace_bytes<AccT>().  n == 0 writes init.
template <class InIt, class AccT, class Op>
cudaError_t reduce_async(InIt in, size_t n, AccT init, Op op, AccT* d_out, void* ws, cudaStream_t stream) {
  char* base = static_cast<char*>(ws);
  ws_header* hdr = reinterpret_cast<ws_header*>(base);
  AccT* partials = reinterpret_cast<AccT*>(base + sizeof(ws_header));
  unsigned* has = reinterpret_cast<unsigned*>(base + sizeof(ws_header) + align_up(REDUCE_MAX_GRID * sizeof(AccT), 256));
  // a result behind the header's own fields is reported too (of 8 bytes at most; its room in the report is 8 bytes whatever its size)
  constexpr size_t RESULT = offsetof(ws_header, aux) + sizeof(unsigned long long);
  ws_header* const rep = sizeof(AccT) <= 8 && reinterpret_cast<char*>(d_out) == base + RESULT ? report_of(hdr, stream) : hdr;
  AccT* const rep_out = rep != hdr ? reinterpret_cast<AccT*>(reinterpret_cast<char*>(rep) + RESULT) : nullptr;
  auto with_result = [&](cudaError_t e) { return reported(e, rep, hdr, RESULT + 8); };
  auto launch = [&](auto vec_tag) -> cudaError_t {
    constexpr int VEC = decltype(vec_tag)::value;
    auto kern = reduce_kernel<InIt, AccT, Op, VEC>;
    const char* const name = VEC > 0 ? "reduce_kernel (16-byte loads)" : "reduce_kernel (generic iterator)";
    using Cluster = reduce_cluster<AccT, Op, VEC>;
    const size_t work_items = VEC > 0 ? n / (VEC > 0 ? VEC : 1) : n;
    timed_launch tl(KID_REDUCE, stream);
    if (cluster_storable<AccT>::value && work_items <= Cluster::MOST) {
      static thread_local unsigned largest[64] = {0};
      bool launched = false;
      unsigned ctas = cluster_ctas((work_items + Cluster::PER_CTA - 1) / Cluster::PER_CTA);
      if (ctas == 0) ctas = CLUSTER_MAX_CTAS;
      const cudaError_t e = cluster_launch(kern, ctas, REDUCE_BLOCK, 0, stream, largest, launched, in, n, init, op, partials, has, hdr, d_out, rep_out, true);
      if (launched) { with_result(e); log_launch(name, ctas, REDUCE_BLOCK, 0, n, stream); }
      if (launched || e != cudaSuccess) return e;
    }
    const cudaError_t e = cudaMemsetAsync(hdr, 0, sizeof(ws_header), stream);
    if (e != cudaSuccess) return e;
    const int grid = reduce_grid(work_items);
    kern<<<grid, REDUCE_BLOCK, 0, stream>>>(in, n, init, op, partials, has, hdr, d_out, rep_out, false);
    log_launch(name, grid, REDUCE_BLOCK, 0, n, stream);
    return with_result(cudaGetLastError());
  };
  if constexpr (std::is_pointer<InIt>::value) {
    using In = typename std::remove_cv<typename std::remove_pointer<InIt>::type>::type;
    if constexpr (std::is_arithmetic<In>::value && 16 % sizeof(In) == 0) {
      if (is_aligned16(in)) return launch(std::integral_constant<int, 16 / (int)sizeof(In)>());
    }
  }
  return launch(std::integral_constant<int, 0>());
}

}  // namespace tb200
