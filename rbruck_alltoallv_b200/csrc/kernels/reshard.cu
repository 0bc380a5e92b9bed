// Sequence <-> head re-sharding on one GPU: the uniform all-to-all of sequence-parallel attention with its pack (or
// unpack) folded in.  When one process hosts every rank a block needs neither a send buffer nor a copy descriptor:
// every element is read once from where the caller has it and written once to where the receiver wants it.
//
// Bound by HBM: two bytes of traffic per byte moved.  The exchange through a packed buffer moves every byte twice (a
// strided copy per rank, then the alltoallv), and for a few MB the launches of the per-rank copies dominate.  Measured on
// one B200, bf16, 32 heads of 128: 8 ranks x 512 positions to heads 92 -> 19 us (host-bound: views and pointer arrays);
// 4 ranks x 4096 positions back 270 -> 43 us (6.2 TB/s).
#include <cuda_runtime.h>

#include <cstdint>

#include "api/ctx_internal.h"
#include "kernels/primitives.cuh"
#include "rbv/device_types.h"
#include "rbv/reshard.h"

namespace rbv {
namespace {

constexpr int kReshardThreads = 256;

struct ReshardArgs {
  unsigned P, vp;                 // vp: vectors per piece
  unsigned row;                   // P * vp: vectors per sequence position on the sequence side
  long long seq, nvec;            // nvec = seq * row: vectors per rank
  char* heap[kMaxProcs];          // for the failure note only
  unsigned long long ctrl_off;
  StatusBlock* host_status;
  char* seq_side[kMaxRanks];
  char* head_side[kMaxRanks];
};

// blockIdx.y: rank r of the sequence side; blockIdx.x: tile of U * 256 consecutive vectors of its array.  The
// sequence side is walked linearly, so it is contiguous for the whole tile; the head side is contiguous per piece.
// All loads of a thread are issued before its first store.
template <typename V, int U, bool TO_HEAD>
__global__ void __launch_bounds__(kReshardThreads) reshard_kernel(const __grid_constant__ ReshardArgs a) {
  const unsigned r = blockIdx.y;
  const long long first = (long long)blockIdx.x * (U * kReshardThreads);
  const long long s0 = first / a.row;                       // one 64-bit division per tile; the rest is 32 bits
  const unsigned rem = (unsigned)(first - s0 * a.row);
  V* seq = reinterpret_cast<V*>(a.seq_side[r]) + first;
  V v[U];
  V* dst[U];
  #pragma unroll
  for (int j = 0; j < U; j++) {
    const unsigned t = (unsigned)j * kReshardThreads + threadIdx.x;
    dst[j] = nullptr;
    if (first + t < a.nvec) {
      const unsigned at = rem + t, ds = at / a.row, in_row = at - ds * a.row, q = in_row / a.vp;
      V* head = reinterpret_cast<V*>(a.head_side[q]) + ((long long)r * a.seq + s0 + ds) * a.vp + (in_row - q * a.vp);
      v[j] = TO_HEAD ? seq[t] : *head;
      dst[j] = TO_HEAD ? head : seq + t;
    }
  }
  #pragma unroll
  for (int j = 0; j < U; j++)
    if (dst[j]) *dst[j] = v[j];
  // like every call on a communicator that failed earlier and was not reset, say so
  if (blockIdx.x == 0 && r == 0 && threadIdx.x == 0) {
    CtrlBlock* my = reinterpret_cast<CtrlBlock*>(a.heap[0] + a.ctrl_off);
    if (dev::ld_relaxed_sys(&my->abort_flag))
      dev::note_failure(a.heap, 1, 0, a.ctrl_off, a.host_status, RBV_ERR_ABORTED, 0, 0, 0);
  }
}

template <typename V>
cudaError_t launch_reshard(const ReshardArgs& a, bool to_head, int sms, cudaStream_t st) {
  // 8 vectors per thread once that still leaves two tiles per SM: enough bytes in flight to run at HBM speed; below
  // that the exchange is a matter of latency and one vector per thread spreads it over all SMs.
  const long long deep = (a.nvec + 8 * kReshardThreads - 1) / (8 * kReshardThreads);
  const bool wide = deep * a.P >= 2ll * sms;
  const long long tiles = wide ? deep : (a.nvec + kReshardThreads - 1) / kReshardThreads;
  if (tiles > 0x7fffffffll) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)tiles, a.P);
  if (wide) {
    if (to_head) reshard_kernel<V, 8, true><<<grid, kReshardThreads, 0, st>>>(a);
    else reshard_kernel<V, 8, false><<<grid, kReshardThreads, 0, st>>>(a);
  } else {
    if (to_head) reshard_kernel<V, 1, true><<<grid, kReshardThreads, 0, st>>>(a);
    else reshard_kernel<V, 1, false><<<grid, kReshardThreads, 0, st>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace
}  // namespace rbv

extern "C" int rbv_reshard_heads(rbv_ctx_t ctx, const void* const* seq_side, const void* const* head_side,
                                 long long seq, long long piece_bytes, int to_head, void* stream) {
  using namespace rbv;
  if (!ctx || !ctx->c || !seq_side || !head_side) return (int)cudaErrorInvalidValue;
  const Context& c = *ctx->c;
  if (c.nproc() != 1 || c.P() > kMaxRanks || seq < 1 || piece_bytes < 1) return (int)cudaErrorInvalidValue;
  ReshardArgs a{};
  a.P = (unsigned)c.P();
  a.seq = seq;
  a.heap[0] = c.heap();
  a.ctrl_off = c.layout().ctrl_off;
  a.host_status = c.host_status_dev();
  // widest vector that divides a piece and every base address (pieces are packed, so all rows then are aligned too)
  uintptr_t bits = (uintptr_t)piece_bytes;
  for (int r = 0; r < c.P(); r++) {
    a.seq_side[r] = static_cast<char*>(const_cast<void*>(seq_side[r]));
    a.head_side[r] = static_cast<char*>(const_cast<void*>(head_side[r]));
    if (!a.seq_side[r] || !a.head_side[r]) return (int)cudaErrorInvalidValue;
    bits |= reinterpret_cast<uintptr_t>(seq_side[r]) | reinterpret_cast<uintptr_t>(head_side[r]);
  }
  const int w = (bits & 15) == 0 ? 16 : (bits & 7) == 0 ? 8 : (bits & 3) == 0 ? 4 : (bits & 1) == 0 ? 2 : 1;
  const long long vp = piece_bytes / w;
  if (vp * a.P > 0x7fffffffll - 8 * kReshardThreads) return (int)cudaErrorInvalidValue;   // 32-bit offsets inside a row
  a.vp = (unsigned)vp;
  a.row = (unsigned)(vp * a.P);
  a.nvec = seq * a.row;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (w) {
    case 16: return (int)launch_reshard<uint4>(a, to_head != 0, c.sm_count(), st);
    case 8: return (int)launch_reshard<uint2>(a, to_head != 0, c.sm_count(), st);
    case 4: return (int)launch_reshard<unsigned>(a, to_head != 0, c.sm_count(), st);
    case 2: return (int)launch_reshard<unsigned short>(a, to_head != 0, c.sm_count(), st);
    default: return (int)launch_reshard<unsigned char>(a, to_head != 0, c.sm_count(), st);
  }
}
