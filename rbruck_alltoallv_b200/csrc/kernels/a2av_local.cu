// Direct alltoallv among ranks that one process hosts, for calls whose counts are not resolved in advance: one-shot
// calls, and persistent calls with counts on the device.  Every rank's counts and displacements can be read where they
// are, so there is nothing to exchange before the data and nobody to wait for after it: each CTA reads the count matrix,
// cuts all blocks into chunks, and its warps copy their share; the end of the kernel is the completion.
//
// The dynamic kernel (a2av_kernel.cu), which serves the same calls across GPUs, publishes the counts into a table, polls
// the table until it is complete, walks an op list and counts arrivals; and a host that does not know the counts has to
// give it one chunk size for every call.  Here the chunk follows from the bytes that the call moves, so that they spread
// over all warps whatever the host knew.  Measured on one B200 (cold caches): counts on the device, 16 ranks, 17 MB in
// blocks of up to 64 KB 29 -> 11.5 us; 1 MB in blocks of up to 16 KB among 8 ranks 12.7 -> 9.2 us; 256 MB in
// blocks of up to 4 MB 124 -> 98 us (5.2 TB/s; 16 vectors per lane in flight move them 7 % faster than 8).
#include <cuda_runtime.h>

#include "kernels/primitives.cuh"
#include "rbv/context.h"
#include "rbv/device_types.h"

namespace rbv {
namespace {

constexpr int kLocalThreads = 512;

// Exclusive scan of one value per thread over the CTA; `total` receives the sum.  All threads take part.
__device__ __forceinline__ unsigned cta_scan(unsigned v, unsigned* s_warp, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned incl = v;
  #pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned n = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += n;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned w = lane < kLocalThreads / 32 ? s_warp[lane] : 0u;
    unsigned s = w;
    #pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned n = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += n;
    }
    s_warp[lane] = s - w;
    if (lane == 31) s_warp[32] = s;
  }
  __syncthreads();
  total = s_warp[32];
  return s_warp[warp] + incl - v;
}

}  // namespace

__global__ void __launch_bounds__(kLocalThreads, 1) a2av_local_kernel(const __grid_constant__ LocalArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* prefix = reinterpret_cast<unsigned*>(smem_raw);    // [P * P + 1] chunks before each pair's block
  __shared__ unsigned s_warp[33];
  __shared__ unsigned long long s_sum[kLocalThreads / 32];
  const int P = a.P, n = P * P, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* sc = a.inline_meta ? a.inl.sendcounts : a.sendcounts;
  const int* rc = a.inline_meta ? a.inl.recvcounts : a.recvcounts;
  const long long* sd = a.inline_meta ? a.inl.sdispls : a.sdispls;
  const long long* rd = a.inline_meta ? a.inl.rdispls : a.rdispls;

  // thread t owns the blocks [t * per, (t + 1) * per): bytes of each (a block larger than its slot is refused)
  const int per = (n + kLocalThreads - 1) / kLocalThreads;
  constexpr int kPer = kMaxRanks * kMaxRanks / kLocalThreads;
  unsigned long long bytes[kPer], mine = 0;
  #pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = tid * per + j;
    bytes[j] = 0;
    if (j < per && i < n) {
      const int s = i / P, d = i - s * P, c = sc[i];
      const int cap = rc ? rc[d * P + s] : -1;
      if (cap >= 0 && c > cap) {
        if (blockIdx.x == 0)
          dev::note_failure(a.heap, 1, 0, a.ctrl_off, a.host_status, RBV_ERR_TRUNCATE, 0, s, d);
      } else if (c > 0) {
        bytes[j] = (unsigned long long)c * (unsigned)a.type_size;
      }
      mine += bytes[j];
    }
  }
  unsigned long long total = mine;
  #pragma unroll
  for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if (lane == 0) s_sum[warp] = total;
  __syncthreads();
  total = 0;
  for (int w = 0; w < kLocalThreads / 32; w++) total += s_sum[w];

  // A chunk is one warp's unit of work: the bytes of the call over the warps of the grid, in a whole number of rounds of
  // at most 64 KB, and at least 2 KB (four vectors per lane; a warp's round of loads is 16, 8 KB).
  const unsigned nwarps = gridDim.x * (kLocalThreads / 32);
  unsigned long long chunk = a.chunk_bytes;
  if (!chunk) {
    const unsigned long long rounds = total / ((unsigned long long)nwarps << 16) + 1;
    chunk = (total + nwarps * rounds - 1) / (nwarps * rounds);
    chunk = chunk < 2048 ? 2048 : (chunk > 65536 ? 65536 : chunk);
    chunk = (chunk + 1023) & ~1023ull;
  }
  unsigned nch[kPer], mych = 0;
  #pragma unroll
  for (int j = 0; j < kPer; j++) {
    nch[j] = (unsigned)((bytes[j] + chunk - 1) / chunk);
    mych += nch[j];
  }
  unsigned items;
  unsigned before = cta_scan(mych, s_warp, items);
  #pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = tid * per + j;
    if (j < per && i < n) prefix[i] = before;
    before += nch[j];
  }
  if (tid == 0) prefix[n] = items;
  __syncthreads();

  // item c goes to warp c / grid of CTA c % grid: a small call runs on as many SMs as it has items
  int pair = 0;
  for (unsigned c = warp * gridDim.x + blockIdx.x; c < items; c += nwarps) {
    pair = dev::find_op(prefix, pair, n, c);
    const int s = pair / P, d = pair - s * P;
    const unsigned long long off = (unsigned long long)(c - prefix[pair]) * chunk;
    const unsigned long long len = min(chunk, (unsigned long long)sc[pair] * (unsigned)a.type_size - off);
    const char* src = a.sendbuf[s] + sd[pair] * a.type_size + off;
    char* dst = a.recvbuf[d] + rd[d * P + s] * a.type_size + off;
    dev::warp_copy<16>(dst, src, len, lane);
  }
  // a communicator that failed earlier and was not reset says so
  if (blockIdx.x == 0 && tid == kLocalThreads - 1) {
    CtrlBlock* my = reinterpret_cast<CtrlBlock*>(a.heap[0] + a.ctrl_off);
    if (dev::ld_relaxed_sys(&my->abort_flag))
      dev::note_failure(a.heap, 1, 0, a.ctrl_off, a.host_status, RBV_ERR_ABORTED, 0, 0, 0);
  }
}

cudaError_t a2av_local_launch(const LocalArgs& args, int grid, cudaStream_t stream) {
  a2av_local_kernel<<<grid, kLocalThreads, 4 * ((size_t)args.P * args.P + 1), stream>>>(args);
  return cudaGetLastError();
}

}  // namespace rbv
