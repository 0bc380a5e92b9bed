// The tables of the static kernel on the host: comm.cu against stand-ins for the CUDA runtime (a "device" pointer is a host
// pointer), every schedule prepared on every process of a communicator, and the items executed as the kernel executes them:
// the chunks that are dealt in any order, a chain at a time, a chunk that waits when its flag is up.  Receive buffers must hold what a
// direct copy would put there, every item must have run, and the arrivals must be the expected ones.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <random>
#include <vector>

#include "rbv/context.h"

extern "C" {
static cudaError_t host_alloc(void** p, size_t n) {
  *p = std::calloc(n, 1);            // zero pages that nobody touches cost nothing: clearing them again would
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMalloc(void** p, size_t n) { return host_alloc(p, n); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return host_alloc(p, n); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { if (v) std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->multiProcessorCount = 4;      // few warps: blocks of tens of KB already take several chunks per warp
  return cudaSuccess;
}
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t* h, void* p) { std::memcpy(h, &p, sizeof p); return cudaSuccess; }
cudaError_t cudaIpcOpenMemHandle(void** p, cudaIpcMemHandle_t h, unsigned) { std::memcpy(p, &h, sizeof *p); return cudaSuccess; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "host"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorInvalidValue; }
}

namespace rbv {
cudaError_t a2av_configure(int, int* ctas) { *ctas = 1; return cudaSuccess; }
int a2av_bulk_ctas_per_sm(int) { return 1; }
cudaError_t a2av_static_configure(int, int* ctas) { *ctas = 1; return cudaSuccess; }
cudaError_t a2av_launch(const KernelArgs&, int, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t a2av_static_launch(const StaticArgs&, int, int, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t a2av_local_launch(const LocalArgs&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t a2av_eager_launch(const KernelArgs&, int, bool, cudaStream_t) { return cudaSuccess; }
}  // namespace rbv

using namespace rbv;

static long g_bad = 0, g_tables = 0, g_chained = 0, g_wide = 0, g_flags = 0;

static void fail(const char* what, int algo, int P, int nproc, int top) {
  if (g_bad++ < 10) std::printf("%s: schedule %d, %d ranks, %d processes, blocks up to %d\n", what, algo, P, nproc, top);
}

// One call of a communicator; false where the schedule does not exist for these ranks.
static bool run(int algo, int P, int nproc, int n, int top, size_t chunk) {
  const int L = P / nproc, ts = 2;
  std::mt19937 gen(algo * 131 + P * 7 + nproc + top);
  std::vector<int> counts(P * P), caps(P * P);
  for (int& v : counts) v = gen() % 5 == 0 ? 0 : gen() % 9 == 0 ? 1 : (int)(gen() % top);
  counts[1] = top;                                           // chunks of 4096 elements: a block that ends with one, and one behind
  if (top > 32768) { counts[P] = 4096 * 8; counts[P - 1] = 4096 * 8 + 1; }
  size_t total = 0;
  for (int s = 0; s < P; s++)
    for (int d = 0; d < P; d++) { caps[d * P + s] = counts[s * P + d]; total += counts[s * P + d]; }
  std::vector<std::unique_ptr<Context>> ctx;
  std::vector<char> handles(64 * nproc);
  for (int q = 0; q < nproc; q++) {
    ctx.emplace_back(new Context(P, nproc, q, 0, 2 * (total + 8 * P * P) * ts + (1 << 20), (size_t)40 * (top + 8) * ts));
    ctx[q]->ipc_handle(&handles[64 * q]);
  }
  for (auto& c : ctx) c->connect(handles.data());
  std::vector<std::vector<char>> send(P);
  std::vector<char*> recv(P);
  std::vector<long long> sd(P * P), rd(P * P);
  std::vector<unsigned long long> off(P);
  std::vector<size_t> room(P);
  for (int r = 0; r < P; r++) {
    long long at = 1, to = 2;
    for (int p = 0; p < P; p++) {
      sd[r * P + p] = at; at += counts[r * P + p] + (int)(gen() % 3);
      rd[r * P + p] = to; to += counts[p * P + r] + (int)(gen() % 3);
    }
    send[r].resize((at + 8) * ts);
    for (char& v : send[r]) v = (char)gen();
    room[r] = (to + 8) * ts;
    recv[r] = static_cast<char*>(ctx[r / L]->symm_alloc(room[r]));
    std::memset(recv[r], 0x5a, room[r]);
    off[r] = recv[r] - ctx[r / L]->heap();
  }
  std::vector<Prepared> calls(nproc);
  for (int q = 0; q < nproc; q++) {
    AlgoSpec spec{};
    spec.algo = algo; spec.P = P; spec.n = n; spec.r = 2; spec.r2 = 2; spec.b = 2; spec.b2 = 2;
    std::vector<const void*> sb;
    std::vector<void*> rb;
    for (int i = 0; i < L; i++) { sb.push_back(send[q * L + i].data()); rb.push_back(recv[q * L + i]); }
    CallArgs ca{};
    ca.sendbufs = sb.data(); ca.recvbufs = rb.data();
    ca.sendcounts = &counts[q * L * P]; ca.recvcounts = &caps[q * L * P];
    ca.sdispls = &sd[q * L * P]; ca.rdispls = &rd[q * L * P];
    ca.bytes_hint = -1;
    if (nproc > 1) { ca.g_counts = counts.data(); ca.g_caps = caps.data(); ca.g_rdispls = rd.data(); ca.g_recvoff = off.data(); }
    CallOptions opt{};
    opt.chunk_bytes = chunk;
    opt.allow_static = true;
    if (ctx[q]->prepare(spec, ts, ca, opt, nullptr, true, &calls[q])) return false;
    if (!calls[q].is_static) { fail("not resolved", algo, P, nproc, top); return true; }
  }
  // ---- execute ----
  std::vector<std::vector<char>> ran(nproc), flag(nproc);
  std::vector<std::vector<unsigned>> left(nproc);            // dealt chunks that have not run
  std::vector<unsigned long long> arrived(P, 0);
  for (int q = 0; q < nproc; q++) {
    const StaticArgs& a = calls[q].sa;
    ran[q].assign(calls[q].static_items, 0);
    flag[q].assign((size_t)L * ctx[q]->layout().flags_per_rank, 0);
    for (unsigned d = 0; d < a.nitems; d++) left[q].push_back(d);
    if (a.wide) g_wide++;
    if (std::memcmp(a.inl, a.items, std::min(calls[q].static_items, (unsigned)kInlineItems) * sizeof(StaticItem)))
      fail("inline items differ", algo, P, nproc, top);
    g_tables++;
  }
  for (bool progress = true; progress;) {
    progress = false;
    for (int q = 0; q < nproc; q++) {
      const StaticArgs& a = calls[q].sa;
      std::vector<unsigned> waiting;
      std::shuffle(left[q].begin(), left[q].end(), gen);     // only flags order anything, and warps run as they like
      for (unsigned d : left[q]) {
        const bool wide = d < a.wide;
        unsigned at = wide ? d >> a.wide_shift : (a.wide >> a.wide_shift) + (d - a.wide);
        const unsigned from = wide ? (d - (at << a.wide_shift)) * a.chunk : 0;
        if (a.items[at].wait_flag != kNoFlag && !flag[q][a.items[at].wait_flag]) { waiting.push_back(d); continue; }
        progress = true;
        if (gen() % 2) { waiting.push_back(d); continue; }
        for (;;) {
          if (at >= calls[q].static_items || from >= a.items[at].len) { fail("no such chunk", algo, P, nproc, top); break; }
          const StaticItem& it = a.items[at];
          ran[q][at] = 1;
          std::memcpy(reinterpret_cast<char*>(it.dst) + from, reinterpret_cast<const char*>(it.src) + from, std::min(it.len - from, a.chunk));
          if (it.flags & ITEM_NEXT) { at = it.signal_flag; g_chained++; continue; }
          if (it.signal_flag == kNoFlag) { if (!(it.flags & ITEM_DST_STAGE)) arrived[it.dst_rank]++; }
          else { flag[it.dst_rank / L][it.signal_flag] = 1; g_flags++; }
          break;
        }
      }
      left[q].swap(waiting);
    }
  }
  for (int q = 0; q < nproc; q++) {
    if (!left[q].empty()) fail("waits for ever", algo, P, nproc, top);
    if (std::count(ran[q].begin(), ran[q].end(), 0)) fail("an item was left out", algo, P, nproc, top);
    for (int i = 0; i < L && nproc > 1; i++)
      if (arrived[q * L + i] != calls[q].sa.expect[i]) fail("arrivals", algo, P, nproc, top);
    ctx[q]->release(calls[q]);
  }
  for (int d = 0; d < P; d++) {
    std::vector<char> want(room[d], 0x5a);
    for (int s = 0; s < P; s++)
      std::memcpy(&want[rd[d * P + s] * ts], &send[s][sd[s * P + d] * ts], (size_t)counts[s * P + d] * ts);
    if (std::memcmp(want.data(), recv[d], room[d])) { fail("wrong bytes", algo, P, nproc, top); break; }
  }
  return true;
}

int main(int argc, char** argv) {
  const int schedules = std::atoi(argv[1]);
  int built = 0;
  for (int chains = 1; chains >= 0; chains--) {
    setenv("RBV_STATIC_CHAINS", chains ? "1" : "0", 1);
    for (int algo = 0; algo < schedules; algo++) {
      bool any = false;
      for (int P : {4, 8, 12})
        for (int nproc : {1, 2, 4})
          for (int top : {3, 150000})
            for (size_t chunk : {(size_t)0, (size_t)4096}) {
              if ((chunk && top < 1000) || (!chains && nproc > 1) || (P != 8 && chunk)) continue;
              any |= run(algo, P, nproc, P == 12 ? 3 : 4, top, chunk);
            }
      if (any) built++;
      else std::printf("schedule %d: never built\n", algo);
    }
  }
  std::printf("%ld tables of %d schedules, %ld hops in chains, %ld flags, %ld tables with wide items, %ld bad\n", g_tables, built / 2,
              g_chained, g_flags, g_wide, g_bad);
  return g_bad != 0 || built != 2 * schedules || !g_chained || !g_flags || !g_wide;
}
