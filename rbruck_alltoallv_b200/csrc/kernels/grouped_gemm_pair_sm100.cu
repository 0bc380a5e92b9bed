// Grouped GEMM for the expert FFN on CTA PAIRS (tcgen05 cta_group::2), weights as the M operand and tokens as the N
// operand.  Two CTAs on neighbouring SMs share one tile of 256 weight rows by up to 256 tokens.  Each CTA fetches its own
// 128 weight rows and its own half of the tile's tokens, so a k-block of a full tile costs 32 KB of shared-memory fill
// per SM.  No counterpart exists in the reference (it has no compute kernels).
//
//   C[rows of group g] = epilogue( A[rows of group g] (M_g x K, K-major) * B_g^T (N x K, K-major) )
//
// Why tokens are N: the M of an MMA is fixed (256 for a pair) while its N is any multiple of 32 up to 256, and the token
// count is the ragged one.  A group of R rows costs ceil(R / 32) * 32 columns, cut into tiles of nearly equal size, where
// tokens as M cost ceil(R / 256) * 256 rows: a group of 16 decoded tokens ran 16 times the MMAs it needed and fetched 16
// times the token rows.  Measured on one B200, MoE layer of 8 experts, hidden 4096, FFN 14336: 64 tokens 660 -> 500 us
// (HBM-bound now: every weight is read once), 8192 tokens, up / down GEMM alone 2.64 / 1.38 -> 2.48 / 1.32 ms (tensor pipe
// busy in 98 % of the cycles, at the clock that the power cap leaves).
//
// One persistent cluster of two CTAs per SM pair walks a static tile schedule (groups in order, weight rows slow, tokens
// fast, so the token tiles of one weight tile run at the same time and share it in L2):
//   warp 0    TMA producer, in both CTAs (own weight rows, own half of the tokens; bytes counted in the rank-0 CTA)
//   warp 1    TMEM allocation in both CTAs; in the rank-0 CTA one elected thread issues the M256 K16 MMAs
//   warps 2-5 epilogue, in both CTAs (each drains the 128 weight rows in its own TMEM: a lane is an output column)
// TMEM holds two 128 x 256 fp32 accumulators per CTA, so the epilogue of tile i overlaps the MMAs of tile i + 1.
// TMA loads carry no cluster multicast.  All waits are bounded; on expiry both CTAs are told, record an error,
// release their TMEM and return.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

#include "kernels/pdl.cuh"
#include "kernels/sm100_ptx.cuh"
#include "kernels/tok_epilogue.cuh"
#include "rbv/moe.h"

namespace rbv {

using namespace sm100;

namespace {

constexpr int PM = 256;            // weight rows (output columns) per pair tile
constexpr int HM = 128;            // weight rows per CTA
constexpr int PT = 256;            // most tokens per tile
constexpr int PU = 32;             // tokens per unit: a tile's token count is a multiple of this
constexpr int PK = 64;             // one 128-byte swizzle atom of bf16
constexpr int PW_BYTES = HM * PK * 2;        // 16 KB of weights
constexpr int PT_BYTES = PT / 2 * PK * 2;    // up to 16 KB of tokens
// Pipeline: 6 stages with room for the tokens of a full tile; where no group has more than 64 rows, 10 stages with room for
// 64.  The kernel then is a stream of weights, and what counts is how many of their bytes are on the way (160 instead of
// 96 KB per SM: up / down GEMM of 64 tokens 316 / 171 -> 299 / 162 us, the layer 472 -> 440 us).
constexpr int PSTAGES = 6, PSTAGE_BYTES = PW_BYTES + PT_BYTES;
constexpr int PSMALL = 64, PSTAGES_SMALL = 10, PSTAGE_BYTES_SMALL = PW_BYTES + PSMALL / 2 * PK * 2;
constexpr int PAIR_THREADS = 192;
constexpr int PAIR_TMEM_COLS = 512;
constexpr size_t PAIR_SMEM = (size_t)PSTAGES_SMALL * PSTAGE_BYTES_SMALL + 1024 /*alignment slack*/;
static_assert(PSTAGES * PSTAGE_BYTES <= PSTAGES_SMALL * PSTAGE_BYTES_SMALL, "shared memory");

// Token boxes of 16, 32, 64 and 128 rows: a CTA's half of a tile is fetched with the smallest that covers it.
struct PairMaps { CUtensorMap w, tok[4]; };

struct PairParams {
  const int* group_start;
  const int* group_rows;
  int G;
  int N, K;
  int ldc;
  long long a_rows;
  void* C;
  int* error;
  int epilogue;   // 0: C = bf16(acc); 1: C[:, j] = bf16(silu(acc[:, 2j]) * acc[:, 2j+1])
  // Push mode (ret != null, epilogue 0): row `pos` of the result goes to row (ret[pos] & 0xffffff) of the [*, N] bf16
  // buffer at offset y2_off of the heap of process ret[pos] >> 24 (a peer mapping over NVLink when that is another
  // GPU): the return all-to-all of the MoE layer, done by the epilogue.
  const unsigned* ret;
  unsigned long long y2_off;
  char* heap[16];
};

struct PairTile { int tok0, ntok, nt, n0, b_row; bool valid; };   // first token row, live tokens, columns, weight rows

// Walks the tile schedule; `at(t)` wants non-decreasing t.
struct PairWalk {
  int g = 0, before = 0;   // tiles of the groups in front of g
  __device__ __forceinline__ PairTile at(const PairParams& p, int t, const int* s_rows, const int* s_start) {
    PairTile r; r.valid = false; r.tok0 = r.ntok = r.nt = r.n0 = r.b_row = 0;
    for (; g < p.G; g++) {
      const int units = (s_rows[g] + PU - 1) / PU, ntm = (units + PT / PU - 1) / (PT / PU);
      const int cnt = ntm * (p.N / PM);
      if (t - before < cnt) {
        const int n = (t - before) / ntm, m = (t - before) - n * ntm;
        const int base = units / ntm, extra = units - base * ntm;     // the first `extra` tiles are one unit larger
        const int u0 = m * base + min(m, extra), nu = base + (m < extra ? 1 : 0);
        r.tok0 = s_start[g] + u0 * PU; r.nt = nu * PU; r.ntok = min(s_rows[g] - u0 * PU, r.nt);
        r.n0 = n * PM; r.b_row = g * p.N + n * PM;
        r.valid = true;
        return r;
      }
      before += cnt;
    }
    return r;
  }
};

// Index of the token box for `half` rows, and its rows.
__device__ __forceinline__ int tok_box(int half) { return half <= 16 ? 0 : half <= 32 ? 1 : half <= 64 ? 2 : 3; }
__device__ __forceinline__ uint32_t tok_box_bytes(int half) { return (16u << tok_box(half)) * PK * 2; }

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
grouped_gemm_pair_kernel(const __grid_constant__ PairMaps maps, const __grid_constant__ PairParams p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[PSTAGES_SMALL];    // used in the rank-0 CTA: bytes of both CTAs' loads
  __shared__ __align__(8) uint64_t empty_bar[PSTAGES_SMALL];   // in each CTA: its stage has been read by the MMAs
  __shared__ __align__(8) uint64_t tfull_bar[2];         // in each CTA: accumulator b is complete
  __shared__ __align__(8) uint64_t tempty_bar[2];        // used in the rank-0 CTA: both CTAs have drained accumulator b
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_rows[kMoeMaxGroups], s_start[kMoeMaxGroups];
  __shared__ int s_abort, s_most;                        // s_most: rows of the largest group

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (tid == 0) {
    for (int s = 0; s < PSTAGES_SMALL; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; b++) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 8); }
    s_abort = 0;
    s_most = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_s, PAIR_TMEM_COLS); tmem_relinquish_pair(); }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  for (int i = tid; i < p.G; i += blockDim.x) {
    s_start[i] = p.group_start[i]; s_rows[i] = rows_inside(p.group_rows[i], s_start[i], p.a_rows, p.error);
    atomicMax(&s_most, s_rows[i]);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();   // barriers of both CTAs are initialised before anything is signalled across
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int num_kb = p.K / PK;
  const int stages = s_most <= PSMALL ? PSTAGES_SMALL : PSTAGES;
  const int stage_bytes = s_most <= PSMALL ? PSTAGE_BYTES_SMALL : PSTAGE_BYTES;
  volatile int* abort_flag = &s_abort;
  const uint32_t peer_abort = mapa_u32(smem_u32(&s_abort), rank ^ 1u);

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      tma_prefetch_desc(&maps.w);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      PairWalk walk;
      for (int t = pair; ok; t += npairs) {
        const PairTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        const int half = tl.nt / 2;
        const CUtensorMap* tok = &maps.tok[tok_box(half)];
        const uint32_t bytes = 2u * (PW_BYTES + tok_box_bytes(half));
        const int w_row = tl.b_row + (int)rank * HM;
        const int t_row = tl.tok0 + (int)rank * half;
        for (int kb = 0; kb < num_kb; kb++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t* sw = tiles + (size_t)stage * stage_bytes;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], bytes);
          const uint32_t bar0 = mapa_u32(smem_u32(&full_bar[stage]), 0);
          tma_load_2d_pair(sw, &maps.w, kb * PK, w_row, bar0);
          tma_load_2d_pair(sw + PW_BYTES, tok, kb * PK, t_row, bar0);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 1); }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (rank-0 CTA only) ----------------
    if (leader && elect_one()) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      int i = 0;
      PairWalk walk;
      for (int t = pair; ok; t += npairs, i++) {
        const PairTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        const uint32_t idesc = umma_idesc(PM, tl.nt, 1 /*bf16*/);
        const int b = i & 1;
        if (!mbar_wait(&tempty_bar[b], (((uint32_t)i >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + (uint32_t)b * PT;
        for (int kb = 0; kb < num_kb; kb++) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint8_t* sw = tiles + (size_t)stage * stage_bytes;
          const uint64_t wdesc = umma_desc_sw128(sw);
          const uint64_t tdesc = umma_desc_sw128(sw + PW_BYTES);
          #pragma unroll
          for (int kk = 0; kk < PK / 16; kk++)
            umma_bf16_pair(d_tmem, wdesc + 2u * kk, tdesc + 2u * kk, idesc, (uint32_t)((kb | kk) != 0));
          umma_commit_pair(&empty_bar[stage]);   // frees this stage in both CTAs
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit_pair(&tfull_bar[b]);   // accumulator complete, both CTAs
      }
      if (!ok) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 2); }
    }
  } else {
    // ---------------- epilogue (both CTAs): warps 2..5, TMEM lane quarter = warp % 4 ----------------
    const int q = warp & 3;
    __nv_bfloat16* C = static_cast<__nv_bfloat16*>(p.C);
    bool ok = true;
    int i = 0;
    PairWalk walk;
    for (int t = pair; ok; t += npairs, i++) {
      const PairTile tl = walk.at(p, t, s_rows, s_start);
      if (!tl.valid) break;
      const int b = i & 1;
      if (!mbar_wait(&tfull_bar[b], ((uint32_t)i >> 1) & 1u, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)b * PT;
      const int nw = tl.n0 + (int)rank * HM + q * 32;   // first of this warp's 32 columns
      #pragma unroll 1
      for (int c = 0; c < tl.nt; c += PU) {
        uint32_t r[32];
        tmem_ld32(taddr + c, r);
        unsigned rv = 0;   // push mode: where the token of this lane's index goes, handed out by shuffle
        if (p.ret && c + lane < tl.ntok) rv = __ldg(p.ret + tl.tok0 + c + lane);
        tmem_ld_wait();
        __nv_bfloat16* rows = C + (size_t)(tl.tok0 + c) * p.ldc;
        if (p.epilogue == 1) {
          tokepi::store_swiglu(r, rows, p.ldc, nw / 2, tl.ntok - c, lane);
        } else if (p.ret) {
          tokepi::store_plain(r, [&](int tok) {
            const unsigned to = __shfl_sync(0xffffffffu, rv, tok);
            return reinterpret_cast<__nv_bfloat16*>(p.heap[to >> 24] + p.y2_off) + (size_t)(to & 0xffffffu) * p.ldc;
          }, nw, tl.ntok - c, lane);
        } else {
          tokepi::store_plain(r, [&](int tok) { return rows + (size_t)tok * p.ldc; }, nw, tl.ntok - c, lane);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty_bar[b]), 0));   // 4 warps x 2 CTAs
    }
    if (!ok && lane == 0) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 3); }
  }

  // ---------------- teardown: nobody leaves while the other CTA may still signal it ----------------
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, PAIR_TMEM_COLS);
  }
}

// ---------------- host side ----------------
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn pair_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// [rows, K] bf16 row-major, box = box_rows x 64 elements, 128-byte swizzle
bool pair_make_map(CUtensorMap* m, const void* base, unsigned long long rows, unsigned long long K, unsigned box_rows) {
  EncodeTiledFn fn = pair_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K * 2};
  cuuint32_t box[2] = {(cuuint32_t)PK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int g_pair_mode = -1;   // -1: not decided yet (environment), 0: one-CTA kernel, 1: CTA pairs

}  // namespace
}  // namespace rbv

extern "C" void rbv_grouped_gemm_set_pair(int on) { rbv::g_pair_mode = on ? 1 : 0; }

extern "C" int rbv_grouped_gemm_pair_enabled() {
  if (rbv::g_pair_mode < 0) {
    const char* e = std::getenv("RBV_GEMM_PAIR");
    rbv::g_pair_mode = (e && e[0] == '0') ? 0 : 1;
  }
  return rbv::g_pair_mode;
}

static int launch_bf16_pair(const void* A, long long a_rows, const void* B, void* C, const int* group_start,
                            const int* group_rows, int G, int N, int K, int ldc, int epilogue, int* error_flag,
                            int max_ctas, void* cuda_stream, const unsigned* ret, const void* const* heaps, int nheaps,
                            unsigned long long y2_off) {
  using namespace rbv;
  if (G < 1 || G > kMoeMaxGroups || N % PM || K % PK || a_rows < 1 || (ldc % 8)) return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return (int)cudaErrorInvalidValue;
  if (ret && (epilogue != 0 || !heaps || nheaps < 1 || nheaps > 16 || (y2_off & 15))) return (int)cudaErrorInvalidValue;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(grouped_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)PAIR_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  PairMaps maps;
  if (!pair_make_map(&maps.w, B, (unsigned long long)G * N, (unsigned long long)K, HM)) return (int)cudaErrorUnknown;
  for (int i = 0; i < 4; i++)
    if (!pair_make_map(&maps.tok[i], A, (unsigned long long)a_rows, (unsigned long long)K, 16u << i)) return (int)cudaErrorUnknown;
  PairParams p;
  p.group_start = group_start; p.group_rows = group_rows; p.G = G; p.N = N; p.K = K; p.ldc = ldc; p.C = C;
  p.a_rows = a_rows; p.error = error_flag; p.epilogue = epilogue;
  p.ret = ret; p.y2_off = y2_off;
  for (int q = 0; q < 16; q++) p.heap[q] = (ret && q < nheaps) ? static_cast<char*>(const_cast<void*>(heaps[q])) : nullptr;
  int grid = max_ctas;
  if (grid <= 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&grid, cudaDevAttrMultiProcessorCount, dev);
  }
  grid &= ~1;   // whole pairs
  if (grid < 2) return (int)cudaErrorInvalidValue;
  return (int)launch_dependent(grouped_gemm_pair_kernel, grid, PAIR_THREADS, PAIR_SMEM,
                               static_cast<cudaStream_t>(cuda_stream), maps, p);
}

extern "C" int rbv_grouped_gemm_bf16_pair(const void* A, long long a_rows, const void* B, void* C,
                                          const int* group_start, const int* group_rows, int G, int N, int K, int ldc,
                                          int epilogue, int* error_flag, int max_ctas, void* cuda_stream) {
  return launch_bf16_pair(A, a_rows, B, C, group_start, group_rows, G, N, K, ldc, epilogue, error_flag, max_ctas,
                          cuda_stream, nullptr, nullptr, 0, 0ull);
}

extern "C" int rbv_grouped_gemm_bf16_push(const void* A, long long a_rows, const void* B, const int* group_start,
                                          const int* group_rows, int G, int N, int K, const unsigned* ret,
                                          const void* const* heaps, int nheaps, unsigned long long y2_off,
                                          int* error_flag, int max_ctas, void* cuda_stream) {
  if (!ret) return (int)cudaErrorInvalidValue;
  // C is only a base for rows that are not pushed (there are none): any aligned address of this process will do
  return launch_bf16_pair(A, a_rows, B, const_cast<void*>(heaps ? heaps[0] : nullptr), group_start, group_rows, G, N, K,
                          N, 0, error_flag, max_ctas, cuda_stream, ret, heaps, nheaps, y2_off);
}
