// Block-scaled fp8 (e4m3) grouped GEMM on CTA pairs for groups of few tokens: same operands, scales and epilogues as
// grouped_gemm_fp8_pair_sm100.cu, with weight rows as the M operand of the MMAs and tokens as the N operand.
//
//   C[rows of g] = epi( sum_kb  sa[kb][row] * sb[g][n / 128][kb] * ( A[rows, kb] * B_g[n-tile, kb]^T ) )
//
// Two CTAs on neighbouring SMs share a tile of 256 weight rows by up to 128 tokens, in multiples of 32: the token count is
// the ragged one, and the M of an MMA is fixed, so that kernel computes and fetches 256 tokens for a group of one.  Per K
// block each CTA fetches its own 128 weight rows and its own half of the tokens, the rank-0 CTA issues four
// tcgen05.mma.cta_group::2.kind::f8f6f4 (M 256, K 32) into one of four 128-column TMEM slots, and the eight scaling /
// epilogue warps of EACH CTA pull the 128 accumulator rows of their own TMEM, scale and accumulate them in registers
// (packed fp32 FMAs) and hand the slot back to the rank-0 CTA across the cluster.  A CTA's weight rows share one scale
// per K block; the tokens' scales, multiplied by it, reach the lanes through a shared-memory row per warp, which is what
// makes a full K block cost more here (450 ns) than with a token per lane (360 ns) and draws the line between the two
// kernels, see rbv_grouped_gemm_fp8_pair.
// TMA loads carry no cluster multicast.  All waits are bounded; on expiry both CTAs are told, record an error, release
// their TMEM and return.  No counterpart in the reference.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels/pdl.cuh"
#include "kernels/sm100_ptx.cuh"
#include "kernels/tok_epilogue.cuh"
#include "rbv/moe.h"

namespace rbv {

using namespace sm100;

namespace {

constexpr int QM = 256;                 // weight rows (output columns) per pair tile
constexpr int QHM = 128;                // weight rows per CTA: one scale block
constexpr int QT = 128;                 // most tokens per tile
constexpr int QU = 32;                  // a tile's token count is a multiple of this
constexpr int QK = 128;                 // one 128-byte swizzle row of fp8
constexpr int QSLOTS = 4;
constexpr int QW_TILE = QHM * QK;       // 16 KB of weights
constexpr int QT_TILE = QT / 2 * QK;    // up to 8 KB of tokens
// Pipeline: 8 stages with room for the tokens of a full tile; where no group has more than 64 rows, 10 with room for 64
constexpr int QSTAGES = 8, QSTAGE = QW_TILE + QT_TILE;
constexpr int QSMALL = 64, QSTAGES_SMALL = 10, QSTAGE_SMALL = QW_TILE + QSMALL / 2 * QK;
constexpr int QSCALERS = 8;             // scaling / epilogue warps
constexpr int QTHREADS = 64 + 32 * QSCALERS;
constexpr size_t QSMEM = (size_t)QSTAGES_SMALL * QSTAGE_SMALL + 1024;
static_assert(QSTAGES * QSTAGE <= QSTAGES_SMALL * QSTAGE_SMALL, "shared memory");

// Token boxes of 16, 32 and 64 rows: a CTA's half of a tile is fetched with the smallest that covers it.
struct Fp8TokMaps { CUtensorMap w, tok[3]; };

struct Fp8TokParams {
  const int* group_start;
  const int* group_rows;
  int G, N, K, ldc;
  long long a_rows;            // rows of A (= leading dimension of the transposed scale array)
  const float* a_scale;        // [K / 128][a_rows]
  const float* b_scale;        // [G][N / 128][K / 128]
  void* C;
  int* error;
  int epilogue;                // bit 0: SwiGLU over interleaved gate / up columns; bit 1: coarse scales
};

struct QTile { int g, tok0, ntok, nt, n0; bool valid; };   // group, first token row, live tokens, columns, first weight row

// Walks the tile schedule (groups in order, weight rows slow, tokens fast); `at(t)` wants non-decreasing t.
struct QWalk {
  int g = 0, before = 0;   // tiles of the groups in front of g
  __device__ __forceinline__ QTile at(const Fp8TokParams& p, int t, const int* s_rows, const int* s_start) {
    QTile r; r.valid = false; r.g = r.tok0 = r.ntok = r.nt = r.n0 = 0;
    const int ntn = (p.N + QM - 1) / QM;     // N is a multiple of 128: the last tile may be half empty
    for (; g < p.G; g++) {
      const int units = (s_rows[g] + QU - 1) / QU, ntm = (units + QT / QU - 1) / (QT / QU);
      const int cnt = ntm * ntn;
      if (t - before < cnt) {
        const int n = (t - before) / ntm, m = (t - before) - n * ntm;
        const int base = units / ntm, extra = units - base * ntm;     // the first `extra` tiles are one unit larger
        const int u0 = m * base + min(m, extra), nu = base + (m < extra ? 1 : 0);
        r.g = g; r.tok0 = s_start[g] + u0 * QU; r.nt = nu * QU; r.ntok = min(s_rows[g] - u0 * QU, r.nt); r.n0 = n * QM;
        r.valid = true;
        return r;
      }
      before += cnt;
    }
    return r;
  }
};

__device__ __forceinline__ int q_tok_box(int half) { return half <= 16 ? 0 : half <= 32 ? 1 : 2; }
__device__ __forceinline__ uint32_t q_tok_box_bytes(int half) { return (16u << q_tok_box(half)) * QK; }

// fp8 (e4m3 x e4m3 -> fp32) MMA of a CTA pair: M 256, issued by one thread of the rank-0 CTA
__device__ __forceinline__ void umma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// What a scaling warp needs besides the tile.
struct Scaler {
  uint64_t* tfull;             // this CTA's slot-full barriers
  uint32_t tempty0;            // cluster address of the rank-0 CTA's slot-free barriers
  volatile int* abort_flag;
  float* row;                  // two rows of 64 scales of this warp, in shared memory
  uint32_t tmem;               // TMEM address of this warp's lanes, column 0 of slot 0
  int q, half, lane, rank;
};

// One tile for a warp that owns HW of its columns (tokens) and 32 weight rows (lanes).  `it`: running slot count.
// Returns false when a wait gave up.
template <int HW>
__device__ __forceinline__ bool scale_tile(const Fp8TokParams& p, const QTile& tl, const Scaler& w, unsigned& it) {
  constexpr int kDepth = 4;                // scales are fetched this many K blocks ahead of their use
  constexpr int kPer = (HW + 31) / 32;     // scales per lane and K block
  const int nkb = p.K / QK, lane = w.lane;
  const int tok = tl.tok0 + w.half * HW;   // this warp's first token row
  const int n_cta = tl.n0 + w.rank * QHM;
  const bool inside = n_cta < p.N;
  const float* sb = p.b_scale + ((size_t)tl.g * (p.N / 128) + (inside ? n_cta / 128 : 0)) * nkb;
  const float* sa = p.a_scale + tok + lane;
  // scale of token i * 32 + lane in K block kb (0 where there is no such token)
  const int in = (int)min((long long)HW, p.a_rows - tok) - lane;
  auto token_scale = [&](int kb, int i) { return i * 32 < in ? __ldg(sa + (size_t)kb * p.a_rows + i * 32) : 0.0f; };
  // Accumulators in the shape of an MMA fragment (tmem_ld_frag16): this lane has, of every group g of 8 tokens, tokens
  // 8 g + 2 (lane % 4) and + 1, of the weight rows lane / 4 + 8 h, h = 0..3, in acc2[4 g + h].  So a pair of scales serves
  // four weight rows; with a weight row per lane every lane would read every token's scale, which keeps the return path
  // of shared memory busy for twice as long as the MMAs of a K block take.
  float2 acc2[HW / 2];
  #pragma unroll
  for (int j = 0; j < HW / 2; j++) acc2[j] = make_float2(0.0f, 0.0f);
  float sa_q[kDepth][kPer], sb_q[kDepth];
  #pragma unroll
  for (int j = 0; j < kDepth; j++) {
    sb_q[j] = j < nkb ? __ldg(sb + j) : 0.0f;
    #pragma unroll
    for (int i = 0; i < kPer; i++) sa_q[j][i] = j < nkb ? token_scale(j, i) : 0.0f;
  }
  const bool coarse = (p.epilogue & 2) != 0;   // scales of K block 0 hold for the whole tile: one slot per tile
  const int steps = coarse ? 1 : nkb;
  for (int kb0 = 0; kb0 < steps; kb0 += kDepth) {
    #pragma unroll
    for (int j = 0; j < kDepth; j++) {
      const int kb = kb0 + j;
      if (kb >= steps) break;
      const int slot = it % QSLOTS;
      float* row = w.row + (kb & 1) * 64;
      #pragma unroll
      for (int i = 0; i < kPer; i++)
        if (i * 32 + lane < HW) row[i * 32 + lane] = sa_q[j][i] * sb_q[j];
      if (kb + kDepth < steps) {
        sb_q[j] = __ldg(sb + kb + kDepth);
        #pragma unroll
        for (int i = 0; i < kPer; i++) sa_q[j][i] = token_scale(kb + kDepth, i);
      }
      if (!mbar_wait(&w.tfull[slot], (it / QSLOTS) & 1u, w.abort_flag)) return false;
      tc_fence_after_sync();
      __syncwarp();                            // the scales are in place (and the other row is no longer read)
      // 16 tokens at a time, the next 16 on their way from TMEM while these are multiplied
      uint32_t r[2][2][8];
      const uint32_t taddr = w.tmem + (uint32_t)slot * QT + (uint32_t)(w.half * HW);
      tmem_ld_frag16(taddr, r[0][0]);
      tmem_ld_frag16(taddr + (16u << 16), r[0][1]);
      #pragma unroll
      for (int c = 0; c < HW; c += 16) {
        float2 s[2];
        #pragma unroll
        for (int g = 0; g < 2; g++) s[g] = *reinterpret_cast<const float2*>(row + c + 8 * g + 2 * (lane & 3));
        tmem_ld_wait();
        if (c + 16 < HW) {
          tmem_ld_frag16(taddr + c + 16, r[(c / 16 + 1) & 1][0]);
          tmem_ld_frag16(taddr + (16u << 16) + c + 16, r[(c / 16 + 1) & 1][1]);
        } else {                               // the slot is free once it sits in registers
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(w.tempty0 + 8u * (uint32_t)slot);
        }
        #pragma unroll
        for (int g = 0; g < 2; g++)
          #pragma unroll
          for (int h = 0; h < 4; h++) {
            const uint32_t* v = &r[(c / 16) & 1][h >> 1][4 * g + 2 * (h & 1)];
            float2& acc = acc2[4 * (c / 8 + g) + h];
            acc = __ffma2_rn(s[g], make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])), acc);
          }
      }
      it++;
    }
  }
  // Neighbouring weight rows (output columns) sit four lanes apart: lanes swap, so that one with an even column keeps the
  // first token of a pair and two columns of it, and its neighbour the second token.
  const int live = inside ? tl.ntok - w.half * HW : 0;
  const int j = lane >> 2;                     // weight row of this lane inside a block of 8
  const bool odd = (j & 1) != 0;
  __nv_bfloat16* rows = static_cast<__nv_bfloat16*>(p.C) + (size_t)tok * p.ldc;
  #pragma unroll
  for (int g = 0; g < HW / 8; g++) {
    const int t = 8 * g + 2 * (lane & 3) + (odd ? 1 : 0);
    __nv_bfloat16* crow = rows + (size_t)t * p.ldc;
    float first[4], second[4];                 // columns 8 h + (j & ~1) and + 1 of token t
    #pragma unroll
    for (int h = 0; h < 4; h++) {
      const float2 v = acc2[4 * g + h];
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 4);
      first[h] = odd ? got : v.x;
      second[h] = odd ? v.y : got;
    }
    if (t >= live) continue;
    const int n = n_cta + w.q * 32 + (j & ~1);
    if (p.epilogue & 1) {                      // (first, second) = (gate, up)
      #pragma unroll
      for (int h = 0; h < 4; h++) crow[(n + 8 * h) / 2] = __float2bfloat16_rn(tokepi::silu(first[h]) * second[h]);
    } else {
      #pragma unroll
      for (int h = 0; h < 4; h++)
        *reinterpret_cast<__nv_bfloat162*>(crow + n + 8 * h) = __floats2bfloat162_rn(first[h], second[h]);
    }
  }
  return true;
}

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(QTHREADS, 1)
grouped_gemm_fp8_tok_kernel(const __grid_constant__ Fp8TokMaps maps, const __grid_constant__ Fp8TokParams p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[QSTAGES_SMALL];    // used in the rank-0 CTA: bytes of both CTAs' loads
  __shared__ __align__(8) uint64_t empty_bar[QSTAGES_SMALL];   // in each CTA: its stage has been read by the MMAs
  __shared__ __align__(8) uint64_t tfull_bar[QSLOTS];    // in each CTA: TMEM slot holds a finished K block (or tile)
  __shared__ __align__(8) uint64_t tempty_bar[QSLOTS];   // used in the rank-0 CTA: all 16 scaling warps took the slot
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_rows[kMoeMaxGroups], s_start[kMoeMaxGroups];
  __shared__ int s_abort, s_most;                        // s_most: rows of the largest group
  __shared__ __align__(16) float s_scale[QSCALERS][2][64];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (tid == 0) {
    for (int s = 0; s < QSTAGES_SMALL; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < QSLOTS; b++) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * QSCALERS); }
    s_abort = 0;
    s_most = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_s, 512); tmem_relinquish_pair(); }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  for (int i = tid; i < p.G; i += blockDim.x) {
    s_start[i] = p.group_start[i]; s_rows[i] = rows_inside(p.group_rows[i], s_start[i], p.a_rows, p.error);
    atomicMax(&s_most, s_rows[i]);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int num_kb = p.K / QK;
  const int stages = s_most <= QSMALL ? QSTAGES_SMALL : QSTAGES;
  const int stage_bytes = s_most <= QSMALL ? QSTAGE_SMALL : QSTAGE;
  volatile int* abort_flag = &s_abort;
  const uint32_t peer_abort = mapa_u32(smem_u32(&s_abort), rank ^ 1u);

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      tma_prefetch_desc(&maps.w);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      QWalk walk;
      for (int t = pair; ok; t += npairs) {
        const QTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        const int half = tl.nt / 2;
        const CUtensorMap* tok = &maps.tok[q_tok_box(half)];
        const uint32_t bytes = 2u * (QW_TILE + q_tok_box_bytes(half));
        // (rows of a half-empty last tile belong to the next expert or lie outside: computed, never stored)
        const int w_row = tl.g * p.N + tl.n0 + (int)rank * QHM;
        const int t_row = tl.tok0 + (int)rank * half;
        for (int kb = 0; kb < num_kb; kb++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t* sw = tiles + (size_t)stage * stage_bytes;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], bytes);
          const uint32_t bar0 = mapa_u32(smem_u32(&full_bar[stage]), 0);
          tma_load_2d_pair(sw, &maps.w, kb * QK, w_row, bar0);
          tma_load_2d_pair(sw + QW_TILE, tok, kb * QK, t_row, bar0);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 1); }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (rank-0 CTA only) ----------------
    if (leader && elect_one()) {
      const bool coarse = (p.epilogue & 2) != 0;
      int stage = 0; uint32_t phase = 0;
      unsigned it = 0;   // running K-block count -> TMEM slot ring
      bool ok = true;
      QWalk walk;
      for (int t = pair; ok; t += npairs) {
        const QTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        const uint32_t idesc = umma_idesc(QM, tl.nt, 0 /*e4m3*/);
        for (int kb = 0; kb < num_kb && ok; kb++) {
          // fine scales: one TMEM slot per K block; coarse scales: one per tile, accumulated over all K blocks
          const int slot = it % QSLOTS;
          if (!coarse || kb == 0)
            if (!mbar_wait(&tempty_bar[slot], ((it / QSLOTS) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
          if (!mbar_wait(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint8_t* sa = tiles + (size_t)stage * stage_bytes;
          const uint64_t adesc = umma_desc_sw128(sa);
          const uint64_t bdesc = umma_desc_sw128(sa + QW_TILE);
          const uint32_t d_tmem = tmem_base + (uint32_t)slot * QT;
          #pragma unroll
          for (int kk = 0; kk < QK / 32; kk++)
            umma_f8_pair(d_tmem, adesc + 2u * kk, bdesc + 2u * kk, idesc,
                         (uint32_t)(coarse ? (kb | kk) != 0 : kk != 0));
          umma_commit_pair(&empty_bar[stage]);
          if (!coarse || kb == num_kb - 1) { umma_commit_pair(&tfull_bar[slot]); it++; }
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 2); }
    }
  } else {
    // ---------------- scaling / epilogue (both CTAs) ----------------
    // warps 2..9: lane quarter = warp % 4, half of the tile's tokens = (warp - 2) / 4
    const int q = warp & 3;
    const Scaler w{tfull_bar, mapa_u32(smem_u32(&tempty_bar[0]), 0), abort_flag, &s_scale[warp - 2][0][0],
                   tmem_base + ((uint32_t)(q * 32) << 16), q, (warp - 2) >> 2, lane, (int)rank};
    unsigned it = 0;
    bool ok = true;
    QWalk walk;
    for (int t = pair; ok; t += npairs) {
      const QTile tl = walk.at(p, t, s_rows, s_start);
      if (!tl.valid) break;
      switch (tl.nt) {
        case 32: ok = scale_tile<16>(p, tl, w, it); break;
        case 64: ok = scale_tile<32>(p, tl, w, it); break;
        case 96: ok = scale_tile<48>(p, tl, w, it); break;
        default: ok = scale_tile<64>(p, tl, w, it); break;
      }
    }
    if (!ok && lane == 0) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 3); }
  }

  // ---------------- teardown: nobody leaves while the other CTA may still signal it ----------------
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ---------------- host side ----------------
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn8t() {
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

// [rows, K] bytes row-major, box = box_rows x 128 bytes, 128-byte swizzle
bool make_map8t(CUtensorMap* m, const void* base, unsigned long long rows, unsigned long long K, unsigned box_rows) {
  EncodeTiledFn fn = encode_fn8t();
  if (!fn) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace rbv

// reached through rbv_grouped_gemm_fp8_pair
extern "C" int rbv_grouped_gemm_fp8_tok(const void* A, const float* a_scale_t, long long a_rows, const void* B,
                                         const float* b_scale, void* C, const int* group_start, const int* group_rows,
                                         int G, int N, int K, int ldc, int epilogue, int* error_flag, int max_ctas,
                                         void* cuda_stream) {
  using namespace rbv;
  if (G < 1 || G > kMoeMaxGroups || N % 128 || K % QK || a_rows < 1 || (ldc % 8)) return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return (int)cudaErrorInvalidValue;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(grouped_gemm_fp8_tok_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)QSMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  Fp8TokMaps maps;
  if (!make_map8t(&maps.w, B, (unsigned long long)G * N, (unsigned long long)K, QHM)) return (int)cudaErrorUnknown;
  for (int i = 0; i < 3; i++)
    if (!make_map8t(&maps.tok[i], A, (unsigned long long)a_rows, (unsigned long long)K, 16u << i)) return (int)cudaErrorUnknown;
  Fp8TokParams p;
  p.group_start = group_start; p.group_rows = group_rows; p.G = G; p.N = N; p.K = K; p.ldc = ldc;
  p.a_rows = a_rows; p.a_scale = a_scale_t; p.b_scale = b_scale; p.C = C; p.error = error_flag; p.epilogue = epilogue;
  int grid = max_ctas;
  if (grid <= 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&grid, cudaDevAttrMultiProcessorCount, dev);
  }
  grid &= ~1;   // whole pairs
  if (grid < 2) return (int)cudaErrorInvalidValue;
  return (int)launch_dependent(grouped_gemm_fp8_tok_kernel, grid, QTHREADS, QSMEM, static_cast<cudaStream_t>(cuda_stream), maps, p);
}
