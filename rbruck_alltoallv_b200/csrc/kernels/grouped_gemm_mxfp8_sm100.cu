// MXFP8 grouped GEMM for the expert FFN: e4m3 operands with one power-of-two (UE8M0) scale per 32 elements along K on
// BOTH operands, applied by the tensor core itself (tcgen05.mma.kind::mxf8f6f4.block_scale), on CTA pairs
// (cta_group::2).  This is the fp8 recipe the hardware scales natively: the accumulator of a tile stays in TMEM for the
// whole K loop and is read out once, where the software-scaled kernel (grouped_gemm_fp8_sm100.cu, fp32 scales per
// 1 x 128 / 128 x 128 block) has to pull it out of TMEM after every K block.  No counterpart in the reference.
//
//   C[rows of g] = epi( sum_k  A[row, k] 2^(sa[row, k / 32] - 127) * B_g[n, k] 2^(sb[g, n, k / 32] - 127) )
//
// Scale storage: one uint32 holds the four scales of one 128-wide K block (lowest byte first); the words of 128
// consecutive rows (of A, or of one expert's weight) sit together as one 512-byte "atom" in the order tcgen05.cp wants,
// word (r % 32) * 4 + (r % 128) / 32 for row r:
//   A: sfa[K / 128][ceil(a_rows / 128)][128]        B: sfb[G][K / 128][N / 128][128]
// so that a tile's scales are one 512-byte TMA box per operand and K block.  For the atoms of A to coincide with tiles,
// every group must start at a multiple of 128 rows (checked in the kernel; the MoE layout pads experts accordingly).
// Weight rows are the M operand and tokens the N operand (the token count is the ragged one, and the M of an MMA is
// fixed): two CTAs on neighbouring SMs share a tile of 256 weight rows by up to 256 tokens.  Tiles start at multiples of
// 64 tokens, so that a tile's token scales start at an even TMEM column of one of three atoms, and hold a multiple of 32.
// Per K block (128 bytes of K) each CTA fetches by TMA (no multicast; bytes counted on a barrier of the rank-0 CTA) its
// own 128 weight rows, its own half of the tile's tokens, the scale atom of its weight rows and the one to three scale
// atoms of the tile's tokens.  The rank-0 CTA copies the scales of both CTAs from shared memory into TMEM
// (tcgen05.cp.32x128b.warpx4, 4 + 12 columns per stage) and issues four MMAs (M 256, K 32), each naming its scale byte in
// the instruction descriptor.
// TMEM: three slots of 128 columns for accumulators and 16 columns of scales per stage.  Two tiles of 256 tokens do not
// fit beside the scales, so they take slots 0, 1 and 1, 2 in turn; the epilogue takes the slot that they share into
// registers first and hands it back at once, and the next tile, whose other slot was free all along, starts a TMEM read
// later.  Tiles of up to 128 tokens alternate between slots 0 and 2.
// Why this tile: per K block an SM's shared memory takes the stage's 34 KB from L2 and gives the MMAs 128 weight rows and
// half the tokens for each 32 bytes of K; the more tokens an MMA has, the less of that is weights.  Measured on one B200,
// 8 experts, hidden 4096, FFN 14336, up / down GEMM in us, against 256 tokens (as M) by 128 weight rows: 64 tokens
// 218 / 122 -> 178 / 105, 1000 tokens 268 / 154 -> 245 / 154, 2000 tokens 456 / 224 -> 423 / 195, 8192 tokens 2098 / 1052
// -> 1534 / 712.  On the way: 128 tokens by 256 weight rows 531 / 270 at 2000 tokens, 192 by 256 455 / 238, two MMAs of
// 128 tokens each instead of one of 256 443 / 205.
// Short K makes the epilogue the bound (1024 / 2816, 4 experts of 616 rows: 88 us with four epilogue warps and tiles of 256
// only, 70 with eight and the tile size below, 77 before).
// Epilogues: bf16; SwiGLU to bf16; SwiGLU followed by the MXFP8 quantiser of the next GEMM's operand (32 tokens at a time
// change hands through shared memory, so that eight lanes hold the 32 values that share a scale); and, for the down GEMM
// of the MoE layer, bf16 rows stored straight into the buffers of the GPUs the tokens came from (the return all-to-all,
// overlapped with the MMAs of the other tiles).  All waits are bounded; on expiry both CTAs are told, record an error,
// release their TMEM and return.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels/mx_quant.cuh"
#include "kernels/pdl.cuh"
#include "kernels/sm100_ptx.cuh"
#include "kernels/tok_epilogue.cuh"
#include "rbv/moe.h"

namespace rbv {

using namespace sm100;

namespace {

constexpr int XM = 256;                 // weight rows (output columns) per pair tile
constexpr int XHM = 128;                // weight rows per CTA
constexpr int XT = 256;                 // most tokens per tile
constexpr int XSUB = 128;               // tokens (columns) per accumulator slot
constexpr int XU = 32;                  // a tile's token count is a multiple of this
constexpr int XS = 64;                  // a tile starts at a multiple of this many tokens of its group
constexpr int XK = 128;                 // bytes of K per pipeline stage (one 128-byte swizzle row, four scale blocks)
constexpr int XW_TILE = XHM * XK;       // 16 KB of weights
constexpr int XT_TILE = XT / 2 * XK;    // up to 16 KB of tokens
constexpr int XSF_TILE = 512;           // an atom: 128 scale words
// Pipeline: 6 stages with room for the tokens (and their three atoms) of a full tile; where no group has more than 64 rows,
// 9 stages with room for 64 tokens and their one atom: the kernel then is a stream of weights, and what counts is how many
// of their bytes are on the way.
constexpr int XSTAGES = 6, XSTAGE = XW_TILE + XT_TILE + 4 * XSF_TILE;                              // 34 KB
constexpr int XSMALL = 64, XSTAGES_SMALL = 9, XSTAGE_SMALL = XW_TILE + XSMALL / 2 * XK + 4 * XSF_TILE;   // 22 KB
static_assert(XSTAGES * XSTAGE >= XSTAGES_SMALL * XSTAGE_SMALL, "shared memory");
constexpr int XEPI = 8;                 // epilogue warps: two groups of four (one per TMEM lane quarter), every other 32 tokens each
constexpr int XTHREADS = 64 + 32 * XEPI;   // and the TMA and the MMA warp
constexpr int XACCS = 3;                // accumulator slots
constexpr int XACC_COLS = XACCS * XSUB;
constexpr int XSF_COLS = 16, XSF_COLS_SMALL = 8;   // TMEM columns of scales per stage: 4 for the weights, 12 (4) for the tokens
static_assert(XACC_COLS + XSTAGES * XSF_COLS <= 512 && XACC_COLS + XSTAGES_SMALL * XSF_COLS_SMALL <= 512, "TMEM");
// quantising epilogue: a buffer of 32 tokens x 64 outputs per group; rows 80 floats apart, so that the even lanes' token and
// the odd lanes' token fall into different halves of the banks
constexpr int XQ_LD = 80;
constexpr int XQ_BUF = XU * XQ_LD * 4;  // 10 KB
constexpr size_t XSMEM = (size_t)XSTAGES * XSTAGE + 2 * XQ_BUF + 1024;

// Token boxes of 16, 32, 64 and 128 rows: a CTA's half of a tile is fetched with the smallest that covers it.
struct MxMaps { CUtensorMap w, sfw, sft, tok[4]; };

struct MxParams {
  const int* group_start;
  const int* group_rows;
  int G, N, K, ldc;
  long long a_rows;            // rows of A
  int a_row_blocks;            // ceil(a_rows / 128): scale atoms of A per K block
  void* C;
  uint32_t* sf_out;            // epilogue 3: scale words of the quantised output, [N / 256][a_row_blocks][128]
  int* error;
  int epilogue;                // 0: C = bf16(acc); 1: SwiGLU over interleaved gate / up columns, bf16;
                               // 3: SwiGLU, then MXFP8 again: C is e4m3 [*, N / 2] (ldc in bytes) with sf_out
  // Push mode (ret != null, epilogue 0): row `pos` of the result goes to row (ret[pos] & 0xffffff) of the [*, N] bf16
  // buffer at offset y2_off of the heap of process ret[pos] >> 24: the return all-to-all of the MoE layer.
  const unsigned* ret;
  unsigned long long y2_off;
  char* heap[16];
};

struct XTile { int g, tok0, ntok, nt, n0; bool valid; };   // group, first token row, live tokens, columns, first weight row

// Walks the tile schedule (groups in order, weight rows slow, tokens fast); `at(t)` wants non-decreasing t.
struct MxWalk {
  const int cap;           // most tokens of a tile, in units of XS
  int g = 0, before = 0;   // tiles of the groups in front of g
  __device__ explicit MxWalk(int c) : cap(c) {}
  __device__ __forceinline__ XTile at(const MxParams& p, int t, const int* s_rows, const int* s_start) {
    XTile r; r.valid = false; r.g = r.tok0 = r.ntok = r.nt = r.n0 = 0;
    const int ntn = (p.N + XM - 1) / XM;     // N is a multiple of 128: the last tile may be half empty
    for (; g < p.G; g++) {
      const int units = (s_rows[g] + XS - 1) / XS, ntm = (units + cap - 1) / cap;
      const int cnt = ntm * ntn;
      if (t - before < cnt) {
        const int n = (t - before) / ntm, m = (t - before) - n * ntm;
        const int base = units / ntm, extra = units - base * ntm;     // the first `extra` tiles are one unit larger
        const int u0 = m * base + min(m, extra), nu = base + (m < extra ? 1 : 0);
        r.g = g; r.tok0 = s_start[g] + u0 * XS; r.n0 = n * XM;
        r.ntok = min(s_rows[g] - u0 * XS, nu * XS); r.nt = (r.ntok + XU - 1) / XU * XU;
        r.valid = true;
        return r;
      }
      before += cnt;
    }
    return r;
  }
};

__device__ __forceinline__ int mx_tok_box(int half) { return half <= 16 ? 0 : half <= 32 ? 1 : half <= 64 ? 2 : 3; }
__device__ __forceinline__ uint32_t mx_tok_box_bytes(int half) { return (16u << mx_tok_box(half)) * XK; }

// Accumulator slots of the tiles of one CTA pair, in order; every role walks the same sequence.
struct MxSlots {
  unsigned odd = 0;            // which of the two places the next tile takes
  uint32_t phases = 0;         // bit s: parity of the uses of slot s so far
  int first, count;            // slots of the current tile
  __device__ __forceinline__ void next(const XTile& t) {
    count = t.nt > XSUB ? 2 : 1;
    first = odd ? (count == 2 ? 1 : 2) : 0;
    odd ^= 1u;
  }
  __device__ __forceinline__ uint32_t phase(int slot) const { return (phases >> slot) & 1u; }
  __device__ __forceinline__ void used(int slot) { phases ^= 1u << slot; }
};

// Scale atoms that cover the tokens of a tile: tok0 is a multiple of 64, and group starts of 128.
__device__ __forceinline__ int mx_tok_atoms(const XTile& t) { return ((t.tok0 & 127) + t.nt + 127) / 128; }

// Instruction descriptor of the block-scaled kinds: e4m3 x e4m3, K-major operands, UE8M0 scales; the scale byte each
// operand uses (0..3 inside its TMEM word) is added per MMA.
__host__ __device__ constexpr uint32_t umma_idesc_block_scaled(int M, int N) {
  return ((uint32_t)(N >> 3) << 17) | (1u << 23) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ uint32_t with_scale_ids(uint32_t idesc, uint32_t a_id, uint32_t b_id) {
  return idesc | (b_id << 4) | (a_id << 29);
}

// Shared-memory descriptor of 32 rows x 16 bytes without swizzle (8-row groups 128 bytes apart): the source of a
// tcgen05.cp.32x128b.
__device__ __forceinline__ uint64_t desc_rows16(const void* smem) {
  const uint64_t addr = (smem_u32(smem) & 0x3FFFFu) >> 4;
  return addr | (8ull << 32) | (1ull << 46);
}

// 32 rows x 128 bits from the shared memory of each CTA of the pair into 4 TMEM columns of that CTA, replicated
// over the four lane quarters.
__device__ __forceinline__ void tmem_cp_scales_pair(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}

// The four epilogue warps of a group: barrier, and barrier with a vote.
__device__ __forceinline__ void epi_barrier(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }
__device__ __forceinline__ bool epi_all(int group, bool pred) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, 128, p;\n\t"
      "selp.b32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"((uint32_t)pred), "r"(1 + group) : "memory");
  return all != 0;
}

__device__ __forceinline__ void umma_mxf8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                               uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(tsfa), "r"(tsfb), "r"(accumulate)
      : "memory");
}

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(XTHREADS, 1)
grouped_gemm_mxfp8_kernel(const __grid_constant__ MxMaps maps, const __grid_constant__ MxParams p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[XSTAGES_SMALL];    // rank-0 CTA: operand and scale bytes of both CTAs
  __shared__ __align__(8) uint64_t empty_bar[XSTAGES_SMALL];   // each CTA: its stage has been read by the MMAs
  __shared__ __align__(8) uint64_t tfull_bar[XACCS];     // each CTA: the accumulator is complete
  __shared__ __align__(8) uint64_t tempty_bar[XACCS];    // rank-0 CTA: both CTAs have taken the accumulator
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_rows[kMoeMaxGroups], s_start[kMoeMaxGroups];
  __shared__ int s_abort, s_bad, s_cap, s_most;          // s_most: rows of the largest group
  __shared__ int s_tiles[3];                             // tiles of the schedule with at most 128, 192, 256 tokens each

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  int npairs = gridDim.x >> 1;

  if (tid == 0) {
    s_bad = 0;
    s_most = 0;
    s_tiles[0] = s_tiles[1] = s_tiles[2] = 0;
    for (int s = 0; s < XSTAGES_SMALL; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < XACCS; b++) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * XEPI); }
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_s, 512); tmem_relinquish_pair(); }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  for (int i = tid; i < p.G; i += blockDim.x) {
    s_start[i] = p.group_start[i]; s_rows[i] = rows_inside(p.group_rows[i], s_start[i], p.a_rows, p.error);
    if (s_rows[i] > 0 && (s_start[i] & 127)) s_bad = 1;   // the scale atoms of A would not coincide with the tiles
    atomicMax(&s_most, s_rows[i]);
    const int units = (s_rows[i] + XS - 1) / XS;
    #pragma unroll
    for (int c = 0; c < 3; c++) atomicAdd(&s_tiles[c], (units + c + 1) / (c + 2) * ((p.N + XM - 1) / XM));
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0) {
    // Rounds of tiles over the SM pairs, times what a K block of such a tile takes: 311 ns with 128 tokens, 380 with 190,
    // 465 with 240, which is about 96 tokens plus its own.  (A few large tiles may leave most pairs idle in the last
    // round, and the same groups in smaller ones fill it.)
    int best = 0x7fffffff;
    for (int c = 2; c >= 0; c--) {
      const int cost = (s_tiles[c] + npairs - 1) / npairs * ((c + 2) * XS + 96);
      if (cost < best) { best = cost; s_cap = c + 2; }
    }
  }
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const int num_kb = s_bad ? 0 : p.K / XK;
  const bool small = s_most <= XSMALL;
  const int stages = small ? XSTAGES_SMALL : XSTAGES;
  const int stage_bytes = small ? XSTAGE_SMALL : XSTAGE, sf_at = stage_bytes - 4 * XSF_TILE;   // scale atoms inside a stage
  const uint32_t sf_cols = small ? XSF_COLS_SMALL : XSF_COLS;
  if (s_bad) {   // both CTAs see the same arrays: nobody does anything, the error is recorded once
    if (blockIdx.x == 0 && tid == 0) atomicExch(p.error, 5);
    npairs = 1 << 30;
  }
  const int first_tile = s_bad ? (1 << 30) : pair;
  volatile int* abort_flag = &s_abort;
  const uint32_t peer_abort = mapa_u32(smem_u32(&s_abort), rank ^ 1u);

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one()) {
      tma_prefetch_desc(&maps.w);
      tma_prefetch_desc(&maps.sfw);
      tma_prefetch_desc(&maps.sft);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      const int nb128 = p.N / 128;
      MxWalk walk(s_cap);
      for (int t = first_tile; ok; t += npairs) {
        const XTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        const int half = tl.nt / 2;
        const CUtensorMap* tok = &maps.tok[mx_tok_box(half)];
        const int atoms = mx_tok_atoms(tl);
        const uint32_t bytes = 2u * (XW_TILE + mx_tok_box_bytes(half) + (uint32_t)(1 + atoms) * XSF_TILE);
        const int n_row = tl.n0 + (int)rank * XHM;
        for (int kb = 0; kb < num_kb; kb++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t* sw = tiles + (size_t)stage * stage_bytes;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], bytes);
          const uint32_t bar0 = mapa_u32(smem_u32(&full_bar[stage]), 0);
          // (rows of a half-empty last tile belong to the next expert or lie outside: computed, never stored)
          tma_load_2d_pair(sw, &maps.w, kb * XK, tl.g * p.N + n_row, bar0);
          tma_load_2d_pair(sw + XW_TILE, tok, kb * XK, tl.tok0 + (int)rank * half, bar0);
          tma_load_2d_pair(sw + sf_at, &maps.sfw, 0, (tl.g * num_kb + kb) * nb128 + n_row / 128, bar0);
          for (int j = 0; j < atoms; j++)
            tma_load_2d_pair(sw + sf_at + (1 + j) * XSF_TILE, &maps.sft, 0,
                             kb * p.a_row_blocks + tl.tok0 / 128 + j, bar0);
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
      MxSlots slots;
      MxWalk walk(s_cap);
      for (int t = first_tile; ok; t += npairs) {
        const XTile tl = walk.at(p, t, s_rows, s_start);
        if (!tl.valid) break;
        slots.next(tl);
        for (int s = slots.first; s < slots.first + slots.count && ok; s++) {
          ok = mbar_wait(&tempty_bar[s], slots.phase(s) ^ 1u, abort_flag);
          slots.used(s);
        }
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t idesc = umma_idesc_block_scaled(XM, tl.nt);
        const uint32_t d_tmem = tmem_base + (uint32_t)slots.first * XSUB;
        const int atoms = mx_tok_atoms(tl);
        const uint32_t sf_shift = (uint32_t)(tl.tok0 & 127) / 32;   // TMEM column of the tile's first token: 0 or 2
        auto copy_scales = [&](int st) {
          const uint8_t* sf = tiles + (size_t)st * stage_bytes + sf_at;
          const uint32_t to = tmem_base + XACC_COLS + (uint32_t)st * sf_cols;
          tmem_cp_scales_pair(to, desc_rows16(sf));
          for (int j = 0; j < atoms; j++) tmem_cp_scales_pair(to + 4u + 4u * (uint32_t)j, desc_rows16(sf + (1 + j) * XSF_TILE));
        };
        // The scales of the next K block are copied in front of the MMAs of this one when they are there already, so that
        // the copies (which MMAs have to wait for) run beside MMAs.
        bool copied = false;
        for (int kb = 0; kb < num_kb; kb++) {
          if (!copied) {
            if (!mbar_wait(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
            tc_fence_after_sync();
            copy_scales(stage);
          }
          const int next = stage + 1 == stages ? 0 : stage + 1;
          const uint32_t next_phase = next ? phase : phase ^ 1u;
          copied = kb + 1 < num_kb && mbar_try_wait(&full_bar[next], next_phase);
          if (copied) {
            tc_fence_after_sync();
            copy_scales(next);
          }
          const uint8_t* sw = tiles + (size_t)stage * stage_bytes;
          const uint64_t wdesc = umma_desc_sw128(sw);
          const uint32_t tsfw = tmem_base + XACC_COLS + (uint32_t)stage * sf_cols;
          const uint64_t tdesc = umma_desc_sw128(sw + XW_TILE);
          #pragma unroll
          for (int kk = 0; kk < XK / 32; kk++)
            umma_mxf8_pair(d_tmem, wdesc + 2u * kk, tdesc + 2u * kk, with_scale_ids(idesc, kk, kk), tsfw, tsfw + 4 + sf_shift,
                           (uint32_t)((kb | kk) != 0));
          umma_commit_pair(&empty_bar[stage]);   // frees this stage (operands and scales) in both CTAs
          stage = next; phase = next_phase;
        }
        for (int s = slots.first; s < slots.first + slots.count && ok; s++) umma_commit_pair(&tfull_bar[s]);
      }
      if (!ok) { s_abort = 1; st_cluster_u32(peer_abort, 1); atomicExch(p.error, 2); }
    }
  } else {
    // ---------------- epilogue (both CTAs): warps 2..9, TMEM lane quarter = warp % 4, group = (warp - 2) / 4 ----------------
    const int q = warp & 3;
    const bool odd = (lane & 1) != 0;
    const int group = (warp - 2) >> 2;
    float* const buf = reinterpret_cast<float*>(tiles + (size_t)XSTAGES * XSTAGE) + group * (XU * XQ_LD);
    __nv_bfloat16* C = static_cast<__nv_bfloat16*>(p.C);
    const uint32_t tempty0 = mapa_u32(smem_u32(&tempty_bar[0]), 0);
    bool ok = true;
    MxSlots slots;
    MxWalk walk(s_cap);
    for (int t = first_tile; ok; t += npairs) {
      const XTile tl = walk.at(p, t, s_rows, s_start);
      if (!tl.valid) break;
      const int n_cta = tl.n0 + (int)rank * XHM;     // this CTA's first output column
      const bool inside = n_cta < p.N;
      const int nw = n_cta + q * 32;
      // tokens c .. c + 31 of the tile
      auto store_chunk = [&](const uint32_t (&r)[32], int c) {
        const int live = inside ? tl.ntok - c : 0;
        unsigned rv = 0;   // push mode: where the token of this lane's index goes, handed out by shuffle
        if (p.ret && c + lane < tl.ntok) rv = __ldg(p.ret + tl.tok0 + c + lane);
        if (p.epilogue == 3) {
          // SwiGLU, then the quantiser of the next GEMM's operand: 32 tokens x 64 outputs of this CTA go through shared
          // memory, after which 16 lanes hold a token's 64 outputs, four each, and 8 lanes the 32 that share a scale.
          #pragma unroll
          for (int k = 0; k < 32; k += 2)
            buf[(k + (odd ? 1 : 0)) * XQ_LD + q * 16 + (lane >> 1)] = tokepi::swiglu_pair(r, k, odd);
          epi_barrier(group);
          #pragma unroll
          for (int u = 0; u < 4; u++) {
            const int tok = u * 8 + q * 2 + (lane >> 4), l16 = lane & 15;
            const float4 o = *reinterpret_cast<const float4*>(buf + tok * XQ_LD + l16 * 4);
            float m = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), fabsf(o.w)));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
            const int e = mx_exponent(m);
            const float inv = mx_inv_scale(e);
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(o.x * inv, o.y * inv), __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(o.z * inv, o.w * inv), __NV_SATFINITE, __NV_E4M3);
            if (tok < live) {
              const unsigned R = (unsigned)(tl.tok0 + c + tok);
              const int n_out = n_cta / 2;
              *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.C) + (size_t)R * p.ldc + n_out + l16 * 4) = lo | (hi << 16);
              if ((l16 & 7) == 0) {
                uint32_t* word = p.sf_out + ((size_t)(n_out / 128) * p.a_row_blocks + R / 128) * 128 + (R % 32) * 4 + (R % 128) / 32;
                reinterpret_cast<uint8_t*>(word)[(n_out / 32 & 3) + (l16 >> 3)] = (uint8_t)(e + 127);
              }
            }
          }
          epi_barrier(group);   // read by all before the next tokens are written
        } else {
          __nv_bfloat16* rows = C + (size_t)(tl.tok0 + c) * p.ldc;
          if (p.epilogue == 1) {
            tokepi::store_swiglu(r, rows, p.ldc, nw / 2, live, lane);
          } else if (p.ret) {
            tokepi::store_plain(r, [&](int tok) {
              const unsigned to = __shfl_sync(0xffffffffu, rv, tok);
              return reinterpret_cast<__nv_bfloat16*>(p.heap[to >> 24] + p.y2_off) + (size_t)(to & 0xffffffu) * p.ldc;
            }, nw, live, lane);
          } else {
            tokepi::store_plain(r, [&](int tok) { return rows + (size_t)tok * p.ldc; }, nw, live, lane);
          }
        }
      };
      slots.next(tl);
      for (int i = 0; i < slots.count; i++) {
        // of two slots the one that the next tile wants, slot 1, goes first
        const int b = slots.count == 2 ? (i == 0 ? 1 : slots.first == 0 ? 0 : 2) : slots.first;
        const int s = b - slots.first;       // tokens s * 128 ...
        // (the four warps of a group meet at a named barrier when they quantise: they leave the loop together, see the vote)
        const bool got_it = mbar_wait(&tfull_bar[b], slots.phase(b), abort_flag);
        slots.used(b);
        if (p.epilogue == 3 ? !epi_all(group, got_it) : !got_it) { ok = false; break; }
        tc_fence_after_sync();
        // this group's tokens of the slot: 32 group ... and 64 + 32 group ...
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * XSUB);
        const int n = min(tl.nt - s * XSUB, XSUB);
        uint32_t r[XSUB / 64][32];
        #pragma unroll
        for (int k = 0; k < XSUB / 64; k++)
          if (k * 64 + group * 32 < n) tmem_ld32(taddr + k * 64 + group * 32, r[k]);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tempty0 + 8u * (uint32_t)b);   // 8 warps x 2 CTAs
        #pragma unroll
        for (int k = 0; k < XSUB / 64; k++)
          if (k * 64 + group * 32 < n) store_chunk(r[k], s * XSUB + k * 64 + group * 32);
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

// Row-wise MXFP8 quantisation of bf16 activations: per (row, 32 columns) a power-of-two scale 2^e >= amax / 448 and
// out = x / 2^e as e4m3.  One half-warp handles one 128-column block: sixteen lanes x 8 bf16 (one 16-byte load
// each), so a block of 32 columns is 4 neighbouring lanes.  The four scale bytes of a 128-column block are packed
// into one word; words are stored in the atom order of the GEMM: sf[K / 128][ceil(rows / 128)][128], word
// (r % 32) * 4 + (r % 128) / 32 of its atom for row r.
__global__ void __launch_bounds__(256)
quantize_rows_mx_kernel(const __nv_bfloat16* __restrict__ x, long long rows, int K, int ldx, uint8_t* __restrict__ out,
                        uint32_t* __restrict__ sf) {
  constexpr int kUnroll = 4;
  const int lane16 = threadIdx.x & 15;
  const unsigned kblocks = (unsigned)(K / 128);
  const unsigned nblk = (unsigned)(rows * kblocks);
  const unsigned groups = (gridDim.x * blockDim.x) >> 4;
  const unsigned g0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const unsigned which = g0 & 1u;
  for (unsigned base = g0 - which; base < nblk; base += groups * kUnroll) {
    uint4 raw[kUnroll];
    unsigned row[kUnroll], kb[kUnroll];
    #pragma unroll
    for (int u = 0; u < kUnroll; u++) {
      const unsigned w = base + which + (unsigned)u * groups;
      raw[u] = make_uint4(0u, 0u, 0u, 0u);
      row[u] = w / kblocks;
      kb[u] = w - row[u] * kblocks;
      if (w < nblk)
        raw[u] = __ldg(reinterpret_cast<const uint4*>(x + (size_t)row[u] * ldx + kb[u] * 128 + lane16 * 8));
    }
    #pragma unroll
    for (int u = 0; u < kUnroll; u++) {
      const unsigned w = base + which + (unsigned)u * groups;
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
      float2 v[4];
      float m = 0.0f;
      #pragma unroll
      for (int j = 0; j < 4; j++) {
        v[j] = __bfloat1622float2(h[j]);
        m = fmaxf(m, fmaxf(fabsf(v[j].x), fabsf(v[j].y)));
      }
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));   // the 4 lanes of one 32-column block
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      const int e = mx_exponent(m);
      const float inv = mx_inv_scale(e);
      const uint32_t byte = (uint32_t)(e + 127);
      // the four blocks of the 128 columns: lanes 0-3, 4-7, 8-11, 12-15 -> bytes 0..3
      uint32_t word = byte << (8 * (lane16 >> 2));
      word |= __shfl_xor_sync(0xffffffffu, word, 4);
      word |= __shfl_xor_sync(0xffffffffu, word, 8);
      if (w < nblk) {
        uint32_t qv[4];
        #pragma unroll
        for (int j = 0; j < 4; j++)
          qv[j] = __nv_cvt_float2_to_fp8x2(make_float2(v[j].x * inv, v[j].y * inv), __NV_SATFINITE, __NV_E4M3);
        *reinterpret_cast<uint2*>(out + (size_t)row[u] * K + kb[u] * 128 + lane16 * 8) =
            make_uint2(qv[0] | (qv[1] << 16), qv[2] | (qv[3] << 16));
        if (lane16 == 0) {
          const unsigned r = row[u], nrb = (unsigned)((rows + 127) / 128);
          sf[((size_t)kb[u] * nrb + r / 128) * 128 + (r % 32) * 4 + (r % 128) / 32] = word;
        }
      }
    }
  }
}

// ---------------- host side ----------------
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn_mx() {
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
bool make_map_mx(CUtensorMap* m, const void* base, unsigned long long rows, unsigned long long K, unsigned box_rows) {
  EncodeTiledFn fn = encode_fn_mx();
  if (!fn) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// scale atoms: [atoms, 128] uint32 row-major, box = one atom (512 bytes), no swizzle
bool make_map_atoms(CUtensorMap* m, const void* base, unsigned long long atoms) {
  EncodeTiledFn fn = encode_fn_mx();
  if (!fn) return false;
  cuuint64_t dims[2] = {128, atoms};
  cuuint64_t strides[1] = {512};
  cuuint32_t box[2] = {128, 1};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace rbv

static int launch_mxfp8(const void* A, const void* sfa, long long a_rows, const void* B, const void* sfb, void* C,
                        void* sf_out, const int* group_start, const int* group_rows, int G, int N, int K, int ldc,
                        int epilogue, int* error_flag, int max_ctas, void* cuda_stream, const unsigned* ret = nullptr,
                        const void* const* heaps = nullptr, int nheaps = 0, unsigned long long y2_off = 0) {
  using namespace rbv;
  if (ret && (epilogue != 0 || !heaps || nheaps < 1 || nheaps > 16 || (y2_off & 15))) return (int)cudaErrorInvalidValue;
  if (G < 1 || G > kMoeMaxGroups || N % 128 || K % XK || a_rows < 1 || (ldc % 8)) return (int)cudaErrorInvalidValue;
  if (epilogue == 3 && (!sf_out || N % 256 || ldc % 16 || (reinterpret_cast<uintptr_t>(sf_out) & 15)))
    return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return (int)cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(sfa) | reinterpret_cast<uintptr_t>(sfb)) & 15) return (int)cudaErrorInvalidValue;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(grouped_gemm_mxfp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)XSMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const unsigned long long nrb = (unsigned long long)((a_rows + 127) / 128), nkb = (unsigned long long)(K / XK);
  MxMaps maps;
  if (!make_map_mx(&maps.w, B, (unsigned long long)G * N, (unsigned long long)K, XHM)) return (int)cudaErrorUnknown;
  for (int i = 0; i < 4; i++)
    if (!make_map_mx(&maps.tok[i], A, (unsigned long long)a_rows, (unsigned long long)K, 16u << i)) return (int)cudaErrorUnknown;
  if (!make_map_atoms(&maps.sft, sfa, nkb * nrb)) return (int)cudaErrorUnknown;
  if (!make_map_atoms(&maps.sfw, sfb, (unsigned long long)G * nkb * (unsigned long long)(N / 128))) return (int)cudaErrorUnknown;
  MxParams p;
  p.group_start = group_start; p.group_rows = group_rows; p.G = G; p.N = N; p.K = K; p.ldc = ldc;
  p.a_rows = a_rows; p.a_row_blocks = (int)nrb;
  p.C = C; p.sf_out = static_cast<uint32_t*>(sf_out); p.error = error_flag; p.epilogue = epilogue;
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
  return (int)launch_dependent(grouped_gemm_mxfp8_kernel, grid, XTHREADS, XSMEM, static_cast<cudaStream_t>(cuda_stream),
                               maps, p);
}

extern "C" int rbv_grouped_gemm_mxfp8(const void* A, const void* sfa, long long a_rows, const void* B, const void* sfb,
                                      void* C, const int* group_start, const int* group_rows, int G, int N, int K,
                                      int ldc, int epilogue, int* error_flag, int max_ctas, void* cuda_stream) {
  if (epilogue != 0 && epilogue != 1) return (int)cudaErrorInvalidValue;
  return launch_mxfp8(A, sfa, a_rows, B, sfb, C, nullptr, group_start, group_rows, G, N, K, ldc, epilogue, error_flag,
                      max_ctas, cuda_stream);
}

extern "C" int rbv_grouped_gemm_mxfp8_push(const void* A, const void* sfa, long long a_rows, const void* B,
                                           const void* sfb, const int* group_start, const int* group_rows, int G,
                                           int N, int K, const unsigned* ret, const void* const* heaps, int nheaps,
                                           unsigned long long y2_off, int* error_flag, int max_ctas,
                                           void* cuda_stream) {
  if (!ret) return (int)cudaErrorInvalidValue;
  return launch_mxfp8(A, sfa, a_rows, B, sfb, const_cast<void*>(heaps ? heaps[0] : nullptr), nullptr, group_start,
                      group_rows, G, N, K, N, 0, error_flag, max_ctas, cuda_stream, ret, heaps, nheaps, y2_off);
}

extern "C" int rbv_grouped_gemm_mxfp8_swiglu_q(const void* A, const void* sfa, long long a_rows, const void* B,
                                               const void* sfb, void* Cq, void* sf_out, const int* group_start,
                                               const int* group_rows, int G, int N, int K, int ldc_bytes,
                                               int* error_flag, int max_ctas, void* cuda_stream) {
  return launch_mxfp8(A, sfa, a_rows, B, sfb, Cq, sf_out, group_start, group_rows, G, N, K, ldc_bytes, 3, error_flag,
                      max_ctas, cuda_stream);
}

extern "C" int rbv_quantize_rows_mxfp8(const void* x_bf16, long long rows, int K, int ldx, void* out_fp8, void* sf,
                                       void* cuda_stream) {
  using namespace rbv;
  if (K % 128 || rows < 1 || (ldx % 8) || (reinterpret_cast<uintptr_t>(x_bf16) & 15) ||
      (reinterpret_cast<uintptr_t>(out_fp8) & 7) || (reinterpret_cast<uintptr_t>(sf) & 15))
    return (int)cudaErrorInvalidValue;
  const long long nblk = rows * (K / 128);
  if (nblk >= (1ll << 31)) return (int)cudaErrorInvalidValue;
  long long grid = (nblk + 63) / 64;
  if (grid > 148 * 8) grid = 148 * 8;
  if (grid < 1) grid = 1;
  quantize_rows_mx_kernel<<<(int)grid, 256, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      static_cast<const __nv_bfloat16*>(x_bf16), rows, K, ldx, static_cast<uint8_t*>(out_fp8),
      static_cast<uint32_t*>(sf));
  return (int)cudaGetLastError();
}
