// Byte copy of any alignment by one warp.  Made of three accesses (ld_cg_v4, ld_cg_u8, st_v4) and shuffles that the
// including file declares first: primitives.cuh on the GPU, stand-ins that check every address in a test on the host.
#pragma once
#include <cstddef>
#include <cstdint>

namespace rbv {
namespace dev {

// The 16 bytes that start `sh` (0..15) bytes into the 32-byte pair (a, b).
__device__ __forceinline__ uint4 shift16(const uint4& a, const uint4& b, unsigned sh) {
  unsigned w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  #pragma unroll
  for (int i = 0; i < 6; i++) w[i] = (sh & 8u) ? w[i + 2] : w[i];
  #pragma unroll
  for (int i = 0; i < 5; i++) w[i] = (sh & 4u) ? w[i + 1] : w[i];
  const unsigned bits = (sh & 3u) * 8u;
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits),
                    __funnelshift_r(w[2], w[3], bits), __funnelshift_r(w[3], w[4], bits));
}

// Output vectors [base, base + 32 V) of a warp's copy, those of them that lie in [0, nvec).  s is aligned; output vector i
// is source vector i (sh = 0) or is cut out of source vectors i and i + 1 at byte sh, where vector i + 1 comes by shuffle
// from the lane that loaded it.  ALL: the range lies inside.  `between` runs when the loads have been issued.
template <int V, bool ALL, typename F>
__device__ __forceinline__ void copy_round(uint4* o, const uint4* s, long long base, long long nvec, unsigned sh, unsigned lane,
                                           F&& between) {
  const long long i0 = base + lane, end = nvec + (sh ? 1 : 0);   // a shifted copy also reads the vector behind the last
  uint4 v[V], more = make_uint4(0u, 0u, 0u, 0u);
  #pragma unroll
  for (int j = 0; j < V; j++) {
    if (!ALL) v[j] = more;
    if (ALL || (i0 + j * 32 >= 0 && i0 + j * 32 < end)) v[j] = ld_cg_v4(s + i0 + j * 32);
  }
  if (sh && lane == 0 && base + V * 32 < end) more = ld_cg_v4(s + base + V * 32);
  between();
  if (sh == 0) {
    #pragma unroll
    for (int j = 0; j < V; j++)
      if (ALL || (i0 + j * 32 >= 0 && i0 + j * 32 < nvec)) st_v4(o + i0 + j * 32, v[j]);
    return;
  }
  #pragma unroll
  for (int j = 0; j < V; j++) {
    // the next vector: of the next lane, and for the last lane of lane 0's next one
    const uint4 give = lane == 0 ? (j + 1 < V ? v[j + 1 < V ? j + 1 : j] : more) : v[j];
    uint4 next;
    next.x = __shfl_sync(0xffffffffu, give.x, (lane + 1) & 31u);
    next.y = __shfl_sync(0xffffffffu, give.y, (lane + 1) & 31u);
    next.z = __shfl_sync(0xffffffffu, give.z, (lane + 1) & 31u);
    next.w = __shfl_sync(0xffffffffu, give.w, (lane + 1) & 31u);
    if (ALL || (i0 + j * 32 >= 0 && i0 + j * 32 < nvec)) st_v4(o + i0 + j * 32, shift16(v[j], next, sh));
  }
}

// Copies n bytes with one warp.  dst and src may have any alignment, relative to each other too; stores are 16-byte
// aligned vectors.  Loads bypass L1 (the source may have been written by another GPU).  All lanes call it together.
//
// Bound by the latency of memory for short blocks and by the bytes in flight for long ones, so that every load of a round
// is issued before anything is stored: the bytes in front of and behind the vectors, and up to U vectors per lane whatever
// the alignment.  (Bytes, the vectors in front of the first line, and the rest one after the other cost a block three
// trips to memory, and a misaligned copy, which blocks of bf16 elements usually are, had four vectors per lane in
// flight.)  Measured on one B200, persistent calls of 8 ranks: Zipf blocks up to 64 KB 6.1 -> 4.65 us; blocks up to 4 MB
// of bf16, direct 103 -> 94 us, two-layer 137 -> 117 us.  A short rest takes a round of its own size: with the
// instructions of a full one Bruck over blocks of up to 1 KB took 10.0 instead of 6.2 us.  U = 16 moves long blocks
// another 7 % faster in a2av_local.cu and nothing else (a2av_static.cu: two-layer 117 -> 123 us).
// The first vector of every round lies on a 128-byte line of the destination (blocks of 1 KB and more): a peer GPU
// receives a line that is written in two pieces as two NVLink packets with one header each, which costs a fifth of the
// link when 512-byte warp stores start in the middle of a line.
template <int U = 8>
__device__ __forceinline__ void warp_copy(char* dst, const char* src, size_t n, unsigned lane) {
  if (n == 0) return;
  size_t head = (16 - ((uintptr_t)dst & 15)) & 15;
  if (head > n) head = n;
  char* const d = dst + head;
  const char* const from = src + head;
  const long long nvec = (long long)((n - head) >> 4);
  const unsigned tail = (unsigned)(n - head) & 15u;
  unsigned char first = 0, last = 0;
  if (lane < head) first = ld_cg_u8((const unsigned char*)src + lane);
  if (lane < tail) last = ld_cg_u8((const unsigned char*)from + (nvec << 4) + lane);
  bool ragged = true;                          // the bytes around the vectors are still to be stored
  auto ends = [&]() {
    if (ragged) {
      if (lane < head) dst[lane] = (char)first;
      if (lane < tail) d[(nvec << 4) + lane] = (char)last;
    }
    ragged = false;
  };
  const unsigned sh = (unsigned)((uintptr_t)from & 15);
  const uint4* const s = reinterpret_cast<const uint4*>(from - sh);
  uint4* const o = reinterpret_cast<uint4*>(d);
  // vector of lane 0 in the first round.  A full round in front of vector 0 masks its lanes; only what follows it is taken
  // without a look at the bounds.
  long long base = nvec >= 64 ? -(long long)(((uintptr_t)d >> 4) & 7) : 0;
  if (base < 0 && nvec - base >= U * 32) {
    copy_round<U, false>(o, s, base, nvec, sh, lane, ends);
    base += U * 32;
  }
  for (; base + U * 32 <= nvec; base += U * 32) copy_round<U, true>(o, s, base, nvec, sh, lane, ends);
  if (nvec - base > 4 * 32) copy_round<U, false>(o, s, base, nvec, sh, lane, ends);
  else if (nvec - base > 32) copy_round<4, false>(o, s, base, nvec, sh, lane, ends);
  else if (nvec - base > 0) copy_round<1, false>(o, s, base, nvec, sh, lane, ends);
  else ends();
}

}  // namespace dev
}  // namespace rbv
