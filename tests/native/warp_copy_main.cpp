// The device byte copy (kernels/warp_copy.cuh) on the host: 32 fibers are the lanes of a warp, a shuffle is a switch to the
// next one, and every access is checked against the block.  Prints the number of copies and of bad ones.
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#define __device__
#define __forceinline__ inline
struct uint4 { unsigned x, y, z, w; };
static inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return uint4{x, y, z, w}; }
static inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned bits) {
  bits &= 31;
  return bits ? (lo >> bits) | (hi << (32 - bits)) : lo;
}

namespace {
constexpr size_t kStack = 64 << 10;
ucontext_t g_main, g_lane[32];
std::vector<char> g_stack(32 * kStack);
int g_current;
unsigned g_given[2][32], g_phase[32];
bool g_done[32];
long g_bad;
const char *g_src, *g_src_end;
char *g_dst, *g_dst_end;
void bad(const char* what) {
  if (!g_bad++) std::printf("%s out of the block\n", what);
}
}  // namespace

static unsigned __shfl_sync(unsigned, unsigned v, unsigned from) {
  const int me = g_current;
  const unsigned slot = g_phase[me]++ & 1;
  g_given[slot][me] = v;
  swapcontext(&g_lane[me], &g_main);   // comes back when every lane has given its value
  return g_given[slot][from];
}

namespace rbv {
namespace dev {
static uint4 ld_cg_v4(const uint4* p) {
  const char* c = reinterpret_cast<const char*>(p);
  // a vector that holds at least one byte of the block
  if (reinterpret_cast<uintptr_t>(p) & 15) bad("misaligned load");
  if (c + 16 <= g_src || c >= g_src_end) { bad("load"); return uint4{}; }
  uint4 v;
  std::memcpy(&v, c, 16);
  return v;
}
static unsigned char ld_cg_u8(const unsigned char* p) {
  const char* c = reinterpret_cast<const char*>(p);
  if (c < g_src || c >= g_src_end) { bad("byte load"); return 0; }
  return *p;
}
static void st_v4(uint4* p, const uint4& v) {
  char* c = reinterpret_cast<char*>(p);
  if (reinterpret_cast<uintptr_t>(p) & 15) bad("misaligned store");
  if (c < g_dst || c + 16 > g_dst_end) { bad("store"); return; }
  std::memcpy(c, &v, 16);
}
}  // namespace dev
}  // namespace rbv

#include "kernels/warp_copy.cuh"

template <int U>
static void lane_main(int lane) {
  rbv::dev::warp_copy<U>(g_dst, g_src, (size_t)(g_dst_end - g_dst), (unsigned)lane);
  g_done[lane] = true;
  swapcontext(&g_lane[lane], &g_main);
}

template <int U>
static void run_warp() {
  for (int l = 0; l < 32; l++) {
    g_done[l] = false;
    g_phase[l] = 0;
    getcontext(&g_lane[l]);
    g_lane[l].uc_stack.ss_sp = g_stack.data() + l * kStack;
    g_lane[l].uc_stack.ss_size = kStack;
    g_lane[l].uc_link = &g_main;
    makecontext(&g_lane[l], reinterpret_cast<void (*)()>(lane_main<U>), 1, l);
  }
  for (bool any = true; any;) {
    any = false;
    for (int l = 0; l < 32; l++)
      if (!g_done[l]) {
        g_current = l;
        swapcontext(&g_main, &g_lane[l]);
        any = true;
      }
    for (int l = 1; l < 32; l++)
      if (g_phase[l] != g_phase[0] || g_done[l] != g_done[0]) { std::printf("lanes part ways\n"); std::exit(1); }
  }
}

template <int U>
static void all_sizes(long* copies, long* wrong) {
  constexpr size_t kRoom = 4096 + 16 * 32 * 16 * 3;
  std::vector<char> from(kRoom + 128), to(kRoom + 128), want(kRoom + 128);
  for (size_t i = 0; i < from.size(); i++) from[i] = (char)(i * 131 + (i >> 8) * 7);
  char* const to0 = to.data() + ((128 - (reinterpret_cast<uintptr_t>(to.data()) & 127)) & 127);
  char* const from0 = from.data() + ((128 - (reinterpret_cast<uintptr_t>(from.data()) & 127)) & 127);
  // vector counts around every limit of the schedule: no vectors, the line rule (64), the small rounds (32, 128), one
  // and two full rounds
  std::vector<int> vectors;
  for (int mid : {0, 32, 64, 128, U * 32, 2 * U * 32})
    for (int d = -10; d <= 10; d++)
      if (mid + d >= 0) vectors.push_back(mid + d);
  for (int line = 0; line < 8; line++)
    for (int db : {0, 15})
      for (int sb : {0, 3})
        for (int nv : vectors) {
          const size_t n = (size_t)nv * 16 + (db ? 1 + 7 : 0);   // a byte up to the first vector, nv vectors, a rest
          std::memset(to.data(), 0x5a, to.size());
          std::memcpy(want.data(), to.data(), to.size());
          g_dst = to0 + 256 + line * 16 + db;
          g_dst_end = g_dst + n;
          g_src = from0 + 256 + sb;
          g_src_end = g_src + n;
          std::memcpy(want.data() + (g_dst - to.data()), g_src, n);
          const long before = g_bad;
          run_warp<U>();
          ++*copies;
          if (g_bad != before || std::memcmp(want.data(), to.data(), to.size())) ++*wrong;
        }
}

int main() {
  long copies = 0, wrong = 0;
  all_sizes<4>(&copies, &wrong);
  all_sizes<8>(&copies, &wrong);
  all_sizes<16>(&copies, &wrong);
  std::printf("%ld copies, %ld bad\n", copies, wrong);
  return wrong ? 1 : 0;
}
