// The copy warp of the fused dispatch on the host: 32 fibres in lockstep between warp collectives, with
// empty headers in place of the PTX wrappers' (test_copy_warp_order.py makes them).  Every fence takes a copy of what its
// lane can see (the slots' route weights, which padding and real rows write with plain stores); every
// announcement is checked against the copy of ITS OWN lane: a fence in another lane does not order this
// lane's reduction behind the stores.
// Prints the announcements that were not covered, all that were made, the blocks that became complete, and
// all blocks.
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#define __device__
#define __forceinline__ inline
struct uint4 { unsigned x, y, z, w; };
static uint4 make_uint4(unsigned a, unsigned b, unsigned c, unsigned d) { return {a, b, c, d}; }
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static int __ffs(unsigned v) { return v ? __builtin_ctz(v) + 1 : 0; }
static int __popc(unsigned v) { return __builtin_popcount(v); }

// ---- 32 lanes as fibres -----------------------------------------------------------------------
static ucontext_t lanes[32], back;
static int cur;
static bool done[32];
static unsigned long long slot[32], all[32];
struct ThreadIdx { struct { operator int() const { return cur; } } x; } threadIdx;
// every lane leaves a value and goes on once all lanes have left theirs
static void exchange(unsigned long long v) { slot[cur] = v; swapcontext(&lanes[cur], &back); }
static void __syncwarp() { exchange(0); }
template <class T> static T __shfl_sync(unsigned, T v, int from) {
  unsigned long long u = 0;
  memcpy(&u, &v, sizeof(T));
  exchange(u);
  T r;
  memcpy(&r, &all[from & 31], sizeof(T));
  return r;
}
static unsigned __ballot_sync(unsigned, int p) {
  exchange(p != 0);
  unsigned m = 0;
  for (int i = 0; i < 32; ++i) m |= (unsigned)(all[i] != 0) << i;
  return m;
}
static int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
static unsigned __match_any_sync(unsigned, unsigned long long v) {
  exchange(v);
  unsigned m = 0;
  for (int i = 0; i < 32; ++i) m |= (unsigned)(all[i] == v) << i;
  return m;
}

// ---- what the lanes see -------------------------------------------------------------------------
static std::vector<int32_t> meta;
static int n_slots, w_off, arrive_off, uncovered, announced;
static std::vector<int32_t> seen[32];
constexpr int32_t UNSET = 0x7f7f7f7f;
namespace mep {
static void fence_sys() { seen[cur].assign(meta.begin() + w_off, meta.begin() + w_off + n_slots); }
static void announce(int32_t* ctr, int v) {
  *ctr += v;
  const int block = (int)(ctr - meta.data()) - arrive_off;
  int ready = 0;
  for (int r = block * 128; r < (block + 1) * 128 && r < (int)seen[cur].size(); ++r) ready += seen[cur][r] != UNSET;
  ++announced;
  if (*ctr > ready) ++uncovered;          // (one part a row)
}
static void red_relaxed_sys_add(int32_t* p, int v) { announce(p, v); }
static void red_release_sys_add(int32_t* p, int v) { fence_sys(); announce(p, v); }
static void fence_proxy_async() {}
static void mbar_expect_tx(uint64_t*, uint32_t) {}
static void bulk_g2s(void* d, const void* s, uint32_t n, uint64_t*) { memcpy(d, s, n); }
static void bulk_s2g(void* d, const void* s, uint32_t n) { memcpy(d, s, n); }
static void bulk_commit() {}
template <int N> static void bulk_wait() {}
}  // namespace mep

#include "device/fused_dispatch.cuh"

static mep::FusedDispatch disp;
static std::vector<uint8_t> ring(8 * mep::FD_PART_CAP);
static uint64_t bars[8];
static int cta_of_run, n_cta;
static void lane_main() {
  mep::fused_dispatch_copy_warp<5>(disp, ring.data(), bars, cta_of_run, n_cta, [](uint64_t*, uint32_t) { return true; });
  done[cur] = true;
  swapcontext(&lanes[cur], &back);
}

int main(int argc, char** argv) {
  // one rank, every group padded to 128 rows: tokens, experts, top-k and CTAs from the command line
  const int S = atoi(argv[1]), E = atoi(argv[2]), K = atoi(argv[3]);
  n_cta = atoi(argv[4]);
  const int N = S * K, row_bytes = 32;
  std::vector<int> count(E), start(E + 1), fill(E), dst(N), order, pads(4 * E);
  std::vector<float> w(N);
  for (int i = 0; i < N; ++i) { count[(i * 7 + i / K) % E]++; w[i] = 1.f + i; }
  for (int e = 0; e < E; ++e) {
    start[e + 1] = start[e] + (count[e] + 127) / 128 * 128;
    pads[2 * e] = start[e] + count[e];
    pads[2 * e + 1] = start[e + 1] - pads[2 * e];
  }
  for (int e = 0; e < E; ++e)
    for (int i = 0; i < N; ++i)
      if ((i * 7 + i / K) % E == e) { dst[i] = start[e] + fill[e]++; order.push_back(i); }
  n_slots = start[E];
  w_off = 0; arrive_off = n_slots;
  const int link = arrive_off + n_slots / 128 + 1, src = link + n_slots;
  meta.assign(src + n_slots, 0);
  for (int i = 0; i < n_slots; ++i) meta[i] = UNSET;
  std::vector<uint8_t> x((size_t)S * row_bytes, 1), rows((size_t)n_slots * row_bytes, 9);
  disp = {};
  disp.x = x.data(); disp.w = w.data(); disp.dst = dst.data(); disp.order = order.data(); disp.zero_fill = pads.data();
  disp.hidden = rows.data(); disp.meta = meta.data();
  disp.weights_off = w_off; disp.link_off = link; disp.src_off = src; disp.arrive_off = arrive_off; disp.NvS = n_slots;
  disp.N = N; disp.K = K; disp.epn = E; disp.R = 1; disp.fresh = 1; disp.row_bytes = row_bytes; disp.nsplit = 1;
  static char stack[32][1 << 16];
  for (cta_of_run = 0; cta_of_run < n_cta; ++cta_of_run) {
    for (int i = 0; i < 32; ++i) {
      done[i] = false;
      seen[i].clear();
      getcontext(&lanes[i]);
      lanes[i].uc_stack.ss_sp = stack[i];
      lanes[i].uc_stack.ss_size = sizeof(stack[i]);
      lanes[i].uc_link = nullptr;
      makecontext(&lanes[i], lane_main, 0);
    }
    while (!done[0]) {
      for (cur = 0; cur < 32; ++cur) swapcontext(&back, &lanes[cur]);
      memcpy(all, slot, sizeof(all));
    }
  }
  int complete = 0;
  for (int b = 0; b < n_slots / 128; ++b) complete += meta[arrive_off + b] == 128;
  printf("%d %d %d %d\n", uncovered, announced, complete, n_slots / 128);
  return 0;
}
