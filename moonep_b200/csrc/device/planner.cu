// Online redundant-expert planner for sm_100a.
//
// What it computes is defined by the CPU oracle (ref/plan_ref.cc), which mirrors the
// reference's oracle (tests/planning_reference.py) and device planner
// (moonep/planning.py:495-1098).  How it computes it differs from the reference:
//  * the reference solves the plan on rank 0 only, parks rank 0's sort on rank 1 and
//    broadcasts three E*R tables through NVLS (planning.py:578-582, 917-934).  Here the
//    gathered tpe[R][E] table (a few KB) is all-gathered with peer stores and EVERY rank
//    solves redundantly in ONE CTA.  The solve is integer-only, hence bit-identical on all
//    ranks, so there is no broadcast, no rank-0 serialisation and ONE cross-rank barrier
//    instead of three.
//  * while CTA 0 exchanges and solves, the other CTAs histogram their slice of top-k.
//  * duplicates of a token on one destination rank are published as per-slot chain links by
//    the SOURCE (common/layout.h) instead of per-slot source records that the destination
//    turns into groups with atomics (dispatch.py:499-681).
#include <cuda_runtime.h>

#include "common/layout.h"
#include "device/planner_core.cuh"
#include "device/sync.cuh"
#include "host/ctx.h"
#include "host/errors.h"

namespace mep {

__global__ void __launch_bounds__(PLAN_THREADS, 1) ep_plan_kernel(const PlanParams p) {
  extern __shared__ int32_t smem[];
  const SyncCtx& sc = p.sync;
  const int R = sc.R, E = p.E, K = p.K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int vr = blockIdx.y, rank = sc.rank_base + vr;
  const int G = gridDim.x, c = blockIdx.x;
  int32_t* st = sync_state_of(sc);
  const int parity = st[3] & 1;
  const int32_t* topk = p.topk + (size_t)vr * p.N;
  int32_t* dst = p.dst + (size_t)vr * p.N;
  int32_t* scratch = p.scratch + (size_t)vr * p.scratch_ints;
  int32_t* hist_g = scratch + (size_t)4 * R * E;
  const int64_t tbl_off = p.tpe_off + (int64_t)parity * R * E;
  pdl_launch_dependents();   // the dispatch kernel that follows may set itself up meanwhile

  // slice of entries owned by this CTA (whole tokens)
  const int tpc = (p.S + G - 1) / G;
  const int tok0 = min(p.S, c * tpc), tok1 = min(p.S, tok0 + tpc);
  const int64_t i0 = (int64_t)tok0 * K, i1 = (int64_t)tok1 * K;

  if (c == 0 && !p.one_device) {
    // all-gather of tpe by peer stores: my row into everyone's table
    const int32_t* my_tpe = p.tpe + (size_t)vr * E;
    for (int64_t i = tid; i < (int64_t)R * E; i += PLAN_THREADS) {
      int peer = (int)(i / E), e = (int)(i % E);
      sc.meta[(size_t)peer * sc.meta_stride + tbl_off + (size_t)rank * E + e] = my_tpe[e];
    }
  }
  // histogram of my slice (smem cnt[E] sits after the solver's area so both can coexist)
  int32_t* cnt = smem;
  for (int e = tid; e < E; e += PLAN_THREADS) cnt[e] = 0;
  __syncthreads();
  for (int64_t i = i0 + tid; i < i1; i += PLAN_THREADS) {
    int e = topk[i];
    if ((unsigned)e < (unsigned)E) atomicAdd(&cnt[e], 1);
    else report_failure(sc, ST_BAD_INDEX, 10, -1, e, E);
  }
  __syncthreads();
  for (int e = tid; e < E; e += PLAN_THREADS) hist_g[(size_t)c * E + e] = cnt[e];
  if (c == 0) {
    // arrival counters of the fused dispatch -> GEMM path start at zero; clearing them before
    // the exchange orders the clear before every peer's first increment of this step
    int32_t* arrive = sc.meta + (size_t)rank * sc.meta_stride + p.arrive_off;
    for (int i = tid; i < p.n_arrive; i += PLAN_THREADS) arrive[i] = 0;
    if (!p.one_device) cta_cross_rank_exchange(sc, 1);
    plan_solve(p, rank, p.one_device ? p.tpe : sc.meta + (size_t)rank * sc.meta_stride + tbl_off, smem,
               p.tables != 0 ? smem + p.tables : nullptr);
  }
  grid_sync(sc, 2);
  if (c == 0 && tid == 0) st[3] = parity ^ 1;

  const int32_t* tpe_cumsum = scratch;
  const int32_t* alloc_cumsum = scratch + (size_t)2 * R * E;
  const int32_t* expert_off = scratch + (size_t)3 * R * E;

  // running count of each expert before my slice: earlier ranks + earlier CTAs of my rank.  With few
  // experts several threads share one's CTAs, and each has sixteen loads in flight.
  for (int e = tid; e < E; e += PLAN_THREADS) cnt[e] = rank > 0 ? tpe_cumsum[(size_t)(rank - 1) * E + e] : 0;
  __syncthreads();
  const int shares = PLAN_THREADS / E > 1 ? PLAN_THREADS / E : 1;
  for (int i = tid; i < E * shares; i += PLAN_THREADS) {
    const int e = i % E;
    int sum = 0;
    for (int c0 = i / E; c0 < c; c0 += 16 * shares) {
      int n[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int cc = c0 + u * shares;
        n[u] = cc < c ? hist_g[(size_t)cc * E + e] : 0;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) sum += n[u];
    }
    if (sum != 0) atomicAdd(&cnt[e], sum);
  }
  // the tables that every entry looks up, in shared memory where the solver's had room there
  if (p.tables != 0) {
    int32_t* at = smem + p.tables + (p.rank_warps > 1 ? p.rank_warps * E : 0);
    for (int i = tid; i < R * E; i += PLAN_THREADS) {
      at[i] = alloc_cumsum[i];
      at[R * E + i] = expert_off[i];
    }
    alloc_cumsum = at;
    expert_off = at + R * E;
  }
  // sending order: exclusive prefix of my per-expert counts in the permuted expert order
  int32_t* pperm = smem + E;
  if (p.send_order != nullptr) {
    const int32_t* my_tpe = p.tpe + (size_t)vr * E;
    for (int e = tid; e < E; e += PLAN_THREADS) pperm[send_perm(e, p.epn, R, rank)] = my_tpe[e];
  }
  __syncthreads();
  if (warp == 0 && p.send_order != nullptr) {
    int run = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int n = e < E ? pperm[e] : 0;
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (e < E) pperm[e] = run + incl - n;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  // Stable rank of every entry among the entries of its expert.  The slice is cut into one part per
  // warp (as many as have room for a counter an expert): each warp counts its part, an exclusive prefix
  // over the warps gives it its starting ranks, and it numbers its entries in order.  (One warp took the
  // whole slice one 32 entries after the other; 1820 entries a CTA, 8 ranks: 55 -> 43 us with the above.)
  const int nw = p.rank_warps;
  int32_t* wcnt = smem + p.rank_counts;                  // [nw][E]
  const int64_t part = (((i1 - i0) + nw - 1) / nw + 31) / 32 * 32;
  const int64_t b0 = min(i1, i0 + warp * part), b1 = min(i1, b0 + part);
  if (nw > 1) {                                          // (a lone warp works on cnt itself)
    for (int i = tid; i < nw * E; i += PLAN_THREADS) wcnt[i] = 0;
  }
  __syncthreads();
  if (nw > 1 && warp < nw) {
    for (int64_t i = b0 + lane; i < b1; i += 32) {
      int e = topk[i];
      if ((unsigned)e >= (unsigned)E) e = 0;
      atomicAdd(&wcnt[warp * E + e], 1);
    }
  }
  __syncthreads();
  for (int e = tid; nw > 1 && e < E; e += PLAN_THREADS) {
    int run = cnt[e];
    for (int w = 0; w < nw; ++w) {
      const int n = wcnt[w * E + e];
      wcnt[w * E + e] = run;
      run += n;
    }
  }
  __syncthreads();
  if (warp < nw) {
    int32_t* mine = wcnt + warp * E;
    for (int64_t b = b0; b < b1; b += 32) {
      int64_t i = b + lane;
      bool valid = i < b1;
      int e = valid ? topk[i] : -1 - lane;
      if (valid && (unsigned)e >= (unsigned)E) e = 0;
      unsigned m = __match_any_sync(0xffffffffu, e);
      int before = __popc(m & ((1u << lane) - 1));
      int base = valid ? mine[e] : 0;
      __syncwarp();
      if (valid && before == 0) mine[e] = base + __popc(m);
      __syncwarp();
      if (valid) dst[i] = base + before;  // global rank of the entry, resolved below
    }
  }
  __syncthreads();
  // destination rank and row of every entry
  for (int64_t i = i0 + tid; i < i1; i += PLAN_THREADS) {
    int e = topk[i];
    if ((unsigned)e >= (unsigned)E) e = 0;
    int g = dst[i];
    const int32_t* ac = alloc_cumsum + (size_t)e * R;
    int lo = 0, hi = R;  // first d with ac[d] > g
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (ac[mid] > g) hi = mid; else lo = mid + 1;
    }
    int dest = lo;
    if (dest >= R) { report_failure(sc, ST_BAD_INDEX, 20, e, g, ac[R - 1]); dest = R - 1; }
    int prev = dest > 0 ? ac[dest - 1] : 0;
    int64_t row = (int64_t)expert_off[(size_t)dest * E + e] + (g - prev);
    if (row < 0 || row >= p.NvS) { report_failure(sc, ST_BAD_INDEX, 21, dest, (int)row, (int)p.NvS); row = 0; }
    dst[i] = (int)((int64_t)dest * p.NvS + row);
    if (p.send_order != nullptr) {
      const int mine_before = rank > 0 ? tpe_cumsum[(size_t)(rank - 1) * E + e] : 0;
      const int64_t pos = (int64_t)pperm[send_perm(e, p.epn, R, rank)] + (g - mine_before);
      if (pos >= 0 && pos < p.N) p.send_order[(size_t)vr * p.N + pos] = (int32_t)i;
      else report_failure(sc, ST_BAD_INDEX, 22, e, (int)pos, (int)p.N);
    }
  }
  __syncthreads();
  // duplicate canonicalisation + chain links: K lanes per token (32 / K tokens per warp), the
  // lanes of a token that share a destination rank find one another with match.any, so nothing
  // is kept in per-thread arrays
  const int tpw = 32 / K;
  const int tl = lane / K, k = lane - tl * K;
  for (int t0 = tok0 + warp * tpw; t0 < tok1; t0 += PLAN_WARPS * tpw) {
    const int t = t0 + tl;
    const bool valid = tl < tpw && t < tok1;
    int32_t* d = dst + (size_t)t * K;
    const int raw = valid ? d[k] : 0;
    const int dr = valid ? (int)(raw / p.NvS) : 0;
    const unsigned m = __match_any_sync(0xffffffffu, valid ? ((tl << 8) | dr) : (0x40000000 | lane));
    const bool dup = (m & ((1u << lane) - 1u)) != 0u;
    const unsigned above = lane < 31 ? (m & ~((2u << lane) - 1u)) : 0u;
    const int nl = above ? __ffs(above) - 1 : lane;
    const int raw_next = __shfl_sync(0xffffffffu, raw, nl);
    if (valid) {
      const int next = above ? (int)(raw_next - (int64_t)dr * p.NvS) : LINK_NONE;
      const int64_t row = raw - (int64_t)dr * p.NvS;
      int32_t* peer = sc.meta + (size_t)dr * sc.meta_stride;
      int32_t* link = p.link_out != nullptr ? p.link_out + (size_t)dr * p.NvS : peer + p.link_off;
      int32_t* src = p.src_out != nullptr ? p.src_out + (size_t)dr * p.NvS : peer + p.src_off;
      link[row] = next | (dup ? LINK_DUP_BIT : 0);
      src[row] = (int32_t)((int64_t)rank * p.N + (int64_t)t * K + k);
      if (dup) d[k] = -raw - 1;
    }
  }
}

}  // namespace mep

using namespace mep;

extern "C" {

// Dynamic shared memory the planner needs for (R, E).
int64_t mep_plan_smem_bytes(int R, int E) {
  return (int64_t)sizeof(int32_t) * (2 * (int64_t)E + 4 * R + (int64_t)PLAN_WARPS * R);
}

// CTAs a rank.  Within one device no more than have 256 entries each: the grid's barrier and the sums over the
// CTAs before one's own cost more than the entries of the smallest calls.  All CTAs of a virtual group's ranks
// are resident at once, and an SM holds one (512 threads of more than 64 registers): a group whose
// num_sms * R is above the number of SMs, which the copy kernels fit twice, takes fewer here.
static int plan_ctas(const BufferCtx& c, bool one_device) {
  const int64_t useful = one_device ? (c.N + 255) / 256 : c.num_sms;
  const int sms = c.sm_count > 0 ? c.sm_count : 148, fit = sms > c.Rv() ? sms / c.Rv() : 1;
  const int most = c.num_sms < fit ? c.num_sms : fit;
  return useful < most ? (int)useful : most;
}

// Ranking warps of a planner launch: one per 64 entries of a CTA within one device (4096 tokens on 256 experts
// 21.6 us, 22.4 with one per 128), per 128 over several (clearing and summing their counters costs more than a few steps of 32
// entries: with sixteen for 8 entries 27 -> 31 us), as many as have room for counters.  Over several devices
// that is 8 KB: the planner and the weight ops wait for other ranks while they hold their SMs, on two
// streams, and beside prefetch_weight's ring (192 KB and its lists) 64 KB do not fit.
static int plan_rank_warps(const BufferCtx& c, bool one_device) {
  const int ctas = plan_ctas(c, one_device);
  const int64_t entries = (int64_t)((c.S + ctas - 1) / ctas) * c.K;
  int64_t w = (one_device ? 64 * 1024 : 8 * 1024) / (int64_t)(sizeof(int32_t) * c.E);
  const int64_t least = one_device ? 64 : 128;
  if (w > entries / least) w = entries / least;
  return w < 1 ? 1 : (w > PLAN_WARPS ? PLAN_WARPS : (int)w);
}

// Where the solver's tables start in shared memory: behind its other arrays, over the ranking warps' counters, which
// are used later.  0 (none) over several devices, where the planner shares SMs (see above), and when they are
// too large.  Tables in shared memory, no exchange within one device, the layout split over all warps: 16 tokens on
// 32 experts 17 -> 15 us, 4096 on 256 28 -> 22, 8 ranks x 17 tokens on 128 experts 29 -> 19, 8 x 4096 on 256 42 -> 35.
static int64_t plan_tables(const BufferCtx& c, bool one_device) {
  const int64_t at = mep_plan_smem_bytes(c.R, c.E);
  return one_device && at + (int64_t)sizeof(int32_t) * solve_table_ints(c.R, c.E) <= 160 * 1024 ? at : 0;
}

static int64_t plan_smem(const BufferCtx& c, bool one_device) {
  const int w = plan_rank_warps(c, one_device);            // (a lone warp counts in place)
  int64_t more = w > 1 ? (int64_t)w * c.E : 0;
  if (plan_tables(c, one_device) != 0) {
    more += 2 * (int64_t)c.R * c.E;            // the tables that are looked up, behind the counters
    if (more < solve_table_ints(c.R, c.E)) more = solve_table_ints(c.R, c.E);
  }
  return mep_plan_smem_bytes(c.R, c.E) + (int64_t)sizeof(int32_t) * more;
}

// CTAs a rank, and dynamic shared memory, of a planner launch of this Buffer.
int mep_plan_launch_ctas(const void* ctx_) {
  const BufferCtx& c = *(const BufferCtx*)ctx_;
  return plan_ctas(c, c.one_device());
}
int64_t mep_plan_launch_smem_bytes(const void* ctx_) {
  const BufferCtx& c = *(const BufferCtx*)ctx_;
  return plan_smem(c, c.one_device());
}

// Fresh plan for this rank (or for all virtual ranks).  send_order [Rv][N] may be null (it is
// only needed by the fused dispatch -> GEMM path).  Leaves the chain links in the peers'
// meta chunks; they become visible with the next cross-rank barrier (the dispatch kernel's
// exit barrier, or an explicit mep_launch_sync).  Within one device link_out and src_out [Rv][NvS] may take the
// records of all real rows instead (the dispatch that follows sets those of padding rows): that saves
// dispatch its exit barrier and the copies behind it, 6 - 9 us.  one_device != 0 only where every rank's counts are
// memory of this device; without it the ranks exchange their counts, a virtual group's too.
int mep_launch_plan(const void* ctx_, const int32_t* topk, const int32_t* tpe, int32_t* dst,
                    int32_t* cu_seqlens, int32_t* zero_fill, int32_t* etc, int32_t* remote_stats,
                    int32_t* send_order, int32_t* link_out, int32_t* src_out, int one_device, cudaStream_t stream) {
  const BufferCtx& c = *(const BufferCtx*)ctx_;
  const bool one = one_device != 0;
  if (one && !c.one_device()) return fail(-2, "plan: the ranks are on several devices");
  if ((link_out != nullptr || src_out != nullptr) && !one)
    return fail(-1, "plan: records go straight into the plan only within one device");
  PlanParams p;
  p.sync = c.sync(KID_PLAN);
  p.E = c.E; p.epn = c.epn; p.S = c.S; p.K = c.K; p.token_padding = c.token_padding;
  p.N = c.N; p.NvS = c.NvS;
  p.tpe_off = c.ml.tpe_off; p.link_off = c.ml.link_off; p.src_off = c.ml.src_off;
  p.topk = topk; p.tpe = tpe; p.dst = dst; p.cu_seqlens = cu_seqlens; p.zero_fill = zero_fill;
  p.etc = etc; p.remote_stats = remote_stats;
  p.scratch = c.plan_scratch; p.scratch_ints = c.plan_scratch_ints;
  p.send_order = send_order; p.arrive_off = c.ml.arrive_off; p.n_arrive = (int)(c.NvS / 128 + 1);
  const size_t smem = (size_t)plan_smem(c, one);
  p.rank_warps = plan_rank_warps(c, one);
  p.one_device = one;
  p.link_out = link_out; p.src_out = src_out;
  p.tables = (int)(plan_tables(c, one) / sizeof(int32_t));
  p.rank_counts = p.rank_warps > 1 ? (int)(mep_plan_smem_bytes(c.R, c.E) / sizeof(int32_t)) : 0;
  static std::atomic<unsigned long long> raised{0};
  MEP_CUDA_OK(raise_smem_limit((const void*)ep_plan_kernel, raised));
  dim3 grid(plan_ctas(c, one), c.Rv());
  MEP_CUDA_OK(launch_coop((const void*)ep_plan_kernel, grid, dim3(PLAN_THREADS), smem, stream, p));
  return 0;
}

}  // extern "C"
