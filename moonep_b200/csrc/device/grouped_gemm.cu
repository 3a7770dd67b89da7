// Grouped bf16 GEMM for sm_100a on the 5th-generation tensor cores: tcgen05.mma issued by one
// thread per CTA, operands staged in shared memory by tiled TMA loads (no cluster multicast),
// fp32 accumulators in tensor memory, read back with tcgen05.ld for fused epilogues.
//
// The reference ships no GEMM: it hands cu_seqlens and the [2*epn, H, H'] compute view to the
// host framework's "VM group GEMM" (README.md:45-68).  These kernels are that GEMM.  One
// persistent CTA (or CTA pair) per SM walks a static tile list derived on the device from
// cu_seqlens (no host synchronisation), with three warp roles: warp 0 TMA producer, warp 1 MMA
// issuer (two 256-column TMEM accumulators), warps 2.. epilogue, overlapped with the next tile's
// main loop through the second accumulator.  Kernels:
//   ep_token_gemm_kernel (token_gemm.cuh): token-major products with bf16 output -- gate/up with
//        SwiGLU, down, both dgrads, the pushed combine, the fused dispatch.
//        Also large products with fp32 output.
//   ep_dense_f32_kernel (dense_f32.cuh): one product with fp32 output (router logits).
//   ep_grouped_gemm_kernel (this file): weight-grad (groups partition the REDUCTION dimension):
//        D[g] (+)= A[rows of g]^T * B[rows of g]   both operands MN-major, fp32 output by TMA
//        store / reduce-add; or (template SGD) the optimizer step fused in: the accumulator is
//        applied straight to the bf16 weights, w = bf16(w - lr * acc), through a per-warp TMA
//        ring of weight blocks, for every local expert that has no replica this step.  Those
//        kernels run eight epilogue warps (two per quarter of the accumulator's lanes, one half
//        of the columns each) and take their split of the shared memory at launch.
// Group g < split reads/writes allocation 0 (local experts), g >= split allocation 1 (this
// rank's prefetch / reduce slots): the [2*epn] compute view never has to be contiguous.
// CTA pairs (template TWO, clusters of two CTAs, tcgen05 cta_group::2): the leader issues
// 256-row MMAs over both CTAs' shared memory; each CTA stages its own 128 rows of A and half
// of the B tile (32 KB per k-block instead of 48 KB, six stages), which lifts the single-CTA
// kernel's limit of 12 KB of operand reads per MMA.  Both CTAs' loads count on the LEADER's full
// barrier, on which only the leader's producer arrives (expecting the bytes of both): a per-stage
// arrival from the peer over the cluster network measured 2x slower overall.  Weight-grad pairs
// cover 256 rows of the weight matrix (+24% over single CTAs, 32 groups x 1024 rows, H=7168, H'=2048).
// Every mbarrier wait is bounded; on expiry the CTA records an error, drains and frees TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "device/fused_dispatch.cuh"
#include "device/tcgen05.cuh"
#include "host/ctx.h"
#include "host/errors.h"

namespace mep {
void* driver_tensor_map_encode();

constexpr int BM = 128, BN = 256, BK = 64, GEMM_STAGES = 4;
constexpr int A_TILE_BYTES = BM * BK * 2;   // 16 KB
constexpr int B_TILE_BYTES = BN * BK * 2;   // 32 KB
constexpr int STAGE_BYTES = A_TILE_BYTES + B_TILE_BYTES;
constexpr int GEMM_THREADS = 192;
// SGD kernels: eight epilogue warps, two per quarter of the accumulator's lanes, each with one
// half of the tile's columns (the read-modify-write stream of a warp is a chain of latencies:
// accumulator load, weight block landed, update, store read; twice the warps run twice the chains)
constexpr int GEMM_THREADS_SGD = 320;
constexpr int MAX_GROUPS = 1024;
// CTA-pair variant: each CTA stages A (16 KB) and half of B (16 KB) per k-block, six stages.
constexpr int GEMM_STAGES2 = 6;
constexpr int STAGE_BYTES2 = A_TILE_BYTES + B_TILE_BYTES / 2;

enum { EPI_BF16 = 0, EPI_SWIGLU = 1, EPI_F32 = 2, EPI_PUSH = 3 };

constexpr int TG_BOXES = 4;

struct GemmKParams {
  CUtensorMap a;           // weight grad: token rows of A in 64 x 64 boxes
  CUtensorMap tok[2][TG_BOXES];   // token rows in boxes of 32, 64, 96 and 128 rows (token_gemm.cuh)
  CUtensorMap b[2][2];
  CUtensorMap c[2];        // weight-grad output (fp32), per allocation
  CUtensorMap b2[2][2];    // K-major B with a 128-row box
  const int32_t* cu_seqlens;
  const int32_t* pads;     // [ngroups][2] first padding row and their number, per group; or null
  int ngroups, split, total_rows, N, K, nseg, rows_per_expert, Mw, accumulate, zero_empty_below;
  int stages, wb;   // SGD kernels: operand stages and weight blocks per epilogue warp of this launch
  // SGD kernels: 1 = only the tiles whose grads are STORED (experts with replicas, slot groups),
  // 2 = only the tiles that are applied to the weights, 0 = all.  Lets the grads that have to
  // travel be computed first, so that their reduce runs beside the rest of the weight grad.
  int wg_select;
  int g_begin; // groups below this index are skipped (a launch may cover a suffix of the groups)
  int vec_out; // outputs allow 16-byte stores
  // weight grad fused with the SGD step: a local expert's tile is applied straight to its bf16
  // weights, w = bf16(w - lr * acc), instead of being stored as an fp32 grad.  Experts whose
  // sgd_keep flag is set (they have replicas elsewhere, whose grads must be added first) and the
  // slot groups are still written as fp32 grads.
  __nv_bfloat16* sgd_w;
  CUtensorMap wmap;        // the same weights as a [G0 * Mw][N] bf16 tensor, 32-row x 64-column boxes, 128B swizzle
  const int32_t* sgd_keep;
  float sgd_lr;
  void* out[3];
  const float* row_scale;
  long long ldc;
  int32_t* status;
  unsigned long long timeout_ns;
  // EPI_PUSH: results go straight to the token's home rank (see the epilogue)
  const int32_t* src_info;
  void* push_base;
  long long push_rank_stride;
  int push_entries, push_ranks;
  FusedDispatch disp;      // DISP kernels only
  long long* trace;        // phase stamps of the fused launches (see sync.cuh), or null
  // DISP: budget of a wait for rows from other ranks.  It is shorter than timeout_ns, which bounds
  // the waits that only follow from it (the MMA thread on the operand ring, the epilogue on the
  // accumulator), so that a missing row is reported as what it is.
  unsigned long long arrive_timeout_ns;
};

struct Tile {
  int g, row0, rows, n0, num_kb, alloc, g_local, m0;
  bool valid;
};

// CLUSTER: the barrier also receives plain arrivals from the pair's other CTA, so the wait
// acquires at cluster scope.  Barriers completed by TMA byte counts or tcgen05.commit do not need it.
template <bool CLUSTER = false, class Params>
__device__ __forceinline__ bool gemm_wait(uint64_t* bar, uint32_t parity, volatile int* s_abort,
                                          const Params& p, int where) {
  auto ready = [&] { return CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
  if (ready()) return true;
  unsigned long long t0 = globaltimer_ns();
  unsigned spins = 0;
  while (!ready()) {
    if ((++spins & 255u) == 0) {
      if (*s_abort) return false;
      if (globaltimer_ns() - t0 > p.timeout_ns) {
        *s_abort = 1;
        if (p.status != nullptr && atomicCAS(p.status, 0, ST_TIMEOUT_MBAR) == 0) {
          p.status[1] = KID_GEMM;
          p.status[2] = where;
          p.status[3] = (int)blockIdx.x;
        }
        return false;
      }
    }
  }
  return true;
}

// Fused dispatch: wait until all rows of the 128-row block have arrived (counter >= expect).
__device__ __forceinline__ bool arrive_wait(const int32_t* ctr, int expect, int block, volatile int* s_abort,
                                            const GemmKParams& p) {
  int seen = ld_acquire_sys(ctr);
  if (seen >= expect) return true;
  unsigned long long t0 = globaltimer_ns();
  unsigned spins = 0;
  while ((seen = ld_acquire_sys(ctr)) < expect) {
    // many CTAs watch the same few counters while the senders' reductions land on them: back off
    __nanosleep(500);
    if ((++spins & 63u) == 0) {
      if (*s_abort) return false;
      if (globaltimer_ns() - t0 > p.arrive_timeout_ns) {
        *s_abort = 1;
        if (p.status != nullptr && atomicCAS(p.status, 0, ST_TIMEOUT_ARRIVAL) == 0) {
          p.status[1] = KID_GEMM;
          p.status[2] = 6;
          p.status[3] = (int)blockIdx.x;
          p.status[4] = block;
          p.status[5] = seen;
          p.status[6] = expect;
        }
        return false;
      }
    }
  }
  return true;
}

// Rows of a group that hold tokens (its real rows if the padding ranges are known); at least one
// for a group that is not empty.
__device__ __forceinline__ int group_valid(const GemmKParams& p, int g, int start, int end) {
  if (p.pads == nullptr || end <= start) return end - start;
  const int first = p.pads[2 * g], n = p.pads[2 * g + 1];
  return (n > 0 && first >= start && first < end) ? max(1, first - start) : end - start;
}

template <bool TWO>
__device__ __forceinline__ Tile get_tile(const GemmKParams& p, int id, const int* s_end, const int* s_valid,
                                         int n_tiles_n, int crank = 0) {
  Tile t;
  t.valid = true;
  constexpr int TMW = TWO ? 2 * BM : BM;       // a pair owns 256 rows of the weight matrix
  const int mt = p.Mw / TMW;
  const int tpg = mt * n_tiles_n;
  t.g = id / tpg;
  int local = id - t.g * tpg;
  int mi = local / n_tiles_n, ni = local - mi * n_tiles_n;
  t.row0 = t.g == 0 ? 0 : s_end[t.g - 1];
  t.rows = s_valid[t.g];                       // padding rows are zero: blocks of nothing else are skipped
  t.m0 = mi * TMW + crank * BM;
  t.n0 = ni * BN;
  t.num_kb = (t.rows + BK - 1) / BK;
  if (t.rows <= 0 && t.g >= p.zero_empty_below) t.valid = false;
  if (t.rows <= 0 && p.sgd_w != nullptr && t.g < p.split &&
      (p.sgd_keep == nullptr || p.sgd_keep[t.g] == 0)) t.valid = false;   // zero grad: nothing to apply
  if (t.g < p.g_begin) t.valid = false;
  t.alloc = t.g >= p.split ? 1 : 0;
  t.g_local = t.alloc ? t.g - p.split : t.g;
  if (p.wg_select != 0 && p.sgd_w != nullptr) {
    const bool applied = t.alloc == 0 && (p.sgd_keep == nullptr || p.sgd_keep[t.g_local] == 0);
    if ((p.wg_select == 2) != applied) t.valid = false;
  }
  return t;
}

// Operand stages of the kernels whose geometry is fixed at compile time.
template <bool TWO> __host__ __device__ constexpr int gemm_stages() { return TWO ? GEMM_STAGES2 : GEMM_STAGES; }
// The SGD kernels (weight grad with the optimizer step in the epilogue) take their geometry at
// launch instead (GemmKParams::stages / wb, sgd_geometry() below): how the shared memory is best
// split between operand stages and weight blocks depends on the group length.
constexpr int SGD_RING_MAX = 8;      // 4 KB weight blocks per epilogue warp, at most
template <bool TWO> __host__ __device__ constexpr int gemm_smem() {   // dynamic shared memory
  return gemm_stages<TWO>() * (TWO ? STAGE_BYTES2 : STAGE_BYTES) + 1024;
}

template <bool TWO, bool SGD>
__global__ void __launch_bounds__(SGD ? GEMM_THREADS_SGD : GEMM_THREADS, 1)
ep_grouped_gemm_kernel(const __grid_constant__ GemmKParams p) {
  // operand stages: a constant, except in the SGD kernels (upper bound; p.stages are used)
  constexpr int GEMM_STAGES = gemm_stages<TWO>();
  const int nst = SGD ? p.stages : GEMM_STAGES;
  constexpr int STAGE_BYTES = TWO ? STAGE_BYTES2 : mep::STAGE_BYTES;
  constexpr int WB_MAX = SGD ? SGD_RING_MAX : 1;
  const int WB = SGD ? p.wb : 1;
  const int crank = TWO ? (int)cluster_cta_rank() : 0;        // 0 = leader of the pair
  const int work_id0 = TWO ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int work_stride = TWO ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full[GEMM_STAGES];
  __shared__ __align__(8) uint64_t empty[GEMM_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_end[MAX_GROUPS];
  __shared__ int s_valid[MAX_GROUPS];
  __shared__ __align__(1024) float s_epi[4 * 32 * 32];      // per-warp staging of stored tiles: a swizzled 4 KB block
  // fused SGD: per epilogue warp a ring of WB 32 x 32 bf16 weight blocks (in dynamic shared
  // memory, behind the operand stages) and their "landed" barriers
  __shared__ __align__(8) uint64_t wbar[SGD ? 8 : 4][WB_MAX];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  volatile int* abortp = &s_abort;

  if (tid == 0) {
    // CTA pairs: both CTAs' loads are credited to the LEADER's full barrier, which only the
    // leader's producer arrives on (expecting the bytes of both CTAs); no per-stage remote arrive
    for (int s = 0; s < GEMM_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], (TWO ? 8 : 4) * (SGD ? 2 : 1)); }
    for (int a = 0; a < (SGD ? 8 : 4) * WB_MAX; ++a) mbar_init(&wbar[a / WB_MAX][a % WB_MAX], 1);
    mbar_fence_init();
    s_abort = 0;
  }
  // group table
  for (int g = tid; g < p.ngroups; g += (int)blockDim.x)
    s_end[g] = p.cu_seqlens != nullptr ? p.cu_seqlens[g] : p.total_rows;
  __syncthreads();
  for (int g = tid; g < p.ngroups; g += (int)blockDim.x)
    s_valid[g] = group_valid(p, g, g == 0 ? 0 : s_end[g - 1], s_end[g]);
  if (warp == 1) {
    if constexpr (TWO) { tmem_alloc2(&s_tmem, 512); tmem_relinquish2(); }
    else { tmem_alloc(&s_tmem, 512); tmem_relinquish(); }
  }
  tc_fence_before();
  if constexpr (TWO) cluster_sync_all();     // the peer's barriers exist before anyone arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;

  const int n_tiles_n = (p.N + BN - 1) / BN;
  const long long total_tiles = (long long)p.ngroups * (p.Mw / (TWO ? 2 * BM : BM)) * n_tiles_n;

  if (warp == 0) {
    // ================= TMA producer =================
    if (lane == 0) {
      tma_prefetch_desc(&p.a);
      tma_prefetch_desc(&p.b[0][0]);
      int it = 0;
      bool ok = true;
      for (long long id = work_id0; id < total_tiles && ok; id += work_stride) {
        Tile t = get_tile<TWO>(p, (int)id, s_end, s_valid, n_tiles_n, crank);
        if (!t.valid) continue;
        for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
          const int s = it % nst;
          if (it >= nst &&
              !gemm_wait(&empty[s], ((uint32_t)(it / nst) & 1u) ^ 1u, abortp, p, 1)) {
            ok = false;
            break;
          }
          uint8_t* sa = tiles + (size_t)s * STAGE_BYTES;
          uint8_t* sb = sa + A_TILE_BYTES;
          uint32_t lead_bar = 0;
          if constexpr (TWO) lead_bar = mapa_u32(&full[s], 0);
          // the peer's bytes may land before this arrival: the pending count keeps the phase open
          if (crank == 0) mbar_expect_tx(&full[s], TWO ? 2 * STAGE_BYTES : STAGE_BYTES);
          const int k0 = kb * BK;
          if constexpr (TWO) {
            // this CTA's 128 columns of A (t.m0 is already its half) and its half of the B tile
#pragma unroll
            for (int j = 0; j < 2; ++j)
              tma_load_2d_pair(sa + j * 8192, &p.a, t.m0 + 64 * j, t.row0 + k0, lead_bar);
#pragma unroll
            for (int j = 0; j < 2; ++j)
              tma_load_2d_pair(sb + j * 8192, &p.b[0][0], t.n0 + 128 * crank + 64 * j, t.row0 + k0, lead_bar);
          } else {
            // A: [token rows][Mw cols], two 64-column blocks; B: [token rows][N cols], four
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_2d(sa + j * 8192, &p.a, t.m0 + 64 * j, t.row0 + k0, &full[s]);
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(sb + j * 8192, &p.b[0][0], t.n0 + 64 * j, t.row0 + k0, &full[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer =================
    if (lane == 0 && TWO && crank != 0) {
      // peer CTA of a pair: the leader issues the MMAs for both
    } else if (lane == 0) {
      constexpr uint32_t idesc = make_instr_desc_bf16(TWO ? 2 * BM : BM, BN, true, true);
      int it = 0, tile_n = 0;
      bool ok = true;
      for (long long id = work_id0; id < total_tiles && ok; id += work_stride) {
        Tile t = get_tile<TWO>(p, (int)id, s_end, s_valid, n_tiles_n, crank);
        if (!t.valid) continue;
        const int acc = tile_n & 1;
        if (tile_n >= 2 &&
            !gemm_wait<TWO>(&acc_empty[acc], ((uint32_t)(tile_n >> 1) & 1u) ^ 1u, abortp, p, 2)) break;
        tc_fence_after();
        const uint32_t tacc = tmem_base + (uint32_t)acc * BN;
        for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
          const int s = it % nst;
          if (!gemm_wait(&full[s], (uint32_t)(it / nst) & 1u, abortp, p, 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + (size_t)s * STAGE_BYTES);
          const uint32_t sb = sa + A_TILE_BYTES;
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const uint64_t da = make_smem_desc(sa + kk * 2048, 8192, 1024);
            const uint64_t db = make_smem_desc(sb + kk * 2048, 8192, 1024);
            if constexpr (TWO) umma_bf16_2cta(tacc, da, db, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            else umma_bf16(tacc, da, db, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          // stage reusable (in both CTAs of a pair) once these MMAs have read it
          if constexpr (TWO) umma_commit_2cta(&empty[s], 3);
          else umma_commit(&empty[s]);
        }
        if (!ok) break;
        if constexpr (TWO) umma_commit_2cta(&acc_full[acc], 3);   // accumulator complete, both halves
        else umma_commit(&acc_full[acc]);
        ++tile_n;
      }
    }
  } else {
    // ================= epilogue (4 warps, one TMEM lane quarter each) =================
    const int q = warp & 3;
    // SGD: warps 2..5 take the tile's first 128 columns, warps 6..9 the other 128
    const int half = SGD ? (warp - 2) >> 2 : 0;
    const int ew = q + 4 * half;
    constexpr int CB = SGD ? BN / 64 / 2 : BN / 64;     // 64-column weight blocks per warp and tile
    const int cofs = half * CB * 64;
    int tile_n = 0;
    // ---- fused SGD: weight blocks stream through this warp's ring, ahead of the tiles ----------
    // Block k of the stream (the 32-row x 64-column blocks of this warp's rows, tile after tile,
    // fused tiles only) lives in buffer k % WB.  The load cursor runs up to WB blocks ahead of the
    // block being updated, across tile boundaries.  Blocks are as wide as the 128B swizzle
    // allows: the TMA engine moves about one box row per 5 cycles per SM whatever its length
    // (measured), so 64-byte rows cap this epilogue at half the HBM rate.
    constexpr int WBLK = 4096, WCOLS = 64;
    uint8_t* wring = tiles + (size_t)nst * STAGE_BYTES + ew * (WB * WBLK);
    int wseq = 0, lseq = 0;                // blocks consumed / loads issued (a few thousand per launch)
    long long lid = work_id0;              // cursor: tile id, block in tile, cached coordinates
    int lc = 0, l_y0 = 0, l_n0 = 0;
    bool l_have = false;
    auto sgd_tile = [&](const Tile& u) {
      return u.valid && u.alloc == 0 && (p.sgd_keep == nullptr || p.sgd_keep[u.g_local] == 0);
    };
    auto cursor_settle = [&]() {           // move to the next existing block at or after (lid, lc)
      while (lid < total_tiles) {
        if (!l_have) {
          const Tile u = get_tile<TWO>(p, (int)lid, s_end, s_valid, n_tiles_n, crank);
          if (sgd_tile(u)) { l_have = true; l_y0 = u.g_local * p.Mw + u.m0 + q * 32; l_n0 = u.n0; lc = 0; }
        }
        if (l_have && lc < CB && l_n0 + cofs + lc * WCOLS < p.N) return;
        l_have = false;
        lid += work_stride;
      }
    };
    auto issue_loads = [&]() {             // lane 0 issues; every lane tracks the cursor
      while (lid < total_tiles && lseq < wseq + WB) {
        if (lane == 0) {
          uint64_t* bar = &wbar[ew][lseq % WB];
          mbar_expect_tx(bar, WBLK);
          tma_load_2d(wring + (lseq % WB) * WBLK, &p.wmap, l_n0 + cofs + lc * WCOLS, l_y0, bar);
        }
        ++lseq;
        ++lc;
        cursor_settle();
      }
    };
    if constexpr (SGD) {
      cursor_settle();
      issue_loads();
    }
    for (long long id = work_id0; id < total_tiles; id += work_stride) {
      Tile t = get_tile<TWO>(p, (int)id, s_end, s_valid, n_tiles_n, crank);
      if (!t.valid) continue;
      const int acc = tile_n & 1;
      bool sgd_fuse = false;
      if constexpr (SGD) sgd_fuse = sgd_tile(t);
      if (!gemm_wait(&acc_full[acc], (uint32_t)(tile_n >> 1) & 1u, abortp, p, 4)) break;
      tc_fence_after();
      const uint32_t tacc = tmem_base + (uint32_t)acc * BN + ((uint32_t)(q * 32) << 16);
      const bool have_acc = t.num_kb > 0;
      {
          const int col_base = t.n0;
          // fp32 weight-grad tiles are 128 KB each and the main loop is short (one group's
          // tokens), so the epilogue must move ~30 GB/s per SM.  Four warps of plain stores
          // cannot (measured: ~14 B/clk/SM), so each warp stages 32x32 blocks in shared memory
          // (128-byte swizzle, conflict-free 16-byte stores) and hands them to the TMA engine:
          // a tiled store, or a tiled reduce-add when accumulating into existing grads.
          uint8_t* pad = reinterpret_cast<uint8_t*>(s_epi) + q * 4096;
          const int y0 = t.g_local * p.Mw + t.m0 + q * 32;
          const CUtensorMap* cmap = &p.c[t.alloc];
          if (SGD && sgd_fuse) {
            // Weights travel by TMA both ways: a block is 32 rows x 64 bf16 (128-byte rows, 128B
            // swizzle); lane i owns row i of the block, exactly the accumulator row it reads from
            // tensor memory, so no transposition is needed.  The block is updated in place,
            // stored back, and its buffer handed to the load cursor.
            const float nlr = -p.sgd_lr;
            bool wok = true;
#pragma unroll 1
            for (int c = 0; c < CB; ++c) {
              if (col_base + cofs + c * WCOLS >= p.N) break;
              const int b = wseq % WB;
              uint8_t* wbuf = wring + b * WBLK;
              uint32_t ra[32], rb[32];
              tmem_ld_32x32(tacc + cofs + c * WCOLS, ra);
              tmem_ld_32x32(tacc + cofs + c * WCOLS + 32, rb);
              if (!gemm_wait(&wbar[ew][b], (uint32_t)(wseq / WB) & 1u, abortp, p, 5)) {
                tmem_ld_wait();
                wok = false;
                break;
              }
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint32_t* g = j < 4 ? ra + 8 * j : rb + 8 * (j - 4);
                uint4* slot = reinterpret_cast<uint4*>(wbuf + lane * 128 + ((j ^ (lane & 7)) << 4));
                uint4 w4 = *slot;
                __nv_bfloat162* w2 = reinterpret_cast<__nv_bfloat162*>(&w4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const float2 x = __bfloat1622float2(w2[i]);
                  w2[i] = __floats2bfloat162_rn(__fmaf_rn(nlr, __uint_as_float(g[2 * i]), x.x),
                                                __fmaf_rn(nlr, __uint_as_float(g[2 * i + 1]), x.y));
                }
                *slot = w4;
              }
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_2d(&p.wmap, col_base + cofs + c * WCOLS, y0, wbuf);
                bulk_commit();
                bulk_wait_read<0>();                // the store has read the buffer: it may be refilled
              }
              ++wseq;
              issue_loads();
            }
            if (!wok) break;
          } else if (half == 0)      // (SGD kernels: a tile that is not applied is stored by warps 2..5 alone)
#pragma unroll 1
          for (int c = 0; c < BN / 32; ++c) {
            uint32_t r[32];
            if (have_acc) {
              tmem_ld_32x32(tacc + c * 32, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            }
            if (lane == 0) bulk_wait_read<0>();     // the previous block has left the pad
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(pad + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                  make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            const int x0 = col_base + c * 32;
            if (lane == 0 && x0 < p.N) {
              if (p.accumulate) tma_reduce_add_2d(cmap, x0, y0, pad);
              else tma_store_2d(cmap, x0, y0, pad);
              bulk_commit();
            }
          }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (TWO && crank != 0) mbar_arrive_remote(&acc_empty[acc], 0);   // the leader issues the MMAs
        else mbar_arrive(&acc_empty[acc]);
      }
      ++tile_n;
    }
  }
  // ---- teardown: everything joins, in-flight work is given time to land on an abort ----------
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  if (warp >= 2 && lane == 0) bulk_wait<0>();   // epilogue TMA stores have completed
  if constexpr (TWO) cluster_sync_all();        // neither CTA leaves while its peer may still touch it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (TWO) tmem_dealloc2(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace mep

#include "device/dense_f32.cuh"
#include "device/token_gemm.cuh"

namespace mep {

// ---- host side -----------------------------------------------------------------------------------
struct GemmDesc {
  int32_t mode, epi, b_mn, nseg;
  int32_t ngroups, split, total_rows, N, K, rows_per_expert, Mw, accumulate, zero_empty_below, grid;
  int32_t g_begin;
  int64_t a_rows;
  int64_t lda[2];
  const void* a[2];
  const void* b[2][2];
  int64_t b_rows[2];
  int64_t ldb;
  const int32_t* cu_seqlens;
  void* out[3];
  int64_t ldc;
  const float* row_scale;
  int32_t* status;
  int64_t timeout_ns;
  const int32_t* src_info;
  void* push_base;
  int64_t push_rank_stride;
  int32_t push_entries, push_ranks;
  int32_t two_cta, wg_select;
  void* sgd_w;
  const int32_t* sgd_keep;
  float sgd_lr;
  // Fused dispatch (0 = off): 1 = only wait for the rows of each tile to arrive, 2 = also send
  // this rank's rows.  disp_ctx is the Buffer's context; the A operand must be the row buffer
  // `disp_shard` of that Buffer.
  int32_t disp_mode;
  const void* disp_ctx;
  const void* disp_x;
  const float* disp_w;
  const int32_t* disp_dst;
  const int32_t* disp_order;
  const int32_t* disp_zero_fill;
  int32_t disp_fresh, disp_shard;
  const int32_t* pads;
};

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                             CUtensorMapFloatOOBfill);

// 2-D fp32 tensor [rows][cols], box 32 x 32 (128-byte rows), 128B swizzle: weight-grad output.
static int make_map_f32(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld) {
  EncodeFn enc = (EncodeFn)driver_tensor_map_encode();
  if (!enc) return fail(-10, "CUDA driver entry cuTensorMapEncodeTiled not available");
  if (((uintptr_t)base & 15) != 0 || (ld * 4) % 16 != 0)
    return fail(-11, "weight-grad output must be 16-byte aligned with a 16-byte multiple row stride");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(-12, "cuTensorMapEncodeTiled (fp32) failed with code %d", (int)r);
  return 0;
}

// 2-D bf16 tensor [rows][cols] (row stride ld elements), box [box_rows][box_cols], 128B swizzle.
static int make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld,
                    int box_cols, int box_rows, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeFn enc = (EncodeFn)driver_tensor_map_encode();
  if (!enc) return fail(-10, "CUDA driver entry cuTensorMapEncodeTiled not available");
  if (((uintptr_t)base & 15) != 0 || (ld * 2) % 16 != 0)
    return fail(-11, "GEMM operand must be 16-byte aligned with a 16-byte multiple row stride");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(-12, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

// Fused dispatch launches: CTAs of different ranks wait for one another's copy warps, so the whole
// grid must be resident at once.  The grid never exceeds what the device holds next to the weight
// ops' CTAs, and a cooperative launch makes the driver guarantee the residency; MOONEP_B200_FD_COOP=0
// launches plainly instead (the waits stay bounded either way).
static bool fused_dispatch_cooperative() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("MOONEP_B200_FD_COOP");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v != 0;
}

// SGD kernels: dynamic shared memory of a launch (operand stages, alignment slack, four rings of
// 4 KB weight blocks) and the most that the kernel may ask for next to its static part.
static int sgd_smem(const GemmKParams& kp, bool two) {
  return kp.stages * (two ? STAGE_BYTES2 : STAGE_BYTES) + 1024 + 8 * kp.wb * 4096;
}
// How an SGD launch splits its shared memory between operand stages and weight blocks (4 KB, per
// epilogue warp).  Measured on the benchmark's shapes (32 x 1024, 64 x 512, 256 x 128 rows): the
// depth of the weight ring hardly matters once eight warps run the read-modify-write chains (a
// warp needs ~1.4 us per block whatever the depth), so the operand ring gets what is left after
// two (pairs) or three (single CTA, whose stages are 48 KB) blocks per warp.
// MOONEP_B200_SGD_RING="stages,blocks" overrides the choice (tuning).
static void sgd_geometry(bool pair, GemmKParams* kp) {
  if (pair) { kp->stages = 4; kp->wb = 2; }
  else { kp->stages = 2; kp->wb = 3; }
  if (const char* e = getenv("MOONEP_B200_SGD_RING")) {
    int a = 0, b = 0;
    if (sscanf(e, "%d,%d", &a, &b) == 2 && a >= 2 && a <= (pair ? GEMM_STAGES2 : GEMM_STAGES) && b >= 2 &&
        b <= SGD_RING_MAX) {
      kp->stages = a; kp->wb = b;
    }
  }
}
static int sgd_smem_limit(const void* kern) {
  cudaFuncAttributes fa;
  int dev = 0, optin = 0;
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) { cudaGetLastError(); return 0; }
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin - (int)fa.sharedSizeBytes;
}

// CTA-pair launch: clusters of two CTAs, one pair per two SMs.  `coop`: the whole grid must be
// resident at once.
struct PairLaunch {
  std::atomic<unsigned long long> raised{0};
  std::atomic<int> max_clusters{-1};
};
static int launch_pair(const void* kern, PairLaunch& once, GemmKParams kp, int grid, int threads, int smem, bool coop,
                       cudaStream_t stream) {
  MEP_CUDA_OK(raise_smem_limit(kern, once.raised));
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(grid / 2 * 2));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = coop ? 2 : 1;
  // A persistent grid must not exceed what is resident at once: not every SM can be paired
  // into a cluster (GPCs with an odd SM count leave one out), and a second wave of persistent
  // CTAs would double the run time.
  int most = once.max_clusters.load(std::memory_order_relaxed);
  if (most < 0) {
    cudaLaunchConfig_t probe = cfg;
    probe.gridDim = dim3(2 * 148);
    if (cudaOccupancyMaxActiveClusters(&most, kern, &probe) != cudaSuccess || most < 1) { cudaGetLastError(); most = 1 << 20; }
    once.max_clusters.store(most, std::memory_order_relaxed);
  }
  int use = most;
  {
    // a launch with a CTA limit shares the GPU with a copy kernel that is placed as SM pairs too:
    // leave it its pairs out of what the device can hold, or this persistent grid would need a
    // second wave
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (grid < sms && most < (1 << 20)) use = most - (sms - grid + 1) / 2;
    if (use < 1) use = 1;
  }
  if ((int)cfg.gridDim.x / 2 > use) cfg.gridDim = dim3((unsigned)(2 * use));
  void* args[] = {(void*)&kp};
  MEP_CUDA_OK(cudaLaunchKernelExC(&cfg, kern, args));
  return 0;
}
static int launch_single(const void* kern, std::atomic<unsigned long long>& raised, GemmKParams kp, int grid, int threads,
                         int smem, bool coop, cudaStream_t stream) {
  MEP_CUDA_OK(raise_smem_limit(kern, raised));
  void* args[] = {(void*)&kp};
  if (coop) MEP_CUDA_OK(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(threads), args, (size_t)smem, stream));
  else MEP_CUDA_OK(cudaLaunchKernel(kern, dim3(grid), dim3(threads), args, (size_t)smem, stream));
  return 0;
}

template <bool SGD>
static int launch_wgrad(const GemmKParams& kp, bool pair, int grid, cudaStream_t stream) {
  const void* kern = pair ? (const void*)ep_grouped_gemm_kernel<true, SGD>
                          : (const void*)ep_grouped_gemm_kernel<false, SGD>;
  const int smem = SGD ? sgd_smem(kp, pair) : (pair ? gemm_smem<true>() : gemm_smem<false>());
  if (SGD && smem > sgd_smem_limit(kern))
    return fail(-3, "gemm: %d operand stages + %d weight blocks do not fit in shared memory", kp.stages, kp.wb);
  const int threads = SGD ? GEMM_THREADS_SGD : GEMM_THREADS;
  if (pair) {
    static PairLaunch once;
    return launch_pair(kern, once, kp, grid, threads, smem, false, stream);
  }
  static std::atomic<unsigned long long> raised{0};
  return launch_single(kern, raised, kp, grid, threads, smem, false, stream);
}

template <bool W_MN>
static int launch_dense_f32(const DenseParams& dp, cudaStream_t stream) {
  const void* kern = (const void*)ep_dense_f32_kernel<W_MN>;
  static std::atomic<unsigned long long> raised{0};
  MEP_CUDA_OK(raise_smem_limit(kern, raised));
  const dim3 grid((unsigned)((dp.S + dp.tok - 1) / dp.tok), (unsigned)((dp.N + BM - 1) / BM));
  // (the MMA reads 128 rows of the weights' part whatever was loaded: 8 KB beyond the last stage may be read)
  const size_t smem = (size_t)dp.stages * dense_stage_bytes(dp.m_rows, dp.tok) + 1024 + 8192;
  void* args[] = {(void*)&dp};
  MEP_CUDA_OK(cudaLaunchKernel(kern, grid, dim3(DN_THREADS), args, smem, stream));
  return 0;
}

template <bool A_MN, int EPI, bool DISP>
static int launch_token(const GemmKParams& kp, bool pair, int grid, cudaStream_t stream) {
  const int threads = TG_THREADS + (DISP ? 32 : 0);
  const bool coop = DISP && fused_dispatch_cooperative();
  if (pair) {
    static PairLaunch once;
    return launch_pair((const void*)ep_token_gemm_kernel<A_MN, EPI, true, DISP>, once, kp, grid, threads,
                       tg_smem<true, DISP>(), coop, stream);
  }
  if (DISP) {
    // CTAs of different ranks wait for one another's copy warps: all of them must be resident
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (grid > sms) grid = sms;
  }
  static std::atomic<unsigned long long> raised{0};
  return launch_single((const void*)ep_token_gemm_kernel<A_MN, EPI, false, DISP>, raised, kp, grid, threads,
                       tg_smem<false, DISP>(), coop, stream);
}

}  // namespace mep

using namespace mep;

extern "C" {

int mep_gemm_desc_bytes() { return (int)sizeof(GemmDesc); }

int mep_gemm_launch(const GemmDesc* d, cudaStream_t stream) {
  if (d->ngroups < 1 || d->ngroups > MAX_GROUPS) return fail(-1, "gemm: ngroups=%d out of range", d->ngroups);
  GemmKParams kp;
  std::memset(&kp, 0, sizeof(kp));
  kp.cu_seqlens = d->cu_seqlens; kp.ngroups = d->ngroups; kp.split = d->split;
  kp.total_rows = d->total_rows; kp.N = d->N; kp.K = d->K; kp.nseg = d->nseg;
  kp.rows_per_expert = d->rows_per_expert; kp.Mw = d->Mw; kp.accumulate = d->accumulate;
  kp.zero_empty_below = d->zero_empty_below;
  kp.g_begin = d->g_begin; kp.pads = d->pads;
  kp.src_info = d->src_info; kp.push_base = d->push_base; kp.push_rank_stride = d->push_rank_stride;
  kp.push_entries = d->push_entries; kp.push_ranks = d->push_ranks;
  kp.out[0] = d->out[0]; kp.out[1] = d->out[1]; kp.out[2] = d->out[2];
  kp.row_scale = d->row_scale; kp.ldc = d->ldc; kp.status = d->status;
  kp.timeout_ns = (unsigned long long)(d->timeout_ns > 0 ? d->timeout_ns : 2000000000ll);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = d->grid > 0 ? d->grid : sms;
  int rc = 0;
  if (d->mode == 1) {
    // weight grad: A [a_rows][Mw] and B [a_rows][N], both read as MN-major 64x64 boxes
    if (d->Mw % BM != 0) return fail(-2, "wgrad: Mw=%d must be a multiple of %d", d->Mw, BM);
    if ((rc = make_map(&kp.a, d->a[0], d->a_rows, d->Mw, d->lda[0], 64, BK))) return rc;
    if ((rc = make_map(&kp.b[0][0], d->b[0][0], d->a_rows, d->N, d->ldb, 64, BK))) return rc;
    if (d->epi != EPI_F32) return fail(-3, "wgrad writes fp32");
    if (d->sgd_w != nullptr) {
      if (d->accumulate) return fail(-13, "wgrad: the fused SGD step cannot accumulate into existing grads");
      if (d->N % 8 != 0 || ((uintptr_t)d->sgd_w & 15) != 0)
        return fail(-14, "wgrad: the fused SGD step needs N %% 8 == 0 and 16-byte aligned weights");
      kp.sgd_w = (__nv_bfloat16*)d->sgd_w; kp.sgd_keep = d->sgd_keep; kp.sgd_lr = d->sgd_lr;
      const int n_w = d->split < d->ngroups ? d->split : d->ngroups;
      if ((rc = make_map(&kp.wmap, d->sgd_w, (int64_t)n_w * d->Mw, d->N, d->ldc, 64, 32))) return rc;
    }
    const int n_local = d->split < d->ngroups ? d->split : d->ngroups;
    if ((rc = make_map_f32(&kp.c[0], d->out[0], (int64_t)n_local * d->Mw, d->N, d->ldc))) return rc;
    kp.c[1] = kp.c[0];
    if (d->ngroups > d->split) {
      if (d->out[1] == nullptr) return fail(-8, "wgrad: groups >= split need a slot grad tensor");
      if ((rc = make_map_f32(&kp.c[1], d->out[1], (int64_t)(d->ngroups - d->split) * d->Mw, d->N, d->ldc))) return rc;
    }
    const bool pair = d->two_cta != 0 && grid >= 2 && d->Mw % (2 * BM) == 0;
    if (kp.sgd_w != nullptr) sgd_geometry(pair, &kp);
    kp.wg_select = kp.sgd_w != nullptr ? d->wg_select : 0;
    if (kp.sgd_w != nullptr)
      return launch_wgrad<true>(kp, pair, grid, stream);
    return launch_wgrad<false>(kp, pair, grid, stream);
  }
  if (d->epi == EPI_F32) {
    // router logits: one group, one segment
    if (d->ngroups != 1 || d->cu_seqlens != nullptr || d->nseg != 1 || d->accumulate)
      return fail(-15, "gemm: fp32 output is one dense product");
    if (d->K % 8 != 0) return fail(-4, "gemm: K=%d must be a multiple of 8", d->K);
    if (d->total_rows < 1) return 0;
  }
  // Router logits: a dense product with fp32 output whose tiles fill the CTAs at most once.  Larger ones take the
  // token-major kernel (same order of the sums), whose CTAs compute on across tiles: 4096 x 4096 -> 4096
  // columns 237 -> 110 us, 16384 x 2048 -> 512 86 -> 46.  Up to 128 columns half of a pair's tile would be empty:
  // single CTAs, from twice as many tiles on (65536 x 512 -> 128 49 -> 34; 32768 x 2048 -> 128 48 either way).
  const long long dn_rows = ((long long)d->total_rows * ((d->N + BM - 1) / BM) + grid - 1) / grid;
  if (d->epi == EPI_F32 && (dn_rows <= DN_MAX_TOK || (d->N <= BM && dn_rows <= 2 * DN_MAX_TOK))) {
    DenseParams dp;
    std::memset(&dp, 0, sizeof(dp));
    dp.out = (float*)d->out[0]; dp.ldc = d->ldc; dp.S = d->total_rows; dp.N = d->N;
    dp.num_kb = (d->K + BK - 1) / BK;
    dp.status = kp.status; dp.timeout_ns = kp.timeout_ns;
    // token tile: as small as fills the CTAs once, in steps of 16
    dp.tok = dn_rows >= DN_MAX_TOK ? DN_MAX_TOK : ((int)dn_rows + 15) / 16 * 16;
    dp.m_rows = dp.N <= 64 ? 64 : 128;
    const int stage = dense_stage_bytes(dp.m_rows, dp.tok);
    dp.stages = DN_RING / stage < DN_MAX_STAGES ? DN_RING / stage : DN_MAX_STAGES;
    if ((rc = make_map(&dp.x, d->a[0], d->a_rows, d->K, d->lda[0], BK, dp.tok))) return rc;
    if (d->b_mn) {
      if ((rc = make_map(&dp.w, d->b[0][0], d->b_rows[0], d->N, d->ldb, 64, BK))) return rc;
      return launch_dense_f32<true>(dp, stream);
    }
    if ((rc = make_map(&dp.w, d->b[0][0], d->b_rows[0], d->K, d->ldb, BK, dp.m_rows))) return rc;
    return launch_dense_f32<false>(dp, stream);
  }
  // A reduction tail is legal: the TMA loads zero-fill A beyond K, which also cancels whatever
  // a MN-major B tile picks up from the next expert's rows.
  if (d->K % 8 != 0) return fail(-4, "gemm: K=%d must be a multiple of 8", d->K);
  if (d->nseg < 1 || d->nseg > 2) return fail(-5, "gemm: nseg=%d", d->nseg);
  for (int s = 0; s < d->nseg; ++s) {
    for (int b = 0; b < TG_BOXES; ++b)
      if ((rc = make_map(&kp.tok[s][b], d->a[s], d->a_rows, d->K, d->lda[s], BK, 32 * (b + 1)))) return rc;
  }
  const int nsel = (d->epi == EPI_SWIGLU) ? 2 : d->nseg;
  // (maps of operands that a launch does not have stay unset: no tile refers to them)
  for (int s = 0; s < nsel; ++s)
    for (int al = 0; al < 2; ++al) {
      if (d->b[s][al] == nullptr) continue;
      if (d->b_mn) {   // [K rows][N cols] per expert
        if ((rc = make_map(&kp.b[s][al], d->b[s][al], d->b_rows[al], d->N, d->ldb, 64, BK))) return rc;
      } else {         // [N rows][K cols] per expert
        if ((rc = make_map(&kp.b2[s][al], d->b[s][al], d->b_rows[al], d->K, d->ldb, BK, BN / 2))) return rc;
      }
    }
  kp.vec_out = d->ldc % 8 == 0 && (((uintptr_t)d->out[0] | (uintptr_t)d->out[1] | (uintptr_t)d->out[2] |
                                    (uintptr_t)d->push_base) & 15) == 0 && d->push_rank_stride % 8 == 0;
  const bool two = d->two_cta != 0 && grid >= 2;
  if (d->disp_mode != 0) {
    // ---- fused dispatch: the A operand is a row buffer of the Buffer behind disp_ctx ----------
    if (d->disp_ctx == nullptr) return fail(-20, "gemm: the fused dispatch needs the Buffer's context");
    const BufferCtx& c = *(const BufferCtx*)d->disp_ctx;
    if (c.virt) return fail(-21, "gemm: the fused dispatch runs one rank per launch (no virtual groups)");
    if (c.token_padding % BM != 0)
      return fail(-22, "gemm: the fused dispatch needs token_padding %% %d == 0 (tiles must not straddle groups)", BM);
    if (d->nseg != 1 || !d->b_mn || (d->epi != EPI_SWIGLU && d->epi != EPI_BF16))
      return fail(-23, "gemm: the fused dispatch feeds the gate/up (SwiGLU) and the down-dgrad GEMMs only");
    uint8_t* rows = (uint8_t*)c.shard_base(d->disp_shard);
    const long long row_bytes = (long long)c.H * 2;
    if (rows == nullptr || (const uint8_t*)d->a[0] != rows + (size_t)c.rank * c.hidden_stride * row_bytes)
      return fail(-24, "gemm: with the fused dispatch the A operand must be this rank's row buffer %d", d->disp_shard);
    const int nsplit = (int)((row_bytes + FD_PART_CAP - 1) / FD_PART_CAP);
    if (row_bytes % (16 * nsplit) != 0)
      return fail(-25, "gemm: a row of %lld bytes cannot travel in %d equal 16-byte multiples", row_bytes, nsplit);
    FusedDispatch& f = kp.disp;
    f.arrive = c.meta + (size_t)c.rank * c.meta_stride + c.ml.arrive_off;
    f.expect = BM * nsplit;
    f.nsplit = nsplit; f.row_bytes = (int)row_bytes;
    f.hidden = rows; f.meta = c.meta;
    f.hidden_stride_bytes = (long long)c.hidden_stride * row_bytes; f.meta_stride = c.meta_stride;
    f.weights_off = c.ml.weights_off; f.link_off = c.ml.link_off; f.src_off = c.ml.src_off;
    f.arrive_off = c.ml.arrive_off; f.NvS = c.NvS;
    f.N = (int)c.N; f.K = c.K; f.epn = c.epn; f.rank = c.rank; f.R = c.R; f.fresh = d->disp_fresh;
    if (d->disp_mode == 2) {
      if (d->disp_x == nullptr || d->disp_dst == nullptr || d->disp_order == nullptr || d->disp_zero_fill == nullptr)
        return fail(-26, "gemm: the fused dispatch needs the token rows, the plan's dst, send order and padding ranges");
      if (((uintptr_t)d->disp_x & 15) != 0) return fail(-27, "gemm: token rows must be 16-byte aligned");
      f.x = (const uint8_t*)d->disp_x; f.w = d->disp_w; f.dst = d->disp_dst; f.order = d->disp_order;
      f.zero_fill = d->disp_zero_fill;
    }
    kp.trace = c.trace;
    kp.arrive_timeout_ns = c.timeout_ns;                       // waits on other ranks: the Buffer's budget
    kp.timeout_ns = c.timeout_ns + c.timeout_ns / 2 + 200000000ull;
    return d->epi == EPI_SWIGLU ? launch_token<true, EPI_SWIGLU, true>(kp, two, grid, stream)
                                : launch_token<true, EPI_BF16, true>(kp, two, grid, stream);
  }
  if (d->epi == EPI_SWIGLU) {
    if (!d->b_mn) return fail(-6, "swiglu epilogue expects MN-major weights");
    return launch_token<true, EPI_SWIGLU, false>(kp, two, grid, stream);
  }
  if (d->epi == EPI_BF16)
    return d->b_mn ? launch_token<true, EPI_BF16, false>(kp, two, grid, stream)
                   : launch_token<false, EPI_BF16, false>(kp, two, grid, stream);
  if (d->epi == EPI_F32)
    return d->b_mn ? launch_token<true, EPI_F32, false>(kp, two && d->N > BM, grid, stream)
                   : launch_token<false, EPI_F32, false>(kp, two && d->N > BM, grid, stream);
  if (d->epi == EPI_PUSH) {
    if (d->src_info == nullptr || d->push_base == nullptr || d->push_entries <= 0)
      return fail(-9, "gemm: the push epilogue needs src_info and a staging buffer");
    return d->b_mn ? launch_token<true, EPI_PUSH, false>(kp, two, grid, stream)
                   : launch_token<false, EPI_PUSH, false>(kp, two, grid, stream);
  }
  return fail(-7, "gemm: unknown epilogue %d", d->epi);
}

}  // extern "C"
