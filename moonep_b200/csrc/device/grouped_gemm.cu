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
//   ep_weight_grad_kernel (weight_grad.cuh): weight grads, fp32 output or with the SGD step in the epilogue.
// Group g < split reads/writes allocation 0 (local experts), g >= split allocation 1 (this
// rank's prefetch / reduce slots): the [2*epn] compute view never has to be contiguous.
// CTA pairs (template TWO, clusters of two CTAs, tcgen05 cta_group::2): the leader issues
// 256-row MMAs over both CTAs' shared memory; each CTA stages its own 128 rows of A and half
// of the B tile (32 KB per k-block instead of 48 KB), which lifts the single-CTA kernel's limit of
// 12 KB of operand reads per MMA.  Both CTAs' loads count on the LEADER's full
// barrier, on which only the leader's producer arrives (expecting the bytes of both): a per-stage
// arrival from the peer over the cluster network measured 2x slower overall.
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

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int MAX_GROUPS = 1024;

enum { EPI_BF16 = 0, EPI_SWIGLU = 1, EPI_F32 = 2, EPI_PUSH = 3 };

constexpr int TG_BOXES = 4;

struct GemmKParams {
  CUtensorMap a;           // weight grad: token rows of A in 64 x 64 boxes (and of B, in b)
  CUtensorMap tok[2][TG_BOXES];   // token rows in boxes of 32, 64, 96 and 128 rows (token_gemm.cuh)
  CUtensorMap b[2][2];
  CUtensorMap b2[2][2];    // K-major B with a 128-row box; weight grad: grads that are added to, 32 x 32 boxes
  const int32_t* cu_seqlens;
  const int32_t* pads;     // [ngroups][2] first padding row and their number, per group; or null
  int ngroups, split, total_rows, N, K, nseg, rows_per_expert, Mw, accumulate, zero_empty_below;
  // weight grad: tiles of a unit; slots of the shared memory for k-blocks of rows and of columns, and for
  // weight pieces of an epilogue warp (SGD)
  int unit, row_slots, col_slots, pieces;
  int vec32;   // weight grad: rows of the weights allow 32-byte accesses
  int products; // weight grad: 2 = a second one with the same A (b[1], out + 2, sgd_w[1])
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
  __nv_bfloat16* sgd_w[2];
  CUtensorMap wmap[2];        // the same weights as a [G0 * Mw][N] bf16 tensor, 16-row x 64-column boxes
  const int32_t* sgd_keep;
  float sgd_lr;
  void* out[4];
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

template <class Params>
__device__ __forceinline__ bool gemm_wait(uint64_t* bar, uint32_t parity, volatile int* s_abort,
                                          const Params& p, int where) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = globaltimer_ns();
  unsigned spins = 0;
  while (!mbar_try_wait(bar, parity)) {
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

}  // namespace mep

#include "device/dense_f32.cuh"
#include "device/token_gemm.cuh"
#include "device/weight_grad.cuh"

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
  void* out[4];            // weight grad: local and slot grads, of the second product behind them
  int64_t ldc;
  const float* row_scale;
  int32_t* status;
  int64_t timeout_ns;
  const int32_t* src_info;
  void* push_base;
  int64_t push_rank_stride;
  int32_t push_entries, push_ranks;
  int32_t two_cta, wg_select;
  void* sgd_w[2];
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
  int32_t rows_used;               // weight grad: rows that hold tokens, on the host's knowledge (0: total_rows)
};

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                             CUtensorMapFloatOOBfill);

// 2-D tensor [rows][cols] of bf16, or with F32 of fp32 (row stride ld elements), box [box_rows][box_cols], 128B swizzle.
template <bool F32 = false>
static int make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld,
                    int box_cols, int box_rows) {
  EncodeFn enc = (EncodeFn)driver_tensor_map_encode();
  if (!enc) return fail(-10, "CUDA driver entry cuTensorMapEncodeTiled not available");
  const int bytes = F32 ? 4 : 2;
  if (((uintptr_t)base & 15) != 0 || (ld * bytes) % 16 != 0)
    return fail(-11, "GEMM operand must be 16-byte aligned with a 16-byte multiple row stride");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * bytes)};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
                   dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   F32 ? CU_TENSOR_MAP_L2_PROMOTION_NONE : CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
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

// How a weight-grad launch splits its shared memory and its tiles, by the average number of k-blocks a group: `rows`
// is the number of rows that hold tokens, where the caller knows it.  (The length of a layer's row tensor is its
// capacity, up to two paddings an expert more: 8 blocks a group where there are 4.)  Every choice computes every
// group.  Figures: the three weight grads of a layer's step (down; gate and up in one launch), padding 128, Zipf 0.3 -
// 0.9, us.
static void wgrad_geometry(GemmKParams* kp, int rows, bool pair) {
  const int local = kp->split < kp->ngroups ? kp->split : kp->ngroups;
  const double kb = (double)rows / (local > 0 ? local : 1) / BK;
  const int tiles_n = (kp->N + BN - 1) / BN;
  kp->pieces = 0;
  kp->unit = 1;
  if (kp->sgd_w[0] != nullptr) {
    // Up to five blocks the stream of old weights needs two pieces a warp in flight, longer groups the operand slots
    // (128 experts, 4096 x 1024, 4 blocks 1528, 1567 with one piece; 64, 2048 x 1536, 8 blocks 809, 788).
    kp->pieces = kb < 5 ? 2 : 1;
    kp->row_slots = (pair ? 7 : 5) - kp->pieces;
    kp->col_slots = pair ? 6 - kp->pieces : 3;
    // Two tiles that share staged rows: with eight column tiles from two blocks on (64 experts, 7168 x 2048: 4 blocks 2683,
    // 2513 so; 2 blocks 2146, 2133), with four and six from eight (2048 x 1536: 4 blocks 1096, 1175; 8 788, 768); not
    // with two (1024 x 512, 8 blocks 155, 173) nor an odd number, which leaves units of unequal length (2048 x 768, 4
    // blocks 627, 788).
    if (tiles_n % 2 == 0 && kb >= (tiles_n >= 8 ? 1.5 : tiles_n >= 4 ? 8 : 1e9)) kp->unit = 2;
  } else if (kp->accumulate) {
    // One warp of a row quarter adds; more of them, with pieces of their own, cost slots and let tiles run
    // ahead of the read-modify-writes in L2 (2048 x 768, 64 experts x 8 blocks 586, 590 with four; 7168 x 2048, 32 x 16 3106,
    // 4124; 4096 x 1024, 128 x 1 2569, 2602).
    kp->row_slots = pair ? 7 : 5;
    kp->col_slots = pair ? 5 : 3;
  } else {
    kp->row_slots = pair ? 7 : 5;
    kp->col_slots = pair ? 6 : 4;
  }
}
static int wgrad_smem(const GemmKParams& kp, bool pair) {
  return kp.row_slots * WG_ROW_BYTES + kp.col_slots * (pair ? wg_col_bytes<true>() : wg_col_bytes<false>()) +
         WG_EPI_WARPS * kp.pieces * WG_PIECE + (kp.accumulate ? 4 * WG_ADD_PIECE : 0) + 1024;
}

template <int MODE>
static int launch_wgrad(const GemmKParams& kp, bool pair, int grid, cudaStream_t stream) {
  const int smem = wgrad_smem(kp, pair);
  if (pair) {
    static PairLaunch once;
    return launch_pair((const void*)ep_weight_grad_kernel<true, MODE>, once, kp, grid, WG_THREADS, smem, false, stream);
  }
  static std::atomic<unsigned long long> raised{0};
  return launch_single((const void*)ep_weight_grad_kernel<false, MODE>, raised, kp, grid, WG_THREADS, smem, false, stream);
}

template <bool W_MN>
static int launch_dense_f32(const DenseParams& dp, cudaStream_t stream) {
  const void* kern = (const void*)ep_dense_f32_kernel<W_MN>;
  static std::atomic<unsigned long long> raised{0};
  MEP_CUDA_OK(raise_smem_limit(kern, raised));
  const dim3 grid((unsigned)((dp.S + dp.tok - 1) / dp.tok), (unsigned)((dp.N + BM - 1) / BM));
  // (the MMA reads 128 rows of the weights' part whatever was loaded: 8 KB beyond the last stage may be read)
  const size_t smem = (size_t)dp.stages * dp.blocks * dense_block_bytes(dp.m_rows, dp.tok) + 1024 + 8192;
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
  kp.out[0] = d->out[0]; kp.out[1] = d->out[1]; kp.out[2] = d->out[2]; kp.out[3] = d->out[3];
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
    if (d->epi != EPI_F32) return fail(-3, "wgrad writes fp32");
    kp.products = d->b[1][0] != nullptr ? 2 : 1;
    if (d->sgd_w[0] != nullptr) {
      if (d->accumulate) return fail(-13, "wgrad: the fused SGD step cannot accumulate into existing grads");
      kp.sgd_keep = d->sgd_keep; kp.sgd_lr = d->sgd_lr;
      kp.vec32 = d->N % 16 == 0;
    }
    for (int i = 0; i < kp.products; ++i) {
      if ((rc = make_map(&kp.b[i][0], d->b[i][0], d->a_rows, d->N, d->ldb, 64, BK))) return rc;
      if (d->sgd_w[0] != nullptr) {
        if (d->N % 8 != 0 || d->sgd_w[i] == nullptr || ((uintptr_t)d->sgd_w[i] & 15) != 0)
          return fail(-14, "wgrad: the fused SGD step needs N %% 8 == 0 and 16-byte aligned weights");
        kp.sgd_w[i] = (__nv_bfloat16*)d->sgd_w[i];
        kp.vec32 = kp.vec32 && ((uintptr_t)d->sgd_w[i] & 31) == 0;
        const int n_w = d->split < d->ngroups ? d->split : d->ngroups;
        if ((rc = make_map(&kp.wmap[i], d->sgd_w[i], (int64_t)n_w * d->Mw, d->N, d->ldc, 64, 16))) return rc;
      }
      if (d->ngroups > d->split && d->out[2 * i + 1] == nullptr) return fail(-8, "wgrad: groups >= split need a slot grad tensor");
      if ((((uintptr_t)d->out[2 * i] | (uintptr_t)d->out[2 * i + 1]) & 15) != 0 || d->ldc % 4 != 0)
        return fail(-11, "weight-grad output must be 16-byte aligned with a 16-byte multiple row stride");
      if (d->accumulate) {
        const int64_t n_local = d->split < d->ngroups ? d->split : d->ngroups;
        if ((rc = make_map<true>(&kp.b2[i][0], d->out[2 * i], n_local * d->Mw, d->N, d->ldc, 32, 32))) return rc;
        if (d->ngroups > d->split &&
            (rc = make_map<true>(&kp.b2[i][1], d->out[2 * i + 1], (d->ngroups - n_local) * d->Mw, d->N, d->ldc, 32, 32))) return rc;
      }
    }
    const bool pair = d->two_cta != 0 && grid >= 2;
    wgrad_geometry(&kp, d->rows_used > 0 ? d->rows_used : d->total_rows, pair);
    kp.wg_select = kp.sgd_w[0] != nullptr ? d->wg_select : 0;
    if (kp.sgd_w[0] != nullptr) return launch_wgrad<WG_SGD>(kp, pair, grid, stream);
    return kp.accumulate ? launch_wgrad<WG_ADD>(kp, pair, grid, stream) : launch_wgrad<WG_STORE>(kp, pair, grid, stream);
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
    const int fit = DN_RING / dense_block_bytes(dp.m_rows, dp.tok);
    // four blocks a stage where four such stages fit (up to 64 experts x 32 tokens), else two (4096 x 7168 -> 128: 28.7 us,
    // 34.8 with four)
    dp.blocks = fit >= 4 * DN_MAX_BLOCKS ? DN_MAX_BLOCKS : 2;
    dp.stages = fit / dp.blocks < DN_MAX_STAGES ? fit / dp.blocks : DN_MAX_STAGES;
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
