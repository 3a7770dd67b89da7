// C[S][N] = A[S][K] * B[K][N] (or B[N][K]) with fp32 output: the router logits.  (Outputs of more tiles than the
// CTAs hold at once go to the token-major kernel.)
//
// The output is small (S x experts) and the reduction long: a CTA walks up to 112 k-blocks one after
// the other, bound by that chain and not by bytes or MMAs (25 us for 8 as for 128 experts; 21 with no MMA but the
// first).  The experts take the M side (128 a tile) and the tokens the N side, in as small a tile as fills the SMs
// once (4096 tokens are 128 CTAs of 32).  Loads and MMAs are issued by one lane of a converged warp, which halved the
// chain (K = 7168 50 -> 25 us for 16 tokens), and one wait and one commit serve two or four k-blocks, which are
// what remains of it: inputs out of L2, 16 x 7168 -> 32 experts 28.5 -> 19.4 us, 1531 29.5 -> 21.4, 4096 31.6 -> 27.6, 4096 ->
// 128 experts 30.7 -> 28.7.  The reduction is NOT split: routing compares these sums, and another order of the
// additions sends tokens at a tie elsewhere.
#pragma once

namespace mep {

constexpr int DN_MAX_STAGES = 16;
constexpr int DN_THREADS = 192;
constexpr int DN_RING = 200 * 1024;
constexpr int DN_MAX_TOK = 128;
constexpr int DN_MAX_BLOCKS = 4;       // k-blocks of a stage, at most

struct DenseParams {
  CUtensorMap x, w;      // tokens: tok x 64 boxes; weights: 64 x 64 (B [K][N]) or m_rows x 64 boxes (B [N][K])
  float* out;
  long long ldc;
  int S, N, num_kb, tok, m_rows, stages, blocks;
  int32_t* status;
  unsigned long long timeout_ns;
};
__host__ __device__ constexpr int dense_block_bytes(int m_rows, int tok) { return (m_rows + tok) * BK * 2; }

template <bool W_MN>
__global__ void __launch_bounds__(DN_THREADS, 1) ep_dense_f32_kernel(const __grid_constant__ DenseParams p) {
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full[DN_MAX_STAGES];
  __shared__ __align__(8) uint64_t empty[DN_MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  volatile int* abortp = &s_abort;
  const int row0 = (int)blockIdx.x * p.tok, m0 = (int)blockIdx.y * BM;
  // (with at most 64 experts only half of the M side is loaded; what the other lanes compute is not stored)
  const int w_bytes = p.m_rows * BK * 2, block_bytes = dense_block_bytes(p.m_rows, p.tok), stage_bytes = p.blocks * block_bytes;

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(&acc_full, 1);
    mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 1) { tmem_alloc(&s_tmem, DN_MAX_TOK); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;

  // a wait has the same outcome in every lane: a warp walks its loop as a whole, one lane issues
  auto warp_wait = [&](uint64_t* bar, uint32_t parity, int where) {
    return __all_sync(0xffffffffu, gemm_wait(bar, parity, abortp, p, where)) != 0;
  };
  if (warp == 0) {
    const bool issue = elect_one();
    if (issue) {
      tma_prefetch_desc(&p.x);
      tma_prefetch_desc(&p.w);
    }
    RingSlot st;
    for (int kb0 = 0; kb0 < p.num_kb; kb0 += p.blocks, st.next(p.stages)) {
      const int s = st.slot, blocks = min(p.blocks, p.num_kb - kb0);
      if (!warp_wait(&empty[s], st.parity ^ 1u, 1)) break;
      if (!issue) continue;
      mbar_expect_tx(&full[s], (uint32_t)(blocks * block_bytes));
      for (int b = 0; b < blocks; ++b) {
        uint8_t* sw = ring + s * stage_bytes + b * block_bytes;
        const int k = (kb0 + b) * BK;
        if constexpr (W_MN) {
          for (int j = 0; j < p.m_rows / 64; ++j) tma_load_2d(sw + j * 8192, &p.w, m0 + 64 * j, k, &full[s]);
        } else {
          tma_load_2d(sw, &p.w, k, m0, &full[s]);
        }
        tma_load_2d(sw + w_bytes, &p.x, k, row0, &full[s]);
      }
    }
  } else if (warp == 1) {
    const bool issue = elect_one();
    const uint32_t idesc = make_instr_desc_bf16(BM, p.tok, W_MN, false);
    // (64 experts: the descriptor's second block of columns / rows is the token part of the stage)
    const uint64_t desc_w = W_MN ? make_smem_desc(smem_u32(ring), 8192, 1024) : make_smem_desc(smem_u32(ring), 16, 1024);
    const uint64_t desc_x = make_smem_desc(smem_u32(ring) + w_bytes, 16, 1024);
    constexpr int W_STEP = (W_MN ? 2048 : 32) >> 4, X_STEP = 32 >> 4;
    RingSlot st;
    bool ok = true;
    for (int kb0 = 0; kb0 < p.num_kb; kb0 += p.blocks, st.next(p.stages)) {
      ok = warp_wait(&full[st.slot], st.parity, 3);
      if (!ok) break;
      tc_fence_after();
      if (issue) {
#pragma unroll
        for (int b = 0; b < DN_MAX_BLOCKS; ++b) {
          if (b >= p.blocks || kb0 + b >= p.num_kb) break;
          const uint32_t at = (uint32_t)((st.slot * stage_bytes + b * block_bytes) >> 4);
          const uint64_t dw = desc_w + at, dx = desc_x + at;
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_bf16(tmem_base, dw + kk * W_STEP, dx + kk * X_STEP, idesc, (kb0 + b > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(&empty[st.slot]);
      }
    }
    if (ok && issue) umma_commit(&acc_full);
  } else {
    // thread = expert: a token's 32 logits of a warp leave as one 128-byte line
    const int q = warp & 3;
    const bool have = gemm_wait(&acc_full, 0, abortp, p, 4);
    __syncwarp();
    tc_fence_after();
    const int col = m0 + q * 32 + lane;
    if (__all_sync(0xffffffffu, have)) {
      for (int c = 0; c < p.tok && row0 + c < p.S; c += 16) {
        uint32_t r[16];
        __syncwarp();
        tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (row0 + c + i < p.S && col < p.N) p.out[(long long)(row0 + c + i) * p.ldc + col] = __uint_as_float(r[i]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_abort) {       // in-flight loads are given time to land
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, DN_MAX_TOK);
  }
}

}  // namespace mep
