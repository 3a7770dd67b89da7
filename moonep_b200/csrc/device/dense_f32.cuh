// C[S][N] = A[S][K] * B[K][N] (or B[N][K]) with fp32 output: the router logits.
//
// The output is small (S x experts) and the reduction long, so 128-row tiles alone leave most SMs
// idle: 4096 tokens are 32 CTAs walking 112 k-blocks one after the other (65 us at K = 7168), 16
// tokens are one (47 us).  A cluster of up to eight CTAs therefore shares a tile: each takes a
// contiguous part of the k-blocks, leaves its fp32 partial tile in its shared memory (over the spent
// operand ring), and after a cluster barrier every CTA sums its share of the tile's rows over the
// cluster's partials through distributed shared memory, in rank order, so the result does not depend
// on timing.  Bound by reading A once (59 MB, 9 us at 4096 x 7168).
// A stage holds 128 rows of A and only as many 64-column blocks of B as the tile has.
#pragma once

namespace mep {

constexpr int DN_MAX_STAGES = 8;
constexpr int DN_THREADS = 192;
constexpr int DN_RING = 200 * 1024;

struct DenseParams {
  CUtensorMap a, b;      // A: 128 x 64 boxes; B: 64 x 64 boxes (either layout)
  float* out;
  long long ldc;
  int S, N, num_kb, tile_n, stages;
  int32_t* status;
  unsigned long long timeout_ns;
};

template <bool B_MN>
__global__ void __launch_bounds__(DN_THREADS, 1) ep_dense_f32_kernel(const __grid_constant__ DenseParams p) {
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full[DN_MAX_STAGES];
  __shared__ __align__(8) uint64_t empty[DN_MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int parts = (int)gridDim.x, part = (int)blockIdx.x;      // one cluster spans grid.x
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  volatile int* abortp = &s_abort;
  const int row0 = (int)blockIdx.y * BM, n0 = (int)blockIdx.z * p.tile_n;
  const int n_here = min(p.tile_n, p.N - n0);
  const int mma_n = (n_here + 15) & ~15, blocks = (n_here + 63) / 64;
  const int stage_bytes = A_TILE_BYTES + (p.tile_n + 63) / 64 * 8192;
  const int kb0 = (int)((long long)p.num_kb * part / parts), kb1 = (int)((long long)p.num_kb * (part + 1) / parts);

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(&acc_full, 1);
    mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 1) { tmem_alloc(&s_tmem, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;

  if (warp == 0 && lane == 0) {
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % p.stages;
      if (it >= p.stages && !gemm_wait(&empty[s], ((uint32_t)(it / p.stages) & 1u) ^ 1u, abortp, p, 1)) break;
      uint8_t* sa = ring + (size_t)s * stage_bytes;
      mbar_expect_tx(&full[s], (uint32_t)(A_TILE_BYTES + blocks * 8192));
      tma_load_2d(sa, &p.a, kb * BK, row0, &full[s]);
      for (int j = 0; j < blocks; ++j) {
        if constexpr (B_MN) tma_load_2d(sa + A_TILE_BYTES + j * 8192, &p.b, n0 + 64 * j, kb * BK, &full[s]);
        else tma_load_2d(sa + A_TILE_BYTES + j * 8192, &p.b, kb * BK, n0 + 64 * j, &full[s]);
      }
    }
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = make_instr_desc_bf16(BM, mma_n, false, B_MN);
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % p.stages;
      if (!gemm_wait(&full[s], (uint32_t)(it / p.stages) & 1u, abortp, p, 3)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sa = smem_u32(ring + (size_t)s * stage_bytes), sb = sa + A_TILE_BYTES;
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) {
        const uint64_t da = make_smem_desc(sa + kk * 32, 16, 1024);
        const uint64_t db = B_MN ? make_smem_desc(sb + kk * 2048, 8192, 1024) : make_smem_desc(sb + kk * 32, 16, 1024);
        umma_bf16(tmem_base, da, db, idesc, (it > 0 || kk > 0) ? 1u : 0u);
      }
      umma_commit(&empty[s]);
    }
    if (ok) umma_commit(&acc_full);
  }
  __syncwarp();
  // ---- partial tile into shared memory: every MMA has read the ring by now --------------------------
  const int pitch = mma_n + 4;       // floats; consecutive rows start 4 banks (mod 16-byte steps) apart
  float* mine = reinterpret_cast<float*>(ring);
  if (warp >= 2) {
    const int q = warp & 3;
    bool have = kb1 > kb0;
    if (have) have = gemm_wait(&acc_full, 0, abortp, p, 4);
    __syncwarp();
    tc_fence_after();
    float* row = mine + (size_t)(q * 32 + lane) * pitch;
    for (int c = 0; c < mma_n; c += 16) {
      uint32_t r[16];
      __syncwarp();
      tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        *reinterpret_cast<float4*>(row + c + i) = kb1 > kb0
            ? make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]))
            : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    tc_fence_before();
  }
  cluster_sync_all();
  // ---- rows [128 part / parts, ..): the sum of the cluster's partials, in rank order -----------------
  const int r_lo = BM * part / parts, r_hi = min(BM * (part + 1) / parts, p.S - row0);
  const int vecs = mma_n / 4;
  const uint32_t base = smem_u32(mine);
  const bool vec_ok = p.ldc % 4 == 0 && n0 % 4 == 0 && ((uintptr_t)p.out & 15) == 0;
  for (int i = tid; i < (r_hi - r_lo) * vecs; i += DN_THREADS) {
    const int r = r_lo + i / vecs, c = (i - (r - r_lo) * vecs) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < parts; ++k) {
      const float4 v = ld_cluster_f4(base + (uint32_t)(r * pitch + c) * 4u, (uint32_t)k);
      if (k == 0) sum = v;
      else { sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w; }
    }
    float* o = p.out + (long long)(row0 + r) * p.ldc + n0 + c;
    if (vec_ok && c + 4 <= n_here) {
      *reinterpret_cast<float4*>(o) = sum;
    } else {
      const float e[4] = {sum.x, sum.y, sum.z, sum.w};
      for (int j = 0; j < 4 && c + j < n_here; ++j) o[j] = e[j];
    }
  }
  if (s_abort) {       // in-flight loads are given time to land
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  cluster_sync_all();  // no CTA leaves while a peer may still read its partial
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

}  // namespace mep
