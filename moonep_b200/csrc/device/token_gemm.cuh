// Token-major grouped GEMM with the WEIGHTS on the M side of the tensor-core tile and the TOKENS on
// its N side:  C[rows of g] = A[rows of g] * B[g]  is computed as  C^T = B[g]^T * A^T.
//
// Why: an MMA has a fixed M (128 rows a CTA, 256 a CTA pair) but any N up to 256 in steps of 32.
// Expert groups are ragged; the weights' output columns are not.  With tokens on M a group of 300
// rows computed 512 (pairs) or 384 (single CTAs, which read 1.5x the operand bytes per MMA);
// with tokens on N it computes 320, always in pairs, and a group that only has 10 rows costs 32.
// The step is power-limited (1.65 of 1.965 GHz), so work on padding costs clocks everywhere.
//
// A tile is 256 (pair; 128 single CTA) output columns x up to 256 tokens of one group.  A group
// of L rows is cut into ceil(L / 256) tiles of equal size, rounded up to 32.  L counts the group's
// real rows when the caller gives the padding ranges (GemmKParams::pads): padding rows beyond the
// last tile are written as zeros, what the product of a zero row is, without being computed.
// Per k-block of 64 each CTA of a pair stages its 128 output columns of the weights (16 KB) and half of
// the tokens (up to 16 KB) in one of six stages (five beside the fused dispatch's copy ring).
//   warp 0  TMA producer (and, with the fused dispatch, 31 arrival watchers)
//   warp 1  MMA issuer   (two 256-column TMEM accumulators)
//   warps 2..5, 6..9 epilogue, two sets of four that take 32 tokens in turn: they are read as matrix
//           fragments, rounded to bf16 and transposed by stmatrix into token rows in shared memory,
//           then leave as 256-byte (SwiGLU: 128-byte) row segments.  A step is a chain of latencies
//           (~0.6 us for 32 tokens), which with one set was a tile's time where the reduction is short:
//           128 groups x 256 rows, H = 1024, H' = 512, gate/up 127 -> 99 us; 280 rows, down 78 -> 68;
//           H' = 64, 53 -> 47; long reductions the same
//   warp 10 copy warp of the fused dispatch
// SwiGLU: a CTA's 128 columns are 64 gate and the same 64 up columns, which meet in the staged rows.
//
// Measured against tokens on M (pairs; isolated launches, 32 groups, H = 7168, H' = 2048), gate/up:
// 1024 rows a group 1435 -> 1433 us (1.34 PFLOP/s), 896: 1423 -> 1358, 640: 1086 -> 1039, 224: 410 -> 388, 128:
// 398 -> 321, 32: 379 -> 284 (the weights' 1.9 GB at the copy rate); down: 680 -> 701, 675 -> 665, 517 -> 508,
// 202 -> 195, 197 -> 172, 188 -> 161.
#pragma once

namespace mep {

constexpr int TG_MAX_N = 256;
constexpr int TG_CHUNK = 32;                                  // tokens per epilogue step
constexpr int TG_SETS = 2;                                    // sets of four epilogue warps
constexpr int TG_THREADS = 64 + TG_SETS * 128;                // and one more warp with the fused dispatch
constexpr int TG_STAGE_ROW = 256 + 16;                        // bytes of a staged token row: 128 columns; the rows
                                                              // of an 8x8 matrix fall into different banks
constexpr int TG_W_BYTES = BM * BK * 2;                       // weights of a k-block, one CTA: 16 KB

template <bool TWO> __host__ __device__ constexpr int tg_stage_bytes() { return TG_W_BYTES + (TWO ? 128 : 256) * BK * 2; }
template <bool TWO, bool DISP> __host__ __device__ constexpr int tg_stages() { return (TWO ? 6 : 4) - (DISP ? 1 : 0); }
// Fused dispatch: stages of the copy ring, in what one operand stage and the slack leave.
constexpr int TG_FD_STAGES = 5;
template <bool TWO, bool DISP> __host__ __device__ constexpr int tg_smem() {
  return tg_stages<TWO, DISP>() * tg_stage_bytes<TWO>() + 1024 + (DISP ? TG_FD_STAGES * FD_PART_CAP : 0);
}

struct TokenTile {
  int g, alloc, g_local;
  int row0, n;             // first token row, tokens computed (a multiple of 32)
  int rows, zero_to;       // rows stored; this tile also zeroes the rows [row0 + rows, zero_to)
  int m0;                  // first output column of the CTA pair (or CTA)
};

__device__ __forceinline__ int token_tiles(int valid) { return (valid + TG_MAX_N - 1) / TG_MAX_N; }

// Eight bf16 of a row, of which `left` lie inside it.
__device__ __forceinline__ void store8(__nv_bfloat16* dst, const uint4& v, int left, bool vec_ok) {
  if (vec_ok && left >= 8) {
    *reinterpret_cast<uint4*>(dst) = v;
  } else {
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&v);
    for (int i = 0; i < 8 && i < left; ++i) dst[i] = e[i];
  }
}
// Barrier of a set's four epilogue warps, and one that also agrees on a condition: true if it held for all of them.
__device__ __forceinline__ void epilogue_sync(int set) { asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory"); }
__device__ __forceinline__ bool epilogue_all(int set, bool mine) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"((uint32_t)mine), "r"(1 + set) : "memory");
  return all != 0;
}

template <bool A_MN, int EPI, bool TWO, bool DISP>
__global__ void __launch_bounds__(TG_THREADS + (DISP ? 32 : 0), 1)
ep_token_gemm_kernel(const __grid_constant__ GemmKParams p) {
  constexpr int NST = tg_stages<TWO, DISP>();
  constexpr int STAGE = tg_stage_bytes<TWO>();
  constexpr int FD_NST = TG_FD_STAGES;
  constexpr int TM = TWO ? 2 * BM : BM;
  constexpr int COLS = EPI == EPI_SWIGLU ? TM / 2 : TM;      // output columns of a tile
  const int crank = TWO ? (int)cluster_cta_rank() : 0;       // 0 = leader of the pair
  const int work_id0 = TWO ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int work_stride = TWO ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full[NST];
  __shared__ __align__(8) uint64_t empty[NST];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ __align__(8) uint64_t fd_full[DISP ? FD_NST : 1];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_groups_ready;
  __shared__ int s_end[MAX_GROUPS];
  __shared__ int s_prefix[MAX_GROUPS + 1];
  __shared__ __align__(128) uint8_t s_stage[TG_SETS][EPI == EPI_F32 ? 16 : TG_CHUNK * TG_STAGE_ROW];
  // per token of a tile: address of its row at the home rank (PUSH) or its scale (SwiGLU); two tiles
  __shared__ unsigned long long s_ptr[EPI == EPI_PUSH ? 2 : 1][EPI == EPI_PUSH ? TG_MAX_N : 1];
  __shared__ float s_scale[EPI == EPI_SWIGLU ? 2 : 1][EPI == EPI_SWIGLU ? TG_MAX_N : 1];

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  uint8_t* stages = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  volatile int* abortp = &s_abort;

  if (tid == 0) {
    // both CTAs' loads count on the LEADER's full barrier, on which only its producer arrives
    for (int s = 0; s < NST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], (TWO ? 8 : 4) * TG_SETS); }
    if constexpr (DISP) for (int a = 0; a < FD_NST; ++a) mbar_init(&fd_full[a], 1);
    mbar_fence_init();
    s_abort = 0;
    s_groups_ready = 0;
  }
  for (int g = tid; g < p.ngroups; g += (int)blockDim.x)
    s_end[g] = p.cu_seqlens != nullptr ? p.cu_seqlens[g] : p.total_rows;
  __syncthreads();
  if (warp == 0) {      // exclusive prefix of token tiles per group
    int run = 0;
    for (int g0 = 0; g0 < p.ngroups; g0 += 32) {
      const int g = g0 + lane;
      int nt = 0;
      if (g < p.ngroups && g >= p.g_begin) {
        const int start = g == 0 ? 0 : s_end[g - 1];
        nt = s_end[g] > start ? token_tiles(group_valid(p, g, start, s_end[g])) : 0;
      }
      int incl = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (g < p.ngroups) s_prefix[g] = run + incl - nt;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_prefix[p.ngroups] = run;
  }
  if (warp == 1) {
    if constexpr (TWO) { tmem_alloc2(&s_tmem, 512); tmem_relinquish2(); }
    else { tmem_alloc(&s_tmem, 512); tmem_relinquish(); }
  }
  tc_fence_before();
  if constexpr (TWO) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;

  const int m_tiles = (p.N + COLS - 1) / COLS;
  const long long total_tiles = (long long)s_prefix[p.ngroups] * m_tiles;
  auto get = [&](int id) {
    TokenTile t;
    int lo = 0, hi = p.ngroups - 1;      // largest g with prefix[g] * m_tiles <= id
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((long long)s_prefix[mid] * m_tiles <= id) lo = mid; else hi = mid - 1;
    }
    t.g = lo;
    const int nt = s_prefix[lo + 1] - s_prefix[lo];
    const int local = id - s_prefix[lo] * m_tiles;
    const int mi = local / nt, ti = local - mi * nt;       // tiles that share weights are neighbours
    const int start = lo == 0 ? 0 : s_end[lo - 1], end = s_end[lo];
    const int valid = group_valid(p, lo, start, end);
    t.n = ((valid + nt - 1) / nt + 31) & ~31;
    t.row0 = start + ti * t.n;
    t.rows = max(0, min(t.n, end - t.row0));
    t.zero_to = ti == nt - 1 ? end : 0;
    t.m0 = mi * COLS;
    t.alloc = lo >= p.split ? 1 : 0;
    t.g_local = t.alloc ? lo - p.split : lo;
    return t;
  };
  const int kb_per_seg = (p.K + BK - 1) / BK;
  // The producer's and the issuer's warps walk their loops as a whole and one lane issues: loop state and
  // descriptors then live in uniform registers.  With the loops in a single lane's branch, the issuer took
  // longer for a k-block than the tensor cores and set the rate.  Isolated launches, H = 7168, H' = 2048, us:
  // 128 groups of 256 rows on average, gate/up 1980 -> 1765, down 1165 -> 1070; 32 groups of 1024, 1530 -> 1440
  // and 850 -> 750; 16 tokens on 32 experts (a stream of the weights) 344 -> 304 and 178 -> 172.
  // A wait has the same outcome in every lane, so that the warp leaves its loops together.  (Beside the
  // arrival watchers of the fused dispatch the producer is one lane.)
  auto warp_wait = [&](uint64_t* bar, uint32_t parity, int where) {
    return __all_sync(0xffffffffu, gemm_wait(bar, parity, abortp, p, where)) != 0;
  };

  if (warp == 0) {
    // ================= TMA producer =================
    if (!DISP || lane == 0) {
      const bool issue = DISP || elect_one();
      if (issue) {
        tma_prefetch_desc(&p.tok[0][TG_BOXES - 1]);
        tma_prefetch_desc(A_MN ? &p.b[0][0] : &p.b2[0][0]);
      }
      RingSlot st;
      bool ok = true;
      int groups_ready = 0;
      if constexpr (DISP) phase_stamp(p.trace, 2, (int)blockIdx.x, 0);
      bool stamped_first = false;
      for (long long id = work_id0; id < total_tiles && ok; id += work_stride) {
        TokenTile t = get((int)id);
        if constexpr (!DISP) {
          // (the same in every lane: said so)
          t.alloc = __shfl_sync(0xffffffffu, t.alloc, 0);
          t.g_local = __shfl_sync(0xffffffffu, t.g_local, 0);
          t.row0 = __shfl_sync(0xffffffffu, t.row0, 0);
          t.n = __shfl_sync(0xffffffffu, t.n, 0);
          t.m0 = __shfl_sync(0xffffffffu, t.m0, 0);
        }
        if constexpr (DISP) {
          // wait for the tile's whole GROUP, published by the watchers below: CTAs then enter a group
          // together and share its rows and weights in L2
          if (p.disp.arrive != nullptr && t.g >= groups_ready) {
            unsigned long long t0 = 0ull;
            unsigned spins = 0;
            while ((groups_ready = *(volatile int*)&s_groups_ready) <= t.g) {
              if ((++spins & 63u) == 0) {
                if (t0 == 0ull) t0 = globaltimer_ns();
                if (*abortp || globaltimer_ns() - t0 > p.timeout_ns) { ok = false; break; }
              }
            }
            if (!ok) break;
            __threadfence_block();
            fence_proxy_async();   // the rows were written through the async proxy (or by plain stores)
            if (!stamped_first) { phase_stamp(p.trace, 2, (int)blockIdx.x, 1); stamped_first = true; }
          }
        }
        const int tok = TWO ? t.n / 2 : t.n;               // tokens staged by this CTA
        const int trow = t.row0 + crank * tok;
        // Tokens arrive in ONE box a stage (a second one above 128, single CTAs), the smallest of four
        // heights that covers them: boxes of 16 rows, exactly covering, cost more than the rows they
        // saved (pairs, 224 tokens: 1722 us with four boxes where 256 tokens in one took 1600).
        const int box = min(4, (tok + 31) / 32);
        const CUtensorMap* tmap = &p.tok[0][0] + (box - 1);
        const uint32_t bytes = (uint32_t)(TG_W_BYTES + box * (!TWO && tok > 128 ? 64 : 32) * BK * 2) * (TWO ? 2u : 1u);
        const int erow = t.g_local * p.rows_per_expert;
        for (int seg = 0; seg < p.nseg && ok; ++seg)
        for (int k0 = 0; k0 < p.K; k0 += BK, st.next(NST)) {
          const int s = st.slot;
          if constexpr (DISP) ok = gemm_wait(&empty[s], st.parity ^ 1u, abortp, p, 1);
          else ok = warp_wait(&empty[s], st.parity ^ 1u, 1);
          if (!ok) break;
          if (!issue) continue;
          uint8_t* sw = stages + (size_t)s * STAGE;
          uint8_t* stok = sw + TG_W_BYTES;
          uint32_t lead_bar = 0;
          if constexpr (TWO) lead_bar = mapa_u32(&full[s], 0);
          if (crank == 0) mbar_expect_tx(&full[s], bytes);
          auto load = [&](uint8_t* dst, const CUtensorMap* map, int x, int y) {
            if constexpr (TWO) tma_load_2d_pair(dst, map, x, y, lead_bar);
            else tma_load_2d(dst, map, x, y, &full[s]);
          };
          if constexpr (A_MN) {            // weights [K rows][N columns]: two blocks of 64 columns
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              if constexpr (EPI == EPI_SWIGLU)
                load(sw + j * 8192, &p.b[j][t.alloc], t.m0 + 64 * crank, erow + k0);
              else
                load(sw + j * 8192, &p.b[seg][t.alloc], t.m0 + 128 * crank + 64 * j, erow + k0);
            }
          } else {                         // weights [N rows][K columns]: 128 rows
            load(sw, &p.b2[seg][t.alloc], k0, erow + t.m0 + 128 * crank);
          }
          load(stok, tmap + seg * TG_BOXES, k0, trow);
          if (!TWO && tok > 128) load(stok + 128 * 128, tmap + seg * TG_BOXES, k0, trow + 128);
        }
      }
      if constexpr (DISP) phase_stamp(p.trace, 2, (int)blockIdx.x, 2);
    } else if (DISP && p.disp.arrive != nullptr) {
      // ---- arrival watchers (lanes 1..31): group after group, wait until every 128-row block of
      // the group has all its rows, then publish the number of complete groups to lane 0 --------
      if constexpr (DISP) {
        for (int g = 0; g < p.ngroups; ++g) {
          const int b0 = (g == 0 ? 0 : s_end[g - 1]) >> 7, b1 = s_end[g] >> 7;
          bool okw = true;
          for (int b = b0 + lane - 1; b < b1 && okw; b += 31)
            okw = arrive_wait(p.disp.arrive + b, p.disp.expect, b, abortp, p);
          if (!__all_sync(0xfffffffeu, okw)) break;
          if (lane == 1) {
            __threadfence_block();
            *(volatile int*)&s_groups_ready = g + 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (the leader issues for both CTAs of a pair) =================
    if (crank == 0) {
      const bool issue = elect_one();
      const int num_kb = p.nseg * kb_per_seg;
      // descriptors of slot 0; a slot further, and a k-step of 16, add to the address field
      const uint64_t desc_w = A_MN ? make_smem_desc(smem_u32(stages), 8192, 1024) : make_smem_desc(smem_u32(stages), 16, 1024);
      const uint64_t desc_t = make_smem_desc(smem_u32(stages) + TG_W_BYTES, 16, 1024);
      constexpr int W_STEP = (A_MN ? 2048 : 32) >> 4, T_STEP = 32 >> 4;
      RingSlot st;
      int tile_n = 0;
      bool ok = true;
      auto tokens = [&](long long id) { return __shfl_sync(0xffffffffu, id < total_tiles ? get((int)id).n : 0, 0); };
      int n = tokens(work_id0);
      for (long long id = work_id0; id < total_tiles && ok; id += work_stride, ++tile_n) {
        const uint32_t idesc = make_instr_desc_bf16(TM, n, A_MN, false);
        const int acc = tile_n & 1;
        if (!warp_wait(&acc_empty[acc], ((uint32_t)(tile_n >> 1) & 1u) ^ 1u, 2)) break;
        tc_fence_after();
        const uint32_t tacc = tmem_base + (uint32_t)acc * TG_MAX_N;
        for (int kb = 0; kb < num_kb; ++kb, st.next(NST)) {
          const int s = st.slot;
          ok = warp_wait(&full[s], st.parity, 3);
          if (!ok) break;
          tc_fence_after();
          if (issue) {
            const uint64_t da = desc_w + (uint32_t)(s * (STAGE >> 4)), db = desc_t + (uint32_t)(s * (STAGE >> 4));
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              if constexpr (TWO) umma_bf16_2cta(tacc, da + kk * W_STEP, db + kk * T_STEP, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
              else umma_bf16(tacc, da + kk * W_STEP, db + kk * T_STEP, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            }
            if constexpr (TWO) umma_commit_2cta(&empty[s], 3);
            else umma_commit(&empty[s]);
          }
          if (kb == 0) n = tokens(id + work_stride);       // (looked up while the tile is being computed)
        }
        if (!ok) break;
        if (issue) {
          if constexpr (TWO) umma_commit_2cta(&acc_full[acc], 3);
          else umma_commit(&acc_full[acc]);
        }
      }
    }
  } else if (DISP && warp >= 2 + 4 * TG_SETS) {
    // ================= fused dispatch: this CTA's share of the all-to-all =================
    if constexpr (DISP) {
      if (p.disp.x != nullptr) {
        uint8_t* ring = stages + (size_t)NST * STAGE;
        if (lane == 0) phase_stamp(p.trace, 3, (int)blockIdx.x, 0);
        fused_dispatch_copy_warp<FD_NST>(
            p.disp, ring, fd_full, (int)blockIdx.x, (int)gridDim.x,
            [&](uint64_t* bar, uint32_t parity) { return gemm_wait(bar, parity, abortp, p, 7); });
        if (lane == 0) phase_stamp(p.trace, 3, (int)blockIdx.x, 1);
      }
    }
  } else {
    // ========= epilogue: two sets of four warps, each warp one quarter of the tile's columns =========
    const int q = warp & 3;
    const int set = (warp - 2) >> 2;
    const int te = tid - 64 - set * 128;                    // 0..127
    // this set's chunks start at tokens first, first + step, ...; the thread's own token in one of them
    const int first = set * TG_CHUNK, step = TG_SETS * TG_CHUNK;
    const int my_tok = (te >> 5) * step + first + (te & 31);
    int tile_n = 0;
    // this thread's row of the matrices that its warp stores: token 8 (lane / 16) + lane % 8, columns
    // 8 (lane / 8 % 2) of the warp's quarter
    uint8_t* const sb = s_stage[set];
    const uint32_t st_addr = smem_u32(sb) +
                             (uint32_t)((8 * (lane >> 4) + (lane & 7)) * TG_STAGE_ROW + q * 64 + ((lane >> 3) & 1) * 16);
    const bool vec_ok = p.vec_out != 0;                     // outputs allow 16-byte stores
    for (long long id = work_id0; id < total_tiles; id += work_stride, ++tile_n) {
      const TokenTile t = get((int)id);
      const int acc = tile_n & 1;
      // home rows of this tile's tokens, looked up while the tile is still being computed
      if constexpr (EPI == EPI_PUSH) {
        for (int i = my_tok; i < t.n; i += 4 * step) {
          const int si = i < t.rows ? p.src_info[t.row0 + i] : -1;
          unsigned long long dptr = 0ull;
          if (si >= 0) {
            const int sr = si / p.push_entries, ent = si - sr * p.push_entries;
            if (sr < p.push_ranks)
              dptr = (unsigned long long)((__nv_bfloat16*)p.push_base + (long long)sr * p.push_rank_stride +
                                          (long long)ent * p.ldc);
          }
          s_ptr[acc][i] = dptr;
        }
      }
      const bool have = gemm_wait(&acc_full[acc], (uint32_t)(tile_n >> 1) & 1u, abortp, p, 4);
      __syncwarp();
      if (!epilogue_all(set, have)) break;      // a set's four warps leave together: they share barriers below
      tc_fence_after();
      const uint32_t tacc = tmem_base + (uint32_t)acc * TG_MAX_N + ((uint32_t)(q * 32) << 16);
      uint32_t r[32];
      auto release_acc = [&] {           // the accumulator has been read: the next tile but one may overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (TWO && crank != 0) mbar_arrive_remote(&acc_empty[acc], 0);
          else mbar_arrive(&acc_empty[acc]);
        }
      };
      if constexpr (EPI == EPI_F32) {
        // thread = output column: a warp's 32 columns of a token leave as one 128-byte line
        const int col = t.m0 + 128 * crank + q * 32 + lane;
#pragma unroll 1
        for (int c = first; c < t.n; c += step) {
          __syncwarp();
          tmem_ld_32x32(tacc + c, r);
          tmem_ld_wait();
          if (c + step >= t.n) release_acc();
          float* o = (float*)p.out[0] + (long long)(t.row0 + c) * p.ldc + col;
#pragma unroll
          for (int i = 0; i < TG_CHUNK; ++i)
            if (c + i < t.rows && col < p.N) o[i * p.ldc] = __uint_as_float(r[i]);
        }
        if (first >= t.n) release_acc();
        continue;
      }
      if (first < t.n) {
        tmem_ld_16x256_x4(tacc + first, r);
        tmem_ld_16x256_x4(tacc + first + (16u << 16), r + 16);
      } else {
        release_acc();
      }
      if constexpr (EPI == EPI_SWIGLU) {
        // (read past L1, and only now: with the fused dispatch another rank wrote the scale along with the
        // row; the first barrier below publishes it)
        for (int i = my_tok; i < t.n; i += 4 * step)
          s_scale[acc][i] = i < t.rows && p.row_scale != nullptr ? __ldcg(p.row_scale + t.row0 + i) : 1.f;
      }
#pragma unroll 1
      for (int c = first; c < t.n; c += step) {
        __syncwarp();
        tmem_ld_wait();
        uint32_t pk[16];       // [16-column half][token block][lower, upper 8 columns]
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          pk[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        if (c + step < t.n) {            // the next 32 tokens travel while these leave
          tmem_ld_16x256_x4(tacc + c + step, r);
          tmem_ld_16x256_x4(tacc + c + step + (16u << 16), r + 16);
        } else {
          release_acc();
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; j += 2)
            stmatrix_x4_trans(st_addr + (uint32_t)(j * 8 * TG_STAGE_ROW + h * 32),
                              pk[8 * h + 2 * j], pk[8 * h + 2 * j + 1], pk[8 * h + 2 * j + 2], pk[8 * h + 2 * j + 3]);
        __syncwarp();
        epilogue_sync(set);
        if constexpr (EPI == EPI_SWIGLU) {
          const int f = (te & 7) * 8, col0 = t.m0 + 64 * crank + f;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int k = (te >> 3) + 16 * i;
            if (c + k >= t.rows || col0 >= p.N) continue;
            const uint4 g4 = *reinterpret_cast<const uint4*>(sb + k * TG_STAGE_ROW + f * 2);
            const uint4 u4 = *reinterpret_cast<const uint4*>(sb + k * TG_STAGE_ROW + 128 + f * 2);
            const float rs = s_scale[acc][c + k];
            uint4 a4;
            const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&g4);
            const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&u4);
            __nv_bfloat162* a2 = reinterpret_cast<__nv_bfloat162*>(&a4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              // the saved gate/up are bf16; the activation is computed from the rounded values so that
              // backward recomputes exactly what forward used
              const float2 fg = __bfloat1622float2(g2[j]), fu = __bfloat1622float2(u2[j]);
              a2[j] = __floats2bfloat162_rn(fg.x / (1.f + __expf(-fg.x)) * fu.x * rs,
                                            fg.y / (1.f + __expf(-fg.y)) * fu.y * rs);
            }
            const long long off = (long long)(t.row0 + c + k) * p.ldc + col0;
            if (p.out[0]) store8((__nv_bfloat16*)p.out[0] + off, g4, p.N - col0, vec_ok);
            if (p.out[1]) store8((__nv_bfloat16*)p.out[1] + off, u4, p.N - col0, vec_ok);
            store8((__nv_bfloat16*)p.out[2] + off, a4, p.N - col0, vec_ok);
          }
        } else {
          const int f = (te & 15) * 8, col0 = t.m0 + 128 * crank + f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = (te >> 4) + 8 * i;
            if (c + k >= t.rows || col0 >= p.N) continue;
            const uint4 v = *reinterpret_cast<const uint4*>(sb + k * TG_STAGE_ROW + f * 2);
            if constexpr (EPI == EPI_PUSH) {
              const unsigned long long pr = s_ptr[acc][c + k];
              if (pr != 0ull) store8(reinterpret_cast<__nv_bfloat16*>(pr) + col0, v, p.N - col0, vec_ok);
            } else {
              store8((__nv_bfloat16*)p.out[0] + (long long)(t.row0 + c + k) * p.ldc + col0, v, p.N - col0, vec_ok);
            }
          }
        }
        epilogue_sync(set);              // every row of the set's buffer has been read: it may be filled again
      }
      if constexpr (EPI != EPI_PUSH) {      // padding rows that no tile computes
        constexpr int V = EPI == EPI_SWIGLU ? 8 : 16;      // vectors of this CTA's columns in a row
        const int f = (te & (V - 1)) * 8, col0 = t.m0 + V * 8 * crank + f;
        if (col0 < p.N)
          for (int r = t.row0 + t.rows + (te + 128 * set) / V; r < t.zero_to; r += 128 * TG_SETS / V) {
            const long long off = (long long)r * p.ldc + col0;
#pragma unroll
            for (int o = 0; o < (EPI == EPI_SWIGLU ? 3 : 1); ++o)
              if (p.out[o]) store8((__nv_bfloat16*)p.out[o] + off, make_uint4(0, 0, 0, 0), p.N - col0, vec_ok);
          }
      }
    }
  }
  // ---- teardown: everything joins, in-flight work is given time to land on an abort ----------
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  // Pushed rows: the home rank reads them behind a cross-rank barrier that this rank enters from a
  // LATER launch of the same stream; one fence here keeps that independent of how that launch arrives.
  if constexpr (EPI == EPI_PUSH) { if (warp >= 2) __threadfence_system(); }
  if constexpr (TWO) cluster_sync_all();        // neither CTA leaves while its peer may still touch it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (TWO) tmem_dealloc2(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace mep
