// Weight-grad GEMM (groups partition the REDUCTION dimension): D[g] (+)= A[rows of g]^T * B[rows of g], both
// operands MN-major; fp32 output (stored, or added: WG_ADD), or WG_SGD, the optimizer step fused in: the accumulator is applied
// straight to the bf16 weights, w = bf16(w - lr * acc), for every local expert that has no replica this step.
//
// A launch may compute the grads of two weights that share A (the gate and up projections): group by group, first
// one's tiles, then the other's.  That is one start and one last round of tiles instead of two, and the rows of A are
// read from memory once (a layer's step, 128 experts x 256 rows: 2048 x 768 stored 2491 -> 2464 us, 7168 x 2048 SGD 12028 ->
// 11971).
//
// What bounds it: bytes between L2 and the SMs, and the power cap.  Reads and writes together move at most 10.4 - 11.7
// TB/s (148 SMs, bulk copies of data that L2 holds beside plain stores; reads alone 12.3), and a 256 x 256 tile of
// a group of 256 rows needs 256 KB of operands beside the 256 KB of its weights or of its fp32 grad.  So
//   * CTA pairs (cta_group::2): each CTA stages its own 128 weight rows and half of the columns;
//   * where reductions are long, two tiles that are neighbours in the columns share the staged rows: a chunk of
//     the reduction for the first, then the same chunk for the second (both accumulators), 3/4 of the bytes;
//   * beside the stream of weights (SGD), loads of groups shorter than the operand slots run one tile ahead, not several
//     (a layer of 128 experts, 4096 x 1024: 1 block a group 1251 -> 1204 us, 4 blocks 1528 -> 1487);
//   * loads and MMAs are issued by converged warps with one elected lane; from a single lane's branch the issuer
//     took longer for a k-block than the tensor cores (without epilogue 32 x 1024 rows 960 -> 620 us);
//   * sixteen epilogue warps move 16-row x 64-column pieces.  The old weights come by TMA through a ring of each
//     warp's own, are updated as matrix fragments, and threads of a quad exchange words so that each holds 32
//     contiguous bytes of a row: stores cover whole 128-byte lines and pass through no shared memory.  fp32 grads
//     leave as 64-byte row segments; where they are added to grads, as 32 x 32 pieces by TMA reductions (128 groups x
//     128 rows, 4096 x 1024: 847 us; 16-byte reductions from registers 917).  (Measured and worse: a row a thread,
//     4.6 TB/s of stores where whole lines reach 6.1; two rows of 64 bytes a warp, 2.5; weights prefetched into
//     registers, 2 TB/s, because outstanding loads need L1 lines and the operand slots leave 28 KB.)
// The three weight grads of a layer's step, Zipf 0.3 - 0.5, us before (TMA both ways, single CTAs below 512 rows a group) ->
// now.  SGD: 64 experts x 256 rows, 7168 x 2048 3190 -> 2450; 128 x 256, 4096 x 1024 1875 -> 1397; 128 x 64 1166 -> 1178; 64 x 32
// rows, 7168 x 2048 2053 -> 2027.  Stored: 128 x 256, 2048 x 768 705 -> 600; 128 x 64, 4096 x 1024 1310 -> 1283.  Added: 128 x 256,
// 4096 x 1024 2727 -> 2745; 32 x 1024, 7168 x 2048 3044 -> 3144.
#pragma once

namespace mep {

enum { WG_STORE = 0, WG_SGD = 1, WG_ADD = 2 };        // what becomes of a tile (SGD: or stored, where it has replicas)
constexpr int WG_EPI_WARPS = 16;
constexpr int WG_THREADS = 64 + WG_EPI_WARPS * 32;
constexpr int WG_STEPS = 32 / WG_EPI_WARPS;           // 16-row x 64-column pieces of a tile that a warp takes
constexpr int WG_ROW_BYTES = BM * BK * 2;             // a k-block of the rows' operand, one CTA: 16 KB
template <bool TWO> __host__ __device__ constexpr int wg_col_bytes() { return (TWO ? BN / 2 : BN) * BK * 2; }
constexpr int WG_MAX_ROW_SLOTS = 7, WG_MAX_COL_SLOTS = 6;
constexpr int WG_PIECE = 16 * 64 * 2;                 // weights of an epilogue step: 16 rows x 64 columns
constexpr int WG_MAX_PIECES = WG_STEPS;
constexpr int WG_ADD_PIECE = 32 * 32 * 4;             // grads that are added to

// One tile, or two that are neighbours in the columns.
struct WgUnit {
  int g, alloc, g_local, row0, num_kb;
  int prod;            // which of the launch's products
  int m0;              // first weight row of this CTA
  int ni, tiles;       // first column tile, and their number
  bool applied;        // goes straight to the weights
};

// Walk over the units of a CTA (pair): first, first + stride, ... in the order group, product and weight rows, columns.
// A step adds the stride digit by digit.
template <bool TWO>
struct WgWalk {
  int g, mi, ui, rt, nm, nn, nu, sg, sm, su;
  __device__ __forceinline__ WgWalk(const GemmKParams& p, int first, int stride) {
    constexpr int TM = TWO ? 2 * BM : BM;
    rt = (p.Mw + TM - 1) / TM;
    nm = rt * p.products;
    nn = (p.N + BN - 1) / BN;
    nu = (nn + p.unit - 1) / p.unit;
    split(first, g, mi, ui);
    split(stride, sg, sm, su);
  }
  __device__ __forceinline__ void split(int id, int& a, int& b, int& c) const {
    a = id / (nm * nu);
    id -= a * (nm * nu);
    b = id / nu;
    c = id - b * nu;
  }
  __device__ __forceinline__ void step() {
    ui += su;
    if (ui >= nu) { ui -= nu; ++mi; }
    mi += sm;
    if (mi >= nm) { mi -= nm; ++g; }
    g += sg;
  }
  // The next unit there is work for, at or after the current position; false when there is none.
  __device__ __forceinline__ bool find(const GemmKParams& p, const int* s_end, const int* s_valid, int crank, WgUnit& t) {
    for (; g < p.ngroups; step()) {
      const int rows = __shfl_sync(0xffffffffu, s_valid[g], 0);   // padding rows are zero: blocks of nothing else are skipped
      t.g = g;
      t.alloc = g >= p.split ? 1 : 0;
      t.g_local = t.alloc ? g - p.split : g;
      t.applied = p.sgd_w[0] != nullptr && t.alloc == 0 && (p.sgd_keep == nullptr || __shfl_sync(0xffffffffu, p.sgd_keep[t.g_local], 0) == 0);
      if (g < p.g_begin || (rows <= 0 && g >= p.zero_empty_below)) continue;
      if (rows <= 0 && t.applied) continue;        // zero grad: nothing to apply
      if (p.wg_select != 0 && (p.wg_select == 2) != t.applied) continue;
      t.row0 = __shfl_sync(0xffffffffu, g == 0 ? 0 : s_end[g - 1], 0);
      t.prod = mi >= rt ? 1 : 0;
      t.m0 = (mi - t.prod * rt) * (TWO ? 2 * BM : BM) + crank * BM;
      t.ni = ui * p.unit;
      t.tiles = min(p.unit, nn - t.ni);
      t.num_kb = (rows + BK - 1) / BK;
      return true;
    }
    return false;
  }
};

// Columns that a tile computes: a multiple of 32.
__device__ __forceinline__ int wg_width(const GemmKParams& p, int ni) { return min(BN, (p.N - ni * BN + 31) & ~31); }

// The k-blocks of a unit in the order in which they are loaded and multiplied: item(tile, kb, row slot, whether
// this is its first use, whether its last).  Rows are staged in chunks of as many blocks as there are slots and
// stay for all tiles of the unit.  Stops when an item returns false.
template <class Item>
__device__ __forceinline__ bool wg_items(const WgUnit& u, int slots, RingSlot& row, Item&& item) {
  for (int k0 = 0; k0 < u.num_kb; k0 += slots) {
    const int k1 = min(u.num_kb, k0 + slots);
    RingSlot s = row;
    for (int i = 0; i < u.tiles; ++i) {
      s = row;
      for (int kb = k0; kb < k1; ++kb, s.next(slots))
        if (!item(i, kb, s, i == 0, i == u.tiles - 1)) return false;
    }
    row = s;
  }
  return true;
}

// ---- epilogue: words of a weight row among the threads of a quad -----------------------------------------
// v[k] of thread c becomes v[c] of thread k (k, c = 0..3): its own inverse.
__device__ __forceinline__ void quad_transpose(uint32_t* v, int c) {
  const bool odd = (c & 1) != 0, high = (c & 2) != 0;
  const uint32_t g0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 1);
  const uint32_t g1 = __shfl_xor_sync(0xffffffffu, odd ? v[2] : v[3], 1);
  const uint32_t a0 = odd ? g0 : v[0], a1 = odd ? v[1] : g0, b0 = odd ? g1 : v[2], b1 = odd ? v[3] : g1;
  const uint32_t h0 = __shfl_xor_sync(0xffffffffu, high ? a0 : b0, 2);
  const uint32_t h1 = __shfl_xor_sync(0xffffffffu, high ? a1 : b1, 2);
  v[0] = high ? h0 : a0;
  v[1] = high ? h1 : a1;
  v[2] = high ? b0 : h0;
  v[3] = high ? b1 : h1;
}
// Sixteen bf16 of a row, `left` before its end: 32 bytes in one access, or two of 16 where rows allow no more.
__device__ __forceinline__ void wg_store16(__nv_bfloat16* dst, int left, bool vec32, const uint32_t* r) {
  if (vec32) {
    if (left > 0)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                   ::"l"(dst), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (left > 8 * i)
        asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};"
                     ::"l"(dst + 8 * i), "r"(r[4 * i]), "r"(r[4 * i + 1]), "r"(r[4 * i + 2]), "r"(r[4 * i + 3]) : "memory");
  }
}

template <bool TWO, int MODE>
__global__ void __launch_bounds__(WG_THREADS, 1) ep_weight_grad_kernel(const __grid_constant__ GemmKParams p) {
  constexpr bool SGD = MODE == WG_SGD;
  constexpr int COL_BYTES = wg_col_bytes<TWO>();
  const int NR = p.row_slots, NC = p.col_slots;
  const int crank = TWO ? (int)cluster_cta_rank() : 0;        // 0 = leader of the pair
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t row_full[WG_MAX_ROW_SLOTS], row_empty[WG_MAX_ROW_SLOTS];
  __shared__ __align__(8) uint64_t col_full[WG_MAX_COL_SLOTS], col_empty[WG_MAX_COL_SLOTS];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t w_full[SGD ? WG_EPI_WARPS : 1][SGD ? WG_MAX_PIECES : 1];   // weight pieces of the epilogue warps
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_end[MAX_GROUPS];
  __shared__ int s_valid[MAX_GROUPS];

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  uint8_t* row_slots = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  uint8_t* col_slots = row_slots + NR * WG_ROW_BYTES;
  volatile int* abortp = &s_abort;

  if (tid == 0) {
    // pairs: both CTAs' loads count on the LEADER's full barriers, on which only its producer arrives
    for (int s = 0; s < NR; ++s) { mbar_init(&row_full[s], 1); mbar_init(&row_empty[s], 1); }
    for (int s = 0; s < NC; ++s) { mbar_init(&col_full[s], 1); mbar_init(&col_empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], WG_EPI_WARPS * (TWO ? 2 : 1)); }
    for (int e = 0; SGD && e < WG_EPI_WARPS * WG_MAX_PIECES; ++e) mbar_init(&w_full[0][0] + e, 1);
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
  __syncthreads();                           // s_valid is complete
  if constexpr (TWO) cluster_sync_all();     // the peer's barriers exist before anyone arrives on them
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;
  WgWalk<TWO> walk(p, TWO ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, TWO ? (int)(gridDim.x >> 1) : (int)gridDim.x);
  WgUnit u;

  // every lane of a warp learns the same outcome, so that a warp leaves its loops together
  auto wait = [&](uint64_t* bar, uint32_t parity, int where) {
    return __all_sync(0xffffffffu, gemm_wait(bar, parity, abortp, p, where)) != 0;
  };

  if (warp == 0) {
    // ================= TMA producer =================
    // (the whole warp walks, one lane issues: loop state and descriptors stay in uniform registers)
    const bool issue = elect_one();
    RingSlot row, col;
    if (issue) { tma_prefetch_desc(&p.a); tma_prefetch_desc(&p.b[0][0]); if (p.products > 1) tma_prefetch_desc(&p.b[1][0]); }
    for (; walk.find(p, s_end, s_valid, crank, u); walk.step()) {
      const int ahead = SGD ? max(1, min(NC, u.tiles * u.num_kb)) : NC;
      const bool ok = wg_items(u, NR, row, [&](int i, int kb, const RingSlot& rs, bool first, bool) {
        const int y = u.row0 + kb * BK;
        // blocks of 64 columns of the [token rows][columns] operands
        auto load = [&](uint8_t* dst, const CUtensorMap* map, int x, uint64_t* bar) {
          if constexpr (TWO) tma_load_2d_pair(dst, map, x, y, mapa_u32(bar, 0));
          else tma_load_2d(dst, map, x, y, bar);
        };
        if (first) {
          if (!wait(&row_empty[rs.slot], rs.parity ^ 1u, 1)) return false;
          if (issue) {
            // the peer's bytes may land before this arrival: the pending count keeps the phase open
            if (crank == 0) mbar_expect_tx(&row_full[rs.slot], WG_ROW_BYTES * (TWO ? 2 : 1));
#pragma unroll
            for (int j = 0; j < 2; ++j)
              load(row_slots + rs.slot * WG_ROW_BYTES + j * 8192, &p.a, u.m0 + 64 * j, &row_full[rs.slot]);
          }
        }
        // a block may be loaded when the one `ahead` before it has been multiplied, which is after its slot is free
        const int back = col.slot - ahead;
        if (!wait(&col_empty[back < 0 ? back + NC : back], back < 0 ? col.parity ^ 1u : col.parity, 1)) return false;
        if (issue) {
          const int n0 = (u.ni + i) * BN, mine = wg_width(p, u.ni + i) / (TWO ? 2 : 1);   // columns of this CTA
          const int blocks = (mine + 63) / 64;
          if (crank == 0) mbar_expect_tx(&col_full[col.slot], (uint32_t)(blocks * 8192 * (TWO ? 2 : 1)));
          for (int j = 0; j < blocks; ++j)
            load(col_slots + col.slot * COL_BYTES + j * 8192, &p.b[u.prod][0], n0 + crank * mine + 64 * j, &col_full[col.slot]);
        }
        col.next(NC);
        return true;
      });
      if (!ok) break;
    }
  } else if (warp == 1) {
    // ================= MMA issuer (the leader issues for both CTAs of a pair) =================
    if (crank == 0) {
      const bool issue = elect_one();
      RingSlot row, col;
      int tile0 = 0;                         // tiles before this unit
      const uint32_t rows_lo = smem_u32(row_slots) >> 4, cols_lo = smem_u32(col_slots) >> 4;
      const uint64_t desc = make_smem_desc(0, 8192, 1024);
      for (; walk.find(p, s_end, s_valid, crank, u); walk.step()) {
        // (an accumulator is empty again when the epilogue has read the tile before the last)
        auto acquire = [&](int tile_n) {
          if (!wait(&acc_empty[tile_n & 1], ((uint32_t)(tile_n >> 1) & 1u) ^ 1u, 2)) return false;
          tc_fence_after();
          return true;
        };
        auto complete = [&](int tile_n) {
          if (!issue) return;
          if constexpr (TWO) umma_commit_2cta(&acc_full[tile_n & 1], 3);
          else umma_commit(&acc_full[tile_n & 1]);
        };
        const bool ok = wg_items(u, NR, row, [&](int i, int kb, const RingSlot& rs, bool first, bool last) {
          const int tile_n = tile0 + i;
          if (kb == 0 && !acquire(tile_n)) return false;
          if (first && !wait(&row_full[rs.slot], rs.parity, 3)) return false;
          if (!wait(&col_full[col.slot], col.parity, 3)) return false;
          tc_fence_after();
          if (issue) {
            const uint32_t idesc = make_instr_desc_bf16(TWO ? 2 * BM : BM, wg_width(p, u.ni + i), true, true);
            const uint64_t da = desc | (rows_lo + rs.slot * (WG_ROW_BYTES >> 4));
            const uint64_t db = desc | (cols_lo + col.slot * (COL_BYTES >> 4));
            const uint32_t tacc = tmem_base + (uint32_t)(tile_n & 1) * BN;
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              if constexpr (TWO) umma_bf16_2cta(tacc, da + kk * 128, db + kk * 128, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
              else umma_bf16(tacc, da + kk * 128, db + kk * 128, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            }
            // slots are reusable (in both CTAs of a pair) once these MMAs have read them
            if constexpr (TWO) { umma_commit_2cta(&col_empty[col.slot], 3); if (last) umma_commit_2cta(&row_empty[rs.slot], 3); }
            else { umma_commit(&col_empty[col.slot]); if (last) umma_commit(&row_empty[rs.slot]); }
          }
          if (kb == u.num_kb - 1) complete(tile_n);
          col.next(NC);
          return true;
        });
        if (!ok) break;
        if (u.num_kb == 0) {                 // an empty group: the epilogue stores zeros
          bool more = true;
          for (int i = 0; i < u.tiles && more; ++i) {
            more = acquire(tile0 + i);
            if (more) complete(tile0 + i);
          }
          if (!more) break;
        }
        tile0 += u.tiles;
      }
    }
  } else {
    // ===== epilogue: four warps for each 64 columns of the tile, 32 rows each =====
    // in pieces of 16 rows x 64 columns, of which a thread has rows lane / 4 and lane / 4 + 8
    const int q = warp & 3, c = lane & 3;
    const bool vec32 = p.vec32 != 0;
    const int rofs = q * 32 + (lane >> 2), cofs = ((warp - 2) >> 2) * 64;
    // weight row of this thread in piece k (rows 16 k) of a tile
    auto row_of = [&](const WgUnit& t, int k) { return (long long)t.g_local * p.Mw + t.m0 + rofs + 16 * k; };
    // SGD: a warp's weight pieces travel through a ring of its own by TMA, as far ahead as the ring is deep.
    // (Loads into registers do not: with this much shared memory in use, what is left as L1 holds 28 KB of
    // outstanding loads, which streams 2 TB/s.)
    // (Grads that are added to: one piece of 32 x 32 fp32 for each of the first four warps.)
    const int ew = warp - 2, depth = p.pieces;
    uint8_t* wring = col_slots + NC * COL_BYTES + ew * (SGD ? depth * WG_PIECE : WG_ADD_PIECE);
    const uint32_t wring_s = smem_u32(wring);
    RingSlot ws;
    auto load_piece = [&](const WgUnit& t, int ni, int k, int slot) {
      if (lane == 0) {
        mbar_expect_tx(&w_full[SGD ? ew : 0][slot], WG_PIECE);
        tma_load_2d(wring + slot * WG_PIECE, &p.wmap[t.prod], ni * BN + cofs, t.g_local * p.Mw + t.m0 + q * 32 + 16 * k,
                    &w_full[SGD ? ew : 0][slot]);
      }
    };
    auto load_first = [&](const WgUnit& t, int ni) {       // of a tile that follows none which is applied
      RingSlot s = ws;
      for (int k = 0; k < depth; ++k, s.next(depth)) load_piece(t, ni, k, s.slot);
    };
    bool more = walk.find(p, s_end, s_valid, crank, u);
    int i = 0;
    if constexpr (SGD) {
      if (more && u.applied) load_first(u, u.ni);
    }
    for (int tile_n = 0; more; ++tile_n) {
      // this tile, and the next one of the walk
      const WgUnit t = u;
      const int ni = u.ni + i;
      if (++i == u.tiles) {
        walk.step();
        more = walk.find(p, s_end, s_valid, crank, u);
        i = 0;
      }
      const bool next_applied = SGD && more && u.applied;
      const int acc = tile_n & 1;
      if (!wait(&acc_full[acc], (uint32_t)(tile_n >> 1) & 1u, 4)) break;
      tc_fence_after();
      const uint32_t tacc = tmem_base + (uint32_t)acc * BN + ((uint32_t)(q * 32) << 16) + (uint32_t)cofs;
      const bool in_rows = t.m0 < p.Mw;      // (the second CTA of a pair may have no rows left)
      bool go_on = true;
      // the accumulator has been read: the next tile but one may overwrite it
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (TWO && crank != 0) mbar_arrive_remote(&acc_empty[acc], 0);   // the leader issues the MMAs
          else mbar_arrive(&acc_empty[acc]);
        }
      };
      if constexpr (MODE == WG_ADD) {
        // 32 x 32 pieces, a row a lane, added by TMA: one warp of a row quarter takes all columns
        const int steps = ew < 4 && t.num_kb > 0 ? BN / 32 : 0;
        if (steps == 0) release();
#pragma unroll 1
        for (int k = 0; k < steps; ++k) {
          uint32_t r[32];
          __syncwarp();
          tmem_ld_32x32(tacc + 32 * k, r);               // (the first four warps' columns start at 0)
          tmem_ld_wait();
          if (k == steps - 1) release();
          if (lane == 0) bulk_wait_read<0>();            // the piece before has left
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(wring + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          const int x0 = ni * BN + 32 * k;
          if (lane == 0 && in_rows && x0 < p.N) {
            tma_reduce_add_2d(&p.b2[t.prod][t.alloc], x0, t.g_local * p.Mw + t.m0 + q * 32, wring);
            bulk_commit();
          }
        }
        continue;
      }
#pragma unroll
      for (int k = 0; k < WG_STEPS; ++k) {
        uint32_t r[32];                      // column block j (of 8): [4j + 2h], [4j + 2h + 1] = columns 2c, 2c + 1 of row lane / 4 + 8h
        __syncwarp();
        if (t.num_kb > 0) {
          tmem_ld_16x256_x8(tacc + ((uint32_t)(16 * k) << 16), r);
          tmem_ld_wait();
        } else {                             // an empty group's grad is zero
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
        if (k == WG_STEPS - 1) release();
        const int col = ni * BN + cofs;
        if (SGD && t.applied) {
          if (!wait(&w_full[ew][ws.slot], ws.parity, 5)) { go_on = false; break; }
          uint32_t w[16];                    // column block j: words [2j + h]
          {
            const int row = (lane & 7) + 8 * ((lane >> 3) & 1), j0 = lane >> 4;
            const uint32_t a = wring_s + ws.slot * WG_PIECE + row * 128;
#pragma unroll
            for (int m = 0; m < 4; ++m) ldmatrix_x4(a + (((2 * m + j0) ^ (lane & 7)) << 4), w + 4 * m);
          }
          __syncwarp();
          // the slot has been read: the piece `depth` further on takes it
          if (k + depth < WG_STEPS) load_piece(t, ni, k + depth, ws.slot);
          else if (next_applied) load_piece(u, u.ni + i, k + depth - WG_STEPS, ws.slot);
          ws.next(depth);
          const float nlr = -p.sgd_lr;
          __nv_bfloat16* dst = p.sgd_w[t.prod] + row_of(t, k) * p.N + col + 16 * c;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t v[8];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                const int j = 2 * b + e;
                const uint32_t* gr = r + 4 * j + 2 * h;
                const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[2 * j + h]));
                const __nv_bfloat162 y = __floats2bfloat162_rn(__fmaf_rn(nlr, __uint_as_float(gr[0]), x.x),
                                                               __fmaf_rn(nlr, __uint_as_float(gr[1]), x.y));
                v[4 * e + b] = *reinterpret_cast<const uint32_t*>(&y);
              }
              quad_transpose(v + 4 * e, c);  // word c of the blocks 2b + e -> all words of block 2c + e
            }
            if (in_rows) wg_store16(dst + 8ll * h * p.N, p.N - col - 16 * c, vec32, v);
          }
        } else {
          // threads 2i and 2i + 1 of a quad trade: 4 contiguous columns of an even block for one, of the next
          // block for the other
          const bool odd = (c & 1) != 0;
          const int x0 = col + (odd ? 8 : 0) + 2 * (c & 2);
          float* dst = (float*)p.out[2 * t.prod + t.alloc] + row_of(t, k) * p.ldc + x0;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const uint32_t* even_b = r + 8 * b + 2 * h;
              const uint32_t* odd_b = even_b + 4;
              const uint32_t g0 = __shfl_xor_sync(0xffffffffu, odd ? even_b[0] : odd_b[0], 1);
              const uint32_t g1 = __shfl_xor_sync(0xffffffffu, odd ? even_b[1] : odd_b[1], 1);
              const uint4 v = odd ? make_uint4(g0, g1, odd_b[0], odd_b[1]) : make_uint4(even_b[0], even_b[1], g0, g1);
              float* o = dst + 8ll * h * p.ldc + 16 * b;
              // The arm that is never taken keeps this a branch.  Predicated, a piece's eight stores leave back to back at its
              // end, and groups of one and two blocks take 3 - 6 % longer (a layer's step, 128 experts, 4096 x 1024: 1
              // block 1317 against 1369 us, 2 blocks 1329 against 1424; as whole lines, two accesses a row, 1397 and 1460).
              if (in_rows && x0 + 16 * b < p.N) {
                if (p.unit < 0) asm volatile("membar.cta;" ::: "memory");
                else *reinterpret_cast<uint4*>(o) = v;
              }
            }
        }
      }
      if (!go_on) break;
      if (SGD && next_applied && !t.applied) load_first(u, u.ni + i);
    }
    if (MODE == WG_ADD && lane == 0) bulk_wait<0>();   // pieces to be added have been read and written
  }
  // ---- teardown: everything joins, in-flight work is given time to land on an abort ----------
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  if constexpr (TWO) cluster_sync_all();        // neither CTA leaves while its peer may still touch it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (TWO) tmem_dealloc2(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace mep
