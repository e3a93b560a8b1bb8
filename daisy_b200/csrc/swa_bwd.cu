// Backward pass of the sliding-window causal softmax attention (the training form,
// models/daisy/attention.py:156-162 under autograd), on tcgen05 tensor cores.
//
// With Z = scale Q K^T (masked), P = softmax(Z), O = P V and the incoming gradient dO:
//     delta_q = sum_d dO[q,d] O[q,d]        dP = dO V^T        dZ = P o (dP - delta)
//     dV = P^T dO        dK = scale dZ^T Q        dQ = scale dZ K
// P is rebuilt from the forward's per-row log2 denominators: P[q,k] = 2^(Z[q,k] log2 e - lse2[q]).
//
// No atomics: results are bitwise reproducible.  swa_bwd_kv_kernel is key block stationary and gives dK, dV, and dZ as operand
// images where there is room for them, from which swa_bwd_dq_kernel gets dQ; without that room swa_bwd_q_kernel, query block
// stationary, forms the scores again.
// All mbarrier waits are bounded (abort flag, DAISY_ETIMEOUT through the status word).
#include "common.cuh"

namespace daisy {

constexpr int WB = 128;                                   // block of queries / keys
constexpr int W_TILE = WB * DAISY_HEAD_DIM * 2;           // 32768
constexpr int W_HALF = W_TILE / 2;
constexpr int W_NST = 2;                                  // stages of streamed (Y0, Y1) tile pairs
constexpr int BWD_THREADS = 576;
constexpr int BWD_WORKERS = 512;                          // threads of warps 0-15
constexpr int BWD_SMEM = 1024 + 2 * W_TILE + W_NST * 2 * W_TILE + 256;
constexpr uint32_t DZ_KBLOCK = 128, DZ_MBLOCK = 2048;     // dZ image: bytes between groups of 8 keys, of 8 queries
static_assert(BWD_SMEM <= 232448, "over the 227 KB a CTA may use");

struct BwdParams {
  const float* lse2;        // [B,H,T]
  const float* delta;       // [B,H,T]
  const int* doc_start;     // null or [.,T], batch stride doc_sb
  int64_t doc_sb;
  __nv_bfloat16 *d0, *d1;   // outputs: dV, dK; or (unused), dQ -- [B,T,H,D] contiguous
  int T, H, B, window, window_blocks;
  float scale, scale_log2;
  int bh0, n_bh;            // the launch's (batch, head) pairs: bh0 .. bh0 + n_bh - 1
  uint8_t* tiles;           // dZ images, [n_bh][query block][tiles_row key blocks] of 32 KB
  int tiles_row;
  int* status;
};

struct BwdBars {
  uint64_t x_full, x_empty, y_full[W_NST], y_empty[W_NST], s_full[2], p_full[2], acc_full, acc_empty;
  uint32_t tmem_base;
  int abort_flag;
};

// First key block that query block `blk` sees, documents aside.
__device__ __forceinline__ int bwd_first_key_block(int blk, int window, int window_blocks) {
  if (window_blocks > 0) return max(0, blk - window_blocks + 1);
  return window > 0 ? max(0, blk * WB - window + 1) / WB : 0;
}

// Streamed block range [lo, hi] of an item: MODE 0, key block stationary; MODE 1, query block stationary.  Both say the same
// about a pair of blocks.
template <int MODE>
__device__ __forceinline__ void bwd_range(int blk, int nblk, int T, int window, int window_blocks, const int* doc_row, int& lo, int& hi) {
  if (MODE == 0) {                                         // key block blk: query blocks that can see it
    lo = blk;
    hi = nblk - 1;
    if (window_blocks > 0) hi = min(hi, blk + window_blocks - 1);
    else if (window > 0) hi = min(hi, (blk * WB + WB - 1 + window - 1) / WB);
    if (doc_row && hi > lo && doc_row[hi * WB] > blk * WB + WB - 1) {
      // later documents see none of these keys: doc_start does not decrease, so the last query block whose first row's
      // document begins at or before the last key is found by bisection (six documents of 8192 tokens under a
      // 2048-token window: the kernel 3.48 -> 2.24 ms at 8 x 8192 tokens, 16 heads)
      int a = lo, c = hi;                                  // a: visible (its own block), c: not
      while (c - a > 1) {
        const int m = (a + c) >> 1;
        if (doc_row[m * WB] > blk * WB + WB - 1) c = m; else a = m;
      }
      hi = a;
    }
  } else {                                                 // query block blk: key blocks inside its window
    hi = blk;
    lo = bwd_first_key_block(blk, window, window_blocks);
    if (doc_row) lo = max(lo, min(doc_row[blk * WB], blk * WB) / WB);  // keys before the first row's document: invisible to all
  }
}

// ---------------------------------------------------------------------------------------------
// dK, dV: key block stationary.  Item = 128 keys of one (batch, head); K_j, V_j stay in shared memory, the query blocks that can
// see them stream through.  Scores are formed TRANSPOSED, S^T = K_j Q_i^T and dP^T = V_j dO_i^T (TMEM lane = key), so P^T and
// dZ^T, rounded to bf16 and written back over them, are exactly the TMEM A operands of dV += P^T dO_i and dK += dZ^T Q_i.
//
// The four products of a tile are issued in the order
//     dV(y)  S(y+1)  dK(y)  dP(y+1)
// with dV waiting for P(y) and dK for dZ(y).  The tensor core executes one thread's products in order, so S(y+1) overwrites the
// columns of P(y), and dP(y+1) those of dZ(y), after they have been read, and whichever of P and dZ the workers rebuild, two
// products of 512 cycles run beside it.  Whole tiles of N = 128: in halves of 64 columns (the form this one replaces) a product
// reads 6 KB of shared memory in the 32 cycles it should take, at 128 bytes a cycle.
//
// 2 x 8192 x 16, window 2048: 684 us in halves -> 486 (tensor pipe 36 -> 53 % of elapsed at 1.62 GHz).  What is left is the workers'
// chain from S to P; a quarter or half of the exponentials by polynomial changed nothing.  Documents: an item's range takes five
// dependent reads, which warp 18 does an item ahead (6 documents of 8192 tokens: 737 -> 705 us a round).
//
// With a place to put them (`tiles`) the workers also leave dZ_ij as 32 KB operand images, from which swa_bwd_dq_kernel gets
// dQ_i = scale sum_j dZ_ij K_j with one product a tile instead of three and no exponentials.
//
// Roles (608 threads): warps 0-15 rebuild P / dZ -- four warpgroups, thread = TMEM lane (key), 32 of a tile's 128 columns each,
// every warpgroup writing its bf16 results over the first 16 columns of its OWN 32 -- and write the results; warp 16 TMA
// producer (Q through three stages, dO, which is spent earlier, through two); warp 17 MMA issuer; warp 18 hands out the items and
// fetches the streamed rows' scalars and each key's last query.
constexpr int KV_THREADS = 608, KV_NQ = 3, KV_NO = 2, KV_NI = 3;
struct KvBars {
  uint64_t k_full, k_empty, v_full, v_empty, q_full[KV_NQ], q_empty[KV_NQ], o_full[KV_NO], o_empty[KV_NO], c_full[2], c_empty[2], e_full, e_empty, i_full[KV_NI], i_empty[KV_NI];
  uint64_t s_full, p_full, dp_full, z_full, acc_full, acc_empty;
  int4 item[KV_NI];         // an item's block (-1: no more), (batch, head), first and last streamed block
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int KV_TILES = (2 + KV_NQ + KV_NO) * W_TILE;
constexpr int KV_SMEM = KV_TILES + 2 * 2 * WB * 4 + WB * 4 + (int)sizeof(KvBars);      // tiles, -lse2 and -delta (two stages), ends, barriers
static_assert(KV_SMEM <= 232448, "over the 227 KB a CTA may use");

// 8 x 8 transpose of 16-byte pieces, or 4 x 4, inside groups of N lanes: afterwards lane l of a group holds piece l of the
// group's rows, so that a store writes whole row segments
template <int N>
__device__ __forceinline__ void exchange_pieces(uint4 (&ch)[N], int lane) {
#pragma unroll
  for (int m = N / 2; m >= 1; m >>= 1) {
    const bool up = (lane & m) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (i & m) continue;
      const uint4 send = up ? ch[i] : ch[i | m];
      uint4 recv;
      recv.x = __shfl_xor_sync(0xffffffffu, send.x, m);
      recv.y = __shfl_xor_sync(0xffffffffu, send.y, m);
      recv.z = __shfl_xor_sync(0xffffffffu, send.z, m);
      recv.w = __shfl_xor_sync(0xffffffffu, send.w, m);
      if (up) ch[i] = recv; else ch[i | m] = recv;
    }
  }
}

template <bool STORE>
__global__ void __launch_bounds__(KV_THREADS, 1)
swa_bwd_kv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t bwd_smem_raw[];          // (no room to align the start by hand: bwd_smem_attr asks)
  uint8_t* x_tiles = bwd_smem_raw;                                   // K_j, V_j
  uint8_t* q_tiles = x_tiles + 2 * W_TILE;
  uint8_t* o_tiles = q_tiles + KV_NQ * W_TILE;
  float* col_f = reinterpret_cast<float*>(x_tiles + KV_TILES);       // [2][-lse2 | -delta][128]
  int* ends = reinterpret_cast<int*>(col_f + 2 * 2 * WB);            // each key's first query that no longer sees it
  KvBars* bars = reinterpret_cast<KvBars*>(ends + WB);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = p.T, nblk = (T + WB - 1) / WB;
  // blocks whose range is cut short by the sequence's end (the last key blocks) go last, longest first
  const int span = p.window_blocks > 0 ? p.window_blocks * WB : p.window;
  const BalancedWalk walk(nblk, p.n_bh, span > 0 ? (span + WB - 1) / WB : nblk, true);

  if (threadIdx.x == 0) {
    mbar_init(&bars->k_full, 1); mbar_init(&bars->k_empty, 1); mbar_init(&bars->v_full, 1); mbar_init(&bars->v_empty, 1);
    for (int i = 0; i < KV_NQ; ++i) { mbar_init(&bars->q_full[i], 1); mbar_init(&bars->q_empty[i], 1); }
    for (int i = 0; i < KV_NO; ++i) { mbar_init(&bars->o_full[i], 1); mbar_init(&bars->o_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->c_full[i], 1); mbar_init(&bars->c_empty[i], 16); }
    mbar_init(&bars->e_full, 1); mbar_init(&bars->e_empty, 16);
    for (int i = 0; i < KV_NI; ++i) { mbar_init(&bars->i_full[i], 1); mbar_init(&bars->i_empty[i], 18); }   // producer, issuer, workers
    mbar_init(&bars->s_full, 1); mbar_init(&bars->p_full, 16); mbar_init(&bars->dp_full, 1); mbar_init(&bars->z_full, 16);
    mbar_init(&bars->acc_full, 1); mbar_init(&bars->acc_empty, 16);
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 17) { tmem_alloc(&bars->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_launch();
  grid_dep_wait();

  // the it-th item as warp 18 published it: false when there are no more, or a wait ran out
  auto next_item = [&](uint32_t it, int4& item) -> bool {
    const uint32_t s = it % KV_NI;
    if (!__all_sync(0xffffffffu, mbar_wait(&bars->i_full[s], (it / KV_NI) & 1, abort_flag, p.status, 10))) return false;
    item = bars->item[s];
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars->i_empty[s]);
    return item.x >= 0;
  };

  if (warp == 16) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) { prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do); }
    uint32_t n = 0;
    bool ok = true;
    int4 item;
    for (uint32_t it = 0; ok && next_item(it, item); ++it) {
      const int blk = item.x, h = item.y % p.H, b = item.y / p.H, lo = item.z, hi = item.w;
      if (lane == 0) {
        auto tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int y) {
          mbar_expect_tx(bar, W_TILE);
          tma_load_4d(dst, tm, bar, 0, y * WB, h, b);
          tma_load_4d(dst + W_HALF, tm, bar, 64, y * WB, h, b);
        };
        // K_j is free after the previous item's last S, V_j after its last dP: both come while that item ends
        ok = mbar_wait(&bars->k_empty, (it & 1) ^ 1, abort_flag, p.status, 1);
        if (ok) tile(x_tiles, &tm_k, &bars->k_full, blk);
        for (int y = lo; ok && y <= hi; ++y, ++n) {
          const int sq = n % KV_NQ, so = n % KV_NO;
          if (!(ok = mbar_wait(&bars->q_empty[sq], ((n / KV_NQ) & 1) ^ 1, abort_flag, p.status, 2))) break;
          tile(q_tiles + sq * W_TILE, &tm_q, &bars->q_full[sq], y);
          if (y == lo) {
            if (!(ok = mbar_wait(&bars->v_empty, (it & 1) ^ 1, abort_flag, p.status, 1))) break;
            tile(x_tiles + W_TILE, &tm_v, &bars->v_full, blk);
          }
          if (!(ok = mbar_wait(&bars->o_empty[so], ((n / KV_NO) & 1) ^ 1, abort_flag, p.status, 2))) break;
          tile(o_tiles + so * W_TILE, &tm_do, &bars->o_full[so], y);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc_s = umma_idesc_bf16(WB, WB, 0, 0);                   // X Y^T: both K-major
    constexpr uint32_t idesc_a = umma_idesc_bf16(WB, DAISY_HEAD_DIM, 0, 1);       // (P | dZ from TMEM) x Y: Y as an MN-major operand
    const uint64_t xd = umma_desc_sw128(smem_u32(x_tiles), 16, 1024), ymn = umma_desc_sw128(smem_u32(q_tiles), W_HALF, 1024);
    const uint32_t x_lo = (uint32_t)xd, k_hi = (uint32_t)(xd >> 32), mn_hi = (uint32_t)(ymn >> 32);
    const uint32_t q_lo = (uint32_t)umma_desc_sw128(smem_u32(q_tiles), 16, 1024), o_lo = (uint32_t)umma_desc_sw128(smem_u32(o_tiles), 16, 1024);
    const uint32_t qmn_lo = (uint32_t)ymn, omn_lo = (uint32_t)umma_desc_sw128(smem_u32(o_tiles), W_HALF, 1024);
    const uint32_t s_t = tmem_base, dp_t = tmem_base + 128, dv_t = tmem_base + 256, dk_t = tmem_base + 384;
    auto score = [&](uint32_t d, uint32_t x, uint32_t y) {
#pragma unroll
      for (int k = 0; k < DAISY_HEAD_DIM / 16; ++k) {
        const uint32_t off = ((k >> 2) * W_HALF + (k & 3) * 32) >> 4;
        umma_ss_lh_p(leader, d, x + off, k_hi, y + off, k_hi, idesc_s, k > 0 ? 1u : 0u);
      }
    };
    auto accumulate = [&](uint32_t d, uint32_t a, uint32_t y, uint32_t acc) {
#pragma unroll
      for (int k = 0; k < WB / 16; ++k)
        umma_ts_lh_p(leader, d, a + (k & 1) * 8 + (k >> 1) * 32, y + k * (2048 >> 4), mn_hi, idesc_a, (acc || k > 0) ? 1u : 0u);
    };
    uint32_t n = 0;
    bool ok = true;
    int4 item;
    for (uint32_t it = 0; ok && next_item(it, item); ++it) {
      const int lo = item.z, hi = item.w;
      if (!mbar_wait(&bars->k_full, it & 1, abort_flag, p.status, 3)) break;
      if (!mbar_wait(&bars->q_full[n % KV_NQ], (n / KV_NQ) & 1, abort_flag, p.status, 4)) break;
      tc_fence_after();
      score(s_t, x_lo, q_lo + (n % KV_NQ) * (W_TILE >> 4));
      tc_commit_p(leader, &bars->s_full);
      if (lo == hi) tc_commit_p(leader, &bars->k_empty);
      if (!mbar_wait(&bars->v_full, it & 1, abort_flag, p.status, 3)) break;
      if (!mbar_wait(&bars->o_full[n % KV_NO], (n / KV_NO) & 1, abort_flag, p.status, 4)) break;
      tc_fence_after();
      score(dp_t, x_lo + (W_TILE >> 4), o_lo + (n % KV_NO) * (W_TILE >> 4));
      tc_commit_p(leader, &bars->dp_full);
      if (lo == hi) tc_commit_p(leader, &bars->v_empty);
      // the first accumulating products overwrite the accumulators: the workers have read out the previous item's
      if (!mbar_wait(&bars->acc_empty, (it & 1) ^ 1, abort_flag, p.status, 8)) break;
      for (int y = lo; y <= hi; ++y, ++n) {
        const uint32_t sq = n % KV_NQ, so = n % KV_NO, sq1 = (n + 1) % KV_NQ, so1 = (n + 1) % KV_NO;
        const bool more = y < hi;
        if (!mbar_wait(&bars->p_full, n & 1, abort_flag, p.status, 5)) { ok = false; break; }
        tc_fence_after();
        accumulate(dv_t, s_t, omn_lo + so * (W_TILE >> 4), y > lo);               // dV += P^T dO
        tc_commit_p(leader, &bars->o_empty[so]);
        if (more) {
          if (!mbar_wait(&bars->q_full[sq1], ((n + 1) / KV_NQ) & 1, abort_flag, p.status, 4)) { ok = false; break; }
          tc_fence_after();
          score(s_t, x_lo, q_lo + sq1 * (W_TILE >> 4));
          tc_commit_p(leader, &bars->s_full);
          if (y + 1 == hi) tc_commit_p(leader, &bars->k_empty);
        }
        if (!mbar_wait(&bars->z_full, n & 1, abort_flag, p.status, 5)) { ok = false; break; }
        tc_fence_after();
        accumulate(dk_t, dp_t, qmn_lo + sq * (W_TILE >> 4), y > lo);              // dK += dZ^T Q
        tc_commit_p(leader, &bars->q_empty[sq]);
        if (more) {
          if (!mbar_wait(&bars->o_full[so1], ((n + 1) / KV_NO) & 1, abort_flag, p.status, 4)) { ok = false; break; }
          tc_fence_after();
          score(dp_t, x_lo + (W_TILE >> 4), o_lo + so1 * (W_TILE >> 4));
          tc_commit_p(leader, &bars->dp_full);
          if (y + 1 == hi) tc_commit_p(leader, &bars->v_empty);
        } else {
          tc_commit_p(leader, &bars->acc_full);
        }
      }
    }
  } else if (warp == 18) {
    // ------------------------------------------------------------------ items, one ahead; scalars: four keys and four streamed queries a lane
    uint32_t n = 0;
    bool ok = true;
    int4 item;
    int end[4];
    auto publish = [&](uint32_t it) -> bool {                         // item `it` and its keys' ends
      const int at = walk.at((int)it);
      item = make_int4(at < 0 ? -1 : at % nblk, at < 0 ? 0 : p.bh0 + at / nblk, 0, 0);
      const int* doc_row = p.doc_start ? p.doc_start + item.y / p.H * p.doc_sb : nullptr;
      if (at >= 0) bwd_range<0>(item.x, nblk, T, p.window, p.window_blocks, doc_row, item.z, item.w);
      const uint32_t s = it % KV_NI;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->i_empty[s], ((it / KV_NI) & 1) ^ 1, abort_flag, p.status, 9))) return false;
      if (lane == 0) { bars->item[s] = item; mbar_arrive(&bars->i_full[s]); }
      if (at < 0) return true;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = item.x * WB + lane + 32 * e;
        int c = min(T, (item.w + 1) * WB);
        if (p.window_blocks <= 0 && p.window > 0) c = min(c, k + min(p.window, T));
        if (doc_row) {                                                // doc_start does not decrease: bisect for the first query of a later document
          int a = k + 1;
          while (a < c) {
            const int m = (a + c) >> 1;
            if (__ldg(doc_row + m) > k) c = m; else a = m + 1;
          }
        }
        end[e] = k < T ? c : 0;
      }
      return true;
    };
    ok = publish(0);
    for (uint32_t it = 0; ok && item.x >= 0; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->e_empty, (it & 1) ^ 1, abort_flag, p.status, 9));
      if (!ok) break;
#pragma unroll
      for (int e = 0; e < 4; ++e) ends[lane + 32 * e] = end[e];
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->e_full);
      const float *lse = p.lse2 + (int64_t)item.y * T, *delta = p.delta + (int64_t)item.y * T;
      const int lo = item.z, hi = item.w;
      for (int y = lo; y <= hi; ++y, ++n) {
        float l[4], d[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = y * WB + lane + 32 * e;
          l[e] = q < T ? -__ldg(lse + q) : 0.f; d[e] = q < T ? -__ldg(delta + q) : 0.f;
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->c_empty[n & 1], ((n >> 1) & 1) ^ 1, abort_flag, p.status, 9));
        if (!ok) break;
        float* cf = col_f + (n & 1) * 2 * WB;
#pragma unroll
        for (int e = 0; e < 4; ++e) { cf[lane + 32 * e] = l[e]; cf[WB + lane + 32 * e] = d[e]; }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->c_full[n & 1]);
        if (y == lo && !(ok = publish(it + 1))) break;                // in the shadow of this item
      }
    }
  } else {
    // ------------------------------------------------------------------ P / dZ rebuild and epilogue: thread = TMEM lane = key
    const int grp = warp >> 2, quarter = warp & 3;                    // which 32 columns; which 32 TMEM lanes
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_t = tmem_base + lane_off + 32 * grp, dp_t = s_t + 128;        // this thread's 32 S and 32 dP columns
    const uint32_t a0_t = tmem_base + lane_off + 256 + 32 * grp, a1_t = a0_t + 128;    // and its 32 output columns of each accumulator
    const uint64_t c2 = pack2f(p.scale_log2, p.scale_log2);
    uint32_t n = 0;
    bool ok = true;
    int4 item;
    for (uint32_t it = 0; ok && next_item(it, item); ++it) {
      const int blk = item.x, h = item.y % p.H, b = item.y / p.H, lo = item.z, hi = item.w;
      const int k = blk * WB + row;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->e_full, it & 1, abort_flag, p.status, 6));
      if (!ok) break;
      const int end = ends[row], first_end = ends[0];                 // ends do not decrease with the key
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->e_empty);
      for (int y = lo; y <= hi; ++y, ++n) {
        const float* cf = col_f + (n & 1) * 2 * WB + 32 * grp;
        const int y0 = y * WB;
        // is every (key, query) pair of this tile visible?
        const bool full = blk * WB + WB - 1 <= y0 && y0 + WB <= first_end;
        // and which of this thread's 32: queries k .. end - 1
        const int v_lo = min(max(k - y0 - 32 * grp, 0), 32), v_hi = min(max(end - y0 - 32 * grp, 0), 32);
        const uint32_t visible = (uint32_t)(((uint64_t)1 << v_hi) - 1) & ~(uint32_t)(((uint64_t)1 << v_lo) - 1);
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->c_full[n & 1], (n >> 1) & 1, abort_flag, p.status, 6) &&
                                     mbar_wait(&bars->s_full, n & 1, abort_flag, p.status, 6));
        if (!ok) break;
        tc_fence_after();
        uint64_t pv[16];                                              // P, fp32 pairs
        {
          uint32_t r[32], pp[16];
          tmem_ld32(s_t, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float l[4];
            *reinterpret_cast<float4*>(l) = *reinterpret_cast<const float4*>(cf + i);
            float x[4];
            unpack2f(ffma2(pack2f(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), c2, pack2f(l[0], l[1])), x[0], x[1]);
            unpack2f(ffma2(pack2f(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), c2, pack2f(l[2], l[3])), x[2], x[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = fast_exp2(x[e]);
            if (!full) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (!((visible >> (i + e)) & 1u)) x[e] = 0.f;
            }
            pp[i >> 1] = pack_bf16(x[0], x[1]); pp[(i >> 1) + 1] = pack_bf16(x[2], x[3]);
            pv[i >> 1] = pack2f(x[0], x[1]); pv[(i >> 1) + 1] = pack2f(x[2], x[3]);
          }
          tmem_st16(s_t, pp);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full);
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->dp_full, n & 1, abort_flag, p.status, 6));
        if (!ok) break;
        tc_fence_after();
        uint32_t pz[16];
        {
          uint32_t r[32];
          tmem_ld32(dp_t, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float d[4], z[4];
            *reinterpret_cast<float4*>(d) = *reinterpret_cast<const float4*>(cf + WB + i);
            unpack2f(fmul2(pv[i >> 1], fadd2(pack2f(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), pack2f(d[0], d[1]))), z[0], z[1]);
            unpack2f(fmul2(pv[(i >> 1) + 1], fadd2(pack2f(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), pack2f(d[2], d[3]))), z[2], z[3]);
            pz[i >> 1] = pack_bf16(z[0], z[1]); pz[(i >> 1) + 1] = pack_bf16(z[2], z[3]);
          }
          tmem_st16(dp_t, pz);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&bars->z_full); mbar_arrive(&bars->c_empty[n & 1]); }
        if (STORE) {
          uint8_t* dst = p.tiles + ((int64_t)((item.y - p.bh0) * nblk + y) * p.tiles_row + blk - bwd_first_key_block(y, p.window, p.window_blocks)) * W_TILE +
                         grp * 4 * DZ_MBLOCK + row * 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(dst + j * DZ_MBLOCK) = make_uint4(pz[4 * j], pz[4 * j + 1], pz[4 * j + 2], pz[4 * j + 3]);
        }
      }
      // ---- epilogue: the item's accumulators -> global rows, 64 bytes of eight rows a store
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, it & 1, abort_flag, p.status, 7));
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const float sc = which == 0 ? 1.f : p.scale;
        uint32_t r[32];
        tmem_ld32(which == 0 ? a0_t : a1_t, r);
        tc_wait_ld();
        if (which == 1) {                                             // the next item's first accumulating products overwrite what was just read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty);
        }
        uint4 ch[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * i + e]) * sc;
          ch[i] = pack8(f);
        }
        exchange_pieces(ch, lane);
        const int k0 = k & ~3;
        __nv_bfloat16* dst = (which == 0 ? p.d0 : p.d1) + (((int64_t)b * T + k0) * p.H + h) * DAISY_HEAD_DIM + 32 * grp + 8 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (k0 + i < T) *reinterpret_cast<uint4*>(dst + (int64_t)i * p.H * DAISY_HEAD_DIM) = ch[i];
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 17) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ---------------------------------------------------------------------------------------------
// dQ_i = scale sum_j dZ_ij K_j from the images swa_bwd_kv_kernel left: a banded product that reads each image once.  Item = 128
// queries of one (batch, head).  Warps 0-3 write the results out of one of two accumulators, warp 4 keeps three stages of
// (dZ_ij, K_j) full, warp 5 issues.  The images are read as MN-major operands without a swizzle: core matrices of 8 keys x 8
// queries in 128 contiguous bytes, which is also how 32 lanes (keys) write 512 contiguous bytes at a time.
// HBM-bound: 6.5 TB/s of the images.  2 x 8192 x 16, window 2048: 176 us, where forming the scores again takes 408.
constexpr int DQ_THREADS = 192, DQ_NST = 3;
struct DqBars {
  uint64_t full[DQ_NST], empty[DQ_NST], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int DQ_SMEM = 1024 + DQ_NST * 2 * W_TILE + (int)sizeof(DqBars);

__global__ void __launch_bounds__(DQ_THREADS, 1) swa_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_k, const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t bwd_smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(bwd_smem_raw) + 1023) & ~uintptr_t(1023));
  DqBars* bars = reinterpret_cast<DqBars*>(stages + DQ_NST * 2 * W_TILE);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = p.T, nblk = (T + WB - 1) / WB;
  const int span = p.window_blocks > 0 ? p.window_blocks * WB : p.window;
  const BalancedWalk walk(nblk, p.n_bh, span > 0 ? (span + WB - 1) / WB : nblk, false);

  if (threadIdx.x == 0) {
    for (int i = 0; i < DQ_NST; ++i) { mbar_init(&bars->full[i], 1); mbar_init(&bars->empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->acc_full[i], 1); mbar_init(&bars->acc_empty[i], 4); }
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 5) { tmem_alloc(&bars->tmem_base, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_launch();
  grid_dep_wait();

  if (warp == 4) {
    if (lane == 0) {
      prefetch_tmap(&tm_k);
      uint32_t n = 0, it = 0;
      bool ok = true;
      for (int item; (item = walk.at((int)it)) >= 0 && ok; ++it) {
        const int blk = item % nblk, bh = p.bh0 + item / nblk, h = bh % p.H, b = bh / p.H;
        int lo, hi;
        bwd_range<1>(blk, nblk, T, p.window, p.window_blocks, p.doc_start ? p.doc_start + b * p.doc_sb : nullptr, lo, hi);
        const uint8_t* row = p.tiles + ((int64_t)item * p.tiles_row - bwd_first_key_block(blk, p.window, p.window_blocks)) * W_TILE;
        for (int y = lo; y <= hi; ++y, ++n) {
          const int st = n % DQ_NST;
          if (!mbar_wait(&bars->empty[st], ((n / DQ_NST) & 1) ^ 1, abort_flag, p.status, 2)) { ok = false; break; }
          uint8_t* dst = stages + st * 2 * W_TILE;
          mbar_expect_tx(&bars->full[st], 2 * W_TILE);
          asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(smem_u32(dst)), "l"(row + (int64_t)y * W_TILE), "r"(W_TILE), "r"(smem_u32(&bars->full[st])) : "memory");
          tma_load_4d(dst + W_TILE, &tm_k, &bars->full[st], 0, y * WB, h, b);
          tma_load_4d(dst + W_TILE + W_HALF, &tm_k, &bars->full[st], 64, y * WB, h, b);
        }
      }
    }
  } else if (warp == 5) {
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = umma_idesc_bf16(WB, DAISY_HEAD_DIM, 1, 1);         // both MN-major
    const uint64_t zd = umma_desc_plain(smem_u32(stages), DZ_KBLOCK, DZ_MBLOCK), kd = umma_desc_sw128(smem_u32(stages) + W_TILE, W_HALF, 1024);
    const uint32_t z_hi = (uint32_t)(zd >> 32), k_hi = (uint32_t)(kd >> 32);
    uint32_t n = 0, it = 0;
    bool ok = true;
    for (int item; (item = walk.at((int)it)) >= 0 && ok; ++it) {
      const int blk = item % nblk, b = (p.bh0 + item / nblk) / p.H;
      int lo, hi;
      bwd_range<1>(blk, nblk, T, p.window, p.window_blocks, p.doc_start ? p.doc_start + b * p.doc_sb : nullptr, lo, hi);
      if (!mbar_wait(&bars->acc_empty[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 8)) break;
      for (int y = lo; y <= hi; ++y, ++n) {
        const uint32_t st = n % DQ_NST, off = st * ((2 * W_TILE) >> 4);
        if (!mbar_wait(&bars->full[st], (n / DQ_NST) & 1, abort_flag, p.status, 4)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < WB / 16; ++k)
          umma_ss_lh_p(leader, tmem_base + 128 * (it & 1), (uint32_t)zd + off + k * ((2 * DZ_KBLOCK) >> 4), z_hi, (uint32_t)kd + off + k * (2048 >> 4), k_hi,
                       idesc, (y > lo || k > 0) ? 1u : 0u);
        tc_commit_p(leader, &bars->empty[st]);
      }
      if (ok) tc_commit_p(leader, &bars->acc_full[it & 1]);
    }
  } else {
    const int row = 32 * warp + lane;
    uint32_t it = 0;
    for (int item; (item = walk.at((int)it)) >= 0; ++it) {
      const int blk = item % nblk, bh = p.bh0 + item / nblk, h = bh % p.H, b = bh / p.H;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->acc_full[it & 1], (it >> 1) & 1, abort_flag, p.status, 7))) break;
      tc_fence_after();
      const int q0 = blk * WB + (row & ~7);
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t r[64];
        tmem_ld32(tmem_base + ((uint32_t)(32 * warp) << 16) + 128 * (it & 1) + 64 * half, r);
        tmem_ld32(tmem_base + ((uint32_t)(32 * warp) << 16) + 128 * (it & 1) + 64 * half + 32, r + 32);
        tc_wait_ld();
        if (half == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty[it & 1]);
        }
        uint4 ch[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * i + e]) * p.scale;
          ch[i] = pack8(f);
        }
        exchange_pieces(ch, lane);
        __nv_bfloat16* dst = p.d1 + (((int64_t)b * T + q0) * p.H + h) * DAISY_HEAD_DIM + 64 * half + 8 * (lane & 7);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (q0 + i < T) *reinterpret_cast<uint4*>(dst + (int64_t)i * p.H * DAISY_HEAD_DIM) = ch[i];
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

// ---------------------------------------------------------------------------------------------
// dQ without the images: query block stationary.  Item = 128 queries; Q_i, dO_i stay, the key blocks of the window stream (K_j,
// V_j);  S = Q_i K_j^T, dP = dO_i V_j^T (TMEM lane = query),  dQ += dZ K_j.  576 threads: warps 0-15 rebuild dZ (four
// warpgroups, thread = TMEM lane, 32 of a tile's 128 columns each) and write the results; warp 16 TMA producer, warp 17 MMA
// issuer.  TMEM: S [0,128) dP [128,256) dQ [384,512).
__global__ void __launch_bounds__(BWD_THREADS, 1)
swa_bwd_q_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t bwd_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(bwd_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x_tiles = smem;                                           // X0, X1
  uint8_t* y_tiles = smem + 2 * W_TILE;                              // per stage: Y0, Y1
  BwdBars* bars = reinterpret_cast<BwdBars*>(y_tiles + W_NST * 2 * W_TILE);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = p.T, nblk = (T + WB - 1) / WB;
  // blocks whose range is cut short by the sequence's start (the first query blocks) go last, longest first
  const int span = p.window_blocks > 0 ? p.window_blocks * WB : p.window;
  const BalancedWalk walk(nblk, p.H * p.B, span > 0 ? (span + WB - 1) / WB : nblk, false);
  const CUtensorMap *tx0 = &tm_q, *tx1 = &tm_do, *ty0 = &tm_k, *ty1 = &tm_v;

  if (threadIdx.x == 0) {
    mbar_init(&bars->x_full, 1); mbar_init(&bars->x_empty, 1);
    for (int i = 0; i < W_NST; ++i) { mbar_init(&bars->y_full[i], 1); mbar_init(&bars->y_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_full[i], BWD_WORKERS / 2); }
    mbar_init(&bars->acc_full, 1); mbar_init(&bars->acc_empty, BWD_WORKERS);
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 17) { tmem_alloc(&bars->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_launch();
  grid_dep_wait();

  if (warp == 16) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do);
      uint32_t n = 0, it = 0;
      bool ok = true;
      for (int item; (item = walk.at((int)it)) >= 0 && ok; ++it) {
        const int blk = item % nblk, bh = item / nblk, h = bh % p.H, b = bh / p.H;
        int lo, hi;
        bwd_range<1>(blk, nblk, T, p.window, p.window_blocks, p.doc_start ? p.doc_start + b * p.doc_sb : nullptr, lo, hi);
        if (!mbar_wait(&bars->x_empty, (it & 1) ^ 1, abort_flag, p.status, 1)) { ok = false; break; }
        mbar_expect_tx(&bars->x_full, 2 * W_TILE);
        tma_load_4d(x_tiles, tx0, &bars->x_full, 0, blk * WB, h, b);
        tma_load_4d(x_tiles + W_HALF, tx0, &bars->x_full, 64, blk * WB, h, b);
        tma_load_4d(x_tiles + W_TILE, tx1, &bars->x_full, 0, blk * WB, h, b);
        tma_load_4d(x_tiles + W_TILE + W_HALF, tx1, &bars->x_full, 64, blk * WB, h, b);
        for (int y = lo; y <= hi && ok; ++y, ++n) {
          const int st = n % W_NST;
          if (!mbar_wait(&bars->y_empty[st], ((n / W_NST) & 1) ^ 1, abort_flag, p.status, 2)) { ok = false; break; }
          uint8_t* dst = y_tiles + st * 2 * W_TILE;
          mbar_expect_tx(&bars->y_full[st], 2 * W_TILE);
          tma_load_4d(dst, ty0, &bars->y_full[st], 0, y * WB, h, b);
          tma_load_4d(dst + W_HALF, ty0, &bars->y_full[st], 64, y * WB, h, b);
          tma_load_4d(dst + W_TILE, ty1, &bars->y_full[st], 0, y * WB, h, b);
          tma_load_4d(dst + W_TILE + W_HALF, ty1, &bars->y_full[st], 64, y * WB, h, b);
        }
      }
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------------ MMA issuer
    // The score tiles are formed and consumed in two halves of 64 streamed rows (= 64 TMEM columns), two worker
    // warpgroups each, and the halves are software-pipelined: while the warpgroups of a half rebuild its dZ, the tensor core
    // forms the other half's scores, accumulates the previous half's products and already forms the NEXT tile's
    // scores of a half as soon as that half's columns have been consumed:
    //   S0(y) S1(y) | wait dZ0(y): A0(y) S0(y+1) | wait dZ1(y): A1(y) S1(y+1) | wait dZ0(y+1): ...
    // (S = both score products of a half, A = the accumulating product).  tcgen05 MMAs of one thread execute in
    // order, so S_h(y+1) overwrites columns that A_h(y) has finished reading.
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc_s = umma_idesc_bf16(WB, WB / 2, 0, 0);               // X Y_half^T: both K-major, 64 streamed rows
    constexpr uint32_t idesc_a = umma_idesc_bf16(WB, DAISY_HEAD_DIM, 0, 1);       // dZ (from TMEM) x Y: Y as an MN-major operand
    const uint64_t xd = umma_desc_sw128(smem_u32(x_tiles), 16, 1024);
    const uint64_t yd = umma_desc_sw128(smem_u32(y_tiles), 16, 1024);
    const uint64_t ymn = umma_desc_sw128(smem_u32(y_tiles), W_HALF, 1024);
    const uint32_t x_lo0 = (uint32_t)xd, y_lo0 = (uint32_t)yd, k_hi = (uint32_t)(xd >> 32);
    const uint32_t ymn_lo0 = (uint32_t)ymn, ymn_hi = (uint32_t)(ymn >> 32);
    const uint32_t s_t = tmem_base, dp_t = tmem_base + 128, a1_t = tmem_base + 384;
    uint32_t n = 0, it = 0;
    bool ok = true;
    // both score products of half hf of the tile in stage st
    auto scores = [&](int st, int hf) {
      const uint32_t y0 = y_lo0 + st * ((2 * W_TILE) >> 4) + hf * ((64 * 128) >> 4), y1 = y0 + (W_TILE >> 4);
#pragma unroll
      for (int k = 0; k < DAISY_HEAD_DIM / 16; ++k) {                            // S = X0 Y0^T
        const uint32_t off = ((k >> 2) * W_HALF + (k & 3) * 32) >> 4;
        umma_ss_lh_p(leader, s_t + 64 * hf, x_lo0 + off, k_hi, y0 + off, k_hi, idesc_s, k > 0 ? 1u : 0u);
      }
#pragma unroll
      for (int k = 0; k < DAISY_HEAD_DIM / 16; ++k) {                            // dP = X1 Y1^T
        const uint32_t off = ((k >> 2) * W_HALF + (k & 3) * 32) >> 4;
        umma_ss_lh_p(leader, dp_t + 64 * hf, x_lo0 + (W_TILE >> 4) + off, k_hi, y1 + off, k_hi, idesc_s, k > 0 ? 1u : 0u);
      }
      tc_commit_p(leader, &bars->s_full[hf]);
    };
    // the accumulating product over the 64 streamed rows of half hf
    auto accumulate = [&](int st, int hf, uint32_t acc) {
      const uint32_t ymn0 = ymn_lo0 + st * ((2 * W_TILE) >> 4);
#pragma unroll
      for (int k = 4 * hf; k < 4 * hf + 4; ++k)                                 // dQ += dZ K
        umma_ts_lh_p(leader, a1_t, dp_t + (k & 1) * 8 + (k >> 1) * 32, ymn0 + k * (2048 >> 4), ymn_hi, idesc_a, (acc || k > 4 * hf) ? 1u : 0u);
    };
    for (int item; (item = walk.at((int)it)) >= 0 && ok; ++it) {
      const int blk = item % nblk, bh = item / nblk, b = bh / p.H;
      int lo, hi;
      bwd_range<1>(blk, nblk, T, p.window, p.window_blocks, p.doc_start ? p.doc_start + b * p.doc_sb : nullptr, lo, hi);
      if (!mbar_wait(&bars->x_full, it & 1, abort_flag, p.status, 3)) { ok = false; break; }
      // the item's first tile
      if (!mbar_wait(&bars->y_full[n % W_NST], (n / W_NST) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      scores(n % W_NST, 0);
      scores(n % W_NST, 1);
      // its first accumulating products overwrite the accumulators: the workers have read out the previous item's
      if (!mbar_wait(&bars->acc_empty, (it & 1) ^ 1, abort_flag, p.status, 8)) { ok = false; break; }
      for (int y = lo; y <= hi && ok; ++y, ++n) {
        const int st = n % W_NST, st_next = (n + 1) % W_NST;
        const bool more = y < hi;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          if (!mbar_wait(&bars->p_full[hf], n & 1, abort_flag, p.status, 5)) { ok = false; break; }
          tc_fence_after();
          accumulate(st, hf, (y == lo && hf == 0) ? 0u : 1u);
          if (hf == 1) tc_commit_p(leader, &bars->y_empty[st]);
          if (more) {
            if (hf == 0) {
              if (!mbar_wait(&bars->y_full[st_next], ((n + 1) / W_NST) & 1, abort_flag, p.status, 4)) { ok = false; break; }
              tc_fence_after();
            }
            scores(st_next, hf);
          }
        }
        if (ok && y == hi) { tc_commit_p(leader, &bars->acc_full); tc_commit_p(leader, &bars->x_empty); }
      }
    }
  } else {
    // ------------------------------------------------------------------ dZ rebuild and epilogue: thread = TMEM lane
    const int grp = warp >> 2, quarter = warp & 3;                    // which 32 columns; which 32 TMEM lanes
    const int half = grp >> 1;                                        // the 64-column half whose barriers this warpgroup uses
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_t = tmem_base + lane_off + 32 * grp, dp_t = s_t + 128;        // this thread's 32 S and 32 dP columns
    const uint32_t a1_t = tmem_base + lane_off + 384 + 32 * grp;                    // and its 32 output columns
    const float c2 = p.scale_log2;
    uint32_t n = 0, it = 0;
    bool ok = true;
    for (int item; (item = walk.at((int)it)) >= 0 && ok; ++it) {
      const int blk = item % nblk, bh = item / nblk, h = bh % p.H, b = bh / p.H;
      const int* doc_row = p.doc_start ? p.doc_start + b * p.doc_sb : nullptr;
      int lo, hi;
      bwd_range<1>(blk, nblk, T, p.window, p.window_blocks, doc_row, lo, hi);
      const int64_t rowbase = ((int64_t)b * p.H + h) * T;
      const int xr = blk * WB + row;                                  // this lane's query
      float my_lse = 0.f, my_delta = 0.f;
      int my_doc = 0;
      if (xr < T) {
        my_lse = p.lse2[rowbase + xr]; my_delta = p.delta[rowbase + xr];
        my_doc = doc_row ? min(doc_row[xr], xr) : 0;
      }
      for (int y = lo; y <= hi; ++y, ++n) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[half], n & 1, abort_flag, p.status, 6));
        if (!ok) break;
        tc_fence_after();
        const int y0 = y * WB;
        // is every (lane, column) pair of this tile pair visible?
        const bool full = (y0 + WB - 1 <= blk * WB) && (p.window_blocks > 0 || p.window <= 0 || blk * WB + WB - 1 - y0 < p.window) &&
                          (!doc_row || doc_row[min(blk * WB + WB - 1, T - 1)] <= y0);
        {                                                             // the results go back over the first 16 of the 32 columns
          uint32_t rs[32], rd[32];
          tmem_ld32(s_t, rs);
          tmem_ld32(dp_t, rd);
          tc_wait_ld();
          uint32_t pz[16];
          const uint64_t nl = pack2f(-my_lse, -my_lse), nd = pack2f(-my_delta, -my_delta);
#pragma unroll
          for (int i = 0; i < 32; i += 2) {                           // two columns per packed instruction: x = S c2 - lse, then dZ = P (dP - delta)
            float x0, x1, z0, z1;
            unpack2f(ffma2(pack2f(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), pack2f(c2, c2), nl), x0, x1);
            float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            if (!full) {
              const int q = xr, k = y0 + 32 * grp + i;
              const int klo = max(my_doc, p.window_blocks > 0 || p.window <= 0 ? 0 : q - p.window + 1);
              if (k > q || k < klo) p0 = 0.f;
              if (k + 1 > q || k + 1 < klo) p1 = 0.f;
            }
            unpack2f(fmul2(pack2f(p0, p1), fadd2(pack2f(__uint_as_float(rd[i]), __uint_as_float(rd[i + 1])), nd)), z0, z1);
            pz[i >> 1] = pack_bf16(z0, z1);
          }
          tmem_st16(dp_t, pz);
        }
        tc_wait_st();
        tc_fence_before();
        mbar_arrive(&bars->p_full[half]);
      }
      // ---- epilogue: the item's accumulators -> global rows (thread = row; 256 contiguous bytes each)
      if (ok) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, it & 1, abort_flag, p.status, 7));
      }
      if (ok) {
        tc_fence_after();
        __nv_bfloat16* dst = p.d1 + (((int64_t)b * T + xr) * p.H + h) * DAISY_HEAD_DIM + 32 * grp;
        uint32_t r[32];
        tmem_ld32(a1_t, r);
        tc_wait_ld();
        if (xr < T) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[i + e]) * p.scale;
            *reinterpret_cast<uint4*>(dst + i) = pack8(f);
          }
        }
        // the next item's first accumulating products overwrite what was just read
        tc_fence_before();
      }
      mbar_arrive(&bars->acc_empty);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 17) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ---------------------------------------------------------------------------------------------
// delta[b,h,t] = sum_d dO[b,t,h,d] O[b,t,h,d]: eight lanes per 256-byte row.
struct DeltaParams {
  const __nv_bfloat16 *o, *d_o;
  int64_t o_sb, o_st, o_sh, g_sb, g_st, g_sh;
  float* delta;
  int B, T, H;
};

__global__ void __launch_bounds__(256) swa_bwd_delta_kernel(const DeltaParams p) {
  grid_dep_launch();
  grid_dep_wait();
  const int64_t rows = (int64_t)p.B * p.T * p.H;
  const int64_t r = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  const int64_t rc = r < rows ? r : rows - 1;
  const int h = (int)(rc % p.H);
  const int64_t bt = rc / p.H;
  const int t = (int)(bt % p.T), b = (int)(bt / p.T);
  const __nv_bfloat16* po = p.o + b * p.o_sb + t * p.o_st + h * p.o_sh + 16 * sub;
  const __nv_bfloat16* pg = p.d_o + b * p.g_sb + t * p.g_st + h * p.g_sh + 16 * sub;
  float acc = 0.f;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    float a[8], g[8];
    unpack8(ld_stream16(po + 8 * u), a);
    unpack8(ld_stream16(pg + 8 * u), g);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc = fmaf(a[e], g[e], acc);
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  if (sub == 0 && r < rows) p.delta[((int64_t)b * p.H + h) * p.T + t] = acc;
}

// ---------------------------------------------------------------------------------------------
// Backward of the q/k/v preparation y = rope(rms_norm(x)) (no RoPE for v), row-wise:
//     g_n = rope^T(g_y),   xh = x r,  r = rsqrt(mean(x^2) + eps),   g_x = r (g_n - xh mean(g_n xh))
// Eight lanes per row; lane `sub` owns elements [8 sub, 8 sub + 8) and [64 + 8 sub, ...), the two halves RoPE pairs.
struct PrepBwdTensor {
  const __nv_bfloat16* x;        // raw input, logical [B,T,H,D] strides
  int64_t sb, st, sh;
  const __nv_bfloat16* gy;       // gradient of the prepared tensor, [B,T,H,D] contiguous
  __nv_bfloat16* gx;             // gradient of the raw input, [B,T,H,D] contiguous
  int do_norm, do_rope;
};
struct PrepBwdParams {
  PrepBwdTensor t[3];
  const float *cos, *sin;
  int B, T, H;
  float eps;
};

__global__ void __launch_bounds__(256) qkv_prep_bwd_kernel(const PrepBwdParams p) {
  const PrepBwdTensor& ten = p.t[blockIdx.y];
  if (ten.x == nullptr) return;
  const int64_t rows = (int64_t)p.B * p.T * p.H;
  const int64_t r = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  const int64_t rc = r < rows ? r : rows - 1;
  const int h = (int)(rc % p.H);
  const int64_t bt = rc / p.H;
  const int t = (int)(bt % p.T), b = (int)(bt / p.T);
  const __nv_bfloat16* px = ten.x + b * ten.sb + t * ten.st + h * ten.sh + 8 * sub;
  const __nv_bfloat16* pg = ten.gy + rc * DAISY_HEAD_DIM + 8 * sub;
  float x1[8], x2[8], g1[8], g2[8];
  unpack8(ld_stream16(px), x1); unpack8(ld_stream16(px + 64), x2);
  unpack8(ld_stream16(pg), g1); unpack8(ld_stream16(pg + 64), g2);
  if (ten.do_rope) {                                               // transpose of the rotation
    const float* cr = p.cos + (int64_t)t * 64 + 8 * sub;
    const float* sr = p.sin + (int64_t)t * 64 + 8 * sub;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float c = cr[e], s = sr[e], a = g1[e], b2 = g2[e];
      g1[e] = a * c - b2 * s;
      g2[e] = a * s + b2 * c;
    }
  }
  if (ten.do_norm) {
    float ss = 0.f, gd = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) { ss += x1[e] * x1[e] + x2[e] * x2[e]; gd += g1[e] * x1[e] + g2[e] * x2[e]; }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) { ss += __shfl_xor_sync(0xffffffffu, ss, o); gd += __shfl_xor_sync(0xffffffffu, gd, o); }
    const float rr = rsqrtf(ss * (1.0f / DAISY_HEAD_DIM) + p.eps);
    const float m = gd * rr * rr * (1.0f / DAISY_HEAD_DIM);        // mean(g_n xh) r = sum(g_n x) r^2 / D
#pragma unroll
    for (int e = 0; e < 8; ++e) { g1[e] = rr * (g1[e] - x1[e] * m); g2[e] = rr * (g2[e] - x2[e] * m); }
  }
  if (r < rows) {
    __nv_bfloat16* dst = ten.gx + rc * DAISY_HEAD_DIM + 8 * sub;
    *reinterpret_cast<uint4*>(dst) = pack8(g1);
    *reinterpret_cast<uint4*>(dst + 64) = pack8(g2);
  }
}

// ---------------------------------------------------------------------------------------------
// The same backward from what the fused projection leaves: the prepared rows y' and 1 / rms.  With y' = R xh (R the
// rotation, orthogonal) the mean in the norm's backward is mean(g_y y') and
//     g_x = R^T ( r (g_y - y' mean(g_y y')) )
// so the raw projections need not be kept or read.  A gated v (v' = g vn + (1 - g) ve) takes vn in place of y' and g g_y in
// place of g_y, and leaves d ve = (1 - g) g_y and the block's share of d g = sum g_y (vn - ve).  The three gradients go
// straight into the merged [M, 3 H 128] matrix that the two projection gradients read.  HBM-bound: 3 x 256 bytes a row.
struct PrepGradParams {
  const __nv_bfloat16* y[3];      // q', k', and v' or vn: [M, H, 128]
  const __nv_bfloat16* gy[3];     // their gradients (of v' where v is gated)
  const float* rstd;              // [M, 3 H]
  __nv_bfloat16* gx;              // [M, 3 H 128]
  const float *cos, *sin;
  const __nv_bfloat16* ve;        // [M, H, 128] or null
  const float* gate_logit;
  __nv_bfloat16* g_ve;            // [M, H, 128]
  float* partial;                 // one per block of the v part
  int M, T, H;
};

// Eight lanes a row, two rows of a block's 64 each, everything they read asked for before the first use.  (One row, the
// rotations asked for after the mean: 769 us at 65536 x 16 rows of q, k and v where the bytes take 370; this form 387.)
constexpr int PG_ROWS = 64;
template <int which>
__device__ __forceinline__ void prep_grad_rows(const PrepGradParams& p) {
  const uint32_t rows = (uint32_t)p.M * (uint32_t)p.H;
  const int sub = threadIdx.x & 7;
  uint4 y[2][2], g[2][2], e[2][2];
  float4 cs[2][4];                                               // cos, cos, sin, sin
  float rr[2];
  uint32_t row[2], m[2], h[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t r = blockIdx.x * PG_ROWS + 32 * i + (threadIdx.x >> 3), rc = min(r, rows - 1);
    row[i] = r; m[i] = rc / (uint32_t)p.H; h[i] = rc - m[i] * p.H;
    const int64_t off = (int64_t)rc * DAISY_HEAD_DIM + 8 * sub;
    y[i][0] = ld_stream16(p.y[which] + off); y[i][1] = ld_stream16(p.y[which] + off + 64);
    g[i][0] = ld_stream16(p.gy[which] + off); g[i][1] = ld_stream16(p.gy[which] + off + 64);
    if (which == 2 && p.ve) { e[i][0] = ld_stream16(p.ve + off); e[i][1] = ld_stream16(p.ve + off + 64); }
    rr[i] = __ldg(p.rstd + ((int64_t)m[i] * 3 + which) * p.H + h[i]);
    if (which < 2) {
      const int64_t t = (int64_t)(m[i] % (uint32_t)p.T) * 64 + 8 * sub;
      cs[i][0] = __ldg(reinterpret_cast<const float4*>(p.cos + t)); cs[i][1] = __ldg(reinterpret_cast<const float4*>(p.cos + t) + 1);
      cs[i][2] = __ldg(reinterpret_cast<const float4*>(p.sin + t)); cs[i][3] = __ldg(reinterpret_cast<const float4*>(p.sin + t) + 1);
    }
  }
  float share = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float x1[8], x2[8], g1[8], g2[8];
    unpack8(y[i][0], x1); unpack8(y[i][1], x2);
    unpack8(g[i][0], g1); unpack8(g[i][1], g2);
    if (which == 2 && p.ve) {
      const float gate = 1.0f / (1.0f + __expf(-*p.gate_logit));
      float e1[8], e2[8], d1[8], d2[8], sh = 0.f;
      unpack8(e[i][0], e1); unpack8(e[i][1], e2);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        sh = fmaf(g1[j], x1[j] - e1[j], sh); sh = fmaf(g2[j], x2[j] - e2[j], sh);
        d1[j] = (1.0f - gate) * g1[j]; d2[j] = (1.0f - gate) * g2[j];
        g1[j] *= gate; g2[j] *= gate;
      }
      if (row[i] < rows) {
        const int64_t off = (int64_t)row[i] * DAISY_HEAD_DIM + 8 * sub;
        *reinterpret_cast<uint4*>(p.g_ve + off) = pack8(d1);
        *reinterpret_cast<uint4*>(p.g_ve + off + 64) = pack8(d2);
        share += sh;
      }
    }
    float gd = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) gd += g1[j] * x1[j] + g2[j] * x2[j];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) gd += __shfl_xor_sync(0xffffffffu, gd, o);
    const float mean = gd * (1.0f / DAISY_HEAD_DIM);
#pragma unroll
    for (int j = 0; j < 8; ++j) { g1[j] = rr[i] * (g1[j] - x1[j] * mean); g2[j] = rr[i] * (g2[j] - x2[j] * mean); }
    if (which < 2) {
      const float c[8] = {cs[i][0].x, cs[i][0].y, cs[i][0].z, cs[i][0].w, cs[i][1].x, cs[i][1].y, cs[i][1].z, cs[i][1].w};
      const float s[8] = {cs[i][2].x, cs[i][2].y, cs[i][2].z, cs[i][2].w, cs[i][3].x, cs[i][3].y, cs[i][3].z, cs[i][3].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = g1[j], b2 = g2[j];
        g1[j] = a * c[j] - b2 * s[j];
        g2[j] = a * s[j] + b2 * c[j];
      }
    }
    if (row[i] < rows) {
      __nv_bfloat16* dst = p.gx + (((int64_t)m[i] * 3 + which) * p.H + h[i]) * DAISY_HEAD_DIM + 8 * sub;
      *reinterpret_cast<uint4*>(dst) = pack8(g1);
      *reinterpret_cast<uint4*>(dst + 64) = pack8(g2);
    }
  }
  if (which == 2 && p.ve) {
    __shared__ float red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) share += __shfl_xor_sync(0xffffffffu, share, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = share;
    __syncthreads();
    if (threadIdx.x == 0) p.partial[blockIdx.x] = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
  }
}

__global__ void __launch_bounds__(256, 3) qkv_prep_grad_kernel(const __grid_constant__ PrepGradParams p) {
  if (blockIdx.y == 0) prep_grad_rows<0>(p);
  else if (blockIdx.y == 1) prep_grad_rows<1>(p);
  else prep_grad_rows<2>(p);
}

// The gate's gradient from the blocks' shares, in a fixed order: d logit = g (1 - g) sum.
__global__ void __launch_bounds__(1024) gate_grad_kernel(const float* partial, int n, const float* gate_logit, float* out) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 1024) s += partial[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
      const float g = 1.0f / (1.0f + __expf(-*gate_logit));
      *out = g * (1.0f - g) * s;
    }
  }
}

}  // namespace daisy

using namespace daisy;

// Most bytes of dZ images that a call asks room for (above that the (batch, head) pairs go in several rounds).  8 x 8192 tokens,
// 16 heads are 4.6 GB at a window of 2048 tokens, three rounds, and 4.3 GB at one of 16 blocks of 128, two.
static constexpr size_t BWD_TILES_MAX = (size_t)2 << 30;

static int bwd_smem_attr() {
  static bool done[daisy_host::MAX_DEVICES] = {};
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  if (done[dev]) return DAISY_OK;
  if (cudaFuncSetAttribute(swa_bwd_kv_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(swa_bwd_kv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(swa_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(swa_bwd_q_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess)
    return DAISY_ECUDA;
  // swa_bwd_kv_kernel's swizzled tiles lie at the start of its dynamic shared memory, behind what the system and the kernel's static
  // variables take: where that is no multiple of 1024 bytes no kernel of the backward is launched
  int reserved = 0;
  if (cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess) return DAISY_ECUDA;
  for (const auto kernel : {swa_bwd_kv_kernel<false>, swa_bwd_kv_kernel<true>}) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess) return DAISY_ECUDA;
    if ((reserved + a.sharedSizeBytes) & 1023) return DAISY_EALIGN;
  }
  done[dev] = true;
  return DAISY_OK;
}

extern "C" size_t daisy_b200_swa_attend_bwd_workspace_bytes(int B, int T, int H) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  return (size_t)B * T * H * sizeof(float);                        // delta
}

// dZ images of one (batch, head): every query block's key blocks inside the window, 32 KB each
static size_t bwd_tiles_row(int T, int window, bool in_blocks) {
  const int64_t nblk = ((int64_t)T + WB - 1) / WB, seen = window <= 0 ? nblk : in_blocks ? window : ((int64_t)window + WB - 2) / WB + 1;
  return (size_t)(seen < nblk ? seen : nblk);
}
static size_t bwd_tiles_bytes(int T, int window, bool in_blocks) {
  return (size_t)((T + WB - 1) / WB) * bwd_tiles_row(T, window, in_blocks) * W_TILE;
}
static size_t bwd_delta_bytes(int B, int T, int H) { return (daisy_b200_swa_attend_bwd_workspace_bytes(B, T, H) + 1023) & ~(size_t)1023; }

// Whether images of `room` (batch, head) pairs at a time are worth their rounds: a tile through them costs 0.78 of one whose
// scores are formed again, but a round of few items lasts as long as its longest, while the other way all items share the SMs.  An
// SM's tiles are taken as the mean and a quarter of the longest item, or as the longest.  Images against scores, us:
// no window: 1 x 24576 x 8 (eight rounds of 192 items, the longest of 192 tiles where the mean of an SM is 125) 4424-4804 / 3880,
// with eight documents 1190 / 787; 1 x 26000 x 8 4750 / 4336, 28000 5266 / 5233, 28700 5450 / 5520 (the rule's line: 28100), 30000 5697 / 6257; 1 x 24576 x 1
// 610 / 840; 1 x 20480 x 8 (four rounds, 160 against 174) 2394 / 2992; 1 x 32000 x 4 2948 / 3365;
// window 8192: 1 x 65536 x 4 3252-3373 / 3521; window 2048: 1 x 65536 x 16 3134 / 4667
static bool bwd_images_pay(int B, int T, int H, int window, bool in_blocks, size_t room) {
  const size_t pairs = (size_t)B * H, rounds = (pairs + room - 1) / room;
  if (rounds == 1) return true;
  const int sms = daisy_host::sm_count_cached();
  const double nblk = (double)(((int64_t)T + WB - 1) / WB), longest = (double)bwd_tiles_row(T, window, in_blocks), tiles = longest * (nblk - (longest - 1) / 2);
  const auto lasts = [&](size_t n) {
    const double sm = n * tiles / (sms > 0 ? sms : 148) + longest / 4;
    return sm > longest ? sm : longest;
  };
  return 0.78 * rounds * lasts((pairs + rounds - 1) / rounds) < lasts(pairs);
}

extern "C" size_t daisy_b200_swa_attend_bwd_workspace_bytes_full(int B, int T, int H, int window, unsigned flags) {
  if (B <= 0 || T <= 0 || H <= 0 || (flags & ~DAISY_WINDOW_BLOCKS)) return 0;
  const bool in_blocks = (flags & DAISY_WINDOW_BLOCKS) != 0;
  const size_t one = bwd_tiles_bytes(T, window, in_blocks), pairs = (size_t)B * H;
  const size_t n = BWD_TILES_MAX / one < pairs ? BWD_TILES_MAX / one : pairs;
  return n && bwd_images_pay(B, T, H, window, in_blocks, n) ? bwd_delta_bytes(B, T, H) + n * one : daisy_b200_swa_attend_bwd_workspace_bytes(B, T, H);
}

// (batch, head) pairs a round takes: rounds of equal size, as many as there is room for images; 0: no room for one pair's
static int bwd_pairs_a_round(int B, int T, int H, int window, bool in_blocks, size_t workspace_bytes) {
  const size_t delta_bytes = bwd_delta_bytes(B, T, H);
  const int64_t room = workspace_bytes > delta_bytes ? (int64_t)((workspace_bytes - delta_bytes) / bwd_tiles_bytes(T, window, in_blocks)) : 0;
  if (room == 0) return 0;
  const int64_t pairs = (int64_t)B * H, rounds = (pairs + room - 1) / room;
  return (int)((pairs + rounds - 1) / rounds);
}

extern "C" int daisy_b200_swa_attend_bwd_rounds(int B, int T, int H, int window, unsigned flags, size_t workspace_bytes) {
  if (B <= 0 || T <= 0 || H <= 0 || (flags & ~DAISY_WINDOW_BLOCKS)) return DAISY_EINVAL;
  if ((int64_t)B * T * H >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  if (workspace_bytes < daisy_b200_swa_attend_bwd_workspace_bytes(B, T, H)) return DAISY_EWORKSPACE;
  const int per = bwd_pairs_a_round(B, T, H, window, (flags & DAISY_WINDOW_BLOCKS) != 0, workspace_bytes);
  return per ? (B * H + per - 1) / per : 1;
}

extern "C" int daisy_b200_swa_attend_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                         int64_t q_sb, int64_t q_st, int64_t q_sh,
                                         int64_t k_sb, int64_t k_st, int64_t k_sh,
                                         int64_t v_sb, int64_t v_st, int64_t v_sh,
                                         int64_t o_sb, int64_t o_st, int64_t o_sh,
                                         int64_t g_sb, int64_t g_st, int64_t g_sh,
                                         const float* lse2, void* dq, void* dk, void* dv,
                                         int B, int T, int H, int D, int window, float scale,
                                         const int32_t* doc_start, int64_t doc_sb, unsigned flags,
                                         void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
  if (!q || !k || !v || !o || !d_o || !lse2 || !dq || !dk || !dv || !workspace || B <= 0 || T <= 0 || H <= 0 || !(scale > 0.f)) return DAISY_EINVAL;
  if (D != DAISY_HEAD_DIM) return DAISY_EUNSUPPORTED;
  if (flags & ~DAISY_WINDOW_BLOCKS) return DAISY_EINVAL;
  if (workspace_bytes < daisy_b200_swa_attend_bwd_workspace_bytes(B, T, H)) return DAISY_EWORKSPACE;
  const void* ptrs[] = {q, k, v, o, d_o, dq, dk, dv, workspace};
  for (const void* x : ptrs) if (!daisy_aligned16(x)) return DAISY_EALIGN;
  if ((q_sb | q_st | q_sh | k_sb | k_st | k_sh | v_sb | v_st | v_sh | o_sb | o_st | o_sh | g_sb | g_st | g_sh) & 7) return DAISY_EALIGN;
  if (q_st <= 0 || k_st <= 0 || v_st <= 0 || g_st <= 0 || o_st <= 0) return DAISY_EINVAL;
  if ((H > 1 && (q_sh <= 0 || k_sh <= 0 || v_sh <= 0 || g_sh <= 0 || o_sh <= 0)) || (B > 1 && (q_sb <= 0 || k_sb <= 0 || v_sb <= 0 || g_sb <= 0 || o_sb <= 0)))
    return DAISY_EINVAL;
  if (doc_start && (doc_sb < 0 || (reinterpret_cast<uintptr_t>(doc_start) & 3))) return DAISY_EINVAL;
  if ((int64_t)B * T * H >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  if (const int arc = bwd_smem_attr(); arc != DAISY_OK) { (void)cudaGetLastError(); return arc; }
  cudaStream_t st = (cudaStream_t)stream;
  float* delta = (float*)workspace;
  {
    DeltaParams dp{(const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, o_sb, o_st, o_sh, g_sb, g_st, g_sh, delta, B, T, H};
    const int64_t rows = (int64_t)B * T * H;
    (void)daisy_host::launch_dependent(swa_bwd_delta_kernel, dim3((unsigned)((rows * 8 + 255) / 256)), dim3(256), 0, st, dp);
    DAISY_CHECK_LAUNCH();
  }
  CUtensorMap tq, tk, tv, tg;
  int rc;
  auto sb = [](int64_t s, int n) { return (uint64_t)(n == 1 ? 16 : s * 2); };
  if ((rc = daisy_host::make_tmap_bf16_dthb(&tq, q, D, T, H, B, q_st * 2, sb(q_sh, H), sb(q_sb, B), 64, WB)) != DAISY_OK) return rc;
  if ((rc = daisy_host::make_tmap_bf16_dthb(&tk, k, D, T, H, B, k_st * 2, sb(k_sh, H), sb(k_sb, B), 64, WB)) != DAISY_OK) return rc;
  if ((rc = daisy_host::make_tmap_bf16_dthb(&tv, v, D, T, H, B, v_st * 2, sb(v_sh, H), sb(v_sb, B), 64, WB)) != DAISY_OK) return rc;
  if ((rc = daisy_host::make_tmap_bf16_dthb(&tg, d_o, D, T, H, B, g_st * 2, sb(g_sh, H), sb(g_sb, B), 64, WB)) != DAISY_OK) return rc;
  BwdParams p;
  p.lse2 = lse2; p.delta = delta; p.doc_start = doc_start; p.doc_sb = doc_sb;
  p.T = T; p.H = H; p.B = B;
  const bool in_blocks = (flags & DAISY_WINDOW_BLOCKS) != 0;
  p.window = in_blocks ? 0 : window;
  p.window_blocks = (in_blocks && window > 0) ? window : 0;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status_word;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  const int nblk = (T + WB - 1) / WB;
  const int room = bwd_pairs_a_round(B, T, H, window, in_blocks, workspace_bytes), pairs = B * H, per = room ? room : pairs;
  p.tiles = (uint8_t*)workspace + bwd_delta_bytes(B, T, H); p.tiles_row = (int)bwd_tiles_row(T, window, in_blocks);
  for (p.bh0 = 0; p.bh0 < pairs; p.bh0 += per) {
    p.n_bh = pairs - p.bh0 < per ? pairs - p.bh0 : per;
    const int64_t items = (int64_t)nblk * p.n_bh;
    const unsigned grid = (unsigned)(items < sms ? items : sms);
    p.d0 = (__nv_bfloat16*)dv; p.d1 = (__nv_bfloat16*)dk;
    (void)daisy_host::launch_dependent(room ? swa_bwd_kv_kernel<true> : swa_bwd_kv_kernel<false>, dim3(grid), dim3(KV_THREADS), KV_SMEM, st, tq, tk, tv, tg, p);
    DAISY_CHECK_LAUNCH();
    p.d0 = nullptr; p.d1 = (__nv_bfloat16*)dq;
    if (room) (void)daisy_host::launch_dependent(swa_bwd_dq_kernel, dim3(grid), dim3(DQ_THREADS), DQ_SMEM, st, tk, p);
    else      (void)daisy_host::launch_dependent(swa_bwd_q_kernel, dim3(grid), dim3(BWD_THREADS), BWD_SMEM, st, tq, tk, tv, tg, p);
    DAISY_CHECK_LAUNCH();
  }
  return DAISY_OK;
}

extern "C" int daisy_b200_qkv_prep_bwd(const void* q, const void* k, const void* v,
                                       int64_t q_sb, int64_t q_st, int64_t q_sh,
                                       int64_t k_sb, int64_t k_st, int64_t k_sh,
                                       int64_t v_sb, int64_t v_st, int64_t v_sh,
                                       const float* cos, const float* sin,
                                       const void* dq_p, const void* dk_p, const void* dv_p,
                                       void* dq, void* dk, void* dv,
                                       int B, int T, int H, int D, float eps, unsigned flags, void* stream) {
  if (B <= 0 || T <= 0 || H <= 0) return DAISY_EINVAL;
  if (D != DAISY_HEAD_DIM) return DAISY_EUNSUPPORTED;
  if (flags & ~DAISY_QKV_DEFAULT) return DAISY_EINVAL;
  if ((q == nullptr) != (dq == nullptr) || (q == nullptr) != (dq_p == nullptr) || (k == nullptr) != (dk == nullptr) ||
      (k == nullptr) != (dk_p == nullptr) || (v == nullptr) != (dv == nullptr) || (v == nullptr) != (dv_p == nullptr)) return DAISY_EINVAL;
  if (!q && !k && !v) return DAISY_EINVAL;
  if ((flags & DAISY_ROPE) && (!cos || !sin)) return DAISY_EINVAL;
  const void* ptrs[] = {q, k, v, dq_p, dk_p, dv_p, dq, dk, dv};
  for (const void* x : ptrs) if (x && !daisy_aligned16(x)) return DAISY_EALIGN;
  if ((q_sb | q_st | q_sh | k_sb | k_st | k_sh | v_sb | v_st | v_sh) & 7) return DAISY_EALIGN;
  if ((int64_t)B * T * H >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  PrepBwdParams p;
  p.t[0] = {(const __nv_bfloat16*)q, q_sb, q_st, q_sh, (const __nv_bfloat16*)dq_p, (__nv_bfloat16*)dq, (flags & DAISY_NORM_Q) ? 1 : 0, (flags & DAISY_ROPE) ? 1 : 0};
  p.t[1] = {(const __nv_bfloat16*)k, k_sb, k_st, k_sh, (const __nv_bfloat16*)dk_p, (__nv_bfloat16*)dk, (flags & DAISY_NORM_K) ? 1 : 0, (flags & DAISY_ROPE) ? 1 : 0};
  p.t[2] = {(const __nv_bfloat16*)v, v_sb, v_st, v_sh, (const __nv_bfloat16*)dv_p, (__nv_bfloat16*)dv, (flags & DAISY_NORM_V) ? 1 : 0, 0};
  p.cos = cos; p.sin = sin; p.B = B; p.T = T; p.H = H; p.eps = eps;
  const int64_t rows = (int64_t)B * T * H;
  dim3 grid((unsigned)((rows * 8 + 255) / 256), 3, 1);
  qkv_prep_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(p);
  DAISY_CHECK_LAUNCH();
  return DAISY_OK;
}

extern "C" int64_t daisy_b200_qkv_prep_grad_blocks(int M, int H) { return M > 0 && H > 0 ? ((int64_t)M * H + PG_ROWS - 1) / PG_ROWS : 0; }

extern "C" int daisy_b200_qkv_prep_grad(const void* q_p, const void* k_p, const void* v_n, const void* dq_p, const void* dk_p, const void* dv_p,
                                        const float* rstd, const float* cos, const float* sin, void* dqkv,
                                        const void* ve, const float* ve_gate_logit, void* d_ve, float* d_logit, float* partial,
                                        int M, int T, int H, int D, void* stream) {
  if (!q_p || !k_p || !v_n || !dq_p || !dk_p || !dv_p || !rstd || !cos || !sin || !dqkv || M <= 0 || T <= 0 || H <= 0) return DAISY_EINVAL;
  if (D != DAISY_HEAD_DIM) return DAISY_EUNSUPPORTED;
  if (ve && (!ve_gate_logit || !d_ve || !d_logit || !partial)) return DAISY_EINVAL;
  const void* ptrs[] = {q_p, k_p, v_n, dq_p, dk_p, dv_p, cos, sin, dqkv, ve, d_ve};
  for (const void* x : ptrs) if (!daisy_aligned16(x)) return DAISY_EALIGN;
  if ((int64_t)M * H >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  PrepGradParams p{};
  p.y[0] = (const __nv_bfloat16*)q_p; p.y[1] = (const __nv_bfloat16*)k_p; p.y[2] = (const __nv_bfloat16*)v_n;
  p.gy[0] = (const __nv_bfloat16*)dq_p; p.gy[1] = (const __nv_bfloat16*)dk_p; p.gy[2] = (const __nv_bfloat16*)dv_p;
  p.rstd = rstd; p.gx = (__nv_bfloat16*)dqkv; p.cos = cos; p.sin = sin;
  p.ve = (const __nv_bfloat16*)ve; p.gate_logit = ve_gate_logit; p.g_ve = (__nv_bfloat16*)d_ve; p.partial = partial;
  p.M = M; p.T = T; p.H = H;
  const int64_t blocks = daisy_b200_qkv_prep_grad_blocks(M, H);
  qkv_prep_grad_kernel<<<dim3((unsigned)blocks, 3, 1), 256, 0, (cudaStream_t)stream>>>(p);
  DAISY_CHECK_LAUNCH();
  if (ve) {
    gate_grad_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(partial, (int)blocks, ve_gate_logit, d_logit);
    DAISY_CHECK_LAUNCH();
  }
  return DAISY_OK;
}
