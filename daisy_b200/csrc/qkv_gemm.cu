// C[M,N] = X[M,K] W[N,K]^T on tcgen05 tensor cores, bf16 in, fp32 accumulation in TMEM, with the projection's
// element-wise tail as the epilogue.
//
// Two uses (the GEMMs either side of the attention core, models/daisy/attention.py:118-125 and :149):
//   EPI_QKV    W = qkvo_w[:3] flattened ([3*H*128, dim]): a 128-column output tile is one head of q, k or v of 128
//              tokens, so the weightless RMS norm over D and the half-rotation RoPE are per-thread work on the
//              accumulator row (thread = token = TMEM lane); q', k', v' leave as [B,T,H,D] bf16 and the separate
//              norm/RoPE pass over q, k, v (1.6 GB at B=8, T=8192, 16 heads) disappears.
//   EPI_PLAIN  bf16 store of C (the output projection); up to three products of one shape in one launch (the Kimi layer's
//              q, k and v projections: 3 x 192 tiles in 8 waves instead of 3 x 3).  Two of the Kimi layer's groups end in its
//              gates: beside the two low-rank products a third of H columns leaves as sigmoid(C) in float32 (the write
//              strength), and the first of the two that follow as  -exp(A_log) softplus(C + dt_bias)  (the log-decay).
//              2 x 3001 tokens, 16 heads: 12.5 + 8.6 + 2.7 us (low-rank products, library product, sigmoid) -> 18.3, 18 + 18.4
//              (second products, gate) -> 33.9; 2 x 127, 12 heads: the layer 86 -> 65 us with three launches fewer.
//
// Persistent CTAs walk 128 x BN output tiles (n fastest, so concurrently running CTAs share X tiles and the
// whole W in L2).  Roles (352 threads): warps 0-7 epilogue, warp 8 MMA issuer, warps 9, 10 TMA producers.  Both
// operands are K-major with 128-byte swizzle (64-element boxes), exactly the Q K^T operand form of the
// attention kernel.  Two accumulators in TMEM (2 x BN columns) let the epilogue of tile i run under the main loop of
// tile i + 1.  At K = 768 the epilogue bounds the QKV form, not the products: with four epilogue warps reading their
// rotations row by row 65536 x 2304 x 768 took 270 us, with eight and rotations through shared memory 219.
// PAIR form (N a multiple of 256): clusters of two CTAs on 256 x 256 tiles with cta_group::2 MMAs.  Each CTA loads its
// own 128 rows of X and its own 128 of the tile's 256 weight rows (plain per-CTA TMA loads), the pair's tensor cores
// read both weight halves, so the shared-memory fill and operand reads per flop drop by a third against the single-CTA
// 128 x 256 tile; rank 0 issues the MMAs, both CTAs run the epilogue on their own 128 accumulator rows.
// All mbarrier waits are bounded (abort flag, DAISY_ETIMEOUT through the status word), as everywhere else.
#include "common.cuh"
#include "kda_gate.cuh"
#include <cuda_fp16.h>

namespace daisy {

constexpr int GM = 128, GK = 64;
constexpr int G_THREADS = 352;                         // 8 epilogue warps, MMA warp, 2 TMA warps
constexpr int G_SMALL_THREADS = 192;                   // 4 epilogue warps, TMA warp, MMA warp
constexpr int G_A_BYTES = GM * GK * 2;                 // 16 KB

template <int BN, bool PAIR, bool QKV> struct GemmCfg {
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;    // weight rows this CTA keeps per stage
  static constexpr int B_BYTES = B_ROWS * GK * 2;
  static constexpr int STAGE = G_A_BYTES + B_BYTES;
  // per epilogue warp: 16 output rows at a time; QKV: before that, two slices of rotations
  static constexpr int WARP_STAGING = QKV ? 2 * 4096 : 4096;
  static constexpr int NST = QKV ? 5 : 6;
  static constexpr int SMEM = 1024 + NST * STAGE + 8 * WARP_STAGING + 256;
  static constexpr int TILE_M = PAIR ? 2 * GM : GM;
};

constexpr int GROUP = 3;
struct GemmMaps { CUtensorMap x[GROUP], w[GROUP]; };

struct GemmParams {
  int M, N, K;
  int epi;                       // 0 plain, 1 qkv
  // plain: up to GROUP products of one shape, columns [i per, (i + 1) per) of N are product i's
  __nv_bfloat16* c[GROUP]; int64_t ldc;
  int per;
  // plain: product 0 as the log-decay gate [M, per] float32; product 2 as sigmoid [M, beta_n] float32, of beta_n weight rows; or null
  float *gate, *beta;
  const float *a_log, *dt_bias;
  int beta_n;
  // qkv
  __nv_bfloat16* out[3];         // q', k', v'  [M, H, 128]
  const float *cos, *sin;        // [T, 64]
  const __nv_bfloat16* ve;       // value embedding [M, H, 128] (row stride ve_ld elements) or null
  int64_t ve_ld;
  const float* ve_gate_logit;    // v' = g * norm(v) + (1 - g) * ve, g = sigmoid(*ve_gate_logit)
  int T, H;
  float eps;
  unsigned flags;
  int* status;
  // optional ring-cache side output: rows t >= ring_first of k' (ring[0]) and v' (ring[1]) also go to slot t % cap of
  // a [B,H,cap,128] ring with element strides (r_sb, r_sh, r_sr); bf16 or (ring_f16) float16 rows
  void* ring[2];
  int64_t r_sb, r_sh, r_sr;
  int cap, ring_first, ring_f16;
  int order;                     // narrow tiles only: ORDER_AHEAD, ORDER_BEHIND (common.cuh) or 0
  // training: 1 / rms of every row and head slot, [M][3 H], and v as normalised before the gate, [M, H, 128]; or null
  float* rstd;
  __nv_bfloat16* vn;
};

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// Two products that end in a gate take what a bf16 store of the product would have left.
// a softplus(bf16(c) + bias), rounded to bf16, of N pairs side by side, each step for all of them before the next (left to itself a
// warp goes through one chain of twenty dependent instructions after the other: 61 us instead of 34 at 6002 x 2048).  softplus is that of
// kda_gate.cuh; its threshold of 20 changes nothing here, where log1p(e^-20) is far below an ulp of 20.
template <int N>
__device__ __forceinline__ void gemm_decay2(uint64_t (&c)[N], const uint64_t (&bias)[2], float a) {
  uint64_t u[N], r[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float x0, x1;
    unpack2f(c[i], x0, x1);
    const uint32_t b = pack_bf16(x0, x1);
    c[i] = fadd2(pack2f(bf16_lo(b), bf16_hi(b)), bias[i & 1]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float x0, x1;
    unpack2f(c[i], x0, x1);
    u[i] = pack2f(fast_exp2(fabsf(x0) * -1.4426950408889634f), fast_exp2(fabsf(x1) * -1.4426950408889634f));
    r[i] = pack2f(LOG1P_C[0], LOG1P_C[0]);
  }
#pragma unroll
  for (int k = 1; k < 10; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = ffma2(r[i], u[i], pack2f(LOG1P_C[k], LOG1P_C[k]));
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float x0, x1, y0, y1;
    unpack2f(c[i], x0, x1);
    unpack2f(fmul2(fadd2(pack2f(fmaxf(x0, 0.f), fmaxf(x1, 0.f)), fmul2(r[i], u[i])), pack2f(a, a)), y0, y1);
    const uint32_t b = pack_bf16(y0, y1);
    c[i] = pack2f(bf16_lo(b), bf16_hi(b));
  }
}
__device__ __forceinline__ float gemm_sigmoid(float c) { return round_bf16(1.f / (1.f + expf(-round_bf16(c)))); }
constexpr int BETA_MAX = 32;

struct GemmBars {
  uint64_t full[6], empty[6];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <int BN, bool PAIR, bool QKV>
__global__ void __launch_bounds__(G_THREADS, 1)
qkv_gemm_kernel(const __grid_constant__ GemmMaps maps, const GemmParams p) {
  using Cfg = GemmCfg<BN, PAIR, QKV>;
  extern __shared__ uint8_t gemm_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stages = smem;
  uint8_t* staging = smem + Cfg::NST * Cfg::STAGE;
  GemmBars* bars = reinterpret_cast<GemmBars*>(staging + 8 * Cfg::WARP_STAGING);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (p.M + Cfg::TILE_M - 1) / Cfg::TILE_M, n_tiles = p.N / BN, kb_n = p.K / GK;
  const int tiles = m_tiles * n_tiles;
  // PAIR: the work item belongs to the cluster; rank 0 issues the MMAs, rank r owns rows r * 128 .. of the tile
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::NST; ++i) { mbar_init(&bars->full[i], 1); mbar_init(&bars->empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->acc_full[i], 1); mbar_init(&bars->acc_empty[i], PAIR ? 512 : 128); }
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 8) {
    if (PAIR) { tmem_alloc_pair(&bars->tmem_base, 2 * BN); tmem_relinquish_pair(); }
    else { tmem_alloc(&bars->tmem_base, 2 * BN); tmem_relinquish(); }
  }
  tc_fence_before();
  if (PAIR) cluster_sync_all();                        // the peer's barriers exist before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_launch();
  grid_dep_wait();

  if (warp >= 9) {
    // ------------------------------------------------------------------ TMA producers: every other k-block each (a turn of the
    // loop takes one thread some 450 cycles, the products of a k-block 256, PAIR 512)
    if (lane == 0) {
      prefetch_tmap(&maps.x[0]); prefetch_tmap(&maps.w[0]);
      uint32_t n = warp - 9, first = 0;                  // my next k-block, and the tile's first, counted over all tiles
      bool ok = true;
      for (int tile = worker; tile < tiles && ok; tile += workers, first += kb_n) {
        const int m0 = (tile / n_tiles) * Cfg::TILE_M + (int)rank * GM, n0 = (tile % n_tiles) * BN;
        const int prod = QKV ? 0 : n0 / p.per, w0 = n0 - prod * p.per + (int)rank * Cfg::B_ROWS;
        const CUtensorMap *tm_x = &maps.x[prod], *tm_w = &maps.w[prod];
        for (; n < first + kb_n; n += 2) {
          const int kb = n - first;
          const int st = n % Cfg::NST;
          if (!mbar_wait(&bars->empty[st], ((n / Cfg::NST) & 1) ^ 1, abort_flag, p.status, 1)) { ok = false; break; }
          uint8_t* dst = stages + st * Cfg::STAGE;
          if (PAIR) {
            // both CTAs' bytes are counted on rank 0's barrier, which the MMA issuer waits on
            const uint32_t full0 = mapa_shared(smem_u32(&bars->full[st]), 0);
            if (rank == 0) mbar_expect_tx(&bars->full[st], 2 * Cfg::STAGE);
            tma_load_3d_pair(dst, tm_x, full0, kb * GK, m0, 0);
            tma_load_3d_pair(dst + G_A_BYTES, tm_w, full0, kb * GK, w0, 0);
          } else {
            mbar_expect_tx(&bars->full[st], Cfg::STAGE);
            tma_load_3d(dst, tm_x, &bars->full[st], kb * GK, m0, 0);
            tma_load_3d(dst + G_A_BYTES, tm_w, &bars->full[st], kb * GK, w0, 0);
          }
        }
      }
    }
  } else if (warp == 8 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = umma_idesc_bf16(Cfg::TILE_M, BN, 0, 0);
    const uint64_t ad = umma_desc_sw128(smem_u32(stages), 16, 1024);
    const uint64_t bd = umma_desc_sw128(smem_u32(stages + G_A_BYTES), 16, 1024);
    const uint32_t a_lo0 = (uint32_t)ad, b_lo0 = (uint32_t)bd, hi = (uint32_t)(ad >> 32);
    uint32_t n = 0, it = 0;
    bool ok = true;
    for (int tile = worker; tile < tiles && ok; tile += workers, ++it) {
      const uint32_t buf = it & 1;
      if (!mbar_wait(&bars->acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 2)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      for (int kb = 0; kb < kb_n; ++kb, ++n) {
        const int st = n % Cfg::NST;
        if (!mbar_wait(&bars->full[st], (n / Cfg::NST) & 1, abort_flag, p.status, 3)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_lo = a_lo0 + st * (Cfg::STAGE >> 4), b_lo = b_lo0 + st * (Cfg::STAGE >> 4);
#pragma unroll
        for (int k = 0; k < GK / 16; ++k) {
          if (PAIR) umma_ss_pair_p(leader, d_tmem, a_lo + k * 2, hi, b_lo + k * 2, hi, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          else umma_ss_lh_p(leader, d_tmem, a_lo + k * 2, hi, b_lo + k * 2, hi, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        if (PAIR) tc_commit_pair_p(leader, &bars->empty[st]);       // both CTAs' producers may refill the stage
        else tc_commit_p(leader, &bars->empty[st]);
      }
      if (ok) {
        if (PAIR) tc_commit_pair_p(leader, &bars->acc_full[buf]);
        else tc_commit_p(leader, &bars->acc_full[buf]);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ epilogue: thread = output row.  Two groups of four warps:
    // PAIR: one takes the tile's columns 0 .. 127, the other 128 .. 255; single: one takes the even tiles, the other the odd ones
    const int grp = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* stg = staging + warp * Cfg::WARP_STAGING;
    const uint32_t s_stg = smem_u32(stg), s_own = s_stg + lane * 128;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = worker; tile < tiles && ok; tile += workers, ++it) {
      const uint32_t buf = it & 1;
      if (!PAIR && (int)buf != grp) continue;
      const int m0 = (tile / n_tiles) * Cfg::TILE_M + (int)rank * GM, n0 = (tile % n_tiles) * BN + (PAIR ? grp * 128 : 0);
      const int m = m0 + row;
      // RoPE: slice i of the rotations (cos, sin of channels 16 i .. 16 i + 15 of the warp's 32 rows) goes through shared memory,
      // two slices ahead: a lane's own row read straight from the tables is 32 lines an instruction, 4096 cycles a 128 x 128 tile
      const bool rope = QKV && (n0 >> 7) < 2 * p.H && (p.flags & DAISY_ROPE);
      const int pos = rope ? min(m, p.M - 1) % p.T : 0;
      auto fetch = [&](int i) {
        const float* tab = ((lane & 4) ? p.sin : p.cos) + 16 * i + 4 * (lane & 3);
        const uint32_t dst = s_stg + (i & 1) * 4096;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int rr = 4 * j + (lane >> 3);
          cp_async16(dst + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4), tab + (size_t)__shfl_sync(0xffffffffu, pos, rr) * 64);
        }
        cp_async_commit();
      };
      if (rope) { fetch(0); fetch(1); }
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full[buf], (it >> 1) & 1, abort_flag, p.status, 4));
      if (!ok) { if (QKV) cp_async_wait<0>(); break; }
      tc_fence_after();
      const uint32_t t0 = tmem_base + lane_off + buf * BN + (PAIR ? grp * 128 : 0);
      if (!QKV && p.gate && n0 < p.per) {
        // 32 columns at a time, transposed through the staging rows: a lane then has four columns of eight rows, eight lanes 128
        // bytes of a row
        const float a = -expf(__ldg(p.a_log + (n0 >> 7)));
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          uint32_t r[32];
          tmem_ld32(t0 + 32 * q, r);
          const int c = 4 * (lane & 7);
          const float4 bias = __ldg(reinterpret_cast<const float4*>(p.dt_bias + n0 + 32 * q + c));
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(stg + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
          __syncwarp();
          float* dst = p.gate + (size_t)(m0 + (warp & 3) * 32) * p.per + n0 + 32 * q + c;
          const uint64_t bias2[2] = {pack2f(bias.x, bias.y), pack2f(bias.z, bias.w)};
          uint64_t v[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = 4 * i + (lane >> 3);
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(stg + rr * 128 + (((lane ^ rr) & 7) << 4));
            v[2 * i] = t.x; v[2 * i + 1] = t.y;
          }
          gemm_decay2(v, bias2, a);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = 4 * i + (lane >> 3);
            if (m0 + (warp & 3) * 32 + rr < p.M) *reinterpret_cast<ulonglong2*>(dst + (size_t)rr * p.per) = make_ulonglong2(v[2 * i], v[2 * i + 1]);
          }
          __syncwarp();
        }
        tc_fence_before();
        if (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&bars->acc_empty[buf]), 0));
        else mbar_arrive(&bars->acc_empty[buf]);
      } else {
        uint32_t r[128];
        tmem_ld32(t0, r); tmem_ld32(t0 + 32, r + 32); tmem_ld32(t0 + 64, r + 64); tmem_ld32(t0 + 96, r + 96);
        tc_wait_ld();
        tc_fence_before();                                         // accumulator read out: the MMA warp may refill it
        if (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&bars->acc_empty[buf]), 0));   // the issuer waits for both CTAs
        else mbar_arrive(&bars->acc_empty[buf]);
        if (!QKV && p.beta && n0 >= 2 * p.per) {
          if (m < p.M) {
#pragma unroll
            for (int i = 0; i < BETA_MAX; ++i)
              if (i < p.beta_n) p.beta[(size_t)m * p.beta_n + i] = gemm_sigmoid(__uint_as_float(r[i]));
          }
          continue;
        }
        __nv_bfloat16* dst_row;                                    // this thread's output row (128 bf16)
        uint8_t* ring_row = nullptr;
        if (QKV) {
          const int nh = n0 >> 7;                   // head slot among 3 H
          const int which = nh / p.H, h = nh - which * p.H;
          const bool do_norm = (p.flags & (which == 0 ? DAISY_NORM_Q : which == 1 ? DAISY_NORM_K : DAISY_NORM_V)) != 0;
          if (do_norm) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < 128; ++i) { const float x = __uint_as_float(r[i]); ss = fmaf(x, x, ss); }
            const float rs = rsqrtf(ss * (1.0f / 128.0f) + p.eps);
            if (p.rstd && m < p.M) p.rstd[(size_t)m * (3 * p.H) + nh] = rs;
#pragma unroll
            for (int i = 0; i < 128; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * rs);
          }
          if (rope) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i < 3) cp_async_wait<1>(); else cp_async_wait<0>();
              __syncwarp();
#pragma unroll
              for (int i4 = 0; i4 < 4; ++i4) {
                const uint32_t a0 = s_own + (i & 1) * 4096;
                const float4 c = ld_shared_f4(a0 + ((i4 ^ (lane & 7)) << 4)), s = ld_shared_f4(a0 + (((4 + i4) ^ (lane & 7)) << 4));
                const float cc[4] = {c.x, c.y, c.z, c.w}, sn[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int j = 16 * i + 4 * i4 + e;
                  const float a = __uint_as_float(r[j]), b2 = __uint_as_float(r[j + 64]);
                  r[j] = __float_as_uint(a * cc[e] + b2 * sn[e]);
                  r[j + 64] = __float_as_uint(b2 * cc[e] - a * sn[e]);
                }
              }
              __syncwarp();
              if (i < 2) fetch(i + 2);
            }
          }
          if (which == 2 && p.vn && m < p.M) {                      // (thread = row: the gated layers of a model are few)
            uint4* vd = reinterpret_cast<uint4*>(p.vn + ((size_t)m * p.H + h) * 128);
#pragma unroll
            for (int c = 0; c < 16; ++c)
              vd[c] = make_uint4(pack_bf16(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])), pack_bf16(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                                 pack_bf16(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])), pack_bf16(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
          }
          if (which == 2 && p.ve) {                                // value-embedding gate on the normalised v
            const float gte = 1.0f / (1.0f + __expf(-*p.ve_gate_logit));
            const uint4* vr = reinterpret_cast<const uint4*>(p.ve + (size_t)min(m, p.M - 1) * p.ve_ld + h * 128);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              float f[8];
              unpack8(vr[c], f);
#pragma unroll
              for (int e = 0; e < 8; ++e) r[8 * c + e] = __float_as_uint(gte * __uint_as_float(r[8 * c + e]) + (1.0f - gte) * f[e]);
            }
          }
          dst_row = p.out[which] + ((size_t)m * p.H + h) * 128;
          if (which >= 1 && p.ring[which - 1] && m < p.M) {        // this row's slot in the ring cache, if it is kept
            const int b = m / p.T, t = m - b * p.T;
            if (t >= p.ring_first)
              ring_row = reinterpret_cast<uint8_t*>(p.ring[which - 1]) + ((int64_t)b * p.r_sb + (int64_t)h * p.r_sh + (int64_t)(t % p.cap) * p.r_sr) * 2;
          }
        } else {
          const int prod = n0 / p.per;
          dst_row = p.c[prod] + (size_t)m * p.ldc + (n0 - prod * p.per);
        }
        // bf16 pack, then through the warp's staging rows so that each store instruction writes two whole rows
        uint4 ch[16];
#pragma unroll
        for (int c = 0; c < 16; ++c)
          ch[c] = make_uint4(pack_bf16(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])),
                             pack_bf16(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                             pack_bf16(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])),
                             pack_bf16(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
          if ((lane >> 4) == pass) {
#pragma unroll
            for (int c = 0; c < 16; ++c) *reinterpret_cast<uint4*>(stg + (lane & 15) * 256 + ((c ^ (lane & 15)) << 4)) = ch[c];
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = 2 * i + (lane >> 4);                    // staged row, = warp row 16 pass + rr
            const uint4 val = *reinterpret_cast<const uint4*>(stg + rr * 256 + (((lane & 15) ^ rr) << 4));
            const int src_lane = 16 * pass + rr;
            // the row's global address lives in the lane that owns the row
            const unsigned long long base = __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(dst_row), src_lane);
            const int mm = __shfl_sync(0xffffffffu, m, src_lane);
            if (mm < p.M) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(base) + (lane & 15) * 16) = val;
            if (QKV && p.ring[0]) {                         // warp-uniform: a ring is attached to this call
              const unsigned long long rb = __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(ring_row), src_lane);
              if (rb) {
                uint4 rv = val;
                if (p.ring_f16) {                                  // the ring keeps float16 rows
                  float f[8];
                  unpack8(val, f);
                  const __half2 h0 = __floats2half2_rn(f[0], f[1]), h1 = __floats2half2_rn(f[2], f[3]);
                  const __half2 h2 = __floats2half2_rn(f[4], f[5]), h3 = __floats2half2_rn(f[6], f[7]);
                  rv = make_uint4(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1),
                                  *reinterpret_cast<const uint32_t*>(&h2), *reinterpret_cast<const uint32_t*>(&h3));
                }
                *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(rb) + (lane & 15) * 16) = rv;
              }
            }
          }
          __syncwarp();
        }
      }
    }
  }

  tc_fence_before();
  if (PAIR) cluster_sync_all();                        // neither CTA leaves while the other may still read its operands
  else __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 2 * BN);
    else tmem_dealloc(tmem_base, 2 * BN);
  }
}


// ---------------------------------------------------------------------- few rows, or few columns
// One tile of at most 128 rows x BN columns per CTA, up to two CTAs to an SM: what these sizes need is the whole chip
// pulling operands, not products per byte.  In the QKV form (BN = 64) a cluster of two CTAs shares a head: CTA r holds the
// head's channels c0 .. c0 + 31 and their rotation partners 64 + c0 .., c0 = 32 r, so RoPE stays inside a thread and only
// each row's sum of squares travels (one float per row and CTA, through the cluster's shared memory).
// Launched as a dependent grid: barriers, TMEM and the hint that brings the weights into L2 come before the wait.
// Bound by latency: launch, first operands, epilogue.  131 x 2304 x 768 with norm and RoPE 17.0 us as one 256 x 256 tile per
// CTA pair, 11.1 as 128 x 128 tiles, 5.9 here; 64 x 6144 x 2048 (25 MB of weights) 110 us in the row-by-row kernel, 8.6 here.
// (A head cut in four, BN = 32, costs more in the exchange than it gains: 9.8 us.)
template <int BN>
struct SmallCfg {
  static constexpr int STAGE = G_A_BYTES + BN * GK * 2;
  static constexpr int MAX_NST = 220 * 1024 / STAGE < 12 ? 220 * 1024 / STAGE : 12;      // alone on its SM
  static constexpr int HALF_NST = 106 * 1024 / STAGE;                                    // two CTAs to an SM
  static constexpr int RANKS = 128 / BN;                                                 // QKV: CTAs to a head
  static constexpr int SMEM0 = 1024 + 1024 + 256;
};
struct GemmWeights { const __nv_bfloat16* p[GROUP]; };
struct SmallBars {
  uint64_t full[12], empty[12], acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

template <int BN, bool QKV>
__global__ void __launch_bounds__(G_SMALL_THREADS, 2)
small_gemm_kernel(const __grid_constant__ GemmMaps maps, const GemmParams p, const int nst,
                  const int tm, const GemmWeights w, const int64_t ldw, const int prefetch) {
  using Cfg = SmallCfg<BN>;
  static_assert(!QKV || BN == 64, "two CTAs to a head");
  constexpr int HB = BN / 2;
  extern __shared__ uint8_t gemm_smem_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(stages + nst * Cfg::STAGE);                     // [rank][row]: sums of squares
  SmallBars* bars = reinterpret_cast<SmallBars*>(part + 2 * 128);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kb_n = p.K / GK;
  const int nx = p.N / BN, bn = (int)blockIdx.x % nx, bm = (int)blockIdx.x / nx;
  const int rank = QKV ? bn % Cfg::RANKS : 0;
  const int nh = bn / Cfg::RANKS;                                                        // QKV: head slot among 3 H
  const int c0 = rank * HB;                                                              // and this CTA's channels of it
  const int m0 = bm * tm;                                                                // tm <= 128 rows of X a tile, a multiple of 8
  const int prod = QKV ? 0 : bn * BN / p.per;                                            // plain: which product
  const int w_lo = QKV ? nh * 128 + c0 : bn * BN - prod * p.per, w_hi = QKV ? w_lo + 64 : w_lo + HB;    // its weight rows: HB and HB

  if (threadIdx.x == 0) {
    for (int i = 0; i < nst; ++i) { mbar_init(&bars->full[i], 1); mbar_init(&bars->empty[i], 1); }
    mbar_init(&bars->acc_full, 1);
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 5) {
    tmem_alloc(&bars->tmem_base, BN);
    tmem_relinquish();
  } else if (prefetch && bm == 0 && threadIdx.x < BN) {
    const int wr = (int)threadIdx.x < HB ? w_lo + (int)threadIdx.x : w_hi + (int)threadIdx.x - HB;
    if (QKV || !p.beta || prod < 2 || wr < p.beta_n) l2_prefetch_bulk(w.p[prod] + (int64_t)wr * ldw, (uint32_t)p.K * 2u);
  }
  if (warp == 4 && lane == 0) { prefetch_tmap(&maps.x[prod]); prefetch_tmap(&maps.w[prod]); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (QKV) asm volatile("barrier.cluster.arrive.release;" ::: "memory");                 // (1) this CTA runs
  const uint32_t tmem_base = bars->tmem_base;
  if (p.order == 0) grid_dep_launch();
  if (p.order != daisy_host::ORDER_BEHIND) grid_dep_wait();
  if (p.order != 0) grid_dep_launch();

  if (warp < 5) {
    // ------------------------------------------------------------------ TMA producers: a turn of the loop takes one thread some
    // 450 cycles, so the epilogue's warps share it before the accumulator is theirs to read.  Never more producers than stages:
    // a producer enters block kb after block kb - np's stage was free, so product kb - np - nst is done; with np <= nst that is
    // no earlier than product kb - 2 nst, and the parity it waits for cannot be that of the round before the last.
    const int np = min(5, nst);
    if (lane == 0 && warp < np) {
      for (int kb = warp; kb < kb_n; kb += np) {
        const int st = kb % nst;
        if (!mbar_wait(&bars->empty[st], ((kb / nst) & 1) ^ 1, abort_flag, p.status, 1)) break;
        uint8_t* dst = stages + st * Cfg::STAGE;
        mbar_expect_tx(&bars->full[st], tm * GK * 2 + BN * GK * 2);
        tma_load_3d(dst + G_A_BYTES, &maps.w[prod], &bars->full[st], kb * GK, w_lo, 0);
        tma_load_3d(dst + G_A_BYTES + HB * GK * 2, &maps.w[prod], &bars->full[st], kb * GK, w_hi, 0);
        tma_load_3d(dst, &maps.x[prod], &bars->full[st], kb * GK, m0, 0);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = umma_idesc_bf16(GM, BN, 0, 0);
    const uint64_t ad = umma_desc_sw128(smem_u32(stages), 16, 1024);
    const uint64_t bd = umma_desc_sw128(smem_u32(stages + G_A_BYTES), 16, 1024);
    const uint32_t a_lo0 = (uint32_t)ad, b_lo0 = (uint32_t)bd, hi = (uint32_t)(ad >> 32);
    bool ok = true;
    for (int kb = 0, st = 0, ph = 0; kb < kb_n; ++kb) {
      if (!mbar_wait(&bars->full[st], ph, abort_flag, p.status, 3)) { ok = false; break; }
      tc_fence_after();
      const uint32_t a_lo = a_lo0 + st * (Cfg::STAGE >> 4), b_lo = b_lo0 + st * (Cfg::STAGE >> 4);
#pragma unroll
      for (int k = 0; k < GK / 16; ++k) umma_ss_lh_p(leader, tmem_base, a_lo + k * 2, hi, b_lo + k * 2, hi, idesc, (kb > 0 || k > 0) ? 1u : 0u);
      tc_commit_p(leader, &bars->empty[st]);
      if (++st == nst) { st = 0; ph ^= 1; }
    }
    if (ok) tc_commit_p(leader, &bars->acc_full);
    __syncwarp();
  }

  if (warp < 4) {
    // ------------------------------------------------------------------ epilogue: thread = output row, r[0 .. HB) low, r[HB ..) high columns
    const int row = warp * 32 + lane, m = m0 + row;
    const int which = nh / p.H, h = nh - which * p.H;                                    // QKV only
    const bool rope = QKV && which < 2 && (p.flags & DAISY_ROPE);
    float4 cs[HB / 4], sn[HB / 4];
    if (rope) {                                                                          // rotations arrive under the products
      const int pos = min(m, p.M - 1) % p.T;
      const float4* cr = reinterpret_cast<const float4*>(p.cos + (size_t)pos * 64 + c0);
      const float4* sr = reinterpret_cast<const float4*>(p.sin + (size_t)pos * 64 + c0);
#pragma unroll
      for (int i = 0; i < HB / 4; ++i) { cs[i] = cr[i]; sn[i] = sr[i]; }
    }
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, 0, abort_flag, p.status, 4)), mine = ok && row < tm && m < p.M;
    tc_fence_after();
    uint32_t r[BN];
    const uint32_t t0 = tmem_base + ((uint32_t)(warp * 32) << 16);
#pragma unroll
    for (int i = 0; i < BN / 32; ++i) tmem_ld32(t0 + 32 * i, r + 32 * i);
    tc_wait_ld();
    if (QKV) {
      const bool do_norm = (p.flags & (which == 0 ? DAISY_NORM_Q : which == 1 ? DAISY_NORM_K : DAISY_NORM_V)) != 0;
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < BN; ++i) { const float x = __uint_as_float(r[i]); ss = fmaf(x, x, ss); }
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");                        // (1) both of the head's CTAs run
#pragma unroll
      for (int j = 0; j < Cfg::RANKS; ++j)
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_shared(smem_u32(part + rank * 128 + row), j)), "f"(ss) : "memory");
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");   // (2)
      ss = 0.f;
#pragma unroll
      for (int j = 0; j < Cfg::RANKS; ++j) ss += part[j * 128 + row];
      if (do_norm) {
        const float rs = rsqrtf(ss * (1.0f / 128.0f) + p.eps);
        if (p.rstd && rank == 0 && mine) p.rstd[(size_t)m * (3 * p.H) + nh] = rs;
#pragma unroll
        for (int i = 0; i < BN; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * rs);
      }
      if (rope) {
#pragma unroll
        for (int i4 = 0; i4 < HB / 4; ++i4) {
          const float cc[4] = {cs[i4].x, cs[i4].y, cs[i4].z, cs[i4].w}, sc[4] = {sn[i4].x, sn[i4].y, sn[i4].z, sn[i4].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = 4 * i4 + e;
            const float a = __uint_as_float(r[i]), b2 = __uint_as_float(r[i + HB]);
            r[i] = __float_as_uint(a * cc[e] + b2 * sc[e]);
            r[i + HB] = __float_as_uint(b2 * cc[e] - a * sc[e]);
          }
        }
      }
    }
    if (!QKV && p.gate && prod == 0) {
      if (mine) {
        const float a = -expf(__ldg(p.a_log + (w_lo >> 7)));
        float4* d = reinterpret_cast<float4*>(p.gate + (size_t)m * p.per + w_lo);
        const float4* bp = reinterpret_cast<const float4*>(p.dt_bias + w_lo);
#pragma unroll
        for (int i = 0; i < BN / 4; ++i) {
          const float4 bias = __ldg(bp + i);
          const uint64_t bias2[2] = {pack2f(bias.x, bias.y), pack2f(bias.z, bias.w)};
          uint64_t v[2] = {pack2f(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1])), pack2f(__uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]))};
          gemm_decay2(v, bias2, a);
          *reinterpret_cast<ulonglong2*>(d + i) = make_ulonglong2(v[0], v[1]);
        }
      }
    } else if (!QKV && p.beta && prod == 2) {
      if (mine) {
#pragma unroll
        for (int i = 0; i < (BN < BETA_MAX ? BN : BETA_MAX); ++i)
          if (w_lo + i < p.beta_n) p.beta[(size_t)m * p.beta_n + w_lo + i] = gemm_sigmoid(__uint_as_float(r[i]));
      }
    } else if (mine) {
      uint32_t hv[HB];                                                                   // bf16 pairs: HB / 2 low, HB / 2 high
      const bool gated = QKV && which == 2 && p.ve;
      // where the high columns follow the low ones, in 16-byte units
      constexpr int HI = QKV ? 8 : HB / 8;
      auto store = [&](void* at) {
        uint4* d = reinterpret_cast<uint4*>(at);
#pragma unroll
        for (int i = 0; i < HB / 8; ++i) {
          d[i] = make_uint4(hv[4 * i], hv[4 * i + 1], hv[4 * i + 2], hv[4 * i + 3]);
          d[HI + i] = make_uint4(hv[HB / 2 + 4 * i], hv[HB / 2 + 4 * i + 1], hv[HB / 2 + 4 * i + 2], hv[HB / 2 + 4 * i + 3]);
        }
      };
      if (gated) {                                                                       // value-embedding gate on the normalised v
        if (p.vn) {
#pragma unroll
          for (int i = 0; i < HB; ++i) hv[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          store(p.vn + ((size_t)m * p.H + h) * 128 + c0);
        }
        const float gte = 1.0f / (1.0f + __expf(-*p.ve_gate_logit));
        const uint4* vr = reinterpret_cast<const uint4*>(p.ve + (size_t)m * p.ve_ld + h * 128 + c0);
#pragma unroll
        for (int c = 0; c < HB / 4; ++c) {
          float f[8];
          unpack8(c < HB / 8 ? vr[c] : vr[8 + c - HB / 8], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) r[8 * c + e] = __float_as_uint(gte * __uint_as_float(r[8 * c + e]) + (1.0f - gte) * f[e]);
        }
      }
#pragma unroll
      for (int i = 0; i < HB; ++i) hv[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      store(QKV ? p.out[which] + ((size_t)m * p.H + h) * 128 + c0 : p.c[prod] + (size_t)m * p.ldc + w_lo);
      if (QKV && which >= 1 && p.ring[which - 1]) {                                      // this row's slot in the ring cache, if it is kept
        const int b = m / p.T, t = m - b * p.T;
        if (t >= p.ring_first) {
          if (p.ring_f16) {                                                              // the bf16 value as float16
#pragma unroll
            for (int i = 0; i < HB; ++i) {
              const __half2 x = __floats2half2_rn(bf16_lo(hv[i]), bf16_hi(hv[i]));
              hv[i] = *reinterpret_cast<const uint32_t*>(&x);
            }
          }
          store(reinterpret_cast<__nv_bfloat16*>(p.ring[which - 1]) + (int64_t)b * p.r_sb + (int64_t)h * p.r_sh + (int64_t)(t % p.cap) * p.r_sr + c0);
        }
      }
    }
  } else if (QKV) {
    asm volatile("barrier.cluster.wait.acquire;\n\tbarrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");   // (1), (2)
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
  if (p.order == daisy_host::ORDER_BEHIND && blockIdx.x == gridDim.x - 1) grid_dep_wait();
}

}  // namespace daisy

using namespace daisy;

template <int BN, bool PAIR, bool QKV>
static int launch_gemm(const GemmMaps& maps, const GemmParams& p, cudaStream_t st) {
  using Cfg = GemmCfg<BN, PAIR, QKV>;
  static_assert(Cfg::SMEM <= 232448, "over the 227 KB a CTA may use");
  static bool attr[daisy_host::MAX_DEVICES] = {};
  static int max_clusters[daisy_host::MAX_DEVICES] = {};
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(G_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = PAIR ? 2 : 1;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(qkv_gemm_kernel<BN, PAIR, QKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    if (PAIR) {                                          // how many CTA pairs the device can hold at once
      cfg.gridDim = dim3((unsigned)(sms & ~1));
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, qkv_gemm_kernel<BN, PAIR, QKV>, &cfg) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        return DAISY_ECUDA;
      }
      max_clusters[dev] = n;
    }
    attr[dev] = true;
  }
  const int64_t tiles = (int64_t)((p.M + Cfg::TILE_M - 1) / Cfg::TILE_M) * (p.N / BN);
  if (PAIR) {
    const int64_t pairs = tiles < max_clusters[dev] ? tiles : max_clusters[dev];
    cfg.gridDim = dim3((unsigned)(2 * pairs));
  } else {
    cfg.gridDim = dim3((unsigned)(tiles < sms ? tiles : sms));
  }
  if (cudaLaunchKernelEx(&cfg, qkv_gemm_kernel<BN, PAIR, QKV>, maps, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return DAISY_ECUDA;
  }
  DAISY_CHECK_LAUNCH();
  return DAISY_OK;
}

static int make_maps(GemmMaps& maps, const void* const* x, int64_t ldx, int x_rows, const void* const* w, int64_t ldw, int w_rows, int n, const GemmParams& p) {
  for (int i = 0; i < n; ++i) {
    int rc = daisy_host::make_tmap_bf16_3d(&maps.x[i], x[i], p.K, p.M, 1, (uint64_t)ldx * 2, (uint64_t)ldx * 2 * p.M, GK, x_rows);
    if (rc != DAISY_OK) return rc;
    const int rows = p.beta && i == 2 ? p.beta_n : p.per;              // rows past the last read as zeros
    rc = daisy_host::make_tmap_bf16_3d(&maps.w[i], w[i], p.K, rows, 1, (uint64_t)ldw * 2, (uint64_t)ldw * 2 * rows, GK, w_rows);
    if (rc != DAISY_OK) return rc;
  }
  for (int i = n; i < GROUP; ++i) { maps.x[i] = maps.x[0]; maps.w[i] = maps.w[0]; }
  return DAISY_OK;
}

constexpr size_t G_PREFETCH_LIMIT = 48u << 20;          // weights up to this size are hinted into L2 ahead of the wait

template <int BN, bool QKV>
static int launch_small(const void* const* x, int64_t ldx, const void* const* w, int64_t ldw, int n, const GemmParams& p, cudaStream_t st) {
  using Cfg = SmallCfg<BN>;
  auto kernel = small_gemm_kernel<BN, QKV>;
  static bool attr[daisy_host::MAX_DEVICES] = {};
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM0 + Cfg::MAX_NST * Cfg::STAGE) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    attr[dev] = true;
  }
  // tiles of equal height: 131 rows are two tiles of 72, not one of 128 and one of 3
  const int mt = (p.M - 1) / GM + 1, tm = ((p.M - 1) / mt + 8) & ~7;
  GemmMaps maps;
  GemmWeights wp{};
  const int rc = make_maps(maps, x, ldx, tm, w, ldw, BN / 2, n, p);
  if (rc != DAISY_OK) return rc;
  for (int i = 0; i < n; ++i) wp.p[i] = (const __nv_bfloat16*)w[i];
  const int tiles = mt * (p.N / BN);
  int nst = tiles <= sms ? Cfg::MAX_NST : Cfg::HALF_NST;
  if (nst > p.K / GK) nst = p.K / GK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles); cfg.blockDim = dim3(G_SMALL_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM0 + nst * Cfg::STAGE; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = Cfg::RANKS; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = QKV ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, maps, p, nst, tm, wp, ldw, (size_t)p.N * p.K * 2 <= G_PREFETCH_LIMIT ? 1 : 0) != cudaSuccess) {
    (void)cudaGetLastError();
    return DAISY_ECUDA;
  }
  DAISY_CHECK_LAUNCH();
  return DAISY_OK;
}

// Which tile.  One wave of narrow tiles as long as they fit the chip (a second wave costs more than wider tiles do:
// 2048 x 768 x 768 7.5 us in 128-column tiles, 8.4 in 64).  From there 128 x 128 tiles against pairs on 256 x 256, by what a
// wave of either was measured to take: a pair's wave is twice the work at 0.7 of the time per product, with a longer start
// and end (ns; 1024 x 2048 x 2048 12.4 against 16.9 us, 2048 x 6144 x 2048 51 against 42, 65536 x 768 x 768 80 against 67).
enum { TILE_32 = 32, TILE_64 = 64, TILE_128 = 128, TILE_PAIR = 256 };
static int gemm_tile(const GemmParams& p, int sms) {
  const int64_t mt = ((int64_t)p.M + GM - 1) / GM;
  if (p.epi == 0 && mt * (p.N / 32) <= sms) return TILE_32;
  if (mt * (p.N / 64) <= sms) return TILE_64;
  if (p.per % 256 != 0) return TILE_128;
  const int64_t w1 = (mt * (p.N / 128) + sms - 1) / sms, w2 = ((mt + 1) / 2 * (p.N / 256) + sms / 2 - 1) / (sms / 2);
  return 4000 + w1 * (37ll * p.K / 10 + 1000) < 7000 + w2 * (53ll * p.K / 10 + 2000) ? TILE_128 : TILE_PAIR;
}

// n products of one shape; p.N counts all their columns, p.per one's
static int gemm_common(const void* const* x, int64_t ldx, const void* const* w, int64_t ldw, int n, GemmParams& p, void* stream) {
  if (p.M <= 0 || p.per <= 0 || p.K <= 0) return DAISY_EINVAL;
  for (int i = 0; i < n; ++i) if (!x[i] || !w[i]) return DAISY_EINVAL;
  if (p.K % GK != 0 || p.per % 128 != 0) return DAISY_EUNSUPPORTED;
  for (int i = 0; i < n; ++i) if (!daisy_aligned16(x[i]) || !daisy_aligned16(w[i])) return DAISY_EALIGN;
  if ((ldx & 7) || (ldw & 7) || ldx < p.K || ldw < p.K) return DAISY_EALIGN;
  p.N = n * p.per;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  cudaStream_t st = (cudaStream_t)stream;
  const int tile = gemm_tile(p, sms);
  if (tile != TILE_32 && tile != TILE_64) p.order = 0;
  if (tile == TILE_32) return launch_small<32, false>(x, ldx, w, ldw, n, p, st);
  if (tile == TILE_64) return p.epi ? launch_small<64, true>(x, ldx, w, ldw, n, p, st) : launch_small<64, false>(x, ldx, w, ldw, n, p, st);
  GemmMaps maps;
  const int rc = make_maps(maps, x, ldx, GM, w, ldw, 128, n, p);
  if (rc != DAISY_OK) return rc;
  if (tile == TILE_PAIR) return p.epi ? launch_gemm<256, true, true>(maps, p, st) : launch_gemm<256, true, false>(maps, p, st);
  return p.epi ? launch_gemm<128, false, true>(maps, p, st) : launch_gemm<128, false, false>(maps, p, st);
}

int daisy_host::gemm_group(const void* const* x, int64_t ldx, const void* const* w, int64_t ldw, void* const* c, int64_t ldc,
                           int n, int M, int N, int K, int* order, int* status_word, void* stream) {
  if (!x || !w || !c || n < 1 || n > GROUP) return DAISY_EINVAL;
  GemmParams p{};
  p.M = M; p.per = N; p.K = K; p.epi = 0; p.ldc = ldc; p.status = status_word;
  for (int i = 0; i < n; ++i) {
    if (!c[i]) return DAISY_EINVAL;
    if (!daisy_aligned16(c[i])) return DAISY_EALIGN;
    p.c[i] = (__nv_bfloat16*)c[i];
  }
  if ((ldc & 7) || ldc < N) return DAISY_EALIGN;
  p.order = *order;
  const int rc = gemm_common(x, ldx, w, ldw, n, p, stream);
  *order = p.order;
  return rc;
}

extern "C" int daisy_b200_gemm_nt_group(const void* const* x, int64_t ldx, const void* const* w, int64_t ldw, void* const* c, int64_t ldc,
                                        int n, int M, int N, int K, int* status_word, void* stream) {
  int order = 0;
  return daisy_host::gemm_group(x, ldx, w, ldw, c, ldc, n, M, N, K, &order, status_word, stream);
}

extern "C" int daisy_b200_kda_low_rank(const void* x, int64_t ldx, const void* f0_w, const void* g0_w, const void* b_w, void* f0, void* g0, float* beta,
                                       int M, int H, int dim, int* status_word, void* stream) {
  if (!f0 || !g0 || !beta || H <= 0) return DAISY_EINVAL;
  if (H > BETA_MAX) return DAISY_EUNSUPPORTED;
  if (!daisy_aligned16(f0) || !daisy_aligned16(g0)) return DAISY_EALIGN;
  const void *xs[3] = {x, x, x}, *w[3] = {f0_w, g0_w, b_w};
  GemmParams p{};
  p.M = M; p.per = 128; p.K = dim; p.ldc = 128; p.status = status_word;
  p.c[0] = (__nv_bfloat16*)f0; p.c[1] = (__nv_bfloat16*)g0; p.beta = beta; p.beta_n = H;
  return gemm_common(xs, ldx, w, dim, 3, p, stream);
}

extern "C" int daisy_b200_kda_gates(const void* f0, const void* g0, const void* f1_w, const void* g1_w, const float* a_log, const float* dt_bias,
                                    float* g, void* gate, int M, int H, int* status_word, void* stream) {
  if (!a_log || !dt_bias || !g || !gate || H <= 0) return DAISY_EINVAL;
  if (!daisy_aligned16(dt_bias) || !daisy_aligned16(g) || !daisy_aligned16(gate)) return DAISY_EALIGN;
  const void *xs[2] = {f0, g0}, *w[2] = {f1_w, g1_w};
  GemmParams p{};
  p.M = M; p.per = H * 128; p.K = 128; p.ldc = p.per; p.status = status_word;
  p.c[1] = (__nv_bfloat16*)gate; p.gate = g; p.a_log = a_log; p.dt_bias = dt_bias;
  return gemm_common(xs, 128, w, 128, 2, p, stream);
}

extern "C" int daisy_b200_gemm_nt(const void* x, int64_t ldx, const void* w, int64_t ldw, void* c, int64_t ldc,
                                  int M, int N, int K, int* status_word, void* stream) {
  return daisy_b200_gemm_nt_group(&x, ldx, &w, ldw, &c, ldc, 1, M, N, K, status_word, stream);
}

static int qkv_gemm_launch(const void* x, int64_t ldx, const void* w_qkv, int64_t ldw, const float* cos, const float* sin,
                           void* q_out, void* k_out, void* v_out, const void* ve, int64_t ve_ld, const float* ve_gate_logit,
                           void* ring_k, void* ring_v, int64_t r_sb, int64_t r_sh, int64_t r_sr, int cap, int ring_first,
                           float* rstd, void* vn, int B, int T, int H, int D, int dim, float eps, unsigned flags,
                           int* status_word, void* stream) {
  if (!q_out || !k_out || !v_out || B <= 0 || T <= 0 || H <= 0) return DAISY_EINVAL;
  if (D != DAISY_HEAD_DIM) return DAISY_EUNSUPPORTED;
  if ((int64_t)B * T >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  if (flags & ~(DAISY_QKV_DEFAULT | DAISY_CACHE_FP16)) return DAISY_EINVAL;
  if ((ring_k == nullptr) != (ring_v == nullptr)) return DAISY_EINVAL;
  if (ring_k) {
    if (cap <= 0 || ring_first < 0 || T - ring_first > cap) return DAISY_EINVAL;          // the kept rows would alias in the ring
    if (!daisy_aligned16(ring_k) || !daisy_aligned16(ring_v) || ((r_sb | r_sh | r_sr) & 7)) return DAISY_EALIGN;
  }
  if ((flags & DAISY_ROPE) && (!cos || !sin)) return DAISY_EINVAL;
  if ((flags & DAISY_ROPE) && (!daisy_aligned16(cos) || !daisy_aligned16(sin))) return DAISY_EALIGN;
  if (!daisy_aligned16(q_out) || !daisy_aligned16(k_out) || !daisy_aligned16(v_out)) return DAISY_EALIGN;
  if (ve && (!ve_gate_logit || !daisy_aligned16(ve) || (ve_ld & 7) || ve_ld < (int64_t)H * D)) return ve_gate_logit ? DAISY_EALIGN : DAISY_EINVAL;
  GemmParams p{};
  p.ve = (const __nv_bfloat16*)ve; p.ve_ld = ve_ld; p.ve_gate_logit = ve_gate_logit;
  p.M = B * T; p.per = 3 * H * D; p.K = dim; p.epi = 1;
  p.out[0] = (__nv_bfloat16*)q_out; p.out[1] = (__nv_bfloat16*)k_out; p.out[2] = (__nv_bfloat16*)v_out;
  p.cos = cos; p.sin = sin; p.T = T; p.H = H; p.eps = eps; p.flags = flags & DAISY_QKV_DEFAULT; p.status = status_word;
  p.ring[0] = ring_k; p.ring[1] = ring_v; p.r_sb = r_sb; p.r_sh = r_sh; p.r_sr = r_sr;
  p.rstd = rstd; p.vn = (__nv_bfloat16*)vn;
  p.cap = cap; p.ring_first = ring_first; p.ring_f16 = (flags & DAISY_CACHE_FP16) ? 1 : 0;
  return gemm_common(&x, ldx, &w_qkv, ldw, 1, p, stream);
}

extern "C" int daisy_b200_qkv_gemm(const void* x, int64_t ldx, const void* w_qkv, int64_t ldw,
                                   const float* cos, const float* sin,
                                   void* q_out, void* k_out, void* v_out,
                                   const void* ve, int64_t ve_ld, const float* ve_gate_logit,
                                   int B, int T, int H, int D, int dim, float eps, unsigned flags,
                                   int* status_word, void* stream) {
  return qkv_gemm_launch(x, ldx, w_qkv, ldw, cos, sin, q_out, k_out, v_out, ve, ve_ld, ve_gate_logit,
                         nullptr, nullptr, 0, 0, 0, 0, 0, nullptr, nullptr, B, T, H, D, dim, eps, flags, status_word, stream);
}

extern "C" int daisy_b200_qkv_gemm_ring(const void* x, int64_t ldx, const void* w_qkv, int64_t ldw,
                                        const float* cos, const float* sin,
                                        void* q_out, void* k_out, void* v_out,
                                        const void* ve, int64_t ve_ld, const float* ve_gate_logit,
                                        void* ring_k, void* ring_v, int64_t r_sb, int64_t r_sh, int64_t r_sr,
                                        int cap, int ring_first,
                                        int B, int T, int H, int D, int dim, float eps, unsigned flags,
                                        int* status_word, void* stream) {
  return qkv_gemm_launch(x, ldx, w_qkv, ldw, cos, sin, q_out, k_out, v_out, ve, ve_ld, ve_gate_logit,
                         ring_k, ring_v, r_sb, r_sh, r_sr, cap, ring_first, nullptr, nullptr, B, T, H, D, dim, eps, flags, status_word, stream);
}

extern "C" int daisy_b200_qkv_gemm_train(const void* x, int64_t ldx, const void* w_qkv, int64_t ldw,
                                         const float* cos, const float* sin,
                                         void* q_out, void* k_out, void* v_out, float* rstd, void* vn_out,
                                         const void* ve, int64_t ve_ld, const float* ve_gate_logit,
                                         int B, int T, int H, int D, int dim, float eps, unsigned flags,
                                         int* status_word, void* stream) {
  if (!rstd || (ve != nullptr) != (vn_out != nullptr) || (flags & DAISY_QKV_DEFAULT) != DAISY_QKV_DEFAULT) return DAISY_EINVAL;
  if (!daisy_aligned16(vn_out)) return DAISY_EALIGN;
  return qkv_gemm_launch(x, ldx, w_qkv, ldw, cos, sin, q_out, k_out, v_out, ve, ve_ld, ve_gate_logit,
                         nullptr, nullptr, 0, 0, 0, 0, 0, rstd, vn_out, B, T, H, D, dim, eps, flags, status_word, stream);
}
