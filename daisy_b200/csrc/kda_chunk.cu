// Kimi delta attention (KDA), chunked forward, chunk = 64, K = V = 128.
//
// Per head the recurrence  S <- diag(e^{g_t}) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;
// o_t = S^T (scale q_t)  is evaluated 64 tokens at a time.  With G_i the inclusive cumulative
// log-decay inside a chunk and S_0 the state entering it:
//     A_kk[i,j] = beta_i sum_c k_ic k_jc e^{G_ic-G_jc} (j < i)     A_qk[i,j] = scale sum_c q_ic k_jc e^{G_ic-G_jc} (j <= i)
//     T = (I + A_kk)^-1          W = T (beta k e^G)          U0 = T (beta v)
//     U = U0 - W S_0             O = (scale q e^G) S_0 + A_qk U          S_C = e^{G_C} S_0 + (k e^{G_C-G})^T U
// Two kernels, on long rows in several parts that run beside one another (kda_split):
//  * kda_intra_kernel  -- everything that does not depend on the state, a small CTA per (batch, head, chunk), three to an SM:
//    Gram products in mma.sync fragments, the blocked solve of (I + A_kk) W = beta k e^G, (I + A_kk) U0 = beta v in register
//    chains.  Per chunk it writes a record of fp16 operand images (16-byte pieces exchanged so that fragment loads are
//    bank-conflict free): W^T, scale q e^G, k e^{G_C-G}, A_qk, U0^T, and e^{G_C}.
//  * kda_state_kernel  -- one CTA per (batch, head), sequential over chunks, on tcgen05: the state in registers, fp16 operands
//    and sums in TMEM, the records through rings in shared memory.
// Tensor-core operands are fp16 (10-bit mantissa, every decay factor and operand here is <= O(1)):
// measured relative error of o against the fp32 token recurrence is ~4e-4, bf16 operands give ~3e-3.
#include <cuda_fp16.h>
#include <type_traits>
#include "common.cuh"

namespace daisy {

constexpr int KC = 64;                 // chunk length
constexpr int KD = 128;                // K = V
// per-chunk record in the workspace (bytes); after a plain bulk copy every image is a 128-byte-swizzled tcgen05 operand: rows of
// 64 fp16 whose 16-byte pieces are exchanged by row (rec_off, panel_off)
constexpr int OFF_WT = 0;                              // W^T      [128 channels][64 tokens] fp16
constexpr int OFF_QT = OFF_WT + KD * KC * 2;           // q~       [2][64 tokens][64 channels] fp16   scale q e^G
constexpr int OFF_KT = OFF_QT + KD * KC * 2;           // k~       [2][64 tokens][64 channels] fp16   k e^{G_C-G}
constexpr int OFF_AQK = OFF_KT + KD * KC * 2;          // A_qk     [64][64]  fp16
constexpr int OFF_D = OFF_AQK + KC * KC * 2;           // e^{G_C}  [128]     fp32
constexpr int SHARED_BYTES = OFF_D + KD * 4;           // 57856: up to here what the state is multiplied with; then what is added
constexpr int OFF_UT = SHARED_BYTES;                   // U0^T     [128 value columns][64 tokens] fp16
constexpr int REC_BYTES = OFF_UT + KD * KC * 2;        // 74240
static_assert(SHARED_BYTES % 16 == 0 && REC_BYTES % 16 == 0, "bulk copies move 16-byte units");
// what a caller provides per record: part of the ABI, from when records had padded rows; the record uses the front of the buffer
constexpr size_t WS_REC_BYTES = 83456;
static_assert(REC_BYTES <= WS_REC_BYTES, "a record fits what callers provide");

// byte offset of (row, token column) in an image of 64-token rows (128 bytes, 16-byte pieces exchanged by row)
__device__ __forceinline__ uint32_t rec_off(int row, int col) { return (uint32_t)(row * 128 + (((col >> 3) ^ (row & 7)) << 4) + (col & 7) * 2); }
// byte offset of 16-byte piece c (0..15) of a 128-channel row kept as two panels of 64 channels
__device__ __forceinline__ uint32_t panel_off(int row, int c) { return (uint32_t)((c >> 3) * (KC * 128) + row * 128 + (((c ^ row) & 7) << 4)); }

// Four 8x8 fp16 matrices from shared memory: lanes 8m..8m+7 give the row addresses of matrix m (16 bytes per
// row); register m of lane l then holds elements (row l/4, columns 2(l%4), 2(l%4)+1) of matrix m -- the B
// fragment layout of mma.m16n8k16 when the rows are the n index and the columns the k index.
__device__ __forceinline__ void ldmatrix_x4(uint32_t* r, uint32_t row_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(row_addr));
}
// The transposing form: register m of lane l holds elements (rows 2(l%4), 2(l%4)+1, column l/4) of matrix m --
// the same B fragment when the stored rows are the k index and the columns the n index.
__device__ __forceinline__ void ldmatrix_x4_t(uint32_t* r, uint32_t row_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(row_addr));
}

__device__ __forceinline__ void mma_f16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_h2(uint64_t v) {
  float lo, hi;
  unpack2f(v, lo, hi);
  return pack_h2(lo, hi);
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float2 unpack_h2(uint32_t u) {
  return __half22float2(*reinterpret_cast<__half2*>(&u));
}
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void st_global16(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// =============================================================================================
// intra-chunk kernel
// =============================================================================================
//
// Gated Gram matrices without a single positive exponent.  e^{G_i - G_j} (i > j) is needed per channel inside the
// contraction over channels, so it must factor into a row term times a column term, and neither term may overflow
// whatever the gates are.
//   * Between different 16-token blocks I > J:  e^{G_i - G_j} = e^{G_i - G_{end J}} e^{G_{end J} - G_j}: the column term is
//     the product of the decays d_t = e^{g_t} <= 1 behind j inside its block (`suf`), the row term the product up to i
//     inside its block (`pre`) times the totals of the blocks between.
//   * Inside a block, pairs are split by the highest bit in which i and j differ ("level" s = 1, 2, 4, 8): i lies in the
//     upper, j in the lower half of an aligned group of 2s tokens, and the same identity holds with the group's middle.
// Every factor is a running product of numbers <= 1 -- ONE exponential per input element, no cumulative sum, and underflow
// is the correct limit.
//
// A CTA of four warps owns one (batch, head, chunk), warp w the tokens 16 w .. 16 w + 15, three CTAs to an SM.  The running
// products are taken with lane = two channels, all 16 tokens in registers (which half of a group a token is in is then
// known at compile time, and no product crosses a lane), 64 channels at a time.  A level's images k f, q f go through 4 KB of
// the warp's own shared memory into m16n8k16 fragments: k and q rows of an octet are stacked into one A operand, two of
// whose four registers are also the B operand, so a level costs one ldmatrix and one product per octet and 16 channels.
// The norms are diagonals of the raw bf16 products, formed the same way.  Blocks meet only through their `suf` images and
// their totals.  Then the four diagonal blocks of I + A_kk are inverted (fp32, one per warp) and W, U0 come from a blocked
// forward substitution on the transposed systems, a warp owning 64 of the 256 rows (see below).
// What bounds it: 22k warp instructions a chunk at some 45 % issue with 12 warps on an SM, latency between.  Rows of k, q and g
// by asynchronous copies before the first wait instead of register loads where they are used: 447 -> 374 us at 4 x 8192 x 16;
// the six products between blocks two to a warp instead of three for the last and none for the first: 357; the halves and the
// solve's tiles rolled, which ended the spills and most waits for instructions: 326.  Lane =
// (2 tokens, 8 channels), as the fragments want it, costs three shuffles and twice the selects per product: 27k instructions.
// Why not tcgen05: the version of this kernel that built six image sets in shared memory for 128 x 64 x 128 tcgen05 products
// was a chain of hand-offs between warp groups (image -> fence -> product -> TMEM load), 20k cycles a chunk with the tensor
// pipe at 10 %; here everything between two barriers stays inside one warp and three CTAs hide each other's latency.
struct KdaIntraParams {
  const __nv_bfloat16 *q, *k, *v;
  const float *g, *beta;
  uint8_t* ws;
  int T, H, NC;            // NC = chunks per sequence
  int c0, behind;          // first chunk of this launch; behind: it runs beside the state's pass over the chunks before (kda_split)
  float scale;
  int l2norm;
  // packed variable-length sequences (B = 1): chunk c of the packed row covers tokens chunk_tab[2c] .. + chunk_tab[2c+1]
  // (1..64 of them; chunks never straddle a sequence boundary); null: chunk c covers tokens 64 c ..
  const int* chunk_tab;
};

constexpr int KI_THREADS = 128;
constexpr int LDAK = 72;                                // halves per row of the A_kk image
constexpr int KI_LD = 256 + 16, KI_LV = 128 + 16;       // bytes between rows of a block's image, and of a level's (64 channels)
struct KdaIntraSmem {
  // each block's k suf, k pre, q pre: [block], 16 token rows of 256 bytes, 16 bytes apart (conflict-free for whole rows and for
  // ldmatrix, with addresses that are constants plus one register).  pk and pq hold the raw rows before and are read by their
  // own warp only, which lays k e^G and its v rows over them afterwards; suf is the level images' room before
  uint8_t suf[4][2 * 16 * KI_LV], pk[4][16 * KI_LD], pq[4][16 * KI_LD];
  __half akh[KC][LDAK];                                 // beta A_kk below the diagonal blocks
  float dg[4][16][20];                                  // beta A_kk, the diagonal blocks, column-major ([j][i])
  __half th[4][16][24];                                 // their inverses (of I + A_kk), row-major
  float tot[4][KD];                                     // product of the decays of each block
  float nrm[4][3][16];                                  // 1 / |k|, 1 / |q|, normalised q . k of each token
  float beta[KC];
};

__device__ __forceinline__ void ki_chunk_span(const int* chunk_tab, int chunk, int T, int& t0, int& rows) {
  if (chunk_tab) { t0 = chunk_tab[2 * chunk]; rows = chunk_tab[2 * chunk + 1]; }
  else { t0 = chunk * KC; rows = min(KC, T - t0); }
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// two fp16 values times fp32 factors, one rounding
__device__ __forceinline__ uint32_t ki_scale(uint32_t a, const float2 f) {
  const float2 x = unpack_h2(a);
  return pack_h2(fmul2(pack2f(x.x, x.y), pack2f(f.x, f.y)));
}
__global__ void __launch_bounds__(KI_THREADS, 3) kda_intra_kernel(const KdaIntraParams p) {
  extern __shared__ __align__(128) uint8_t kda_smem_raw[];
  KdaIntraSmem& sm = *reinterpret_cast<KdaIntraSmem*>(kda_smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
  const int chunk = p.c0 + blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  if (!p.behind) grid_dep_wait();
  grid_dep_launch();
  int t0, rows;
  ki_chunk_span(p.chunk_tab, chunk, p.T, t0, rows);
  if (rows <= 0) return;                                                           // a table made for as many chunks as there can be
  uint8_t* rec = p.ws + ((size_t)(b * p.H + h) * p.NC + chunk) * REC_BYTES;
  const size_t tok = ((size_t)b * p.T + t0) * p.H + h, ts = (size_t)p.H * KD;      // row of token i: tok * KD + i * ts

  const int r0 = 16 * warp + g8, r1 = r0 + 8;                                      // this lane's two rows in the products
  const int nrow = rows - 16 * warp;                                               // rows of this block that exist (<= 0: none)
  const uint32_t s_suf = smem_u32(sm.suf[warp]), s_pk = smem_u32(sm.pk[warp]), s_pq = smem_u32(sm.pq[warp]);
  // fragment addresses: A = {k octet, q octet} x 16 channels from images at s_pk, s_pq; lane l gives row (l & 7) of matrix l >> 3
  const uint32_t s_kq = (lane & 8) ? s_pq : s_pk;

  // ---- everything the levels read is on its way before the first wait: the raw rows of k and q (bf16), then g, 64 channels at a
  //      time (fp32): the first half where the level images come later, the second where this warp's rows of the solve's operands do
  const uint32_t s_akh = smem_u32(&sm.akh[16 * warp][0]), s_dg = smem_u32(sm.dg[warp]), s_th = smem_u32(sm.th[warp]);
  auto g1_row = [&](int r) { return r < 9 ? s_akh + 256 * r : r < 14 ? s_dg + 256 * (r - 9) : s_th + 256 * (r - 14); };
  static_assert(sizeof(sm.akh) / 4 >= 9 * 256 && sizeof(sm.dg[0]) >= 5 * 256 && sizeof(sm.th[0]) >= 2 * 256, "room for 16 rows of g");
  {
    const size_t base = tok * KD + (size_t)(16 * warp) * ts;
    const int c = lane & 15;
    auto copy = [&](uint32_t dst, const void* src, bool ok) {                      // rows past the end: zeros
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16u : 0u) : "memory");
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 2 * i + (lane >> 4);
      const bool ok = r < nrow;
      const size_t at = ok ? base + r * ts + 8 * c : tok * KD;
      copy(s_pk + r * KI_LD + 16 * c, p.k + at, ok);
      copy(s_pq + r * KI_LD + 16 * c, p.q + at, ok);
    }
    if (lane < 16)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                   ::"r"(smem_u32(&sm.beta[16 * warp + lane])), "l"(p.beta + tok + (size_t)(lane < nrow ? 16 * warp + lane : 0) * p.H), "r"(lane < nrow ? 4u : 0u) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 2 * i + (lane >> 4);
        const bool ok = r < nrow;
        copy((hf ? g1_row(r) : s_suf + 256 * r) + 16 * c, p.g + (ok ? base + r * ts + 64 * hf + 4 * c : tok * KD), ok);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  }
  // v is needed last: ask L2 for it now
  for (int i = tid; i < 2 * rows; i += KI_THREADS)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.v + tok * KD + (size_t)(i >> 1) * ts + 64 * (i & 1)));
  // 1 / |k|, 1 / |q| and q . k are diagonals of products
  asm volatile("cp.async.wait_group 2;" ::: "memory");
  __syncwarp();
  {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float ck[4] = {0.f, 0.f, 0.f, 0.f}, cq[4] = {0.f, 0.f, 0.f, 0.f};            // {k; q} k^T, {k; q} q^T
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a[4];
        ldmatrix_x4(a, s_kq + (8 * u + (lane & 7)) * KI_LD + 32 * ks + 16 * (lane >> 4));
        mma_bf16(ck, a, a[0], a[2]);
        mma_bf16(cq, a, a[1], a[3]);
      }
      if ((g8 >> 1) == t4) {                                                       // the lane with column g8
        const float kk = (g8 & 1) ? ck[1] : ck[0], qk = (g8 & 1) ? ck[3] : ck[2], qq = (g8 & 1) ? cq[3] : cq[2];
        const float rk = p.l2norm ? rsqrtf(kk + 1e-6f) : 1.f, rq = p.l2norm ? rsqrtf(qq + 1e-6f) : 1.f;
        sm.nrm[warp][0][8 * u + g8] = rk; sm.nrm[warp][1][8 * u + g8] = rq; sm.nrm[warp][2][8 * u + g8] = rk * rq * qk;
      }
    }
  }
  __syncwarp();

  // ---- in-block levels, 64 channels at a time.  lv[s][octet]: {kk(g8, 2 t4), kk(g8, 2 t4 + 1), qk.., qk..} of levels 1, 2, 4;
  //      l8: rows 8 + g8 against columns 2 t4, 2 t4 + 1
  float lv[3][2][4], l8[4];
#pragma unroll
  for (int s = 0; s < 3; ++s)
#pragma unroll
    for (int u = 0; u < 2; ++u) { lv[s][u][0] = lv[s][u][1] = lv[s][u][2] = lv[s][u][3] = 0.f; }
  l8[0] = l8[1] = l8[2] = l8[3] = 0.f;
  uint32_t sh[16];                                                                 // k suf of the first 64 channels
  const uint32_t s_lv = s_suf + ((lane & 8) ? 16 * KI_LV : 0) + (lane & 7) * KI_LV + 16 * (lane >> 4);   // level images: k rows, then q rows
#pragma unroll 1
  for (int hf = 0; hf < 2; ++hf) {                                                 // (rolled: the instruction cache bounds three CTAs too)
    uint64_t pre[16], suf[16];                                                     // fp32 pairs: the lane's two channels
    uint32_t kh[16], qh[16];                                                       // normalised, fp16 pairs
    {
      if (hf == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      uint2 gv[16];
#pragma unroll
      for (int t = 0; t < 16; ++t)
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(gv[t].x), "=r"(gv[t].y) : "r"((hf ? g1_row(t) : s_suf + 256 * t) + 8 * lane) : "memory");
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        pre[t] = pack2f(fast_exp2(__uint_as_float(gv[t].x) * 1.4426950408889634f), fast_exp2(__uint_as_float(gv[t].y) * 1.4426950408889634f));
        suf[t] = pack2f(1.f, 1.f);
      }
    }
#pragma unroll
    for (int t4_ = 0; t4_ < 16; t4_ += 4) {
      float rk[4], rq[4];
      *reinterpret_cast<float4*>(rk) = *reinterpret_cast<const float4*>(&sm.nrm[warp][0][t4_]);
      *reinterpret_cast<float4*>(rq) = *reinterpret_cast<const float4*>(&sm.nrm[warp][1][t4_]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = t4_ + e;
        const uint32_t off = t * KI_LD + 128 * hf + 4 * lane;
        const uint32_t kr = *reinterpret_cast<const uint32_t*>(sm.pk[warp] + off), qr = *reinterpret_cast<const uint32_t*>(sm.pq[warp] + off);
        kh[t] = pack_h2(bf16_lo(kr) * rk[e], bf16_hi(kr) * rk[e]);
        qh[t] = pack_h2(bf16_lo(qr) * rq[e], bf16_hi(qr) * rq[e]);
      }
    }
    auto level = [&](auto S) {                                                     // S = 1, 2, 4, 8
      constexpr int s = decltype(S)::value;
      __syncwarp();                                                                // the previous level's fragments are loaded
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        float f0, f1;
        unpack2f((t & s) ? pre[t] : suf[t], f0, f1);
        const uint32_t f = pack_h2(f0, f1), off = t * KI_LV + 4 * lane;
        *reinterpret_cast<uint32_t*>(sm.suf[warp] + off) = hmul2_u32(kh[t], f);
        if (t & s) *reinterpret_cast<uint32_t*>(sm.suf[warp] + 16 * KI_LV + off) = hmul2_u32(qh[t], f);   // (lower tokens' results are not used)
      }
      __syncwarp();
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (s < 8) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint32_t a[4];
            ldmatrix_x4(a, s_lv + 8 * u * KI_LV + 32 * ks);
            mma_f16(lv[s == 1 ? 0 : s == 2 ? 1 : 2][u], a, a[0], a[2]);
          }
        } else {
          uint32_t a[4], c[4];
          ldmatrix_x4(a, s_lv + 8 * KI_LV + 32 * ks);
          ldmatrix_x4(c, s_lv + 32 * ks);
          mma_f16(l8, a, c[0], c[2]);
        }
      }
      // both products from aligned blocks of s to blocks of 2 s: upper block: prefix times the lower block's total; lower block:
      // suffix times the upper block's total
#pragma unroll
      for (int a = 0; a < 16; a += 2 * s) {
        const uint64_t tl = pre[a + s - 1], tu = pre[a + 2 * s - 1];
#pragma unroll
        for (int i = 0; i < s; ++i) { pre[a + s + i] = fmul2(pre[a + s + i], tl); suf[a + i] = fmul2(suf[a + i], tu); }
      }
    };
    level(std::integral_constant<int, 1>{});
    level(std::integral_constant<int, 2>{});
    level(std::integral_constant<int, 4>{});
    level(std::integral_constant<int, 8>{});
    __syncwarp();
    // the block's images, from the unrounded rows
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const float rk = sm.nrm[warp][0][t], rq = sm.nrm[warp][1][t];
      const uint32_t off = t * KI_LD + 128 * hf + 4 * lane;
      const uint32_t kr = *reinterpret_cast<const uint32_t*>(sm.pk[warp] + off), qr = *reinterpret_cast<const uint32_t*>(sm.pq[warp] + off);
      const uint64_t kf = pack2f(bf16_lo(kr) * rk, bf16_hi(kr) * rk), qf = pack2f(bf16_lo(qr) * rq, bf16_hi(qr) * rq);
      *reinterpret_cast<uint32_t*>(sm.pk[warp] + off) = pack_h2(fmul2(kf, pre[t]));
      *reinterpret_cast<uint32_t*>(sm.pq[warp] + off) = pack_h2(fmul2(qf, pre[t]));
      const uint32_t ks = pack_h2(fmul2(kf, suf[t]));
      if (hf == 0) sh[t] = ks;
      else {
        *reinterpret_cast<uint32_t*>(sm.suf[warp] + off - 128) = sh[t];
        *reinterpret_cast<uint32_t*>(sm.suf[warp] + off) = ks;
      }
    }
    float d0, d1;
    unpack2f(pre[15], d0, d1);
    *reinterpret_cast<float2*>(&sm.tot[warp][64 * hf + 2 * lane]) = make_float2(d0, d1);
  }
  __syncwarp();
  __syncthreads();

  // ---- products with the earlier blocks: (1, 0); (2, 1), (2, 0); (3, 2), (3, 1) and, by warp 0, which has none of its own, (3, 0)
  const float b0 = sm.beta[r0], b1 = sm.beta[r1];
  const int I = warp ? warp : 3;
#pragma unroll 1
  for (int J = warp ? warp - 1 : 0; J >= (warp == 3 ? 1 : 0); --J) {
    const int i0 = 16 * I + g8, i1 = i0 + 8;
    const float bi0 = sm.beta[i0], bi1 = sm.beta[i1];
    const uint32_t s_ki = smem_u32(sm.pk[I]), s_qi = smem_u32(sm.pq[I]);
    float kk[2][4], qk[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) { kk[n][0] = kk[n][1] = kk[n][2] = kk[n][3] = 0.f; qk[n][0] = qk[n][1] = qk[n][2] = qk[n][3] = 0.f; }
    const uint32_t s_c = smem_u32(sm.suf[J]) + ((lane & 7) + 8 * (lane >> 4)) * KI_LD + 16 * ((lane >> 3) & 1);
    const uint32_t ao = ((lane & 7) + 8 * ((lane >> 3) & 1)) * KI_LD + 16 * (lane >> 4);
#pragma unroll 2
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t c[4], kr[4], qr[4];
      ldmatrix_x4(c, s_c + 32 * ks);
      ldmatrix_x4(kr, s_ki + ao + 32 * ks);
      ldmatrix_x4(qr, s_qi + ao + 32 * ks);
      if (J < I - 1) {                                                          // blocks lie between: their totals
        float2 f0 = *reinterpret_cast<const float2*>(&sm.tot[J + 1][16 * ks + 2 * t4]), f1 = *reinterpret_cast<const float2*>(&sm.tot[J + 1][16 * ks + 8 + 2 * t4]);
        if (J < I - 2) {
          const float2 e0 = *reinterpret_cast<const float2*>(&sm.tot[J + 2][16 * ks + 2 * t4]), e1 = *reinterpret_cast<const float2*>(&sm.tot[J + 2][16 * ks + 8 + 2 * t4]);
          f0.x *= e0.x; f0.y *= e0.y; f1.x *= e1.x; f1.y *= e1.y;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) { kr[i] = ki_scale(kr[i], i < 2 ? f0 : f1); qr[i] = ki_scale(qr[i], i < 2 ? f0 : f1); }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mma_f16(kk[n], kr, c[2 * n], c[2 * n + 1]);
        mma_f16(qk[n], qr, c[2 * n], c[2 * n + 1]);
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int col = 16 * J + 8 * n + 2 * t4;
      *reinterpret_cast<uint32_t*>(&sm.akh[i0][col]) = pack_h2(bi0 * kk[n][0], bi0 * kk[n][1]);
      *reinterpret_cast<uint32_t*>(&sm.akh[i1][col]) = pack_h2(bi1 * kk[n][2], bi1 * kk[n][3]);
      *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(i0, col)) = pack_h2(p.scale * qk[n][0], p.scale * qk[n][1]);
      *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(i1, col)) = pack_h2(p.scale * qk[n][2], p.scale * qk[n][3]);
    }
  }
  if (warp == 0) { __syncwarp(); asm volatile("bar.arrive 1, 64;" ::: "memory"); }  // block 3's images may change

  // ---- the diagonal block: each entry from its level
  {
    const int jc = 2 * t4;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float kk[2], qk[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int x = g8 ^ (jc + e);                                               // highest differing bit of the two token numbers
        const float a = x >= 4 ? lv[2][u][e] : x >= 2 ? lv[1][u][e] : lv[0][u][e];
        const float c = x >= 4 ? lv[2][u][2 + e] : x >= 2 ? lv[1][u][2 + e] : lv[0][u][2 + e];
        const bool low = jc + e < g8;
        kk[e] = low ? (u ? b1 : b0) * a : 0.f;
        qk[e] = p.scale * (low ? c : jc + e == g8 ? sm.nrm[warp][2][8 * u + g8] : 0.f);                 // the diagonal: q_i . k_i, no decay
        sm.dg[warp][8 * u + jc + e][8 * u + g8] = kk[e];
      }
      *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(16 * warp + 8 * u + g8, 16 * warp + 8 * u + jc)) = pack_h2(qk[0], qk[1]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) { sm.dg[warp][jc + e][8 + g8] = b1 * l8[e]; sm.dg[warp][8 + jc + e][g8] = 0.f; }
    *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(r1, 16 * warp + jc)) = pack_h2(p.scale * l8[2], p.scale * l8[3]);
    *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(r0, 16 * warp + 8 + jc)) = 0u;
  }
  for (int J = warp + 1; J < 4; ++J) st_global16(rec + OFF_AQK + rec_off(16 * warp + (lane >> 1), 16 * J + 8 * (lane & 1)), 0u, 0u, 0u, 0u);   // j > i
  __syncwarp();
  // ---- its inverse in fp32, lane = column: a column sweep (once t_j is final every later row takes its update at once)
  if (lane < 16) {
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = (i == lane) ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 15; ++j) {
      float a[16];
#pragma unroll
      for (int i4 = (j + 1) & ~3; i4 < 16; i4 += 4) *reinterpret_cast<float4*>(&a[i4]) = *reinterpret_cast<const float4*>(&sm.dg[warp][j][i4]);
#pragma unroll
      for (int i = j + 1; i < 16; ++i) t[i] = fmaf(-a[i], t[j], t[i]);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) sm.th[warp][i][lane] = __float2half_rn(t[i]);
  }

  if (warp == 3) asm volatile("bar.sync 1, 64;" ::: "memory");
  // ---- state-pass operands: k e^G (shared memory), q e^G scale and k e^{G_C - G} (record)
  {
    const int c = lane & 15;                                                       // this lane's eight channels, in every other row
    float f[8], s[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) { f[e] = 1.f; s[e] = 1.f; }
    for (int K = 0; K < 4; ++K) {
      if (K == warp) continue;
      const float4 lo = *reinterpret_cast<const float4*>(&sm.tot[K][8 * c]), hi = *reinterpret_cast<const float4*>(&sm.tot[K][8 * c + 4]);
      const float t[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) { f[e] *= K < warp ? t[e] : 1.f; s[e] *= K < warp ? 1.f : t[e]; }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 2 * i + (lane >> 4);
      const uint32_t off = r * KI_LD + 16 * c, roff = panel_off(16 * warp + r, c);
      uint32_t q[4], k[4], z[4];
      *reinterpret_cast<uint4*>(q) = *reinterpret_cast<const uint4*>(sm.pq[warp] + off);
      *reinterpret_cast<uint4*>(k) = *reinterpret_cast<const uint4*>(sm.pk[warp] + off);
      *reinterpret_cast<uint4*>(z) = *reinterpret_cast<const uint4*>(sm.suf[warp] + off);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 fj = make_float2(f[2 * j], f[2 * j + 1]);
        k[j] = ki_scale(k[j], fj);
        q[j] = ki_scale(q[j], make_float2(fj.x * p.scale, fj.y * p.scale));
        z[j] = ki_scale(z[j], make_float2(s[2 * j], s[2 * j + 1]));
      }
      *reinterpret_cast<uint4*>(sm.pk[warp] + off) = *reinterpret_cast<const uint4*>(k);
      st_global16(rec + OFF_QT + roff, q[0], q[1], q[2], q[3]);
      st_global16(rec + OFF_KT + roff, z[0], z[1], z[2], z[3]);
    }
    __syncwarp();
    const uint32_t vb = s_pq;                                                      // v takes the place of q pre
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 2 * i + (lane >> 4);
      const uint32_t n = r < nrow ? 16u : 0u;                                      // rows past the end: zeros
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                   ::"r"(vb + r * KI_LD + 16 * c), "l"(p.v + tok * KD + (size_t)(r < nrow ? 16 * warp + r : 0) * ts + 8 * c), "r"(n) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  reinterpret_cast<float*>(rec + OFF_D)[tid] = (sm.tot[0][tid] * sm.tot[1][tid]) * (sm.tot[2][tid] * sm.tot[3][tid]);   // e^{G_C}
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- W and U0 by blocked forward substitution on the transposed systems
  //          W^T (I + A)^T = (diag(beta) k e^G)^T,      U0^T (I + A)^T = (diag(beta) v)^T
  //      A warp owns 64 of the 256 rows (channels of W^T: warps 0, 1, value columns of U0^T: warps 2, 3) for all four
  //      16-token block columns I, so there is nothing to exchange between warps:
  //          Z_I = R_I - sum_{J<I} Z_J A_IJ^T,   then   Z_I <- Z_I T_II^T
  //      with every product an m16n8k16 tile whose fp32 accumulators, rounded to fp16, are the A fragment of the products
  //      that follow.  Two row tiles of a warp are independent chains issued side by side, twice (all four unrolled were more
  //      registers and more code than they hid: 336 -> 326 us).
  {
    const bool is_w = warp < 2;
    uint8_t* dst = rec + (is_w ? OFF_WT : OFF_UT);
#pragma unroll 1
    for (int c0 = 64 * (warp & 1), end = c0 + 64; c0 < end; c0 += 32) {               // first row (channel or value column) of two tiles
      const uint32_t src = smem_u32(is_w ? sm.pk : sm.pq) + ((lane & 7) + 8 * (lane >> 4)) * KI_LD + 2 * c0 + 16 * ((lane >> 3) & 1);
      uint32_t zf[2][3][4];                                                          // Z_J as fp16 A fragments: [row tile][J][4]
#pragma unroll
      for (int I = 0; I < 4; ++I) {
        float acc[2][2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int n = 0; n < 2; ++n) { acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f; }
#pragma unroll
        for (int J = 0; J < I; ++J) {
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            const __half* arow = &sm.akh[I * 16 + n * 8 + g8][J * 16 + 2 * t4];
            const uint32_t w0 = *reinterpret_cast<const uint32_t*>(arow), w1 = *reinterpret_cast<const uint32_t*>(arow + 8);
#pragma unroll
            for (int m = 0; m < 2; ++m) mma_f16(acc[m][n], zf[m][J], w0, w1);
          }
        }
        uint32_t tw[2][2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const __half* trow = &sm.th[I][n * 8 + g8][2 * t4];
          tw[n][0] = *reinterpret_cast<const uint32_t*>(trow); tw[n][1] = *reinterpret_cast<const uint32_t*>(trow + 8);
        }
        const float2 bt0 = *reinterpret_cast<const float2*>(&sm.beta[I * 16 + 2 * t4]), bt1 = *reinterpret_cast<const float2*>(&sm.beta[I * 16 + 8 + 2 * t4]);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          // right-hand side: tokens 16 I .. + 15 x rows c0 + 16 m .. + 15, transposed: register i = (tokens 8 (i >> 1) + 2 t4 (+1),
          // row 8 (i & 1) + g8)
          uint32_t rr[4];
          ldmatrix_x4_t(rr, src + I * (16 * KI_LD) + 32 * m);
          uint32_t a[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int n = i >> 1, hi = i & 1;
            const float2 r = is_w ? unpack_h2(rr[i]) : make_float2(bf16_lo(rr[i]), bf16_hi(rr[i]));
            const float2 bt = n ? bt1 : bt0;
            a[2 * n + hi] = pack_h2(r.x * bt.x - acc[m][n][2 * hi], r.y * bt.y - acc[m][n][2 * hi + 1]);
          }
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            float z[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(z, a, tw[n][0], tw[n][1]);
            const uint32_t zl = pack_h2(z[0], z[1]), zh = pack_h2(z[2], z[3]);
            if (I < 3) { zf[m][I][2 * n] = zl; zf[m][I][2 * n + 1] = zh; }
            const int cr = c0 + 16 * m + g8;
            *reinterpret_cast<uint32_t*>(dst + rec_off(cr, I * 16 + n * 8 + 2 * t4)) = zl;
            *reinterpret_cast<uint32_t*>(dst + rec_off(cr + 8, I * 16 + n * 8 + 2 * t4)) = zh;
          }
        }
      }
    }
  }
  if (p.behind && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1) grid_dep_wait();
}

// =============================================================================================
// inter-chunk state kernel
// =============================================================================================
struct KdaStateParams {
  const uint8_t* ws;
  const float* h0;         // state before the first chunk (null: zero) and after the last (null: not kept)
  float* hT;
  void* o;
  int64_t ld_in, ld_out;   // floats between the states of two CTAs
  int T, H, NC, out_fp32;
  int c0, c1, more;        // dense: chunks of this launch; more: another one follows it (kda_split)
  int* status;
  // packed variable-length sequences (B = 1): blockIdx.x = sequence * H + head, the sequence's chunks are
  // seq_ptr[s] .. seq_ptr[s + 1] - 1 of the packed row's NC chunks, chunk_tab as in the intra kernel; null: dense
  const int* chunk_tab;
  const int* seq_ptr;
};


// One CTA per (batch, head); TMEM lane = value column, so all products have M = 128 and
//     U^T [V x 64]   = U0^T - S^T W^T            S^T as fp16 from TMEM, W^T as the record has it (channels = depth)
//     O^T [V x 64]   = S^T q~^T + U^T A_qk^T
//     S^T [V x 128] <- S^T diag(e^{G_C}) + U^T k~  the product summed in TMEM, added to the state in registers
// The chain from chunk to chunk is all that matters (a (batch, head) is serial, and there are rarely more of them than SMs):
// S to fp16, 8 products of N = 64, U to fp16, 4 products of N = 128.  Warps 0-7 (thread = half a value column) run it with the
// state in fp32 registers, scaled while the U products run; TMEM carries only fp16 operands and fresh sums.  Two warps to a
// scheduler: one warp's conversions alone are twice as long as the products.  q~'s products fill the tensor pipe while U is
// converted, warps 8-11 write O out of two accumulators, transposed through shared memory, warp 12 issues, warps 13 and 14
// keep the rings full.
// The same recurrence in mma.sync fragments, 64 value columns to a CTA, took 3700 cycles a chunk (212 products of a warp on
// one tensor pipe and as many cycles of ldmatrix): 500 us at 4 x 16384 x 16.  With the state in TMEM, scaled there, 2850
// cycles, 418 us; with one three-stage ring of whole records, which the output held back, 2560 cycles, 370 us; this form 344.
// The record comes in two parts with rings of their own: W^T, D and U0^T are spent when U is there, the rest a product later
constexpr int KS_A = 3, KS_B = 2;
constexpr int KS_A_BYTES = 33 * 1024, KS_B_BYTES = 40 * 1024;  // operands start on 1024-byte boundaries
constexpr int KS_AD = KD * KC * 2, KS_AU = KS_AD + KD * 4;     // in part A: W^T, then D and U0^T
constexpr int KS_OUT = 16 * 1024;                              // output of one chunk, bf16
constexpr int KS_THREADS = 480;
static_assert(OFF_KT - OFF_QT == 16384 && OFF_AQK - OFF_QT == 32768 && OFF_D - OFF_QT == KS_B_BYTES && OFF_UT - OFF_D == KD * 4, "q~, k~, A_qk in one copy; D, U0^T in another");
constexpr int TM_D = 0, TM_S16 = 128, TM_U = 192, TM_U16 = 256, TM_O = 288;      // TMEM columns; D: the state's increment; O: two accumulators of 64
struct KdaStateBars {
  uint64_t a_full[KS_A], a_empty[KS_A], b_full[KS_B], b_empty[KS_B];
  uint64_t s16[2], u, u16, s, o_full[2], o_free[2];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int KS_SMEM = 1024 + KS_A * KS_A_BYTES + KS_B * KS_B_BYTES + KS_OUT + (int)sizeof(KdaStateBars);
static_assert(KS_SMEM <= 232448, "over the 227 KB a CTA may use");

__device__ __forceinline__ void ld_shared16(uint32_t* r, uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

__global__ void __launch_bounds__(KS_THREADS, 1) kda_state_kernel(const KdaStateParams p) {
  extern __shared__ uint8_t kda_smem_raw[];
  uint8_t* part_a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(kda_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *part_b = part_a + KS_A * KS_A_BYTES, *out = part_b + KS_B * KS_B_BYTES;
  KdaStateBars* bars = reinterpret_cast<KdaStateBars*>(out + KS_OUT);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < KS_A; ++i) { mbar_init(&bars->a_full[i], 1); mbar_init(&bars->a_empty[i], 9); }     // warps 0-7, one commit
    for (int i = 0; i < KS_B; ++i) { mbar_init(&bars->b_full[i], 1); mbar_init(&bars->b_empty[i], 1); }
    mbar_init(&bars->s16[0], 128); mbar_init(&bars->s16[1], 128); mbar_init(&bars->u, 1); mbar_init(&bars->u16, 256); mbar_init(&bars->s, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->o_full[i], 1); mbar_init(&bars->o_free[i], 128); }
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 12) { tmem_alloc(&bars->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  if (p.more) grid_dep_launch();
  grid_dep_wait();

  const int bh = blockIdx.x, h = bh % p.H, b = p.seq_ptr ? 0 : bh / p.H;           // bh also indexes h0 / hT
  const int c_begin = p.seq_ptr ? p.seq_ptr[bh / p.H] : p.c0, c_end = p.seq_ptr ? p.seq_ptr[bh / p.H + 1] : p.c1;
  const int n_chunks = c_end - c_begin;

  const uint8_t* recs = p.ws + ((size_t)(b * p.H + h) * p.NC + c_begin) * REC_BYTES;
  if (warp == 13) {
    // ------------------------------------------------------------ producers: part A, part B
    if (lane == 0) {
      for (int c = 0; c < n_chunks; ++c) {
        const int s = c % KS_A;
        const uint8_t* rec = recs + (size_t)c * REC_BYTES;
        if (!mbar_wait(&bars->a_empty[s], ((c / KS_A) & 1) ^ 1, abort_flag, p.status, 1)) break;
        mbar_expect_tx(&bars->a_full[s], KS_AU + KD * KC * 2);
        bulk_g2s(part_a + s * KS_A_BYTES, rec + OFF_WT, KD * KC * 2, &bars->a_full[s]);
        bulk_g2s(part_a + s * KS_A_BYTES + KS_AD, rec + OFF_D, KD * 4 + KD * KC * 2, &bars->a_full[s]);
      }
    }
    __syncwarp();
  } else if (warp == 14) {
    if (lane == 0) {
      for (int c = 0; c < n_chunks; ++c) {
        const int s = c % KS_B;
        if (!mbar_wait(&bars->b_empty[s], ((c / KS_B) & 1) ^ 1, abort_flag, p.status, 1)) break;
        mbar_expect_tx(&bars->b_full[s], KS_B_BYTES);
        bulk_g2s(part_b + s * KS_B_BYTES, recs + (size_t)c * REC_BYTES + OFF_QT, KS_B_BYTES, &bars->b_full[s]);
      }
    }
    __syncwarp();
  } else if (warp == 12) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t id_u = umma_idesc_f16(128, KC, 0, 1), id_o = umma_idesc_f16(128, KC, 0, 0), id_s = umma_idesc_f16(128, KD, 0, 1);
    const uint32_t base = smem_u32(part_b);
    const uint64_t wd = umma_desc_sw128(smem_u32(part_a), KC * 128, 1024), kd = umma_desc_sw128(base + OFF_KT - OFF_QT, KC * 128, 1024);   // depth = rows
    const uint64_t qd = umma_desc_sw128(base, 16, 1024), ad = umma_desc_sw128(base + OFF_AQK - OFF_QT, 16, 1024);              // depth along the row
    const uint32_t w_hi = (uint32_t)(wd >> 32), k_hi = (uint32_t)(kd >> 32), q_hi = (uint32_t)(qd >> 32), a_hi = (uint32_t)(ad >> 32);
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t sa = c % KS_A, sb = c % KS_B, ao = sa * (KS_A_BYTES >> 4), bo = sb * (KS_B_BYTES >> 4), o = tmem + TM_O + KC * (c & 1);
      if (!mbar_wait(&bars->a_full[sa], (c / KS_A) & 1, abort_flag, p.status, 2)) break;
      if (!mbar_wait(&bars->s16[0], c & 1, abort_flag, p.status, 3)) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_ts_lh_p(leader, tmem + TM_U, tmem + TM_S16 + 8 * k, (uint32_t)wd + ao + k * (2048 >> 4), w_hi, id_u, k ? 1u : 0u);
      if (!mbar_wait(&bars->s16[1], c & 1, abort_flag, p.status, 3)) break;
      tc_fence_after();
#pragma unroll
      for (int k = 4; k < 8; ++k) umma_ts_lh_p(leader, tmem + TM_U, tmem + TM_S16 + 8 * k, (uint32_t)wd + ao + k * (2048 >> 4), w_hi, id_u, 1u);
      tc_commit_p(leader, &bars->u);
      tc_commit_p(leader, &bars->a_empty[sa]);
      if (!mbar_wait(&bars->b_full[sb], (c / KS_B) & 1, abort_flag, p.status, 2)) break;
      if (!mbar_wait(&bars->o_free[c & 1], ((c >> 1) & 1) ^ 1, abort_flag, p.status, 4)) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 8; ++k) umma_ts_lh_p(leader, o, tmem + TM_S16 + 8 * k, (uint32_t)qd + bo + ((k >> 2) * (KC * 128) + (k & 3) * 32) / 16, q_hi, id_o, k ? 1u : 0u);
      if (!mbar_wait(&bars->u16, c & 1, abort_flag, p.status, 5)) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_ts_lh_p(leader, tmem + TM_D, tmem + TM_U16 + 8 * k, (uint32_t)kd + bo + k * (2048 >> 4), k_hi, id_s, k ? 1u : 0u);
      tc_commit_p(leader, &bars->s);
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_ts_lh_p(leader, o, tmem + TM_U16 + 8 * k, (uint32_t)ad + bo + k * 2, a_hi, id_o, 1u);
      tc_commit_p(leader, &bars->o_full[c & 1]);
      tc_commit_p(leader, &bars->b_empty[sb]);
    }
    __syncwarp();
  } else if (warp < 8) {
    // ------------------------------------------------------------ the chain: thread = half of a value column
    const int half = warp >> 2, v = 32 * (warp & 3) + lane;
    const uint32_t t = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    float S[64];                                                                   // row v of S^T, channels 64 half ..
    {
      const float* hp = p.h0 ? p.h0 + bh * p.ld_in + 64 * half * KD + v : nullptr;
#pragma unroll
      for (int i = 0; i < 64; ++i) S[i] = hp ? __ldcg(hp + (size_t)i * KD) : 0.f;      // (L2: the part before may have written it)
    }
    bool ok = true;
    for (int c = 0; c <= n_chunks; ++c) {
      if (c > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->s, (c - 1) & 1, abort_flag, p.status, 6));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t x[32];
          tmem_ld32(t + TM_D + 64 * half + 32 * j, x);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) S[32 * j + i] += __uint_as_float(x[i]);
        }
      }
      if (c == n_chunks) break;
      uint32_t y[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) y[i] = pack_h2(S[2 * i], S[2 * i + 1]);
      tmem_st32(t + TM_S16 + 32 * half, y);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->s16[half]);
      // beside the U products: scale the state, fetch this column's 32 tokens of U0
      const int s = c % KS_A;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->a_full[s], (c / KS_A) & 1, abort_flag, p.status, 7));
      if (!ok) break;
      const uint32_t rec = smem_u32(part_a) + s * KS_A_BYTES;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t d[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) ld_shared16(d + 4 * i, rec + KS_AD + 256 * half + 128 * j + 16 * i);
#pragma unroll
        for (int i = 0; i < 32; ++i) S[32 * j + i] *= __uint_as_float(d[i]);
      }
      uint32_t u0[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) ld_shared16(u0 + 4 * j, rec + KS_AU + rec_off(v, 32 * half + 8 * j));
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->a_empty[s]);
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->u, c & 1, abort_flag, p.status, 8));
      if (!ok) break;
      tc_fence_after();
      tmem_ld32(t + TM_U + 32 * half, y);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 u = unpack_h2(u0[i]);
        u0[i] = pack_h2(u.x - __uint_as_float(y[2 * i]), u.y - __uint_as_float(y[2 * i + 1]));
      }
      tmem_st16(t + TM_U16 + 16 * half, u0);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->u16);
    }
    if (ok && p.hT) {
      float* hp = p.hT + bh * p.ld_out + 64 * half * KD + v;
#pragma unroll
      for (int i = 0; i < 64; ++i) hp[(size_t)i * KD] = S[i];
    }
  } else {
    // ------------------------------------------------------------ output: a warp's 64 tokens x 32 columns, bf16 in 64-byte stores.
    // Its columns lie as rows of 64 tokens in shared memory, from where a transposing ldmatrix gives a lane eight columns of a token:
    // rows 2 j, 2 j + 1 of matrix m are columns 8 j + 2 m, + 1.  Pieces are exchanged by (v & 7) ^ 2 (v >> 3): both the eight
    // lanes of a store and the eight rows of a matrix hit different banks
    const int w = warp - 8;
    const uint32_t t = tmem + ((uint32_t)(32 * w) << 16) + TM_O;
    const int vr = 8 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);           // the row this lane addresses
    for (int c = 0; c < n_chunks; ++c) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->o_full[c & 1], (c >> 1) & 1, abort_flag, p.status, 10))) break;
      tc_fence_after();
      uint32_t x[64];
      tmem_ld32(t + KC * (c & 1), x);
      tmem_ld32(t + KC * (c & 1) + 32, x + 32);
      tc_wait_ld();
      tc_fence_before();
      mbar_arrive(&bars->o_free[c & 1]);
      int t0, rows;
      ki_chunk_span(p.chunk_tab, c_begin + c, p.T, t0, rows);
      const size_t off = (((size_t)b * p.T + t0) * p.H + h) * KD + 32 * w, ts = (size_t)p.H * KD;
      if (p.out_fp32) {
        float* o = reinterpret_cast<float*>(p.o) + off + lane;
#pragma unroll
        for (int i = 0; i < KC; ++i) if (i < rows) o[i * ts] = __uint_as_float(x[i]);
      } else {
        const uint32_t stg = smem_u32(out) + w * 4096;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t* xx = x + 8 * j;
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};"
                       ::"r"(stg + lane * 128 + ((j ^ ((lane & 7) ^ (2 * (lane >> 3)))) << 4)),
                       "r"(pack_bf16(__uint_as_float(xx[0]), __uint_as_float(xx[1]))), "r"(pack_bf16(__uint_as_float(xx[2]), __uint_as_float(xx[3]))),
                       "r"(pack_bf16(__uint_as_float(xx[4]), __uint_as_float(xx[5]))), "r"(pack_bf16(__uint_as_float(xx[6]), __uint_as_float(xx[7]))) : "memory");
        }
        __syncwarp();
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.o) + off + 8 * (lane & 3);
#pragma unroll
        for (int j = 0; j < 8; ++j) ldmatrix_x4_t(x + 4 * j, stg + vr * 128 + ((j ^ ((vr & 7) ^ (2 * (vr >> 3)))) << 4));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int tok = 8 * j + (lane >> 2);
          if (tok < rows) st_global16(o + tok * ts, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Chunk table and sequences' first chunks of a packed row, from its lengths where they lie: one CTA, one thread a sequence.  For the
// host to make them it has to wait for the lengths, with the device idle until the tables are back (11 sequences, 5003 tokens of
// 16 heads: 122 us a call, 110 with this).  Lengths that do not begin at 0, decrease or do not end at T give tables without chunks.
constexpr int KT_MAX_SEQ = 1023;
template <typename E>
__global__ void __launch_bounds__(1024) kda_tables_kernel(const E* cu, int n, int T, int cap, int2* tab, int* ptr) {
  __shared__ int first[1024], at[1024], sums[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_dep_launch();
  grid_dep_wait();
  const long long v = tid <= n ? (long long)cu[tid] : T, next = tid < n ? (long long)cu[tid + 1] : T;
  const bool bad = v < 0 || v > T || next < v || (tid == 0 && v != 0) || (tid == n && v != T);
  first[tid] = (int)v;
  const bool none = __syncthreads_or(bad) != 0;
  int scan = none || tid >= n ? 0 : ((int)(next - v) + KC - 1) / KC;
  const int own = scan;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) { const int up = __shfl_up_sync(0xffffffffu, scan, d); if (lane >= d) scan += up; }
  if (lane == 31) sums[warp] = scan;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += sums[w];
  at[tid] = before + scan - own;
  if (tid <= n) ptr[tid] = at[tid];
  __syncthreads();
  const int total = at[n];
  for (int c = tid; c < cap; c += 1024) {
    int2 e = make_int2(0, 0);
    if (c < total) {
      int lo = 0, hi = n;                              // the last sequence whose first chunk is not behind c
      while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (at[mid] <= c) lo = mid; else hi = mid; }
      e.x = first[lo] + KC * (c - at[lo]);
      e.y = min(KC, first[lo + 1] - e.x);
    }
    tab[c] = e;
  }
}

}  // namespace daisy

using namespace daisy;

extern "C" int daisy_b200_kda_chunk_tables(const void* cu, int elem_bytes, int n_seq, int T_total, int32_t* chunk_tab, int max_chunks, int32_t* seq_ptr, void* stream) {
  if (!cu || !chunk_tab || !seq_ptr || n_seq <= 0 || T_total <= 0) return DAISY_EINVAL;
  if (n_seq > KT_MAX_SEQ || (elem_bytes != 4 && elem_bytes != 8)) return DAISY_EUNSUPPORTED;
  if (max_chunks < T_total / KC + n_seq) return DAISY_EWORKSPACE;
  if ((reinterpret_cast<uintptr_t>(chunk_tab) & 7) || (reinterpret_cast<uintptr_t>(seq_ptr) & 3) || (reinterpret_cast<uintptr_t>(cu) & (elem_bytes - 1))) return DAISY_EALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  if (elem_bytes == 4) (void)daisy_host::launch_dependent(kda_tables_kernel<int32_t>, dim3(1), dim3(1024), 0, st, (const int32_t*)cu, n_seq, T_total, max_chunks, (int2*)chunk_tab, seq_ptr);
  else                 (void)daisy_host::launch_dependent(kda_tables_kernel<int64_t>, dim3(1), dim3(1024), 0, st, (const int64_t*)cu, n_seq, T_total, max_chunks, (int2*)chunk_tab, seq_ptr);
  DAISY_CHECK_LAUNCH();
  return DAISY_OK;
}

extern "C" size_t daisy_b200_kda_workspace_bytes(int B, int T, int H, int K, int V) {
  if (B <= 0 || T <= 0 || H <= 0 || K != KD || V != KD) return 0;
  const size_t nc = (size_t)(T + KC - 1) / KC;
  return (size_t)B * H * nc * WS_REC_BYTES;
}

// Where to cut a row of chunks, so that the state's pass over one part runs beside the intra-chunk pass over the next: the state
// takes a CTA per (batch, head), the other SMs are the next part's.  Launches: intra, state, intra, state, ..  A launch may start
// when every CTA of the one before has started; the state's waits for the intra-chunk launch before it, which ends only after the
// state's launch before that has (its last CTA waits for it).  An intra-chunk launch after the first waits for nothing at its
// start: all CTAs of the first have waited for what the stream held before.  The state goes from part to part in fp32 through the
// room of a record that is spent, so the results have the same bits.
// Each part takes as long beside the state's pass as that pass: by the measured 5.7 us of an SM per record, 1.35 us of the chain per
// chunk alone and 1.8 beside the other pass, and 5 us that a cut costs (SMs run empty, the state is stored and read).
// One pass each -> in parts: 4 x 16384 x 16 977 -> 874 us, 2 x 8192 x 16 343 -> 287, 1 x 16384 x 16 512 -> 427, 3 x 7000 x 12
// 312 -> 262, 2 x 3001 x 16 136 -> 119, 2 x 1000 x 16 54 -> 49; rows of fewer chunks do not gain what a cut costs (2 x 700 x 16 level).
constexpr int KDA_PARTS = 4;
static_assert(KD * KD * 4 <= REC_BYTES, "a state fits a record");
static int kda_split(int rows, int NC, int sms, int* end) {
  if (rows >= sms * 7 / 8) return 1;
  const double intra = 5.7 * rows / sms, beside = 5.7 * rows / (sms - rows), chain = 1.35, slow = 1.8, cost = 5;
  int best = 1;
  double best_us = NC * (intra + chain);
  for (int n = 2; n <= KDA_PARTS; ++n) {
    double sum = 0, part = 1;
    for (int i = 0; i < n; ++i, part *= slow / beside) sum += part;
    int cut[KDA_PARTS], at = 0;
    double us = 0, size = NC / sum;
    bool ok = true;
    for (int i = 0, before = 0; i < n; ++i, size *= slow / beside) {
      const int len = i + 1 == n ? NC - at : (int)(size + 0.5);
      ok = ok && len >= 4;
      const double state = before * slow, own = len * beside;
      us += i == 0 ? len * intra : cost + (state > own ? state : own);
      cut[i] = at += len;
      before = len;
      if (i + 1 == n) us += len * chain;
    }
    if (!ok || us >= best_us) continue;
    best = n; best_us = us;
    for (int i = 0; i < n; ++i) end[i] = cut[i];
  }
  return best;
}

extern "C" int daisy_b200_kda_parts(int B, int T, int H) {
  if (B <= 0 || T <= 0 || H <= 0) return DAISY_EINVAL;
  const int sms = daisy_host::sm_count_cached();
  int end[KDA_PARTS];
  return sms > 0 ? kda_split(B * H, (T + KC - 1) / KC, sms, end) : DAISY_ENODEV;
}

// Shared launcher.  Dense: NC = ceil(T / 64) chunks per (batch, head) row, n_seq = B.  Packed variable-length (B = 1):
// chunk_tab [NC][2] and seq_ptr [n_seq + 1] (both in device memory) say which tokens each chunk covers and which
// chunks each sequence owns; h0 / hT are [n_seq, H, K, V].
static int kda_launch(const void* q, const void* k, const void* v, const float* g, const float* beta, const float* h0, void* o,
                      float* hT, int B, int T, int H, int K, int V, int chunk, float scale, unsigned flags,
                      void* workspace, size_t workspace_bytes, int NC, int n_seq, const int* chunk_tab, const int* seq_ptr,
                      int* status_word, void* stream) {
  if (!q || !k || !v || !g || !beta || !o || !workspace || B <= 0 || T <= 0 || H <= 0 || NC <= 0 || n_seq <= 0) return DAISY_EINVAL;
  if (K != KD || V != KD || chunk != KC) return DAISY_EUNSUPPORTED;
  if (B > 65535 || H > 65535 || (size_t)n_seq * H > 65535) return DAISY_EUNSUPPORTED;
  if (workspace_bytes < (size_t)B * H * NC * WS_REC_BYTES) return DAISY_EWORKSPACE;
  if (!daisy_aligned16(q) || !daisy_aligned16(k) || !daisy_aligned16(v) || !daisy_aligned16(g) || !daisy_aligned16(o) ||
      !daisy_aligned16(workspace) || (h0 && !daisy_aligned16(h0)) || (hT && !daisy_aligned16(hT)))
    return DAISY_EALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  static bool attr[daisy_host::MAX_DEVICES] = {};             // the attribute is per device
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  constexpr int intra_smem = (int)sizeof(KdaIntraSmem);
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(kda_intra_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, intra_smem) != cudaSuccess ||
        cudaFuncSetAttribute(kda_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KS_SMEM) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    attr[dev] = true;
  }
  if ((int64_t)B * H * NC >= ((int64_t)1 << 31)) return DAISY_EUNSUPPORTED;
  KdaIntraParams ip;
  ip.q = (const __nv_bfloat16*)q; ip.k = (const __nv_bfloat16*)k; ip.v = (const __nv_bfloat16*)v; ip.g = g;
  ip.beta = beta; ip.ws = (uint8_t*)workspace;
  ip.T = T; ip.H = H; ip.NC = NC;
  ip.scale = scale > 0.f ? scale : 1.0f / sqrtf((float)K);
  ip.l2norm = (flags & DAISY_KDA_L2NORM_QK) ? 1 : 0;
  ip.chunk_tab = chunk_tab;
  KdaStateParams sp;
  sp.ws = (const uint8_t*)workspace; sp.o = o;
  sp.T = T; sp.H = H; sp.NC = NC; sp.out_fp32 = (flags & DAISY_KDA_OUT_FP32) ? 1 : 0;
  sp.status = status_word;
  sp.chunk_tab = chunk_tab; sp.seq_ptr = seq_ptr;

  int end[KDA_PARTS];
  const int parts = seq_ptr ? 1 : kda_split(n_seq * H, NC, daisy_host::sm_count_cached(), end);
  if (parts == 1) end[0] = NC;
  float* kept = nullptr;                                      // the state between two parts
  for (int i = 0, c0 = 0; i < parts; c0 = end[i++]) {
    const bool last = i + 1 == parts;
    ip.c0 = c0; ip.behind = i > 0;
    if (daisy_host::launch_dependent(kda_intra_kernel, dim3(end[i] - c0, H, B), dim3(KI_THREADS), intra_smem, st, ip) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    DAISY_CHECK_LAUNCH();
    const int64_t ld_rec = (int64_t)NC * (REC_BYTES / 4);
    sp.h0 = i ? kept : h0; sp.ld_in = i ? ld_rec : KD * KD;
    kept = reinterpret_cast<float*>((uint8_t*)workspace + (size_t)c0 * REC_BYTES);      // over a record this part has read
    sp.hT = last ? hT : kept; sp.ld_out = last ? KD * KD : ld_rec;
    sp.c0 = c0; sp.c1 = end[i]; sp.more = !last;
    if (daisy_host::launch_dependent(kda_state_kernel, dim3(n_seq * H), dim3(KS_THREADS), KS_SMEM, st, sp) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    DAISY_CHECK_LAUNCH();
  }
  return DAISY_OK;
}

extern "C" int daisy_b200_kda_chunk_fwd(const void* q, const void* k, const void* v, const float* g,
                                        const float* beta, const float* h0, void* o, float* hT,
                                        int B, int T, int H, int K, int V, int chunk, float scale,
                                        unsigned flags, void* workspace, size_t workspace_bytes,
                                        int* status_word, void* stream) {
  if (T <= 0) return DAISY_EINVAL;
  return kda_launch(q, k, v, g, beta, h0, o, hT, B, T, H, K, V, chunk, scale, flags, workspace, workspace_bytes,
                    (T + KC - 1) / KC, B, nullptr, nullptr, status_word, stream);
}

extern "C" size_t daisy_b200_kda_varlen_workspace_bytes(int n_chunks, int H, int K, int V) {
  if (n_chunks <= 0 || H <= 0 || K != KD || V != KD) return 0;
  return (size_t)H * n_chunks * WS_REC_BYTES;
}

extern "C" int daisy_b200_kda_chunk_fwd_varlen(const void* q, const void* k, const void* v, const float* g,
                                               const float* beta, const float* h0, void* o, float* hT,
                                               int T_total, int H, int K, int V, int chunk, float scale, unsigned flags,
                                               const int32_t* chunk_tab, int n_chunks, const int32_t* seq_ptr, int n_seq,
                                               void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
  if (!chunk_tab || !seq_ptr || n_chunks <= 0 || n_seq <= 0) return DAISY_EINVAL;
  if ((reinterpret_cast<uintptr_t>(chunk_tab) & 7) || (reinterpret_cast<uintptr_t>(seq_ptr) & 3)) return DAISY_EALIGN;
  return kda_launch(q, k, v, g, beta, h0, o, hT, 1, T_total, H, K, V, chunk, scale, flags, workspace, workspace_bytes,
                    n_chunks, n_seq, chunk_tab, seq_ptr, status_word, stream);
}
