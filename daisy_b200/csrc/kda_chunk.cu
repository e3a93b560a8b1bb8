// Kimi delta attention (KDA), chunked forward, chunk = 64, K = V = 128.
//
// Per head the recurrence  S <- diag(e^{g_t}) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;
// o_t = S^T (scale q_t)  is evaluated 64 tokens at a time.  With G_i the inclusive cumulative
// log-decay inside a chunk and S_0 the state entering it:
//     A_kk[i,j] = beta_i sum_c k_ic k_jc e^{G_ic-G_jc} (j < i)     A_qk[i,j] = scale sum_c q_ic k_jc e^{G_ic-G_jc} (j <= i)
//     T = (I + A_kk)^-1          W = T (beta k e^G)          U0 = T (beta v)
//     U = U0 - W S_0             O = (scale q e^G) S_0 + A_qk U          S_C = e^{G_C} S_0 + (k e^{G_C-G})^T U
// Two kernels:
//  * kda_intra_kernel  -- everything that does not depend on the state, a small CTA per (batch, head, chunk), three to an SM:
//    Gram products in mma.sync fragments, the blocked solve of (I + A_kk) W = beta k e^G, (I + A_kk) U0 = beta v in register
//    chains.  Per chunk it writes a record of fp16 operand images (16-byte pieces exchanged so that fragment loads are
//    bank-conflict free): W^T, scale q e^G, k e^{G_C-G}, A_qk, U0^T, and e^{G_C}.
//  * kda_state_kernel  -- one CTA per (batch, head, V-slice), sequential over chunks: a producer warp
//    bulk-copies the images of chunk c+1.. into a shared-memory ring while the compute warps hold their
//    slice of S^T (16 V-rows x 128 K-columns per warp) in fp32 accumulator registers and chain the
//    three products through register-resident fragments (an accumulator tile pair is exactly the next
//    product's A fragment), so the state never leaves the register file between chunks.  With few (batch, head)
//    pairs per GPU two warps share a slice, each holding half of the K-columns.
// Tensor-core operands are fp16 (10-bit mantissa, every decay factor and operand here is <= O(1)):
// measured relative error of o against the fp32 token recurrence is ~4e-4, bf16 operands give ~3e-3.
#include <cuda_fp16.h>
#include <type_traits>
#include "common.cuh"

namespace daisy {

constexpr int KC = 64;                 // chunk length
constexpr int KD = 128;                // K = V
// per-chunk record in the workspace (bytes); every image is laid out so that ldmatrix reads it without bank conflicts after
// a plain bulk copy (rec_off, ki_off)
constexpr int OFF_WT = 0;                              // W^T      [128 channels][64 tokens] fp16
constexpr int OFF_QT = OFF_WT + KD * KC * 2;           // q~       [64 tokens][128 channels] fp16   scale q e^G
constexpr int OFF_KT = OFF_QT + KD * KC * 2;           // k~       [64 tokens][128 channels] fp16   k e^{G_C-G}
constexpr int OFF_AQK = OFF_KT + KD * KC * 2;          // A_qk     [64][64]  fp16
constexpr int OFF_D = OFF_AQK + KC * KC * 2;           // e^{G_C}  [128]     fp32
constexpr int SHARED_BYTES = OFF_D + KD * 4;           // 57856: identical for every V-slice
constexpr int OFF_UT = SHARED_BYTES;                   // U0^T     [128 value columns][64 tokens] fp16
constexpr int REC_BYTES = OFF_UT + KD * KC * 2;        // 74240
static_assert(SHARED_BYTES % 16 == 0 && REC_BYTES % 16 == 0, "bulk copies move 16-byte units");

// byte offset of (row, token column) in an image of 64-token rows (128 bytes, 16-byte pieces exchanged by row)
__device__ __forceinline__ uint32_t rec_off(int row, int col) { return (uint32_t)(row * 128 + (((col >> 3) ^ (row & 7)) << 4) + (col & 7) * 2); }
// byte offset of 16-byte piece c (0..15) of a row in an image of 128-channel rows: the eight lanes that store two half rows,
// and the eight rows of a (transposing) ldmatrix, all hit different banks
__device__ __forceinline__ uint32_t ki_off(int row, int c) { return (uint32_t)(row * 256 + ((c ^ (((row & 1) << 2) | ((row >> 1) & 3))) << 4)); }

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
// What bounds it: 22k warp instructions a chunk at 35 % issue, the rest waits for the rows of g and v with 12 warps on an SM
// (asking L2 for them at the start: 433 -> 425 us at 4 x 8192 x 16).  Lane = (2 tokens, 8 channels), as the fragments want
// it, costs three shuffles and twice the selects per product: 27k instructions, 937 us at 4 x 16384 x 16 where this takes 840.
// Why not tcgen05: the version of this kernel that built six image sets in shared memory for 128 x 64 x 128 tcgen05 products
// was a chain of hand-offs between warp groups (image -> fence -> product -> TMEM load), 20k cycles a chunk with the tensor
// pipe at 10 %; here everything between two barriers stays inside one warp and three CTAs hide each other's latency.
struct KdaIntraParams {
  const __nv_bfloat16 *q, *k, *v;
  const float *g, *beta;
  uint8_t* ws;
  int T, H, NC;            // NC = chunks per sequence
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
__device__ __forceinline__ uint4 ld_nc16(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

__device__ __forceinline__ uint2 ld_nc8(const void* p) {
  uint2 r;
  asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  return r;
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
  const int chunk = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  int t0, rows;
  ki_chunk_span(p.chunk_tab, chunk, p.T, t0, rows);
  uint8_t* rec = p.ws + ((size_t)(b * p.H + h) * p.NC + chunk) * REC_BYTES;
  const size_t tok = ((size_t)b * p.T + t0) * p.H + h, ts = (size_t)p.H * KD;      // row of token i: tok * KD + i * ts

  if (tid < KC) sm.beta[tid] = tid < rows ? p.beta[tok + (size_t)tid * p.H] : 0.f;
  for (int i = tid; i < 4 * rows; i += KI_THREADS)                                 // g and v are needed later: ask L2 for them now
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.g + tok * KD + (size_t)(i >> 2) * ts + 32 * (i & 3)));
  for (int i = tid; i < 2 * rows; i += KI_THREADS)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.v + tok * KD + (size_t)(i >> 1) * ts + 64 * (i & 1)));
  const int r0 = 16 * warp + g8, r1 = r0 + 8;                                      // this lane's two rows in the products
  const int nrow = rows - 16 * warp;                                               // rows of this block that exist (<= 0: none)
  const uint32_t s_suf = smem_u32(sm.suf[warp]), s_pk = smem_u32(sm.pk[warp]), s_pq = smem_u32(sm.pq[warp]);
  // fragment addresses: A = {k octet, q octet} x 16 channels from images at s_pk, s_pq; lane l gives row (l & 7) of matrix l >> 3
  const uint32_t s_kq = (lane & 8) ? s_pq : s_pk;

  // ---- raw rows (bf16) through shared memory: 1 / |k|, 1 / |q| and q . k are diagonals of products
  {
    const size_t base = tok * KD + (size_t)(16 * warp) * ts;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 2 * i + (lane >> 4), c = lane & 15;
      const bool ok = r < nrow;
      const uint4 kv = ok ? ld_nc16(p.k + base + r * ts + 8 * c) : make_uint4(0, 0, 0, 0), qv = ok ? ld_nc16(p.q + base + r * ts + 8 * c) : make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(sm.pk[warp] + r * KI_LD + 16 * c) = kv;
      *reinterpret_cast<uint4*>(sm.pq[warp] + r * KI_LD + 16 * c) = qv;
    }
  }
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
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    uint64_t pre[16], suf[16];                                                     // fp32 pairs: the lane's two channels
    uint32_t kh[16], qh[16];                                                       // normalised, fp16 pairs
    {
      const float* gp = p.g + tok * KD + (size_t)(16 * warp) * ts + 64 * hf + 2 * lane;
      uint2 gv[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) gv[t] = t < nrow ? ld_nc8(gp + t * ts) : make_uint2(0, 0);
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

  // ---- products with the earlier blocks
  const float b0 = sm.beta[r0], b1 = sm.beta[r1];
#pragma unroll 1
  for (int J = warp - 1; J >= 0; --J) {
    float kk[2][4], qk[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) { kk[n][0] = kk[n][1] = kk[n][2] = kk[n][3] = 0.f; qk[n][0] = qk[n][1] = qk[n][2] = qk[n][3] = 0.f; }
    const uint32_t s_c = smem_u32(sm.suf[J]) + ((lane & 7) + 8 * (lane >> 4)) * KI_LD + 16 * ((lane >> 3) & 1);
    const uint32_t ao = ((lane & 7) + 8 * ((lane >> 3) & 1)) * KI_LD + 16 * (lane >> 4);
#pragma unroll 2
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t c[4], kr[4], qr[4];
      ldmatrix_x4(c, s_c + 32 * ks);
      ldmatrix_x4(kr, s_pk + ao + 32 * ks);
      ldmatrix_x4(qr, s_pq + ao + 32 * ks);
      if (J < warp - 1) {                                                          // blocks lie between: their totals
        float2 f0 = *reinterpret_cast<const float2*>(&sm.tot[J + 1][16 * ks + 2 * t4]), f1 = *reinterpret_cast<const float2*>(&sm.tot[J + 1][16 * ks + 8 + 2 * t4]);
        if (J < warp - 2) {
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
      *reinterpret_cast<uint32_t*>(&sm.akh[r0][col]) = pack_h2(b0 * kk[n][0], b0 * kk[n][1]);
      *reinterpret_cast<uint32_t*>(&sm.akh[r1][col]) = pack_h2(b1 * kk[n][2], b1 * kk[n][3]);
      *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(r0, col)) = pack_h2(p.scale * qk[n][0], p.scale * qk[n][1]);
      *reinterpret_cast<uint32_t*>(rec + OFF_AQK + rec_off(r1, col)) = pack_h2(p.scale * qk[n][2], p.scale * qk[n][3]);
    }
  }

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
      const uint32_t off = r * KI_LD + 16 * c, roff = 4096 * warp + ki_off(r, c);
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
  //      that follow.  The four row tiles of a warp are independent chains issued side by side.
  {
    const bool is_w = warp < 2;
    uint8_t* dst = rec + (is_w ? OFF_WT : OFF_UT);
    const int c0 = 64 * (warp & 1);                                                // first row (channel or value column)
    const uint32_t src = smem_u32(is_w ? sm.pk : sm.pq) + ((lane & 7) + 8 * (lane >> 4)) * KI_LD + 2 * c0 + 16 * ((lane >> 3) & 1);
    uint32_t zf[4][3][4];                                                          // Z_J as fp16 A fragments: [row tile][J][4]
#pragma unroll
    for (int I = 0; I < 4; ++I) {
      float acc[4][2][4];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) { acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f; }
#pragma unroll
      for (int J = 0; J < I; ++J) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const __half* arow = &sm.akh[I * 16 + n * 8 + g8][J * 16 + 2 * t4];
          const uint32_t w0 = *reinterpret_cast<const uint32_t*>(arow), w1 = *reinterpret_cast<const uint32_t*>(arow + 8);
#pragma unroll
          for (int m = 0; m < 4; ++m) mma_f16(acc[m][n], zf[m][J], w0, w1);
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
      for (int m = 0; m < 4; ++m) {
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

// =============================================================================================
// inter-chunk state kernel
// =============================================================================================
struct KdaStateParams {
  const uint8_t* ws;
  const float* h0;
  float* hT;
  void* o;
  int T, H, NC, out_fp32;
  int* status;
  // packed variable-length sequences (B = 1): blockIdx.y = sequence * H + head, the sequence's chunks are
  // seq_ptr[s] .. seq_ptr[s + 1] - 1 of the packed row's NC chunks, chunk_tab as in the intra kernel; null: dense
  const int* chunk_tab;
  const int* seq_ptr;
};


// NW V-slices of 16 rows per CTA, each owned by KS warps that split the K dimension of the state between them.
// KS = 1: a warp keeps its 16 V-rows x 128 K-columns of S^T in accumulator registers and chains everything through
// register fragments.  KS > 1 (few (batch, head) pairs per GPU, where the serial chain over the chunks -- 212
// dependent mma.sync per chunk and warp -- is all that is left): warp kq holds K-columns [128 kq / KS, 128 (kq+1) / KS);
// the two products that contract over K (S^T W^T and S^T q~^T) become partial sums that the slice's warps exchange
// through shared memory once per chunk (fragment order, double-buffered, one named barrier), after which every warp
// has the whole U^T, finishes the output for its own token tiles and updates its own K-columns of the state.
template <int NW, int KS, int NST>
struct KdaStateSmem {
  static constexpr int VS = 16 * NW;
  static constexpr int CW = NW * KS;                     // compute warps
  static constexpr int U_BYTES = VS * KC * 2;
  static constexpr int STAGE = SHARED_BYTES + U_BYTES;
  static constexpr int O_LD = VS + 4;                    // floats; staging of one chunk of output
  static constexpr int XCH_WARP = 2 * 8 * 32 * 16;       // one warp's two partial accumulators: 8 tiles x 32 lanes x float4
  static constexpr int XCH = KS > 1 ? CW * XCH_WARP : 0;
  static constexpr int BYTES = NST * STAGE + KC * O_LD * 4 + XCH + 64;
};

template <int NW, int KS, int NST>
__global__ void __launch_bounds__(32 * (NW * KS + 1), 1) kda_state_kernel(const KdaStateParams p) {
  using L = KdaStateSmem<NW, KS, NST>;
  constexpr int KDA_NST = NST;                             // ring stages of chunk records
  constexpr int VS = L::VS, CW = L::CW;
  constexpr int NKT = 16 / KS;                             // this warp's 8-column tiles of the state
  constexpr int NKS = 8 / KS;                              // and its 16-deep steps of the contractions over K
  constexpr int TPW = 8 / KS;                              // token tiles whose output this warp finishes
  extern __shared__ __align__(128) uint8_t kda_smem_raw[];
  uint8_t* stages = kda_smem_raw;
  float* o_stage = reinterpret_cast<float*>(kda_smem_raw + KDA_NST * L::STAGE);
  float4* xch = reinterpret_cast<float4*>(kda_smem_raw + KDA_NST * L::STAGE + KC * L::O_LD * 4);
  uint64_t* full = reinterpret_cast<uint64_t*>(kda_smem_raw + KDA_NST * L::STAGE + KC * L::O_LD * 4 + L::XCH);
  uint64_t* empty = full + KDA_NST;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + KDA_NST);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int vsl = blockIdx.x, bh = blockIdx.y;              // bh also indexes h0 / hT
  const int h = bh % p.H;
  const int b = p.seq_ptr ? 0 : bh / p.H;
  const int c_begin = p.seq_ptr ? p.seq_ptr[bh / p.H] : 0, c_end = p.seq_ptr ? p.seq_ptr[bh / p.H + 1] : p.NC;
  const int v_base = vsl * VS;
  const uint8_t* recs = p.ws + ((size_t)(b * p.H + h) * p.NC + c_begin) * REC_BYTES;    // this sequence's first record
  const int n_chunks = c_end - c_begin;

  if (threadIdx.x == 0) {
    for (int s = 0; s < KDA_NST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], CW); }
    *abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();

  if (warp == CW) {
    // ------------------------------------------------------------ producer: bulk copies into the ring
    if (lane == 0) {
      for (int c = 0; c < n_chunks; ++c) {
        const int s = c % KDA_NST;
        if (!mbar_wait(&empty[s], ((c / KDA_NST) & 1) ^ 1, abort_flag, p.status, 1)) break;
        const uint8_t* rec = recs + (size_t)c * REC_BYTES;
        mbar_expect_tx(&full[s], L::STAGE);
        bulk_g2s(stages + s * L::STAGE, rec, SHARED_BYTES, &full[s]);
        bulk_g2s(stages + s * L::STAGE + SHARED_BYTES, rec + OFF_UT + (size_t)v_base * KC * 2, L::U_BYTES, &full[s]);
      }
    }
    return;
  }

  // ------------------------------------------------------------ compute warps: 16 V rows, 128 / KS K columns each
  const int vs = warp / KS, kq = warp % KS;
  const int vr0 = vs * 16 + g8, vr1 = vr0 + 8;                     // rows inside the CTA's V range
  float st[NKT][4];                                                // S^T[v][k]: tile j -> k = 8 (kq NKT + j) + 2 t4 (+1)
#pragma unroll
  for (int j = 0; j < NKT; ++j) {
    if (p.h0) {
      const float* hp = p.h0 + (size_t)bh * KD * KD;
      const int k0 = (kq * NKT + j) * 8 + 2 * t4;
      st[j][0] = hp[(size_t)k0 * KD + v_base + vr0]; st[j][1] = hp[(size_t)(k0 + 1) * KD + v_base + vr0];
      st[j][2] = hp[(size_t)k0 * KD + v_base + vr1]; st[j][3] = hp[(size_t)(k0 + 1) * KD + v_base + vr1];
    } else {
      st[j][0] = st[j][1] = st[j][2] = st[j][3] = 0.f;
    }
  }

  for (int c = 0; c < n_chunks; ++c) {
    const int s = c % KDA_NST;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (c / KDA_NST) & 1, abort_flag, p.status, 2));
    if (!ok) break;
    const uint8_t* sb = stages + s * L::STAGE;
    const uint32_t Wt = smem_u32(sb + OFF_WT), Qt = smem_u32(sb + OFF_QT), Kt = smem_u32(sb + OFF_KT), Aq = smem_u32(sb + OFF_AQK);
    const float* dv = reinterpret_cast<const float*>(sb + OFF_D);
    const uint8_t* Ut = sb + SHARED_BYTES;

    // (1) accU = S^T W^T   and   (2a) accO = S^T q~^T      [16 x 64 tokens each], over this warp's K columns
    float au[8][4], ao[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) { au[nt][0] = au[nt][1] = au[nt][2] = au[nt][3] = 0.f; ao[nt][0] = ao[nt][1] = ao[nt][2] = ao[nt][3] = 0.f; }
#pragma unroll
    for (int ksl = 0; ksl < NKS; ++ksl) {
      const int ks = kq * NKS + ksl;
      uint32_t a[4];
      a[0] = pack_h2(st[2 * ksl][0], st[2 * ksl][1]); a[1] = pack_h2(st[2 * ksl][2], st[2 * ksl][3]);
      a[2] = pack_h2(st[2 * ksl + 1][0], st[2 * ksl + 1][1]); a[3] = pack_h2(st[2 * ksl + 1][2], st[2 * ksl + 1][3]);
      // B fragments of two token tiles per ldmatrix.x4, matrix m = (channel octet m & 1, token tile nt + (m >> 1)): W^T rows
      // are channels (transposing form), q~ rows are tokens
      const int wrow = ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), qrow = (lane & 7) + 8 * (lane >> 4), qpc = 2 * ks + ((lane >> 3) & 1);
#pragma unroll
      for (int nt = 0; nt < 8; nt += 2) {
        uint32_t bw[4], bq[4];
        ldmatrix_x4_t(bw, Wt + rec_off(wrow, (nt + (lane >> 4)) * 8));
        ldmatrix_x4(bq, Qt + ki_off(nt * 8 + qrow, qpc));
        mma_f16(au[nt], a, bw[0], bw[1]);
        mma_f16(ao[nt], a, bq[0], bq[1]);
        mma_f16(au[nt + 1], a, bw[2], bw[3]);
        mma_f16(ao[nt + 1], a, bq[2], bq[3]);
      }
    }
    if (KS > 1) {
      // exchange: every warp of the slice needs the whole accU; accO only for the token tiles it finishes.  The sums
      // run over the warps in a fixed order, so all of them hold the same bits.
      float4* mine = xch + (size_t)warp * (L::XCH_WARP / 16);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        mine[nt * 32 + lane] = make_float4(au[nt][0], au[nt][1], au[nt][2], au[nt][3]);
        mine[256 + nt * 32 + lane] = make_float4(ao[nt][0], ao[nt][1], ao[nt][2], ao[nt][3]);
      }
      named_bar(2 + vs, 32 * KS);
      const float4* slice = xch + (size_t)(vs * KS) * (L::XCH_WARP / 16);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        float4 t = slice[nt * 32 + lane];
#pragma unroll
        for (int q = 1; q < KS; ++q) {
          const float4 u = slice[q * (L::XCH_WARP / 16) + nt * 32 + lane];
          t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
        }
        au[nt][0] = t.x; au[nt][1] = t.y; au[nt][2] = t.z; au[nt][3] = t.w;
      }
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        if (nt / TPW != kq) continue;                                // compile-time tile index, warp-uniform test
        float4 t = slice[256 + nt * 32 + lane];
#pragma unroll
        for (int q = 1; q < KS; ++q) {
          const float4 u = slice[q * (L::XCH_WARP / 16) + 256 + nt * 32 + lane];
          t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
        }
        ao[nt][0] = t.x; ao[nt][1] = t.y; ao[nt][2] = t.z; ao[nt][3] = t.w;
      }
      named_bar(2 + vs, 32 * KS);                                    // everybody has read: the next chunk may overwrite
    }
    // U^T = U0^T - accU, as fp16 A fragments over the token axis
    uint32_t ua[4][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int tok = nt * 8 + 2 * t4;
      const float2 u0 = unpack_h2(*reinterpret_cast<const uint32_t*>(Ut + rec_off(vr0, tok)));
      const float2 u1 = unpack_h2(*reinterpret_cast<const uint32_t*>(Ut + rec_off(vr1, tok)));
      const uint32_t lo = pack_h2(u0.x - au[nt][0], u0.y - au[nt][1]);
      const uint32_t hi = pack_h2(u1.x - au[nt][2], u1.y - au[nt][3]);
      ua[nt >> 1][(nt & 1) * 2 + 0] = lo;
      ua[nt >> 1][(nt & 1) * 2 + 1] = hi;
    }
    // (2b) accO += U^T A_qk^T, for the token tiles this warp finishes
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const int lrow = (lane >> 4) * 8 + (lane & 7), lcol = ks * 16 + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int nt = 2 * ks; nt < 8; nt += 2) {                     // A_qk[i][j] = 0 for j > i: tiles below 2 ks are empty
        if (KS > 1 && nt / TPW != kq) continue;
        uint32_t ba[4];
        ldmatrix_x4(ba, Aq + rec_off(nt * 8 + lrow, lcol));
        mma_f16(ao[nt], ua[ks], ba[0], ba[1]);
        mma_f16(ao[nt + 1], ua[ks], ba[2], ba[3]);
      }
    }
    // (3) S^T = S^T diag(e^{G_C}) + U^T k~, this warp's K columns
#pragma unroll
    for (int j = 0; j < NKT; ++j) {
      const float2 d2 = *reinterpret_cast<const float2*>(&dv[(kq * NKT + j) * 8 + 2 * t4]);
      st[j][0] *= d2.x; st[j][1] *= d2.y; st[j][2] *= d2.x; st[j][3] *= d2.y;
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const int krow = ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);            // k~ rows are tokens: transposing form
#pragma unroll
      for (int j = 0; j < NKT; j += 2) {
        uint32_t bk[4];
        ldmatrix_x4_t(bk, Kt + ki_off(krow, kq * NKT + j + (lane >> 4)));
        mma_f16(st[j], ua[ks], bk[0], bk[1]);
        mma_f16(st[j + 1], ua[ks], bk[2], bk[3]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);                         // this warp is done with the stage

    // output: stage [token][v] in shared memory, then coalesced rows
    asm volatile("bar.sync 1, %0;" ::"n"(32 * CW) : "memory");    // previous chunk's copy-out finished
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      if (KS > 1 && nt / TPW != kq) continue;
      const int tok = nt * 8 + 2 * t4;
      o_stage[tok * L::O_LD + vr0] = ao[nt][0]; o_stage[(tok + 1) * L::O_LD + vr0] = ao[nt][1];
      o_stage[tok * L::O_LD + vr1] = ao[nt][2]; o_stage[(tok + 1) * L::O_LD + vr1] = ao[nt][3];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * CW) : "memory");
    int t0, rows;
    ki_chunk_span(p.chunk_tab, c_begin + c, p.T, t0, rows);
    for (int idx = threadIdx.x; idx < KC * (VS / 4); idx += 32 * CW) {
      const int tok = idx / (VS / 4), v4 = (idx % (VS / 4)) * 4;
      if (tok >= rows) continue;
      const float4 x = *reinterpret_cast<const float4*>(&o_stage[tok * L::O_LD + v4]);
      const size_t off = (((size_t)b * p.T + (size_t)t0 + tok) * p.H + h) * KD + v_base + v4;
      if (p.out_fp32) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.o) + off) = x;
      } else {
        uint2 pk = make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.o) + off) = pk;
      }
    }
  }

  if (p.hT) {
    float* hp = p.hT + (size_t)bh * KD * KD;
#pragma unroll
    for (int j = 0; j < NKT; ++j) {
      const int k0 = (kq * NKT + j) * 8 + 2 * t4;
      hp[(size_t)k0 * KD + v_base + vr0] = st[j][0]; hp[(size_t)(k0 + 1) * KD + v_base + vr0] = st[j][1];
      hp[(size_t)k0 * KD + v_base + vr1] = st[j][2]; hp[(size_t)(k0 + 1) * KD + v_base + vr1] = st[j][3];
    }
  }
}

}  // namespace daisy

using namespace daisy;

extern "C" size_t daisy_b200_kda_workspace_bytes(int B, int T, int H, int K, int V) {
  if (B <= 0 || T <= 0 || H <= 0 || K != KD || V != KD) return 0;
  const size_t nc = (size_t)(T + KC - 1) / KC;
  return (size_t)B * H * nc * REC_BYTES;
}

template <int NW, int KS, int NST>
static int launch_state(const KdaStateParams& sp, int BH, cudaStream_t st) {
  using L = KdaStateSmem<NW, KS, NST>;
  static_assert(L::BYTES <= 232448, "over the 227 KB a CTA may use");
  static bool attr[daisy_host::MAX_DEVICES] = {};             // the attribute is per device
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(kda_state_kernel<NW, KS, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES) != cudaSuccess) return DAISY_ECUDA;
    attr[dev] = true;
  }
  kda_state_kernel<NW, KS, NST><<<dim3(KD / L::VS, BH), 32 * (L::CW + 1), L::BYTES, st>>>(sp);
  return cudaGetLastError() == cudaSuccess ? DAISY_OK : DAISY_ECUDA;
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
  if (workspace_bytes < (size_t)B * H * NC * REC_BYTES) return DAISY_EWORKSPACE;
  if (!daisy_aligned16(q) || !daisy_aligned16(k) || !daisy_aligned16(v) || !daisy_aligned16(g) || !daisy_aligned16(o) ||
      !daisy_aligned16(workspace) || (h0 && !daisy_aligned16(h0)) || (hT && !daisy_aligned16(hT)))
    return DAISY_EALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  static bool attr[daisy_host::MAX_DEVICES] = {};             // the attribute is per device
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  constexpr int intra_smem = (int)sizeof(KdaIntraSmem);
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(kda_intra_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, intra_smem) != cudaSuccess) {
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
  kda_intra_kernel<<<dim3(NC, H, B), KI_THREADS, intra_smem, st>>>(ip);
  DAISY_CHECK_LAUNCH();

  KdaStateParams sp;
  sp.ws = (const uint8_t*)workspace; sp.h0 = h0; sp.hT = hT; sp.o = o;
  sp.T = T; sp.H = H; sp.NC = NC; sp.out_fp32 = (flags & DAISY_KDA_OUT_FP32) ? 1 : 0;
  sp.status = status_word;
  sp.chunk_tab = chunk_tab; sp.seq_ptr = seq_ptr;
  const int BH = n_seq * H;
  // V-slices: 64 rows (4 warps) fill the machine when there are >= 48 (sequence, head) pairs; fewer take narrower slices
  int rc;
  if (BH * 2 >= 96) rc = launch_state<4, 1, 2>(sp, BH, st);
  else if (BH * 4 >= 96) rc = launch_state<2, 2, 2>(sp, BH, st);
  else rc = launch_state<1, 2, 3>(sp, BH, st);
  if (rc != DAISY_OK) { (void)cudaGetLastError(); return rc; }
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
  return (size_t)H * n_chunks * REC_BYTES;
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
