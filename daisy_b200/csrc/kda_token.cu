// One decoded token through a Kimi-delta-attention layer: the projections, the short convolutions with their
// carried state, the decay gate, the recurrent state update, the gated norm and the output projection
// (KimiLinearSelfAttention.step, models/daisy/attention_kimi.py:128-211 with T = 1 and the cached states).  One launch up to
// TK_MAX_B rows and KT_ONE_PAIRS (row, head) pairs, four above (kda_batch_kernel).
//
// Bound: HBM and latency -- at dim 2048 and batch 1 the weights are 35 MB (5.4 us at copy bandwidth) and the state 2 MB, but
// as seventeen dependent launches of 2-5 us the step took 79 us replayed as a graph and 278 us issued from Python.  As in
// swa_token.cu a persistent CTA per SM streams its share of the weights through per-warp rings that run ahead of the
// phases, and the phases exchange vectors as tagged words:
//   Phase A  16-row tiles of [q; k; v; f0; g0; b] x -> the thread that sums a q / k / v row owns that channel's convolution
//            state, so convolution, SiLU and the state's shift are the projection's epilogue
//   Phase B  one CTA per (batch, head): decay gate (f1 row block x f0), output gate (g1 row block x g0), the 128 x 128 state in
//            registers (8 warps), gated norm -> o.  Its 128 KB of state and weights are asked of L2 when the kernel starts.
//   Phase C  16-row tiles of the output projection -> y
// Every value is rounded to bf16 where the chain of kernels stores it as bf16, so both give the same numbers up to the order
// of fp32 sums.
#include "token_common.cuh"

namespace daisy {

struct KdaTokenParams {
  CUtensorMap tw[7];                                  // q, k, v [dim, dim]; f0, g0 [128, dim]; b [H, dim]; o [dim, dim]
  const __nv_bfloat16 *f1, *g1, *g1_bias, *norm_w;    // [dim, 128], [dim, 128], [dim] or null, [128] or null
  const __nv_bfloat16 *conv_w[3], *conv_b[3];         // [dim, 4], [dim] or null
  __nv_bfloat16* conv_s[3];                           // [B, dim, 4], shifted in place
  const float *a_log, *dt_bias;                       // [H], [dim]
  float* state;                                       // [B, H, 128, 128], updated in place
  const __nv_bfloat16* x; int64_t x_sb;
  __nv_bfloat16* y;
  int B, H, dim, depth, silu;
  float eps, scale;
  unsigned* epoch;
  uint2 *qkv, *fg, *bl, *o;                           // words: [B, 3 dim / 2], [B, 128], [B, 8], [TK_COPIES][B, dim / 2]
  int* status;
};

struct KdaTokenBars {
  uint64_t full[TK_CW * TK_DEPTH];
  int abort_flag;
};

struct KdaTokenStream : TokenRing {
  const KdaTokenParams& p;
  int t0, na, c0, nc, ks_n, i;                        // first tile and pieces of phases A and C; next piece to load
  __device__ explicit KdaTokenStream(const KdaTokenParams& p_) : p(p_) {}
  // tile of phase A -> matrix and first row
  static __device__ __forceinline__ int matrix(int tile, int dim, int& row) {
    const int per = dim / 16;
    if (tile < 3 * per) { const int m = tile < per ? 0 : tile < 2 * per ? 1 : 2; row = 16 * (tile - m * per); return m; }
    tile -= 3 * per;
    row = 16 * (tile & 7);
    return 3 + (tile >> 3);
  }
  __device__ __forceinline__ void load(int at) {
    if (i >= na + nc) return;
    mbar_expect_tx(&full[at], TK_PIECE);
    const int k = i < na ? i : i - na, tile = k / ks_n, kb = k - tile * ks_n;
    int m = 6, row = 16 * (c0 + tile);
    if (i < na) m = matrix(t0 + tile, p.dim, row);
    tk_tma3(buf + at * TK_PIECE, &p.tw[m], &full[at], 0, row, kb * (TK_KW / 64));
    i += TK_CW;
  }
};

__device__ __forceinline__ float kt_sigmoid(float a) { return __fdividef(1.f, 1.f + fast_exp2(a * -1.4426950408889634f)); }

// two channels of the short convolution: state s (the last four inputs of each, oldest first), taps w, new inputs v
__device__ __forceinline__ void kt_conv(const uint4& s, const uint4& w, uint32_t v, const __nv_bfloat16* bias, int silu, float* out) {
  float st[8], wt[8];
  unpack8(s, st); unpack8(w, wt);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float cur = e ? bf16_hi(v) : bf16_lo(v);
    float a = bias ? __bfloat162float(bias[e]) : 0.f;
    a = fmaf(wt[4 * e], st[4 * e + 1], a);
    a = fmaf(wt[4 * e + 1], st[4 * e + 2], a);
    a = fmaf(wt[4 * e + 2], st[4 * e + 3], a);
    a = fmaf(wt[4 * e + 3], cur, a);
    out[e] = silu ? a * kt_sigmoid(a) : a;
  }
}
__device__ __forceinline__ uint4 kt_shift(const uint4& s, uint32_t v) {
  return make_uint4(s.x >> 16 | s.y << 16, s.y >> 16 | v << 16, s.z >> 16 | s.w << 16, s.w >> 16 | (v & 0xffff0000u));
}

// ---- one (batch, head), its vectors in shared memory: sv [9][128] = q, k, v, f0, g0, decay, output gate, two partial sums; sv[9 * 128]
//      the write strength
// decay gate (f1 row block x f0) and output gate (g1 row block x g0): half-warp hw takes rows hw, hw + HW, ..  (A sum at a time, its gate by
// one lane of sixteen: the exponentials eleven or sixteen times one after the other.)
template <int HW> struct KtGateRows { static constexpr int N = (256 + HW - 1) / HW; uint4 w[N]; };
template <int HW>
__device__ __forceinline__ void kt_gate_rows(KtGateRows<HW>& rows, const __nv_bfloat16* f1, const __nv_bfloat16* g1, int h, int tid) {
  const int hw = tid >> 4, sub = tid & 15;
#pragma unroll
  for (int k = 0; k < KtGateRows<HW>::N; ++k) {
    const int r = hw + HW * k;
    if (r < 256) rows.w[k] = __ldg(reinterpret_cast<const uint4*>((r < 128 ? f1 : g1) + ((size_t)h * 128 + (r & 127)) * 128 + 8 * sub));
  }
}
template <int HW>
__device__ __forceinline__ void kt_gates(float* sv, const KtGateRows<HW>& rows, const __nv_bfloat16* g1_bias, const float* a_log, const float* dt_bias, int h, int tid) {
  const int hw = tid >> 4, sub = tid & 15;
  float f[8], g[8];
  *reinterpret_cast<float4*>(f) = reinterpret_cast<const float4*>(sv + 3 * 128)[2 * sub]; *reinterpret_cast<float4*>(f + 4) = reinterpret_cast<const float4*>(sv + 3 * 128)[2 * sub + 1];
  *reinterpret_cast<float4*>(g) = reinterpret_cast<const float4*>(sv + 4 * 128)[2 * sub]; *reinterpret_cast<float4*>(g + 4) = reinterpret_cast<const float4*>(sv + 4 * 128)[2 * sub + 1];
  constexpr int N = KtGateRows<HW>::N;
  static_assert(N <= 16, "a row for each lane of a half-warp");
  float d[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    d[k] = 0.f;
    const int r = hw + HW * k;
    if (k < N && r < 256) {
      float w[8];
      unpack8(rows.w[k < N ? k : 0], w);
#pragma unroll
      for (int e = 0; e < 8; ++e) d[k] = fmaf(w[e], r < 128 ? f[e] : g[e], d[k]);
    }
  }
  // sixteen sums over sixteen lanes, half of them handed on at each step: lane `sub` ends with row hw + HW sub
#pragma unroll
  for (int m = 8; m >= 1; m >>= 1) {
    const bool up = (sub & m) != 0;
#pragma unroll
    for (int i = 0; i < m; ++i) d[i] = (up ? d[i + m] : d[i]) + __shfl_xor_sync(0xffffffffu, up ? d[i] : d[i + m], m);
  }
  const int r = hw + HW * sub;
  if (r < 256) {
    float x = __bfloat162float(__float2bfloat16_rn(d[0]));
    if (r < 128) {                                    // decay e^g, g = -exp(A) softplus(f + dt_bias) at bf16
      const float z = x + __ldg(dt_bias + h * 128 + r);
      const float sp_ = z > 20.f ? z : log1pf(expf(z));
      sv[5 * 128 + r] = __expf(__bfloat162float(__float2bfloat16_rn(-expf(__ldg(a_log + h)) * sp_)));
    } else {
      if (g1_bias) x = __bfloat162float(__float2bfloat16_rn(x + __bfloat162float(g1_bias[h * 128 + r - 128])));
      sv[6 * 128 + r - 128] = x;
    }
  }
}
// state update and gated norm by 256 threads (value column tid & 127, keys 64 (tid >> 7) ..); store(columns 4 lane, + 1; + 2, + 3) by warp 0
template <typename Store>
__device__ __forceinline__ void kt_update(float (&S)[64], float* sv, const __nv_bfloat16* norm_w, float eps, int tid, Store&& store) {
  const int vcol = tid & 127, kq = tid >> 7, lane = tid & 31;
    const float* dk = sv + 5 * 128 + 64 * kq;
    const float* kk = sv + 128 + 64 * kq;
    float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      const float4 d4 = *reinterpret_cast<const float4*>(dk + i), k4 = *reinterpret_cast<const float4*>(kk + i);
      S[i] *= d4.x; S[i + 1] *= d4.y; S[i + 2] *= d4.z; S[i + 3] *= d4.w;
      dot[0] = fmaf(S[i], k4.x, dot[0]); dot[1] = fmaf(S[i + 1], k4.y, dot[1]);
      dot[2] = fmaf(S[i + 2], k4.z, dot[2]); dot[3] = fmaf(S[i + 3], k4.w, dot[3]);
    }
    sv[(7 + kq) * 128 + vcol] = (dot[0] + dot[1]) + (dot[2] + dot[3]);
    named_bar(2, 256);
    const float ut = sv[9 * 128] * (sv[2 * 128 + vcol] - (sv[7 * 128 + vcol] + sv[8 * 128 + vcol]));
    named_bar(2, 256);
    const float* qq = sv + 64 * kq;
    float od[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      const float4 k4 = *reinterpret_cast<const float4*>(kk + i), q4 = *reinterpret_cast<const float4*>(qq + i);
      S[i] = fmaf(k4.x, ut, S[i]); S[i + 1] = fmaf(k4.y, ut, S[i + 1]); S[i + 2] = fmaf(k4.z, ut, S[i + 2]); S[i + 3] = fmaf(k4.w, ut, S[i + 3]);
      od[0] = fmaf(S[i], q4.x, od[0]); od[1] = fmaf(S[i + 1], q4.y, od[1]); od[2] = fmaf(S[i + 2], q4.z, od[2]); od[3] = fmaf(S[i + 3], q4.w, od[3]);
    }
    sv[(7 + kq) * 128 + vcol] = (od[0] + od[1]) + (od[2] + od[3]);
    named_bar(2, 256);
    if (tid < 32) {                                // gated norm: lane = 4 value columns
      float4 a = reinterpret_cast<const float4*>(sv + 7 * 128)[lane], c = reinterpret_cast<const float4*>(sv + 8 * 128)[lane];
      const float4 gt = reinterpret_cast<const float4*>(sv + 6 * 128)[lane];
      const uint32_t o01 = pack_bf16(a.x + c.x, a.y + c.y), o23 = pack_bf16(a.z + c.z, a.w + c.w);
      float x[4] = {bf16_lo(o01), bf16_hi(o01), bf16_lo(o23), bf16_hi(o23)};
      const float gg[4] = {gt.x, gt.y, gt.z, gt.w};
      const float rstd = rsqrtf(tk_warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]) * (1.0f / 128) + eps);
      float r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float n = x[e] * (rstd * (norm_w ? __bfloat162float(norm_w[4 * lane + e]) : 1.f)), s = kt_sigmoid(gg[e]);
        r[e] = __bfloat162float(__float2bfloat16_rn(n * gg[e] * s)) * __bfloat162float(__float2bfloat16_rn(s));
      }
      const uint32_t r01 = pack_bf16(r[0], r[1]), r23 = pack_bf16(r[2], r[3]);
      store(r01, r23);
    }
}

template <int NB>
__global__ void __launch_bounds__(TK_CT, 1) kda_token_kernel(const __grid_constant__ KdaTokenParams p) {
  extern __shared__ __align__(128) uint8_t kt_smem[];
  KdaTokenBars* bars = reinterpret_cast<KdaTokenBars*>(kt_smem);
  const uint32_t ring = (smem_u32(kt_smem) + sizeof(KdaTokenBars) + 1023) & ~1023u;
  uint8_t* after = kt_smem + (ring - smem_u32(kt_smem)) + TK_CW * p.depth * TK_PIECE;
  float* sv = reinterpret_cast<float*>(after);        // [9][128]: q, k, v, f0, g0, decay, output gate, two partial sums
  uint8_t* xs = after + 10 * 512;
  const int xs_ld = (p.dim + 8) * 2;
  float* psum = reinterpret_cast<float*>(xs + p.B * xs_ld);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;

  if (tid == 0) {
    for (int i = 0; i < TK_CW * TK_DEPTH; ++i) mbar_init(&bars->full[i], 1);
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  const uint32_t tag = *p.epoch + 1;
  const int ks_n = (p.dim + TK_KW - 1) / TK_KW, per = p.dim / 16, ta = 3 * per + 16 + (p.H + 15) / 16;
  const int t0 = cta * ta / G, t1 = (cta + 1) * ta / G, o0 = cta * per / G, o1 = (cta + 1) * per / G;
  __syncthreads();
  KdaTokenStream in(p);
  in.full = bars->full + warp * TK_DEPTH; in.buf = ring + warp * (p.depth * TK_PIECE);
  in.depth = p.depth; in.st = in.par = 0; in.skip = warp; in.abort_flag = abort_flag; in.status = p.status;
  in.t0 = t0; in.na = (t1 - t0) * ks_n; in.c0 = o0; in.nc = (o1 - o0) * ks_n; in.ks_n = ks_n; in.i = warp;
  if (lane == 0)
    for (int i = 0; i < p.depth; ++i) in.load(i);
  const int units = p.B * p.H;
  if (cta < units && tid < 4) {                       // this CTA's (batch, head): state, f1 and g1 blocks
    const int h = cta % p.H;
    if (tid < 2) l2_prefetch_bulk(p.state + (size_t)cta * 128 * 128 + tid * 8192, 32768);
    else l2_prefetch_bulk((tid == 2 ? p.f1 : p.g1) + (size_t)h * 128 * 128, 32768);
  }
  // the convolution's inputs of this thread's first row pair, ahead of the sums
  const int pairs = (t1 - t0) * 8;
  uint4 cs = make_uint4(0, 0, 0, 0), cw = cs;
  if (tid < pairs * p.B) {
    const int b = p.B == 1 ? 0 : tid / pairs, r = 2 * (tid - b * pairs);
    int row;
    const int m = KdaTokenStream::matrix(t0 + (r >> 4), p.dim, row);
    if (m < 3) {
      cs = *reinterpret_cast<const uint4*>(p.conv_s[m] + ((size_t)b * p.dim + row + (r & 15)) * 4);
      cw = __ldg(reinterpret_cast<const uint4*>(p.conv_w[m] + (size_t)(row + (r & 15)) * 4));
    }
  }
  uint32_t swz[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = (lane & 7) + 8 * ((lane >> 3) & 1);
    swz[j] = row * 128 + (((2 * j + (lane >> 4)) ^ (row & 7)) << 4);
  }
  // ---- phase A
  for (int b = 0; b < p.B; ++b)
    for (int k = tid; k < p.dim / 8; k += TK_CT) *reinterpret_cast<uint4*>(xs + b * xs_ld + k * 16) = ld_cg16(p.x + b * p.x_sb + k * 8);
  tk_project<NB>(in, psum, smem_u32(xs), xs_ld, p.B, p.dim, in.na, pairs, swz, lane, [&](bool first, int b, int r, float s0, float s1) {
    int row;
    const int m = KdaTokenStream::matrix(t0 + (r >> 4), p.dim, row);
    row += r & 15;
    uint32_t v = pack_bf16(s0, s1);                   // as the projection stores it
    if (m < 3) {
      __nv_bfloat16* sp = p.conv_s[m] + ((size_t)b * p.dim + row) * 4;
      uint4 s = cs, w = cw;
      if (!first) { s = *reinterpret_cast<const uint4*>(sp); w = __ldg(reinterpret_cast<const uint4*>(p.conv_w[m] + (size_t)row * 4)); }
      float out[2];
      kt_conv(s, w, v, p.conv_b[m] ? p.conv_b[m] + row : nullptr, p.silu, out);
      *reinterpret_cast<uint4*>(sp) = kt_shift(s, v);
      tk_put2(p.qkv + (size_t)b * 3 * (p.dim / 2) + m * (p.dim / 2) + (row >> 1), pack_bf16(out[0], out[1]), tag);
    } else if (m < 5) {
      tk_put2(p.fg + (size_t)b * 128 + (m - 3) * 64 + (row >> 1), v, tag);
    } else {
      tk_put2(p.bl + (size_t)b * 8 + (row >> 1), v, tag);
    }
  });
  // ---- phase B
  for (int u = cta; u < units; u += G) {
    const int b = u / p.H, h = u - b * p.H;
    float S[64];                                      // threads 0 .. 255: value column tid & 127, keys 64 (tid >> 7) ..
    float* sp = p.state + (size_t)u * 128 * 128 + (size_t)(tid >> 7) * 64 * 128 + (tid & 127);
    if (tid < 256) {
#pragma unroll
      for (int i = 0; i < 64; ++i) S[i] = __ldcg(sp + i * 128);
    }
    KtGateRows<TK_CT / 16> gate_rows;                 // on their way while the vectors are waited for
    kt_gate_rows(gate_rows, p.f1, p.g1, h, tid);
    if (warp < 5) {                                   // q, k, v, f0, g0
      const uint2* src = warp < 3 ? p.qkv + (size_t)b * 3 * (p.dim / 2) + warp * (p.dim / 2) + h * 64 : p.fg + (size_t)b * 128 + (warp - 3) * 64;
      uint4 r[1];
      tk_get(reinterpret_cast<const uint4*>(src) + lane, 0, r, tag, abort_flag, p.status);
      float x[4] = {bf16_lo(r[0].x), bf16_hi(r[0].x), bf16_lo(r[0].z), bf16_hi(r[0].z)};
      if (warp < 2) {                                 // q, k: L2 norm
        const float n = rsqrtf(tk_warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]) + 1e-6f) * (warp == 0 ? p.scale : 1.f);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] *= n;
      }
      reinterpret_cast<float4*>(sv + warp * 128)[lane] = make_float4(x[0], x[1], x[2], x[3]);
    } else if (tid == 160) {                          // the write strength: sigmoid at bf16, as the layer computes it
      uint4 r[1];
      tk_get(reinterpret_cast<const uint4*>(p.bl + (size_t)b * 8) + (h >> 2), 0, r, tag, abort_flag, p.status);
      const uint32_t w = (h & 2) ? r[0].z : r[0].x;
      const float z = (h & 1) ? bf16_hi(w) : bf16_lo(w);
      sv[9 * 128] = __bfloat162float(__float2bfloat16_rn(kt_sigmoid(z)));
    }
    named_bar(1, TK_CT);
    kt_gates(sv, gate_rows, p.g1_bias, p.a_log, p.dt_bias, h, tid);
    named_bar(1, TK_CT);
    if (tid < 256) {
      kt_update(S, sv, p.norm_w, p.eps, tid, [&](uint32_t r01, uint32_t r23) {
#pragma unroll
        for (int c4 = 0; c4 < TK_COPIES; ++c4)
          tk_put4(reinterpret_cast<uint4*>(p.o + (size_t)(c4 * p.B + b) * (p.dim / 2) + h * 64) + lane, r01, r23, tag);
      });
#pragma unroll
      for (int i = 0; i < 64; ++i) sp[i * 128] = S[i];
    }
    if (u + G < units) named_bar(1, TK_CT);           // the next unit overwrites the staged vectors
  }
  // ---- phase C
  for (int b = 0; b < p.B; ++b)
    tk_gather(xs + b * xs_ld, p.o + (size_t)(cta % TK_COPIES * p.B + b) * (p.dim / 2), p.dim / 4, tag, abort_flag, p.status);
  tk_project<NB>(in, psum, smem_u32(xs), xs_ld, p.B, p.dim, in.nc, (o1 - o0) * 8, swz, lane, [&](bool, int b, int r, float s0, float s1) {
    *reinterpret_cast<uint32_t*>(p.y + (size_t)b * p.dim + 16 * o0 + r) = pack_bf16(s0, s1);
  });
  in.drain();
  if (tid == 0 && cta == 0) *p.epoch = tag;           // every CTA has contributed by now, hence read the tag
}

// ---------------------------------------------------------------------------------------------
// The same step for batches that are not the launch above's (kt_one_launch): projections by the GEMM, everything between by this
// kernel, one CTA per (batch, head).  It is bound by the state, 64 KB in and out (12 heads x 54 rows: 85 MB, 13 us at copy
// bandwidth); the gates' second projections are formed here (64 KB of weights a CTA, from L2) rather than as two more products.
struct KdaBatchParams {
  const __nv_bfloat16 *x, *pr[3], *f0, *g0;           // [B, dim] (row stride x_sb); projections [B, dim] and [B, 128]
  const __nv_bfloat16 *b_w, *f1, *g1, *g1_bias, *norm_w, *conv_w[3], *conv_b[3];
  __nv_bfloat16 *conv_s[3], *o;                       // o [B, dim]
  const float *a_log, *dt_bias;
  float* state;
  int64_t x_sb;
  int H, dim, silu;
  float eps, scale;
};

__global__ void __launch_bounds__(256, 2) kda_batch_kernel(const __grid_constant__ KdaBatchParams p) {
  __shared__ __align__(16) float sv[9 * 128 + 4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, u = blockIdx.x, h = u % p.H, b = u / p.H;
  if (tid < 2) l2_prefetch_bulk(p.state + (size_t)u * 128 * 128 + tid * 8192, 32768);
  else if (tid < 4) l2_prefetch_bulk((tid == 2 ? p.f1 : p.g1) + (size_t)h * 128 * 128, 32768);
  grid_dep_launch();
  grid_dep_wait();
  float S[64];
  float* sp = p.state + (size_t)u * 128 * 128 + (size_t)(tid >> 7) * 64 * 128 + (tid & 127);
#pragma unroll
  for (int i = 0; i < 64; ++i) S[i] = __ldcg(sp + i * 128);
  if (warp < 3) {                                     // convolution of q, k, v: four channels a lane
    const int ch = h * 128 + 4 * lane;
    __nv_bfloat16* cs = p.conv_s[warp] + ((size_t)b * p.dim + ch) * 4;
    const uint2 cur2 = *reinterpret_cast<const uint2*>(p.pr[warp] + (size_t)b * p.dim + ch);
    float x[4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint32_t v = half ? cur2.y : cur2.x;
      const uint4 s = *reinterpret_cast<const uint4*>(cs + 8 * half), w = __ldg(reinterpret_cast<const uint4*>(p.conv_w[warp] + (size_t)(ch + 2 * half) * 4));
      float out[2];
      kt_conv(s, w, v, p.conv_b[warp] ? p.conv_b[warp] + ch + 2 * half : nullptr, p.silu, out);
      *reinterpret_cast<uint4*>(cs + 8 * half) = kt_shift(s, v);
      const uint32_t r = pack_bf16(out[0], out[1]);
      x[2 * half] = bf16_lo(r); x[2 * half + 1] = bf16_hi(r);
    }
    if (warp < 2) {                                   // q, k: L2 norm
      const float n = rsqrtf(tk_warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]) + 1e-6f) * (warp == 0 ? p.scale : 1.f);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] *= n;
    }
    reinterpret_cast<float4*>(sv + warp * 128)[lane] = make_float4(x[0], x[1], x[2], x[3]);
  } else if (warp < 5) {
    const uint2 r = *reinterpret_cast<const uint2*>((warp == 3 ? p.f0 : p.g0) + (size_t)b * 128 + 4 * lane);
    reinterpret_cast<float4*>(sv + warp * 128)[lane] = make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
  } else if (warp == 5) {                             // the write strength: sigmoid at bf16, as the layer computes it
    float d = 0.f;
#pragma unroll 4
    for (int k = 8 * lane; k < p.dim; k += 256) {
      float a[8], w[8];
      unpack8(*reinterpret_cast<const uint4*>(p.x + b * p.x_sb + k), a);
      unpack8(__ldg(reinterpret_cast<const uint4*>(p.b_w + (size_t)h * p.dim + k)), w);
#pragma unroll
      for (int e = 0; e < 8; ++e) d = fmaf(a[e], w[e], d);
    }
    d = tk_warp_sum(d);
    if (lane == 0) sv[9 * 128] = __bfloat162float(__float2bfloat16_rn(kt_sigmoid(__bfloat162float(__float2bfloat16_rn(d)))));
  }
  __syncthreads();
  KtGateRows<16> gate_rows;
  kt_gate_rows(gate_rows, p.f1, p.g1, h, tid);
  kt_gates(sv, gate_rows, p.g1_bias, p.a_log, p.dt_bias, h, tid);
  __syncthreads();
  kt_update(S, sv, p.norm_w, p.eps, tid, [&](uint32_t r01, uint32_t r23) {
    *reinterpret_cast<uint2*>(p.o + (size_t)b * p.dim + h * 128 + 4 * lane) = make_uint2(r01, r23);
  });
#pragma unroll
  for (int i = 0; i < 64; ++i) sp[i * 128] = S[i];
}

}  // namespace daisy

using namespace daisy;

static inline size_t kt_align(size_t n) { return (n + 255) / 256 * 256; }

// One launch, or four: the one gives each (batch, head) pair a CTA and has to take turns where there are more than SMs.  One launch
// against four, us: 16 heads 9 rows (144 pairs) 23.1 / 26.4, 11 (176) 27.4 / 26.6, 16 (256) 32.7 / 27.1; 12 heads 13 rows (156)
// 27.4 / 28.2, 16 (192) 29.4 / 28.4; 8 heads 16 rows (128) 23.2 / 26.0.
constexpr int KT_ONE_PAIRS = 168;
static bool kt_one_launch(int B, int H) { return B <= TK_MAX_B && B * H <= KT_ONE_PAIRS; }
// the exchange's words, up to TK_MAX_B rows; scratch of the four launches lies behind them, so that a buffer serves both
static size_t kt_words(size_t B, size_t dim) {
  if (B > TK_MAX_B) return 0;
  return 256 + kt_align(B * 3 * dim * 4) + kt_align(B * 128 * 8) + kt_align(B * 64) + TK_COPIES * kt_align(B * dim * 4);
}

extern "C" size_t daisy_b200_kda_token_workspace_bytes(int B, int H, int D) {
  if (B <= 0 || H <= 0 || D != 128 || H * D > TK_MAX_DIM) return 0;
  const size_t dim = (size_t)H * D;
  return kt_words(B, dim) + (kt_one_launch(B, H) ? 0 : 4 * kt_align(B * dim * 2) + 2 * kt_align((size_t)B * 128 * 2));   // q, k, v, o; f0, g0
}

template <int NB>
static int launch_kda_token(KdaTokenParams& p, int sms, cudaStream_t st) {
  static bool attr[daisy_host::MAX_DEVICES] = {};
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(kda_token_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, TK_SMEM_LIMIT) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    attr[dev] = true;
  }
  const int tiles = 3 * (p.dim / 16) + 16 + (p.H + 15) / 16, grid = sms < tiles ? sms : tiles;   // every CTA has a tile of phase A
  const int fixed = 2048 + 10 * 512 + p.B * (p.dim + 8) * 2 + tk_psum_bytes(p.dim, (tiles + grid - 1) / grid, NB);
  p.depth = fixed + TK_CW * TK_DEPTH * TK_PIECE <= TK_SMEM_LIMIT ? TK_DEPTH : 1;
  const int smem = fixed + TK_CW * p.depth * TK_PIECE;
  if (smem > TK_SMEM_LIMIT) return DAISY_EUNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(TK_CT); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kda_token_kernel<NB>, p) != cudaSuccess) { (void)cudaGetLastError(); return DAISY_ECUDA; }
  return DAISY_OK;
}

// More rows or pairs than a launch of kda_token_kernel is for: four launches for all of them.
static int kda_batch_step(const daisy_b200_kda_layer* ly, const void* x, int64_t x_sb, void* y, float* state, void* conv_q, void* conv_k, void* conv_v,
                          int B, int H, float eps, unsigned flags, void* workspace, int* status_word, void* stream) {
  const int dim = H * 128;
  if ((int64_t)B * H >= (int64_t)1 << 31) return DAISY_EUNSUPPORTED;
  uint8_t* ws = (uint8_t*)workspace + kt_words(B, dim);
  void *pr[3], *o, *low[2];
  for (void*& c : pr) { c = ws; ws += kt_align((size_t)B * dim * 2); }
  o = ws; ws += kt_align((size_t)B * dim * 2);
  for (void*& c : low) { c = ws; ws += kt_align((size_t)B * 128 * 2); }
  const void *xs[3] = {x, x, x}, *w1[3] = {ly->q_w, ly->k_w, ly->v_w}, *w2[2] = {ly->f0_w, ly->g0_w};
  int rc, order = daisy_host::ORDER_AHEAD;                  // the low-rank products take 8 CTAs, 9 us: beside the others (18 rows of 16 heads 32.1 -> 27.4 us, 64 rows 61.2 -> 57.5)
  if ((rc = daisy_host::gemm_group(xs, x_sb, w2, dim, low, 128, 2, B, 128, dim, &order, status_word, stream)) != DAISY_OK) return rc;
  if (order) order = daisy_host::ORDER_BEHIND;
  if ((rc = daisy_host::gemm_group(xs, x_sb, w1, dim, pr, dim, 3, B, dim, dim, &order, status_word, stream)) != DAISY_OK) return rc;
  KdaBatchParams p;
  p.x = (const __nv_bfloat16*)x; p.x_sb = x_sb; p.f0 = (const __nv_bfloat16*)low[0]; p.g0 = (const __nv_bfloat16*)low[1];
  p.b_w = (const __nv_bfloat16*)ly->b_w; p.f1 = (const __nv_bfloat16*)ly->f1_w; p.g1 = (const __nv_bfloat16*)ly->g1_w;
  p.g1_bias = (const __nv_bfloat16*)ly->g1_bias; p.norm_w = (const __nv_bfloat16*)ly->norm_w;
  void* cs[3] = {conv_q, conv_k, conv_v};
  for (int i = 0; i < 3; ++i) {
    p.pr[i] = (const __nv_bfloat16*)pr[i];
    p.conv_w[i] = (const __nv_bfloat16*)ly->conv_w[i]; p.conv_b[i] = (const __nv_bfloat16*)ly->conv_bias[i]; p.conv_s[i] = (__nv_bfloat16*)cs[i];
  }
  p.o = (__nv_bfloat16*)o; p.a_log = ly->a_log; p.dt_bias = ly->dt_bias; p.state = state;
  p.H = H; p.dim = dim; p.silu = (flags & DAISY_KDA_CONV_SILU) ? 1 : 0; p.eps = eps; p.scale = 1.0f / sqrtf(128.f);
  (void)daisy_host::launch_dependent(kda_batch_kernel, dim3((unsigned)(B * H)), dim3(256), 0, (cudaStream_t)stream, p);
  DAISY_CHECK_LAUNCH();
  return daisy_b200_gemm_nt(o, dim, ly->o_w, dim, y, dim, B, dim, dim, status_word, stream);
}

extern "C" int daisy_b200_kda_token_step(const daisy_b200_kda_layer* ly, const void* x, int64_t x_sb, void* y, float* state,
                                         void* conv_q, void* conv_k, void* conv_v, int B, int H, int D, float eps, unsigned flags,
                                         void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
  if (!ly || !x || !y || !state || !conv_q || !conv_k || !conv_v || !workspace || B <= 0 || H <= 0) return DAISY_EINVAL;
  const size_t need = daisy_b200_kda_token_workspace_bytes(B, H, D);
  if (!need) return DAISY_EUNSUPPORTED;
  if (workspace_bytes < need) return DAISY_EWORKSPACE;
  if (flags & ~DAISY_KDA_CONV_SILU) return DAISY_EINVAL;
  const void* all[] = {ly->q_w, ly->k_w, ly->v_w, ly->f0_w, ly->g0_w, ly->b_w, ly->o_w, ly->f1_w, ly->g1_w, ly->a_log, ly->dt_bias,
                       ly->conv_w[0], ly->conv_w[1], ly->conv_w[2]};
  for (const void* a : all) {
    if (!a) return DAISY_EINVAL;
    if (!daisy_aligned16(a)) return DAISY_EALIGN;
  }
  if (!daisy_aligned16(x) || !daisy_aligned16(y) || !daisy_aligned16(state) || !daisy_aligned16(conv_q) || !daisy_aligned16(conv_k) ||
      !daisy_aligned16(conv_v) || (x_sb & 7) || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return DAISY_EALIGN;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  const int dim = H * D;
  if (!kt_one_launch(B, H)) return kda_batch_step(ly, x, x_sb, y, state, conv_q, conv_k, conv_v, B, H, eps, flags, workspace, status_word, stream);
  KdaTokenParams p;
  const void* w[7] = {ly->q_w, ly->k_w, ly->v_w, ly->f0_w, ly->g0_w, ly->b_w, ly->o_w};
  const int rows[7] = {dim, dim, dim, 128, 128, H, dim};
  int rc;
  for (int i = 0; i < 7; ++i)
    if ((rc = tk_make_weight_map(&p.tw[i], w[i], rows[i], dim)) != DAISY_OK) return rc;
  p.f1 = (const __nv_bfloat16*)ly->f1_w; p.g1 = (const __nv_bfloat16*)ly->g1_w;
  p.g1_bias = (const __nv_bfloat16*)ly->g1_bias; p.norm_w = (const __nv_bfloat16*)ly->norm_w;
  void* cs[3] = {conv_q, conv_k, conv_v};
  for (int i = 0; i < 3; ++i) {
    p.conv_w[i] = (const __nv_bfloat16*)ly->conv_w[i]; p.conv_b[i] = (const __nv_bfloat16*)ly->conv_bias[i]; p.conv_s[i] = (__nv_bfloat16*)cs[i];
  }
  p.a_log = ly->a_log; p.dt_bias = ly->dt_bias; p.state = state;
  p.x = (const __nv_bfloat16*)x; p.x_sb = x_sb; p.y = (__nv_bfloat16*)y;
  p.B = B; p.H = H; p.dim = dim; p.silu = (flags & DAISY_KDA_CONV_SILU) ? 1 : 0;
  p.eps = eps; p.scale = 1.0f / sqrtf((float)D);
  uint8_t* ws = (uint8_t*)workspace;
  p.epoch = (unsigned*)ws; ws += 256;
  p.qkv = (uint2*)ws; ws += kt_align((size_t)B * 3 * dim * 4);
  p.fg = (uint2*)ws; ws += kt_align((size_t)B * 128 * 8);
  p.bl = (uint2*)ws; ws += kt_align((size_t)B * 64);
  p.o = (uint2*)ws;
  p.status = status_word;
  return B <= 8 ? launch_kda_token<1>(p, sms, (cudaStream_t)stream) : launch_kda_token<2>(p, sms, (cudaStream_t)stream);
}
