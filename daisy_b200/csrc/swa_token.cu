// One decoded token through a stack of attention layers in ONE launch: per layer the merged QKV projection, the norm /
// RoPE / value-embedding gate of the new token, the windowed attention over the ring cache, the ring store and the output
// projection (CausalSelfAttention.step called layer after layer by Generator._step, models/daisy/attention.py:181-202,
// inference/generate.py:231-248).
//
// Bound: HBM -- every weight and every cache row in the window is read once (67 MB per layer at dim 2048, window 4096,
// batch 1: 10 us at copy bandwidth).  As three launches per layer the step took 22 us a layer: each kernel is only 5-15 us
// long and pays its own launch, ramp-up and tail.  Here a persistent CTA per SM (cooperative launch) keeps the memory
// pipe busy across those boundaries instead: nothing the step streams depends on what it computes -- the addresses of all
// weight rows and cache rows of all layers are known at the start.  The CTA's stream (weight rows, cache rows, weight rows,
// next layer, ...) is cut into 8 KB pieces; piece n belongs to warp n % 12, which keeps two of its pieces in flight and, as
// soon as it has used one, starts the copy of its next but one into the same place -- whatever phase or layer that belongs
// to.  (One producer thread for all warps needs ~400 cycles for a piece, which caps the stream at 20 bytes a cycle and SM
// however large the copies in flight: 3.8 TB/s.  Twelve warps refill in parallel and need no barrier to hand a slot back.)
//   Phase A  QKV rows [c N / G, (c+1) N / G) of the merged weight                       -> qkv
//   Phase B  an equal share of the flattened (batch, head, 64-row piece) range          -> partial (max, sum, acc) per segment;
//            the CTA with a (batch, head)'s last part merges them with the new token    -> o, ring row
//   Phase C  rows of the output projection                                              -> next layer's x, or y
// Exchanges carry their own flags: every 8-byte word is {4 bytes of data, the launch's and layer's tag}, written with one
// store, and the reader polls the words it needs until the tags match.  That is one trip to L2 and back (~1.2k cycles)
// where a counter barrier followed by the load was three (barrier alone: 2.4k), needs no fence, no atomic and nothing reset
// between launches.  A buffer is rewritten one layer later, which needs the whole next x, hence the reads done of every CTA
// that contributes to it.  With 256 channels 20 of 148 CTAs have no row of the output projection: nobody waits for those, and
// one head's next o could be stored while such a CTA, owner of q, k or v rows of the other head only, still reads the old one.
// So a CTA without rows does not read the vector (tk_gathers); in the last phase, after which nothing is rewritten, all do.
// Both contractions run as m16n8k16 tensor-core products (16 weight rows or cache rows x batch rows or q) -- not for their
// rate (HBM is the bound) but because a piece then costs a quarter of the instructions.  q and the softmax weights stay at
// fp32 precision: each is split into a high and a low 16-bit part that occupy two of the product's empty columns / rows.
// All waits are bounded; a CTA that gives up keeps walking through its barriers (its waits return at once), so nobody is
// left behind, and every warp waits for the copies it has in flight before it leaves.
#include "token_common.cuh"

namespace daisy {

constexpr int TK_MAX_SEG = 4;                         // (batch, head) segments of one CTA's range
constexpr int TK_MAX_LAYERS = 16;
constexpr float TK_NEG = -1.0e30f;

struct TokenLayer {
  CUtensorMap tw, tk, tv;                             // [4 dim, dim] weights; rings
  void *kc, *vc;
  const __nv_bfloat16* ve;
  const float* ve_gate;
  __nv_bfloat16 *k_new, *v_new;
  const float *cos, *sin;                             // [table_rows, 64]
};

struct TokenParams {
  TokenLayer layer[TK_MAX_LAYERS];
  int L, B, H, dim, depth;
  const __nv_bfloat16* x; int64_t x_sb;
  __nv_bfloat16* y;                                   // [B, dim]
  int64_t c_sb, c_sh, c_sr, ve_sb;
  long long t;                                        // position, unless t_dev holds it
  const long long* t_dev;
  long long* t_advance;                               // counter to step once the token is done, or null
  int cap, window, table_rows;
  float qscale, eps;
  unsigned flags;
  // workspace: tagged words (see above)
  unsigned* epoch;                                    // tag of the last layer of the previous launch
  uint2* qkv;                                         // [B, 3 dim / 2]: two bf16 and the tag
  uint2 *o, *xmid;                                    // [TK_COPIES][B, dim / 2]
  uint4* part;                                        // [G * TK_MAX_SEG][65]: 128 accumulators, then (max, sum)
  int* status;
};

struct TokenBars {
  uint64_t full[TK_CW * TK_DEPTH];
  int abort_flag;
  float wm[TK_CW], wl[TK_CW];
  float sm[TK_MAX_SEG], sl[TK_MAX_SEG], s_self[TK_MAX_SEG];
};
constexpr int TK_FIXED = TK_MAX_SEG * (512 + 1024 + 512);   // shared memory of the segments: q halves, k and v, own partial
constexpr int TK_PART = 65;                           // uint4 words of a partial

// Position-dependent geometry of the step, and this CTA's share of the tiles.
struct TokenGeom {
  int start, n1, n2, t1, tpb;                         // context rows: n1 from slot `start`, n2 from slot 0; pieces: t1 + the rest = tpb
  int new_slot;
  int tot, parts;                                     // all pieces; CTAs that share them
  int lo, hi;                                         // this CTA's pieces
  long long pos;
};
// First row of a CTA's share of a projection, in pairs of rows; whether a CTA of `rows` rows reads the vector it multiplies.
__host__ __device__ __forceinline__ int tk_row(int cta, int ctas, int rows) { return 2 * (cta * (rows / 2) / ctas); }
__host__ __device__ __forceinline__ bool tk_gathers(int rows, bool last) { return rows > 0 || last; }
// every CTA has rows of q, k or v, so that whoever has seen all of them knows every CTA's reads of x, position and tag done
static_assert(daisy_host::MAX_SMS <= 3 * DAISY_HEAD_DIM / 2, "row pairs of the smallest QKV projection");
// (the launcher keeps pieces x CTAs below 2^31)
__device__ __forceinline__ int tk_lo(int c, int tot, int parts) { return (int)tk_div((unsigned)c * (unsigned)tot, (unsigned)parts); }
__device__ __forceinline__ int tk_owner(int tile, int tot, int parts) { return (int)tk_div(((unsigned)tile + 1u) * (unsigned)parts - 1u, (unsigned)tot); }
__device__ __forceinline__ TokenGeom tk_geom(const TokenParams& p) {
  TokenGeom g;
  const long long t = p.t_dev ? *p.t_dev : p.t;
  long long r = t < p.cap ? t : p.cap;
  if (p.window > 0 && r > (long long)p.window - 1) r = p.window - 1;
  g.start = p.cap > 0 ? (int)((t - r) % p.cap) : 0;
  g.new_slot = p.cap > 0 ? (int)(t % p.cap) : 0;
  g.n1 = min((int)r, p.cap - g.start); g.n2 = (int)r - g.n1;
  g.t1 = (g.n1 + 15) / 16;
  g.tpb = g.t1 + (g.n2 + 15) / 16;
  g.tot = p.B * p.H * g.tpb;
  g.parts = min((int)gridDim.x, g.tot);
  const int c = (int)blockIdx.x;
  g.lo = c < g.parts ? tk_lo(c, g.tot, g.parts) : 0;
  g.hi = c < g.parts ? tk_lo(c + 1, g.tot, g.parts) : 0;
  g.pos = t;
  if (g.pos >= p.table_rows) {                        // past the RoPE table: report, stay in bounds
    g.pos = p.table_rows - 1;
    if (p.status && threadIdx.x == 0 && blockIdx.x == 0) p.status[0] = DAISY_EINVAL;
  }
  return g;
}

// This warp's pieces of the CTA's stream: weight rows, cache rows, weight rows of each layer.
struct TokenStream : TokenRing {
  const TokenParams& p;
  const TokenGeom& g;
  int na, nb, nc, ks_n, a0, c0;                       // pieces of the phases of a layer; pieces of a row tile; first rows
  int l, i;                                           // next to load: layer, piece of the layer

  __device__ TokenStream(const TokenParams& p_, const TokenGeom& g_) : p(p_), g(g_) {}
  __device__ __forceinline__ void load(int at) {
    if (l >= p.L) return;
    const TokenLayer& ly = p.layer[l];
    const uint32_t dst = buf + at * TK_PIECE;
    mbar_expect_tx(&full[at], TK_PIECE);
    if (i >= na && i < na + nb) {
      const int x = g.lo + i - na, bh = x / g.tpb, b = bh / p.H, h = bh - b * p.H, j = x - bh * g.tpb;
      const int row = j < g.t1 ? g.start + 16 * j : 16 * (j - g.t1);
      tk_tma5(dst, &ly.tk, &full[at], row, h, b);
      tk_tma5(dst + 2 * TK_BLK, &ly.tv, &full[at], row, h, b);
    } else {                                          // (a last row tile brings rows of the next CTA: not used)
      const int k = i < na ? i : i - na - nb, tile = k / ks_n, kb = k - tile * ks_n;
      tk_tma3(dst, &ly.tw, &full[at], 0, (i < na ? a0 : 3 * p.dim + c0) + 16 * tile, kb * (TK_KW / 64));
    }
    step();
  }
  __device__ __forceinline__ void step() {
    i += TK_CW;
    while (i >= na + nb + nc) { i -= na + nb + nc; ++l; }
  }
};

// One warp: the raw q / k / v row (lane = 4 consecutive elements) -> normalised, rotated.
__device__ __forceinline__ void tk_norm_rope(float (&x)[4], bool norm, bool rope, float eps, const float4 c, const float4 s, int lane) {
  if (norm) {
    const float r = rsqrtf(tk_warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]) * (1.0f / DAISY_HEAD_DIM) + eps);
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] *= r;
  }
  if (rope) {
    const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x, s.y, s.z, s.w};
    const float sgn = lane < 16 ? 1.f : -1.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, x[e], 16);
      x[e] = x[e] * cc[e] + sgn * other * ss[e];
    }
  }
}
__device__ __forceinline__ void tk_unpack(const uint4& u, float (&x)[4]) {
  x[0] = bf16_lo(u.x); x[1] = bf16_hi(u.x); x[2] = bf16_lo(u.z); x[3] = bf16_hi(u.z);
}

// One warp prepares a segment: q, scaled, as high and low halves; the new row's k and v as the cache will hold them, its
// score, and -- where this CTA merges the segment -- the ring row and the copies the caller asked for.  (The ring slot may
// still be attended to when the window exceeds the ring: the row is stored by tk_finish.)
template <bool F16>
__device__ __forceinline__ void tk_prepare(const TokenParams& p, const TokenGeom& g, const TokenLayer& ly, TokenBars* bars, uint16_t* qs,
                                           float* kv, int bh, int sg, bool merger, uint32_t tag, int lane) {
  const int b = bh / p.H, h = bh - b * p.H;
  const float4 cs = __ldg(reinterpret_cast<const float4*>(ly.cos + g.pos * 64) + (lane & 15));
  const float4 sn = __ldg(reinterpret_cast<const float4*>(ly.sin + g.pos * 64) + (lane & 15));
  float q[4], k[4], v[4];
  {
    uint4 r[3];
    tk_get(reinterpret_cast<const uint4*>(p.qkv + (size_t)b * 3 * (p.dim / 2) + h * 64) + lane, p.dim / 4, r, tag, &bars->abort_flag, p.status);
    tk_unpack(r[0], q); tk_unpack(r[1], k); tk_unpack(r[2], v);
  }
  tk_norm_rope(q, p.flags & DAISY_NORM_Q, p.flags & DAISY_ROPE, p.eps, cs, sn, lane);
  uint16_t hi[4], lo[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) tk_split<F16>(q[e] * p.qscale, hi[e], lo[e]);
  *reinterpret_cast<uint2*>(qs + sg * 256 + 4 * lane) = make_uint2(hi[0] | (uint32_t)hi[1] << 16, hi[2] | (uint32_t)hi[3] << 16);
  *reinterpret_cast<uint2*>(qs + sg * 256 + 128 + 4 * lane) = make_uint2(lo[0] | (uint32_t)lo[1] << 16, lo[2] | (uint32_t)lo[3] << 16);
  if (!merger) return;
  tk_norm_rope(k, p.flags & DAISY_NORM_K, p.flags & DAISY_ROPE, p.eps, cs, sn, lane);
  tk_norm_rope(v, p.flags & DAISY_NORM_V, false, p.eps, cs, sn, lane);
  if (ly.ve) {
    const float gate = 1.0f / (1.0f + __expf(-*ly.ve_gate));
    const uint2 u = *reinterpret_cast<const uint2*>(ly.ve + b * p.ve_sb + h * 128 + 4 * lane);
    const float e4[4] = {bf16_lo(u.x), bf16_hi(u.x), bf16_lo(u.y), bf16_hi(u.y)};
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = gate * v[e] + (1.0f - gate) * e4[e];
  }
  if (ly.k_new) *reinterpret_cast<uint2*>(ly.k_new + (size_t)bh * 128 + 4 * lane) = make_uint2(pack_bf16(k[0], k[1]), pack_bf16(k[2], k[3]));
  if (ly.v_new) *reinterpret_cast<uint2*>(ly.v_new + (size_t)bh * 128 + 4 * lane) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
#pragma unroll
  for (int e = 0; e < 4; ++e) {                                                 // at the precision of the cache
    k[e] = F16 ? __half2float(__float2half_rn(k[e])) : __bfloat162float(__float2bfloat16_rn(k[e]));
    v[e] = F16 ? __half2float(__float2half_rn(v[e])) : __bfloat162float(__float2bfloat16_rn(v[e]));
  }
  const float s_self = tk_warp_sum((q[0] * k[0] + q[1] * k[1] + q[2] * k[2] + q[3] * k[3]) * p.qscale);
  reinterpret_cast<float4*>(kv + sg * 256)[lane] = make_float4(k[0], k[1], k[2], k[3]);
  reinterpret_cast<float4*>(kv + sg * 256 + 128)[lane] = make_float4(v[0], v[1], v[2], v[3]);
  if (lane == 0) bars->s_self[sg] = s_self;
}

// One warp: the segment's own partial (sg) and, if `others`, what the warps gathered from the other parts, merged with the
// new row -> attention output, ring row.
template <bool F16>
__device__ __forceinline__ void tk_finish(const TokenParams& p, const TokenGeom& g, const TokenLayer& ly, const TokenBars* bars, const float* kv,
                                          const float* own, const float* wacc, bool any, bool others, int bh, int sg, uint32_t tag, int lane) {
  __syncwarp();
  const int b = bh / p.H, h = bh - b * p.H;
  const float4 k = reinterpret_cast<const float4*>(kv + sg * 256)[lane], v = reinterpret_cast<const float4*>(kv + sg * 256 + 128)[lane];
  const float s_self = bars->s_self[sg];
  float M = any ? fmaxf(s_self, bars->sm[sg]) : s_self;
  if (others) {
#pragma unroll
    for (int w = 0; w < TK_CW; ++w) M = fmaxf(M, bars->wm[w]);
  }
  const float w0 = fast_exp2(s_self - M);
  float den = w0, num[4] = {w0 * v.x, w0 * v.y, w0 * v.z, w0 * v.w};
  auto add = [&](float f, float l, const float4 a) {
    den = fmaf(f, l, den);
    num[0] = fmaf(f, a.x, num[0]); num[1] = fmaf(f, a.y, num[1]); num[2] = fmaf(f, a.z, num[2]); num[3] = fmaf(f, a.w, num[3]);
  };
  if (any) add(fast_exp2(bars->sm[sg] - M), bars->sl[sg], reinterpret_cast<const float4*>(own + sg * 128)[lane]);
  if (others) {
#pragma unroll
    for (int w = 0; w < TK_CW; ++w) add(fast_exp2(bars->wm[w] - M), bars->wl[w], reinterpret_cast<const float4*>(wacc + w * 128)[lane]);
  }
  const float inv = 1.0f / den;
  const uint32_t o01 = pack_bf16(num[0] * inv, num[1] * inv), o23 = pack_bf16(num[2] * inv, num[3] * inv);
#pragma unroll
  for (int c = 0; c < TK_COPIES; ++c) tk_put4(reinterpret_cast<uint4*>(p.o + (size_t)(c * p.B + b) * (p.dim / 2) + h * 64) + lane, o01, o23, tag);
  if (p.flags & DAISY_WRITE_RING) {
    const int64_t at = b * p.c_sb + h * p.c_sh + (int64_t)g.new_slot * p.c_sr + 4 * lane;
    uint2 kr, vr;
    if (F16) {
      const __half2 k0 = __floats2half2_rn(k.x, k.y), k1 = __floats2half2_rn(k.z, k.w), v0 = __floats2half2_rn(v.x, v.y), v1 = __floats2half2_rn(v.z, v.w);
      kr = make_uint2(*reinterpret_cast<const uint32_t*>(&k0), *reinterpret_cast<const uint32_t*>(&k1));
      vr = make_uint2(*reinterpret_cast<const uint32_t*>(&v0), *reinterpret_cast<const uint32_t*>(&v1));
    } else {
      kr = make_uint2(pack_bf16(k.x, k.y), pack_bf16(k.z, k.w));
      vr = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
    }
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(ly.kc) + at) = kr;
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(ly.vc) + at) = vr;
  }
}

template <bool F16, int NB>
__global__ void __launch_bounds__(TK_CT, 1) swa_token_kernel(const __grid_constant__ TokenParams p) {
  extern __shared__ __align__(128) uint8_t tk_smem[];
  TokenBars* bars = reinterpret_cast<TokenBars*>(tk_smem);
  const uint32_t ring = (smem_u32(tk_smem) + sizeof(TokenBars) + 1023) & ~1023u;       // swizzled blocks: 1 KB boundaries
  static_assert(sizeof(TokenBars) <= 1024, "barrier block");
  uint8_t* after = tk_smem + (ring - smem_u32(tk_smem)) + TK_CW * p.depth * TK_PIECE;
  uint16_t* qs = reinterpret_cast<uint16_t*>(after);                            // [TK_MAX_SEG][2][128]: high and low half of q
  float* kv = reinterpret_cast<float*>(after + TK_MAX_SEG * 512);               // [TK_MAX_SEG][2][128]: the new row's k, v
  float* own = kv + TK_MAX_SEG * 256;                                           // [TK_MAX_SEG][128]: partials of the segments merged here
  uint8_t* xs = after + TK_FIXED;
  const int xs_ld = (p.dim + 8) * 2;
  float* psum = reinterpret_cast<float*>(xs + p.B * xs_ld);                     // also the warps' attention accumulators
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;

  if (threadIdx.x == 0) {
    for (int i = 0; i < TK_CW * TK_DEPTH; ++i) mbar_init(&bars->full[i], 1);
    bars->abort_flag = 0;
    mbar_init_fence();
  }
  const TokenGeom g = tk_geom(p);
  const uint32_t tag0 = *p.epoch + 1;                                           // stepped by the last act of CTA 0
  // rows of the projections, in pairs
  const int a0 = tk_row(cta, G, 3 * p.dim), a1 = tk_row(cta + 1, G, 3 * p.dim);
  const int c0 = tk_row(cta, G, p.dim), c1 = tk_row(cta + 1, G, p.dim);
  __syncthreads();

  const int ks_n = (p.dim + TK_KW - 1) / TK_KW, na = (a1 - a0 + 15) / 16 * ks_n, nb = g.hi - g.lo, nc = (c1 - c0 + 15) / 16 * ks_n;
  TokenStream in(p, g);
  in.full = bars->full + warp * TK_DEPTH; in.buf = ring + warp * (p.depth * TK_PIECE);
  in.depth = p.depth; in.st = in.par = 0; in.skip = warp; in.abort_flag = abort_flag; in.status = p.status;
  in.na = na; in.nb = nb; in.nc = nc; in.ks_n = ks_n; in.a0 = a0; in.c0 = c0; in.l = 0; in.i = warp - TK_CW;
  in.step();                                                                    // the warp's first piece
  if (lane == 0)
    for (int i = 0; i < p.depth; ++i) in.load(i);
  const bool any = g.tot > 0;                                                   // is there a context at all
  const int bh_lo = any ? (g.hi > g.lo ? g.lo / g.tpb : 0) : cta;
  const int nseg = any ? (g.hi > g.lo ? (g.hi - 1) / g.tpb - bh_lo + 1 : 0) : (p.B * p.H - 1 - cta) / G + (cta < p.B * p.H ? 1 : 0);
  const int seg_step = any ? 1 : G;
  // this CTA merges the segments whose last tile it has: all but perhaps its last one; only the first of them can have
  // parts elsewhere, `others` of them, from CTA part0 on
  const int merged = any ? (nseg > 0 && g.hi == (bh_lo + nseg) * g.tpb ? nseg : nseg - 1) : nseg;
  int part0 = 0, others = 0;
  if (any && merged > 0 && g.lo > bh_lo * g.tpb) { part0 = tk_owner(bh_lo * g.tpb, g.tot, g.parts); others = cta - part0; }
  uint32_t swz[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = (lane & 7) + 8 * ((lane >> 3) & 1);
    swz[j] = row * 128 + (((2 * j + (lane >> 4)) ^ (row & 7)) << 4);
  }
#pragma unroll 1
  for (int ph = 0; ph < 2 * p.L; ++ph) {
    const int l = ph >> 1;
    const bool is_c = ph & 1;
    const TokenLayer& ly = p.layer[l];
    const uint32_t tag = tag0 + l;
    // ---- phases A and C: the vector, then the projection
    const bool gathers = tk_gathers(is_c ? c1 - c0 : a1 - a0, ph == 2 * p.L - 1);
#pragma unroll 1
    for (int b = 0; gathers && b < p.B; ++b) {
      if (ph == 0) {
        for (int k = threadIdx.x; k < p.dim / 8; k += TK_CT) *reinterpret_cast<uint4*>(xs + b * xs_ld + k * 16) = ld_cg16(p.x + b * p.x_sb + k * 8);
      } else {
        tk_gather(xs + b * xs_ld, (is_c ? p.o : p.xmid) + (size_t)(cta % TK_COPIES * p.B + b) * (p.dim / 2), p.dim / 4, is_c ? tag : tag - 1, abort_flag, p.status);
      }
    }
    const int n0 = is_c ? c0 : a0, out_ld = (is_c ? 1 : 3) * (p.dim / 2);
    __nv_bfloat16* plain = ph == 2 * p.L - 1 ? p.y : nullptr;
    tk_project<NB>(in, psum, smem_u32(xs), xs_ld, p.B, p.dim, is_c ? nc : na, (is_c ? c1 - c0 : a1 - a0) >> 1, swz, lane,
                   [&](bool, int b, int row, float s0, float s1) {
      const uint32_t v = pack_bf16(s0, s1);
      if (plain) *reinterpret_cast<uint32_t*>(plain + (size_t)b * p.dim + n0 + row) = v;
      else if (!is_c) tk_put2(p.qkv + (size_t)b * out_ld + ((n0 + row) >> 1), v, tag);
      else
        for (int c = 0; c < TK_COPIES; ++c) tk_put2(p.xmid + (size_t)(c * p.B + b) * out_ld + ((n0 + row) >> 1), v, tag);
    });
    if (is_c) continue;
    // ---- phase B
#pragma unroll 1
    for (int sg = warp; sg < nseg; sg += TK_CW)
      tk_prepare<F16>(p, g, ly, bars, qs, kv, bh_lo + sg * seg_step, sg, sg < merged, tag, lane);
    int piece = g.lo + in.phase(nb);
#pragma unroll 1
    for (int sg = 0; any && sg < nseg; ++sg) {
      const int bh = bh_lo + sg, p_end = min(g.hi, (bh + 1) * g.tpb);
      // B operand of the scores: column 0 the high, column 1 the low half of q
      const uint32_t* qrow = reinterpret_cast<const uint32_t*>(qs + sg * 256 + (g8 & 1) * 128 + 2 * t4);
      float m = TK_NEG, lsum = 0.f, acc[16][4];
#pragma unroll
      for (int j = 0; j < 16; ++j) { acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f; }
      if (sg == 0) named_bar(1, TK_CT);                                         // q is in shared memory
#pragma unroll 1
      for (; piece < p_end; piece += TK_CW) {
        const uint32_t blk = in.wait();
        {
          const int j0 = piece - bh * g.tpb, valid = j0 < g.t1 ? g.n1 - 16 * j0 : g.n2 - 16 * (j0 - g.t1);
          float sc[4][4];
#pragma unroll
          for (int j = 0; j < 16; ++j) sc[j >> 2][j & 3] = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint32_t a[4];
            tk_ldm4(a, blk + (j >> 2) * TK_BLK + swz[j & 3]);
            const uint32_t b0 = qrow[j * 8], b1 = qrow[j * 8 + 4];
            tk_mma<F16>(sc[j & 3], a, g8 < 2 ? b0 : 0u, g8 < 2 ? b1 : 0u);
          }
          // high + low column: lane t4 = 0 of each quad has rows g8 and g8 + 8
          float s0 = ((sc[0][0] + sc[1][0]) + (sc[2][0] + sc[3][0])) + ((sc[0][1] + sc[1][1]) + (sc[2][1] + sc[3][1]));
          float s1 = ((sc[0][2] + sc[1][2]) + (sc[2][2] + sc[3][2])) + ((sc[0][3] + sc[1][3]) + (sc[2][3] + sc[3][3]));
          s0 = __shfl_sync(0xffffffffu, s0, lane & 28); s1 = __shfl_sync(0xffffffffu, s1, lane & 28);
          if (g8 >= valid) s0 = -INFINITY;
          if (g8 + 8 >= valid) s1 = -INFINITY;
          float mt = fmaxf(s0, s1);
          mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 4));
          mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 8));
          mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 16));
          if (mt > m) {
            const float alpha = fast_exp2(m - mt);
            lsum *= alpha;
#pragma unroll
            for (int j = 0; j < 16; ++j) { acc[j][0] *= alpha; acc[j][1] *= alpha; acc[j][2] *= alpha; acc[j][3] *= alpha; }
            m = mt;
          }
          const float p0 = fast_exp2(s0 - m), p1 = fast_exp2(s1 - m);
          lsum += p0 + p1;
          // A operand: row 0 the high, row 8 the low half of the 16 weights
          const float w0 = __shfl_sync(0xffffffffu, p0, 8 * t4), w1 = __shfl_sync(0xffffffffu, p0, 8 * t4 + 4);
          const float w2 = __shfl_sync(0xffffffffu, p1, 8 * t4), w3 = __shfl_sync(0xffffffffu, p1, 8 * t4 + 4);
          uint16_t h0, h1, h2, h3, l0, l1, l2, l3;
          tk_split<F16>(w0, h0, l0); tk_split<F16>(w1, h1, l1); tk_split<F16>(w2, h2, l2); tk_split<F16>(w3, h3, l3);
          uint32_t a[4] = {h0 | (uint32_t)h1 << 16, l0 | (uint32_t)l1 << 16, h2 | (uint32_t)h3 << 16, l2 | (uint32_t)l3 << 16};
#pragma unroll
          for (int j = 0; j < 4; ++j) a[j] = g8 == 0 ? a[j] : 0u;
          // V rows past the context hold whatever an earlier sequence left in the ring: their weights are zero, but zero times
          // an infinity is not.  The lanes that address such rows read the last row of the context instead.
          const int vr = min((lane & 7) + 8 * ((lane >> 3) & 1), valid - 1);
          const uint32_t vrow = blk + 2 * TK_BLK + vr * 128 + (((lane >> 4) ^ (vr & 7)) << 4);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint32_t bv[4];
            tk_ldm4_t(bv, (vrow ^ ((j & 3) << 5)) + (j >> 2) * TK_BLK);
            tk_mma<F16>(acc[2 * j], a, bv[0], bv[1]);
            tk_mma<F16>(acc[2 * j + 1], a, bv[2], bv[3]);
          }
        }
        in.done(in, lane);
      }
      // the warps' shares of the segment
      lsum += __shfl_xor_sync(0xffffffffu, lsum, 4);
      lsum += __shfl_xor_sync(0xffffffffu, lsum, 8);
      lsum += __shfl_xor_sync(0xffffffffu, lsum, 16);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (g8 == 0) *reinterpret_cast<float2*>(psum + warp * 128 + j * 8 + 2 * t4) = make_float2(acc[j][0] + acc[j][2], acc[j][1] + acc[j][3]);
      if (lane == 0) { bars->wm[warp] = m; bars->wl[warp] = lsum; }
      named_bar(1, TK_CT);
      if (threadIdx.x < 128) {
        float f[TK_CW], M = TK_NEG, a = 0.f, L = 0.f;
#pragma unroll
        for (int w = 0; w < TK_CW; ++w) { f[w] = bars->wm[w]; M = fmaxf(M, f[w]); }
#pragma unroll
        for (int w = 0; w < TK_CW; ++w) {
          f[w] = fast_exp2(f[w] - M);
          a = fmaf(f[w], psum[w * 128 + threadIdx.x], a);
          L = fmaf(f[w], bars->wl[w], L);
        }
        if (sg < merged) {
          own[sg * 128 + threadIdx.x] = a;
          if (threadIdx.x == 0) { bars->sm[sg] = M; bars->sl[sg] = L; }
        } else {
          uint4* dst = p.part + (size_t)(cta * TK_MAX_SEG + sg) * TK_PART;
          tk_put2(reinterpret_cast<uint2*>(dst) + threadIdx.x, __float_as_uint(a), tag);
          if (threadIdx.x == 0) tk_put4(dst + 64, __float_as_uint(M), __float_as_uint(L), tag);
        }
      }
      named_bar(1, TK_CT);
    }
    if (others) {                                                               // the first segment's other parts, spread over the warps
      float m = TK_NEG, lsum = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int i = warp; i < others; i += TK_CW) {
        const int c = part0 + i, seg = bh_lo - tk_lo(c, g.tot, g.parts) / g.tpb;
        const uint4* src = p.part + (size_t)(c * TK_MAX_SEG + seg) * TK_PART;
        uint4 r[2], ml[1];
        tk_get(src + 2 * lane, 1, r, tag, abort_flag, p.status);
        tk_get(src + 64, 0, ml, tag, abort_flag, p.status);
        const float mi = __uint_as_float(ml[0].x), mn = fmaxf(m, mi), fa = fast_exp2(m - mn), fb = fast_exp2(mi - mn);
        a[0] = a[0] * fa + fb * __uint_as_float(r[0].x); a[1] = a[1] * fa + fb * __uint_as_float(r[0].z);
        a[2] = a[2] * fa + fb * __uint_as_float(r[1].x); a[3] = a[3] * fa + fb * __uint_as_float(r[1].z);
        lsum = lsum * fa + fb * __uint_as_float(ml[0].z);
        m = mn;
      }
      reinterpret_cast<float4*>(psum + warp * 128)[lane] = make_float4(a[0], a[1], a[2], a[3]);
      if (lane == 0) { bars->wm[warp] = m; bars->wl[warp] = lsum; }
      named_bar(1, TK_CT);
    }
#pragma unroll 1
    for (int sg = warp; sg < merged; sg += TK_CW)
      tk_finish<F16>(p, g, ly, bars, kv, own, psum, any, others > 0 && sg == 0, bh_lo + sg * seg_step, sg, tag, lane);
  }
  in.drain();
  // CTA 0 has read the last o: every CTA has contributed, hence read the position and the tag
  if (threadIdx.x == 0 && cta == 0) {
    *p.epoch = tag0 + p.L - 1;
    if (p.t_advance) *p.t_advance += 1;
  }
}

}  // namespace daisy

using namespace daisy;

static inline size_t tk_align(size_t n) { return (n + 255) / 256 * 256; }

extern "C" size_t daisy_b200_swa_token_workspace_bytes(int B, int H, int D) {
  if (B <= 0 || H <= 0 || D != DAISY_HEAD_DIM || B > TK_MAX_B || H * D > TK_MAX_DIM) return 0;
  const size_t dim = (size_t)H * D;
  const size_t parts = (size_t)daisy_host::MAX_SMS * TK_MAX_SEG;
  return 256 + tk_align(B * 3 * dim * 4) + 2 * TK_COPIES * tk_align(B * dim * 4) + parts * TK_PART * 16;
}

extern "C" int daisy_b200_swa_token_rows(int cta, int ctas, int dim, int phase, int* first, int* end) {
  if (ctas <= 0 || cta < 0 || cta >= ctas || dim <= 0 || dim % DAISY_HEAD_DIM || dim > TK_MAX_DIM || phase < 0 || phase > 2 || !first || !end) return DAISY_EINVAL;
  const int rows = phase ? dim : 3 * dim;
  *first = tk_row(cta, ctas, rows); *end = tk_row(cta + 1, ctas, rows);
  return tk_gathers(*end - *first, phase == 2) ? 1 : 0;
}

template <bool F16, int NB>
static int launch_token(TokenParams& p, int sms, cudaStream_t st) {
  static bool attr[daisy_host::MAX_DEVICES] = {};
  const int dev = daisy_host::device_slot();
  if (dev < 0) return DAISY_ENODEV;
  constexpr int limit = TK_SMEM_LIMIT;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(swa_token_kernel<F16, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) {
      (void)cudaGetLastError();
      return DAISY_ECUDA;
    }
    attr[dev] = true;
  }
  int psum = tk_psum_bytes(p.dim, ((3 * p.dim / 2 + sms - 1) / sms * 2 + 15) / 16, NB);
  if (psum < TK_CW * 512) psum = TK_CW * 512;                             // also the warps' attention accumulators
  const int fixed = 2048 + TK_FIXED + p.B * (p.dim + 8) * 2 + psum;
  p.depth = fixed + TK_CW * TK_DEPTH * TK_PIECE <= limit ? TK_DEPTH : 1;
  const int smem = fixed + TK_CW * p.depth * TK_PIECE;
  if (smem > limit) return DAISY_EUNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms); cfg.blockDim = dim3(TK_CT); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, swa_token_kernel<F16, NB>, p) != cudaSuccess) { (void)cudaGetLastError(); return DAISY_ECUDA; }
  return DAISY_OK;
}

extern "C" int daisy_b200_swa_token_step(const daisy_b200_token_layer* layers, int n_layers, const void* x, int64_t x_sb, void* y,
                                         int64_t c_sb, int64_t c_sh, int64_t c_sr, int64_t t, const int64_t* t_dev, int64_t* t_advance,
                                         int cap, int window, int table_rows, int64_t ve_sb,
                                         int B, int H, int D, float scale, float eps, unsigned flags,
                                         void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
  if (!layers || n_layers <= 0 || !x || !y || !workspace || B <= 0 || H <= 0 || t < 0 || cap < 0 || table_rows <= 0) return DAISY_EINVAL;
  if (D != DAISY_HEAD_DIM || n_layers > TK_MAX_LAYERS) return DAISY_EUNSUPPORTED;
  const size_t need = daisy_b200_swa_token_workspace_bytes(B, H, D);
  if (!need) return DAISY_EUNSUPPORTED;
  if (workspace_bytes < need) return DAISY_EWORKSPACE;
  if (flags & ~(DAISY_QKV_DEFAULT | DAISY_WRITE_RING | DAISY_CACHE_FP16)) return DAISY_EINVAL;
  if ((flags & DAISY_WRITE_RING) && cap == 0) return DAISY_EINVAL;
  if (!t_dev && t >= table_rows) return DAISY_EINVAL;
  if ((reinterpret_cast<uintptr_t>(t_dev) & 7) || (reinterpret_cast<uintptr_t>(t_advance) & 7)) return DAISY_EINVAL;
  const bool need_cache = (flags & DAISY_WRITE_RING) || (cap > 0 && window != 1 && (t_dev || t > 0));
  if (!daisy_aligned16(x) || !daisy_aligned16(y) || (reinterpret_cast<uintptr_t>(workspace) & 255) || (x_sb & 7) ||
      (need_cache && ((c_sb | c_sh | c_sr) & 7)))
    return DAISY_EALIGN;
  // a zero stride on a dimension longer than 1 is a broadcast (expanded) view, which the tile loads cannot express
  if (need_cache && (c_sb < 0 || c_sh < 0 || c_sr < 0 || (B > 1 && c_sb == 0) || (H > 1 && c_sh == 0) || (cap > 1 && c_sr == 0))) return DAISY_EINVAL;
  const int sms = daisy_host::sm_count_cached();
  if (sms <= 0) return DAISY_ENODEV;
  // segments of a CTA's range: at most BH / G + 2 of them (see TK_MAX_SEG)
  if ((int64_t)B * H * ((int64_t)cap / 16 + 2) * sms >= ((int64_t)1 << 31)) return DAISY_EUNSUPPORTED;
  if (sms > daisy_host::MAX_SMS || (int64_t)B * H > (int64_t)sms * (TK_MAX_SEG - 2)) return DAISY_EUNSUPPORTED;
  // a dimension of length 1 may come with any stride; the encoder wants a non-zero multiple of 16 bytes
  auto stride = [](int64_t s, int n) { return (cuuint64_t)(n == 1 ? 16 : s * 2); };
  static_assert(sizeof(TokenParams) <= 32764, "kernel parameters");
  TokenParams p;
  const int dim = H * D;
  for (int l = 0; l < n_layers; ++l) {
    const daisy_b200_token_layer& s = layers[l];
    if (!s.qkvo_w || !s.cos || !s.sin || (need_cache && (!s.kcache || !s.vcache)) || (s.ve && !s.ve_gate_logit)) return DAISY_EINVAL;
    if (!daisy_aligned16(s.qkvo_w) || (need_cache && (!daisy_aligned16(s.kcache) || !daisy_aligned16(s.vcache))) || !daisy_aligned16(s.ve) ||
        !daisy_aligned16(s.k_new_out) || !daisy_aligned16(s.v_new_out) || !daisy_aligned16(s.cos) || !daisy_aligned16(s.sin) || (s.ve && (ve_sb & 7)))
      return DAISY_EALIGN;
    TokenLayer& ly = p.layer[l];
    int rc;
    if ((rc = tk_make_weight_map(&ly.tw, s.qkvo_w, 4 * dim, dim)) != DAISY_OK) return rc;
    if (need_cache) {                                 // a ring as (64 elements, slots, halves of a row, h, b)
      const cuuint64_t dims[5] = {64, (cuuint64_t)cap, 2, (cuuint64_t)H, (cuuint64_t)B};
      const cuuint64_t st[4] = {stride(c_sr, cap), 128, stride(c_sh, H), stride(c_sb, B)};
      const cuuint32_t box[5] = {64, 16, 2, 1, 1};
      if ((rc = tk_make_map(&ly.tk, s.kcache, 5, dims, st, box)) != DAISY_OK) return rc;
      if ((rc = tk_make_map(&ly.tv, s.vcache, 5, dims, st, box)) != DAISY_OK) return rc;
    }
    ly.kc = s.kcache; ly.vc = s.vcache; ly.ve = (const __nv_bfloat16*)s.ve; ly.ve_gate = s.ve_gate_logit;
    ly.k_new = (__nv_bfloat16*)s.k_new_out; ly.v_new = (__nv_bfloat16*)s.v_new_out; ly.cos = s.cos; ly.sin = s.sin;
  }
  p.L = n_layers; p.B = B; p.H = H; p.dim = dim;
  p.x = (const __nv_bfloat16*)x; p.x_sb = x_sb; p.y = (__nv_bfloat16*)y;
  p.c_sb = c_sb; p.c_sh = c_sh; p.c_sr = c_sr; p.ve_sb = ve_sb;
  p.t = t; p.t_dev = (const long long*)t_dev; p.t_advance = (long long*)t_advance; p.cap = cap; p.window = window; p.table_rows = table_rows;
  p.qscale = scale * 1.4426950408889634f; p.eps = eps; p.flags = flags;
  uint8_t* ws = (uint8_t*)workspace;
  p.epoch = (unsigned*)ws; ws += 256;
  p.qkv = (uint2*)ws; ws += tk_align((size_t)B * 3 * dim * 4);
  p.o = (uint2*)ws; ws += TK_COPIES * tk_align((size_t)B * dim * 4);
  p.xmid = (uint2*)ws; ws += TK_COPIES * tk_align((size_t)B * dim * 4);
  p.part = (uint4*)ws;
  p.status = status_word;
  const bool f16 = (flags & DAISY_CACHE_FP16) != 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (B <= 8) return f16 ? launch_token<true, 1>(p, sms, st) : launch_token<false, 1>(p, sms, st);
  return f16 ? launch_token<true, 2>(p, sms, st) : launch_token<false, 2>(p, sms, st);
}
