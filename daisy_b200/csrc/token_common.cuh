// What the single-launch decode kernels (swa_token.cu, kda_token.cu) share: the warps' private rings of streamed pieces, the
// projection of the batch's vectors, and the exchange of vectors between CTAs as tagged words.
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>

namespace daisy {

constexpr int TK_CW = 12;                             // warps
constexpr int TK_CT = 32 * TK_CW;
constexpr int TK_DEPTH = 2;                           // pieces of a warp in flight (one where the vectors of a large batch take the room)
constexpr int TK_KW = 256;                            // weight columns of a piece
// A piece is 16 weight rows x 256 columns, or 16 K rows + 16 V rows: blocks of 16 rows x 128 bytes, 128-byte swizzle
constexpr int TK_PIECE = 8192, TK_BLK = 2048;
constexpr int TK_COPIES = 4;                          // of a vector that all CTAs read: 148 of them at the same 8 KB queue at its L2 slices
constexpr int TK_MAX_DIM = 2048, TK_MAX_B = 16;
constexpr int TK_SMEM_LIMIT = 232448;

static __device__ __noinline__ unsigned tk_div(unsigned a, unsigned b) { return a / b; }
template <bool F16>
__device__ __forceinline__ void tk_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if (F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void tk_ldm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tk_ldm4_t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tk_tma3(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tk_tma5(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int row, int h, int b) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5, %6}], [%2];"
               ::"r"(dst), "l"(m), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(h), "r"(b) : "memory");
}
__device__ __forceinline__ float tk_warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// high and low 16-bit halves of a value: h + l carries 16 (bf16) to 21 (fp16) bits of it
template <bool F16>
__device__ __forceinline__ void tk_split(float x, uint16_t& hi, uint16_t& lo) {
  if (F16) {
    const __half h = __float2half_rn(x);
    hi = __half_as_ushort(h); lo = __half_as_ushort(__float2half_rn(x - __half2float(h)));
  } else {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    hi = __bfloat16_as_ushort(h); lo = __bfloat16_as_ushort(__float2bfloat16_rn(x - __bfloat162float(h)));
  }
}
// Tagged words: {4 bytes of data, tag}.  Each 8-byte half of a 16-byte access is written and read as one unit.
__device__ __forceinline__ void tk_put2(uint2* p, uint32_t a, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(tag) : "memory");
}
__device__ __forceinline__ void tk_put4(void* p, uint32_t a, uint32_t b, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %3, %2, %3};" ::"l"(p), "r"(a), "r"(b), "r"(tag) : "memory");
}
__device__ __forceinline__ uint4 tk_peek(const void* p) {
  uint4 r;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
  return r;
}
constexpr long long TK_PATIENCE = 4000000000ll;      // cycles a wait lasts at most: about two seconds
static __device__ __noinline__ void tk_give_up(volatile int* abort_flag, int* status) {
  *abort_flag = 9;
  if (status) status[0] = DAISY_ETIMEOUT;
}
// N 16-byte words at p, p + step, .. once all of them carry the tag.  Bounded: the caller then gets whatever is there and
// the launch reports it.
template <int N>
__device__ __forceinline__ void tk_get(const uint4* p, int step, uint4 (&r)[N], uint32_t tag, volatile int* abort_flag, int* status) {
  const long long t0 = clock64();
  while (true) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = tk_peek(p + i * step);
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && r[i].y == tag && r[i].w == tag;
    if (ok || *abort_flag) return;
    if (clock64() - t0 > TK_PATIENCE) { tk_give_up(abort_flag, status); return; }
  }
}
__device__ __forceinline__ bool tk_bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > TK_PATIENCE) { tk_give_up(abort_flag, status); return false; }
  }
  return true;
}
// n tagged words of 4 bf16 each (two per 8-byte half) into a plain row in shared memory, by all threads
__device__ __forceinline__ void tk_gather(uint8_t* dst, const uint2* src, int n, uint32_t tag, volatile int* abort_flag, int* status) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += 2 * TK_CT) {
    const int d = i + TK_CT < n ? TK_CT : 0;                                    // (the same word twice at the end)
    uint4 r[2];
    tk_get(s + i, d, r, tag, abort_flag, status);
    *reinterpret_cast<uint2*>(dst + i * 8) = make_uint2(r[0].x, r[0].z);
    *reinterpret_cast<uint2*>(dst + (i + d) * 8) = make_uint2(r[1].x, r[1].z);
  }
}

// The consuming half of a warp's stream: TK_DEPTH (or one) buffers that are waited for in turn.  Derived classes know what
// the stream consists of: load(at) starts the copy of the warp's next piece into buffer `at`.
struct TokenRing {
  uint64_t* full;                                     // this warp's barriers
  uint32_t buf;                                       // and buffers
  int depth, st, par;                                 // next to consume
  int skip;                                           // pieces of the stream before the phase's first one of this warp
  volatile int* abort_flag;
  int* status;

  __device__ __forceinline__ uint32_t wait() {        // -> shared address of the piece
    (void)tk_bar_wait(&full[st], par, abort_flag, status);
    __syncwarp();
    return buf + st * TK_PIECE;
  }
  template <class S>
  __device__ __forceinline__ void done(S& s, int lane) {                       // the piece is used up: refill its place
    __syncwarp();
    if (lane == 0 && !*abort_flag) s.load(st);
    if (++st == depth) { st = 0; par ^= 1; }
  }
  // the warp's first piece among the next n of the stream, which then move on
  __device__ __forceinline__ int phase(int n) {
    const int first = skip;
    int k = skip - n;
    while (k < 0) k += TK_CW;
    skip = k;
    return first;
  }
  __device__ __forceinline__ void drain() {           // after a wait gave up: leave only when no copy is in flight any more
    if (!*abort_flag) return;
    const long long t0 = clock64();
    for (int i = 0; i < depth; ++i)
      while (!mbar_try_wait(&full[i], i < st ? par ^ 1 : par) && clock64() - t0 < TK_PATIENCE / 1000) {}
  }
};

// Rows of a weight times the batch's vectors: partial products per piece (16 rows x 256 columns) into psum, summed over the
// pieces of a row tile in a fixed order; emit(first, b, row, s0, s1) gets batch b's results of rows `row` (even) and row + 1,
// `first` true on a thread's first turn.  swz[j]: byte offset, inside a swizzled 16 x 128-byte block, of this lane's row and
// 16-byte piece 2 j (+ 1).  xs: the vectors in shared memory, once every thread has arrived here.
template <int NB, class Stream, class Emit>
__device__ __forceinline__ void tk_project(Stream& in, float* psum, uint32_t xs, int xs_ld, int B, int dim, int count, int pairs,
                                           const uint32_t (&swz)[4], int lane, Emit&& emit) {
  const int ks_n = (dim + TK_KW - 1) / TK_KW, g8 = lane >> 2, t4 = lane & 3;
  const int first = in.phase(count);
  const uint32_t xrow0 = xs + min(lane & 7, B - 1) * xs_ld + 16 * (lane >> 3), xrow1 = xs + min(8 + (lane & 7), B - 1) * xs_ld + 16 * (lane >> 3);
  int kb = first % ks_n;
  named_bar(1, TK_CT);                                                          // the vector is in shared memory
#pragma unroll 1
  for (int i = first; i < count; i += TK_CW) {
    uint32_t blk = in.wait(), xo = kb * (TK_KW * 2);
    float c[NB][2][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int j = 0; j < 8; ++j) c[nb][j >> 2][j & 3] = 0.f;
    const int blocks = min(TK_KW, dim - kb * TK_KW) / 64;
#pragma unroll 4
    for (int k = 0; k < blocks; ++k, blk += TK_BLK, xo += 128) {                // a 16 x 64 block of the piece
      uint32_t a[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) tk_ldm4(a[j], blk + swz[j]);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        uint32_t b[2][4];
        tk_ldm4(b[0], (nb ? xrow1 : xrow0) + xo); tk_ldm4(b[1], (nb ? xrow1 : xrow0) + xo + 64);
#pragma unroll
        for (int j = 0; j < 4; ++j) tk_mma<false>(c[nb][j & 1], a[j], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
      }
    }
    in.done(in, lane);
    float* ps = psum + i * (16 * 8 * NB) + g8 * (8 * NB) + 2 * t4;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      *reinterpret_cast<float2*>(ps + nb * 8) = make_float2(c[nb][0][0] + c[nb][1][0], c[nb][0][1] + c[nb][1][1]);
      *reinterpret_cast<float2*>(ps + 8 * (8 * NB) + nb * 8) = make_float2(c[nb][0][2] + c[nb][1][2], c[nb][0][3] + c[nb][1][3]);
    }
    kb += TK_CW;
    while (kb >= ks_n) kb -= ks_n;
  }
  named_bar(1, TK_CT);
#pragma unroll 1
  for (int i = threadIdx.x; i < pairs * B; i += TK_CT) {
    const int b = B == 1 ? 0 : (int)tk_div(i, pairs), row = 2 * (i - b * pairs);
    const float* ps = psum + (row >> 4) * ks_n * (16 * 8 * NB) + (row & 15) * (8 * NB) + b;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
    for (int k = 0; k < ks_n; ++k, ps += 16 * 8 * NB) { s0 += ps[0]; s1 += ps[8 * NB]; }
    emit(i < TK_CT, b, row, s0, s1);
  }
}

// bytes of psum for `tiles` row tiles of a CTA
static inline int tk_psum_bytes(int dim, int tiles, int NB) { return (dim + TK_KW - 1) / TK_KW * tiles * 16 * 8 * NB * 4; }

}  // namespace daisy

// weights [rows][dim] as (64 columns, rows, blocks of 64 columns), one piece a box
static inline int tk_make_map(CUtensorMap* m, const void* base, int nd, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  daisy_host::EncodeTiledFn enc = daisy_host::get_encode_tiled();
  if (!enc) return DAISY_ECUDA;
  const cuuint32_t one[5] = {1, 1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, nd, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? DAISY_OK : DAISY_ECUDA;
}
static inline int tk_make_weight_map(CUtensorMap* m, const void* base, int rows, int dim) {
  const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)dim / 64}, st[2] = {(cuuint64_t)dim * 2, 128};
  const cuuint32_t box[3] = {64, 16, daisy::TK_KW / 64};
  return tk_make_map(m, base, 3, dims, st, box);
}
