// Forward and backward for narrow heads (Dk, Dv <= 32, M <= 128 latents, bf16, softmax, token-causal) on the tensor cores at
// the precision of the fp32 kernels they stand in for (narrow_exact.cu).
//
// Tiles of 16 tokens; a warp owns 16 latents and all columns, and everything of a tile stays in its registers.  With the
// running maximum c through the tile as frame, E = exp2(s - c), D = d + cumsum E, R = (decode weight) / D, A = V dY^T:
//   forward   W = tril(R^T E)      Y = R^T U + W V      U += E V
//   backward  P = U dY^T + E A     X = G V^T + R A^T    dS = g (P / D - delta) + E (X - C - suffix sum of R P / D)
//             dV = E^T G + (E^T R) dY    dK = dS^T Q    dQ += dS K    G += R dY    C += sum of R P / D
// (A, W and E^T R masked to the causal half), the algebra of the kernels for wide heads.  The products run as bf16
// mma.sync.m16n8k16: every operand that is not the caller's own bf16 tensor (E, R, W, A, U, G, dS) enters as the sum of three
// bf16 values, all the 24 bits of its mantissa; terms below 2^-24 of a product are left out, and what lives over many tiles (U, G,
// dQ, the carries) takes a tile's product in one rounded fp32 addition.  The accumulator layout of one product is the A operand
// layout of the next one; the transposes that are left are movmatrix on the packed pairs.
// Why not tcgen05: the smallest product it takes is 64 rows against tensor memory, and a tile here is 16 x 16 x 32 with a scan
// over the tokens between every two products; per token and latent the work is the exponentials and the packing.
// The recurrence walked token by token (narrow_exact.cu) has a chain of 16 dependent steps where this has one.
//
// Warps share the tile's K, V (dY) in shared memory and meet twice per 32 tokens: partial read-outs (each warp in its own
// decode frame) and partial dV, dK are summed over the warps there.  Segments of the sequence run concurrently: states of the
// segments alone, folded by every CTA for itself; the backward's replay leaves the carries of the segments alone the same way.
//
// Sharp scores: the frame is the maximum through the tile, so a running maximum that grows by more than 2^57 inside a tile would
// flush weights that still count.  Such a tile is taken in windows, each with a frame of its own, that end before the token that
// outgrows them (at worst one token each); the reverse sweep finds the same windows again from the frame before the tile.  So only
// results that are not finite raise the CTA's gate word and let the fp32 kernels standing by redo the lane (forward) or the call
// (backward).  One CTA walks a whole lane there: before tiles were taken in windows, B=2 N=1000 H=4 M=64 D=32 with a standard
// deviation of 200 of the scores took 611 us forward and 950 us a step; 63 and 320 us in windows (85 and 383 us on the fp32 kernels).
// Code of its own for the tile that is one window: with one for both, every step took 5 % longer (516 us the one below).
//
// Precision: the distances of the bf16 outputs from 64 bits equal those of the fp32 kernels to 1 part in 10^6, either way, over
// M = 32 .. 128, N = 128 .. 4096, and 0.1 % of the outputs at most are rounded the other way, as there.  (Two values per operand
// were faster, 386 us for the step below where three took 472 before the windows, but left 0.1 to 0.5 % of the outputs rounded
// the other way and an fp32 dQ ten times as far from 64 bits.)  What is left is the tensor cores' own addition, which cuts off
// instead of rounding: 3.7e-7 of an fp32 dQ whatever N is, where the fp32 kernels have 2.8e-7 (N = 128) to 5.2e-7 (N = 4096).  A
// caller that wants dQ in fp32 gets the fp32 kernels.
//
// B200, training step B=8 N=2048 H=16 M=64 D=32: 1823 us on the fp32 kernels, 493 us on these; the forward alone 632
// and 132 us.
#include "narrow_mma.cuh"

#include <string.h>

#include <type_traits>

#include "bwd_exact.cuh"
#include "sm100_ptx.cuh"

namespace flare {

namespace {

using sm100::ex2_approx;
using sm100::pack_bf16;
using sm100::rcp_approx;
using sm100::smem_u32;

constexpr int BT = 32;         // tokens per staged block (two tiles)
constexpr int LD = 40;         // bf16 per staged row: 80 bytes, so that the eight rows of an ldmatrix lie in different banks
constexpr int LDP = 40;        // floats per row of a warp's partial outputs
constexpr int STAGE = BT * LD; // bf16 elements of a staged tensor
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kGrowth = 57.f;  // growth of the running maximum inside a window (log2 units) up to which nothing is lost: a
                                 // weight flushed to zero (below 2^-126) then stood for less than 2^-69 of its row's sum

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool on) {
  const int n = on ? 16 : 0;  // (0: zeros)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// tokens [t0, t0 + BT) as rows of 32 columns; zeros beyond t_end and beyond D
__device__ __forceinline__ void stage(__nv_bfloat16* dst, const void* src, int64_t off, int64_t stride_n, int t0, int t_end, int D) {
  const __nv_bfloat16* base = reinterpret_cast<const __nv_bfloat16*>(src) + off;
  for (int i = threadIdx.x; i < BT * 4; i += blockDim.x) {
    const int t = i >> 2, c = (i & 3) * 8;
    const bool on = t0 + t < t_end && c < D;
    cp_async16(dst + t * LD + c, on ? base + (int64_t)(t0 + t) * stride_n + c : base, on);
  }
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Thread (g, q) = (lane / 4, lane % 4).  An accumulator x[j] covers rows g (elements 0, 1) and g + 8 (2, 3) and columns
// 8 j + 2 q, + 1.  A 16 x 16 operand is the four 8 x 8 blocks (rows 0-7 | 8-15, columns 0-7), (rows 0-7 | 8-15, columns 8-15).
struct Split {
  uint32_t hi[4], mid[4], lo[4];
};
__device__ __forceinline__ void split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  mid = pack_bf16(x, y);
  lo = pack_bf16(x - __uint_as_float(mid << 16), y - __uint_as_float(mid & 0xffff0000u));
}
// accumulators of columns 0-7 and 8-15 as an A operand
__device__ __forceinline__ void split_tile(Split& p, const float (&x0)[4], const float (&x1)[4]) {
  split(x0[0], x0[1], p.hi[0], p.mid[0], p.lo[0]);
  split(x0[2], x0[3], p.hi[1], p.mid[1], p.lo[1]);
  split(x1[0], x1[1], p.hi[2], p.mid[2], p.lo[2]);
  split(x1[2], x1[3], p.hi[3], p.mid[3], p.lo[3]);
}
// the transposed 16 x 16 operand in A order; as B operand of a product over its own rows: columns 0-7 = blocks 0, 2 and
// columns 8-15 = blocks 1, 3 of this
__device__ __forceinline__ void transpose_blocks(uint32_t (&t)[4], const uint32_t (&p)[4]) {
  t[0] = transpose8(p[0]); t[1] = transpose8(p[2]); t[2] = transpose8(p[1]); t[3] = transpose8(p[3]);
}
__device__ __forceinline__ void transpose_tile(Split& t, const Split& p) {
  transpose_blocks(t.hi, p.hi);
  transpose_blocks(t.mid, p.mid);
  transpose_blocks(t.lo, p.lo);
}
// d += a b, small terms first: b exact, or both split (what is left out is below 2^-24 of the product)
__device__ __forceinline__ void mma_exact(float (&d)[4], const Split& a, uint32_t b0, uint32_t b1) {
  mma(d, a.lo, b0, b1);
  mma(d, a.mid, b0, b1);
  mma(d, a.hi, b0, b1);
}
struct Col {  // eight columns of a split B operand
  uint32_t hi0, hi1, mid0, mid1, lo0, lo1;
};
__device__ __forceinline__ void mma_split(float (&d)[4], const Split& a, const Col& b) {
  mma(d, a.lo, b.hi0, b.hi1);
  mma(d, a.hi, b.lo0, b.lo1);
  mma(d, a.mid, b.mid0, b.mid1);
  mma(d, a.mid, b.hi0, b.hi1);
  mma(d, a.hi, b.mid0, b.mid1);
  mma(d, a.hi, b.hi0, b.hi1);
}
template <int I>  // columns 8 I .. + 7 of an operand in the order above
__device__ __forceinline__ Col col(const Split& t) {
  return Col{t.hi[I], t.hi[I + 2], t.mid[I], t.mid[I + 2], t.lo[I], t.lo[I + 2]};
}
// an accumulator (16 rows, 8 columns) as B operand of a product over its rows
__device__ __forceinline__ Col as_col(const float (&x)[4]) {
  Col c;
  split(x[0], x[1], c.hi0, c.mid0, c.lo0);
  split(x[2], x[3], c.hi1, c.mid1, c.lo1);
  c.hi0 = transpose8(c.hi0); c.hi1 = transpose8(c.hi1);
  c.mid0 = transpose8(c.mid0); c.mid1 = transpose8(c.mid1);
  c.lo0 = transpose8(c.lo0); c.lo1 = transpose8(c.lo1);
  return c;
}
// Sums that live over many tiles take a tile's product in one rounded addition: the tensor cores cut off what does not fit
// the accumulator, always towards zero.
__device__ __forceinline__ void add_product(float (&sum)[4], const Split& a, uint32_t b0, uint32_t b1) {
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  mma_exact(d, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) sum[i] += d[i];
}

// rows of a staged tile (16 tokens): f[h][piece] = tokens 8 h .. + 7, columns 8 piece .. + 7.  B operand of a product over the
// columns (tokens as its columns): tile h, k-step s = f[h][2 s], f[h][2 s + 1].  A operand (tokens as rows): k-step s =
// f[0][2 s], f[1][2 s], f[0][2 s + 1], f[1][2 s + 1].
__device__ __forceinline__ void load_rows(uint32_t (&f)[2][4], const __nv_bfloat16* tile, int lane) {
  const __nv_bfloat16* p = tile + (lane & 7) * LD + (lane >> 3) * 8;
  ldsm4(f[0], p);
  ldsm4(f[1], p + 8 * LD);
}
// the same rows as B operand of a product over the tokens: columns 8 n .. + 7 = f[n][0], f[n][1]
__device__ __forceinline__ void load_cols(uint32_t (&f)[4][2], const __nv_bfloat16* tile, int lane) {
  const __nv_bfloat16* p = tile + (((lane >> 3) & 1) * 8 + (lane & 7)) * LD + (lane >> 4) * 8;
  ldsm4t(f[0][0], f[0][1], f[1][0], f[1][1], p);
  ldsm4t(f[2][0], f[2][1], f[3][0], f[3][1], p + 16);
}
__device__ __forceinline__ void as_rows(uint32_t (&a)[4], const uint32_t (&f)[2][4], int s) {
  a[0] = f[0][2 * s]; a[1] = f[1][2 * s]; a[2] = f[0][2 * s + 1]; a[3] = f[1][2 * s + 1];
}

// latent bank rows of this warp as A operand of the score product
__device__ __forceinline__ void load_bank(uint32_t (&qa)[2][4], const NarrowMmaParams& p, int h, int m0, int lane) {
  const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(p.q) + (int64_t)h * p.q_stride_h;
  const int g = lane >> 2, c = (lane & 3) * 2;
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = s * 16 + (i >> 1) * 8 + c, row = m0 + g + (i & 1) * 8;
      qa[s][i] = col < p.Dk ? *reinterpret_cast<const uint32_t*>(q + (int64_t)row * p.q_stride_m + col) : 0u;
    }
}

// scores (log2 units) of 16 latents and 16 tokens
__device__ __forceinline__ void scores(float (&s)[2][4], const uint32_t (&qa)[2][4], const uint32_t (&kf)[2][4], float sc2) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[j][i] = 0.f;
    mma(s[j], qa[0], kf[j][0], kf[j][1]);
    mma(s[j], qa[1], kf[j][2], kf[j][3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) s[j][i] *= sc2;
  }
}

// running maximum cn of the rows through the tokens [lo, end) of the tile
__device__ __forceinline__ void maximum_through(float (&cn)[2], const float (&s)[2][4], const float (&c)[2], int lo, int end, int lane) {
  const int q2 = (lane & 3) * 2;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float top = kNegInf;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int t = 8 * j + q2 + x;
        if (t >= lo && t < end) top = fmaxf(top, s[j][2 * r + x]);
      }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    cn[r] = fmaxf(c[r], top);
  }
}
__device__ __forceinline__ void change_frame(float (&c)[2], float (&alpha)[2], const float (&cn)[2]) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    alpha[r] = ex2_approx(c[r] - cn[r]);  // (an empty state: 0)
    c[r] = cn[r];
  }
}
// Frame through the tile: c becomes the running maximum, alpha the factor from the old frame.  False, and nothing done, where one
// frame may not hold the tile (the first tile of all among them, which has nothing to grow from).
__device__ __forceinline__ bool tile_frame(const float (&s)[2][4], float (&c)[2], float (&alpha)[2], int nvalid, int lane) {
  float cn[2];
  maximum_through(cn, s, c, 0, nvalid, lane);
  if (__any_sync(0xffffffffu, cn[0] - c[0] > kGrowth || cn[1] - c[1] > kGrowth)) return false;
  change_frame(c, alpha, cn);
  return true;
}
// The same for a window of the tile that begins at token lo.  Returns its end: the first token that outgrows it, else nvalid.
__device__ __forceinline__ int window_frame(const float (&s)[2][4], float (&c)[2], float (&alpha)[2], int lo, int nvalid, int lane) {
  const int q2 = (lane & 3) * 2;
  float low[2], cn[2];  // what the window grows from, its maximum
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float mine = (lo & 8) ? ((lo & 1) ? s[1][2 * r + 1] : s[1][2 * r]) : ((lo & 1) ? s[0][2 * r + 1] : s[0][2 * r]);
    low[r] = fmaxf(c[r], __shfl_sync(0xffffffffu, mine, (lane & ~3) + ((lo >> 1) & 3)));
  }
  int end = nvalid;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = 8 * j + q2 + (i & 1);
      if (t > lo && t < end && s[j][i] - low[i >> 1] > kGrowth) end = t;
    }
  end = __reduce_min_sync(0xffffffffu, end);
  maximum_through(cn, s, c, lo, end, lane);
  change_frame(c, alpha, cn);
  return end;
}
// whether a token is of a window that is the whole tile (then all that is checked is the sequence's end), or a part of it
template <bool WHOLE>
__device__ __forceinline__ bool in_window(int t, int lo, int hi) { return WHOLE ? t < hi : t >= lo && t < hi; }

// encoder weights in the frame c of the window [lo, hi), zero outside
template <bool WHOLE>
__device__ __forceinline__ void encode(float (&e)[2][4], const float (&s)[2][4], const float (&c)[2], int lo, int hi, int lane) {
  const int q2 = (lane & 3) * 2;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = 8 * j + q2 + (i & 1);
      e[j][i] = in_window<WHOLE>(t, lo, hi) ? ex2_approx(s[j][i] - c[i >> 1]) : 0.f;
    }
}

// den = base + running sum over the tokens; base becomes the sum through the tile
__device__ __forceinline__ void scan(float (&den)[2][4], const float (&e)[2][4], float (&base)[2], int lane) {
  const int q = lane & 3;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float run = e[j][2 * r] + e[j][2 * r + 1];
      float t = __shfl_up_sync(0xffffffffu, run, 1, 4);
      if (q >= 1) run += t;
      t = __shfl_up_sync(0xffffffffu, run, 2, 4);
      if (q >= 2) run += t;
      const float before = __shfl_up_sync(0xffffffffu, run, 1, 4);
      const float total = __shfl_sync(0xffffffffu, run, 3, 4);
      den[j][2 * r] = (q >= 1 ? base[r] + before : base[r]) + e[j][2 * r];
      den[j][2 * r + 1] = den[j][2 * r] + e[j][2 * r + 1];
      base[r] += total;
    }
}

__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
// Sum over the warp's latents of a per-token value: v[j][x] = this thread's part for token 8 j + 2 q + x.  The thread keeps the
// sum of one of its four tokens, summed_token (threads that differ in bit 2 of the lane hold the same).
__device__ __forceinline__ float sum_latents(float (&v)[2][2], int lane) {
  const bool up = lane & 16, up2 = lane & 8;
  float a = up ? v[1][0] : v[0][0], b = up ? v[1][1] : v[0][1];
  a += __shfl_xor_sync(0xffffffffu, up ? v[0][0] : v[1][0], 16);
  b += __shfl_xor_sync(0xffffffffu, up ? v[0][1] : v[1][1], 16);
  float x = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
  return x + __shfl_xor_sync(0xffffffffu, x, 4);
}
__device__ __forceinline__ int summed_token(int lane) { return ((lane & 16) ? 8 : 0) + (lane & 3) * 2 + ((lane & 8) ? 1 : 0); }

// decode frame of the warp's latents per token: maximum score
__device__ __forceinline__ void decode_frame(float (&kap)[2][2], const float (&s)[2][4]) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      float t = fmaxf(s[j][x], s[j][2 + x]);
      t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 4));
      t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 8));
      kap[j][x] = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 16));
    }
}
__device__ __forceinline__ float summed_frame(const float (&kap)[2][2], int lane) {  // that of summed_token
  return (lane & 16) ? ((lane & 8) ? kap[1][1] : kap[1][0]) : ((lane & 8) ? kap[0][1] : kap[0][0]);
}

// a warp's partial rows of a tile: this thread's pieces of rows g and g + 8; windows after the first one add theirs
__device__ __forceinline__ void put_rows(float* dst, const float (&x)[4], bool add) {
  float2 *const a = reinterpret_cast<float2*>(dst), *const b = reinterpret_cast<float2*>(dst + 8 * LDP);
  float2 p = make_float2(x[0], x[1]), q = make_float2(x[2], x[3]);
  if (add) {
    const float2 p0 = *a, q0 = *b;
    p.x += p0.x; p.y += p0.y; q.x += q0.x; q.y += q0.y;
  }
  *a = p;
  *b = q;
}

template <int ROWS>
__device__ __forceinline__ void zero(float (&x)[ROWS][4]) {
#pragma unroll
  for (int n = 0; n < ROWS; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) x[n][i] = 0.f;
}

// state before segment `seg` (frame c in log2 units, d, u in the accumulator layout): the segments before it, folded in order
__device__ __forceinline__ void prefix_state(const NarrowMmaParams& p, int lane_id, int seg, int m0, int lane, float (&c)[2],
                                             float (&d)[2], float (&u)[4][4]) {
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  c[0] = c[1] = kNegInf;
  d[0] = d[1] = 0.f;
  zero(u);
  for (int s = 0; s < seg; ++s) {
    const int64_t st = ((int64_t)lane_id * p.nseg + s) * p.M + m0 + g;
    float mb[2] = {p.seg_m[st] * kLog2e, p.seg_m[st + 8] * kLog2e}, db[2] = {p.seg_d[st], p.seg_d[st + 8]};
    float2 ub[4][2];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        ub[n][r] = 8 * n + q2 < p.Dv ? *reinterpret_cast<const float2*>(p.seg_u + (st + 8 * r) * p.Dv + 8 * n + q2) : make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float cn = fmaxf(c[r], mb[r]), fa = ex2_approx(c[r] - cn), fb = ex2_approx(mb[r] - cn);
      c[r] = cn;
      d[r] = d[r] * fa + db[r] * fb;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        u[n][2 * r] = u[n][2 * r] * fa + ub[n][r].x * fb;
        u[n][2 * r + 1] = u[n][2 * r + 1] * fa + ub[n][r].y * fb;
      }
    }
  }
}

__device__ __forceinline__ void rescale(float (&u)[4][4], const float (&f)[2]) {
  if (__any_sync(0xffffffffu, f[0] != 1.f || f[1] != 1.f)) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) u[n][i] *= f[i >> 1];
  }
}

// ---------------------------------------------------------------------------------------------
// forward: the state of a segment alone (WRITE_Y false), or its read-out
// ---------------------------------------------------------------------------------------------
template <int THREADS, bool WRITE_Y>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) narrow_mma_forward_kernel(const NarrowMmaParams p) {
  pdl_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q2 = (lane & 3) * 2;
  __nv_bfloat16* const kv = reinterpret_cast<__nv_bfloat16*>(smem_raw);  // two stages of (K, V)
  float* const ypart = reinterpret_cast<float*>(kv + 4 * STAGE);         // [nw][BT][LDP]
  float* const kap_s = ypart + nw * BT * LDP;                            // [nw][BT]
  float* const sum_s = kap_s + nw * BT;                                  // [nw][BT]
  const int lane_id = blockIdx.x, seg = blockIdx.y, b = lane_id / p.H, h = lane_id % p.H, m0 = warp * 16;
  const int tbeg = seg * p.seg_len, tend = min(p.N, tbeg + p.seg_len);
  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t y_off = (int64_t)b * p.y_stride_b + (int64_t)h * p.y_stride_h;
  const float sc2 = p.scale * kLog2e;
  stage(kv, p.k, k_off, p.k_stride_n, tbeg, tend, p.Dk);
  stage(kv + STAGE, p.v, v_off, p.v_stride_n, tbeg, tend, p.Dv);
  cp_async_commit();
  uint32_t qa[2][4];
  load_bank(qa, p, h, m0, lane);
  float c[2], d[2], u[4][4];
  prefix_state(p, lane_id, WRITE_Y ? seg : 0, m0, lane, c, d, u);
  bool ok = true;
  for (int t0 = tbeg, buf = 0; t0 < tend; t0 += BT, buf ^= 1) {
    cp_async_wait_all();
    __syncthreads();  // this block is in place, and everyone is done with the one before and its partial outputs
    if (t0 + BT < tend) {
      stage(kv + (buf ^ 1) * 2 * STAGE, p.k, k_off, p.k_stride_n, t0 + BT, tend, p.Dk);
      stage(kv + (buf ^ 1) * 2 * STAGE + STAGE, p.v, v_off, p.v_stride_n, t0 + BT, tend, p.Dv);
      cp_async_commit();
    }
#pragma unroll 1
    for (int tile = 0; tile < 2; ++tile) {
      const int nvalid = min(16, tend - t0 - tile * 16);
      if (nvalid <= 0) break;
      const __nv_bfloat16* const ks = kv + buf * 2 * STAGE + tile * 16 * LD;
      const __nv_bfloat16* const vs = ks + STAGE;
      auto tile_scores = [&](float (&s)[2][4]) {
        uint32_t kf[2][4];
        load_rows(kf, ks, lane);
        scores(s, qa, kf, sc2);
      };
      // the window [lo, hi) of the tile, whose frame is c
      auto window = [&](auto whole, const float (&s)[2][4], const float (&alpha)[2], int lo, int hi) {
        constexpr bool WHOLE = decltype(whole)::value;
        float e[2][4];
        encode<WHOLE>(e, s, c, lo, hi, lane);
        d[0] *= alpha[0];
        d[1] *= alpha[1];
        rescale(u, alpha);
        uint32_t vt[4][2];
        load_cols(vt, vs, lane);
        Split ep;
        split_tile(ep, e[0], e[1]);
        if constexpr (WRITE_Y) {
          float den[2][4];
          scan(den, e, d, lane);
          // decode weights in the warp's own frame, their sum, R
          float kap[2][2], part[2][2], r[2][4];
          decode_frame(kap, s);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) r[j][i] = ex2_approx(s[j][i] - kap[j][i & 1]);
            part[j][0] = r[j][0] + r[j][2];
            part[j][1] = r[j][1] + r[j][3];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int t = 8 * j + q2 + (i & 1);
              r[j][i] = in_window<WHOLE>(t, lo, hi) ? r[j][i] * rcp_approx(den[j][i]) : 0.f;
            }
          }
          const float sum = sum_latents(part, lane);
          if (!(lane & 4)) {
            const int t = warp * BT + tile * 16 + summed_token(lane);
            sum_s[t] = sum;
            kap_s[t] = summed_frame(kap, lane);
          }
          Split rp, rt, et;
          split_tile(rp, r[0], r[1]);
          transpose_tile(rt, rp);  // A operand: tokens x latents
          transpose_tile(et, ep);  // B operand over the latents
          float y[4][4];
          zero(y);
          {
            float w[2][4];
            zero(w);
            mma_split(w[0], rt, col<0>(et));
            mma_split(w[1], rt, col<1>(et));
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int i = 0; i < 4; ++i) w[j][i] = 8 * j + q2 + (i & 1) <= g + (i >> 1) * 8 ? w[j][i] : 0.f;
            Split wp;
            split_tile(wp, w[0], w[1]);
#pragma unroll
            for (int n = 0; n < 4; ++n) mma_exact(y[n], wp, vt[n][0], vt[n][1]);
          }
#pragma unroll
          for (int n = 0; n < 4; ++n) mma_split(y[n], rt, as_col(u[n]));
          float* const dst = ypart + (warp * BT + tile * 16 + g) * LDP + q2;
#pragma unroll
          for (int n = 0; n < 4; ++n) put_rows(dst + 8 * n, y[n], !WHOLE && lo > 0);
        } else {
#pragma unroll
          for (int r = 0; r < 2; ++r) d[r] += quad_sum((e[0][2 * r] + e[0][2 * r + 1]) + (e[1][2 * r] + e[1][2 * r + 1]));
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) add_product(u[n], ep, vt[n][0], vt[n][1]);
      };
      float s[2][4], alpha[2];
      tile_scores(s);
      if constexpr (!WRITE_Y) {  // (what is lost in a frame too high counts for nothing at the segment's end)
        float cn[2];
        maximum_through(cn, s, c, 0, nvalid, lane);
        change_frame(c, alpha, cn);
        window(std::true_type(), s, alpha, 0, nvalid);
      } else if (tile_frame(s, c, alpha, nvalid, lane)) {
        window(std::true_type(), s, alpha, 0, nvalid);
      } else {
#pragma unroll 1
        for (int lo = 0, hi; lo < nvalid; lo = hi) {
          tile_scores(s);
          hi = window_frame(s, c, alpha, lo, nvalid, lane);
          window(std::false_type(), s, alpha, lo, hi);
        }
      }
    }
    if constexpr (WRITE_Y) {
      __syncthreads();
      // read-out rows: the warps' partial sums in a common decode frame; thread = (token, 8 columns)
      for (int i = threadIdx.x; i < BT * 4; i += blockDim.x) {
        const int t = i >> 2, col = (i & 3) * 8;
        if (t0 + t >= tend || col >= p.Dv) continue;
        float top = kap_s[t];
        for (int w = 1; w < nw; ++w) top = fmaxf(top, kap_s[w * BT + t]);
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, total = 0.f;
        for (int w = 0; w < nw; ++w) {
          const float f = ex2_approx(kap_s[w * BT + t] - top);
          total = fmaf(f, sum_s[w * BT + t], total);
          const float4* src = reinterpret_cast<const float4*>(ypart + (w * BT + t) * LDP + col);
          const float4 x = src[0], z = src[1];
          acc[0] = fmaf(f, x.x, acc[0]); acc[1] = fmaf(f, x.y, acc[1]); acc[2] = fmaf(f, x.z, acc[2]); acc[3] = fmaf(f, x.w, acc[3]);
          acc[4] = fmaf(f, z.x, acc[4]); acc[5] = fmaf(f, z.y, acc[5]); acc[6] = fmaf(f, z.z, acc[6]); acc[7] = fmaf(f, z.w, acc[7]);
        }
        const float inv = 1.0f / total;
        float check = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[j] *= inv;
          check = fmaf(acc[j], 0.f, check);
        }
        ok = ok && check == 0.f;  // (0 x inf and 0 x NaN are not)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.y) + y_off + (int64_t)(t0 + t) * p.y_stride_n + col) =
            make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
      }
    }
  }
  if constexpr (WRITE_Y) {
    const int bad = __syncthreads_or(!ok);
    if (threadIdx.x == 0) {
      p.gate[1 + (int64_t)lane_id * p.gate_stride + seg] = bad;
      if (lane_id == 0 && seg == 0) p.gate[0] = p.gate_stride;
    }
  } else {
    // (what leaves the domain here does so in the pass that walks the segment again, or arrives there as a NaN)
    const int64_t st = ((int64_t)lane_id * p.nseg + seg) * p.M + m0 + g;
    if (q2 == 0) {
      p.seg_m[st] = c[0] * kLn2;
      p.seg_m[st + 8] = c[1] * kLn2;
      p.seg_d[st] = d[0];
      p.seg_d[st + 8] = d[1];
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (8 * n + q2 < p.Dv)
          *reinterpret_cast<float2*>(p.seg_u + (st + 8 * r) * p.Dv + 8 * n + q2) = make_float2(u[n][2 * r], u[n][2 * r + 1]);
  }
}

// ---------------------------------------------------------------------------------------------
// backward, replay: per-tile frames and denominators, p of every (token, latent), per-token log-sum-exp and <dY, y>, the
// carries of the segment alone
// ---------------------------------------------------------------------------------------------
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 384 / THREADS) narrow_mma_replay_kernel(const NarrowMmaParams p) {
  pdl_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q2 = (lane & 3) * 2;
  __nv_bfloat16* const kv = reinterpret_cast<__nv_bfloat16*>(smem_raw);  // two stages of (K, V, dY)
  float* const kap_s = reinterpret_cast<float*>(kv + 6 * STAGE);         // [2][nw][BT] (block parity)
  float* const sum_s = kap_s + 2 * nw * BT;                              // [2][nw][BT]
  float* const del_s = sum_s + 2 * nw * BT;                              // [2][nw][BT]
  const int lane_id = blockIdx.x, seg = blockIdx.y, b = lane_id / p.H, h = lane_id % p.H, m0 = warp * 16;
  const int tbeg = seg * p.seg_len, tend = min(p.N, tbeg + p.seg_len);
  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t dy_off = (int64_t)b * p.dy_stride_b + (int64_t)h * p.dy_stride_h;
  const float sc2 = p.scale * kLog2e;
  auto stage_all = [&](int buf, int t0) {
    __nv_bfloat16* const dst = kv + buf * 3 * STAGE;
    stage(dst, p.k, k_off, p.k_stride_n, t0, tend, p.Dk);
    stage(dst + STAGE, p.v, v_off, p.v_stride_n, t0, tend, p.Dv);
    stage(dst + 2 * STAGE, p.dy, dy_off, p.dy_stride_n, t0, tend, p.Dv);
    cp_async_commit();
  };
  stage_all(0, tbeg);
  uint32_t qa[2][4];
  load_bank(qa, p, h, m0, lane);
  float c[2], d[2], u[4][4], b0[4][4], c0[2] = {0.f, 0.f};
  prefix_state(p, lane_id, seg, m0, lane, c, d, u);
  zero(b0);
  const float c_start[2] = {c[0], c[1]};
  const bool carries = seg > 0;
  bool ok = true;
  for (int t0 = tbeg, buf = 0; t0 < tend; t0 += BT, buf ^= 1) {
    cp_async_wait_all();
    __syncthreads();
    if (t0 + BT < tend) stage_all(buf ^ 1, t0 + BT);
    const __nv_bfloat16* const block = kv + buf * 3 * STAGE;
    // decode log-sum-exp of the block's tokens over all latents
#pragma unroll 1
    for (int tile = 0; tile < 2; ++tile) {
      float s[2][4], kap[2][2], part[2][2];
      uint32_t kf[2][4];
      load_rows(kf, block + tile * 16 * LD, lane);
      scores(s, qa, kf, sc2);
      decode_frame(kap, s);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int x = 0; x < 2; ++x) part[j][x] = ex2_approx(s[j][x] - kap[j][x]) + ex2_approx(s[j][2 + x] - kap[j][x]);
      const float sum = sum_latents(part, lane);
      if (!(lane & 4)) {
        const int t = (buf * nw + warp) * BT + tile * 16 + summed_token(lane);
        sum_s[t] = sum;
        kap_s[t] = summed_frame(kap, lane);
      }
    }
    __syncthreads();
    float l2;  // of token t0 + lane
    {
      const float* const kp = kap_s + buf * nw * BT + lane;
      const float* const sp = sum_s + buf * nw * BT + lane;
      float top = kp[0], total = 0.f;
      for (int w = 1; w < nw; ++w) top = fmaxf(top, kp[w * BT]);
      for (int w = 0; w < nw; ++w) total = fmaf(ex2_approx(kp[w * BT] - top), sp[w * BT], total);
      l2 = top + log2f(total);
      if (warp == 0 && t0 + lane < tend) p.tok_l2[(int64_t)lane_id * p.ntiles * 16 + t0 + lane] = l2;
      // (the sums of <dY, y> of the block before: complete since the barrier at the top of this one)
      if (warp == 0 && t0 > tbeg) {
        const float* const dp = del_s + (buf ^ 1) * nw * BT + lane;
        float delta = dp[0];
        for (int w = 1; w < nw; ++w) delta += dp[w * BT];
        p.tok_delta[(int64_t)lane_id * p.ntiles * 16 + t0 - BT + lane] = delta;
      }
    }
#pragma unroll 1
    for (int tile = 0; tile < 2; ++tile) {
      const int nvalid = min(16, tend - t0 - tile * 16);
      if (nvalid <= 0) break;
      const int64_t tile_id = (int64_t)lane_id * p.ntiles + (t0 >> 4) + tile;
      const __nv_bfloat16* const ks = block + tile * 16 * LD;
      auto tile_scores = [&](float (&s)[2][4]) {
        uint32_t kf[2][4];
        load_rows(kf, ks, lane);
        scores(s, qa, kf, sc2);
      };
      auto window = [&](auto whole, const float (&s)[2][4], const float (&alpha)[2], int lo, int hi) {
        constexpr bool WHOLE = decltype(whole)::value;
        float e[2][4], den[2][4], r[2][4];
        encode<WHOLE>(e, s, c, lo, hi, lane);
        if ((WHOLE || lo == 0) && (lane & 3) == 0) {
#pragma unroll
          for (int i = 0; i < 2; ++i) p.stat_d[tile_id * p.M + m0 + g + 8 * i] = !WHOLE && hi < nvalid ? -d[i] : d[i];
        }
        d[0] *= alpha[0];
        d[1] *= alpha[1];
        rescale(u, alpha);
        scan(den, e, d, lane);
        float dec[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int t = 8 * j + q2 + x;
            const float l = __shfl_sync(0xffffffffu, l2, tile * 16 + t);
#pragma unroll
            for (int i = x; i < 4; i += 2) {
              dec[j][i] = t < nvalid ? ex2_approx(s[j][i] - l) : 0.f;
              r[j][i] = in_window<WHOLE>(t, lo, hi) ? rcp_approx(den[j][i]) : 0.f;  // 1 / D
            }
          }
        Split ep;
        split_tile(ep, e[0], e[1]);
        uint32_t vf[2][4], df[2][4];
        load_rows(vf, ks + STAGE, lane);
        load_rows(df, ks + 2 * STAGE, lane);
        float pp[2][4];
        zero(pp);
        {
          // A^T = dY V^T, masked to tau <= t, as B operand of a product over tau
          float at[2][4];
          zero(at);
#pragma unroll
          for (int k2 = 0; k2 < 2; ++k2) {
            uint32_t a[4];
            as_rows(a, df, k2);
            mma(at[0], a, vf[0][2 * k2], vf[0][2 * k2 + 1]);
            mma(at[1], a, vf[1][2 * k2], vf[1][2 * k2 + 1]);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) at[j][i] = 8 * j + q2 + (i & 1) <= g + (i >> 1) * 8 ? at[j][i] : 0.f;
          Split ap;
          split_tile(ap, at[0], at[1]);  // blocks (t 0-7 | 8-15, tau 0-7), (t 0-7 | 8-15, tau 8-15)
          mma_split(pp[0], ep, col<0>(ap));
          mma_split(pp[1], ep, col<1>(ap));
        }
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          Split up;
          split_tile(up, u[2 * k2], u[2 * k2 + 1]);
          mma_exact(pp[0], up, df[0][2 * k2], df[0][2 * k2 + 1]);
          mma_exact(pp[1], up, df[1][2 * k2], df[1][2 * k2 + 1]);
        }
        float part[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            pp[j][i] *= r[j][i];   // p
            r[j][i] *= dec[j][i];  // R
          }
          part[j][0] = dec[j][0] * pp[j][0] + dec[j][2] * pp[j][2];
          part[j][1] = dec[j][1] * pp[j][1] + dec[j][3] * pp[j][3];
          // (zero outside the window)
          float4* const out = p.p + ((tile_id * nw + warp) * 2 + j) * 32 + lane;
          float4 x = make_float4(pp[j][0], pp[j][1], pp[j][2], pp[j][3]);
          if (!WHOLE && lo > 0) {
            const float4 y = *out;
            x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
          }
          *out = x;
        }
        const float sum = sum_latents(part, lane);
        if (!(lane & 4)) {
          float* const out = del_s + (buf * nw + warp) * BT + tile * 16 + summed_token(lane);
          *out = !WHOLE && lo > 0 ? *out + sum : sum;
        }
        {
          uint32_t vt[4][2];
          load_cols(vt, ks + STAGE, lane);
#pragma unroll
          for (int n = 0; n < 4; ++n) add_product(u[n], ep, vt[n][0], vt[n][1]);
        }
        if (carries) {
          // in the frame before the segment (the frames only grow, so the factors stay below 1)
          const float f[2] = {ex2_approx(c_start[0] - c[0]), ex2_approx(c_start[1] - c[1])};
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              r[j][i] *= f[i >> 1];
              c0[i >> 1] = fmaf(r[j][i], pp[j][i], c0[i >> 1]);
            }
          Split rp;
          split_tile(rp, r[0], r[1]);
          uint32_t dt[4][2];
          load_cols(dt, ks + 2 * STAGE, lane);
#pragma unroll
          for (int n = 0; n < 4; ++n) add_product(b0[n], rp, dt[n][0], dt[n][1]);
        }
      };
      float s[2][4], alpha[2];
      tile_scores(s);
      if (tile_frame(s, c, alpha, nvalid, lane)) {
        window(std::true_type(), s, alpha, 0, nvalid);
      } else {
#pragma unroll 1
        for (int lo = 0, hi; lo < nvalid; lo = hi) {
          tile_scores(s);
          hi = window_frame(s, c, alpha, lo, nvalid, lane);
          window(std::false_type(), s, alpha, lo, hi);
        }
      }
      if ((lane & 3) == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) p.stat_c[tile_id * p.M + m0 + g + 8 * i] = c[i];
      }
      ok = ok && c[0] < INFINITY && c[1] < INFINITY;
    }
  }
  const int bad = __syncthreads_or(!ok);
  const int nblocks = (tend - tbeg + BT - 1) / BT;
  if (warp == 0) {
    const int t_last = tbeg + (nblocks - 1) * BT;
    const float* const dp = del_s + ((nblocks - 1) & 1) * nw * BT + lane;
    float delta = dp[0];
    for (int w = 1; w < nw; ++w) delta += dp[w * BT];
    if (t_last + lane < tend) p.tok_delta[(int64_t)lane_id * p.ntiles * 16 + t_last + lane] = delta;
    if (lane == 0) p.gate[lane_id * p.nseg + seg] = bad;
  }
  const int64_t st = ((int64_t)lane_id * p.nseg + seg) * p.M + m0 + g;
  const float cs[2] = {quad_sum(c0[0]), quad_sum(c0[1])};
  if ((lane & 3) == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      p.start_c[st + 8 * i] = c_start[i];
      p.seg_c[st + 8 * i] = cs[i];
    }
  }
  if (carries) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (8 * n + q2 < p.Dv)
          *reinterpret_cast<float2*>(p.seg_b + (st + 8 * i) * p.Dv + 8 * n + q2) = make_float2(b0[n][2 * i], b0[n][2 * i + 1]);
  }
}

// ---------------------------------------------------------------------------------------------
// backward, reverse sweep: dV, dK and this segment's part of dQ
// ---------------------------------------------------------------------------------------------
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 384 / THREADS) narrow_mma_reverse_kernel(const NarrowMmaParams p) {
  pdl_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, q2 = q * 2;
  __nv_bfloat16* const kv = reinterpret_cast<__nv_bfloat16*>(smem_raw);  // two stages of (K, V, dY)
  float* const part = reinterpret_cast<float*>(kv + 6 * STAGE);          // [dV | dK][nw][BT][LDP]
  __nv_bfloat16* const qs = reinterpret_cast<__nv_bfloat16*>(part + 2 * nw * BT * LDP);  // [M][LD] latent bank
  const int lane_id = blockIdx.x, seg = blockIdx.y, b = lane_id / p.H, h = lane_id % p.H, m0 = warp * 16;
  const int tbeg = seg * p.seg_len, tend = min(p.N, tbeg + p.seg_len);
  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t dy_off = (int64_t)b * p.dy_stride_b + (int64_t)h * p.dy_stride_h;
  const float sc2 = p.scale * kLog2e;
  auto stage_all = [&](int buf, int t0) {
    __nv_bfloat16* const dst = kv + buf * 3 * STAGE;
    stage(dst, p.k, k_off, p.k_stride_n, t0, tend, p.Dk);
    stage(dst + STAGE, p.v, v_off, p.v_stride_n, t0, tend, p.Dv);
    stage(dst + 2 * STAGE, p.dy, dy_off, p.dy_stride_n, t0, tend, p.Dv);
    cp_async_commit();
  };
  const int t_top = tbeg + (tend - tbeg - 1) / BT * BT;
  {
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(p.q) + (int64_t)h * p.q_stride_h;
    for (int i = threadIdx.x; i < p.M * 4; i += blockDim.x) {
      const int m = i >> 2, col = (i & 3) * 8;
      cp_async16(qs + m * LD + col, col < p.Dk ? src + (int64_t)m * p.q_stride_m + col : src, col < p.Dk);
    }
  }
  stage_all(0, t_top);
  uint32_t qa[2][4];
  load_bank(qa, p, h, m0, lane);
  // carries of the later segments, each in the frame before it, into the frame behind this segment
  float gr[4][4], dq[4][4], cc[2] = {0.f, 0.f};
  zero(gr);
  zero(dq);
  {
    float c_from[2] = {0.f, 0.f};
    for (int s = p.nseg - 1; s > seg; --s) {
      const int64_t st = ((int64_t)lane_id * p.nseg + s) * p.M + m0 + g;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float c_to = p.start_c[st + 8 * r];
        const float f = s == p.nseg - 1 ? 0.f : ex2_approx(c_to - c_from[r]);
        c_from[r] = c_to;
        cc[r] = fmaf(cc[r], f, p.seg_c[st + 8 * r]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float2 x = 8 * n + q2 < p.Dv ? *reinterpret_cast<const float2*>(p.seg_b + (st + 8 * r) * p.Dv + 8 * n + q2) : make_float2(0.f, 0.f);
          gr[n][2 * r] = fmaf(gr[n][2 * r], f, x.x);
          gr[n][2 * r + 1] = fmaf(gr[n][2 * r + 1], f, x.y);
        }
      }
    }
  }
  bool ok = true;
  for (int t0 = t_top, buf = 0; t0 >= tbeg; t0 -= BT, buf ^= 1) {
    const int64_t tok = (int64_t)lane_id * p.ntiles * 16 + t0 + lane;
    const bool in = t0 + lane < tend;
    const float l2 = in ? p.tok_l2[tok] : 0.f, delta = in ? p.tok_delta[tok] : 0.f;
    cp_async_wait_all();
    __syncthreads();
    if (t0 - BT >= tbeg) stage_all(buf ^ 1, t0 - BT);
    const __nv_bfloat16* const block = kv + buf * 3 * STAGE;
#pragma unroll 1
    for (int tile = 1; tile >= 0; --tile) {
      const int nvalid = min(16, tend - t0 - tile * 16);
      if (nvalid <= 0) continue;
      const int64_t tile_id = (int64_t)lane_id * p.ntiles + (t0 >> 4) + tile;
      const __nv_bfloat16* const ks = block + tile * 16 * LD;
      const float4* const pt = p.p + ((tile_id * nw + warp) * 2) * 32 + lane;
      const int64_t so = tile_id * p.M + m0 + g;
      // frame before the tile
      const float* const cb = t0 + tile * 16 > tbeg ? p.stat_c + so - p.M : p.start_c + ((int64_t)lane_id * p.nseg + seg) * p.M + m0 + g;
      // the window of the tile that ends at `end`; returns its begin
      auto window = [&](auto whole, int end) -> int {
        constexpr bool WHOLE = decltype(whole)::value;
        int begin = 0;
        float e[2][4], r[2][4], ds[2][4], rp[2][4], phi[2];  // (phi: the factor to the frame before the window)
        {
          const float4 p0 = pt[0], p1 = pt[32];
          const float pv[2][4] = {{p0.x, p0.y, p0.z, p0.w}, {p1.x, p1.y, p1.z, p1.w}};
          float c[2] = {cb[0], cb[8]}, run[2] = {p.stat_d[so], p.stat_d[so + 8]};
          float s[2][4], den[2][4];
          uint32_t kf[2][4];
          load_rows(kf, ks, lane);
          scores(s, qa, kf, sc2);
          if constexpr (WHOLE) {
            const float cn[2] = {p.stat_c[so], p.stat_c[so + 8]};
            change_frame(c, phi, cn);
          } else {
            run[0] = fabsf(run[0]);
            run[1] = fabsf(run[1]);
#pragma unroll 1
            for (;;) {
              const int hi = window_frame(s, c, phi, begin, nvalid, lane);
              if (hi >= end) break;
              encode<false>(e, s, c, begin, hi, lane);
              run[0] *= phi[0];
              run[1] *= phi[1];
              scan(den, e, run, lane);
              begin = hi;
            }
          }
          encode<WHOLE>(e, s, c, begin, end, lane);
          run[0] *= phi[0];
          run[1] *= phi[1];
          scan(den, e, run, lane);
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int t = 8 * j + q2 + x;
              const float l = __shfl_sync(0xffffffffu, l2, tile * 16 + t), dl = __shfl_sync(0xffffffffu, delta, tile * 16 + t);
#pragma unroll
              for (int i = x; i < 4; i += 2) {
                const bool on = in_window<WHOLE>(t, begin, end);
                const float dec = on ? ex2_approx(s[j][i] - l) : 0.f;
                r[j][i] = WHOLE || on ? dec * rcp_approx(den[j][i]) : 0.f;
                rp[j][i] = r[j][i] * pv[j][i];
                ds[j][i] = dec * (pv[j][i] - dl);  // decode part
              }
            }
        }
        Split ep, rs;
        split_tile(ep, e[0], e[1]);
        split_tile(rs, r[0], r[1]);
        uint32_t vf[2][4], dt[4][2];
        load_rows(vf, ks + STAGE, lane);
        load_cols(dt, ks + 2 * STAGE, lane);
        {
          // X = G V^T + R (A masked)^T
          float x[2][4], a[2][4];
          zero(x);
          zero(a);
          {
            uint32_t df[2][4];
            load_rows(df, ks + 2 * STAGE, lane);
#pragma unroll
            for (int k2 = 0; k2 < 2; ++k2) {
              uint32_t va[4];
              as_rows(va, vf, k2);
              mma(a[0], va, df[0][2 * k2], df[0][2 * k2 + 1]);
              mma(a[1], va, df[1][2 * k2], df[1][2 * k2 + 1]);
            }
          }
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) a[j][i] = 8 * j + q2 + (i & 1) >= g + (i >> 1) * 8 ? a[j][i] : 0.f;  // row tau, column t
          Split ap;
          split_tile(ap, a[0], a[1]);  // blocks (tau 0-7 | 8-15, t 0-7), (tau 0-7 | 8-15, t 8-15)
          mma_split(x[0], rs, col<0>(ap));
          mma_split(x[1], rs, col<1>(ap));
#pragma unroll
          for (int k2 = 0; k2 < 2; ++k2) {
            Split gp;
            split_tile(gp, gr[2 * k2], gr[2 * k2 + 1]);
            mma_exact(x[0], gp, vf[0][2 * k2], vf[0][2 * k2 + 1]);
            mma_exact(x[1], gp, vf[1][2 * k2], vf[1][2 * k2 + 1]);
          }
          // encoder part: C + sum of R p from the token on
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float behind = cc[i];
#pragma unroll
            for (int j = 1; j >= 0; --j) {
              float suf = rp[j][2 * i] + rp[j][2 * i + 1];
              float t = __shfl_down_sync(0xffffffffu, suf, 1, 4);
              if (q <= 2) suf += t;
              t = __shfl_down_sync(0xffffffffu, suf, 2, 4);
              if (q <= 1) suf += t;
              const float later = __shfl_down_sync(0xffffffffu, suf, 1, 4), total = __shfl_sync(0xffffffffu, suf, 0, 4);
              const float from1 = (q <= 2 ? behind + later : behind) + rp[j][2 * i + 1], from0 = from1 + rp[j][2 * i];
              ds[j][2 * i] = fmaf(e[j][2 * i], x[j][2 * i] - from0, ds[j][2 * i]);
              ds[j][2 * i + 1] = fmaf(e[j][2 * i + 1], x[j][2 * i + 1] - from1, ds[j][2 * i + 1]);
              behind += total;
            }
            cc[i] = behind;
          }
        }
        Split et;
        transpose_tile(et, ep);
        float out[4][4];
        zero(out);
        {
          // dV = E^T G + (E^T R masked) dY
          float w[2][4];
          zero(w);
          Split rt;
          transpose_tile(rt, rs);
          mma_split(w[0], et, col<0>(rt));
          mma_split(w[1], et, col<1>(rt));
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) w[j][i] = 8 * j + q2 + (i & 1) >= g + (i >> 1) * 8 ? w[j][i] : 0.f;
          Split wp;
          split_tile(wp, w[0], w[1]);
#pragma unroll
          for (int n = 0; n < 4; ++n) mma_exact(out[n], wp, dt[n][0], dt[n][1]);
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_split(out[n], et, as_col(gr[n]));
        float* dst = part + (warp * BT + tile * 16 + g) * LDP + q2;
#pragma unroll
        for (int n = 0; n < 4; ++n) put_rows(dst + 8 * n, out[n], !WHOLE && end < nvalid);
        // G += R dY, then into the frame before the window
#pragma unroll
        for (int n = 0; n < 4; ++n) add_product(gr[n], rs, dt[n][0], dt[n][1]);
        rescale(gr, phi);
        cc[0] *= phi[0];
        cc[1] *= phi[1];
        // dK = dS^T Q, dQ += dS K
        Split dsp, dst_t;
        split_tile(dsp, ds[0], ds[1]);
        transpose_tile(dst_t, dsp);
        {
          uint32_t qf[4][2];
          load_cols(qf, qs + m0 * LD, lane);
          zero(out);
#pragma unroll
          for (int n = 0; n < 4; ++n) mma_exact(out[n], dst_t, qf[n][0], qf[n][1]);
        }
        dst += nw * BT * LDP;
#pragma unroll
        for (int n = 0; n < 4; ++n) put_rows(dst + 8 * n, out[n], !WHOLE && end < nvalid);
        {
          uint32_t kt[4][2];
          load_cols(kt, ks, lane);
#pragma unroll
          for (int n = 0; n < 4; ++n) add_product(dq[n], dsp, kt[n][0], kt[n][1]);
        }
        return begin;
      };
      if (!signbit(p.stat_d[so])) {
        window(std::true_type(), nvalid);
      } else {  // (the tile was taken in several windows: from the last to the first)
#pragma unroll 1
        for (int end = nvalid; end > 0;) end = window(std::false_type(), end);
      }
    }
    __syncthreads();
    // rows of dV and dK: sums over the warps; thread = (tensor, token, 8 columns)
    for (int i = threadIdx.x; i < 2 * BT * 4; i += blockDim.x) {
      const int which = i >> 7, t = (i >> 2) & (BT - 1), col = (i & 3) * 8, D = which ? p.Dk : p.Dv;
      if (t0 + t >= tend || col >= D) continue;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int w = 0; w < nw; ++w) {
        const float4* src = reinterpret_cast<const float4*>(part + ((which * nw + w) * BT + t) * LDP + col);
        const float4 x = src[0], z = src[1];
        acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
        acc[4] += z.x; acc[5] += z.y; acc[6] += z.z; acc[7] += z.w;
      }
      float check = 0.f;
      const float f = which ? p.scale : 1.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[j] *= f;
        check = fmaf(acc[j], 0.f, check);
      }
      ok = ok && check == 0.f;
      *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(which ? p.dk : p.dv) + (((int64_t)b * p.N + t0 + t) * p.H + h) * D + col) =
          make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
    }
  }
  float* const dst = p.dq_part + ((((int64_t)b * p.nseg + seg) * p.H + h) * p.M + m0 + g) * p.Dk;
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (8 * n + q2 < p.Dk) {
        const float x = dq[n][2 * i] * p.scale, z = dq[n][2 * i + 1] * p.scale;
        ok = ok && fmaf(x, 0.f, z * 0.f) == 0.f;
        *reinterpret_cast<float2*>(dst + (int64_t)8 * i * p.Dk + 8 * n + q2) = make_float2(x, z);
      }
  const int bad = __syncthreads_or(!ok);
  if (threadIdx.x == 0) p.gate[(gridDim.x + lane_id) * p.nseg + seg] = bad;
}

// dq[i] = sum of the partials in fixed order; block 0 also gathers the CTAs' words into the word of the call
__global__ void __launch_bounds__(256) narrow_mma_sum_kernel(const float* part, int64_t n, int count, void* out, int out_dtype,
                                                             const int* words, int nwords, int* gate) {
  pdl_begin();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < n) {
    float acc = 0.f;
    for (int s = 0; s < count; ++s) acc += part[(int64_t)s * n + i];
    store1(out, out_dtype, i, acc);
  }
  if (blockIdx.x == 0) {
    int bad = 0;
    for (int w = threadIdx.x; w < nwords; w += 256) bad |= words[w];
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) *gate = bad;
  }
}

template <typename Kern>
int launch(Kern kern, const char* name, const NarrowMmaParams& p, int nseg_grid, size_t smem, cudaStream_t stream) {
  LaunchTimer timer(name, stream);
  FLARE_CUDA_CHECK(allow_smem(kern));
  FLARE_CUDA_CHECK(launch_pdl(kern, dim3(p.B * p.H, nseg_grid), dim3(p.M * 2), smem, stream, p));
  return FLARE_OK;
}

int launch_state(const NarrowMmaParams& p, cudaStream_t stream) {
  const size_t smem = 4 * STAGE * 2;
  return p.M <= 64 ? launch(narrow_mma_forward_kernel<128, false>, "narrow_mma_forward_kernel (state only)", p, p.nseg - 1, smem, stream)
                   : launch(narrow_mma_forward_kernel<256, false>, "narrow_mma_forward_kernel (state only)", p, p.nseg - 1, smem, stream);
}

bool shape_ok(const flare_fwd_args_t& f) {
  return f.path == FLARE_PATH_AUTO && f.dtype == FLARE_BF16 && f.variant == FLARE_SOFTMAX && f.B > 0 && f.N > 0 &&
         narrow_shape(f.M, f.Dk, f.Dv, f.block_size, f.q_dec != nullptr || f.k_dec != nullptr) && f.state_in.u == nullptr &&
         f.keep == nullptr && f.lengths == nullptr;
}

void fill(NarrowMmaParams& p, const flare_fwd_args_t& f) {
  memset(&p, 0, sizeof(p));
  p.q = f.q; p.k = f.k; p.v = f.v;
  p.B = f.B; p.N = f.N; p.H = f.H; p.M = f.M; p.Dk = f.Dk; p.Dv = f.Dv;
  p.q_stride_h = f.q_stride_h; p.q_stride_m = f.q_stride_m;
  p.k_stride_b = f.k_stride_b; p.k_stride_n = f.k_stride_n; p.k_stride_h = f.k_stride_h;
  p.v_stride_b = f.v_stride_b; p.v_stride_n = f.v_stride_n; p.v_stride_h = f.v_stride_h;
  p.scale = f.scale;
}

struct Plan {
  int nseg, seg_len, ntiles;
  size_t off_words, off_m, off_d, off_u, off_b, off_c, off_start, off_sc, off_sd, off_p, off_l2, off_delta, off_dq, total;
};
Plan plan(const flare_fwd_args_t& f) {
  Plan pl;
  const int64_t lanes = (int64_t)f.B * f.H;
  narrow_mma_segments(lanes, f.N, f.M, true, kNarrowMmaSegments, &pl.nseg, &pl.seg_len);
  pl.ntiles = (f.N + 15) / 16;
  size_t off = 0;
  auto take = [&](size_t words) {
    const size_t o = off;
    off += align_up(words * 4, 256);
    return o;
  };
  const size_t ls = (size_t)lanes * pl.nseg, lt = (size_t)lanes * pl.ntiles;
  pl.off_words = take(2 * ls);
  pl.off_m = take(ls * f.M);
  pl.off_d = take(ls * f.M);
  pl.off_u = take(ls * f.M * f.Dv);
  pl.off_b = take(ls * f.M * f.Dv);
  pl.off_c = take(ls * f.M);
  pl.off_start = take(ls * f.M);
  pl.off_sc = take(lt * f.M);
  pl.off_sd = take(lt * f.M);
  pl.off_p = take(lt * f.M * 16);
  pl.off_l2 = take(lt * 16);
  pl.off_delta = take(lt * 16);
  pl.off_dq = take((size_t)f.B * pl.nseg * f.H * f.M * f.Dk);
  pl.total = off;
  return pl;
}

}  // namespace

bool narrow_mma_forward_supported(const flare_fwd_args_t* a) {
  return shape_ok(*a) && a->mask == nullptr && a->y != nullptr && a->state_out.u == nullptr && a->lse_dec == nullptr && a->lse_enc == nullptr;
}

bool narrow_mma_backward_supported(const flare_bwd_args_t& a) {
  const bool span = a.carry_b || a.carry_c || a.carry_rho || a.span_b0 || a.span_c0 || a.span_gam || a.span_rho_first || a.phase != 0;
  // (dQ in fp32: nothing would hide how the tensor cores add, see above)
  return shape_ok(a.fwd) && a.dq_dtype != FLARE_F32 && !span && (reinterpret_cast<uintptr_t>(a.dy) & 15u) == 0 && a.dy_stride_b % 8 == 0 &&
         a.dy_stride_n % 8 == 0 && a.dy_stride_h % 8 == 0;
}

// As many segments as fill the SMs with 16 (backward: 12) warps, of 64 tokens at least; a second pass over all but one of them
// pays from two segments on because a CTA alone leaves its SM mostly idle.
void narrow_mma_segments(int64_t lanes, int N, int M, bool backward, int64_t room, int* nseg_out, int* seg_len_out) {
  int64_t n = (backward ? 12LL : 16LL) * sm_count() / (lanes * (M / 16));
  if (n > N / 64) n = N / 64;
  if (n > kNarrowMmaSegments) n = kNarrowMmaSegments;
  if (n > room) n = room;
  if (n < 1) n = 1;
  const int len = (int)(((N + n - 1) / n + BT - 1) / BT * BT);
  *seg_len_out = len;
  *nseg_out = (N + len - 1) / len;
}

int narrow_mma_forward(const flare_fwd_args_t& f, float* seg_m, float* seg_d, float* seg_u, int nseg, int seg_len, int* gate,
                       cudaStream_t stream) {
  NarrowMmaParams p;
  fill(p, f);
  p.y = f.y;
  p.y_stride_b = f.y_stride_b; p.y_stride_n = f.y_stride_n; p.y_stride_h = f.y_stride_h;
  p.seg_m = seg_m; p.seg_d = seg_d; p.seg_u = seg_u;
  p.nseg = nseg; p.seg_len = seg_len;
  p.gate = gate; p.gate_stride = nseg;
  if (nseg > 1) {
    const int rc = launch_state(p, stream);
    if (rc != FLARE_OK) return rc;
  }
  const size_t smem = 4 * STAGE * 2 + (size_t)(f.M / 16) * BT * (LDP + 2) * 4;
  return f.M <= 64 ? launch(narrow_mma_forward_kernel<128, true>, "narrow_mma_forward_kernel", p, nseg, smem, stream)
                   : launch(narrow_mma_forward_kernel<256, true>, "narrow_mma_forward_kernel", p, nseg, smem, stream);
}

size_t narrow_mma_backward_bytes(const flare_bwd_args_t& a) { return plan(a.fwd).total; }

int narrow_mma_backward(const flare_bwd_args_t& a, char* ws, int* gate, cudaStream_t stream) {
  const flare_fwd_args_t& f = a.fwd;
  const Plan pl = plan(f);
  auto at = [&](size_t off) { return reinterpret_cast<float*>(ws + off); };
  NarrowMmaParams p;
  fill(p, f);
  p.dy = a.dy;
  p.dy_stride_b = a.dy_stride_b; p.dy_stride_n = a.dy_stride_n; p.dy_stride_h = a.dy_stride_h;
  p.seg_len = pl.seg_len; p.nseg = pl.nseg; p.ntiles = pl.ntiles;
  p.seg_m = at(pl.off_m); p.seg_d = at(pl.off_d); p.seg_u = at(pl.off_u);
  p.seg_b = at(pl.off_b); p.seg_c = at(pl.off_c); p.start_c = at(pl.off_start);
  p.stat_c = at(pl.off_sc); p.stat_d = at(pl.off_sd); p.p = reinterpret_cast<float4*>(ws + pl.off_p);
  p.tok_l2 = at(pl.off_l2); p.tok_delta = at(pl.off_delta); p.dq_part = at(pl.off_dq);
  p.gate = reinterpret_cast<int*>(ws + pl.off_words);
  p.dk = a.dk; p.dv = a.dv;
  const int nw = f.M / 16;
  int rc;
  if (pl.nseg > 1) {
    rc = launch_state(p, stream);
    if (rc != FLARE_OK) return rc;
  }
  const size_t smem1 = 6 * STAGE * 2 + (size_t)6 * nw * BT * 4;
  rc = f.M <= 64 ? launch(narrow_mma_replay_kernel<128>, "narrow_mma_replay_kernel", p, pl.nseg, smem1, stream)
                 : launch(narrow_mma_replay_kernel<256>, "narrow_mma_replay_kernel", p, pl.nseg, smem1, stream);
  if (rc != FLARE_OK) return rc;
  const size_t smem2 = 6 * STAGE * 2 + (size_t)2 * nw * BT * LDP * 4 + (size_t)f.M * LD * 2;
  rc = f.M <= 64 ? launch(narrow_mma_reverse_kernel<128>, "narrow_mma_reverse_kernel", p, pl.nseg, smem2, stream)
                 : launch(narrow_mma_reverse_kernel<256>, "narrow_mma_reverse_kernel", p, pl.nseg, smem2, stream);
  if (rc != FLARE_OK) return rc;
  const int64_t n = (int64_t)f.H * f.M * f.Dk;
  LaunchTimer timer("narrow_mma_sum_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(narrow_mma_sum_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, p.dq_part, n,
                              f.B * pl.nseg, a.dq, a.dq_dtype, p.gate, (int)(2 * (int64_t)f.B * f.H * pl.nseg), gate));
  return FLARE_OK;
}

}  // namespace flare
