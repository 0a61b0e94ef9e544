// Exact (fp32, CUDA-core) forward walk, backward replay and reverse walk for narrow heads: Dk, Dv <= 32, M <= 128 latents,
// token-causal read-out, shared decode weights; softmax or stablemax encoder.
//
// The general kernels (walk_exact.cu, bwd_exact.cu) spread the value columns over the 32 lanes of a warp and the latents
// over eight warps.  At 32 columns a lane then holds one column of M / 8 latents, every product over the columns is a
// reduction over all 32 lanes and three broadcast loads feed two FMAs.  Here a warp owns 32 latents and all 32 columns:
// lane = (group of 8 latents, group of 4 columns), 32 state entries per thread.  A product over the columns is four FMAs
// and 7 shuffles for 8 latents (its result for latent 32 w + lane lands in that lane), a sum over the latents eight FMAs
// and 3 shuffles for 4 columns.  The per-latent statistics run with one latent per lane.  The latents of a warp are
// touched by no other warp, so only the decode softmax and the cross-latent sums need CTA barriers.
// Bound by the latency and issue of the fp32 passes; one CTA (M / 32 warps) per (lane, segment), segments so short that
// about twelve warps per SM are in flight.  bf16 softmax calls run on the tensor cores at the same precision (narrow_mma.cu);
// these kernels serve the rest (fp32, fp16, stablemax, states, masks) and stand by behind those.  B200: training step B=8 N=2048 H=16 M=64 D=32 4007 us with the general kernels,
// 1823 us with these.
#include "narrow_exact.cuh"

#include "walk_device.cuh"

namespace flare {

namespace {

constexpr int BT = 16;  // tokens per tile
constexpr int W = 32;   // columns of a staged row (zero beyond the head width)

// rows [t0, t0 + BT) as fp32, columns beyond D and rows from t_end on are zero
__device__ __forceinline__ void stage_rows(float* dst, const void* src, int dtype, int64_t off, int64_t stride_n, int t0,
                                           int t_end, int D) {
  for (int idx = threadIdx.x; idx < BT * (W / 8); idx += blockDim.x) {
    const int t = idx >> 2, c = (idx & 3) * 8;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t0 + t < t_end && c < D) load8(src, dtype, off + (int64_t)(t0 + t) * stride_n + c, x);
    *reinterpret_cast<float4*>(dst + t * W + c) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(dst + t * W + c + 4) = make_float4(x[4], x[5], x[6], x[7]);
  }
}

__device__ __forceinline__ void load8s(const float* p, float (&x)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
// (zeros for a thread whose latents lie beyond M, so that a non-finite value does not meet its zero weights)
__device__ __forceinline__ void load4s(const float* p, float (&x)[4], bool on) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  x[0] = on ? a.x : 0.f; x[1] = on ? a.y : 0.f; x[2] = on ? a.z : 0.f; x[3] = on ? a.w : 0.f;
}

// Sum of v[i] over the 8 lanes that differ in their low three bits; lane l keeps the total of v[l & 7].
__device__ __forceinline__ float reduce_columns(float (&v)[8], int lane) {
#pragma unroll
  for (int s = 4; s >= 1; s >>= 1) {
    const bool upper = (lane & s) != 0;
#pragma unroll
    for (int k = 0; k < s; ++k) {
      const float send = upper ? v[k] : v[k + s], keep = upper ? v[k + s] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
  return v[0];
}
// Sum of v[j] over the 4 lanes that differ in bits 3 and 4; lane l keeps the total of v[l >> 3].
__device__ __forceinline__ float reduce_latents(float (&v)[4], int lane) {
#pragma unroll
  for (int s = 2; s >= 1; s >>= 1) {
    const bool upper = (lane & (s * 8)) != 0;
#pragma unroll
    for (int k = 0; k < s; ++k) {
      const float send = upper ? v[k] : v[k + s], keep = upper ? v[k + s] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, s * 8);
    }
  }
  return v[0];
}

// scores of TS tokens for this thread's latent (its bank row in registers)
template <int TS>
__device__ __forceinline__ void score_rows(float (&s)[TS], const float* ks, const float (&q)[W], float scale) {
#pragma unroll
  for (int t = 0; t < TS; ++t) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int c = 0; c < W; c += 4) {
      const float4 x = *reinterpret_cast<const float4*>(ks + t * W + c);
      a0 = fmaf(q[c], x.x, a0);
      a1 = fmaf(q[c + 1], x.y, a1);
      a2 = fmaf(q[c + 2], x.z, a2);
      a3 = fmaf(q[c + 3], x.w, a3);
    }
    s[t] = ((a0 + a1) + (a2 + a3)) * scale;
  }
}

// Maximum of v[t] over the lanes of the warp; lane l keeps that of token l % TS (16 shuffles for 16 tokens).
template <int TS>
__device__ __forceinline__ float reduce_max(float (&v)[TS], int lane) {
#pragma unroll
  for (int s = TS / 2; s >= 1; s >>= 1) {
    const bool upper = (lane & s) != 0;
#pragma unroll
    for (int k = 0; k < s; ++k) {
      const float send = upper ? v[k] : v[k + s], keep = upper ? v[k + s] : v[k];
      v[k] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, send, s));
    }
  }
  float r = v[0];
#pragma unroll
  for (int o = TS; o < 32; o <<= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

// Decode softmax of TS tokens over all latents: a[t] = weight of this thread's latent.  red: [2][nw] rows of BT floats, of which
// these tokens have their own.  Contains two CTA barriers.
template <int TS>
__device__ __forceinline__ void decode_weights(float (&a)[TS], const float (&s)[TS], bool live, float* red, float* lse, int t0,
                                               int t_end, const int* valid) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int t = 0; t < TS; ++t) a[t] = live ? s[t] : kNegInf;
  const float mx = reduce_max<TS>(a, lane);
  if (lane < TS) red[warp * BT + lane] = mx;
  __syncthreads();
  float e[TS];
#pragma unroll
  for (int t = 0; t < TS; ++t) {
    float m = red[t];
    for (int w = 1; w < nw; ++w) m = fmaxf(m, red[w * BT + t]);
    a[t] = live ? __expf(s[t] - m) : 0.f;
    e[t] = a[t];
  }
  walk::warp_reduce_scatter<TS>(e, lane);
  float* sums = red + nw * BT;
  if (lane < TS) sums[warp * BT + lane] = e[0];
  __syncthreads();
#pragma unroll
  for (int t = 0; t < TS; ++t) {
    float sum = sums[t];
    for (int w = 1; w < nw; ++w) sum += sums[w * BT + t];
    a[t] *= 1.0f / sum;
  }
  if (lse != nullptr && threadIdx.x < TS && t0 + (int)threadIdx.x < t_end) {
    const int t = threadIdx.x;
    float m = red[t], sum = sums[t];
    for (int w = 1; w < nw; ++w) {
      m = fmaxf(m, red[w * BT + t]);
      sum += sums[w * BT + t];
    }
    lse[t] = valid[t] ? m + logf(sum) : 0.f;
  }
}

__device__ __forceinline__ void load_bank_row(float (&q)[W], const void* src, int dtype, int64_t off, int Dk, bool live) {
#pragma unroll
  for (int c = 0; c < W; c += 8) {
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (live && c < Dk) load8(src, dtype, off + c, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) q[c + j] = x[j];
  }
}

// U *= gam, skipped while no running maximum of the warp's latents has grown (multiplying by one)
__device__ __forceinline__ void decay_state(float (&U)[8][4], const float* gam_row) {
  float gam[8];
  load8s(gam_row, gam);
  bool grown = false;
#pragma unroll
  for (int i = 0; i < 8; ++i) grown |= gam[i] != 1.f;
  if (__any_sync(0xffffffffu, grown)) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) U[i][j] *= gam[i];
  }
}

// ---------------------------------------------------------------------------------------------
// forward walk
// ---------------------------------------------------------------------------------------------
// Scores and statistics are taken for eight tokens at a time and the state is walked without unrolling.  Unrolled for the 16 tokens
// of a tile the code was most of the time of a CTA that walks two tiles (half of the warps' cycles waited for an instruction),
// and held more registers: B200, fp32 B=1 N=256 H=8 M=64 D=32 47.2 -> 43.1 us, B=8 N=4096 H=16 1256 -> 1124 us, fp16 B=4
// N=2048 H=16 M=128 637 -> 568 us.  (Four tokens at a time: 44.3, 1148, 579.)
constexpr int TS = 8;
template <bool STABLE>
__global__ void __launch_bounds__(128, 4) walk_narrow_kernel(const WalkParams p) {
  pdl_begin();
  extern __shared__ __align__(16) float smem_raw[];
  const int nw = blockDim.x >> 5, ms = nw * 32;
  float* ks = smem_raw;
  float* vs = ks + BT * W;
  float* s_s = vs + BT * W;      // eta
  float* g_s = s_s + BT * ms;    // decay of the state
  float* w_s = g_s + BT * ms;    // read-out weight
  float* ypart = w_s + BT * ms;  // [nw][BT][W]
  float* red = ypart + nw * BT * W;  // [2][nw][BT]
  int* valid = reinterpret_cast<int*>(red + 2 * nw * BT);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, seg = blockIdx.y;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int M = p.M;
  const int seg_begin = seg * p.seg_len, seg_end = min(p.N, seg_begin + p.seg_len);
  const int m = warp * 32 + lane;                       // this thread's latent in the statistics
  const int mb = warp * 32 + (lane >> 3) * 8;           // first of its 8 latents in the state
  const int cb = (lane & 7) * 4;                        // first of its 4 columns
  const bool live = m < M;

  float q[W];
  load_bank_row(q, p.q, p.dtype, (int64_t)h * p.q_stride_h + (int64_t)m * p.q_stride_m, p.Dk, live);
  const int64_t sidx = (int64_t)lane_id * p.in_lane_stride + (int64_t)seg * p.in_seg_stride;
  float mr = STABLE ? 0.f : kNegInf, dr = 0.f;
  if (live && p.in_m != nullptr) {
    mr = p.in_m[sidx * M + m];
    dr = p.in_d[sidx * M + m];
  }
  float U[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      U[i][j] = (p.in_u != nullptr && mb + i < M && cb + j < p.Dv) ? p.in_u[(sidx * M + mb + i) * p.Dv + cb + j] : 0.f;

  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t y_off = (int64_t)b * p.y_stride_b + (int64_t)h * p.y_stride_h;
  const bool write_y = p.write_y != 0;
  for (int t0 = seg_begin; t0 < seg_end; t0 += BT) {
    __syncthreads();
    if (tid < BT) {
      const int t = t0 + tid;
      valid[tid] = t < seg_end && (p.mask == nullptr || p.mask[(int64_t)b * p.N + t] != 0);
    }
    stage_rows(ks, p.k, p.dtype, k_off, p.k_stride_n, t0, seg_end, p.Dk);
    stage_rows(vs, p.v, p.dtype, v_off, p.v_stride_n, t0, seg_end, p.Dv);
    __syncthreads();
#pragma unroll 1
    for (int t1 = 0; t1 < BT; t1 += TS) {
      float sv[TS], aw[TS];
      score_rows<TS>(sv, ks + t1 * W, q, p.scale);
      if (write_y)
        decode_weights<TS>(aw, sv, live, red + t1, p.lse_dec != nullptr ? p.lse_dec + (int64_t)lane_id * p.N + t0 + t1 : nullptr,
                           t0 + t1, seg_end, valid + t1);
      // running statistics of this thread's latent
#pragma unroll
      for (int t = 0; t < TS; ++t) {
        const bool on = valid[t1 + t] != 0;
        float gam = 1.f, eta;
        if constexpr (STABLE) {
          eta = on ? stablemax_sigma(sv[t], p.power) : 0.f;
          dr += eta;
        } else {
          const float mn = on ? fmaxf(mr, sv[t]) : mr;
          if (on) gam = (mr == kNegInf) ? 0.f : __expf(mr - mn);
          eta = on ? __expf(sv[t] - mn) : 0.f;
          dr = dr * gam + eta;
          mr = mn;
        }
        if (write_y) w_s[(t1 + t) * ms + m] = aw[t] * (1.0f / (dr > 0.f ? dr : 1.f));
        if constexpr (!STABLE) g_s[(t1 + t) * ms + m] = gam;
        s_s[(t1 + t) * ms + m] = eta;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < BT; ++t) {
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      if (valid[t]) {
        float v[4], eta[8];
        load4s(vs + t * W + cb, v, mb < M);
        load8s(s_s + t * ms + mb, eta);
        if constexpr (!STABLE) decay_state(U, g_s + t * ms + mb);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) U[i][j] = fmaf(eta[i], v[j], U[i][j]);
        if (write_y) {
          float w[8];
          load8s(w_s + t * ms + mb, w);
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = fmaf(w[i], U[i][j], y[j]);
        }
      }
      if (write_y) ypart[(warp * BT + t) * W + cb + (lane >> 3)] = reduce_latents(y, lane);
    }
    if (write_y) {
      __syncthreads();
      for (int idx = tid; idx < BT * (W / 4); idx += blockDim.x) {
        const int t = idx >> 3, c = (idx & 7) * 4;
        if (t0 + t >= seg_end || c >= p.Dv) continue;
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        for (int w = 0; w < nw; ++w) {
          const float4 x = *reinterpret_cast<const float4*>(ypart + (w * BT + t) * W + c);
          a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
        }
        store4(p.y, p.dtype, y_off + (int64_t)(t0 + t) * p.y_stride_n + c, a[0], a[1], a[2], a[3]);
      }
    }
  }
  if (p.out_u != nullptr && (p.out_mode == 1 || (p.out_mode == 2 && seg == p.nseg_total - 1))) {
    const int64_t so = (int64_t)lane_id * p.out_lane_stride + (int64_t)seg * p.out_seg_stride;
    if (live) {
      p.out_m[so * M + m] = mr;
      p.out_d[so * M + m] = dr;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)  // (the caller's state need not be 16-byte aligned)
        if (mb + i < M && cb + j < p.Dv) p.out_u[(so * M + mb + i) * p.Dv + cb + j] = U[i][j];
  }
}

// ---------------------------------------------------------------------------------------------
// backward, replay: e, g, p of every (token, latent) and the carries of the segment for a zero carry-in,
//   b0[m, :] = sum_t X dY_t,  c0[m] = sum_t X p,   X[t, m] = g prod_{tau = a+1 .. t} (1 - e[tau, m])
// ---------------------------------------------------------------------------------------------
template <bool STABLE>
__global__ void __launch_bounds__(128, 3) narrow_replay_kernel(const NarrowBwdParams p) {
  pdl_begin();
  if (p.gate != nullptr && *p.gate == 0) return;
  extern __shared__ __align__(16) float smem_raw[];
  const int nw = blockDim.x >> 5, ms = nw * 32;
  float* ks = smem_raw;
  float* vs = ks + BT * W;
  float* dos = vs + BT * W;
  float* s_s = dos + BT * W;   // eta
  float* g_s = s_s + BT * ms;  // decay of the state
  float* x_s = g_s + BT * ms;  // carry weights
  float* r_s = x_s + BT * ms;  // 1 / denominator
  float* red = r_s + BT * ms;  // [2][nw][BT]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, seg = blockIdx.y;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int M = p.M, N = p.N;
  const int tbeg = seg * p.seg_len, tend = min(N, tbeg + p.seg_len);
  const int m = warp * 32 + lane, mb = warp * 32 + (lane >> 3) * 8, cb = (lane & 7) * 4;
  const bool live = m < M;
  const int64_t st = (int64_t)lane_id * p.nseg + seg;
  const bool carries = p.nseg > 1;

  float q[W];
  load_bank_row(q, p.q, p.dtype, (int64_t)h * p.q_stride_h + (int64_t)m * p.q_stride_m, p.Dk, live);
  float mr = STABLE ? 0.f : kNegInf, dr = 0.f, gp = 1.f, c0 = 0.f;
  if (live && p.in_m != nullptr) {
    mr = p.in_m[st * M + m];
    dr = p.in_d[st * M + m];
  }
  float U[8][4], b0[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      U[i][j] = (p.in_u != nullptr && mb + i < M && cb + j < p.Dv) ? p.in_u[(st * M + mb + i) * p.Dv + cb + j] : 0.f;
      b0[i][j] = 0.f;
    }
  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t dy_off = (int64_t)b * p.dy_stride_b + (int64_t)h * p.dy_stride_h;
  const int64_t row0 = (int64_t)lane_id * N;
  for (int t0 = tbeg; t0 < tend; t0 += BT) {
    const int nt = min(BT, tend - t0);
    __syncthreads();
    stage_rows(ks, p.k, p.dtype, k_off, p.k_stride_n, t0, tend, p.Dk);
    stage_rows(vs, p.v, p.dtype, v_off, p.v_stride_n, t0, tend, p.Dv);
    stage_rows(dos, p.dy, p.dtype, dy_off, p.dy_stride_n, t0, tend, p.Dv);
    __syncthreads();
    float sv[BT], aw[BT];
    score_rows<BT>(sv, ks, q, p.scale);
    decode_weights<BT>(aw, sv, live, red, nullptr, t0, tend, nullptr);
#pragma unroll
    for (int t = 0; t < BT; ++t) {
      if (t >= nt) break;
      const float sc = sv[t];
      float gam, eta;
      if constexpr (STABLE) {
        gam = 1.f;
        eta = stablemax_sigma(sc, p.power);
        dr += eta;
      } else {
        const float mn = fmaxf(mr, sc);
        gam = (mr == kNegInf) ? 0.f : __expf(mr - mn);
        eta = __expf(sc - mn);
        dr = dr * gam + eta;
        mr = mn;
      }
      const float rinv = 1.0f / dr, e = eta * rinv;
      if (t0 + t != tbeg) gp *= 1.0f - e;  // the segment's first token carries no decay
      g_s[t * ms + m] = gam;
      s_s[t * ms + m] = eta;
      r_s[t * ms + m] = rinv;
      x_s[t * ms + m] = aw[t] * gp;
      if (live) {
        const int64_t o = (row0 + t0 + t) * M + m;
        p.E[o] = e;
        p.G[o] = aw[t];
        if constexpr (STABLE) p.W2[o] = e * stablemax_slope_ratio(sc, p.power);
      }
    }
    __syncwarp();
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      float v[4], dy[4], eta[8], pp[8];
      load4s(vs + t * W + cb, v, mb < M);
      load4s(dos + t * W + cb, dy, mb < M);
      load8s(s_s + t * ms + mb, eta);
      if constexpr (!STABLE) decay_state(U, g_s + t * ms + mb);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        pp[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          U[i][j] = fmaf(eta[i], v[j], U[i][j]);
          pp[i] = fmaf(U[i][j], dy[j], pp[i]);
        }
      }
      const float pv = reduce_columns(pp, lane) * r_s[t * ms + m];
      if (live) p.P[(row0 + t0 + t) * M + m] = pv;
      if (carries) {
        float x[8];
        load8s(x_s + t * ms + mb, x);
        c0 = fmaf(x_s[t * ms + m], pv, c0);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) b0[i][j] = fmaf(x[i], dy[j], b0[i][j]);
      }
    }
  }
  if (carries) {
    if (live) {
      p.seg_c[st * M + m] = c0;
      p.seg_gam[st * M + m] = gp;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (mb + i < M && cb < p.Dv)
        *reinterpret_cast<float4*>(p.seg_b + (st * M + mb + i) * p.Dv + cb) = make_float4(b0[i][0], b0[i][1], b0[i][2], b0[i][3]);
  }
}

// ---------------------------------------------------------------------------------------------
// backward, reverse walk: dV, dK and this segment's part of dQ (the dS rows never leave the CTA)
// ---------------------------------------------------------------------------------------------
template <bool STABLE>
__global__ void __launch_bounds__(128, 4) narrow_reverse_kernel(const NarrowBwdParams p) {
  pdl_begin();
  if (p.gate != nullptr && *p.gate == 0) return;
  extern __shared__ __align__(16) float smem_raw[];
  const int nw = blockDim.x >> 5, ms = nw * 32;
  float* ks = smem_raw;
  float* vs = ks + BT * W;
  float* dos = vs + BT * W;
  float* e_s = dos + BT * W;
  float* rho_s = e_s + BT * ms;  // decay from the next token into this one
  float* g_s = rho_s + BT * ms;
  float* ds_s = g_s + BT * ms;     // p -> dS
  float* q_s = ds_s + BT * ms;     // [ms][W] latent bank
  float* dvpart = q_s + ms * W;    // [nw][BT][W]
  float* gps = dvpart + nw * BT * W;  // [nw][BT]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, seg = blockIdx.y;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int M = p.M, N = p.N;
  const int tbeg = seg * p.seg_len, tend = min(N, tbeg + p.seg_len);
  const int m = warp * 32 + lane, mb = warp * 32 + (lane >> 3) * 8, cb = (lane & 7) * 4;
  const bool live = m < M;
  const int64_t st = (int64_t)lane_id * p.nseg + seg;
  const int64_t row0 = (int64_t)lane_id * N;
  const bool carry_in = p.nseg > 1 && tend < N;
  {
    float q[W];
    load_bank_row(q, p.q, p.dtype, (int64_t)h * p.q_stride_h + (int64_t)m * p.q_stride_m, p.Dk, live);
#pragma unroll
    for (int c = 0; c < W; c += 4)
      *reinterpret_cast<float4*>(q_s + m * W + c) = make_float4(q[c], q[c + 1], q[c + 2], q[c + 3]);
  }
  float Bc[8][4], dq[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      Bc[i][j] = (carry_in && mb + i < M && cb + j < p.Dv) ? p.seg_b[(st * M + mb + i) * p.Dv + cb + j] : 0.f;
      dq[i][j] = 0.f;
    }
  float c = (carry_in && live) ? p.seg_c[st * M + m] : 0.f;
  // decay of the first step = 1 - e of the first token of the segment to the right
  float rho = (tend < N && live) ? 1.0f - p.E[(row0 + tend) * M + m] : 0.f;
  const int64_t k_off = (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h;
  const int64_t v_off = (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h;
  const int64_t dy_off = (int64_t)b * p.dy_stride_b + (int64_t)h * p.dy_stride_h;
  for (int t0 = tbeg + (tend - 1 - tbeg) / BT * BT; t0 >= tbeg; t0 -= BT) {
    const int nt = min(BT, tend - t0);
    __syncthreads();
    stage_rows(ks, p.k, p.dtype, k_off, p.k_stride_n, t0, tend, p.Dk);
    stage_rows(vs, p.v, p.dtype, v_off, p.v_stride_n, t0, tend, p.Dv);
    stage_rows(dos, p.dy, p.dtype, dy_off, p.dy_stride_n, t0, tend, p.Dv);
    // this thread's latent: e, g, p of the tile; tokens beyond the sequence stand for nothing
    {
      float gpr[BT];
#pragma unroll
      for (int t = BT - 1; t >= 0; --t) {
        const bool in = live && t < nt;
        const int64_t o = (row0 + t0 + t) * M + m;
        const float e = in ? p.E[o] : 0.f, g = in ? p.G[o] : 0.f, pv = in ? p.P[o] : 0.f;
        e_s[t * ms + m] = e;
        g_s[t * ms + m] = g;
        ds_s[t * ms + m] = pv;
        rho_s[t * ms + m] = rho;
        if (t < nt) rho = 1.0f - e;
        gpr[t] = g * pv;
      }
      walk::warp_reduce_scatter<BT>(gpr, lane);
      if (lane < BT) gps[warp * BT + lane] = gpr[0];
    }
    __syncthreads();
#pragma unroll 2
    for (int t = nt - 1; t >= 0; --t) {
      float dy[4], v[4], g[8], r[8], e[8];
      load4s(dos + t * W + cb, dy, mb < M);
      load4s(vs + t * W + cb, v, mb < M);
      load8s(g_s + t * ms + mb, g);
      load8s(rho_s + t * ms + mb, r);
      load8s(e_s + t * ms + mb, e);
      float bv[8], dv[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        bv[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          Bc[i][j] = fmaf(Bc[i][j], r[i], g[i] * dy[j]);
          bv[i] = fmaf(Bc[i][j], v[j], bv[i]);
          dv[j] = fmaf(e[i], Bc[i][j], dv[j]);
        }
      }
      const float bvm = reduce_columns(bv, lane);
      dvpart[(warp * BT + t) * W + cb + (lane >> 3)] = reduce_latents(dv, lane);
      float gp = 0.f;
      for (int w = 0; w < nw; ++w) gp += gps[w * BT + t];
      const float gm = g_s[t * ms + m], pm = ds_s[t * ms + m];
      c = gm * pm + rho_s[t * ms + m] * c;
      float w2 = e_s[t * ms + m];
      if constexpr (STABLE) w2 = live ? p.W2[(row0 + t0 + t) * M + m] : 0.f;
      ds_s[t * ms + m] = w2 * (bvm - c) + gm * (pm - gp);
    }
    __syncthreads();
    // dQ += dS^T K: this thread's 8 latents and 4 columns
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      float kk[4], d[8];
      load4s(ks + t * W + cb, kk, mb < M);
      load8s(ds_s + t * ms + mb, d);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dq[i][j] = fmaf(d[i], kk[j], dq[i][j]);
    }
    // dV and dK rows: thread = (token, 4 columns)
    for (int idx = tid; idx < nt * (W / 4); idx += blockDim.x) {
      const int t = idx >> 3, cc = (idx & 7) * 4;
      const int64_t row = ((int64_t)b * N + t0 + t) * p.H + h;
      if (cc < p.Dv) {
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        for (int w = 0; w < nw; ++w) {
          const float4 x = *reinterpret_cast<const float4*>(dvpart + (w * BT + t) * W + cc);
          a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
        }
        store4(p.dv, p.dtype, row * p.Dv + cc, a[0], a[1], a[2], a[3]);
      }
      if (cc < p.Dk) {
        float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int mm = 0; mm < M; mm += 4) {
          const float4 d = *reinterpret_cast<const float4*>(ds_s + t * ms + mm);
          const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 x = *reinterpret_cast<const float4*>(q_s + (mm + u) * W + cc);
            a[0] = fmaf(dd[u], x.x, a[0]);
            a[1] = fmaf(dd[u], x.y, a[1]);
            a[2] = fmaf(dd[u], x.z, a[2]);
            a[3] = fmaf(dd[u], x.w, a[3]);
          }
        }
        store4(p.dk, p.dtype, row * p.Dk + cc, a[0] * p.scale, a[1] * p.scale, a[2] * p.scale, a[3] * p.scale);
      }
    }
  }
  float* part = p.dq_part + (((int64_t)b * p.nseg + seg) * p.H + h) * M * p.Dk;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (mb + i < M && cb < p.Dk)
      *reinterpret_cast<float4*>(part + (int64_t)(mb + i) * p.Dk + cb) =
          make_float4(dq[i][0] * p.scale, dq[i][1] * p.scale, dq[i][2] * p.scale, dq[i][3] * p.scale);
}

template <typename Kern, typename P>
int launch(Kern kern, const char* name, const P& p, int nseg_grid, int floats, cudaStream_t stream) {
  LaunchTimer timer(name, stream);
  FLARE_CUDA_CHECK(allow_smem(kern));
  FLARE_CUDA_CHECK(launch_pdl(kern, dim3(p.B * p.H, nseg_grid), dim3(narrow_warps(p.M) * 32), floats * sizeof(float), stream, p));
  return FLARE_OK;
}

}  // namespace

int launch_walk_narrow(const WalkParams& p, int nseg_grid, cudaStream_t stream) {
  const int nw = narrow_warps(p.M), ms = nw * 32;
  const int floats = 2 * BT * W + 3 * BT * ms + nw * BT * W + 2 * nw * BT + BT;
  return launch(p.variant == FLARE_STABLEMAX ? walk_narrow_kernel<true> : walk_narrow_kernel<false>,
                "walk_exact_kernel (narrow heads)", p, nseg_grid, floats, stream);
}

int launch_narrow_replay(const NarrowBwdParams& p, cudaStream_t stream) {
  const int nw = narrow_warps(p.M), ms = nw * 32;
  const int floats = 3 * BT * W + 4 * BT * ms + 2 * nw * BT;
  return launch(p.variant == FLARE_STABLEMAX ? narrow_replay_kernel<true> : narrow_replay_kernel<false>,
                "bwd_replay_kernel (narrow heads)", p, p.nseg, floats, stream);
}

int launch_narrow_reverse(const NarrowBwdParams& p, cudaStream_t stream) {
  const int nw = narrow_warps(p.M), ms = nw * 32;
  const int floats = 3 * BT * W + 4 * BT * ms + ms * W + nw * BT * W + nw * BT;
  return launch(p.variant == FLARE_STABLEMAX ? narrow_reverse_kernel<true> : narrow_reverse_kernel<false>,
                "bwd_reverse_kernel (narrow heads)", p, p.nseg, floats, stream);
}

}  // namespace flare
