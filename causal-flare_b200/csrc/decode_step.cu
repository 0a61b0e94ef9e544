// One decode token per (batch, head) lane: HBM-bound in-place update of the fp32 latent state.
//
// Per lane the kernel reads and writes u [M, Dv] fp32 once (128-bit accesses, streaming cache hints so the
// shared latent bank Q stays resident in L2), plus m, d [M].  Phases inside a CTA (one CTA per lane):
//   0. issue the first batch of state loads so they are in flight while scores are computed (few lanes: all of them, the lane's
//      value columns shared by the CTAs of a cluster)
//   1. scores s[m] = scale <q_m, k>, 8 lanes per latent, 16-byte loads of Q, 3-step shuffle reduction
//   2. running max / denominator update per latent, decode softmax over the M latents (block reductions)
//   3. stream u: u' = gamma u + eta v,  y += (softmax / d') u'; thread-private y columns, reduced once
#include "decode_step.cuh"

#include "sm100_ptx.cuh"

namespace flare {

namespace {

constexpr int NT = 256;
constexpr int NW = NT / 32;

__device__ __forceinline__ float block_reduce(float v, float* red, bool is_max) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) r = is_max ? fmaxf(r, red[w]) : r + red[w];
  return r;
}

// scores of latents mb .. me - 1 against one token vector held in shared memory (fp32), AHEAD latent rows in flight per thread;
// SLICED: into the same place of every CTA of the cluster
template <int AHEAD, bool SLICED>
__device__ __forceinline__ void lane_scores(float* out, const float* tok, const void* lat, int dtype, int64_t lat_off,
                                            int64_t lat_stride_m, int mb, int me, int Dk, float scale, int slices) {
  const int grp = threadIdx.x >> 3, gl = threadIdx.x & 7;
  // (latents come in multiples of 16, so a warp's four rows are all there, or its part of a slice ends inside it)
  constexpr bool ALL_THERE = AHEAD == 1 && !SLICED;
  for (int m0 = mb; m0 + (grp & ~3) < me; m0 += AHEAD * (NT / 8)) {  // (whole warps: the shuffles below)
    float acc[AHEAD];
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) acc[a] = 0.f;
    for (int d0 = gl * 8; d0 < Dk; d0 += 64) {
      float qv[AHEAD][8];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a)
        load8(lat, dtype, lat_off + (int64_t)(ALL_THERE ? m0 + grp : min(m0 + a * (NT / 8) + grp, me - 1)) * lat_stride_m + d0, qv[a]);
#pragma unroll
      for (int a = 0; a < AHEAD; ++a)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[a] += qv[a][i] * tok[d0 + i];
    }
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) {
      acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], 4);
      acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], 2);
      acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], 1);
      const int m = m0 + a * (NT / 8) + grp;
      if (!ALL_THERE && m >= me) continue;
      if constexpr (SLICED) {
        // (one thread of the latent's eight for every CTA of the cluster: eight at most)
        if (gl < slices) sm100::st_cluster_f32(sm100::mapa_shared(sm100::smem_u32(out + m), gl), acc[a] * scale);
      } else if (gl == 0) {
        out[m] = acc[a] * scale;
      }
    }
  }
}

}  // namespace

// PRE: state vectors per thread issued before the score phase; UNR: state vectors in flight per thread in the
// streaming loop (0: PRE vectors are all there is); MINB: CTAs per SM the register budget is held to; AHEAD: latent rows in flight per
// thread in the scores
// SLICED: the lane's value columns are shared by the CTAs of a cluster (blockIdx.y).  Each computes the scores of its part of the
// latents and sends them to the others; the statistics are the business of all of them and written by the first.
template <int PRE, int UNR, int MINB, int AHEAD, bool SLICED>
__global__ void __launch_bounds__(NT, MINB) decode_step_kernel(const DecodeParams p) {
  extern __shared__ __align__(16) float smem[];
  const int lane_id = blockIdx.x;
  pdl_begin();
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int M = p.M, Dk = p.Dk, Dv = p.Dv;
  const int tid = threadIdx.x;
  const int dtype = p.dtype;
  const int slices = SLICED ? (int)gridDim.y : 1, slice = SLICED ? (int)blockIdx.y : 0;
  const int dv4 = Dv >> 2, cols = dv4 / slices;
  const int rows_per_pass = NT / cols;
  const int col4 = slice * cols + tid % cols, row0 = tid / cols;

  float* s_sc = smem;           // [M] encode scores -> eta
  float* a_sc = s_sc + M;       // [M] decode scores -> read-out weight
  float* gam = a_sc + M;        // [M]
  float* ktok = gam + M;        // [Dk]
  float* qtok = ktok + Dk;      // [Dk]
  float* vtok = qtok + Dk;      // [Dv]
  float* red = vtok + Dv;       // [NW]
  float4* ypart = reinterpret_cast<float4*>(red + NW);  // [NT]

  if (p.mask != nullptr && p.mask[b] == 0) {
    // masked lane: state untouched, y = 0
    if (slice == 0)
      for (int i = tid; i < Dv; i += NT) store1(p.y, dtype, (int64_t)lane_id * Dv + i, 0.f);
    return;
  }

  if constexpr (SLICED) sm100::cluster_arrive();  // (a CTA may be written to once it runs)
  // rows row0, row0 + rows_per_pass, ... of this thread's columns: NT * slices vectors apart, a constant for a whole lane
  float4* const u4 = reinterpret_cast<float4*>(p.u + (int64_t)lane_id * M * Dv) + (SLICED ? row0 * dv4 + col4 : tid);
  const int step = NT * slices;

  // phase 0: first state vectors in flight, and the statistics of this thread's first latent
  float4 pre[PRE];
#pragma unroll
  for (int i = 0; i < PRE; ++i) {
    const int r = row0 + i * rows_per_pass;
    pre[i] = r < M ? load_streaming(u4 + i * step) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float* gm = p.m + (int64_t)lane_id * M;
  float* gd = p.d + (int64_t)lane_id * M;
  float m_first = 0.f, d_first = 0.f;
  if (SLICED && tid < M) {
    m_first = gm[tid];
    d_first = gd[tid];
  }

  // token vectors -> smem fp32
  for (int i = tid; i < Dk; i += NT) {
    ktok[i] = load1(p.k, dtype, (int64_t)b * p.k_stride_b + (int64_t)h * p.k_stride_h + i);
    if (p.qd != nullptr) qtok[i] = load1(p.qd, dtype, (int64_t)b * p.qd_stride_b + (int64_t)h * p.qd_stride_h + i);
  }
  for (int i = tid; i < Dv; i += NT) vtok[i] = load1(p.v, dtype, (int64_t)b * p.v_stride_b + (int64_t)h * p.v_stride_h + i);
  __syncthreads();
  if constexpr (SLICED) sm100::cluster_wait();

  // phase 1: scores
  const int ms = SLICED ? (M + slices - 1) / slices : M, mb = slice * ms, me = min(M, mb + ms);
  lane_scores<AHEAD, SLICED>(s_sc, ktok, p.q, dtype, (int64_t)h * p.q_stride_h, p.q_stride_m, mb, me, Dk, p.scale, slices);
  const bool shared_w = p.qd == nullptr && p.kd == nullptr;
  if (!shared_w) {
    lane_scores<AHEAD, SLICED>(a_sc, p.qd ? qtok : ktok, p.kd ? p.kd : p.q, dtype,
                               p.kd ? (int64_t)h * p.kd_stride_h : (int64_t)h * p.q_stride_h, p.kd ? p.kd_stride_m : p.q_stride_m,
                               mb, me, Dk, p.scale, slices);
  }
  // (sliced: every CTA of the lane has all scores, and has read the statistics that the first one rewrites below)
  if constexpr (SLICED) sm100::cluster_sync_all();
  else __syncthreads();

  // phase 2: decode softmax over latents and per-latent statistics
  float amax = kNegInf;
  for (int m = tid; m < M; m += NT) amax = fmaxf(amax, shared_w ? s_sc[m] : a_sc[m]);
  amax = block_reduce(amax, red, true);
  float asum = 0.f;
  for (int m = tid; m < M; m += NT) {
    const float e = __expf((shared_w ? s_sc[m] : a_sc[m]) - amax);
    a_sc[m] = e;
    asum += e;
  }
  asum = block_reduce(asum, red, false);
  const float ainv = 1.0f / asum;
  for (int m = tid; m < M; m += NT) {
    const float s = s_sc[m];
    const float mo = SLICED ? m_first : gm[m], dold = SLICED ? d_first : gd[m];
    const float mn = fmaxf(mo, s);
    const float g = (mo == kNegInf) ? 0.f : __expf(mo - mn);
    const float eta = __expf(s - mn);
    const float dn = dold * g + eta;
    if (slice == 0) {
      gm[m] = mn;
      gd[m] = dn;
    }
    gam[m] = g;
    s_sc[m] = eta;
    a_sc[m] = a_sc[m] * ainv / (dn > 0.f ? dn : 1.f);
  }
  __syncthreads();

  // phase 3: stream the state
  const float4 v4 = reinterpret_cast<const float4*>(vtok)[col4];
  float4 yacc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto apply = [&](float4 x, int row, int at) {
    const float g = gam[row], e = s_sc[row], w = a_sc[row];
    x.x = x.x * g + e * v4.x;
    x.y = x.y * g + e * v4.y;
    x.z = x.z * g + e * v4.z;
    x.w = x.w * g + e * v4.w;
    __stcs(u4 + at, x);
    yacc.x += w * x.x;
    yacc.y += w * x.y;
    yacc.z += w * x.z;
    yacc.w += w * x.w;
  };
#pragma unroll
  for (int i = 0; i < PRE; ++i) {
    const int r = row0 + i * rows_per_pass;
    if (r < M) apply(pre[i], r, i * step);
  }
  if constexpr (UNR > 0) {
    int r = row0 + PRE * rows_per_pass, at = PRE * step;
    for (; r + (UNR - 1) * rows_per_pass < M; r += UNR * rows_per_pass, at += UNR * step) {
      float4 x[UNR];
#pragma unroll
      for (int i = 0; i < UNR; ++i) x[i] = load_streaming(u4 + at + i * step);
#pragma unroll
      for (int i = 0; i < UNR; ++i) apply(x[i], r + i * rows_per_pass, at + i * step);
    }
    if constexpr (MINB == 4) {  // what is left, together too (the registers of the others do not allow it, or the code costs more)
      float4 x[UNR - 1];
#pragma unroll
      for (int i = 0; i < UNR - 1; ++i)
        if (r + i * rows_per_pass < M) x[i] = load_streaming(u4 + at + i * step);
#pragma unroll
      for (int i = 0; i < UNR - 1; ++i)
        if (r + i * rows_per_pass < M) apply(x[i], r + i * rows_per_pass, at + i * step);
    } else {
      for (; r < M; r += rows_per_pass, at += step) apply(load_streaming(u4 + at), r, at);
    }
  }

  // reduce y over the row groups that share a column
  ypart[tid] = yacc;
  __syncthreads();
  if (tid < cols) {
    float4 acc = ypart[tid];
    for (int r = 1; r < rows_per_pass; ++r) {
      const float4 x = ypart[tid + r * cols];
      acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
    store4(p.y, p.dtype, (int64_t)lane_id * Dv + col4 * 4, acc.x, acc.y, acc.z, acc.w);
  }
}

bool decode_step_supported(int M, int Dk, int Dv) {
  const int dv4 = Dv / 4;
  if (dv4 > NT || (NT % dv4) != 0) return false;
  const size_t smem = (size_t)(3 * M + 2 * Dk + Dv + NW) * 4 + NT * 16;
  return smem <= 200 * 1024;
}

template <int PRE, int UNR, int MINB, int AHEAD, bool SLICED>
static int launch_variant(const DecodeParams& p, size_t smem, int slices, cudaStream_t stream) {
  auto kern = decode_step_kernel<PRE, UNR, MINB, AHEAD, SLICED>;
  if (smem > 48 * 1024) FLARE_CUDA_CHECK(allow_smem(kern));
  LaunchTimer timer("decode_step_kernel", stream);
  if constexpr (SLICED) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.B * p.H, slices);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = slices;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FLARE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, p));
  } else {
    FLARE_CUDA_CHECK(launch_pdl(kern, dim3(p.B * p.H), dim3(NT), smem, stream, p));
  }
  return FLARE_OK;
}

template <int PRE, int UNR, int MINB, bool SLICED>
static int launch_ahead(const DecodeParams& p, size_t smem, int slices, cudaStream_t stream) {
  // rows of 32 latents per round of the scores: as many as there are, or what loads the fewest of them twice
  const int rows = ((p.M + slices - 1) / slices + 31) / 32;
  constexpr int MOST = MINB == 8 ? 2 : 4;  // (more do not fit 32 registers)
  const int ahead = rows <= MOST ? rows : (MOST == 2 ? 2 : (rows % 4 == 1 || rows % 4 == 2 ? 3 : 4));
  if (ahead == 1) return launch_variant<PRE, UNR, MINB, 1, SLICED>(p, smem, slices, stream);
  if (ahead == 2) return launch_variant<PRE, UNR, MINB, 2, SLICED>(p, smem, slices, stream);
  if constexpr (MOST == 4) {
    if (ahead == 3) return launch_variant<PRE, UNR, MINB, 3, SLICED>(p, smem, slices, stream);
    return launch_variant<PRE, UNR, MINB, 4, SLICED>(p, smem, slices, stream);
  }
  return FLARE_ERR_UNSUPPORTED;
}

int launch_decode_step(const DecodeParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)(3 * p.M + 2 * p.Dk + p.Dv + NW) * 4 + NT * 16;
  // What counts is how much of the state is on its way: a thread needs registers for the vectors that it has asked for.  At 32
  // registers (eight CTAs per SM) the compiler asks for one at a time.  Per step, us on B200 with the state cold, eight CTAs / four /
  // two, in columns of their own / sliced:
  //   2048 lanes of 128 KB 121 / 97 / 99 / 108     2048 lanes of 64 KB 65 / 52 / 56 / 69      768 lanes of 32 KB 19 / 16 / 18 / 23
  //    256 lanes of 128 KB  49 / 21 / 17 / 18        96 lanes of 64 KB 12.4 / 10.9 / 8.0 / 7.8     16 lanes of 128 KB 16.6 / 11.2 / 9.3 / 6.8
  // So: four CTAs per SM while there are lanes for more than two, else two with twice the vectors, and a lane whose state does
  // not fit the vectors asked for ahead is cut into column slices (128 bytes wide at least) while two per SM hold them all.
  // Small states of many lanes have little to ask for; there eight CTAs per SM, which hide the phases before the state, are the
  // better ones.  Us a step among others, eight / four: 2048 lanes of 8 KB (M = 32, D = 64) 15.2 / 17.4, 1024 lanes 9.1 / 9.7, 2048 lanes
  // with M = 16 and keys 512 wide 18.3 / 23.2; of 16 KB (M = 64) 21.1 / 21.6 with 2048 lanes, 12.4 / 12.1 with 1024.
  // The rows of the latent bank in flight follow the latents that there are: four CTAs with four rows were 19.1 us at M = 32.
  // Measured and rejected on the largest shape: one kernel for the coefficients of all lanes and one that only streams (98 to
  // 103), 128-thread CTAs (121.7 against 112), bulk async copies through a shared-memory ring (115.5 to 207).
  const int64_t lanes = (int64_t)p.B * p.H, sms = sm_count();
  const int vectors = p.M * (p.Dv / 4);
  if (lanes > 4 * sms && vectors <= 2 * NT) return launch_ahead<2, 0, 8, false>(p, smem, 1, stream);
  if (lanes > 8 * sms && vectors <= 4 * NT) return launch_ahead<2, 4, 8, false>(p, smem, 1, stream);
  if (lanes > 2 * sms) return launch_ahead<4, 4, 4, false>(p, smem, 1, stream);
  constexpr int PRE = 8;
  int slices = 1;  // (eight at most: what a cluster may have without being asked for more, and what lane_scores serves)
  while (slices < 8 && p.M <= NT && vectors > slices * PRE * NT && lanes * slices * 2 <= 2 * sms && p.Dv / 4 % (slices * 16) == 0)
    slices *= 2;
  return slices == 1 ? launch_ahead<PRE, 8, 2, false>(p, smem, 1, stream) : launch_ahead<PRE, 8, 2, true>(p, smem, slices, stream);
}

}  // namespace flare
