// Exact (fp32, CUDA-core) backward of causal FLARE: softmax / stablemax encoders, token-causal or
// block-causal read-out, shared or separate decode weights.  Nothing is saved by the forward; the
// forward recurrence is replayed here.
//
// With e[t,m] the normalised encoder weight of token t at its read-out time (softmax exp(s - L_t),
// stablemax sigma(s)/D_t) the read-out state obeys z_t = (1 - e_t) z_{t-1} + e_t v_t, hence
//   p[t,m]   = <z_t[m,:], dY_t>                        g[t,:] = softmax_m(a[t,:])
//   b_t[m,:] = g dY_t + (1 - e_{t+1}) b_{t+1}           c_t[m] = g p + (1 - e_{t+1}) c_{t+1}
//   dV_t     = sum_m e b_t[m,:]
//   dS_enc   = e * slope * (<b_t[m,:], v_t> - c_t[m])    slope = 1 | sigma'(s)/sigma(s)
//   dS_dec   = g (p - sum_m g p)
//   dK = scale dS Q,  dQ = scale sum_{b,t} dS^T k_t  (decode-side products go to dQ_dec / dK_dec when separate)
// For block-causal read-out the state is read at block ends, so e, b, c are per block.
//
// Kernels: (1) replay: forward walk that stores e, g and the partial p of its Dv tile;
// (2) reverse: reverse walk carrying (b, c), emits dV and the dS planes; (3) rows: dK / dQ_dec = dS Lat;
// (4) latents: per-split partial dQ / dK_dec = dS^T Rows; (5) fixed-order sum of the partials
// (deterministic: no atomics anywhere).
// Heads up to 32 wide take narrow_exact.cu instead: its replay also forms the segment carries, its reverse walk also dK
// and dQ, so (3), (4) and the dS planes fall away; bf16 softmax calls among those take narrow_mma.cu.  The kernels' bodies are in
// bwd_cta.cuh: behind the tensor-core backward they stand by as the tasks of one kernel (bwd_standby.cu).
#include "bwd_exact.cuh"

#include <string.h>

#include "bwd_cta.cuh"
#include "narrow_exact.cuh"
#include "narrow_mma.cuh"
#include "prefill_tc.cuh"
#include "state_ops.cuh"
#include "walk_cta.cuh"
#include "walk_exact.cuh"

namespace flare {

// defined once per MM_MAX in {2, 8, 16, 32, 64}, each in its own translation unit; stage 0 = replay, 1 = reverse
template <int MM_MAX>
int launch_bwd_mm(const BwdParams& p, int dd, dim3 grid, size_t smem1, size_t smem2, cudaStream_t stream, int stage);

namespace {

#ifdef FLARE_WALK_MM
template <int MM_MAX, int DD>
__global__ void __launch_bounds__(NT, (MM_MAX * DD <= 32) ? 2 : 1) bwd_replay_kernel(const BwdParams p) {
  pdl_begin();
  replay_cta<MM_MAX, DD>(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

template <int MM_MAX, int DD>
__global__ void __launch_bounds__(NT, (MM_MAX * DD <= 32) ? 2 : 1) bwd_reverse_kernel(const BwdParams p) {
  pdl_begin();
  reverse_cta<MM_MAX, DD>(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

#else
__global__ void __launch_bounds__(NT) bwd_rows_kernel(const RowsParams p) {
  pdl_begin();
  rows_cta(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

__global__ void __launch_bounds__(NT) bwd_lat_kernel(const LatParams p) {
  pdl_begin();
  lat_cta(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

__global__ void __launch_bounds__(NT) bwd_seg_carry_kernel(const CarryParams p) {
  pdl_begin();
  carry_cta(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

// (gate: of the narrow kernels standing by, which come one by one)
__global__ void __launch_bounds__(256) bwd_seg_scan_kernel(const ScanParams p, const int* gate) {
  pdl_begin();
  if (gate != nullptr && *gate == 0) return;
  scan_element(p, (int64_t)blockIdx.x * 256 + threadIdx.x);
}

__global__ void __launch_bounds__(256) bwd_sum_splits_kernel(const SumParams p, const int* gate) {
  pdl_begin();
  if (gate != nullptr && *gate == 0) return;
  sum_element(p, (int64_t)blockIdx.x * 256 + threadIdx.x);
}

struct BwdPlan {
  bool narrow;
  int dd, DT, splits, rows_per_split;
  int nseg, seg_len;  // sequence segments of the replay / reverse walks (token-causal read-out only)
  int64_t plane;
  size_t off_E, off_G, off_W2, off_P, off_dSe, off_dSd, off_part_q, off_part_kd, total;
  size_t off_seg_m, off_seg_d, off_seg_u, off_seg_b, off_seg_c, off_seg_gam, off_X, off_RHO;
};

// a span of a longer sequence: prefix state, carries from the right or a summary wanted
bool span_mode(const flare_bwd_args_t& a) {
  return a.fwd.state_in.u != nullptr || a.carry_b != nullptr || a.span_b0 != nullptr || a.phase != 0;
}

BwdPlan plan_backward(const flare_bwd_args_t& a) {
  const flare_fwd_args_t& f = a.fwd;
  BwdPlan pl;
  memset(&pl, 0, sizeof(pl));
  pl.narrow = !span_mode(a) && narrow_shape(f.M, f.Dk, f.Dv, f.block_size, f.q_dec != nullptr || f.k_dec != nullptr);
  if (pl.narrow) {
    // as many segments as keep about twelve warps per SM in flight (the replay's registers allow no more), of 64 tokens at least
    const int64_t lanes = (int64_t)f.B * f.H;
    int64_t nseg = 12LL * sm_count() / (lanes * narrow_warps(f.M));
    if (nseg > f.N / 64) nseg = f.N / 64;
    if (nseg < 1) nseg = 1;
    pl.seg_len = (int)(((f.N + nseg - 1) / nseg + 15) / 16 * 16);
    pl.nseg = (f.N + pl.seg_len - 1) / pl.seg_len;
    pl.plane = lanes * f.N * f.M;
    size_t off = 0;
    auto take = [&](size_t floats) {
      const size_t o = off;
      off += align_up(floats * 4, 256);
      return o;
    };
    pl.off_E = take((size_t)pl.plane);
    pl.off_G = take((size_t)pl.plane);
    pl.off_W2 = f.variant == FLARE_STABLEMAX ? take((size_t)pl.plane) : pl.off_E;
    pl.off_P = take((size_t)pl.plane);
    pl.off_part_q = take((size_t)f.B * pl.nseg * f.H * f.M * f.Dk);
    if (pl.nseg > 1) {
      const size_t ls = (size_t)lanes * pl.nseg;
      pl.off_seg_m = take(ls * f.M);
      pl.off_seg_d = take(ls * f.M);
      pl.off_seg_u = take(ls * f.M * f.Dv);
      pl.off_seg_b = take(ls * f.M * f.Dv);
      pl.off_seg_c = take(ls * f.M);
      pl.off_seg_gam = take(ls * f.M);
    }
    pl.total = off;
    return pl;
  }
  pl.dd = walk_exact_dd(f.M, f.Dv);
  pl.DT = (f.Dv + 32 * pl.dd - 1) / (32 * pl.dd);
  // The walks are sequential in the tokens; with few (lane, value tile) CTAs the sequence is cut into segments that
  // run concurrently (prefix states for the replay, carries (b, c) for the reverse walk, see bwd_exact()).
  // Measured at B=4, N=4096, H=16, M=64, D=128 (ms per training step): 2 segments 6.09, 4: 3.87, 8: 3.91, 16: 3.95;
  // narrower value tiles (more CTAs, repeated score work) are slower once the sequence is segmented (5.1-8.9).
  pl.nseg = 1;
  pl.seg_len = f.N;
  {
    // segments are whole 128-token chunks (forward kernels) and whole blocks (block-causal read-out)
    int unit = 128;
    if (f.block_size > 1) {
      int a = f.block_size, b = 128;
      while (b != 0) { const int t = a % b; a = b; b = t; }
      unit = f.block_size / a * 128;
    }
    const int min_seg = unit > 256 ? unit : 256;
    const int64_t ctas = (int64_t)f.B * f.H * pl.DT, target = 4LL * sm_count();
    int nseg = (int)((target + ctas - 1) / ctas);
    const int max_seg = f.N / min_seg;
    if (nseg > max_seg) nseg = max_seg;
    if (nseg > 1) {
      int seg_len = (f.N + nseg - 1) / nseg;
      seg_len = (seg_len + unit - 1) / unit * unit;
      pl.seg_len = seg_len;
      pl.nseg = (f.N + seg_len - 1) / seg_len;
    }
  }
  pl.plane = (int64_t)f.B * f.H * f.N * f.M;
  const bool stablemax = f.variant == FLARE_STABLEMAX;
  const bool shared_w = f.q_dec == nullptr && f.k_dec == nullptr;
  const int64_t rows = (int64_t)f.B * f.N;
  const int mt = (f.M + LM - 1) / LM, dkc = (f.Dk + LDK - 1) / LDK;
  int64_t splits = (2LL * sm_count() + (int64_t)f.H * mt * dkc - 1) / ((int64_t)f.H * mt * dkc);
  const int64_t max_splits = (rows + 255) / 256;
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  int64_t rps = (rows + splits - 1) / splits;
  rps = (rps + LT - 1) / LT * LT;
  splits = (rows + rps - 1) / rps;
  pl.splits = (int)splits;
  pl.rows_per_split = (int)rps;
  size_t off = 0;
  auto take = [&](size_t floats) {
    const size_t o = off;
    off += align_up(floats * 4, 256);
    return o;
  };
  const size_t plane = (size_t)pl.plane;
  pl.off_E = take(plane);
  pl.off_G = take(plane);
  pl.off_W2 = stablemax ? take(plane) : pl.off_E;
  pl.off_P = take(plane * pl.DT);
  pl.off_dSe = take(plane * pl.DT);
  pl.off_dSd = shared_w ? 0 : take(plane);
  const size_t lat = (size_t)f.H * f.M * f.Dk;
  pl.off_part_q = take(lat * pl.splits);
  pl.off_part_kd = f.k_dec ? take(lat * pl.splits) : 0;
  pl.off_seg_m = pl.off_seg_d = pl.off_seg_u = pl.off_seg_b = pl.off_seg_c = pl.off_seg_gam = pl.off_X = pl.off_RHO = 0;
  if (pl.nseg > 1 || span_mode(a)) {
    const size_t ls = (size_t)f.B * f.H * pl.nseg;
    pl.off_seg_m = take(ls * f.M);
    pl.off_seg_d = take(ls * f.M);
    pl.off_seg_u = take(ls * f.M * f.Dv);
    pl.off_seg_b = take(ls * f.M * f.Dv);
    pl.off_seg_c = take(ls * f.M);
    pl.off_seg_gam = take(ls * f.M);
    pl.off_X = take(plane);
    pl.off_RHO = f.block_size > 1 ? take((size_t)f.B * f.H * (f.N / f.block_size) * f.M) : 0;
  }
  pl.total = off;
  return pl;
}

#endif

}  // namespace

#ifdef FLARE_WALK_MM
template <int MM_MAX, int DD>
static int launch_bwd_one(const BwdParams& p, dim3 grid, size_t smem1, size_t smem2, cudaStream_t stream, int stage) {
  if (stage == 0) {
    auto k1 = bwd_replay_kernel<MM_MAX, DD>;
    FLARE_CUDA_CHECK(allow_smem(k1));
    LaunchTimer timer("bwd_replay_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(k1, grid, dim3(NT), smem1, stream, p));
  } else {
    auto k2 = bwd_reverse_kernel<MM_MAX, DD>;
    FLARE_CUDA_CHECK(allow_smem(k2));
    LaunchTimer timer("bwd_reverse_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(k2, grid, dim3(NT), smem2, stream, p));
  }
  return FLARE_OK;
}

template <>
int launch_bwd_mm<FLARE_WALK_MM>(const BwdParams& p, int dd, dim3 grid, size_t smem1, size_t smem2, cudaStream_t stream,
                                 int stage) {
  constexpr int MM_MAX = FLARE_WALK_MM;
  if (dd == 1) return launch_bwd_one<MM_MAX, 1>(p, grid, smem1, smem2, stream, stage);
  if (dd == 2) {
    if constexpr (MM_MAX * 2 <= 64) return launch_bwd_one<MM_MAX, 2>(p, grid, smem1, smem2, stream, stage);
  }
  if (dd == 4) {
    if constexpr (MM_MAX * 4 <= 64) return launch_bwd_one<MM_MAX, 4>(p, grid, smem1, smem2, stream, stage);
  }
  return FLARE_ERR_UNSUPPORTED;
}
#else

constexpr size_t kGateBytes = 256;

size_t bwd_exact_workspace_bytes(const flare_bwd_args_t& a) {
  if (a.fwd.B == 0 || a.fwd.N == 0) return 0;
  const size_t exact = plan_backward(a).total;
  if (!narrow_mma_backward_supported(a)) return exact;
  const size_t mma = narrow_mma_backward_bytes(a);  // (shares its space with the pass standing by; the gate word comes first)
  return kGateBytes + (mma > exact ? mma : exact);
}

static int bwd_narrow(const flare_bwd_args_t& a, const BwdPlan& pl, cudaStream_t stream, const int* gate) {
  const flare_fwd_args_t& f = a.fwd;
  char* ws = reinterpret_cast<char*>(f.workspace);
  auto at = [&](size_t off) { return reinterpret_cast<float*>(ws + off); };
  NarrowBwdParams p;
  memset(&p, 0, sizeof(p));
  p.q = f.q; p.k = f.k; p.v = f.v; p.dy = a.dy;
  p.B = f.B; p.N = f.N; p.H = f.H; p.M = f.M; p.Dk = f.Dk; p.Dv = f.Dv;
  p.q_stride_h = f.q_stride_h; p.q_stride_m = f.q_stride_m;
  p.k_stride_b = f.k_stride_b; p.k_stride_n = f.k_stride_n; p.k_stride_h = f.k_stride_h;
  p.v_stride_b = f.v_stride_b; p.v_stride_n = f.v_stride_n; p.v_stride_h = f.v_stride_h;
  p.dy_stride_b = a.dy_stride_b; p.dy_stride_n = a.dy_stride_n; p.dy_stride_h = a.dy_stride_h;
  p.scale = f.scale; p.power = f.power; p.dtype = f.dtype; p.variant = f.variant;
  p.E = at(pl.off_E); p.G = at(pl.off_G); p.W2 = at(pl.off_W2); p.P = at(pl.off_P);
  p.seg_len = pl.seg_len; p.nseg = pl.nseg;
  p.dk = a.dk; p.dv = a.dv; p.dq_part = at(pl.off_part_q);
  p.gate = gate;
  int rc;
  if (pl.nseg > 1) {
    p.in_m = at(pl.off_seg_m); p.in_d = at(pl.off_seg_d); p.in_u = at(pl.off_seg_u);
    p.seg_b = at(pl.off_seg_b); p.seg_c = at(pl.off_seg_c); p.seg_gam = at(pl.off_seg_gam);
    rc = segment_prefix_states(&f, pl.nseg, pl.seg_len, at(pl.off_seg_m), at(pl.off_seg_d), at(pl.off_seg_u), nullptr, stream,
                               gate);
    if (rc != FLARE_OK) return rc;
  }
  rc = launch_narrow_replay(p, stream);
  if (rc != FLARE_OK) return rc;
  if (pl.nseg > 1) {
    const int64_t lanes = (int64_t)f.B * f.H, nscan = lanes * f.M * (f.Dv + 1);
    LaunchTimer timer("bwd_seg_scan_kernel", stream);
    ScanParams sc;
    memset(&sc, 0, sizeof(sc));
    sc.seg_b = p.seg_b; sc.seg_c = p.seg_c; sc.seg_gam = p.seg_gam; sc.nseg = pl.nseg; sc.seg_len = pl.seg_len; sc.lanes = lanes;
    sc.N = f.N; sc.M = f.M; sc.Dv = f.Dv; sc.E = p.E; sc.block_size = 1; sc.write_slots = 1;
    FLARE_CUDA_CHECK(launch_pdl(bwd_seg_scan_kernel, dim3((unsigned)((nscan + 255) / 256)), dim3(256), 0, stream, sc, gate));
  }
  rc = launch_narrow_reverse(p, stream);
  if (rc != FLARE_OK) return rc;
  const int64_t lat_n = (int64_t)f.H * f.M * f.Dk;
  LaunchTimer timer("bwd_sum_splits_kernel", stream);
  const SumParams sum{a.dq, a.dq_dtype, p.dq_part, lat_n, f.B * pl.nseg};
  FLARE_CUDA_CHECK(launch_pdl(bwd_sum_splits_kernel, dim3((unsigned)((lat_n + 255) / 256)), dim3(256), 0, stream, sum, gate));
  return FLARE_OK;
}

int bwd_exact(const flare_bwd_args_t& a, cudaStream_t stream, const int* gate, int* sync) {
  const flare_fwd_args_t& f = a.fwd;
  if (f.B == 0 || f.N == 0) return FLARE_OK;
  if (f.M > 512) return FLARE_ERR_UNSUPPORTED;
  if (gate == nullptr && narrow_mma_backward_supported(a)) {
    if (f.workspace == nullptr || f.workspace_bytes < bwd_exact_workspace_bytes(a) || (reinterpret_cast<uintptr_t>(f.workspace) & 15u))
      return FLARE_ERR_WORKSPACE;
    char* ws = reinterpret_cast<char*>(f.workspace);
    int* word = reinterpret_cast<int*>(ws);
    const int rc = narrow_mma_backward(a, ws + kGateBytes, word, stream);
    if (rc != FLARE_OK) return rc;
    flare_bwd_args_t ex = a;  // standing by: every kernel returns at once unless the word is set
    ex.fwd.path = FLARE_PATH_EXACT;
    ex.fwd.workspace = ws + kGateBytes;
    ex.fwd.workspace_bytes = f.workspace_bytes - kGateBytes;
    return bwd_exact(ex, stream, word);
  }
  const BwdPlan pl = plan_backward(a);
  if (f.workspace == nullptr || f.workspace_bytes < pl.total || (reinterpret_cast<uintptr_t>(f.workspace) & 15u))
    return FLARE_ERR_WORKSPACE;
  if (pl.narrow) return bwd_narrow(a, pl, stream, gate);
  char* ws = reinterpret_cast<char*>(f.workspace);
  const bool stablemax = f.variant == FLARE_STABLEMAX;
  const bool shared_w = f.q_dec == nullptr && f.k_dec == nullptr;
  BwdParams p;
  memset(&p, 0, sizeof(p));
  p.q = f.q; p.k = f.k; p.v = f.v; p.qd = f.q_dec; p.kd = f.k_dec; p.dy = a.dy;
  p.B = f.B; p.N = f.N; p.H = f.H; p.M = f.M; p.Dk = f.Dk; p.Dv = f.Dv;
  p.q_stride_h = f.q_stride_h; p.q_stride_m = f.q_stride_m;
  p.k_stride_b = f.k_stride_b; p.k_stride_n = f.k_stride_n; p.k_stride_h = f.k_stride_h;
  p.v_stride_b = f.v_stride_b; p.v_stride_n = f.v_stride_n; p.v_stride_h = f.v_stride_h;
  p.qd_stride_b = f.qd_stride_b; p.qd_stride_n = f.qd_stride_n; p.qd_stride_h = f.qd_stride_h;
  p.kd_stride_h = f.kd_stride_h; p.kd_stride_m = f.kd_stride_m;
  p.dy_stride_b = a.dy_stride_b; p.dy_stride_n = a.dy_stride_n; p.dy_stride_h = a.dy_stride_h;
  p.scale = f.scale; p.power = f.power; p.dtype = f.dtype; p.variant = f.variant; p.block_size = f.block_size;
  p.E = reinterpret_cast<float*>(ws + pl.off_E);
  p.G = reinterpret_cast<float*>(ws + pl.off_G);
  p.W2 = reinterpret_cast<float*>(ws + pl.off_W2);
  p.P = reinterpret_cast<float*>(ws + pl.off_P);
  p.dSe = reinterpret_cast<float*>(ws + pl.off_dSe);
  p.dSd = shared_w ? nullptr : reinterpret_cast<float*>(ws + pl.off_dSd);
  p.DT = pl.DT; p.plane = pl.plane; p.dv_out = a.dv;
  p.nseg = pl.nseg; p.seg_len = pl.seg_len; p.seg_first = 0;
  const int64_t lanes = (int64_t)f.B * f.H;
  const bool seg_mode = pl.nseg > 1 || span_mode(a);
  if (a.phase < 0 || a.phase > 2 || (a.span_b0 != nullptr && !(a.span_c0 && a.span_gam && a.span_rho_first)) ||
      (a.carry_b != nullptr && !(a.carry_c && a.carry_rho)) || (span_mode(a) && f.block_size > 1 && f.N % f.block_size))
    return FLARE_ERR_BAD_POINTER;
  float *seg_m = nullptr, *seg_d = nullptr, *seg_u = nullptr;
  if (seg_mode) {
    seg_m = reinterpret_cast<float*>(ws + pl.off_seg_m);
    seg_d = reinterpret_cast<float*>(ws + pl.off_seg_d);
    seg_u = reinterpret_cast<float*>(ws + pl.off_seg_u);
    p.in_m = seg_m; p.in_d = seg_d; p.in_u = seg_u;
    p.seg_b = reinterpret_cast<float*>(ws + pl.off_seg_b);
    p.seg_c = reinterpret_cast<float*>(ws + pl.off_seg_c);
    p.seg_gam = reinterpret_cast<float*>(ws + pl.off_seg_gam);
    p.X = reinterpret_cast<float*>(ws + pl.off_X);
    p.RHO = f.block_size > 1 ? reinterpret_cast<float*>(ws + pl.off_RHO) : nullptr;
  }
  p.carry_b = a.carry_b; p.carry_c = a.carry_c; p.carry_rho = a.carry_rho;

  const int mm = f.M / NW;
  const size_t smem1 = replay_smem(f.M, f.Dk, pl.dd), smem2 = reverse_smem(f.M, pl.dd, stablemax);
  if (smem1 > 227 * 1024 || smem2 > 227 * 1024) return FLARE_ERR_UNSUPPORTED;
  auto walk = [&](int stage, int seg_first, int seg_count) -> int {
    BwdParams q = p;
    q.seg_first = seg_first;
    dim3 grid(f.B * f.H, pl.DT, seg_count);
    if (mm <= 2) return launch_bwd_mm<2>(q, pl.dd, grid, smem1, smem2, stream, stage);
    if (mm <= 8) return launch_bwd_mm<8>(q, pl.dd, grid, smem1, smem2, stream, stage);
    if (mm <= 16) return launch_bwd_mm<16>(q, pl.dd, grid, smem1, smem2, stream, stage);
    if (mm <= 32) return launch_bwd_mm<32>(q, pl.dd, grid, smem1, smem2, stream, stage);
    return launch_bwd_mm<64>(q, pl.dd, grid, smem1, smem2, stream, stage);
  };
  const int64_t nscan = lanes * f.M * (f.Dv + 1);
  auto scan_params = [&](bool write_slots, bool with_carry, bool summary) {
    ScanParams sc;
    memset(&sc, 0, sizeof(sc));
    sc.seg_b = p.seg_b; sc.seg_c = p.seg_c; sc.seg_gam = p.seg_gam; sc.nseg = pl.nseg; sc.seg_len = pl.seg_len; sc.lanes = lanes;
    sc.N = f.N; sc.M = f.M; sc.Dv = f.Dv; sc.E = p.E; sc.RHO = p.RHO; sc.block_size = f.block_size;
    if (with_carry) {
      sc.carry_b = a.carry_b; sc.carry_c = a.carry_c; sc.carry_rho = a.carry_rho;
    }
    sc.write_slots = write_slots ? 1 : 0;
    sc.span_b0 = summary ? a.span_b0 : nullptr;
    sc.span_c0 = a.span_c0; sc.span_gam = a.span_gam; sc.span_rho_first = a.span_rho_first;
    return sc;
  };
  auto scan = [&](bool write_slots, bool with_carry, bool summary) -> int {
    LaunchTimer timer("bwd_seg_scan_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(bwd_seg_scan_kernel, dim3((unsigned)((nscan + 255) / 256)), dim3(256), 0, stream,
                                scan_params(write_slots, with_carry, summary), nullptr));
    return FLARE_OK;
  };
  CarryParams carry;
  memset(&carry, 0, sizeof(carry));
  carry.X = p.X; carry.P = p.P; carry.p_parts = pl.DT; carry.plane = pl.plane; carry.dy = a.dy; carry.dtype = f.dtype;
  carry.dy_stride_b = a.dy_stride_b; carry.dy_stride_n = a.dy_stride_n; carry.dy_stride_h = a.dy_stride_h;
  carry.seg_b = p.seg_b; carry.seg_c = p.seg_c; carry.nseg = pl.nseg; carry.seg_len = pl.seg_len;
  carry.N = f.N; carry.H = f.H; carry.M = f.M; carry.Dv = f.Dv;
  const int mt = (f.M + LM - 1) / LM, dkc = (f.Dk + LDK - 1) / LDK;
  const int64_t lat_n = (int64_t)f.H * f.M * f.Dk;
  const dim3 carry_grid((unsigned)(lanes * mt), pl.nseg, (f.Dv + LDK - 1) / LDK);
  const dim3 rows_grid(f.B * f.H, (f.N + RT - 1) / RT, (f.Dk + RC - 1) / RC), lat_grid(f.H * mt, pl.splits, dkc);
  auto fill_rows = [&](RowsParams& r) {
    r.plane = pl.plane; r.B = f.B; r.N = f.N; r.H = f.H; r.M = f.M; r.Dk = f.Dk; r.dtype = f.dtype; r.scale = f.scale;
  };
  auto fill_lat = [&](LatParams& l, float* partial) {
    l.plane = pl.plane; l.B = f.B; l.N = f.N; l.H = f.H; l.M = f.M; l.Dk = f.Dk; l.dtype = f.dtype; l.scale = f.scale;
    l.rows_per_split = pl.rows_per_split; l.splits = pl.splits; l.partial = partial;
  };
  if (gate != nullptr) {
    // standing by: the whole pass as one kernel
    if (!shared_w || span_mode(a) || sync == nullptr) return FLARE_ERR_UNSUPPORTED;
    StandbyParams s;
    memset(&s, 0, sizeof(s));
    auto tasks = [&](int phase, dim3 g) { s.nx[phase] = (int)g.x; s.ny[phase] = (int)g.y; s.nz[phase] = (int)g.z; };
    s.bwd = p;
    if (seg_mode) {
      segment_state_params(&f, pl.nseg, pl.seg_len, seg_m, seg_d, seg_u, &s.walk, &s.fold);
      tasks(0, dim3((unsigned)lanes, pl.nseg - 1, pl.DT));
      tasks(1, dim3((unsigned)lanes, (f.M + NW - 1) / NW, 1));
      s.carry = carry;
      tasks(3, carry_grid);
      s.scan = scan_params(true, false, false);
      tasks(4, dim3((unsigned)((nscan + NT - 1) / NT), 1, 1));
    }
    tasks(2, dim3((unsigned)lanes, pl.DT, pl.nseg));
    tasks(5, dim3((unsigned)lanes, pl.DT, pl.nseg));
    s.rows.out = a.dk;
    s.rows.ds[0] = p.dSe; s.rows.parts[0] = pl.DT; s.rows.lat[0] = f.q;
    s.rows.lat_stride_h[0] = f.q_stride_h; s.rows.lat_stride_m[0] = f.q_stride_m; s.rows.nsrc = 1;
    fill_rows(s.rows);
    tasks(6, rows_grid);
    float* const partial = reinterpret_cast<float*>(ws + pl.off_part_q);
    s.lat.ds[0] = p.dSe; s.lat.parts[0] = pl.DT; s.lat.rows[0] = f.k;
    s.lat.rows_stride_b[0] = f.k_stride_b; s.lat.rows_stride_n[0] = f.k_stride_n; s.lat.rows_stride_h[0] = f.k_stride_h;
    s.lat.nsrc = 1;
    fill_lat(s.lat, partial);
    tasks(7, lat_grid);
    s.sum = SumParams{a.dq, a.dq_dtype, partial, lat_n, pl.splits};
    tasks(8, dim3((unsigned)((lat_n + NT - 1) / NT), 1, 1));
    s.gate = gate;
    s.sync = sync;
    const int rc = tc_error_word(&s.err);
    if (rc != FLARE_OK) return rc;
    size_t smem = walk_exact_smem_bytes(f.M, f.Dk, pl.dd);
    for (size_t need : {smem1, smem2, kRowsSmem, kLatSmem})
      if (need > smem) smem = need;
    if (mm <= 2) return launch_bwd_standby<2>(s, pl.dd, smem, stream);
    if (mm <= 8) return launch_bwd_standby<8>(s, pl.dd, smem, stream);
    if (mm <= 16) return launch_bwd_standby<16>(s, pl.dd, smem, stream);
    if (mm <= 32) return launch_bwd_standby<32>(s, pl.dd, smem, stream);
    return launch_bwd_standby<64>(s, pl.dd, smem, stream);
  }
  int rcw = FLARE_OK;
  if (a.phase != 2) {
    if (seg_mode) {
      // exclusive prefix state of every segment, from the forward kernels (slot 0: the state before the span)
      rcw = segment_prefix_states(&f, pl.nseg, pl.seg_len, seg_m, seg_d, seg_u,
                                  f.state_in.u != nullptr ? &f.state_in : nullptr, stream);
      if (rcw != FLARE_OK) return rcw;
    }
    rcw = walk(0, 0, pl.nseg);  // replay: planes e, g, p (and X, the carry weights, when segmented)
    if (rcw != FLARE_OK) return rcw;
    if (seg_mode) {
      // carries of every segment for a zero carry-in, as products over the planes
      LaunchTimer timer("bwd_seg_carry_kernel", stream);
      FLARE_CUDA_CHECK(launch_pdl(bwd_seg_carry_kernel, carry_grid, dim3(NT), kLatSmem, stream, carry));
      if (a.span_b0 != nullptr) {
        rcw = scan(false, false, true);  // summary of the span for a zero carry-in from the right
        if (rcw != FLARE_OK) return rcw;
      }
    }
    if (a.phase == 1) return FLARE_OK;
  }
  if (seg_mode) {
    rcw = scan(true, true, false);  // right-to-left scan: every segment's true carry-in
    if (rcw != FLARE_OK) return rcw;
  }
  rcw = walk(1, 0, pl.nseg);  // reverse walk: dV and the dS planes
  if (rcw != FLARE_OK) return rcw;

  // ---- dK (+ dQ_dec): products of the dS planes with the latent banks ------------------------------
  auto rows_launch = [&](RowsParams& r) -> int {
    fill_rows(r);
    LaunchTimer timer("bwd_rows_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(bwd_rows_kernel, rows_grid, dim3(NT), kRowsSmem, stream, r));
    return FLARE_OK;
  };
  {
    RowsParams r;
    memset(&r, 0, sizeof(r));
    r.out = a.dk;
    r.ds[0] = p.dSe; r.parts[0] = pl.DT; r.lat[0] = f.q; r.lat_stride_h[0] = f.q_stride_h; r.lat_stride_m[0] = f.q_stride_m;
    r.nsrc = 1;
    if (!shared_w && f.q_dec == nullptr) {  // decode queries are the keys: their gradient lands on K
      r.ds[1] = p.dSd; r.parts[1] = 1; r.lat[1] = f.k_dec; r.lat_stride_h[1] = f.kd_stride_h; r.lat_stride_m[1] = f.kd_stride_m;
      r.nsrc = 2;
    }
    int rc = rows_launch(r);
    if (rc != FLARE_OK) return rc;
  }
  if (f.q_dec != nullptr) {
    RowsParams r;
    memset(&r, 0, sizeof(r));
    r.out = a.dq_dec;
    r.ds[0] = p.dSd; r.parts[0] = 1;
    r.lat[0] = f.k_dec ? f.k_dec : f.q;
    r.lat_stride_h[0] = f.k_dec ? f.kd_stride_h : f.q_stride_h;
    r.lat_stride_m[0] = f.k_dec ? f.kd_stride_m : f.q_stride_m;
    r.nsrc = 1;
    int rc = rows_launch(r);
    if (rc != FLARE_OK) return rc;
  }

  // ---- dQ (+ dK_dec): split partial sums, then a fixed-order reduction -------------------------------
  auto lat_launch = [&](LatParams& l, float* partial, void* out, int out_dtype) -> int {
    fill_lat(l, partial);
    {
      LaunchTimer timer("bwd_lat_kernel", stream);
      FLARE_CUDA_CHECK(launch_pdl(bwd_lat_kernel, lat_grid, dim3(NT), kLatSmem, stream, l));
    }
    const SumParams sum{out, out_dtype, partial, lat_n, pl.splits};
    LaunchTimer timer("bwd_sum_splits_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(bwd_sum_splits_kernel, dim3((unsigned)((lat_n + 255) / 256)), dim3(256), 0, stream, sum, nullptr));
    return FLARE_OK;
  };
  {
    LatParams l;
    memset(&l, 0, sizeof(l));
    l.ds[0] = p.dSe; l.parts[0] = pl.DT; l.rows[0] = f.k;
    l.rows_stride_b[0] = f.k_stride_b; l.rows_stride_n[0] = f.k_stride_n; l.rows_stride_h[0] = f.k_stride_h;
    l.nsrc = 1;
    if (!shared_w && f.k_dec == nullptr) {  // decode keys are the latent queries: their gradient lands on Q
      l.ds[1] = p.dSd; l.parts[1] = 1; l.rows[1] = f.q_dec;
      l.rows_stride_b[1] = f.qd_stride_b; l.rows_stride_n[1] = f.qd_stride_n; l.rows_stride_h[1] = f.qd_stride_h;
      l.nsrc = 2;
    }
    int rc = lat_launch(l, reinterpret_cast<float*>(ws + pl.off_part_q), a.dq, a.dq_dtype);
    if (rc != FLARE_OK) return rc;
  }
  if (f.k_dec != nullptr) {
    LatParams l;
    memset(&l, 0, sizeof(l));
    l.ds[0] = p.dSd; l.parts[0] = 1;
    l.rows[0] = f.q_dec ? f.q_dec : f.k;
    l.rows_stride_b[0] = f.q_dec ? f.qd_stride_b : f.k_stride_b;
    l.rows_stride_n[0] = f.q_dec ? f.qd_stride_n : f.k_stride_n;
    l.rows_stride_h[0] = f.q_dec ? f.qd_stride_h : f.k_stride_h;
    l.nsrc = 1;
    int rc = lat_launch(l, reinterpret_cast<float*>(ws + pl.off_part_kd), a.dk_dec, FLARE_F32);
    if (rc != FLARE_OK) return rc;
  }
  return FLARE_OK;
}
#endif

}  // namespace flare
