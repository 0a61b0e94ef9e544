// Exact (fp32, CUDA-core) sequential walk over the tokens of one (batch, head) lane.
//
// This is the general path of the library: any dtype, any M/Dk/Dv that are multiples of 16,
// separate decode weights, attention masks, carry-in / carry-out state, token-causal or
// block-causal read-out, softmax or stablemax encoder weights.  It evaluates the online
// recurrence token by token, so it is exact for arbitrarily sharp score distributions.
//
// Work split: grid = (lane, segment, Dv tile).  A CTA walks the tokens of its segment in tiles
// of 16: (1) stage the K/V rows in shared memory as fp32, (2) all 16 x M scores with fp32 FMAs,
// (3) decode softmax over the latents, one warp per token, (4) per-latent running statistics,
// one thread per latent, (5) the state replay: warp w owns latents [w*M/8, (w+1)*M/8), lane l owns
// value columns l, l+32, ... of the tile; state and per-token output partials live in registers,
// (6) cross-warp reduction of the output partials through shared memory.
#include "walk_exact.cuh"

#include "narrow_exact.cuh"
#include "walk_cta.cuh"

namespace flare {

template <int MM_MAX, int DD>
__global__ void __launch_bounds__(NT, (MM_MAX * DD <= 32) ? 2 : 1) walk_exact_kernel(const WalkParams p) {
  pdl_wait();
  if (p.gate != nullptr) {
    int raised = 0;  // (a lane of a long sequence has up to 74 words)
    for (int i = threadIdx.x; i < p.gate_count; i += NT) raised |= p.gate[(int64_t)blockIdx.x * p.gate_stride + i];
    if (!__syncthreads_or(raised)) return;
  }
  walk_cta<MM_MAX, DD>(p, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z));
}

#ifdef FLARE_WALK_MM
// One translation unit per latents-per-warp bound, so the instantiations compile in parallel.
template <int MM_MAX, int DD>
static int launch_one(const WalkParams& p, dim3 grid, size_t smem, cudaStream_t stream) {
  auto kern = walk_exact_kernel<MM_MAX, DD>;
  FLARE_CUDA_CHECK(allow_smem(kern));
  LaunchTimer timer(p.gate != nullptr ? "walk_exact_kernel (standby)" : "walk_exact_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(kern, grid, dim3(NT), smem, stream, p));
  return FLARE_OK;
}

template <>
int launch_walk_mm<FLARE_WALK_MM>(const WalkParams& p, int dd, dim3 grid, size_t smem, cudaStream_t stream) {
  constexpr int MM_MAX = FLARE_WALK_MM;
  if (dd == 1) return launch_one<MM_MAX, 1>(p, grid, smem, stream);
  if (dd == 2) {
    if constexpr (MM_MAX * 2 <= 64) return launch_one<MM_MAX, 2>(p, grid, smem, stream);
  }
  if (dd == 4) {
    if constexpr (MM_MAX * 4 <= 64) return launch_one<MM_MAX, 4>(p, grid, smem, stream);
  }
  return FLARE_ERR_UNSUPPORTED;
}
#else
int walk_exact_dd(int M, int Dv) {
  const int mm = M / NW;
  int dd = 1;
  while (dd < 4 && dd * 32 < Dv && mm * dd * 2 <= 64) dd *= 2;
  return dd;
}

int launch_walk_exact(const WalkParams& p, int nseg_grid, cudaStream_t stream) {
  if (p.M % 16 != 0 || p.M > 512) return FLARE_ERR_UNSUPPORTED;
  if (nseg_grid <= 0 || p.B * p.H <= 0) return FLARE_OK;
  if (p.gate == nullptr && narrow_shape(p.M, p.Dk, p.Dv, p.block_size, p.qd != nullptr || p.kd != nullptr))
    return launch_walk_narrow(p, nseg_grid, stream);
  const int mm = p.M / NW;
  const int dd = walk_exact_dd(p.M, p.Dv);
  const int dvt = 32 * dd;
  dim3 grid(p.B * p.H, nseg_grid, (p.Dv + dvt - 1) / dvt);
  const size_t smem = walk_exact_smem_bytes(p.M, p.Dk, dd);
  if (smem > 227 * 1024) return FLARE_ERR_UNSUPPORTED;
  if (mm <= 2) return launch_walk_mm<2>(p, dd, grid, smem, stream);
  if (mm <= 8) return launch_walk_mm<8>(p, dd, grid, smem, stream);
  if (mm <= 16) return launch_walk_mm<16>(p, dd, grid, smem, stream);
  if (mm <= 32) return launch_walk_mm<32>(p, dd, grid, smem, stream);
  return launch_walk_mm<64>(p, dd, grid, smem, stream);
}
#endif

}  // namespace flare
