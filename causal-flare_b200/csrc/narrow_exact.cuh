// Exact kernels for narrow heads (see narrow_exact.cu).
#pragma once
#include "flare_common.cuh"
#include "walk_exact.cuh"

namespace flare {

// Head widths up to 32 and at most 128 latents, token-causal read-out with shared decode weights.
inline bool narrow_shape(int M, int Dk, int Dv, int block_size, bool separate_weights) {
  return M <= 128 && Dk <= 32 && Dv <= 32 && block_size <= 1 && !separate_weights;
}
inline int narrow_warps(int M) { return (M + 31) / 32; }  // warps per CTA, one CTA per (lane, segment)

int launch_walk_narrow(const WalkParams& p, int nseg_grid, cudaStream_t stream);

struct NarrowBwdParams {
  const void *q, *k, *v, *dy;
  int B, N, H, M, Dk, Dv;
  int64_t q_stride_h, q_stride_m;
  int64_t k_stride_b, k_stride_n, k_stride_h;
  int64_t v_stride_b, v_stride_n, v_stride_h;
  int64_t dy_stride_b, dy_stride_n, dy_stride_h;
  float scale, power;
  int dtype, variant;
  float *E, *G, *W2, *P;             // [lanes][N][M]: e, decode softmax, e * slope (stablemax), p
  int seg_len, nseg;
  const float *in_m, *in_d, *in_u;   // exclusive prefix states of the segments; null with one segment
  float *seg_b, *seg_c, *seg_gam;    // replay: carries of the segment alone; reverse: the carries that enter it
  void *dk, *dv;                     // [B, N, H, D] contiguous, input dtype
  float* dq_part;                    // [B * nseg][H][M][Dk]
  const int* gate;                   // optional: nothing is done unless *gate != 0
};
int launch_narrow_replay(const NarrowBwdParams& p, cudaStream_t stream);
int launch_narrow_reverse(const NarrowBwdParams& p, cudaStream_t stream);

}  // namespace flare
