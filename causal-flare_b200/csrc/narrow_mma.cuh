// Tensor-core kernels for narrow heads at single precision (see narrow_mma.cu).
#pragma once
#include "flare_common.cuh"
#include "narrow_exact.cuh"

namespace flare {

constexpr int kNarrowMmaSegments = 24;  // a CTA folds the states (carries) of all segments before (behind) its own

struct NarrowMmaParams {
  const void *q, *k, *v, *dy;
  int B, N, H, M, Dk, Dv;
  int64_t q_stride_h, q_stride_m;
  int64_t k_stride_b, k_stride_n, k_stride_h;
  int64_t v_stride_b, v_stride_n, v_stride_h;
  int64_t dy_stride_b, dy_stride_n, dy_stride_h;
  float scale;
  int seg_len, nseg;                  // seg_len a multiple of 32
  float *seg_m, *seg_d, *seg_u;       // states of every segment but the last, alone: [lanes][nseg][M], .., [lanes][nseg][M][Dv]
  void* y;
  int64_t y_stride_b, y_stride_n, y_stride_h;
  int* gate;                          // one word for every CTA, written when it ends: 1 if it met values outside its domain
  int gate_stride;                    // forward: words per lane, behind a leading one
  // backward
  int ntiles;                         // tiles of 16 tokens in a lane
  float *stat_c, *stat_d;             // [lanes][ntiles][M]: frame after the tile (log2 units); denominator before the tile, in the frame
                                      // before it, with a minus sign where the tile was taken in several windows
  float *start_c;                     // [lanes][nseg][M]: frame before the segment
  float4* p;                          // [lanes][ntiles][M / 16][2][32]: p = <z_t[m], dY_t>, in the order of a warp's registers
  float *tok_l2, *tok_delta;          // [lanes][ntiles * 16]: decode log-sum-exp (log2 units), <dY_t, y_t>
  float *seg_b, *seg_c;               // [lanes][nseg][M][Dv], [lanes][nseg][M]: carries of the segment alone, in its start frame
  void *dk, *dv;                      // [B, N, H, D] contiguous
  float* dq_part;                     // [B * nseg][H][M][Dk]
};

// What these kernels take: bf16, softmax encoder, token-causal, shared weights, heads up to 32 wide, at most 128 latents, no
// mask and no state on either side (states are returned in fp32: those calls stay on the fp32 kernels).
bool narrow_mma_forward_supported(const flare_fwd_args_t* a);
bool narrow_mma_backward_supported(const flare_bwd_args_t& a);
// sequence segments of a call (`room`: segments per lane that there is scratch for)
void narrow_mma_segments(int64_t lanes, int N, int M, bool backward, int64_t room, int* nseg, int* seg_len);
// seg_*: the segments' states (fp32, [lanes][nseg] of them); gate: 1 + lanes * nseg words
int narrow_mma_forward(const flare_fwd_args_t& f, float* seg_m, float* seg_d, float* seg_u, int nseg, int seg_len, int* gate,
                       cudaStream_t stream);

size_t narrow_mma_backward_bytes(const flare_bwd_args_t& a);
// writes *gate: 1 if the fp32 kernels have to redo the call
int narrow_mma_backward(const flare_bwd_args_t& a, char* ws, int* gate, cudaStream_t stream);

}  // namespace flare
