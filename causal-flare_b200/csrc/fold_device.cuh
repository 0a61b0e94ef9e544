// One latent row of a fold / scan of states (state_ops.cu describes it), by one warp.
#pragma once
#include "state_ops.cuh"

namespace flare {
namespace fold {

constexpr int DCH = 4;  // value columns per lane per pass (32 * DCH columns per pass)

__device__ __forceinline__ void merge_factors(float ma, float mb, float& mn, float& fa, float& fb) {
  mn = fmaxf(ma, mb);
  if (mn == kNegInf) {
    fa = 1.f;
    fb = 1.f;
  } else {
    fa = (ma == kNegInf) ? 0.f : __expf(ma - mn);
    fb = (mb == kNegInf) ? 0.f : __expf(mb - mn);
  }
}

// Bound by latency: every state waits for the one before it only in a few multiplications, but a loop that loads a state where
// it needs it waits for memory `count` times.  The next kAhead states are in registers before they are folded.
constexpr int kAhead = 4;
__device__ __forceinline__ void fold_row(const FoldParams& p, int64_t lane_id, int m, int lane) {
  const int M = p.M, Dv = p.Dv;
  const int have = p.mode == 1 ? p.count : p.count - 1;  // states that are folded (a scan does not need the last)
  for (int dv0 = 0; dv0 < Dv; dv0 += 32 * DCH) {
    float rm = p.a_m ? p.a_m[lane_id * M + m] : (p.stablemax ? 0.f : kNegInf);
    float rd = p.a_d ? p.a_d[lane_id * M + m] : 0.f;
    float ru[DCH];
#pragma unroll
    for (int j = 0; j < DCH; ++j) {
      const int dv = dv0 + lane + 32 * j;
      ru[j] = (p.a_u && dv < Dv) ? p.a_u[(lane_id * M + m) * Dv + dv] : 0.f;
    }
    // the statistics are rewritten only in the last column pass: earlier passes still need the originals
    const bool first = (dv0 + 32 * DCH >= Dv) && lane == 0;
    for (int j0 = 0; j0 < p.count; j0 += kAhead) {
      float bm[kAhead], bd[kAhead], bu[kAhead][DCH];
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int64_t sidx = lane_id * p.lane_stride + (int64_t)(j0 + a) * p.seg_stride;
        const bool on = j0 + a < have;
        bm[a] = on ? p.s_m[sidx * M + m] : kNegInf;
        bd[a] = on ? p.s_d[sidx * M + m] : 0.f;
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          const int dv = dv0 + lane + 32 * c;
          bu[a][c] = on && dv < Dv ? p.s_u[(sidx * M + m) * Dv + dv] : 0.f;
        }
      }
      // all lanes of the warp have read the slots before anyone overwrites them
      if (p.mode == 0) __syncwarp();
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int j = j0 + a;
        if (j >= p.count) break;
        if (p.mode == 0) {
          const int64_t sidx = lane_id * p.lane_stride + (int64_t)j * p.seg_stride;
          if (first) {
            p.s_m[sidx * M + m] = rm;
            p.s_d[sidx * M + m] = rd;
          }
#pragma unroll
          for (int c = 0; c < DCH; ++c) {
            const int dv = dv0 + lane + 32 * c;
            if (dv < Dv) p.s_u[(sidx * M + m) * Dv + dv] = ru[c];
          }
        }
        if (j < have) {
          float mn, fa, fb;
          merge_factors(rm, bm[a], mn, fa, fb);
          rm = mn;
          rd = rd * fa + bd[a] * fb;
#pragma unroll
          for (int c = 0; c < DCH; ++c) ru[c] = ru[c] * fa + bu[a][c] * fb;
        }
      }
    }
    if (p.mode == 1) {
      if (first) {
        p.o_m[lane_id * M + m] = rm;
        p.o_d[lane_id * M + m] = rd;
      }
#pragma unroll
      for (int c = 0; c < DCH; ++c) {
        const int dv = dv0 + lane + 32 * c;
        if (dv < Dv) p.o_u[(lane_id * M + m) * Dv + dv] = ru[c];
      }
    }
  }
}

}  // namespace fold
}  // namespace flare
