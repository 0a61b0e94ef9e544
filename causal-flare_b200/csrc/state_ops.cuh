// Associative combination of online-softmax states (see state_ops.cu).
#pragma once
#include "flare_common.cuh"

namespace flare {

struct FoldParams {
  // optional left operand (all null: the empty state); one state per lane
  const float *a_m, *a_d, *a_u;
  // `count` states per lane, state j of lane l at index l * lane_stride + j * seg_stride
  float *s_m, *s_d, *s_u;
  int64_t lane_stride, seg_stride;
  int count;
  // mode 0: s[j] <- a (+) s[0] (+) ... (+) s[j-1] in place (exclusive scan; s[count-1] is only written)
  // mode 1: o <- a (+) s[0] (+) ... (+) s[count-1]
  int mode;
  float *o_m, *o_d, *o_u;
  int64_t lanes;
  int M, Dv;
  int stablemax;  // the empty state has m = 0 instead of -inf
  const int* gate;  // optional: the kernel does nothing unless *gate != 0
};

int launch_fold(const FoldParams& p, cudaStream_t stream);

// Copy of a tensor of rows, fp16 <-> bf16 or as it is: n0 x n1 x n2 rows of d contiguous 2-byte elements (d a multiple of 8, row
// starts 16-byte aligned), row (i0, i1, i2) at element offset i0 * s0 + i1 * s1 + i2 * s2 on either side.
struct CastParams {
  const void* in;
  void* out;
  int64_t n0, n1, n2, d;
  int64_t is0, is1, is2;
  int64_t os0, os1, os2;
};

enum Cast { CAST_TO_BF16 = 0, CAST_TO_F16 = 1, CAST_COPY = 2 };
// up to four tensors in one launch, all alike
int launch_cast_rows(const CastParams* p, int count, Cast cast, cudaStream_t stream);

// Compaction of masked rows (2-byte elements, head widths that are multiples of 8, 16-byte aligned rows).
// slot[b][n] = number of valid tokens before token n of row b, or -1 for a masked token; lens[b] = valid tokens of the row.
// start (may be null): start[b] = N - lens[b] for a row whose valid tokens are its last ones (left padding, or none), else -1.
int launch_mask_slots(const int* mask, int B, int N, int* slot, int* lens, int* start, cudaStream_t stream);
// Rows with start[b] >= 0 (start may be null: none) stay where they are: pack skips them, unpack only zeroes their padding.
// pack: out[b][slot[n]] = in[b][n] for the valid tokens of up to two tensors; rows lens[b] .. up to the end of their 128-token
// chunk become zero, later rows stay as they are.  unpack: out[b][n] = in[b][slot[n]], zero for masked tokens.
struct MoveRowsParams {
  const void* in[2];
  void* out[2];
  int64_t is_b[2], is_n[2], is_h[2], os_b[2], os_n[2], os_h[2];
  int d[2];
  int B, N, H, unpack;
  const int *slot, *lens, *start;
};
int launch_move_rows(const MoveRowsParams& p, int tensors, cudaStream_t stream);

}  // namespace flare
