// Fold / exclusive scan of (m, d, u) states: the chunk-state scan of the segmented prefill, the carry-in
// merge, and the cross-GPU prefix fold all use this one kernel.
//
// (m_a, d_a, u_a) (+) (m_b, d_b, u_b) = (m, d_a e^{m_a-m} + d_b e^{m_b-m}, u_a e^{m_a-m} + u_b e^{m_b-m}),
// m = max(m_a, m_b); a side whose max is -inf contributes with factor 0 (factor 1 if both are -inf).
#include "state_ops.cuh"

#include <string.h>

#include "fold_device.cuh"

namespace flare {

namespace {

constexpr int NT = 128;
constexpr int LAT_PER_CTA = NT / 32;

__global__ void __launch_bounds__(NT) fold_kernel(const FoldParams p) {
  pdl_begin();
  if (p.gate != nullptr && *p.gate == 0) return;
  const int m = blockIdx.y * LAT_PER_CTA + (threadIdx.x >> 5);
  if (m < p.M) fold::fold_row(p, blockIdx.x, m, threadIdx.x & 31);
}

struct CastList {
  CastParams t[4];
};

// blockIdx.y = tensor.  Bound by memory; a tensor that is one dense run needs no index arithmetic (three 64-bit divisions for
// every 16-byte piece otherwise).
template <Cast CAST>
__global__ void __launch_bounds__(256) cast_rows_kernel(const __grid_constant__ CastList list) {
  pdl_begin();
  const CastParams& p = list.t[blockIdx.y];
  const int64_t c8n = p.d >> 3;
  const int64_t total = p.n0 * p.n1 * p.n2 * c8n;
  const bool dense = c8n == total;
  const uint16_t* in = reinterpret_cast<const uint16_t*>(p.in);
  uint16_t* out = reinterpret_cast<uint16_t*>(p.out);
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t io = idx * 8, oo = idx * 8;
    if (!dense) {
      const int64_t c8 = idx % c8n;
      int64_t r = idx / c8n;
      const int64_t i2 = r % p.n2;
      r /= p.n2;
      const int64_t i1 = r % p.n1;
      const int64_t i0 = r / p.n1;
      io = i0 * p.is0 + i1 * p.is1 + i2 * p.is2 + c8 * 8;
      oo = i0 * p.os0 + i1 * p.os1 + i2 * p.os2 + c8 * 8;
    }
    const uint4 x = *reinterpret_cast<const uint4*>(in + io);
    uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (CAST == CAST_TO_F16) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
        const __half2 h = __floats2half2_rn(f.x, f.y);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
      } else if (CAST == CAST_TO_BF16) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    *reinterpret_cast<uint4*>(out + oo) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// One CTA per batch row: ranks by ballots within a warp, then over the warps.
__global__ void __launch_bounds__(1024) mask_slots_kernel(const int* mask, int N, int* slot, int* lens, int* start) {
  pdl_begin();
  __shared__ int sums[32], firsts[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * N;
  int base = 0, first = N;  // first valid token among this thread's
  for (int n0 = 0; n0 < N; n0 += 1024) {
    const int n = n0 + threadIdx.x;
    const bool on = n < N && mask[row + n] != 0;
    if (on && n < first) first = n;
    const unsigned votes = __ballot_sync(0xffffffffu, on);
    __syncthreads();  // (the sums of the tile before have been read)
    if (lane == 0) sums[warp] = __popc(votes);
    __syncthreads();
    int before = base, all = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? sums[w] : 0;
      all += sums[w];
    }
    if (n < N) slot[row + n] = on ? before + __popc(votes & ((1u << lane) - 1u)) : -1;
    base += all;
  }
  if (threadIdx.x == 0) lens[blockIdx.x] = base;
  if (start != nullptr) {
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) firsts[warp] = first;
    __syncthreads();
    if (warp == 0) {
      first = __reduce_min_sync(0xffffffffu, firsts[lane]);
      if (lane == 0) start[blockIdx.x] = first == N - base ? first : -1;
    }
  }
}

// A streaming copy of 16-byte pieces, both tensors of a pack in one launch (blockIdx.z).  Bound by memory: every valid row is
// read and written once.  One block takes kMoveTokens tokens of a batch row (blockIdx.y): a call whose rows all stay where
// they are is a few hundred blocks that return at once, and the index arithmetic stays a few 32-bit operations.
constexpr int kMoveTokens = 16;
__global__ void __launch_bounds__(256) move_rows_kernel(const MoveRowsParams p) {
  pdl_begin();
  const int w = blockIdx.z, b = blockIdx.y;
  const int first = p.start != nullptr ? p.start[b] : -1;
  const int n0 = blockIdx.x * kMoveTokens, n1 = min(p.N, n0 + kMoveTokens);
  if (first >= 0 && (!p.unpack || n0 >= first)) return;
  const uint16_t* in = reinterpret_cast<const uint16_t*>(p.in[w]) + b * p.is_b[w];
  uint16_t* out = reinterpret_cast<uint16_t*>(p.out[w]) + b * p.os_b[w];
  const int* slot = p.slot + (int64_t)b * p.N;
  const int c8n = p.d[w] >> 3, pieces = p.H * c8n;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const int len = p.unpack ? 0 : p.lens[b];
  for (int i = threadIdx.x; i < (n1 - n0) * pieces; i += 256) {
    const int t = i / pieces, n = n0 + t, r = i - t * pieces;
    const int h = r / c8n, c = (r - h * c8n) * 8;
    const int s = slot[n];
    const uint16_t* src = in + h * p.is_h[w] + c;
    uint16_t* dst = out + h * p.os_h[w] + c;
    if (p.unpack) {
      if (s < 0) *reinterpret_cast<uint4*>(dst + n * p.os_n[w]) = zero;
      else if (first < 0) *reinterpret_cast<uint4*>(dst + n * p.os_n[w]) = *reinterpret_cast<const uint4*>(src + s * p.is_n[w]);
    } else {
      if (s >= 0) *reinterpret_cast<uint4*>(dst + s * p.os_n[w]) = *reinterpret_cast<const uint4*>(src + n * p.is_n[w]);
      if (n >= len && n < (len + 127) / 128 * 128) *reinterpret_cast<uint4*>(dst + n * p.os_n[w]) = zero;
    }
  }
}

}  // namespace

int launch_mask_slots(const int* mask, int B, int N, int* slot, int* lens, int* start, cudaStream_t stream) {
  LaunchTimer timer("mask_slots_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(mask_slots_kernel, dim3((unsigned)B), dim3(1024), 0, stream, mask, N, slot, lens, start));
  return FLARE_OK;
}

int launch_move_rows(const MoveRowsParams& p, int tensors, cudaStream_t stream) {
  if ((int64_t)p.B * p.N > 0x7fffffff) return FLARE_ERR_UNSUPPORTED;
  for (int w = 0; w < tensors; ++w)
    if (p.d[w] % 8) return FLARE_ERR_BAD_SHAPE;
  LaunchTimer timer(p.unpack ? "move_rows_kernel (unpack)" : "move_rows_kernel (pack)", stream);
  const unsigned blocks = (unsigned)((p.N + kMoveTokens - 1) / kMoveTokens);
  MoveRowsParams q = p;
  for (int b0 = 0; b0 < p.B; b0 += 65535) {  // (what grid.y holds)
    q.B = p.B - b0 < 65535 ? p.B - b0 : 65535;
    FLARE_CUDA_CHECK(launch_pdl(move_rows_kernel, dim3(blocks, (unsigned)q.B, tensors), dim3(256), 0, stream, q));
    q.slot += (int64_t)65535 * p.N;
    if (q.lens != nullptr) q.lens += 65535;
    if (q.start != nullptr) q.start += 65535;
    for (int w = 0; w < tensors; ++w) {
      q.in[w] = reinterpret_cast<const uint16_t*>(q.in[w]) + 65535 * p.is_b[w];
      q.out[w] = reinterpret_cast<uint16_t*>(q.out[w]) + 65535 * p.os_b[w];
    }
  }
  return FLARE_OK;
}

int launch_cast_rows(const CastParams* p, int count, Cast cast, cudaStream_t stream) {
  CastList list;
  memset(&list, 0, sizeof(list));
  int64_t most = 0;
  for (int i = 0; i < count; ++i) {
    CastParams c = p[i];
    if (c.d % 8) return FLARE_ERR_BAD_SHAPE;
    // rows that lie behind one another on both sides become one longer row
    for (int level = 0; level < 3 && (c.n2 == 1 || (c.is2 == c.d && c.os2 == c.d)); ++level) {
      c.d *= c.n2;
      c.n2 = c.n1; c.is2 = c.is1; c.os2 = c.os1;
      c.n1 = c.n0; c.is1 = c.is0; c.os1 = c.os0;
      c.n0 = 1;
    }
    const int64_t total = c.n0 * c.n1 * c.n2 * (c.d >> 3);
    if (total > most) most = total;
    list.t[i] = c;
  }
  if (most <= 0) return FLARE_OK;
  int64_t blocks = (most + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  const char* const names[] = {"cast_rows_kernel<fp16 to bf16>", "cast_rows_kernel<bf16 to fp16>", "cast_rows_kernel<copy>"};
  auto* const kernel = cast == CAST_COPY ? cast_rows_kernel<CAST_COPY>
                                         : (cast == CAST_TO_F16 ? cast_rows_kernel<CAST_TO_F16> : cast_rows_kernel<CAST_TO_BF16>);
  LaunchTimer timer(names[cast], stream);
  FLARE_CUDA_CHECK(launch_pdl(kernel, dim3((unsigned)blocks, count), dim3(256), 0, stream, list));
  return FLARE_OK;
}

int launch_fold(const FoldParams& p, cudaStream_t stream) {
  if (p.lanes <= 0 || p.count <= 0) return FLARE_OK;
  dim3 grid((unsigned)p.lanes, (p.M + LAT_PER_CTA - 1) / LAT_PER_CTA);
  LaunchTimer timer("fold_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(fold_kernel, grid, dim3(NT), 0, stream, p));
  return FLARE_OK;
}

}  // namespace flare
