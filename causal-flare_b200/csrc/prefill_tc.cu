// Tensor-core (tcgen05 + TMEM + TMA) chunked causal prefill, bf16 operands, fp32 accumulation and statistics.
// Shape class: M <= 512 latents (multiple of 16, in groups of 128 rows, the last one padded), (Dk, Dv) = (64, 64),
// (128, 128) or (64, 128), shared decode weights; softmax encoder token- or block-causal, stablemax encoder
// token-causal; optional per-row lengths (right padding).
//
// One CTA owns a (batch, head, sequence segment, slice of 64 value columns, group of 128 latents) and walks its chunks
// of C = 128 tokens in order ((128, 128) heads on a grid that would not fit the SMs at once: one CTA for all 128
// value columns, the "wide" instance below).  With more than one latent group every CTA emits a partial read-out
// (normalised over its own latents, fp16) and the log2 of its weight mass per token; a small kernel merges the
// groups.  Read-out rows leave the CTA as tiled bulk stores of 32 x 32 tiles staged in shared memory.  The CTA carries the
// latent state on chip: U [128 latents x 64] fp32 in tensor memory, the latent bank Q in shared memory (Dk = 64) or
// as packed bf16 in tensor memory (Dk = 128; A operand of the score MMA), running max c and denominator d per latent
// in registers of the thread that owns the latent (TMEM lane = thread).  Per chunk, with the frame c_m = running
// max after the chunk and kappa = max_m c_m:
//
//   S^T = Q K_c^T                          MMA1  (128 x 128, k = 64)      latents on lanes, tokens on columns
//   E[m,t]   = exp(s[m,t] - c_m)           one exp per element, thread m scans its row
//   D[m,t]   = d_m + cumsum_t E[m,t]       (d_m already rescaled into the new frame)
//   R[m,t]   = E[m,t] exp(c_m - kappa) / D[m,t]        = softmax-numerator / encoder denominator
//   [W | Y | Den0] = R^T [E | U_bf16 | d]   MMA2  ONE product of width 208 (256 with two value blocks, Den0 separate):
//                                                  W = R^T E (tokens x tokens), Y = R^T U_bf16, Den0 = R^T d
//   W -> causal mask + bf16, written back to TMEM (token group)
//   U   += E V_c                           MMA3
//   Y   += tril(W) V_c                     MMA4  (A operand from TMEM)
//   y_t  = Y[t,:] / (Den0[t] + rowsum tril(W)[t,:])
//
// Operands E, R (written by the latent threads row-wise) feed MMAs both K-major and MN-major from the same
// 128-byte-swizzled buffers, so no transposition pass exists.  E, the bf16 copy of the state and the block whose
// column 0 is d lie behind one another in shared memory, so that they form ONE MN-major B operand and R is read once
// for all three products (28 MMA instructions per chunk at Dk = 64 instead of 44: every instruction costs 100-190
// cycles from issue to issue in this kernel whatever its width, 60-100 where an elected thread issues, 49-130 alone).
//
// Warp roles (14 warps): 0-7 "latent group" (two warps per lane quarter, each half of the chunk's tokens): scores ->
// E, R, state rescale (chunk i+1);  8-11 "token group": causal mask of W, normalisation and store of Y (chunk i);
// 12: MMA issuer (one thread);  13: TMA producer (one thread);  training: 14 stores the kept states.  The three stages
// work on consecutive chunks concurrently.  E and R have one buffer each (every product that reads them is issued when the latent group has
// finished the chunk; the latent group waits for the state update of the previous chunk before it writes E), the
// accumulators [W | Y | Den0] are single and go back to the MMA issuer as soon as the token group has them in
// registers, K is single-buffered (free as soon as its score MMA has run), V has two stages.
#include "prefill_tc.cuh"

#include <cuda.h>
#include <stdlib.h>
#include <string.h>

#include "sm100_ptx.cuh"
#include "tc_device.cuh"

// polling rounds of every wait of the prefill kernel before it suspends (see tc::wait_or_abort)
#ifndef FLARE_TC_FWD_POLLS
#define FLARE_TC_FWD_POLLS 24
#endif

namespace flare {

using namespace sm100;

namespace {

constexpr int C = 128;    // tokens per chunk
constexpr int M = 128;    // latents
constexpr int D = 64;     // value columns per CTA, and width of one 128-byte operand block
// (keep: a warp that stores the kept states)
constexpr int nthreads(bool keep) { return keep ? 480 : 448; }
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// shared memory map (bytes, every operand buffer 1024-aligned for the 128B swizzle)
// DKB = Dk / 64 = number of 64-wide key blocks
// WIDE: one CTA handles both 64-column value blocks of Dv = 128 (Dk = 128 only), see the kernel's comment
template <int DKB, bool WIDE = false>
struct Lay {
  static_assert(!WIDE || DKB == 2, "the wide instance is the (128, 128) head shape");
  // Dk = 64: the latent bank stays in shared memory (TMA-loaded); Dk = 128 has no room for it there and keeps it in
  // tensor memory as the A operand of the score MMA
  static constexpr bool Q_SMEM = DKB == 1;
  // Every product that reads R (W, Y0, Den0) is ONE tcgen05.mma sequence over a B operand of adjacent 64-wide
  // MN-major blocks [E t-block 0 | E t-block 1 | U_bf16 ... | d], issued when the latent group has finished a chunk:
  // R is read once, and E and R need one buffer each (free long before the next chunk writes them).
  static constexpr int VB = WIDE ? 2 : 1;                  // 64-column value blocks per CTA
  static constexpr int OFF_Q = 0;                          // [128 m][64] bf16, K-major                 16 KB or 0
  static constexpr int OFF_K = Q_SMEM ? 16384 : 0;         // DKB x [128 t][64] bf16                    16 KB each
  static constexpr int OFF_V = OFF_K + DKB * 16384;        // 2 stages x [VB value blocks][128 t][64]   16 KB each
  static constexpr int OFF_E = OFF_V + 2 * VB * 16384;     // [2 t-blocks][128 m][64 t] bf16            32 KB
  // merged product: the bf16 state operand follows E directly; with one value block the denominator follows as a
  // fourth MN-major block [128 m][64] of which column 0 holds d (product width 128 + 64 + 16 = 208); with two value
  // blocks the width is 256 already and Den0 stays a product of its own over the small K-major d tile
  static constexpr int OFF_U = OFF_E + 32768;              // [VB][128 m][64 dv] bf16                    16 KB each
  static constexpr int OFF_B16 = OFF_U + VB * 16384;       // d: MN-major block 16 KB, or (wide) the K-major tile
                                                           // [2 m-blocks][16 n][64 m] 4 KB
  static constexpr int D_BYTES = WIDE ? 4096 : 16384;
  static constexpr int OFF_R = OFF_B16 + D_BYTES;          // [2 t-blocks][128 m][64 t] bf16              32 KB
  static constexpr int OFF_MISC = OFF_R + 32768;           // barriers, tmem slot, reductions          4608 B
  static constexpr int OFF_STAGE = OFF_MISC + 4608;        // 4 token warps x [32 t][32 columns] 16-bit: source of the
                                                           // read-out's bulk stores (64-byte swizzle)     8 KB
  // wide, two latent groups merged on chip: the partner CTA's normalised partial rows of the value block this CTA
  // finalises, [128 t][64] fp16 (16-byte pieces swizzled by row), and the log2 weight mass per row
  static constexpr int OFF_XCH = OFF_STAGE + 8192;         //                                          16 KB + 512 B
  static constexpr int OFF_KEEP = (OFF_XCH + 1023) / 1024 * 1024;  // training (not wide): the chunk's kept state, [128 m][64] bf16
  static constexpr int smem_bytes(bool keep) {  // + slack for manual 1024-byte alignment
    return (keep ? OFF_KEEP + 16384 : OFF_XCH + (WIDE ? 16384 + 512 : 0)) + 1024;
  }
  static_assert(smem_bytes(!WIDE) <= 232448, "shared memory");
  // tensor-memory columns.  [W | Y | Den] are adjacent (one product writes them); single accumulators, handed back by
  // the token group as soon as it has them in registers.  Wide: W shares the columns of S (the latent group has the
  // next chunk's scores in registers before W of this chunk is written) and U takes 128 columns.
  static constexpr uint32_t TM_S = 0, TM_W = WIDE ? 0 : 128, TM_Y = TM_W + 128, TM_DEN = WIDE ? 384 : TM_Y + 64,
                            TM_U = WIDE ? 256 : TM_DEN + 16, TM_Q = WIDE ? 400 : TM_U + 64 /* packed bf16 (Dk = 128 only) */;
  static_assert(TM_Q + (Q_SMEM ? 0 : DKB * 32) <= 512, "tensor memory columns");
};
constexpr uint32_t TM_COLS = 512;

struct Misc {
  uint64_t q_full, k_full, k_empty, v_full[2], v_empty[2], v_conv[2];
  uint64_t keep_free, s_ready, s_free, kap_done, p1_done, u_done, w_ready, p2_done, y_ready, y_free;
  uint64_t pmax[4], psum[4];  // pair barriers of the two latent half-groups, one per lane quarter
  uint64_t xfull[4], xfree[4];  // on-chip merge of two latent groups, per token warp: the partner's rows have arrived /
                                // the partner has read the rows this CTA sent
  uint32_t tmem_base;
  volatile int abort_flag;
  volatile int out_of_domain;  // some token of this CTA left the numeric domain
  float wmax[4][4];  // (the packed instance uses four slots, the others two: see there)
  float kap[4];  // decode frame of chunk i in slot i % 4, for the token group (log-sum-exp, weight mass of a latent group)
  // exchange of the token parts' row maxima and sums of E: [chunk parity][part][latent]
  union {
    struct {
      float xmax[2][2][128], xsum[2][2][128];
    };
    float x4[2][2][4][64];  // packed instance: (maxima, sums)
  };
};


// optional cycle trace of CTA (0, 0): [role][chunk < 16][slot < 8] clock64 stamps (diagnostic hook, null in normal use)
#define TC_TRACE(role, chunk, slot)                                                                   \
  do {                                                                                                \
    if (p.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (chunk) < 16)                   \
      p.trace[((role) * 16 + (chunk)) * 8 + (slot)] = clock64();                                      \
  } while (0)

using tc::swz_chunk_off;
using tc::warp_arrive;
using tc::sigma8;

// bounded wait that also gives up as soon as another role of the CTA has given up
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, Misc* misc) {
  return tc::wait_or_abort(bar, parity, &misc->abort_flag, FLARE_TC_FWD_POLLS);
}

// eight of a thread's values (fp32 bits) as bf16
__device__ __forceinline__ uint4 pack_piece(const uint32_t (&r)[32], int ch) {
  return make_uint4(pack_bf16(__uint_as_float(r[ch * 8 + 0]), __uint_as_float(r[ch * 8 + 1])),
                    pack_bf16(__uint_as_float(r[ch * 8 + 2]), __uint_as_float(r[ch * 8 + 3])),
                    pack_bf16(__uint_as_float(r[ch * 8 + 4]), __uint_as_float(r[ch * 8 + 5])),
                    pack_bf16(__uint_as_float(r[ch * 8 + 6]), __uint_as_float(r[ch * 8 + 7])));
}

// The store of the block-causal wide instance with latent groups.  Through the kernel's store_e, which computes the address
// itself, this one instance spills more (88 bytes of loads instead of 72) and takes 2087 instead of 1992 us at B=2 N=65536 H=32
// M=256 D=128 with blocks of 64; the others spill less with store_e (the wide one without groups 0 instead of 36 bytes).
__device__ __forceinline__ void put_piece(uint8_t* at, const uint4& v) { *reinterpret_cast<uint4*>(at) = v; }

// eight values as fp16 or bf16 pairs
__device__ __forceinline__ void pack_out(const float (&y)[8], bool f16, uint32_t (&o)[4]) {
  if (f16) {
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = pack_f16(y[2 * j], y[2 * j + 1]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = pack_bf16(y[2 * j], y[2 * j + 1]);
  }
}

// grid.z = latent group * DKB + value slice.  First value column of this CTA's slice (a compile-time zero when there
// is one slice) and first latent of its group (zero without the latent split).
template <int DVB, bool SPLIT>
__device__ __forceinline__ int value_col0() {
  return DVB == 1 ? 0 : (SPLIT ? (int)blockIdx.z % DVB : (int)blockIdx.z) * D;
}
template <int DVB, bool SPLIT>
__device__ __forceinline__ int latent0() {
  return SPLIT ? ((int)blockIdx.z / DVB) * M : 0;
}

}  // namespace

// The kernel instances are compiled in separate translation units (FLARE_TC_UNIT = 0..7: head widths (64, 64) / (128, 128) / (64, 128), without /
// with the latent-group split, and the wide ones; FLARE_TC_MODE = 0..2) to keep build times short; the unit without
// FLARE_TC_UNIT holds the host side.
template <int UNIT, int MODE>
int launch_prefill_tc_unit(int lat, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& ty, const CUtensorMap* in,
                           const TcParams& p, dim3 grid, cudaStream_t stream);

#ifdef FLARE_TC_UNIT


// LAT: 0 = groups of 128 latents, 1 = the (last) group is padded, 2 = at most 64 latents (PACK).  The full-width instance
//        carries none of the padding predicates.
// PACK: at most 64 latents would leave half of the 128 tensor-memory lanes, and with them half of the latent warps, without
//        work.  The latent bank is laid down twice (rows 0..63 and 64..127), so the score product gives every latent's
//        scores on two lanes, and a thread takes 32 tokens of the chunk instead of 64: four warps per 32 latents, the two
//        of the lower lanes the even quarters of the chunk, the two of the upper lanes the odd ones.  E is stored on both
//        rows, so both lanes carry the state; each lane maintains half of its columns (the others are never read).
//        Products over the latents take four 16-latent steps instead of eight.
// SPLIT: more than 128 latents, partial read-outs
// BLOCK: block-causal (semi-autoregressive) read-out with blocks of 16, 32, 64 or 128 tokens: a token reads the state
//        at the end of its block, so the denominator of a block's tokens is the one at the block's end and the mask
//        of W is "column <= end of the row's block"
// MODE 2 (STABLE): stablemax encoder weights sigma(s) = (1+s)^p | (1-s)^-p.  The encoder side then has no frames
//        (E = sigma(s), D = plain running sum, the state is never rescaled); the decode weights stay a softmax over
//        the latents, whose numerator exp2(s - c) a_m is formed with the same running-max machinery as before.
// DVB = Dv / 64 = number of value slices (grid.z); Dv may differ from Dk (Dk = 64 with Dv = 128)
// KEEP: training forward that leaves the per-chunk prefix states for the backward pass (a separate instance: the
//       extra live values cost the register-capped latent group about 5 % when the code is merely present)
// WIDE: (Dk, Dv) = (128, 128) with ONE CTA per (lane, latent group) that carries all 128 value columns, instead of two
//       CTAs that each repeat the score / E / R work for 64 of them.  Used when the two-slice grid would not fit the
//       SMs in one wave.  Differences: U and Y are 128 columns wide; W and Y0 = R^T U_bf16 come out of ONE product of
//       width 256 ([E | U_bf16] as one B operand, [W | Y] adjacent in tensor memory), so R is read once for both; W
//       shares the columns of S; E and R are single-buffered.
// FL:   0 = bf16, every row N tokens long; 1 = bf16 with per-row lengths and, of a masked call, rows that were not packed;
//       2 = fp16, with lengths or not.  Instances of their own: as run-time choices they cost every bf16 call 2 to 3 % (B200:
//       B=8 N=8192 H=16 M=128 D=64 182.3 -> 185.8 us, training B=4 N=4096 H=16 M=64 D=128 411 -> 424 us), and the type of y in
//       the epilogue of the wide instance 5 to 8 %.
template <int LAT, int DKB, int DVB, bool SPLIT, int MODE, bool KEEP, bool WIDE, int FL>
__global__ void __launch_bounds__(nthreads(KEEP && !WIDE), 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_y,
                  const __grid_constant__ CUtensorMap tm_k_in, const __grid_constant__ CUtensorMap tm_v_in, const TcParams p) {
  using L = Lay<DKB, WIDE>;
  constexpr bool PADDED = LAT != 0, PACK = LAT == 2;
  static_assert(!WIDE || (DVB == 2 && !PADDED), "wide instance");
  static_assert(!KEEP || FL == 0, "training forwards are bf16 and know no lengths");
  constexpr bool LENS = FL != 0, F16 = FL == 2;
  static_assert(!PACK || !SPLIT, "one group of at most 64 latents");
  // The kept states leave through a bulk store of the chunk's tile by a warp of its own (its tensor map comes as tm_k_in, which no
  // training forward needs).  Stored by the latent threads, 32 bytes of a row each (512 transactions a chunk, packed), they made
  // the state pass of a chunk 1 300 instead of 350 cycles.  B200, us a training step: B=4 N=4096 H=16 M=128 D=64 442 -> 432, M=64
  // D=128 354 -> 348, B=2 N=2048 M=256 D=128 288 -> 283.  (Wide: no room for the tile.)
  constexpr bool KEEP_TILE = KEEP && !WIDE;
  constexpr int NTHREADS = nthreads(KEEP_TILE);
  constexpr int NP = PACK ? 4 : 2;       // token parts of a chunk = latent warps per 32 latents
  constexpr int TOK = C / NP;            // tokens per latent thread
  constexpr int ROWS = PACK ? 64 : 128;  // latent rows of the operand buffers that the products over the latents read
  constexpr int KSM = ROWS / 16;         // their 16-latent steps
  constexpr int WS = PACK ? 4 : 2;       // slots of the frame maximum's exchange
  // The elected thread issues a chunk's products in 2 700 instead of 3 700 cycles (see elect_one).  B200, us, lane 0 -> elected, medians
  // that move by up to 0.5 % from run to run.  Packed: B=1 N=777 H=16 M=64 D=64 20.7 -> 19.4, fp16 B=4 N=4096 H=16 M=64 D=128 88.9 ->
  // 83.6.  Wide: block-causal B=2 N=65536 H=32 M=256 D=128 2 024 -> 1 949.  Whole groups at (64, 64), H=16 M=128: stablemax B=8 N=8192
  // 442.9 -> 423.3, fp16 193.8 -> 187.4, bf16 175.6 -> 175.4, B=1 N=3000 36.9 -> 36.3, B=2 N=1000 H=8 27.6 -> 27.9, training B=4 N=4096
  // 435.5 -> 428.9.  The others keep lane 0: with 64 tokens a thread the latent warps are the longest chain by far, and products that
  // follow one another faster may get in their way as well as help them (two slices, M=128 D=128: B=4 N=4096 H=8 91.7 -> 94.4, B=1
  // N=3000 H=16 51.1 -> 49.3; B=4 N=4096 H=16 M=192 D=64 120.8 -> 121.5, M=96 89.9 -> 90.2, M=96 D=128 96.8 -> 94.3).
  constexpr bool ELECT = PACK || WIDE || (LAT == 0 && DKB == 1 && DVB == 1 && !SPLIT);
  constexpr int ZS = WIDE ? 1 : DVB;  // value slices on grid.z
  constexpr bool XM = WIDE && SPLIT && FL != 1;  // may merge two latent groups on chip (never in a call with lengths)
  constexpr bool BLOCK = MODE == 1, STABLE = MODE == 2;
  constexpr int OFF_K = L::OFF_K, OFF_V = L::OFF_V, OFF_E = L::OFF_E, OFF_R = L::OFF_R, OFF_U = L::OFF_U,
                OFF_B16 = L::OFF_B16, OFF_Q = L::OFF_Q, OFF_MISC = L::OFF_MISC, VB = L::VB, D_BYTES = L::D_BYTES;
  constexpr bool Q_SMEM = L::Q_SMEM;
  constexpr uint32_t TM_S = L::TM_S, TM_W = L::TM_W, TM_U = L::TM_U, TM_Y = L::TM_Y, TM_DEN = L::TM_DEN, TM_Q = L::TM_Q;
  pdl_wait();
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + OFF_MISC);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, seg = blockIdx.y;
  // This CTA's slice of the value columns starts at blockIdx.z * D (a compile-time zero when Dv = 64); the
  // roles read it where they need it instead of keeping it in a register across their chunk loops, because the
  // latent group runs at the register cap and an extra live value there cost 4 % of the kernel's time.
  constexpr int DV = DVB * D;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int seg_begin = seg * p.seg_len;
  // rows beyond the batch row's own length are right padding: they are not walked
  const int n_row = LENS && p.lens != nullptr ? min(p.N, max(0, p.lens[b])) : p.N;
  const int seg_end = max(seg_begin, min(n_row, seg_begin + p.seg_len));
  const int nchunks = (seg_end - seg_begin + C - 1) / C;

  if (tid == 0) {
    mbar_init(&misc->q_full, Q_SMEM ? 1 : 8);
    mbar_init(&misc->k_full, 1);
    mbar_init(&misc->k_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&misc->v_full[i], 1);
      mbar_init(&misc->v_empty[i], 1);
      mbar_init(&misc->v_conv[i], 1);
    }
    mbar_init(&misc->keep_free, 1);
    mbar_init(&misc->s_ready, 1);
    mbar_init(&misc->s_free, 8);
    mbar_init(&misc->kap_done, 4);
    mbar_init(&misc->p1_done, 8);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&misc->pmax[i], NP);
      mbar_init(&misc->psum[i], NP);
    }
    mbar_init(&misc->u_done, 1);
    mbar_init(&misc->w_ready, 1);
    mbar_init(&misc->p2_done, 4);
    mbar_init(&misc->y_ready, 1);
    mbar_init(&misc->y_free, 4);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&misc->xfull[i], 1);
      mbar_init(&misc->xfree[i], 32);
    }
    misc->abort_flag = 0;
    misc->out_of_domain = 0;
    fence_barrier_init();
  }
  // zero the denominator operand tile once (rows 1..15 stay zero for the whole kernel)
  for (int i = tid; i < D_BYTES / 16; i += NTHREADS) reinterpret_cast<uint4*>(smem + OFF_B16)[i] = make_uint4(0, 0, 0, 0);

  if (warp == 12) {
    tmem_alloc(&misc->tmem_base, TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // on-chip merge: the partner CTA arrives on this CTA's barriers, which must be initialised first
  const bool xmerge = XM && p.cluster_merge != 0;
  if (xmerge) cluster_sync_all();
  const uint32_t tmem = misc->tmem_base;
  bool ok = true;
  // No read-out wanted (segment states for a scan, prefix states): only E and U += E V are computed; R, W, the
  // read-out MMAs and the token group are skipped.
  const bool state_only = p.y == nullptr;

  if (warp == 13) {
    // ======================================= TMA producer =======================================
    if constexpr (FL == 0) {
      if (ELECT ? elect_one() : lane == 0) {
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
        if (Q_SMEM) {
          mbar_arrive_expect_tx(&misc->q_full, 16384);
          tma_load_3d(smem + OFF_Q, &tm_q, &misc->q_full, 0, latent0<ZS, SPLIT>(), h);  // rows beyond M read as zero
          if (PACK) tma_load_3d(smem + OFF_Q + 8192, &tm_q, &misc->q_full, 0, 0, h);    // (boxes of 64 rows)
        }
        const int vc0 = value_col0<ZS, SPLIT>();
        for (int i = 0; ok && i < nchunks; ++i) {
          const int t0 = seg_begin + i * C;
          // K tile: free once the score MMA of the previous chunk has run
          if (i > 0 && !(ok = wait_or_abort(&misc->k_empty, (i - 1) & 1, misc))) break;
          mbar_arrive_expect_tx(&misc->k_full, DKB * 16384);
#pragma unroll
          for (int kb = 0; kb < DKB; ++kb) tma_load_4d(smem + OFF_K + kb * 16384, &tm_k, &misc->k_full, kb * 64, h, t0, b);
          // V tile: stage i & 1, free once chunk i - 2 has been folded into Y
          const int st = i & 1;
          if (i >= 2 && !(ok = wait_or_abort(&misc->v_empty[st], ((i - 2) >> 1) & 1, misc))) break;
          mbar_arrive_expect_tx(&misc->v_full[st], VB * 16384);
#pragma unroll
          for (int vb = 0; vb < VB; ++vb)
            tma_load_4d(smem + OFF_V + (st * VB + vb) * 16384, &tm_v, &misc->v_full[st], vc0 + vb * 64, h, t0, b);
        }
      }
    } else {
      // fp16 inputs: Q and K go to the score product as they are; V, which meets bf16 weights, is rounded to bf16 in place by
      // this warp (one tile behind the loads, so that the next chunk's K never waits for it).  B200, B=4 N=4096 H=16 M=64 D=128:
      // 130 us with bf16 copies of K and V made before the kernel (a pass of 42 us over them), 93 us this way.
      constexpr unsigned active = F16 ? 0xffffffffu : 1u;  // (bf16: the one thread that issues the loads)
      auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(active, wait_or_abort(bar, parity, misc)) != 0; };
      auto convert_v = [&](int i) -> bool {
        const int st = i & 1;
        if (!wait_all(&misc->v_full[st], (i >> 1) & 1)) return false;
        uint4* tile = reinterpret_cast<uint4*>(smem + OFF_V + st * VB * 16384);
#pragma unroll 1
        for (int c = lane; c < VB * 1024; c += 32 * 8) {
          uint4 x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = tile[c + u * 32];
#pragma unroll
          for (int u = 0; u < 8; ++u) tile[c + u * 32] = make_uint4(f16x2_to_bf16x2(x[u].x), f16x2_to_bf16x2(x[u].y),
                                                                    f16x2_to_bf16x2(x[u].z), f16x2_to_bf16x2(x[u].w));
        }
        fence_proxy_async_smem();
        warp_arrive(&misc->v_conv[st], lane);
        return true;
      };
      if (lane == 0 || F16) {
        const int vc0 = value_col0<ZS, SPLIT>();
        // a row of a masked call that was not packed: its tokens are the last ones of the caller's row
        const int row0 = p.row_start != nullptr ? p.row_start[b] : -1;
        const CUtensorMap* const mk = row0 >= 0 ? &tm_k_in : &tm_k;
        const CUtensorMap* const mv = row0 >= 0 ? &tm_v_in : &tm_v;
        if (lane == 0) {
          prefetch_tensormap(mk);
          prefetch_tensormap(mv);
          if (Q_SMEM) {
            mbar_arrive_expect_tx(&misc->q_full, 16384);
            tma_load_3d(smem + OFF_Q, &tm_q, &misc->q_full, 0, latent0<ZS, SPLIT>(), h);  // rows beyond M read as zero
            if (PACK) tma_load_3d(smem + OFF_Q + 8192, &tm_q, &misc->q_full, 0, 0, h);    // (boxes of 64 rows)
          }
        }
        for (int i = 0; ok && i < nchunks; ++i) {
          const int t0 = seg_begin + i * C + max(row0, 0);
          // K tile: free once the score MMA of the previous chunk has run
          if (i > 0 && !(ok = wait_all(&misc->k_empty, (i - 1) & 1))) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(&misc->k_full, DKB * 16384);
#pragma unroll
            for (int kb = 0; kb < DKB; ++kb) tma_load_4d(smem + OFF_K + kb * 16384, mk, &misc->k_full, kb * 64, h, t0, b);
          }
          if (F16 && i > 0 && !(ok = convert_v(i - 1))) break;
          // V tile: stage i & 1, free once chunk i - 2 has been folded into Y
          const int st = i & 1;
          if (i >= 2 && !(ok = wait_all(&misc->v_empty[st], ((i - 2) >> 1) & 1))) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(&misc->v_full[st], VB * 16384);
#pragma unroll
            for (int vb = 0; vb < VB; ++vb)
              tma_load_4d(smem + OFF_V + (st * VB + vb) * 16384, mv, &misc->v_full[st], vc0 + vb * 64, h, t0, b);
          }
        }
        if (F16 && ok && nchunks > 0) ok = convert_v(nchunks - 1);
      }
    }
  } else if (KEEP_TILE && warp == 14) {
    // ======================================= kept states =======================================
    if (elect_one()) {
      prefetch_tensormap(&tm_k_in);
      for (int i = 0; ok && i < nchunks; ++i) {
        if (!(ok = wait_or_abort(&misc->p1_done, i & 1, misc))) break;
        tma_store_4d(&tm_k_in, smem + L::OFF_KEEP, value_col0<ZS, SPLIT>(), latent0<ZS, SPLIT>(), seg_begin / C + i, lane_id);
        bulk_commit_group();
        bulk_wait_group_read0();
        mbar_arrive(&misc->keep_free);
      }
      bulk_wait_group0();
    }
  } else if (warp == 12) {
    // ======================================= MMA issuer =======================================
    if (ELECT ? elect_one() : lane == 0) {
      const uint32_t k_addr = smem_u32(smem + OFF_K);
      const uint32_t b16_addr = smem_u32(smem + OFF_B16);
      // Q (TMEM) x K_c (K-major): both as the caller has them, bf16 or fp16
      constexpr uint32_t ID_S = F16 ? make_idesc_f16(128, 128, 0, 0) : make_idesc_bf16(128, 128, 0, 0);
      uint64_t* const v_ready = F16 ? misc->v_conv : misc->v_full;  // the V tile is in place, as bf16
      constexpr uint32_t ID_U = make_idesc_bf16(128, WIDE ? 128 : 64, 0, 1);  // E (K-major) x V (MN-major)
      constexpr uint32_t ID_DEN = make_idesc_bf16(128, 16, 1, 0);  // R (MN-major) x d tile (K-major)
      constexpr uint32_t ID_Y1 = make_idesc_bf16(128, WIDE ? 128 : 64, 0, 1);  // tril(W) (TMEM) x V (MN-major)
      // merged: R (MN-major) x [E | U_bf16 (| d)] (MN-major), width 256 with two value blocks, 208 with one
      constexpr uint32_t ID_WY = make_idesc_bf16(128, WIDE ? 256 : 208, 1, 1);

      // descriptors are built once; inside the loops only the start-address field (units of 16 bytes) advances
      const uint64_t dk = make_desc_sw128(k_addr, 16, 1024);
      const uint64_t dq = make_desc_sw128(smem_u32(smem + OFF_Q), 16, 1024);
      const uint64_t db16 = make_desc_sw128(b16_addr, 16, 1024);
      // second buffer of a double-buffered operand = first + its byte distance (in 16-byte units)
      const uint64_t de_k0 = make_desc_sw128(smem_u32(smem + OFF_E), 16, 1024);
      const uint64_t de_mn0 = make_desc_sw128(smem_u32(smem + OFF_E), 16384, 1024);
      const uint64_t dr_mn0 = make_desc_sw128(smem_u32(smem + OFF_R), 16384, 1024);
      // (wide: the two 64-column value blocks are 16384 bytes apart, the leading-dimension stride of the N = 128 operand)
      const uint64_t dv_mn0 = make_desc_sw128(smem_u32(smem + OFF_V), WIDE ? 16384 : 1024, 1024);
      constexpr int V_STAGE = VB * 16384;

      auto issue_scores = [&](int i) -> bool {  // S^T of chunk i; K tile and the S columns must be free
        if (!wait_or_abort(&misc->k_full, i & 1, misc)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int j = 0; j < 4 * DKB; ++j) {
          const uint64_t dkj = dk + (((j >> 2) * 16384 + (j & 3) * 32) >> 4);
          if (Q_SMEM) mma_ss(tmem + TM_S, dq + (j * 32 >> 4), dkj, ID_S, j > 0);
          else mma_ts(tmem + TM_S, tmem + TM_Q + j * 8, dkj, ID_S, j > 0);
        }
        tc_commit(&misc->s_ready);
        tc_commit(&misc->k_empty);
        return true;
      };
      auto issue_tail = [&](int i) -> bool {  // Y += tril(W) V of chunk i, after the token group masked W
        if (!wait_or_abort(&misc->p2_done, i & 1, misc)) return false;
        tc_fence_after_sync();
        const uint64_t dv = dv_mn0 + (uint64_t)((i & 1) * (V_STAGE >> 4));
#pragma unroll
        for (int j = 0; j < 8; ++j)
          mma_ts(tmem + TM_Y, tmem + TM_W + j * 8, dv + (j * 2048 >> 4), ID_Y1, 1);
        tc_commit(&misc->y_ready);
        tc_commit(&misc->v_empty[i & 1]);
        return true;
      };

      ok = wait_or_abort(&misc->q_full, 0, misc);  // the latent bank is in place
      tc_fence_after_sync();
      if (ok && nchunks > 0) ok = issue_scores(0);
      for (int i = 0; ok && i < nchunks; ++i) {
        const uint32_t par = i & 1;
        TC_TRACE(2, i, 0);
        // Next chunk's scores first: the latent group took S of chunk i long ago, while the token group is still
        // masking W of chunk i - 1, which the read-out product below waits for.  (Wide: the scores go into the columns
        // that hold the packed W of chunk i - 1 until that product has read them, so they come second there.)
        if (!WIDE && i + 1 < nchunks) {
          if (!(ok = wait_or_abort(&misc->s_free, par, misc))) break;
          if (!(ok = issue_scores(i + 1))) break;
        }
        TC_TRACE(2, i, 2);
        if (!state_only && i >= 1 && !(ok = issue_tail(i - 1))) break;
        TC_TRACE(2, i, 1);
        if (WIDE && i + 1 < nchunks) {
          // the latent group has read S of chunk i: the columns can take the next chunk's scores
          if (!(ok = wait_or_abort(&misc->s_free, par, misc))) break;
          if (!(ok = issue_scores(i + 1))) break;
        }
        if (!(ok = wait_or_abort(&misc->p1_done, par, misc))) break;
        if (!(ok = wait_or_abort(&v_ready[i & 1], (i >> 1) & 1, misc))) break;
        tc_fence_after_sync();
        TC_TRACE(2, i, 3);
        const uint64_t dek = de_k0, dem = de_mn0, drm = dr_mn0;
        const uint64_t dv = dv_mn0 + (uint64_t)((i & 1) * (V_STAGE >> 4));
        if (!state_only) {
          // Single-buffered accumulators: the token group must have taken Y of chunk i - 1.
          if (i >= 1) {
            if (!(ok = wait_or_abort(&misc->y_free, (i - 1) & 1, misc))) break;
            tc_fence_after_sync();
          }
          {
            // wide: W shares the columns of S: the latent group must have taken the next chunk's scores
            if (WIDE && i + 1 < nchunks) {
              if (!(ok = wait_or_abort(&misc->s_free, (i + 1) & 1, misc))) break;
              tc_fence_after_sync();
            }
            // [W | Y0 (| Den0)] = R^T [E | U_bf16 (| d)]: one product (k = latents); the B operand's four 64-wide blocks
            // lie 16384 bytes apart: the E t-blocks, then the two value blocks of the bf16 state, or its one value
            // block and the block whose column 0 is d
#pragma unroll
            for (int j = 0; j < KSM; ++j) mma_ss(tmem + TM_W, drm + (j * 2048 >> 4), dem + (j * 2048 >> 4), ID_WY, j > 0);
            tc_commit(&misc->w_ready);
            TC_TRACE(2, i, 5);
            if constexpr (WIDE) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                mma_ss(tmem + TM_DEN, drm + (j * 2048 >> 4), db16 + (((j >> 2) * 2048 + (j & 3) * 32) >> 4), ID_DEN, j > 0);
            }
          }
          TC_TRACE(2, i, 6);
        }
        // U += E V_c  (k = tokens of the chunk)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          mma_ss(tmem + TM_U, dek + (((j >> 2) * 16384 + (j & 3) * 32) >> 4), dv + (j * 2048 >> 4), ID_U, 1);
        tc_commit(&misc->u_done);
        if (state_only) tc_commit(&misc->v_empty[i & 1]);  // no read-out MMA will read this V stage
        TC_TRACE(2, i, 4);
      }
      if (!state_only && ok && nchunks > 0) ok = issue_tail(nchunks - 1);
    }
  } else if (warp < 8) {
    // ===================== latent group: 8 warps, thread = (latent = TMEM lane, half of the chunk's tokens) =====================
    // Warps q and q + 4 own the same 32 latents and split the 128 tokens of a chunk in halves, so that two warps
    // per scheduler overlap the special-function, ALU and FMA pipes.  The halves exchange the row maximum and the
    // row sum of E through shared memory.
    const int hf = warp >> 2, q = warp & 3;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
    const int lm = q * 32 + lane;                       // TMEM lane
    const int m = PACK ? (lm & 63) : lm;                // latent of the group
    const int tp = PACK ? hf * 2 + (q >> 1) : hf;       // token part of this thread
    const int pq = PACK ? (q & 1) : q;                  // exchange group: the NP warps of the same 32 latents
    // exchange arrays [chunk parity][part][latent]
    auto xs = [&](int par_, int part) -> float& {
      if constexpr (PACK) return misc->x4[1][par_][part][m];
      else return misc->xsum[par_][part][m];
    };
    auto xm = [&](int par_, int part) -> float& {
      if constexpr (PACK) return misc->x4[0][par_][part][m];
      else return misc->xmax[par_][part][m];
    };
    auto xsum_all = [&](int par_) -> float {
      float t = xs(par_, 0) + xs(par_, 1);
      if constexpr (PACK) t += xs(par_, 2) + xs(par_, 3);
      return t;
    };
    auto xmax_all = [&](int par_) -> float {
      float t = fmaxf(xm(par_, 0), xm(par_, 1));
      if constexpr (PACK) t = fmaxf(t, fmaxf(xm(par_, 2), xm(par_, 3)));
      return t;
    };
    const float sc2 = p.scale * kLog2e;
    const int64_t st_idx = (int64_t)lane_id * p.in_lane_stride + (int64_t)seg * p.in_seg_stride;
    // Fewer than 128 latents: the missing rows are padding (zero rows of Q).  A padding latent gets the frame +inf,
    // so its E = exp2(0 - inf) is exactly zero without any predicate in the element loops, and a denominator of 1.
    const bool live = !PADDED || latent0<ZS, SPLIT>() + m < p.M;
    float c2 = -INFINITY, dsum = 0.f;  // running max (log2 units) and the denominator in that frame
    if (!live) {
      c2 = 0.f;
      dsum = 1.f;
    } else if (p.in_m != nullptr) {
      // (stablemax: the carried m is a constant zero and not a frame; the decode frame starts empty)
      if (!STABLE) c2 = p.in_m[st_idx * p.M + latent0<ZS, SPLIT>() + m] * kLog2e;
      dsum = p.in_d[st_idx * p.M + latent0<ZS, SPLIT>() + m];
    }
    float d_prev = 0.f;                                  // denominator before the chunk in flight, in its frame
    if constexpr (!Q_SMEM) {
      // latent bank row m -> tensor memory as packed bf16 (element k in column k / 2); each half-group thread
      // writes half of the row.  Rows beyond M are zero.
      uint32_t r[DKB * 16];
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.q) +
                                                        (int64_t)h * p.q_stride_h +
                                                        (int64_t)(live ? latent0<ZS, SPLIT>() + m : 0) * p.q_stride_m +
                                                        hf * (DKB * 32));
#pragma unroll
      for (int i = 0; i < DKB * 4; ++i) {
        const uint4 x = live ? src[i] : make_uint4(0, 0, 0, 0);
        r[4 * i] = x.x; r[4 * i + 1] = x.y; r[4 * i + 2] = x.z; r[4 * i + 3] = x.w;
      }
      static_assert(Q_SMEM || DKB == 2, "store width");
      tmem_st32(tl + TM_Q + hf * 32, r);
      tmem_wait_st();
      tc_fence_before_sync();
      warp_arrive(&misc->q_full, lane);
    }
    // columns of the numerator each thread looks after: 32 of the CTA's 64, (wide) 64 of its 128, (packed) 16 of 64
    constexpr int UW = WIDE ? 64 : (PACK ? 16 : 32);
    const int ucol = PACK ? (q >> 1) * 32 + hf * 16 : hf * UW;
    if constexpr (PACK) {
      // carry-in numerator -> tensor memory (the columns of the row's other copy are whatever is there: never read)
      uint32_t r[16];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        r[i] = (p.in_u && live) ? __float_as_uint(p.in_u[(st_idx * p.M + m) * DV + value_col0<ZS, SPLIT>() + ucol + i]) : 0u;
      tmem_st16(tl + TM_U + ucol, r);
      tmem_wait_st();
    } else {
#pragma unroll
      for (int c0 = 0; c0 < UW; c0 += 32) {
        // carry-in numerator -> tensor memory
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; ++i)
          r[i] = (p.in_u && live) ? __float_as_uint(p.in_u[(st_idx * p.M + latent0<ZS, SPLIT>() + m) * DV +
                                                           value_col0<ZS, SPLIT>() + ucol + c0 + i])
                                  : 0u;
        tmem_st32(tl + TM_U + ucol + c0, r);
        tmem_wait_st();
      }
    }

    for (int i = 0; ok && i < nchunks; ++i) {
      const uint32_t par = i & 1;
      const int nvalid = min(C, seg_end - (seg_begin + i * C));
      const int tok0 = tp * TOK;
      uint8_t* e_row = smem + OFF_E + (tok0 >> 6) * 16384;  // this thread's t-block of the operand buffers
      uint8_t* r_row = smem + OFF_R + (tok0 >> 6) * 16384;
      const int ch0 = PACK ? (tp & 1) * 4 : 0;              // and its first 8-token piece there
      if (!(ok = wait_or_abort(&misc->s_ready, par, misc))) break;
      tc_fence_after_sync();
      if (tid == 0) TC_TRACE(0, i, 0);
      // the 64 (packed: 32) scores of this thread stay in registers for the whole chunk
      uint32_t ra[32], rb[32];
      tmem_ld32(tl + TM_S + tok0, ra);
      if constexpr (!PACK) tmem_ld32(tl + TM_S + tok0 + 32, rb);
      // Frame of this chunk.  Chunk 0 exchanges the two halves' maxima synchronously (the carried frame may be
      // empty).  Later chunks use the running max through the PREVIOUS chunk, known without waiting (this bookkeeping
      // runs while the scores are on their way out of tensor memory); E may then exceed 1 by the growth of the max
      // inside one chunk, which fp32 / bf16 hold easily.  This chunk's own row maximum is taken along with the E pass
      // and enters the next chunk's frame.  The state is put into the exact running-max frame when it is written out.
      float c_new = c2;
      if (i > 0) {
        // bookkeeping of chunk i - 1: both halves' sums and maxima are published once its psum phase completed
        if (!(ok = wait_or_abort(&misc->psum[pq], (i - 1) & 1, misc))) break;
        dsum = d_prev + xsum_all(par ^ 1);
        c_new = fmaxf(c2, xmax_all(par ^ 1));
      }
      tmem_wait_ld();
      tmem_fence_regs(ra);
      if constexpr (!PACK) tmem_fence_regs(rb);
      tc_fence_before_sync();
      warp_arrive(&misc->s_free, lane);  // the S columns may take the next chunk's scores
      if (i == 0) {
        // row maximum over the valid tokens of this half, exchanged with the other half
        float cm0 = -INFINITY, cm2 = -INFINITY;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          if (tok0 + k < nvalid) cm0 = fmaxf(cm0, __uint_as_float(ra[k]) * sc2);
          if (!PACK && tok0 + 32 + k < nvalid) cm2 = fmaxf(cm2, __uint_as_float(rb[k]) * sc2);
        }
        xm(0, tp) = live ? fmaxf(cm0, cm2) : -INFINITY;
        warp_arrive(&misc->pmax[pq], lane);
        if (!(ok = wait_or_abort(&misc->pmax[pq], 0, misc))) break;
        c_new = fmaxf(c2, xmax_all(0));
      }
      float alpha = STABLE ? 1.0f : ex2_approx(c2 - c_new);  // 0 when the old state is empty
      // kappa: common frame of the decode weights = max over latents of the running max.  Chunk 0 synchronises;
      // later chunks use the value published during the previous chunk (one chunk stale, which only changes a
      // per-token scale that cancels in y).  (Publishing behind the E pass and reading the value of two chunks before,
      // to take the warp reduction off the start of the chunk, measured 3 % slower: the E pass grew by more.)
      if (hf == 0) {  // (both half-groups hold the same frames: one of them publishes)
        float wm = live ? c_new : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, o));
        // (Two slots suffice: the slot written now is read by the other warps at the top of the NEXT chunk and
        // rewritten at the top of the one after; a warp gets that far only after every warp has finished this chunk -
        // the state update it waits for follows the product that waits for all of them - and has 3 000 cycles of passes
        // of its own in between, while a reader needs a few hundred from the end of this chunk to its read.  Four
        // slots indexed by chunk % 4 measured 4 % slower: one more live value in a register-capped loop.)
        // (The packed instance has registers to spare and passes half as long: four slots there.)
        if (lane == 0) misc->wmax[i & (WS - 1)][q] = wm;
      }
      if (i == 0) {
        if (hf == 0 && lane == 0) mbar_arrive(&misc->kap_done);
        if (!(ok = wait_or_abort(&misc->kap_done, 0, misc))) break;
      }
      const float* wsrc = misc->wmax[i == 0 ? 0 : ((i - 1) & (WS - 1))];
      const float kappa = fmaxf(fmaxf(wsrc[0], wsrc[1]), fmaxf(wsrc[2], wsrc[3]));
      // ordered before the token group's read by the barrier chain
      if ((SPLIT || BLOCK || p.lse_dec != nullptr) && tid == 0) misc->kap[i & 3] = kappa;
      if (tid == 0) TC_TRACE(0, i, 1);
      float a_m = ex2_approx(c_new - kappa);
      float d_carry = dsum * alpha;  // denominator of the carried state in the new frame
      if (PADDED && !live) {
        c_new = INFINITY;
        alpha = 1.0f;
        a_m = 0.f;
        d_carry = 1.0f;
      }
      c2 = c_new;
      // phase a: E for the 64 tokens of this half (in place of the scores), their sum, E operand rows
      float tot0 = 0.f, tot1 = 0.f;
      float g16[4] = {0.f, 0.f, 0.f, 0.f};  // BLOCK: sums of the four groups of 16 tokens of this half
      // this half's row maximum of s - c_new (log2 units), taken along with the pass
      float cma = -INFINITY, cmb = -INFINITY;
      // single E / R buffers: the products that read the previous chunk's E and R (they are all issued together and
      // the state update comes last) must have run
      if (STABLE && i > 0) {
        if (!(ok = wait_or_abort(&misc->u_done, (i - 1) & 1, misc))) break;
        tc_fence_after_sync();
      }
      auto store_e = [&](int ch, const uint4& v) {  // 8 tokens of the E operand's row (packed: both copies of it)
        *reinterpret_cast<uint4*>(e_row + swz_chunk_off(m, ch0 + ch)) = v;
        if constexpr (PACK) *reinterpret_cast<uint4*>(e_row + 8192 + swz_chunk_off(m, ch0 + ch)) = v;
      };
      if constexpr (STABLE) {
        // encoder weights sigma(s): packed and stored 8 tokens at a time; the raw scores stay in ra / rb for phase b (packed:
        // rb is free there and keeps the weights)
#pragma unroll
        for (int ch = 0; ch < TOK / 8; ++ch) {
          float sg[8], x[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float raw = __uint_as_float(ch < 4 ? ra[ch * 8 + j] : rb[(ch - 4) * 8 + j]);
            if (tok0 + ch * 8 + j < nvalid) cma = fmaxf(cma, raw * sc2 - c_new);
            x[j] = raw * p.scale;
          }
          sigma8(x, p.power, sg);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (tok0 + ch * 8 + j >= nvalid) sg[j] = 0.f;
            tot0 += sg[j];
            if constexpr (PACK) rb[ch * 8 + j] = __float_as_uint(sg[j]);
          }
          store_e(ch, make_uint4(pack_bf16(sg[0], sg[1]), pack_bf16(sg[2], sg[3]), pack_bf16(sg[4], sg[5]), pack_bf16(sg[6], sg[7])));
        }
      } else if (nvalid == C) {
        // two tokens per FMA / add instruction (packed fp32 pairs): the passes are bound by instruction issue
        const uint64_t sc2p = f2_pack(sc2, sc2), cnp = f2_pack(-c_new, -c_new);
        uint64_t sa[2] = {f2_pack(0.f, 0.f), f2_pack(0.f, 0.f)}, sb[2] = {f2_pack(0.f, 0.f), f2_pack(0.f, 0.f)};
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          float xa0, xa1;
          f2_unpack(f2_fma(f2_pack(__uint_as_float(ra[k]), __uint_as_float(ra[k + 1])), sc2p, cnp), xa0, xa1);
          cma = fmax3(cma, xa0, xa1);
          const float ea0 = ex2_approx(xa0), ea1 = ex2_approx(xa1);
          ra[k] = __float_as_uint(ea0);
          ra[k + 1] = __float_as_uint(ea1);
          sa[BLOCK ? (k >> 4) : 0] = f2_add(sa[BLOCK ? (k >> 4) : 0], f2_pack(ea0, ea1));
          if constexpr (!PACK) {
            float xb0, xb1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(rb[k]), __uint_as_float(rb[k + 1])), sc2p, cnp), xb0, xb1);
            cmb = fmax3(cmb, xb0, xb1);
            const float eb0 = ex2_approx(xb0), eb1 = ex2_approx(xb1);
            rb[k] = __float_as_uint(eb0);
            rb[k + 1] = __float_as_uint(eb1);
            sb[BLOCK ? (k >> 4) : 0] = f2_add(sb[BLOCK ? (k >> 4) : 0], f2_pack(eb0, eb1));
          }
        }
        float lo, hi;
        if (BLOCK) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            f2_unpack(sa[g], lo, hi);
            g16[g] = lo + hi;
            if constexpr (!PACK) {
              f2_unpack(sb[g], lo, hi);
              g16[2 + g] = lo + hi;
            }
          }
        } else {
          f2_unpack(sa[0], lo, hi);
          tot0 = lo + hi;
          if constexpr (!PACK) {
            f2_unpack(sb[0], lo, hi);
            tot1 = lo + hi;
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          const float x0 = __uint_as_float(ra[k]) * sc2 - c_new;
          if (tok0 + k < nvalid) cma = fmaxf(cma, x0);
          const float e0 = (tok0 + k < nvalid) ? ex2_approx(x0) : 0.f;
          ra[k] = __float_as_uint(e0);
          if (BLOCK) g16[k >> 4] += e0;
          else tot0 += e0;
          if constexpr (!PACK) {
            const float x1 = __uint_as_float(rb[k]) * sc2 - c_new;
            if (tok0 + 32 + k < nvalid) cmb = fmaxf(cmb, x1);
            const float e1 = (tok0 + 32 + k < nvalid) ? ex2_approx(x1) : 0.f;
            rb[k] = __float_as_uint(e1);
            if (BLOCK) g16[2 + (k >> 4)] += e1;
            else tot1 += e1;
          }
        }
      }
      if (BLOCK) {
        tot0 = g16[0] + g16[1];
        tot1 = g16[2] + g16[3];
      }
      xs(par, tp) = tot0 + tot1;
      // (chunk 0 published its maximum before the pass; an empty part stays at -inf)
      if (i > 0) xm(par, tp) = live ? fmaxf(cma, cmb) + c_new : -INFINITY;
      if (!(tot0 + tot1 < 1.15e18f)) {
        // the running max grew by more than 60 powers of two inside one chunk (the frame is the max through the
        // previous chunk): the denominators of this row leave the range in which the read-out weights are safe, see
        // the token group's check; an overflow (or a NaN) lands here as well.  Outside the numeric domain of this path.
        atomicOr(p.err, 2);
        misc->out_of_domain = 1;
      }
      warp_arrive(&misc->psum[pq], lane);
      // E has one buffer: the products that read the previous chunk's E and R (issued together, the state update last)
      // must have run.  (Storing inside the pass would need this wait before it, where it is not yet satisfied.)
      if (!STABLE && i > 0) {
        if (!(ok = wait_or_abort(&misc->u_done, (i - 1) & 1, misc))) break;
        tc_fence_after_sync();
      }
      if constexpr (!STABLE)
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        if constexpr (BLOCK && WIDE && SPLIT && !KEEP) {
          put_piece(e_row + swz_chunk_off(m, ch0 + ch), pack_piece(ra, ch));
          put_piece(e_row + swz_chunk_off(m, ch0 + 4 + ch), pack_piece(rb, ch));
        } else {
          store_e(ch, pack_piece(ra, ch));
          if constexpr (!PACK) store_e(4 + ch, pack_piece(rb, ch));
        }
      }
      d_prev = d_carry;
      // a later part continues the earlier parts' running denominator; the first one needs nothing from its partners
      // (except for blocks that end in a later part)
      float run = d_carry;
      if (!state_only && (tp || (BLOCK && p.block > TOK))) {
        if (!(ok = wait_or_abort(&misc->psum[pq], par, misc))) break;
        if constexpr (PACK) {
#pragma unroll
          for (int t = 0; t < NP - 1; ++t) run += t < tp ? xs(par, t) : 0.f;
        } else {
          run += xs(par, 0);
          if (BLOCK && p.block > TOK && hf == 0) run = d_carry;  // lower half: only the wait was needed
        }
      }
      if (tid == 0) TC_TRACE(0, i, 2);
      if (state_only) {
        // no read-out: R is not needed
      } else if constexpr (STABLE) {
        // phase b, stablemax: D = running sum of sigma (kept, or recomputed), decode numerator exp2(s - c) a_m, R = numerator / D
#pragma unroll
        for (int ch = 0; ch < TOK / 8; ++ch) {
          float s[8], sg[8], r[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = __uint_as_float(ch < 4 ? ra[ch * 8 + j] : rb[(ch - 4) * 8 + j]);
          if constexpr (PACK) {
#pragma unroll
            for (int j = 0; j < 8; ++j) sg[j] = __uint_as_float(rb[ch * 8 + j]);
          } else {
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = s[j] * p.scale;
            sigma8(x, p.power, sg);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (tok0 + ch * 8 + j >= nvalid) sg[j] = 0.f;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            run += sg[j];
            r[j] = ex2_approx(s[j] * sc2 - c_new) * (a_m * rcp_approx(run));
          }
          *reinterpret_cast<uint4*>(r_row + swz_chunk_off(m, ch0 + ch)) =
              make_uint4(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]), pack_bf16(r[4], r[5]), pack_bf16(r[6], r[7]));
        }
      } else if constexpr (!BLOCK) {
        // phase b: D = running denominator, R = E a_m / D, R operand rows.  Reciprocals run on the special-function
        // unit (25-35 % busy); a Newton reciprocal on the FMA pipe for every other element cost 1-9 % of the kernel
        // depending on the box, and carrying the denominator pre-divided by a_m (one FMA + reciprocal + multiply per
        // element) measured 1.5 % slower than this form.
#pragma unroll
        for (int blk = 0; blk < TOK / 32; ++blk) {
          uint32_t rp[16];
#pragma unroll
          for (int k = 0; k < 32; k += 2) {
            const float e0 = __uint_as_float(blk ? rb[k] : ra[k]);
            const float e1 = __uint_as_float(blk ? rb[k + 1] : ra[k + 1]);
            run += e0;
            const float i0 = rcp_approx(run);
            run += e1;
            const float i1 = rcp_approx(run);
            float r0, r1;  // e * (a_m / D), two tokens per multiply
            f2_unpack(f2_mul(f2_pack(e0, e1), f2_mul(f2_pack(i0, i1), f2_pack(a_m, a_m))), r0, r1);
            rp[k >> 1] = pack_bf16(r0, r1);
          }
#pragma unroll
          for (int ch = 0; ch < 4; ++ch)
            *reinterpret_cast<uint4*>(r_row + swz_chunk_off(m, ch0 + blk * 4 + ch)) =
                make_uint4(rp[ch * 4], rp[ch * 4 + 1], rp[ch * 4 + 2], rp[ch * 4 + 3]);
        }
      } else {
        // phase b, block-causal: the denominator of a token is the one at the end of its block.  dend[g] is that
        // value for the g-th group of 16 tokens of this half (`run` = denominator before this half).
        const int bs = p.block;
        constexpr int NG = TOK / 16;
        float dend[NG];
        if constexpr (PACK) {
          const float p0 = run + g16[0], p1 = p0 + g16[1];
          if (bs == 16) {
            dend[0] = p0; dend[1] = p1;
          } else if (bs == 32) {
            dend[0] = dend[1] = p1;
          } else {
            // the block ends in a later part (or this one): add the parts up to its last one
            const int last = bs == 64 ? (tp | 1) : NP - 1;
            float t = p1;
#pragma unroll
            for (int u = 1; u < NP; ++u) t += (u > tp && u <= last) ? xs(par, u) : 0.f;
            dend[0] = dend[1] = t;
          }
        } else {
          const float p0 = run + g16[0], p1 = p0 + g16[1], p2 = p1 + g16[2], p3 = p2 + g16[3];
          if (bs == 16) {
            dend[0] = p0; dend[1] = p1; dend[2] = p2; dend[3] = p3;
          } else if (bs == 32) {
            dend[0] = dend[1] = p1; dend[2] = dend[3] = p3;
          } else if (bs == 64) {
            dend[0] = dend[1] = dend[2] = dend[3] = p3;
          } else {
            // one block per chunk: both halves use the chunk's end
            const float whole = d_carry + xsum_all(par);
            dend[0] = dend[1] = dend[2] = dend[3] = whole;
          }
        }
        // log normaliser after each block that ends in this half (natural log, exact-frame independent)
        if (p.lse_enc != nullptr && live && value_col0<ZS, SPLIT>() == 0) {
          const int t_half = seg_begin + i * C + tok0;  // first token of this half in the sequence
          float* dst = p.lse_enc + ((int64_t)lane_id * (p.N / bs)) * p.M + latent0<ZS, SPLIT>() + m;
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            const int t_end = t_half + g * 16 + 15;            // last token of the group
            const bool ends = ((t_end + 1) % bs) == 0;         // a block ends with this group
            if (ends && tok0 + g * 16 < nvalid) dst[(int64_t)(t_end / bs) * p.M] = (c_new + __log2f(dend[g])) * kLn2;
          }
        }
        float inv[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) inv[g] = a_m * rcp_approx(dend[g]);
#pragma unroll
        for (int blk = 0; blk < TOK / 32; ++blk) {
          uint32_t rp[16];
#pragma unroll
          for (int k = 0; k < 32; k += 2) {
            const float w = inv[blk * 2 + (k >> 4)];
            float r0, r1;
            f2_unpack(f2_mul(f2_pack(__uint_as_float(blk ? rb[k] : ra[k]), __uint_as_float(blk ? rb[k + 1] : ra[k + 1])),
                             f2_pack(w, w)), r0, r1);
            rp[k >> 1] = pack_bf16(r0, r1);
          }
#pragma unroll
          for (int ch = 0; ch < 4; ++ch)
            *reinterpret_cast<uint4*>(r_row + swz_chunk_off(m, ch0 + blk * 4 + ch)) =
                make_uint4(rp[ch * 4], rp[ch * 4 + 1], rp[ch * 4 + 2], rp[ch * 4 + 3]);
        }
      }
      if (tid == 0) TC_TRACE(0, i, 3);
      // state part: needs the numerator update of the previous chunk to have landed (waited for before the E rows
      // were written)
      if (tid == 0) TC_TRACE(0, i, 4);
      if (tp == 0 && !state_only) {
        // d of the carried state: column 0 of row m of the MN-major block (merged product with one value block), or
        // element m of row 0 of the small K-major tile
        if (!WIDE)
          *reinterpret_cast<__nv_bfloat16*>(smem + OFF_B16 + swz_chunk_off(m, 0)) = __float2bfloat16_rn(d_carry);
        else
          *reinterpret_cast<__nv_bfloat16*>(smem + OFF_B16 + (m >> 6) * 2048 + ((m & 63) >> 3) * 16 + (m & 7) * 2) =
              __float2bfloat16_rn(d_carry);
      }
      const bool need = __any_sync(0xffffffffu, alpha != 1.0f);
      if constexpr (WIDE) {
        // 64 value columns per thread = value block hf of the bf16 state operand (free: the products that read it
        // were issued before the state update this thread has just waited for)
        if (!state_only || need) {
#pragma unroll
          for (int c0 = 0; c0 < 64; c0 += 32) {
            uint32_t r[32];
            tmem_ld32(tl + TM_U + hf * 64 + c0, r);
            tmem_wait_ld();
            tmem_fence_regs(r);
            if (need) {
#pragma unroll
              for (int k = 0; k < 32; k += 2) {
                float u0, u1;
                f2_unpack(f2_mul(f2_pack(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), f2_pack(alpha, alpha)), u0, u1);
                r[k] = __float_as_uint(u0);
                r[k + 1] = __float_as_uint(u1);
              }
              tmem_st32(tl + TM_U + hf * 64 + c0, r);
            }
            if (!state_only) {
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) {
                uint4 v;
                v.x = pack_bf16(__uint_as_float(r[ch * 8 + 0]), __uint_as_float(r[ch * 8 + 1]));
                v.y = pack_bf16(__uint_as_float(r[ch * 8 + 2]), __uint_as_float(r[ch * 8 + 3]));
                v.z = pack_bf16(__uint_as_float(r[ch * 8 + 4]), __uint_as_float(r[ch * 8 + 5]));
                v.w = pack_bf16(__uint_as_float(r[ch * 8 + 6]), __uint_as_float(r[ch * 8 + 7]));
                *reinterpret_cast<uint4*>(smem + OFF_U + hf * 16384 + swz_chunk_off(m, (c0 >> 3) + ch)) = v;
              }
              if constexpr (KEEP) {
                // training: the state before this chunk in the exact running-max frame through it (see below)
                if (c0 == 0 && !(ok = wait_or_abort(&misc->psum[pq], par, misc))) break;
                float fin = 1.0f, c_true = c2;
                if (!STABLE) {
                  c_true = fmaxf(c2, xmax_all(par));
                  fin = ex2_approx(c2 - c_true);
                }
                const int64_t o = ((int64_t)lane_id * p.dump_nch + (seg_begin / C + i)) * p.M + latent0<ZS, SPLIT>() + m;
                uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dump_u) + o * DV + hf * 64 + c0);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                  uint4 v;
                  v.x = pack_bf16(__uint_as_float(r[ch * 8 + 0]) * fin, __uint_as_float(r[ch * 8 + 1]) * fin);
                  v.y = pack_bf16(__uint_as_float(r[ch * 8 + 2]) * fin, __uint_as_float(r[ch * 8 + 3]) * fin);
                  v.z = pack_bf16(__uint_as_float(r[ch * 8 + 4]) * fin, __uint_as_float(r[ch * 8 + 5]) * fin);
                  v.w = pack_bf16(__uint_as_float(r[ch * 8 + 6]) * fin, __uint_as_float(r[ch * 8 + 7]) * fin);
                  dst[ch] = v;
                }
                if (hf == 0 && c0 == 0) {
                  p.dump_c[o] = c_true;
                  p.dump_d[o] = d_carry * fin;
                }
              }
            }
          }
          if (!ok) break;
          if (need) tmem_wait_st();
        }
      } else
      if (!state_only || need) {
        constexpr int NU = PACK ? 16 : 32;  // columns of this thread
        uint32_t r[NU];
        if constexpr (PACK) tmem_ld16(tl + TM_U + ucol, r);
        else tmem_ld32(tl + TM_U + ucol, r);
        tmem_wait_ld();
        if constexpr (PACK) tmem_fence_regs16(r);
        else tmem_fence_regs(r);
        if (need) {
#pragma unroll
          for (int k = 0; k < NU; k += 2) {
            float u0, u1;
            f2_unpack(f2_mul(f2_pack(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), f2_pack(alpha, alpha)), u0, u1);
            r[k] = __float_as_uint(u0);
            r[k + 1] = __float_as_uint(u1);
          }
          if constexpr (PACK) tmem_st16(tl + TM_U + ucol, r);
          else tmem_st32(tl + TM_U + ucol, r);
        }
        if (!state_only) {
#pragma unroll
          for (int ch = 0; ch < NU / 8; ++ch) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(r[ch * 8 + 0]), __uint_as_float(r[ch * 8 + 1]));
            v.y = pack_bf16(__uint_as_float(r[ch * 8 + 2]), __uint_as_float(r[ch * 8 + 3]));
            v.z = pack_bf16(__uint_as_float(r[ch * 8 + 4]), __uint_as_float(r[ch * 8 + 5]));
            v.w = pack_bf16(__uint_as_float(r[ch * 8 + 6]), __uint_as_float(r[ch * 8 + 7]));
            *reinterpret_cast<uint4*>(smem + OFF_U + swz_chunk_off(m, (ucol >> 3) + ch)) = v;
          }
          if constexpr (KEEP) {
            // Training: the state before this chunk is kept for the backward pass, in the EXACT running-max frame
            // through this chunk (= the frame the next chunk will use), so that the backward's encoder weights of
            // the chunk never exceed 1.  All parts' maxima of this chunk are published once its psum phase completed.
            if (!(ok = wait_or_abort(&misc->psum[pq], par, misc))) break;
            float fin = 1.0f, c_true = c2;
            if (!STABLE) {
              c_true = fmaxf(c2, xmax_all(par));
              fin = ex2_approx(c2 - c_true);
            }
            if (i > 0 && !(ok = wait_or_abort(&misc->keep_free, (i - 1) & 1, misc))) break;  // the tile has been read
#pragma unroll
            for (int ch = 0; ch < NU / 8; ++ch) {  // (rows beyond M are clipped)
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[ch * 8 + 0]) * fin, __uint_as_float(r[ch * 8 + 1]) * fin);
              v.y = pack_bf16(__uint_as_float(r[ch * 8 + 2]) * fin, __uint_as_float(r[ch * 8 + 3]) * fin);
              v.z = pack_bf16(__uint_as_float(r[ch * 8 + 4]) * fin, __uint_as_float(r[ch * 8 + 5]) * fin);
              v.w = pack_bf16(__uint_as_float(r[ch * 8 + 6]) * fin, __uint_as_float(r[ch * 8 + 7]) * fin);
              *reinterpret_cast<uint4*>(smem + L::OFF_KEEP + swz_chunk_off(m, (ucol >> 3) + ch)) = v;
            }
            if (live) {
              const int64_t o = ((int64_t)lane_id * p.dump_nch + (seg_begin / C + i)) * p.M + latent0<ZS, SPLIT>() + m;
              if (tp == 0 && value_col0<ZS, SPLIT>() == 0) {
                p.dump_c[o] = c_true;          // log2 units (unused for the stablemax encoder)
                p.dump_d[o] = d_carry * fin;   // denominator before the chunk in that frame
              }
            }
          }
        }
        if (need) tmem_wait_st();
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      warp_arrive(&misc->p1_done, lane);
      if (tid == 0) TC_TRACE(0, i, 5);
    }
    // carry-out state
    if (ok && p.out_u != nullptr && (p.out_mode == 1 || (p.out_mode == 2 && seg == p.nseg_total - 1))) {
      float fin = 1.0f;  // factor from the last chunk's frame to the exact running-max frame
      if (nchunks > 0) {
        const int lp = (nchunks - 1) & 1;
        ok = wait_or_abort(&misc->u_done, lp, misc) && wait_or_abort(&misc->psum[pq], lp, misc);
        if (ok) {
          dsum = d_prev + xsum_all(lp);
          if (!STABLE) {
            const float c_true = fmaxf(c2, xmax_all(lp));
            fin = ex2_approx(c2 - c_true);
            c2 = c_true;
          }
        }
      }
      tc_fence_after_sync();
      if (ok) {
        const int64_t so = (int64_t)lane_id * p.out_lane_stride + (int64_t)seg * p.out_seg_stride;
        const int mg = latent0<ZS, SPLIT>() + m;  // latent index in the whole bank
        if (tp == 0 && live && value_col0<ZS, SPLIT>() == 0) {
          p.out_m[so * p.M + mg] = STABLE ? 0.f : c2 * kLn2;
          p.out_d[so * p.M + mg] = dsum * fin;
        }
        constexpr int NU = PACK ? 16 : 32;
#pragma unroll
        for (int c0 = 0; c0 < UW; c0 += NU) {
          uint32_t r[NU];
          if constexpr (PACK) tmem_ld16(tl + TM_U + ucol + c0, r);
          else tmem_ld32(tl + TM_U + ucol + c0, r);
          tmem_wait_ld();
          if constexpr (PACK) tmem_fence_regs16(r);
          else tmem_fence_regs(r);
          float4* dst = reinterpret_cast<float4*>(p.out_u + (so * p.M + (live ? mg : 0)) * DV +
                                                  value_col0<ZS, SPLIT>() + ucol + c0);
#pragma unroll
          for (int k = 0; k < NU / 4; ++k)
            if (live) dst[k] = make_float4(__uint_as_float(r[4 * k]) * fin, __uint_as_float(r[4 * k + 1]) * fin,
                                 __uint_as_float(r[4 * k + 2]) * fin, __uint_as_float(r[4 * k + 3]) * fin);
        }
      }
    }
  } else {
    // ============================ token group: thread = token of the chunk = TMEM lane ============================
    const int wq = warp - 8;  // lane quarter
    const uint32_t tl = tmem + ((uint32_t)(wq * 32) << 16);
    const int tt = wq * 32 + lane;  // token index inside the chunk
    uint8_t* const stage = smem + L::OFF_STAGE + wq * 2048;
    // latent-group split: dense fp16 partials [group][B][N][H][DV] and log2 weight masses [group][B][N][H]
    const int64_t part_row0 = SPLIT ? (((int64_t)(blockIdx.z / ZS) * (gridDim.x / p.H) + b) * p.N) : 0;
    const int row0 = LENS && p.row_start != nullptr ? p.row_start[b] : 0;  // (-1: a packed row, whose y goes to the packed copy)
    // Two latent groups merged on chip: a chunk's own rows wait in registers and are merged with the partner's behind the next chunk's
    // mask, while that chunk's tril(W) V runs and the rows are long there.  B200, B=2 N=65536 H=32 M=256 D=128 blocks of 64: 1 899
    // us, 1 967 with the merge at the end of its own chunk (a chunk's period 6 200 and 6 800 cycles).
    uint32_t own[XM ? 2 : 1][XM ? 32 : 1];
    float lw_own = 0.f, inv_own = 0.f;
    auto receive = [&](int i) {
      if constexpr (XM) {
        const int t0 = seg_begin + i * C, nvalid = min(C, seg_end - t0);
        const uint32_t rank = cluster_ctarank();
        if (!(ok = tc::wait_or_abort_cluster(&misc->xfull[wq], i & 1, &misc->abort_flag))) return;
        const float lw_p = *reinterpret_cast<const float*>(smem + L::OFF_XCH + 16384 + tt * 4);
        uint4 xp[8];
#pragma unroll
        for (int ch = 0; ch < 8; ++ch)  // [warp][32-column half][32 rows x 64 bytes, 16-byte pieces swizzled as in the staging tile]
          xp[ch] = *reinterpret_cast<const uint4*>(smem + L::OFF_XCH + wq * 4096 + (ch >> 2) * 2048 + lane * 64 +
                                                   (((ch & 3) ^ ((lane >> 1) & 3)) << 4));
        const float mx = fmaxf(lw_own, lw_p);
        float ca = 0.f, cb = 0.f;  // coefficients of the raw accumulator values and of the partner's normalised rows
        if (mx == -INFINITY) {
          // every group's weights underflowed: outside the numeric domain of this path
          if (rank == 0 && tt < nvalid) {
            atomicOr(p.err, 2);
            misc->out_of_domain = 1;
          }
        } else {
          const float wa = ex2_approx(lw_own - mx), wb = ex2_approx(lw_p - mx);
          const float iw = rcp_approx(wa + wb);
          ca = wa * iw * inv_own;
          cb = wb * iw;
          if (rank == 0 && p.lse_dec != nullptr && tt < nvalid)
            p.lse_dec[(int64_t)lane_id * p.N + t0 + tt] = (mx + __log2f(wa + wb)) * kLn2;
        }
        // The merged rows go out from the exchange tile itself (its layout is the bulk store's 64-byte swizzle and
        // the partner's rows are in registers by now): both 32-column tiles are stored without waiting on each other.
        uint8_t* const xt = smem + L::OFF_XCH + wq * 4096;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint32_t(&r)[32] = own[half];
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            const uint4 x = xp[half * 4 + ch];
            const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
            uint32_t o[4];
            float y[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&xw[j]));
              // own raw values * ca + partner's normalised values * cb, two columns per instruction
              f2_unpack(f2_fma(f2_pack(__uint_as_float(r[ch * 8 + 2 * j]), __uint_as_float(r[ch * 8 + 2 * j + 1])),
                               f2_pack(ca, ca), f2_mul(f2_pack(f.x, f.y), f2_pack(cb, cb))), y[2 * j], y[2 * j + 1]);
            }
            pack_out(y, F16, o);
            *reinterpret_cast<uint4*>(xt + half * 2048 + lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_4d(&tm_y, xt, (int)rank * 64, h, t0 + wq * 32, b);
          tma_store_4d(&tm_y, xt + 2048, (int)rank * 64 + 32, h, t0 + wq * 32, b);
          bulk_commit_group();
        }
        // (the partner learns that the tile is free in the epilogue of the chunk in flight, which waits for these stores to have read it)
      }
    };
    for (int i = 0; !state_only && ok && i < nchunks; ++i) {
      const uint32_t par = i & 1;
      const int t0 = seg_begin + i * C;
      const int nvalid = min(C, seg_end - t0);
      // causal mask of W, bf16 pack, row sums
      if (!(ok = wait_or_abort(&misc->w_ready, par, misc))) break;
      tc_fence_after_sync();
      // This chunk's decode frame, taken now: the latent group is one to two chunks ahead and reuses the slot four
      // chunks on (read late, in the epilogue, from a two-slot array, a slow token group saw a later chunk's frame:
      // wrong weight masses for the merge of latent groups)
      const float kap_i = misc->kap[i & 3];
      if (tid == 256) TC_TRACE(1, i, 0);
      uint64_t rs2 = f2_pack(0.f, 0.f);  // row sum of the bf16-rounded masked W (the values the read-out MMA multiplies), as a pair of partial sums
      // last column (token of the chunk) this row may see: itself, or the end of its block
      const int be = BLOCK ? (tt | (p.block - 1)) : tt;
      // (with the rows of the chunk before in registers 16 columns at a time, else 32)
      constexpr int MW = XM ? 16 : 32;
#pragma unroll 1
      for (int j = 0; j < C / MW; ++j) {
        uint32_t wp[MW / 2];
        // (token-causal, 32 columns: the block below the diagonal, on it or above it is the same for the whole warp)
        const bool any = MW == 32 ? (BLOCK ? j * MW <= be : j <= wq) : __any_sync(0xffffffffu, j * MW <= be);
        if (any) {
          uint32_t r[MW];
          tmem_read(tl + TM_W + j * MW, r);
          if (MW == 32 ? (BLOCK ? j * MW + MW - 1 <= be : j < wq) : __all_sync(0xffffffffu, j * MW + MW - 1 <= be)) {
            // all of these columns are visible to every row of this warp
#pragma unroll
            for (int k = 0; k < MW; k += 2) {
              const uint32_t pk = pack_bf16(__uint_as_float(r[k]), __uint_as_float(r[k + 1]));
              wp[k >> 1] = pk;
              rs2 = f2_add(rs2, f2_pack(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u)));
            }
          } else {
#pragma unroll
            for (int k = 0; k < MW; k += 2) {
              const bool v0 = MW == 32 && !BLOCK ? k <= lane : j * MW + k <= be;
              const bool v1 = MW == 32 && !BLOCK ? k + 1 <= lane : j * MW + k + 1 <= be;
              const uint32_t pk = pack_bf16(v0 ? __uint_as_float(r[k]) : 0.f, v1 ? __uint_as_float(r[k + 1]) : 0.f);
              wp[k >> 1] = pk;
              rs2 = f2_add(rs2, f2_pack(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u)));
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < MW / 2; ++k) wp[k] = 0u;
        }
        tmem_write(tl + TM_W + j * (MW / 2), wp);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      warp_arrive(&misc->p2_done, lane);
      if (tid == 256) TC_TRACE(1, i, 1);

      if (XM && xmerge && i > 0) {
        receive(i - 1);
        if (!ok) break;
      }
      // normalise and store (wide: the first of the two value blocks; two accumulator phases per chunk)
      if (!(ok = wait_or_abort(&misc->y_ready, par, misc))) break;
      tc_fence_after_sync();
      if (tid == 256) TC_TRACE(1, i, 2);
      uint32_t den0;
      tmem_ld1(tl + TM_DEN, den0);
      tmem_wait_ld();
      float rs_lo, rs_hi;
      f2_unpack(rs2, rs_lo, rs_hi);
      const float den = __uint_as_float(den0) + (rs_lo + rs_hi);
      // Numeric domain of this path.  The read-out weight of (token, latent) is R = E a_m / D: it is flushed to zero
      // below 2^-126, while what it stands for, R D = the token's decode weight in the frame kappa, may still matter
      // when the whole token's weight mass is small.  With the row denominators held below 2^60 (checked by the latent
      // group) a flushed weight is below 2^-66, so a token whose mass is at least 2^-40 loses nothing it can see in
      // bf16; below that, or with a mass that overflowed or is not a number, the token is flagged and the exact path,
      // which has no such limit, redoes its lane.  With several latent groups each group's own mass is held to this
      // (the frames differ between groups, so a group that looks empty in its own frame may carry the token).
      const bool den_ok = den >= 9.1e-13f && den < INFINITY;
      if (tt < nvalid && !den_ok) {
        atomicOr(p.err, 2);
        misc->out_of_domain = 1;
      }
      const float inv = (SPLIT && !den_ok) ? 0.f : rcp_approx(den);  // (a true division compiles to a call here)
      if (SPLIT && !xmerge && p.part_y != nullptr && tt < nvalid && value_col0<ZS, SPLIT>() == 0)
        p.part_lw[(part_row0 + t0 + tt) * p.H + h] = den_ok ? kap_i + __log2f(den) : -INFINITY;
      // log-sum-exp of the token's decode scores = log of the decode weights' mass in the frame kappa
      if (!SPLIT && p.lse_dec != nullptr && tt < nvalid && value_col0<ZS, SPLIT>() == 0)
        p.lse_dec[(int64_t)lane_id * p.N + t0 + tt] = (kap_i + __log2f(den)) * kLn2;
      if constexpr (XM) {
        if (xmerge) {
          // Two latent groups = two CTAs of a cluster.  CTA r finalises value block r: it sends its normalised
          // partial of the OTHER block (fp16) and the log2 of its weight mass into the partner's shared memory,
          // takes the partner's rows for its own block, and stores y = sum_g w_g y_g / sum_g w_g.
          const uint32_t rank = cluster_ctarank(), peer = rank ^ 1u;
          lw_own = den_ok ? kap_i + __log2f(den) : -INFINITY;
          inv_own = inv;
          uint32_t pk[32];
          uint32_t(&ra)[32] = own[0], (&rb)[32] = own[1];
          // The exchange tile was the source of the previous chunk's bulk stores: once they have read it the partner
          // may send this chunk's rows (32 rows x 128 bytes and 32 weight masses per warp), which the barrier counts.
          if (lane == 0) {
            bulk_wait_group_read0();
            mbar_arrive_expect_tx(&misc->xfull[wq], 4096 + 128);
          }
          __syncwarp();
          if (i > 0) mbar_arrive_cluster_relaxed(mapa_shared(smem_u32(&misc->xfree[wq]), peer));
          // the partner's block, normalised, as fp16 pairs; then this CTA's block; the accumulator is free again
          tmem_ld32(tl + TM_Y + peer * 64, ra);
          tmem_ld32(tl + TM_Y + peer * 64 + 32, rb);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const uint64_t inv2 = f2_pack(inv, inv);
            float a0, a1, b0, b1;
            f2_unpack(f2_mul(f2_pack(__uint_as_float(ra[2 * k]), __uint_as_float(ra[2 * k + 1])), inv2), a0, a1);
            f2_unpack(f2_mul(f2_pack(__uint_as_float(rb[2 * k]), __uint_as_float(rb[2 * k + 1])), inv2), b0, b1);
            pk[k] = pack_f16(a0, a1);
            pk[16 + k] = pack_f16(b0, b1);
          }
          tmem_ld32(tl + TM_Y + rank * 64, ra);
          tmem_ld32(tl + TM_Y + rank * 64 + 32, rb);
          tmem_wait_ld();
          tc_fence_before_sync();
          warp_arrive(&misc->y_free, lane);
          // (1) send: the rows sent for chunk i - 1 must have been read by the partner.  The stores are asynchronous and
          // count their bytes on the partner's barrier: plain remote stores followed by a releasing arrive cost 1600
          // cycles per chunk here.  Every thread sends the eight 16-byte pieces of its row, in the tile's layout.
          if (i > 0 && !(ok = tc::wait_or_abort_cluster(&misc->xfree[wq], (i - 1) & 1, &misc->abort_flag))) break;
          {
            const uint32_t xw = mapa_shared(smem_u32(smem + L::OFF_XCH + wq * 4096), peer);
            const uint32_t xbar = mapa_shared(smem_u32(&misc->xfull[wq]), peer);
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
              for (int ch = 0; ch < 4; ++ch)
                st_async_v4(xw + half * 2048 + lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4),
                            make_uint4(pk[half * 16 + ch * 4], pk[half * 16 + ch * 4 + 1], pk[half * 16 + ch * 4 + 2],
                                       pk[half * 16 + ch * 4 + 3]), xbar);
            st_async_b32(mapa_shared(smem_u32(smem + L::OFF_XCH + 16384 + tt * 4), peer), __float_as_uint(lw_own), xbar);
          }
          if (tid == 256) TC_TRACE(1, i, 4);
          if (tid == 256) TC_TRACE(1, i, 3);
          continue;
        }
      }
      // The accumulator goes back to the MMA issuer as soon as its columns are in registers (single-buffered
      // instances); scaling and the stores follow.  Wide: two value blocks of 64 columns, handed back after the second.
#pragma unroll
      for (int vb = 0; vb < VB; ++vb) {
        uint32_t ra[32], rb[32];
        tmem_ld32(tl + TM_Y + vb * 64, ra);
        tmem_ld32(tl + TM_Y + vb * 64 + 32, rb);
        tmem_wait_ld();
        if (vb == VB - 1) {
          tc_fence_before_sync();
          warp_arrive(&misc->y_free, lane);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint32_t(&r)[32] = half ? rb : ra;
          const int col = value_col0<ZS, SPLIT>() + vb * 64 + half * 32;
          // 32 columns of this thread's row as 16-bit values: y in its type, or fp16 of a latent group's partial
          uint4 v[4];
          const uint64_t inv2 = f2_pack(inv, inv);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            uint32_t o[4];
            float y[8];
#pragma unroll
            for (int j = 0; j < 4; ++j)  // two columns per multiply
              f2_unpack(f2_mul(f2_pack(__uint_as_float(r[ch * 8 + 2 * j]), __uint_as_float(r[ch * 8 + 2 * j + 1])), inv2), y[2 * j],
                        y[2 * j + 1]);
            pack_out(y, SPLIT || F16, o);
            v[ch] = make_uint4(o[0], o[1], o[2], o[3]);
          }
          if (p.y_tma && (!LENS || row0 >= 0)) {
            // One tiled bulk store per warp and 32 x 32 tile.  A thread storing its own row straight to global
            // memory costs 32 separate 16-byte transactions per instruction; the latent warps' operand stores to
            // shared memory queued behind those and the whole kernel ran 12 % slower.  Rows beyond the sequence end
            // are clipped by the copy.
            if (lane == 0) bulk_wait_group_read0();  // the previous tile has left the staging buffer
            __syncwarp();
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)  // 64-byte swizzle: 16-byte piece index ^ (row / 2) % 4
              *reinterpret_cast<uint4*>(stage + lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4)) = v[ch];
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_4d(&tm_y, stage, col, h, t0 + row0 + wq * 32, SPLIT ? (int)(blockIdx.z / ZS) * (int)(gridDim.x / p.H) + b : b);
              bulk_commit_group();
            }
          } else if (SPLIT) {
            if (p.part_y != nullptr && tt < nvalid) {
              uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.part_y) +
                                                    ((part_row0 + t0 + tt) * p.H + h) * DV + col);
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) dst[ch] = v[ch];
            }
          } else if (p.y != nullptr && tt < nvalid) {
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.y) + (int64_t)b * p.y_stride_b +
                                                  (int64_t)h * p.y_stride_h + (int64_t)(t0 + tt) * p.y_stride_n + col);
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) dst[ch] = v[ch];
          }
        }
      }
      if (!ok) break;
      if (tid == 256) TC_TRACE(1, i, 3);
    }
    if (XM && xmerge && !state_only && ok && nchunks > 0) receive(nchunks - 1);
    if (lane == 0) bulk_wait_group0();  // the bulk stores of this warp are complete
  }
  if (!ok) {
    misc->abort_flag = 1;
    atomicOr(p.err, 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && p.gate != nullptr) {
    p.gate[1 + (int64_t)lane_id * p.gate_stride + p.gate_off + (int)(blockIdx.y * gridDim.z + blockIdx.z)] = misc->out_of_domain;
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) p.gate[0] = p.gate_stride;  // (both passes write the same)
  }
  // the partner may still write to this CTA's shared memory or arrive on its barriers until it is done as well
  if (xmerge) cluster_sync_all();
  if (warp == 12) tmem_dealloc(tmem, TM_COLS);
}



namespace {

template <int LAT, int DKB, int DVB, bool SPLIT, int MODE, bool KEEP, bool WIDE, int FL>
int launch_keep(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& ty, const CUtensorMap* in,
                const TcParams& p, dim3 grid, cudaStream_t stream) {
  auto kern = prefill_tc_kernel<LAT, DKB, DVB, SPLIT, MODE, KEEP, WIDE, FL>;
  FLARE_CUDA_CHECK(allow_smem(kern));
  LaunchTimer timer(p.y == nullptr ? "prefill_tc_kernel (state only)" : (WIDE ? "prefill_tc_kernel (wide)" : "prefill_tc_kernel"),
                    stream);
  if (WIDE && SPLIT && p.cluster_merge) {
    // the two latent-group CTAs of a lane (adjacent in grid.z) as one thread-block cluster
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(nthreads(KEEP && !WIDE));
    cfg.dynamicSmemBytes = Lay<DKB, WIDE>::smem_bytes(KEEP && !WIDE);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 2;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FLARE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, ty, in[0], in[1], p));
  } else {
    FLARE_CUDA_CHECK(launch_pdl(kern, grid, dim3(nthreads(KEEP && !WIDE)), Lay<DKB, WIDE>::smem_bytes(KEEP && !WIDE), stream, tq, tk, tv, ty, in[0], in[1], p));
  }
  return FLARE_OK;
}

template <int LAT, int DKB, int DVB, bool SPLIT, int MODE, bool WIDE>
int launch_instance(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& ty, const CUtensorMap* in,
                    const TcParams& p, dim3 grid, cudaStream_t stream) {
  if (p.dump_u != nullptr)  // training forward that keeps its per-chunk states
    return launch_keep<LAT, DKB, DVB, SPLIT, MODE, true, WIDE, 0>(tq, tk, tv, ty, in, p, grid, stream);
  if (p.f16) return launch_keep<LAT, DKB, DVB, SPLIT, MODE, false, WIDE, 2>(tq, tk, tv, ty, in, p, grid, stream);
  if constexpr (MODE != 1) {  // (no lengths in block-causal calls)
    if (p.lens != nullptr) return launch_keep<LAT, DKB, DVB, SPLIT, MODE, false, WIDE, 1>(tq, tk, tv, ty, in, p, grid, stream);
  }
  return launch_keep<LAT, DKB, DVB, SPLIT, MODE, false, WIDE, 0>(tq, tk, tv, ty, in, p, grid, stream);
}

}  // namespace

template <>
int launch_prefill_tc_unit<FLARE_TC_UNIT, FLARE_TC_MODE>(int lat, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                                         const CUtensorMap& ty, const CUtensorMap* in, const TcParams& p,
                                                         dim3 grid, cudaStream_t stream) {
  // units 0..2: (Dk, Dv) = (64, 64), (128, 128), (64, 128); units 3..5: the same with the latent-group split;
  // units 6, 7: the wide (128, 128) instance (one CTA for both value blocks) without / with the latent-group split
  constexpr int MODE = FLARE_TC_MODE;
#if FLARE_TC_UNIT >= 6
  (void)lat;
  return launch_instance<0, 2, 2, FLARE_TC_UNIT == 7, MODE, true>(tq, tk, tv, ty, in, p, grid, stream);
#else
  constexpr int COMBO = FLARE_TC_UNIT % 3;
  constexpr int DKB = COMBO == 1 ? 2 : 1;
  constexpr int DVB = COMBO == 0 ? 1 : 2;
  constexpr bool SPLIT = FLARE_TC_UNIT >= 3;
  // one instance family per kind of latent bank; the packed one exists for a single group only
  if (lat == 0) return launch_instance<0, DKB, DVB, SPLIT, MODE, false>(tq, tk, tv, ty, in, p, grid, stream);
  if constexpr (!SPLIT) {
    if (lat == 2) return launch_instance<2, DKB, DVB, SPLIT, MODE, false>(tq, tk, tv, ty, in, p, grid, stream);
  }
  return launch_instance<1, DKB, DVB, SPLIT, MODE, false>(tq, tk, tv, ty, in, p, grid, stream);
#endif
}

#else  // host side and the merge kernel

__device__ int g_tc_error = 0;

#define FLARE_TC_DECLARE(U, MODE)                                                                                            \
  template <>                                                                                                               \
  int launch_prefill_tc_unit<U, MODE>(int, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&,  \
                                      const CUtensorMap*, const TcParams&, dim3, cudaStream_t);
#define FLARE_TC_DECLARE_UNIT(U) FLARE_TC_DECLARE(U, 0) FLARE_TC_DECLARE(U, 1) FLARE_TC_DECLARE(U, 2)
FLARE_TC_DECLARE_UNIT(0)
FLARE_TC_DECLARE_UNIT(1)
FLARE_TC_DECLARE_UNIT(2)
FLARE_TC_DECLARE_UNIT(3)
FLARE_TC_DECLARE_UNIT(4)
FLARE_TC_DECLARE_UNIT(5)
FLARE_TC_DECLARE_UNIT(6)
FLARE_TC_DECLARE_UNIT(7)
#undef FLARE_TC_DECLARE_UNIT
#undef FLARE_TC_DECLARE

// -------------------------------------------------------------------------------------------------
// host side
// -------------------------------------------------------------------------------------------------
namespace {

bool make_map(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const int64_t* strides_elems,
              const uint32_t* box) {
  return tc::make_map_bf16(map, base, rank, dims, strides_elems, box);
}

}  // namespace

bool prefill_tc_stride(int64_t st) { return st > 0 && (st % 8) == 0 && st < (int64_t(1) << 39); }

bool prefill_tc_supported(const flare_fwd_args_t* a) { return a->dtype == FLARE_BF16 && prefill_tc_shape(a); }

bool prefill_tc_supported_f16(const flare_fwd_args_t* a) {
  return a->dtype == FLARE_F16 && a->keep == nullptr && prefill_tc_shape(a);
}

bool prefill_tc_shape(const flare_fwd_args_t* a) {
  const int bs = a->block_size;
  const bool block_ok = bs == 1 || ((bs == 16 || bs == 32 || bs == 64 || bs == 128) && a->N % bs == 0);
  // the per-block encoder normalisers exist in block-causal mode only; the decode log-sum-exp in every mode
  const bool lse_ok = a->lse_enc == nullptr || bs > 1;
  if (a->lengths != nullptr && bs > 1) return false;  // per-row lengths: token-causal only
  // stablemax encoder weights: token-causal only
  const bool variant_ok = a->variant == FLARE_SOFTMAX || (a->variant == FLARE_STABLEMAX && bs == 1 && a->power > 0.f);
  // (of a tensor expanded over heads, with a stride of 0, fp16 calls make a copy; bf16 ones are served by the exact kernels)
  const int64_t strides[] = {a->k_stride_b, a->k_stride_n, a->k_stride_h, a->v_stride_b, a->v_stride_n, a->v_stride_h,
                             a->q_stride_h, a->q_stride_m};
  for (int64_t st : strides)
    if (!prefill_tc_stride(st)) return false;
  return variant_ok && block_ok && lse_ok && a->M <= 4 * M && a->M >= 16 &&
         (a->M % 16) == 0 && ((a->Dk == 64 && (a->Dv == 64 || a->Dv == 128)) || (a->Dk == 128 && a->Dv == 128)) && a->q_dec == nullptr &&
         a->k_dec == nullptr && a->mask == nullptr && a->N >= 1;
}

// Merge of the latent groups' partial read-outs: y = sum_g w_g y_g / sum_g w_g with w_g = exp2(lw_g - max lw).
// One thread per (token, head, 8 value columns).
__global__ void __launch_bounds__(256) tc_merge_groups_kernel(const __half* part_y, const float* part_lw,
                                                               int groups, int64_t rows /* B*N*H */, int N, int H, int dv,
                                                               uint16_t* y, int y_f16, int64_t y_stride_b, int64_t y_stride_n,
                                                               int64_t y_stride_h, float* lse_dec /* [B, H, N] or null */,
                                                               const int32_t* lens /* [B] or null */,
                                                               const int32_t* row_start /* [B] or null */, uint16_t* y_in,
                                                               int64_t yi_stride_b, int64_t yi_stride_n, int64_t yi_stride_h,
                                                               int* gate, int gate_stride, int gate_off) {
  pdl_begin();
  const int cols8 = dv >> 3;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * cols8) return;
  const int64_t row = idx / cols8;
  const int c8 = (int)(idx % cols8);
  if (lens != nullptr && (int)((row / H) % N) >= lens[row / ((int64_t)H * N)]) return;  // right padding: nothing emitted
  float lw[4], mx = -INFINITY;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    lw[g] = g < groups ? part_lw[g * rows + row] : -INFINITY;
    mx = fmaxf(mx, lw[g]);
  }
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, wsum = 0.f;
  if (mx == -INFINITY) {
    if (c8 == 0) {  // every group's weights underflowed: outside the numeric domain
      atomicOr(&g_tc_error, 2);
      // (the lane's words were written by the CTAs before this kernel: raise the first of them)
      if (gate != nullptr) gate[1 + ((row / ((int64_t)H * N)) * H + (row % H)) * gate_stride + gate_off] = 1;
    }
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      if (g >= groups) break;
      const float w = exp2f(lw[g] - mx);
      wsum += w;
      const uint4 raw = *reinterpret_cast<const uint4*>(part_y + (g * rows + row) * dv + c8 * 8);
      const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&rw[j]));
        acc[2 * j] += w * f.x;
        acc[2 * j + 1] += w * f.y;
      }
    }
  }
  const float inv = wsum > 0.f ? 1.0f / wsum : 0.f;
  const int h = (int)(row % H);
  const int64_t bn = row / H;
  const int n = (int)(bn % N);
  const int64_t b = bn / N;
  if (lse_dec != nullptr && c8 == 0) lse_dec[(b * H + h) * N + n] = (mx + log2f(wsum)) * kLn2;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] *= inv;
  uint32_t o[4];
  pack_out(acc, y_f16 != 0, o);
  const int row0 = row_start != nullptr ? row_start[b] : -1;  // (>= 0: a row of a masked call that was not packed)
  uint16_t* const dst = row0 >= 0 ? y_in + b * yi_stride_b + (int64_t)(n + row0) * yi_stride_n + (int64_t)h * yi_stride_h
                                  : y + b * y_stride_b + (int64_t)n * y_stride_n + (int64_t)h * y_stride_h;
  *reinterpret_cast<uint4*>(dst + c8 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}


int prefill_tc_latent_groups(const flare_fwd_args_t* a) { return (a->M + M - 1) / M; }

int prefill_tc_grid_z(const flare_fwd_args_t* a, bool wide) { return prefill_tc_latent_groups(a) * (wide ? 1 : a->Dv / D); }

// Which instance of the (128, 128) head shape runs - two CTAs per (lane, latent group), each repeating the score / E / R
// work for 64 value columns, or the wide one, one CTA for all 128 columns (not for a padded latent bank) - and into how
// many sequence segments a lane is cut: whatever an estimate of the call's time makes shortest.  Segments cost a state-only
// pass over all but the last and a scan of the segment states, and are taken only as far as all CTAs run in ONE wave (64
// lanes in 3 segments = 192 CTAs measured 0.140 ms for the read-out pass alone against 0.185 ms unsegmented).
// The constants are fits to runs on B200 in us per chunk of 128 tokens and pass: two-slice or 64-column instance 2.55
// (M = 64, 128 at D = 64; M = 128 at D = 128) and 1.4 for its state-only pass, wide 3.2 and 1.3; launch and fill 8, with
// segments 22 and 3 per MB of segment states.  Measured against the choices of the rule before it (half a wave of CTAs is
// the most that is cut, at 256 tokens or more per segment; wide only beyond one wave): B=1 H=16 M=128 D=128 N=32768
// 306 -> 190 us (4 segments of two slices -> 9 wide), B=1 H=32 N=8192 166 -> 124 us, B=1 H=16 M=64 D=64 N=777
// 32 -> 26 us (3 segments -> 1).
static bool can_wide(const flare_fwd_args_t* a) { return a->Dk == 128 && a->Dv == 128 && (a->M % M) == 0; }

// estimated time of the call on one instance, and the segments that give it
static double plan_instance(const flare_fwd_args_t* a, bool wide, size_t state_bytes, int* nseg_out) {
  const int nch = (a->N + C - 1) / C;
  const int64_t lanes = (int64_t)a->B * a->H;
  const int sms = sm_count();
  const double pass = wide ? 3.2 : 2.55, state_pass = wide ? 1.3 : 1.4;
  const int64_t ctas = lanes * prefill_tc_grid_z(a, wide);
  const double waves = (double)((ctas + sms - 1) / sms);
  double best = 8.0 + waves * nch * pass;
  *nseg_out = 1;
  if (ctas * 2 > sms) return best;
  int most = (int)(sms / ctas) < nch ? (int)(sms / ctas) : nch;
  const size_t room = state_bytes / ((size_t)lanes * (2 * a->M + (size_t)a->M * a->Dv) * sizeof(float));
  if ((size_t)most > room) most = (int)room;
  if (most < 2) return best;
  const int len = (nch + most - 1) / most, n = (nch + len - 1) / len;  // chunks per segment, segments that many make
  const double t = 22.0 + 3e-6 * (double)lanes * n * a->M * a->Dv * 4 + len * (pass + state_pass);
  if (1.1 * t < best) best = t, *nseg_out = n;  // (worth two more launches)
  return best;
}

void prefill_tc_plan(const flare_fwd_args_t* a, size_t state_bytes, int* nseg_out, bool* wide_out) {
  bool try_wide[2] = {true, can_wide(a)};
  if (const char* env = getenv("FLARE_B200_WIDE")) {  // 0 / 1 forces the instance
    try_wide[0] = env[0] != '1' || !try_wide[1];
    try_wide[1] = env[0] == '1' && try_wide[1];
  }
  double best = 1e30;
  for (int w = 0; w < 2; ++w) {
    if (!try_wide[w]) continue;
    int n = 1;
    const double t = plan_instance(a, w != 0, state_bytes, &n);
    // (segments are worth it only if they also beat the other instance by a tenth)
    if ((n > 1 ? 1.1 * t : t) < best) best = t, *nseg_out = n, *wide_out = w != 0;
  }
}

int prefill_tc_gate_stride(const flare_fwd_args_t* a, int nseg, bool wide) {
  return (2 * nseg - 1) * prefill_tc_grid_z(a, wide);  // state pass over all segments but the last, read-out over all
}

int prefill_tc_max_gate_stride(const flare_fwd_args_t* a) {
  int most = 0;
  for (int w = 0; w < (can_wide(a) ? 2 : 1); ++w) {
    int n = 1;
    plan_instance(a, w != 0, SIZE_MAX, &n);
    const int stride = prefill_tc_gate_stride(a, n, w != 0);
    if (stride > most) most = stride;
  }
  return most;
}

// fp16 partial read-outs [groups][B][N][H][Dv], then fp32 weight masses [groups][B][N][H]
size_t prefill_tc_partial_lw_offset(const flare_fwd_args_t* a) {
  const int groups = prefill_tc_latent_groups(a);
  return align_up((size_t)groups * a->B * a->N * a->H * a->Dv * sizeof(__half), 256);
}

size_t prefill_tc_partial_bytes(const flare_fwd_args_t* a) {
  const int groups = prefill_tc_latent_groups(a);
  if (groups == 1) return 0;
  return prefill_tc_partial_lw_offset(a) + (size_t)groups * a->B * a->N * a->H * sizeof(float);
}

bool prefill_tc_rows_in_place(const flare_fwd_args_t* a) {
  if (!prefill_tc_shape(a)) return false;
  if (a->y == nullptr) return true;
  for (int64_t st : {a->y_stride_b, a->y_stride_n, a->y_stride_h})
    if (!prefill_tc_stride(st)) return false;
  return (reinterpret_cast<uintptr_t>(a->y) % 16) == 0;
}

int launch_prefill_tc(const flare_fwd_args_t* a, const TcParams& p_in, int nseg_grid, bool wide, const flare_fwd_args_t* direct,
                      cudaStream_t stream) {
  TcParams p = p_in;
  {
    const int rc = tc_error_word(&p.err);
    if (rc != FLARE_OK) return rc;
  }
  p.block = a->block_size;
  p.power = a->power;
  p.lens = a->lengths;
  p.lse_dec = a->lse_dec;
  p.lse_enc = a->lse_enc;
  if (p.y == nullptr) {  // state-only passes emit nothing else
    p.lse_dec = p.lse_enc = nullptr;
    p.dump_u = nullptr;
  }
  if (p.row_start == nullptr) direct = nullptr;
  CUtensorMap tq, tk, tv, in[2];
  {
    // latent bank (used by the Dk = 64 instances only; any valid map otherwise)
    const uint64_t dims[3] = {(uint64_t)a->Dk, (uint64_t)a->M, (uint64_t)a->H};
    const int64_t str[2] = {a->q_stride_m, a->q_stride_h};
    const uint32_t box[3] = {64, a->M <= 64 ? 64u : 128u, 1};
    if (!make_map(&tq, a->q, 3, dims, str, box)) {
      set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (latent bank)");
      return FLARE_ERR_CUDA;
    }
  }
  {
    const uint64_t dimk[4] = {(uint64_t)a->Dk, (uint64_t)a->H, (uint64_t)a->N, (uint64_t)a->B};
    const uint64_t dimv[4] = {(uint64_t)a->Dv, (uint64_t)a->H, (uint64_t)a->N, (uint64_t)a->B};
    const uint32_t box[4] = {64, 1, 128, 1};
    const int64_t strk[3] = {a->k_stride_h, a->k_stride_n, a->k_stride_b};
    const int64_t strv[3] = {a->v_stride_h, a->v_stride_n, a->v_stride_b};
    if (!make_map(&tk, a->k, 4, dimk, strk, box) || !make_map(&tv, a->v, 4, dimv, strv, box)) {
      set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (keys / values)");
      return FLARE_ERR_CUDA;
    }
    in[0] = tk;
    in[1] = tv;
    if (direct != nullptr) {
      const int64_t sk[3] = {direct->k_stride_h, direct->k_stride_n, direct->k_stride_b};
      const int64_t sv[3] = {direct->v_stride_h, direct->v_stride_n, direct->v_stride_b};
      if (!make_map(&in[0], direct->k, 4, dimk, sk, box) || !make_map(&in[1], direct->v, 4, dimv, sv, box)) {
        set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (keys / values of a masked call)");
        return FLARE_ERR_CUDA;
      }
    }
  }
  if (p.dump_u != nullptr && !wide) {
    // kept states [lanes][chunks][M][Dv], a value slice of a latent group at a time
    const uint64_t dims[4] = {(uint64_t)a->Dv, (uint64_t)a->M, (uint64_t)p.dump_nch, (uint64_t)a->B * a->H};
    const int64_t str[3] = {a->Dv, (int64_t)a->M * a->Dv, (int64_t)p.dump_nch * a->M * a->Dv};
    const uint32_t box[4] = {64, a->M <= 64 ? 64u : 128u, 1, 1};
    if (!tc::make_map_bf16(&in[0], p.dump_u, 4, dims, str, box)) {
      set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (kept states)");
      return FLARE_ERR_CUDA;
    }
  }
  const int groups = prefill_tc_latent_groups(a);
  // packed below 65 latents (see PACK)
  const int lat = a->M <= 64 ? 2 : ((a->M % M) != 0 ? 1 : 0);
  const int mode = a->variant == FLARE_STABLEMAX ? 2 : (a->block_size > 1 ? 1 : 0);
  // Read-out rows leave through tiled bulk stores of 32 tokens x 32 columns (64-byte swizzle): into y, or with several
  // latent groups into the dense fp16 partials.  Per-row lengths (rows beyond a length stay untouched) and output
  // strides the tiled copy cannot express fall back to per-thread stores.
  CUtensorMap ty = tk;
  p.y_tma = 0;
  p.cluster_merge = 0;
  if (p.y != nullptr && a->lengths == nullptr) {
    const uint32_t box[4] = {32, 1, 32, 1};
    const int64_t str[3] = {p.y_stride_h, p.y_stride_n, p.y_stride_b};
    bool y_ok = (reinterpret_cast<uintptr_t>(p.y) % 16) == 0;
    for (int64_t st : str) y_ok = y_ok && prefill_tc_stride(st);
    const uint64_t ydims[4] = {(uint64_t)a->Dv, (uint64_t)a->H, (uint64_t)a->N, (uint64_t)a->B};
    // wide instance with exactly two latent groups: the two CTAs of a lane merge on chip (thread-block cluster) and
    // store y themselves.  FLARE_B200_CLUSTER=0 keeps the partials in global memory and the merge kernel.
    bool cluster = wide && groups == 2 && y_ok;
    if (const char* env = getenv("FLARE_B200_CLUSTER"))
      if (env[0] == '0') cluster = false;
    if (cluster && tc::make_map_bf16(&ty, p.y, 4, ydims, str, box, CU_TENSOR_MAP_SWIZZLE_64B)) {
      p.y_tma = 1;
      p.cluster_merge = 1;
    } else if (groups > 1) {
      const uint64_t dims[4] = {(uint64_t)a->Dv, (uint64_t)a->H, (uint64_t)a->N, (uint64_t)groups * a->B};
      const int64_t pstr[3] = {a->Dv, (int64_t)a->H * a->Dv, (int64_t)a->N * a->H * a->Dv};
      p.y_tma = tc::make_map_bf16(&ty, p.part_y, 4, dims, pstr, box, CU_TENSOR_MAP_SWIZZLE_64B) ? 1 : 0;
    } else {
      p.y_tma = y_ok && tc::make_map_bf16(&ty, p.y, 4, ydims, str, box, CU_TENSOR_MAP_SWIZZLE_64B) ? 1 : 0;
    }
  }
  if (direct != nullptr && p.y != nullptr && groups == 1) {
    // rows of a masked call that stay where they are: their y goes straight to the caller's tensor
    const uint32_t box[4] = {32, 1, 32, 1};
    const int64_t str[3] = {direct->y_stride_h, direct->y_stride_n, direct->y_stride_b};
    const uint64_t ydims[4] = {(uint64_t)a->Dv, (uint64_t)a->H, (uint64_t)a->N, (uint64_t)a->B};
    if (!tc::make_map_bf16(&ty, direct->y, 4, ydims, str, box, CU_TENSOR_MAP_SWIZZLE_64B)) {
      set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (output of a masked call)");
      return FLARE_ERR_CUDA;
    }
    p.y_tma = 1;
  } else if (const char* env = getenv("FLARE_B200_ROW_STORES"))  // diagnostic: per-thread row stores instead
    if (env[0] == '1' && !p.cluster_merge) p.y_tma = 0;
  const dim3 grid(a->B * a->H, nseg_grid, prefill_tc_grid_z(a, wide));
  const int combo = a->Dk == 128 ? 1 : (a->Dv == 128 ? 2 : 0);  // (64, 64), (128, 128), (64, 128)
  const int unit = wide ? (groups > 1 ? 7 : 6) : combo + (groups > 1 ? 3 : 0);
  using Launch = int (*)(int, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const CUtensorMap*,
                         const TcParams&, dim3, cudaStream_t);
#define FLARE_TC_UNIT_ROW(U) {launch_prefill_tc_unit<U, 0>, launch_prefill_tc_unit<U, 1>, launch_prefill_tc_unit<U, 2>}
  static constexpr Launch launch[8][3] = {FLARE_TC_UNIT_ROW(0), FLARE_TC_UNIT_ROW(1), FLARE_TC_UNIT_ROW(2), FLARE_TC_UNIT_ROW(3),
                                          FLARE_TC_UNIT_ROW(4), FLARE_TC_UNIT_ROW(5), FLARE_TC_UNIT_ROW(6), FLARE_TC_UNIT_ROW(7)};
#undef FLARE_TC_UNIT_ROW
  const int rc = launch[unit][mode](lat, tq, tk, tv, ty, in, p, grid, stream);
  if (rc != FLARE_OK || groups == 1 || p.y == nullptr || p.cluster_merge) return rc;
  const int64_t rows = (int64_t)a->B * a->N * a->H;
  const int64_t threads = rows * (a->Dv / 8);
  LaunchTimer timer("tc_merge_groups_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(tc_merge_groups_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, stream,
                              reinterpret_cast<const __half*>(p.part_y), p.part_lw, groups, rows, a->N, a->H, a->Dv,
                              reinterpret_cast<uint16_t*>(p.y), p.f16, p.y_stride_b, p.y_stride_n, p.y_stride_h, p.lse_dec, p.lens,
                              p.row_start, direct != nullptr ? reinterpret_cast<uint16_t*>(direct->y) : nullptr,
                              direct != nullptr ? direct->y_stride_b : 0, direct != nullptr ? direct->y_stride_n : 0,
                              direct != nullptr ? direct->y_stride_h : 0, p.gate, p.gate_stride, p.gate_off));
  return FLARE_OK;
}

int tc_error_word(int** device_address) {
  void* err = nullptr;
  FLARE_CUDA_CHECK(cudaGetSymbolAddress(&err, g_tc_error));  // of the current device and context: not remembered
  *device_address = reinterpret_cast<int*>(err);
  return FLARE_OK;
}

int prefill_tc_error_flag(int* host_value, bool reset) {
  int v = 0;
  FLARE_CUDA_CHECK(cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)));
  if (reset && v != 0) {
    const int zero = 0;
    FLARE_CUDA_CHECK(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int)));
  }
  *host_value = v;
  return FLARE_OK;
}

#endif  // FLARE_TC_UNIT

}  // namespace flare
