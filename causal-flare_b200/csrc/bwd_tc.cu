// Tensor-core (tcgen05 + TMEM + TMA) backward of causal FLARE, bf16 operands, fp32 accumulation and statistics.
// Shape class: the one of the tensor-core forward (prefill_tc.cu) with shared decode weights: softmax encoder token-
// or block-causal (blocks of 16 / 32 / 64 / 128), stablemax encoder token-causal; (Dk, Dv) = (64, 64), (128, 128),
// (64, 128); M a multiple of 16, up to 256 (Dk = 128) or 512 (Dk = 64).
//
// Per (batch, head) lane, chunks of C = 128 tokens are walked from the last to the first.  The forward kernel has
// left, per chunk i, the frame c_i[m] (log2 units), the encoder denominator d_i[m] and the numerator U_i[m, :] (bf16)
// of the state BEFORE the chunk, and per token the decode log-sum-exp L_t; delta_t = <dY_t, y_t>.  With
//   E[m,t] = exp2(s2[m,t] - c_i[m])   (stablemax: sigma(s))        D[m,t] = d_i[m] + sum_{tau <= t} E[m,tau]
//   g[m,t] = exp2(s2[m,t] - L_t)      decode softmax               R[m,t] = g / D
//   A[tau,t] = <v_tau, dY_t>,  vis(tau, t) = tau <= t  (block-causal: tau <= end of the block of t; D at block ends)
// and the reverse carries G[m,:] = sum_{t in later chunks} R dY_t, Cc[m] = sum_{t later} R p (both in the frame c_i):
//   P    = U_i dY^T + E (A . vis)                          p = P / D = <z_t[m], dY_t>
//   X    = G V^T   + R (A . vis)^T
//   dS   = R (P - D delta_t)  +  E slope (X - Cc - sum_{t' >= t} R p)          slope = 1 | sigma'/sigma
//   dV   = E^T G + (E^T R . vis) dY
//   G   += R dY,  Cc += sum_t R p,  then both are rescaled by exp2(c_{i-1} - c_i) for the next chunk.
// dS is written per latent as a hi and a lo bf16 row over the tokens ([lane][2][m][t], dS = hi + lo); a second tensor-core
// kernel forms dK = scale dS^T Q per chunk and dQ = scale sum_t dS K per (lane, split) (fp32 partials, summed in fixed order:
// no atomics, deterministic).
//
// Main kernel, one CTA per (lane, group of 128 latents, sequence segment), 23 warps: 0-15 latent group (thread = latent = TMEM
// lane, the four warps of a lane quarter take 32 tokens each; packed: see PACK), 16-19 token group (thread = token = TMEM lane:
// causal masks of A and E^T R, dV store), 20 MMA issuer, 21 TMA producer, 22 stores of dS (elected threads: with lane 0
// of the issuer and the producer, a training step B=4 N=4096 H=16 M=128 D=64 took 496 instead of 484 us).  Ten MMAs per chunk;
// every operand that the latent / token threads produce (E, R, masked A, G as bf16) is written once into a 128-byte-swizzled
// buffer and read K-major or MN-major as the product needs, so there is no transposition pass.
#include "bwd_tc.cuh"

#include <cuda.h>
#include <string.h>

#include "bwd_exact.cuh"
#include "prefill_tc.cuh"
#include "sm100_ptx.cuh"
#include "tc_device.cuh"

namespace flare {

using namespace sm100;
using tc::bf16_hi;
using tc::bf16_lo;
using tc::kmaj_step;
using tc::mnmaj_step;
using tc::sigma8;
using tc::swz_chunk_off;
using tc::warp_arrive;

constexpr int kMaxBwdSegments = 16;

struct BwdTcParams {
  const void* q;  // bf16 latent bank [H, M, Dk]
  int64_t q_stride_h, q_stride_m;
  int N, H, M;  // M: all latents
  int nch;      // chunks of 128 tokens per lane
  int npad;     // nch * 128
  int block;    // 1 or 16 / 32 / 64 / 128
  float scale, power;
  const float *chunk_c, *chunk_d;  // [lanes][nch][M]
  const float *tok_l2, *tok_delta;  // [lanes][npad]
  // Sequence segments (grid.z = the segments from seg_first on, segment s = chunks seg_begin[s] .. seg_begin[s + 1] - 1).
  int nseg, seg_first;
  int lead;       // the CTA of a segment first walks all later chunks for their carries alone (no exchange)
  int emit_only;  // carries of the segment alone, written to xg / xc in the frame of the chunk before the segment
  float *xg, *xc;  // [lanes][nseg][M][Dv], [lanes][nseg][M]; null: no exchange
  int seg_begin[kMaxBwdSegments + 1];
  int* gate;  // per-call gate word (may be null): raised when a carry turns non-finite (inputs outside the numeric domain)
  int* err;
  long long* trace;  // optional diagnostic cycle stamps of CTA (0, 0), see BT_TRACE; null in normal use
};

struct GradTcParams {
  int H, M;
  int nch, groups;
  int nsplit, chunks_per_split;
  float scale;
  int plane, nds, nk;  // bytes of a dS plane of the ring, stages (see grad_rings)
  float* dq_part;  // fp32 [B * nsplit][H][M][Dk]
  int* err;
};

// one instance family per head-width combination, compiled in its own translation unit
template <int UNIT>
int launch_bwd_tc_unit(int mode, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdy, const CUtensorMap& tu,
                       const CUtensorMap& tds, const CUtensorMap& tdv, const BwdTcParams& p, dim3 grid, cudaStream_t stream);

namespace {

constexpr int C = 128;
constexpr int LW = 4;                           // latent warps per lane quarter
// Latent warps, token warps, MMA issuer, TMA producer, dS stores: six warps on a scheduler, 80 registers a thread, and the latent warps
// spill.  Bytes of spill stores, softmax / block-causal / stablemax, at (Dk, Dv) = (64, 64) 132 / 44 / 128, (128, 128) 212 / 132 / 232,
// (64, 128) 200 / 144 / 220; packed 4 / 0 / 4, 56 / 48 / 64, 12 / 52 / 16.  (With dS and dV stored by their threads, at the same 80
// registers, the packed ones spilled at most 12 and the others up to 188; the kernel with tiles is the faster one all the same.)
constexpr int NT_MAIN = (4 * LW + 4 + 3) * 32;
constexpr int W_TOKEN = 4 * LW, W_MMA = 4 * LW + 4, W_TMA = 4 * LW + 5, W_OUT = 4 * LW + 6;  // (W_TOKEN: the first of four)
constexpr float kLog2e = 1.4426950408889634f;

// shared memory map of the main kernel (bytes; every operand buffer 1024-aligned for the 128B swizzle)
template <int DVB>
struct BL {
  static constexpr int OFF_KA = 0;                      // K tile [DKB][128 t][64]; later the masked A [2][128 tau][64 t]
  static constexpr int OFF_V = 32768;                   // [DVB][128 t][64]
  static constexpr int OFF_DY = OFF_V + DVB * 16384;    // [DVB][128 t][64]
  // U_i [DVB][128 m][64], and the chunk's dV rows on their way out, DV / 32 tiles of 32 x 32 for each of the four token warps:
  // at Dv = 64 behind U_i, at Dv = 128 in its place
  static constexpr int OFF_UR = OFF_DY + DVB * 16384;
  static constexpr int DV_TILES = DVB * 2 * 2048;  // bytes of a token warp's tiles
  static constexpr int OFF_DVT = OFF_UR + (DVB == 1 ? 16384 : 0);
  static constexpr int OFF_GC = OFF_UR + 32768;         // G as bf16 [DVB][128 m][64]
  static_assert(OFF_DVT + 4 * DV_TILES <= OFF_GC && OFF_DVT % 1024 == 0, "tiles of dV");
  static constexpr int OFF_E = OFF_GC + DVB * 16384;    // [2 t-blocks][128 m][64 t]
  static constexpr int OFF_R = OFF_E + 32768;
  static constexpr int OFF_MISC = OFF_R + 32768;
  static constexpr int SMEM_BYTES = OFF_MISC + 3072;  // Misc + what the manual 1024-byte alignment may cost
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};
// tensor-memory columns: T0 / T1 transient accumulators, T2 the masked E^T R as bf16 (A operand), TQ the latent bank
// as packed bf16 (A operand of the score product), TG the carry G (fp32)
constexpr uint32_t T0 = 0, T1 = 128, T2 = 256, TQ = 320, TG = 384, TM_COLS = 512;

struct Misc {
  uint64_t k_full, v_full, dy_full, u_full, q_ready;
  uint64_t s_ready, a_ready, px_ready, g_ready, wt_ready, dv_ready;
  uint64_t er_done, am_done, p_free, x_done, wm_done, dv_free, gc_done, ds_out, dv_out;
  uint64_t psum[4], prp[4];
  uint32_t tmem_base;
  volatile int abort_flag;
  float xch[LW * 128];  // exchange between the token parts of a latent row, [part][latent]: sums of E, then sums of R p
};
static_assert(sizeof(Misc) <= 2560, "Misc must leave room for the alignment slack");

// waits between roles are long (thousands of cycles): one quick look, then suspend
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, Misc* misc) {
  return tc::wait_or_abort(bar, parity, &misc->abort_flag, 1);
}
// exchange between the four warps of a lane quarter, which run in step: poll
__device__ __forceinline__ bool wait_partner(uint64_t* bar, uint32_t parity, Misc* misc) {
  return tc::wait_or_abort(bar, parity, &misc->abort_flag, 48);
}

// optional cycle trace of CTA (0, 0): [role < 4][chunk step < 8][slot < 8] clock64 stamps (diagnostic hook)
#define BT_TRACE(role, step, slot)                                                             \
  do {                                                                                         \
    if (p.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (step) < 8) \
      p.trace[((role) * 8 + (step)) * 8 + (slot)] = clock64();                                 \
  } while (0)

__device__ __forceinline__ float unpack8(const uint4& v, int j) {
  const uint32_t w = j < 2 ? v.x : (j < 4 ? v.y : (j < 6 ? v.z : v.w));
  return (j & 1) ? bf16_hi(w) : bf16_lo(w);
}
// slope sigma'(s) / sigma(s) = p / (1 + |s|) recovered from the (rounded) weight: 1 + |s| = E^(1/p) for s >= 0
// (E >= 1) and E^(-1/p) for s < 0; eight weights at a time, so that the power is looked at once for all of them.  The default
// power takes one reciprocal square root instead of a logarithm and an exponential (a weight of zero stays a slope of zero).
__device__ __forceinline__ void slope8_from_sigma(const float (&e)[8], float p, float (&slope)[8]) {
  if (p == 2.0f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float r = rsqrtf(fmaxf(e[j], 1e-37f));
      slope[j] = 2.0f * (e[j] >= 1.0f ? r : e[j] * r);
    }
  } else {
    const float inv_p = 1.0f / p;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float l = __log2f(e[j]) * inv_p;
      slope[j] = p * ex2_approx(e[j] >= 1.0f ? -l : l);
    }
  }
}

}  // namespace

#ifdef FLARE_BT_UNIT

// MODE 0: softmax encoder, token-causal; 1: block-causal read-out; 2: stablemax encoder, token-causal
// PACK: at most 64 latents would leave half of the 128 tensor-memory lanes, and with them the latent warps of two of the
//       four schedulers, without work in a kernel that is bound by the instructions of the latent passes.  As in the
//       forward the bank is laid down twice (rows 0..63 and 64..127): every latent's scores, P and X appear on two lanes, a
//       thread takes 16 tokens of the chunk instead of 32 and the two lanes share the columns of G (each maintains its own
//       ones, the others of its lane are never read).  Products over the latents read rows 0..63 only.
//       B200: training step B=4 N=4096 H=16 M=64 D=128 504 -> 412 us.
template <int DKB, int DVB, int MODE, bool PACK>
__global__ void __launch_bounds__(NT_MAIN, 1)
bwd_tc_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
              const __grid_constant__ CUtensorMap tm_dy, const __grid_constant__ CUtensorMap tm_u,
              const __grid_constant__ CUtensorMap tm_ds, const __grid_constant__ CUtensorMap tm_dv, const BwdTcParams p) {
  using L = BL<DVB>;
  constexpr bool BLOCK = MODE == 1, STABLE = MODE == 2;
  constexpr int DV = DVB * 64;
  constexpr int NP = PACK ? 2 * LW : LW;  // token parts of a chunk = latent warps per 32 latents
  constexpr int TOK = C / NP;             // tokens per latent thread
  constexpr int NG = TOK / 16;            // groups of 16 tokens among them
  constexpr int NCH = TOK / 8;            // 16-byte pieces of its operand rows
  constexpr int XL = PACK ? 64 : 128;     // latents of an exchange row
  // dS and dV leave through tiled bulk stores.  A thread storing its own row straight to global memory costs a transaction for every
  // 16 bytes, 4 096 (dS) and 2 048 (dV) a chunk at M = D = 128, and everything else that goes through the load / store unit waits
  // behind them: at M = 64, D = 128 the descending pass took 4 400 of a chunk's 15 700 cycles and the dV rows 4 200.
  // dS is laid down where E (hi) and R (lo) were: packed, in their second copies, which are free when P, X and G have been formed;
  // else in place, when the chunk's last product has run.  dV goes through U's slot, of which Dv = 64 uses half; at Dv = 128 the next
  // chunk's U comes when the rows have left.  B200, us a training step, dS (and dV where R's copy or U's slot had room) by threads -> in
  // tiles: B=4 N=4096 H=16 M=128 D=64 482 -> 450, M=64 D=128 376 -> 362, B=8 M=64 D=64 432 -> 392; all dV rows through U's slot: B=4
  // N=4096 H=32 M=128 D=128 723 -> 680, B=2 N=3000 H=8 M=96 D=128 165 -> 159, M <= 64 the same.
  pdl_wait();
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + L::OFF_MISC);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, group = blockIdx.y;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int nch = p.nch;
  // This CTA walks the chunks first - 1 .. begin.  Those from full_end on only move the carries (G, Cc): no X, no dV,
  // no dS.  All barriers run through the same phases in both kinds of chunk.
  const int seg = p.seg_first + blockIdx.z;
  const int begin = p.seg_begin[seg], end = p.seg_begin[seg + 1];
  const int full_end = p.emit_only ? begin : end;
  const int first = p.lead ? nch : end;
  const int steps = first - begin;
  const bool carry_in = p.xg != nullptr && !p.emit_only && seg + 1 < p.nseg;  // carries of the later segments, exchanged
  if ((int)(smem - smem_dyn) + L::OFF_MISC + (int)sizeof(Misc) > L::SMEM_BYTES) {
    // the dynamic shared memory window starts less aligned than this layout can absorb: report, do nothing
    if (tid == 0) atomicOr(p.err, 1);
    return;
  }

  if (tid == 0) {
    mbar_init(&misc->k_full, 1);
    mbar_init(&misc->v_full, 1);
    mbar_init(&misc->dy_full, 1);
    mbar_init(&misc->u_full, 1);
    mbar_init(&misc->q_ready, 4 * LW);
    mbar_init(&misc->s_ready, 1);
    mbar_init(&misc->a_ready, 1);
    mbar_init(&misc->px_ready, 1);
    mbar_init(&misc->g_ready, 1);
    mbar_init(&misc->wt_ready, 1);
    mbar_init(&misc->dv_ready, 1);
    mbar_init(&misc->er_done, 4 * LW);
    mbar_init(&misc->am_done, 4);
    mbar_init(&misc->p_free, 4 * LW);
    mbar_init(&misc->x_done, 4 * LW);
    mbar_init(&misc->wm_done, 4);
    mbar_init(&misc->dv_free, 4);
    mbar_init(&misc->gc_done, 4 * LW);
    mbar_init(&misc->ds_out, 1);
    mbar_init(&misc->dv_out, 4);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&misc->psum[i], NP);
      mbar_init(&misc->prp[i], NP);
    }
    misc->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == W_MMA) {
    tmem_alloc(&misc->tmem_base, TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = misc->tmem_base;
  bool ok = true;
  const int rows_here = min(128, p.M - group * 128);  // latents of this group
  const int ksm = (rows_here + 15) >> 4;              // 16-latent steps of a contraction over the latents

  if (warp == W_TMA) {
    // ======================================= TMA producer =======================================
    if (elect_one()) {
      prefetch_tensormap(&tm_k);
      prefetch_tensormap(&tm_v);
      prefetch_tensormap(&tm_dy);
      prefetch_tensormap(&tm_u);
      for (int j = 0; ok && j < steps; ++j) {
        const int i = first - 1 - j, t0 = i * C;
        const uint32_t pp = (j - 1) & 1;
        // K, V: free once the previous chunk's P / X products (which read the masked A and V) have run
        if (j > 0 && !(ok = wait_or_abort(&misc->px_ready, pp, misc))) break;
        mbar_arrive_expect_tx(&misc->k_full, DKB * 16384);
#pragma unroll
        for (int kb = 0; kb < DKB; ++kb) tma_load_4d(smem + L::OFF_KA + kb * 16384, &tm_k, &misc->k_full, kb * 64, h, t0, b);
        mbar_arrive_expect_tx(&misc->v_full, DVB * 16384);
#pragma unroll
        for (int vb = 0; vb < DVB; ++vb) tma_load_4d(smem + L::OFF_V + vb * 16384, &tm_v, &misc->v_full, vb * 64, h, t0, b);
        // dY: read by the previous chunk's dV and G products
        if (j > 0 && !(ok = wait_or_abort(&misc->dv_ready, pp, misc))) break;
        mbar_arrive_expect_tx(&misc->dy_full, DVB * 16384);
#pragma unroll
        for (int vb = 0; vb < DVB; ++vb) tma_load_4d(smem + L::OFF_DY + vb * 16384, &tm_dy, &misc->dy_full, vb * 64, h, t0, b);
        // U_i: read by the previous chunk's P product (which has run: px_ready above); at Dv = 128 the previous (full) chunk's dV rows
        // have left its slot
        if (DVB == 2 && j > 0 && i + 1 < full_end && !(ok = wait_or_abort(&misc->dv_out, (j - 1 - (first - full_end)) & 1, misc))) break;
        mbar_arrive_expect_tx(&misc->u_full, DVB * 16384);
#pragma unroll
        for (int vb = 0; vb < DVB; ++vb) {
          tma_load_4d(smem + L::OFF_UR + vb * 16384, &tm_u, &misc->u_full, vb * 64, group * 128, i, lane_id);
          if constexpr (PACK)  // (boxes of 64 rows)
            tma_load_4d(smem + L::OFF_UR + vb * 16384 + 8192, &tm_u, &misc->u_full, vb * 64, 0, i, lane_id);
        }
      }
      pdl_trigger();
    }
  } else if (warp == W_MMA) {
    // ======================================= MMA issuer =======================================
    if (elect_one()) {
      // All operands are bf16: tcgen05.mma kind::f16 wants A and B in ONE format (a descriptor that mixes fp16 and
      // bf16 operands is rejected by the hardware as an illegal instruction), and everything that scales with the
      // caller's data (V, dY, U, G, the masked A, R) needs the bf16 range.
      constexpr uint32_t ID_SS = make_idesc_bf16(128, 128, 0, 0);   // K-major x K-major (scores, A, U dY^T, G V^T, R A^T)
      constexpr uint32_t ID_PE = make_idesc_bf16(128, 128, 0, 1);   // E (K-major) x masked A (MN-major)
      constexpr uint32_t ID_WT = make_idesc_bf16(128, 128, 1, 1);   // E (MN-major) x R (MN-major)
      constexpr uint32_t ID_DV1 = make_idesc_bf16(128, DV, 1, 1);   // E (MN-major) x G (MN-major)
      constexpr uint32_t ID_DV2 = make_idesc_bf16(128, DV, 0, 1);   // masked E^T R (TMEM) x dY (MN-major)
      constexpr uint32_t ID_G = make_idesc_bf16(128, DV, 0, 1);     // R (K-major) x dY (MN-major)
      const uint64_t d_k = make_desc_sw128(smem_u32(smem + L::OFF_KA), 16, 1024);        // K tile, K-major
      const uint64_t d_am_k = d_k;                                                        // masked A, K-major (N = tau)
      const uint64_t d_am_mn = make_desc_sw128(smem_u32(smem + L::OFF_KA), 16384, 1024);  // masked A, MN-major (N = t)
      const uint64_t d_v_k = make_desc_sw128(smem_u32(smem + L::OFF_V), 16, 1024);
      const uint64_t d_dy_k = make_desc_sw128(smem_u32(smem + L::OFF_DY), 16, 1024);
      const uint64_t d_dy_mn = make_desc_sw128(smem_u32(smem + L::OFF_DY), 16384, 1024);
      const uint64_t d_u_k = make_desc_sw128(smem_u32(smem + L::OFF_UR), 16, 1024);
      const uint64_t d_g_k = make_desc_sw128(smem_u32(smem + L::OFF_GC), 16, 1024);
      const uint64_t d_g_mn = make_desc_sw128(smem_u32(smem + L::OFF_GC), 16384, 1024);
      const uint64_t d_e_k = make_desc_sw128(smem_u32(smem + L::OFF_E), 16, 1024);
      const uint64_t d_e_mn = make_desc_sw128(smem_u32(smem + L::OFF_E), 16384, 1024);
      const uint64_t d_r_k = make_desc_sw128(smem_u32(smem + L::OFF_R), 16, 1024);
      const uint64_t d_r_mn = make_desc_sw128(smem_u32(smem + L::OFF_R), 16384, 1024);

      ok = wait_or_abort(&misc->q_ready, 0, misc);  // the latent bank is in tensor memory
      tc_fence_after_sync();
      for (int j = 0; ok && j < steps; ++j) {
        const uint32_t par = j & 1, pp = (j - 1) & 1;
        const bool full = first - 1 - j < full_end;
        const uint32_t fpar = (j - (first - full_end)) & 1;  // parity among the full chunks
        const uint32_t have = (j > 0 || carry_in) ? 1u : 0u;  // G holds something
        // scores S^T = Q K^T -> T1 (the previous chunk's X has been read)
        if (!(ok = wait_or_abort(&misc->k_full, par, misc))) break;
        if (j > 0 && !(ok = wait_or_abort(&misc->x_done, pp, misc))) break;
        tc_fence_after_sync();
        BT_TRACE(2, j, 0);
#pragma unroll
        for (int s = 0; s < 4 * DKB; ++s) mma_ts(tmem + T1, tmem + TQ + s * 8, kmaj_step(d_k, s), ID_SS, s > 0);
        tc_commit(&misc->s_ready);
        // A = V dY^T -> T0 (the previous chunk's dV has been stored)
        if (!(ok = wait_or_abort(&misc->v_full, par, misc))) break;
        if (!(ok = wait_or_abort(&misc->dy_full, par, misc))) break;
        if (j > 0 && !(ok = wait_or_abort(&misc->dv_free, pp, misc))) break;
        tc_fence_after_sync();
        BT_TRACE(2, j, 1);
#pragma unroll
        for (int s = 0; s < 4 * DVB; ++s) mma_ss(tmem + T0, kmaj_step(d_v_k, s), kmaj_step(d_dy_k, s), ID_SS, s > 0);
        tc_commit(&misc->a_ready);
        // P -> T0, X -> T1, then G += R dY
        if (!(ok = wait_or_abort(&misc->er_done, par, misc))) break;
        if (!(ok = wait_or_abort(&misc->am_done, par, misc))) break;
        if (!(ok = wait_or_abort(&misc->u_full, par, misc))) break;
        if (j > 0 && !(ok = wait_or_abort(&misc->gc_done, pp, misc))) break;
        tc_fence_after_sync();
        BT_TRACE(2, j, 2);
#pragma unroll
        for (int s = 0; s < 4 * DVB; ++s) mma_ss(tmem + T0, kmaj_step(d_u_k, s), kmaj_step(d_dy_k, s), ID_SS, s > 0);
#pragma unroll
        for (int s = 0; s < 8; ++s) mma_ss(tmem + T0, kmaj_step(d_e_k, s), mnmaj_step(d_am_mn, s), ID_PE, 1);
        if (full) {
          if (have) {
#pragma unroll
            for (int s = 0; s < 4 * DVB; ++s) mma_ss(tmem + T1, kmaj_step(d_g_k, s), kmaj_step(d_v_k, s), ID_SS, s > 0);
          }
#pragma unroll
          for (int s = 0; s < 8; ++s) mma_ss(tmem + T1, kmaj_step(d_r_k, s), kmaj_step(d_am_k, s), ID_SS, s > 0 ? 1u : have);
        }
        tc_commit(&misc->px_ready);
#pragma unroll
        for (int s = 0; s < 8; ++s)
          mma_ss(tmem + TG, kmaj_step(d_r_k, s), mnmaj_step(d_dy_mn, s), ID_G, s > 0 ? 1u : have);
        tc_commit(&misc->g_ready);
        if (!full) tc_commit(&misc->dv_ready);  // (no dV: E, R and dY have been read)
        // W^T = E^T R -> T0 (P has been read; the wt_ready / wm_done phases count the full chunks only)
        if (!(ok = wait_or_abort(&misc->p_free, par, misc))) break;
        tc_fence_after_sync();
        BT_TRACE(2, j, 3);
        if (!full) continue;
        for (int s = 0; s < ksm; ++s) mma_ss(tmem + T0, mnmaj_step(d_e_mn, s), mnmaj_step(d_r_mn, s), ID_WT, s > 0);
        tc_commit(&misc->wt_ready);
        // dV = E^T G + (masked W^T) dY -> T0
        if (!(ok = wait_or_abort(&misc->wm_done, fpar, misc))) break;
        tc_fence_after_sync();
        BT_TRACE(2, j, 4);
        if (have)
          for (int s = 0; s < ksm; ++s) mma_ss(tmem + T0, mnmaj_step(d_e_mn, s), mnmaj_step(d_g_mn, s), ID_DV1, s > 0);
#pragma unroll
        for (int s = 0; s < 8; ++s) mma_ts(tmem + T0, tmem + T2 + s * 8, mnmaj_step(d_dy_mn, s), ID_DV2, s > 0 ? 1u : have);
        tc_commit(&misc->dv_ready);
      }
    }
  } else if (warp == W_OUT) {
    // ======================================= dS stores =======================================
    if (elect_one()) {
      prefetch_tensormap(&tm_ds);
      for (int j = 0; ok && j < steps; ++j) {
        const int i = first - 1 - j;
        if (!(ok = wait_or_abort(&misc->x_done, j & 1, misc))) break;
        if (i < full_end) {
          constexpr int COPY = PACK ? 8192 : 0;
#pragma unroll
          for (int tb = 0; tb < 2; ++tb) {  // (rows beyond M are clipped)
            tma_store_4d(&tm_ds, smem + L::OFF_E + tb * 16384 + COPY, i * C + tb * 64, group * 128, 0, lane_id);
            tma_store_4d(&tm_ds, smem + L::OFF_R + tb * 16384 + COPY, i * C + tb * 64, group * 128, 1, lane_id);
          }
          bulk_commit_group();
          bulk_wait_group_read0();
        }
        // In the chunks that only move the carries too, where there is nothing to store: the latent warps wait for this phase before
        // their next chunk, so that x_done cannot complete twice before this warp has looked at it (it would look unfinished then).
        mbar_arrive(&misc->ds_out);
      }
      bulk_wait_group0();
    }
  } else if (warp < 4 * LW) {
    // ======== latent group: thread = (latent = TMEM lane, part of the chunk's tokens); 4 warps per lane quarter ========
    const int tq = warp >> 2, q = warp & 3;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
    const int m = PACK ? (q & 1) * 32 + lane : q * 32 + lane;  // latent of the group
    const int tp = PACK ? tq * 2 + (q >> 1) : tq;              // token part
    const int pq = PACK ? (q & 1) : q;                         // exchange group: the NP warps of the same 32 latents
    auto xch = [&](int part) -> float& { return misc->xch[part * XL + m]; };
    // one 16-byte piece of an operand row (packed: of both copies)
    auto put = [&](uint8_t* rows, int ch, const uint4& v) {
      *reinterpret_cast<uint4*>(rows + swz_chunk_off(m, ch)) = v;
      if constexpr (PACK) *reinterpret_cast<uint4*>(rows + 8192 + swz_chunk_off(m, ch)) = v;
    };
    const int mg = group * 128 + m;
    const bool live = mg < p.M;
    const float sc2 = p.scale * kLog2e;
    const int tok0 = tp * TOK;
    // this thread's tokens are the 16-byte pieces from ch0 on of row m in t-block tok0 / 64 of the [2][128][64] buffers
    const int ch0 = (tok0 & 63) >> 3;
    uint8_t* const e_row = smem + L::OFF_E + (tok0 >> 6) * 16384;
    uint8_t* const r_row = smem + L::OFF_R + (tok0 >> 6) * 16384;
    {
      // latent bank row -> tensor memory as packed bf16 (element k in column k / 2); each warp of the quarter writes
      // 32 elements of the row (Dk = 64: the first two warps)
      if (tq * 32 < DKB * 64) {
        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.q) + (int64_t)h * p.q_stride_h +
                                                          (int64_t)(live ? mg : 0) * p.q_stride_m + tq * 32);
        uint32_t r[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 x = live ? src[i] : make_uint4(0, 0, 0, 0);
          r[4 * i] = x.x; r[4 * i + 1] = x.y; r[4 * i + 2] = x.z; r[4 * i + 3] = x.w;
        }
        tmem_st16(tl + TQ + tq * 16, r);
        tmem_wait_st();
      }
      tc_fence_before_sync();
      if (!carry_in) warp_arrive(&misc->q_ready, lane);
    }
    float cc_carry = 0.f;  // Cc: sum over later chunks of R p, in the current chunk's frame
    const int64_t stat0 = (int64_t)lane_id * nch * p.M + mg;
    // value columns of G this warp rescales and repacks
    constexpr int GCOLS = DV / NP;
    const int gcol = tp * GCOLS;
    uint8_t* const g_dst = smem + L::OFF_GC + (gcol >> 6) * 16384;
    const int gch0 = (gcol & 63) >> 3;
    if (carry_in) {
      // Carries of the later segments, summed from the last one on: every segment's are in the frame of the chunk before
      // it, and the frames only grow with the chunk, so the factors between them never exceed 1.
      float g[GCOLS];
#pragma unroll
      for (int k = 0; k < GCOLS; ++k) g[k] = 0.f;
      if (live) {
        float c_from = 0.f;
        for (int s = p.nseg - 1; s > seg; --s) {
          const int64_t xo = ((int64_t)lane_id * p.nseg + s) * p.M + mg;
          const float c_to = STABLE ? 0.f : p.chunk_c[stat0 + (int64_t)(p.seg_begin[s] - 1) * p.M];
          const float f = s == p.nseg - 1 ? 0.f : (STABLE ? 1.f : ex2_approx(c_to - c_from));
          c_from = c_to;
          cc_carry = fmaf(cc_carry, f, p.xc[xo]);
          const float4* src = reinterpret_cast<const float4*>(p.xg + xo * DV + gcol);
#pragma unroll
          for (int k = 0; k < GCOLS / 4; ++k) {
            const float4 x = src[k];
            g[4 * k] = fmaf(g[4 * k], f, x.x);
            g[4 * k + 1] = fmaf(g[4 * k + 1], f, x.y);
            g[4 * k + 2] = fmaf(g[4 * k + 2], f, x.z);
            g[4 * k + 3] = fmaf(g[4 * k + 3], f, x.w);
          }
        }
      }
      uint32_t r[GCOLS];
#pragma unroll
      for (int k = 0; k < GCOLS; ++k) r[k] = __float_as_uint(g[k]);
      tmem_write(tl + TG + gcol, r);
#pragma unroll
      for (int ch = 0; ch < GCOLS / 8; ++ch)
        put(g_dst, gch0 + ch,
            make_uint4(pack_bf16(g[ch * 8 + 0], g[ch * 8 + 1]), pack_bf16(g[ch * 8 + 2], g[ch * 8 + 3]),
                       pack_bf16(g[ch * 8 + 4], g[ch * 8 + 5]), pack_bf16(g[ch * 8 + 6], g[ch * 8 + 7])));
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      warp_arrive(&misc->q_ready, lane);
    }

    if (!__any_sync(0xffffffffu, live)) {
      // A warp whose 32 latents all lie beyond M (M <= 96, or the ragged last group): its operand rows are zero for
      // the whole kernel and it only keeps the barrier phases in step with the working warps.
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        put(e_row, ch0 + ch, make_uint4(0, 0, 0, 0));
        put(r_row, ch0 + ch, make_uint4(0, 0, 0, 0));
      }
#pragma unroll
      for (int ch = 0; ch < GCOLS / 8; ++ch) put(g_dst, gch0 + ch, make_uint4(0, 0, 0, 0));
      fence_proxy_async_smem();
      for (int j = 0; ok && j < steps; ++j) {
        const uint32_t par = j & 1, pp = (j - 1) & 1;
        if (j > 0 && !(ok = wait_or_abort(&misc->dv_ready, pp, misc))) break;
        if (!(ok = wait_or_abort(&misc->s_ready, par, misc))) break;
        warp_arrive(&misc->er_done, lane);
        if (!(ok = wait_or_abort(&misc->px_ready, par, misc))) break;
        warp_arrive(&misc->p_free, lane);
        warp_arrive(&misc->x_done, lane);
        if (j + 1 < steps) {
          if (!(ok = wait_or_abort(&misc->dv_ready, par, misc))) break;
          warp_arrive(&misc->gc_done, lane);
        }
      }
    } else {
      auto emit_g = [&](const uint32_t(&r)[GCOLS]) {  // this thread's columns of the segment's G, for the segments before
        if (!live) return;
        float4* dst = reinterpret_cast<float4*>(p.xg + (((int64_t)lane_id * p.nseg + seg) * p.M + mg) * DV + gcol);
#pragma unroll
        for (int k = 0; k < GCOLS / 4; ++k)
          dst[k] = make_float4(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]), __uint_as_float(r[4 * k + 2]),
                               __uint_as_float(r[4 * k + 3]));
      };
      // Per-chunk statistics of this thread's latent and per-token statistics of this warp's tokens (lane l keeps
      // token tok0 + l % TOK; the loops broadcast them with shuffles), all fetched one chunk ahead so that the global-memory
      // latency never sits between two phases.
      const float* const l2_row = p.tok_l2 + (int64_t)lane_id * p.npad + tok0 + (lane & (TOK - 1));
      const float* const dl_row = p.tok_delta + (int64_t)lane_id * p.npad + tok0 + (lane & (TOK - 1));
      float c_cur = (live && !STABLE) ? p.chunk_c[stat0 + (int64_t)(first - 1) * p.M] : 0.f;
      float d_cur = live ? p.chunk_d[stat0 + (int64_t)(first - 1) * p.M] : 1.f;
      float c_nxt = (live && !STABLE && first > 1) ? p.chunk_c[stat0 + (int64_t)(first - 2) * p.M] : c_cur;
      float l2_cur = l2_row[(int64_t)(first - 1) * C], dl_cur = dl_row[(int64_t)(first - 1) * C];

      for (int j = 0; ok && j < steps; ++j) {
        const int i = first - 1 - j, t0 = i * C;
        const uint32_t par = j & 1, pp = (j - 1) & 1;
        const int nvalid = min(C, p.N - t0);
        const int lim = live ? nvalid - tok0 : 0;  // tokens of this thread's part that exist (may be <= 0)
        const bool fast = __all_sync(0xffffffffu, lim >= TOK);
        const float c_i = c_cur, d_i = d_cur;
        const float c_prev = i > 0 ? c_nxt : c_i;
        const float l2_mine = l2_cur, dl_mine = dl_cur;
        // the next chunk's (i - 1) values, used one iteration from now
        if (tid == 0) BT_TRACE(3, j, 0);
        const float d_pre = (live && i > 0) ? ld_pinned(p.chunk_d + stat0 + (int64_t)(i - 1) * p.M) : 1.f;
        const float c_pre = (live && !STABLE && i > 1) ? ld_pinned(p.chunk_c + stat0 + (int64_t)(i - 2) * p.M) : c_nxt;
        const float l2_pre = i > 0 ? ld_pinned(l2_row + (int64_t)(i - 1) * C) : 0.f;
        const float dl_pre = i > 0 ? ld_pinned(dl_row + (int64_t)(i - 1) * C) : 0.f;
        // E / R buffers: the previous chunk's products have read them, and its dS has left them
        if (j > 0 && !(ok = wait_or_abort(&misc->dv_ready, pp, misc) && wait_or_abort(&misc->ds_out, pp, misc))) break;
        if (!(ok = wait_or_abort(&misc->s_ready, par, misc))) break;
        tc_fence_after_sync();
        if (tid == 0) BT_TRACE(0, j, 0);
        uint32_t rs[TOK];  // the raw scores of this thread
        tmem_read(tl + T1 + tok0, rs);
        if (tid == 0) BT_TRACE(3, j, 1);
        // ---- phase 1a: E rows (bf16) and their sums
        float g16[NG] = {};  // sums of the rounded E per 16 tokens
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          float e[8];
          if constexpr (STABLE) {
            float x[8];
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) x[jj] = __uint_as_float(rs[ch * 8 + jj]) * p.scale;
            sigma8(x, p.power, e);
          }
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            const int k = ch * 8 + jj;
            if constexpr (!STABLE) e[jj] = ex2_approx(fmaf(__uint_as_float(rs[k]), sc2, -c_i));
            if (!fast) e[jj] = k < lim ? e[jj] : 0.f;
          }
          uint4 v;
          v.x = pack_bf16(e[0], e[1]); v.y = pack_bf16(e[2], e[3]); v.z = pack_bf16(e[4], e[5]); v.w = pack_bf16(e[6], e[7]);
          g16[ch >> 1] += (bf16_lo(v.x) + bf16_hi(v.x)) + (bf16_lo(v.y) + bf16_hi(v.y)) + (bf16_lo(v.z) + bf16_hi(v.z)) +
                          (bf16_lo(v.w) + bf16_hi(v.w));
          put(e_row, ch0 + ch, v);
        }
        xch(tp) = NG == 2 ? g16[0] + g16[NG - 1] : g16[0];
        warp_arrive(&misc->psum[pq], lane);
        if (tid == 0) BT_TRACE(3, j, 2);
        if (!(ok = wait_partner(&misc->psum[pq], par, misc))) break;
        if (tid == 0) BT_TRACE(3, j, 3);
        // denominator before this thread's first token
        float base_run = d_i;
#pragma unroll
        for (int t = 0; t < NP - 1; ++t) base_run += t < tp ? xch(t) : 0.f;
        float dend[NG], invg[NG];  // block-causal: denominator at the end of the block of each 16-token group
        if constexpr (BLOCK) {
          const int bs = p.block;
          if (bs <= TOK) {  // the blocks end inside this part
            const float p0 = base_run + g16[0];
            dend[0] = p0;
            if constexpr (NG == 2) {
              dend[1] = p0 + g16[1];
              if (bs == 32) dend[0] = dend[1];
            }
          } else {
            // the block ends in a later part (or with this one): add the parts up to its last one
            const int last = tp | (bs / TOK - 1);
            float tot = base_run + xch(tp);
#pragma unroll
            for (int t = 1; t < NP; ++t) tot += (t > tp && t <= last) ? xch(t) : 0.f;
#pragma unroll
            for (int g = 0; g < NG; ++g) dend[g] = tot;
          }
#pragma unroll
          for (int g = 0; g < NG; ++g) invg[g] = rcp_approx(dend[g]);
        }
        // ---- phase 1b: R = g / D rows (bf16)
        {
          float run = base_run;
#pragma unroll
          for (int ch = 0; ch < NCH; ++ch) {
            const uint4 ev = *reinterpret_cast<const uint4*>(e_row + swz_chunk_off(m, ch0 + ch));
            float r[8];
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const int k = ch * 8 + jj;
              const float l2 = __shfl_sync(0xffffffffu, l2_mine, k);
              const float g = ex2_approx(fmaf(__uint_as_float(rs[k]), sc2, -l2));
              float inv;
              if constexpr (BLOCK) {
                inv = invg[ch >> 1];
              } else {
                run += unpack8(ev, jj);
                inv = rcp_approx(run);
              }
              float x = g * inv;
              if (!fast) x = k < lim ? x : 0.f;
              r[jj] = x;
            }
            put(r_row, ch0 + ch,
                make_uint4(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]), pack_bf16(r[4], r[5]), pack_bf16(r[6], r[7])));
          }
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        warp_arrive(&misc->er_done, lane);
        if (tid == 0) BT_TRACE(0, j, 1);

        // ---- phase 2a (ascending): p = P / D, R p, decode part of dS - everything stays in registers
        if (!(ok = wait_or_abort(&misc->px_ready, par, misc))) break;
        tc_fence_after_sync();
        if (tid == 0) BT_TRACE(0, j, 2);
        uint32_t pd[TOK];       // P accumulators of the tokens, replaced in place by the decode-side dS (fp32)
        uint32_t rpk[TOK / 2];  // R p, packed bf16 pairs
        float rg16[NG] = {};    // sums of the rounded R p per 16 tokens
        tmem_read(tl + T0 + tok0, pd);
        tc_fence_before_sync();
        warp_arrive(&misc->p_free, lane);  // T0 may take E^T R
        {
          float run = base_run;
#pragma unroll
          for (int ch = 0; ch < NCH; ++ch) {
            const uint4 ev = *reinterpret_cast<const uint4*>(e_row + swz_chunk_off(m, ch0 + ch));
            const uint4 rv = *reinterpret_cast<const uint4*>(r_row + swz_chunk_off(m, ch0 + ch));
            float rp[8];
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const int k = ch * 8 + jj;
              const float pacc = __uint_as_float(pd[k]);
              const float rbv = unpack8(rv, jj);
              const float dl = __shfl_sync(0xffffffffu, dl_mine, k);
              float dcur, inv;
              if constexpr (BLOCK) {
                dcur = dend[ch >> 1];
                inv = invg[ch >> 1];
              } else {
                run += unpack8(ev, jj);
                dcur = run;
                inv = rcp_approx(run);
              }
              rp[jj] = rbv * (pacc * inv);
              pd[k] = __float_as_uint(rbv * fmaf(-dcur, dl, pacc));
            }
#pragma unroll
            for (int jj = 0; jj < 8; jj += 2) {
              const uint32_t w = pack_bf16(rp[jj], rp[jj + 1]);
              rpk[ch * 4 + (jj >> 1)] = w;
              rg16[ch >> 1] += bf16_lo(w) + bf16_hi(w);
            }
          }
        }
        if (tid == 0) BT_TRACE(0, j, 3);
        const float rp_mine = NG == 2 ? rg16[0] + rg16[NG - 1] : rg16[0];
        xch(tp) = rp_mine;
        warp_arrive(&misc->prp[pq], lane);
        if (!(ok = wait_partner(&misc->prp[pq], par, misc))) break;
        if (tid == 0) BT_TRACE(3, j, 4);
        float rp_later = 0.f, rp_all = 0.f;  // R p of the parts after this one, and of the whole chunk
#pragma unroll
        for (int t = 0; t < NP; ++t) {
          const float x = xch(t);
          rp_all += x;
          rp_later += t > tp ? x : 0.f;
        }

        // ---- phase 2b (descending): encoder part, dS as a hi + lo pair into the tiles that the store warp sends off
        if (i < full_end) {
          // dS may be laid down (where E and R were, see the top of the kernel)
          if (!(ok = PACK ? wait_or_abort(&misc->g_ready, par, misc) : wait_or_abort(&misc->dv_ready, par, misc))) break;
          float ccg[NG];  // block-causal: Cc + sum of R p from the start of the group's block on
          float cc = cc_carry + rp_later;
          if constexpr (BLOCK) {
            const int bs = p.block;
            if (bs <= TOK) {
              ccg[NG - 1] = cc + rg16[NG - 1];
              if constexpr (NG == 2) {
                ccg[0] = ccg[1] + rg16[0];
                if (bs == 32) ccg[1] = ccg[0];
              }
            } else {
              // the block starts in an earlier (or this) part: add the parts from its first one on
              const int from = tp & ~(bs / TOK - 1);
              float tot = cc + rp_mine;
#pragma unroll
              for (int t = 0; t < NP - 1; ++t) tot += (t >= from && t < tp) ? xch(t) : 0.f;
#pragma unroll
              for (int g = 0; g < NG; ++g) ccg[g] = tot;
            }
          }
#pragma unroll
          for (int blk = NG - 1; blk >= 0; --blk) {
            uint32_t xr[16];
            tmem_read(tl + T1 + tok0 + blk * 16, xr);
#pragma unroll
            for (int c2 = 1; c2 >= 0; --c2) {
              const int ch = blk * 2 + c2;
              const uint4 ev = *reinterpret_cast<const uint4*>(e_row + swz_chunk_off(m, ch0 + ch));
              float ds[8], e8[8], slope[8];
#pragma unroll
              for (int jj = 0; jj < 8; ++jj) e8[jj] = unpack8(ev, jj);
              if constexpr (STABLE) slope8_from_sigma(e8, p.power, slope);
#pragma unroll
              for (int jj = 7; jj >= 0; --jj) {
                const int k = ch * 8 + jj;
                const float x = __uint_as_float(xr[c2 * 8 + jj]);
                const float eb = e8[jj];
                float csub;
                if constexpr (BLOCK) {
                  csub = ccg[ch >> 1];
                } else {
                  const uint32_t w = rpk[k >> 1];
                  cc += (k & 1) ? bf16_hi(w) : bf16_lo(w);
                  csub = cc;
                }
                float enc = eb * (x - csub);
                if constexpr (STABLE) enc *= slope[jj];
                ds[jj] = __uint_as_float(pd[k]) + ((STABLE && eb == 0.f) ? 0.f : enc);
              }
              // dS = hi + lo, two bf16 values: the dK / dQ products then see it with 16 mantissa bits
              uint32_t hi[4], lo[4];
#pragma unroll
              for (int jj = 0; jj < 8; jj += 2) {
                hi[jj >> 1] = pack_bf16(ds[jj], ds[jj + 1]);
                lo[jj >> 1] = pack_bf16(ds[jj] - bf16_lo(hi[jj >> 1]), ds[jj + 1] - bf16_hi(hi[jj >> 1]));
              }
              constexpr int COPY = PACK ? 8192 : 0;
              *reinterpret_cast<uint4*>(e_row + COPY + swz_chunk_off(m, ch0 + ch)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
              *reinterpret_cast<uint4*>(r_row + COPY + swz_chunk_off(m, ch0 + ch)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
          }
          fence_proxy_async_smem();
        }
        if (tid == 0) BT_TRACE(3, j, 5);
        tc_fence_before_sync();
        warp_arrive(&misc->x_done, lane);
        if (tid == 0) BT_TRACE(0, j, 4);
        // carries into the previous chunk's frame
        const float phi = STABLE ? 1.0f : ex2_approx(c_prev - c_i);
        cc_carry = (cc_carry + rp_all) * phi;
        if (!(fabsf(cc_carry) < INFINITY)) {
          // an overflow or 0 / 0 upstream (score spreads beyond what these frames hold) has reached the carries: the
          // results of this call are invalid; the exact kernels standing by behind this pass redo it
          atomicOr(p.err, 2);
          if (p.gate != nullptr) p.gate[0] = 1;
        }
        if (p.emit_only && i == begin && tp == 0 && live)
          p.xc[((int64_t)lane_id * p.nseg + seg) * p.M + mg] = cc_carry;
        if (i > begin || p.emit_only) {
          // G has taken this chunk's R dY: rescale this warp's value columns in tensor memory and pack them as bf16.
          // The shared-memory copy is still read by this chunk's dV product, so the packed rows wait in registers
          // until that product has run.
          if (!(ok = wait_or_abort(&misc->g_ready, par, misc))) break;
          tc_fence_after_sync();
          if (tid == 0) BT_TRACE(0, j, 5);
          const bool need = __any_sync(0xffffffffu, phi != 1.0f);
          uint4 gv[GCOLS / 8];
          uint32_t r[GCOLS];
          tmem_read(tl + TG + gcol, r);
          if (need) {
#pragma unroll
            for (int k = 0; k < GCOLS; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) * phi);
            tmem_write(tl + TG + gcol, r);
          }
          if (i == begin) emit_g(r);
#pragma unroll
          for (int ch = 0; ch < GCOLS / 8; ++ch)
            gv[ch] = make_uint4(pack_bf16(__uint_as_float(r[ch * 8 + 0]), __uint_as_float(r[ch * 8 + 1])),
                                pack_bf16(__uint_as_float(r[ch * 8 + 2]), __uint_as_float(r[ch * 8 + 3])),
                                pack_bf16(__uint_as_float(r[ch * 8 + 4]), __uint_as_float(r[ch * 8 + 5])),
                                pack_bf16(__uint_as_float(r[ch * 8 + 6]), __uint_as_float(r[ch * 8 + 7])));
          if (need) tmem_wait_st();
          if (tid == 0) BT_TRACE(3, j, 6);
          if (!(ok = wait_or_abort(&misc->dv_ready, par, misc))) break;
          if (i == begin) break;
          if (tid == 0) BT_TRACE(0, j, 6);
#pragma unroll
          for (int ch = 0; ch < GCOLS / 8; ++ch) put(g_dst, gch0 + ch, gv[ch]);
          fence_proxy_async_smem();
          tc_fence_before_sync();
          warp_arrive(&misc->gc_done, lane);
          if (tid == 0) BT_TRACE(0, j, 7);
        }
        c_cur = c_prev;
        d_cur = d_pre;
        c_nxt = c_pre;
        l2_cur = l2_pre;
        dl_cur = dl_pre;
      }
    }  // working warp
  } else {
    // ============================ token group: thread = token of the chunk = TMEM lane ============================
    const int wq = warp - W_TOKEN;
    const uint32_t tl = tmem + ((uint32_t)(wq * 32) << 16);
    const int tt = wq * 32 + lane;
    const int lo = BLOCK ? (tt & ~(p.block - 1)) : tt;  // first column (token) this row keeps
    uint8_t* const dv_stage = smem + L::OFF_DVT + wq * L::DV_TILES;  // this warp's tiles of the dV rows
    for (int j = 0; ok && j < steps; ++j) {
      const int i = first - 1 - j, t0 = i * C;
      const uint32_t par = j & 1, fpar = (j - (first - full_end)) & 1;
      // masked A (bf16) into the K tile's buffer
      if (!(ok = wait_or_abort(&misc->a_ready, par, misc))) break;
      tc_fence_after_sync();
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 0);
#pragma unroll 1
      for (int jb = 0; jb < 4; ++jb) {
        uint32_t wp[16];
        if (jb * 32 + 31 >= lo) {
          uint32_t r[32];
          tmem_ld32(tl + T0 + jb * 32, r);
          tmem_wait_ld();
          tmem_fence_regs(r);
          if (jb * 32 >= lo) {
#pragma unroll
            for (int k = 0; k < 32; k += 2) wp[k >> 1] = pack_bf16(__uint_as_float(r[k]), __uint_as_float(r[k + 1]));
          } else {
#pragma unroll
            for (int k = 0; k < 32; k += 2)
              wp[k >> 1] = pack_bf16(jb * 32 + k >= lo ? __uint_as_float(r[k]) : 0.f,
                                     jb * 32 + k + 1 >= lo ? __uint_as_float(r[k + 1]) : 0.f);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) wp[k] = 0u;
        }
        uint8_t* blk = smem + L::OFF_KA + (jb >> 1) * 16384;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(blk + swz_chunk_off(tt, (jb & 1) * 4 + ch)) =
              make_uint4(wp[ch * 4], wp[ch * 4 + 1], wp[ch * 4 + 2], wp[ch * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      warp_arrive(&misc->am_done, lane);
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 1);
      if (i >= full_end) {  // carries only: T0 holds nothing of this group's
        warp_arrive(&misc->dv_free, lane);
        continue;
      }
      // masked E^T R (bf16) into tensor memory
      if (!(ok = wait_or_abort(&misc->wt_ready, fpar, misc))) break;
      tc_fence_after_sync();
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 2);
#pragma unroll 1
      for (int jb = 0; jb < 4; ++jb) {
        uint32_t wp[16];
        if (jb * 32 + 31 >= lo) {
          uint32_t r[32];
          tmem_ld32(tl + T0 + jb * 32, r);
          tmem_wait_ld();
          tmem_fence_regs(r);
          if (jb * 32 >= lo) {
#pragma unroll
            for (int k = 0; k < 32; k += 2) wp[k >> 1] = pack_bf16(__uint_as_float(r[k]), __uint_as_float(r[k + 1]));
          } else {
#pragma unroll
            for (int k = 0; k < 32; k += 2)
              wp[k >> 1] = pack_bf16(jb * 32 + k >= lo ? __uint_as_float(r[k]) : 0.f,
                                     jb * 32 + k + 1 >= lo ? __uint_as_float(r[k + 1]) : 0.f);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) wp[k] = 0u;
        }
        tmem_st16(tl + T2 + jb * 16, wp);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      warp_arrive(&misc->wm_done, lane);
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 3);
      // dV rows
      if (!(ok = wait_or_abort(&misc->dv_ready, par, misc))) break;
      tc_fence_after_sync();
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 4);
#pragma unroll
      for (int half = 0; half < DV / 32; ++half) {
        uint32_t r[32];
        tmem_ld32(tl + T0 + half * 32, r);
        tmem_wait_ld();
        tmem_fence_regs(r);
        if (half == DV / 32 - 1) {
          tc_fence_before_sync();
          warp_arrive(&misc->dv_free, lane);
        }
        uint4 v[4];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          v[ch] = make_uint4(pack_bf16(__uint_as_float(r[ch * 8 + 0]), __uint_as_float(r[ch * 8 + 1])),
                             pack_bf16(__uint_as_float(r[ch * 8 + 2]), __uint_as_float(r[ch * 8 + 3])),
                             pack_bf16(__uint_as_float(r[ch * 8 + 4]), __uint_as_float(r[ch * 8 + 5])),
                             pack_bf16(__uint_as_float(r[ch * 8 + 6]), __uint_as_float(r[ch * 8 + 7])));
        // a 32 x 32 tile (64-byte swizzle)
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(dv_stage + half * 2048 + lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4)) = v[ch];
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int half = 0; half < DV / 32; ++half)  // (rows beyond the sequence end are clipped)
          tma_store_4d(&tm_dv, dv_stage + half * 2048, half * 32, h, t0 + wq * 32, group * (int)(gridDim.x / p.H) + b);
        bulk_commit_group();
        bulk_wait_group_read0();
      }
      if constexpr (DVB == 2) warp_arrive(&misc->dv_out, lane);
      else __syncwarp();
      if (tid == W_TOKEN * 32) BT_TRACE(1, j, 5);
    }
    if (lane == 0) bulk_wait_group0();
  }
  if (!ok) {
    misc->abort_flag = 1;
    atomicOr(p.err, 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == W_MMA) tmem_dealloc(tmem, TM_COLS);
}

namespace {

template <int DKB, int DVB, int MODE, bool PACK>
int launch_main(const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdy, const CUtensorMap& tu,
                const CUtensorMap& tds, const CUtensorMap& tdv, const BwdTcParams& p, dim3 grid, cudaStream_t stream) {
  auto kern = bwd_tc_kernel<DKB, DVB, MODE, PACK>;
  FLARE_CUDA_CHECK(allow_smem(kern));
  LaunchTimer timer("bwd_tc_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(kern, grid, dim3(NT_MAIN), BL<DVB>::SMEM_BYTES, stream, tk, tv, tdy, tu, tds, tdv, p));
  return FLARE_OK;
}

}  // namespace

template <>
int launch_bwd_tc_unit<FLARE_BT_UNIT>(int mode, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdy,
                                      const CUtensorMap& tu, const CUtensorMap& tds, const CUtensorMap& tdv, const BwdTcParams& p,
                                      dim3 grid, cudaStream_t stream) {
  // units 0..2: (Dk, Dv) = (64, 64), (128, 128), (64, 128); units 3..5: the same, packed
  constexpr int W = FLARE_BT_UNIT % 3;
  constexpr int DKB = W == 1 ? 2 : 1;
  constexpr int DVB = W == 0 ? 1 : 2;
  constexpr bool PACK = FLARE_BT_UNIT >= 3;
  if (mode == 1) return launch_main<DKB, DVB, 1, PACK>(tk, tv, tdy, tu, tds, tdv, p, grid, stream);
  if (mode == 2) return launch_main<DKB, DVB, 2, PACK>(tk, tv, tdy, tu, tds, tdv, p, grid, stream);
  return launch_main<DKB, DVB, 0, PACK>(tk, tv, tdy, tu, tds, tdv, p, grid, stream);
}

#else  // host side, the dK / dQ kernel and the small helper kernels

#define FLARE_BT_DECLARE(U)                                                                                                    \
  template <>                                                                                                               \
  int launch_bwd_tc_unit<U>(int, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, \
                            const CUtensorMap&, const BwdTcParams&, dim3, cudaStream_t);
FLARE_BT_DECLARE(0)
FLARE_BT_DECLARE(1)
FLARE_BT_DECLARE(2)
FLARE_BT_DECLARE(3)
FLARE_BT_DECLARE(4)
FLARE_BT_DECLARE(5)
#undef FLARE_BT_DECLARE

namespace {

// -------------------------------------------------------------------------------------------------
// per-token statistics: delta_t = <dY_t, y_t> and the decode log-sum-exp in log2 units, rows padded to whole chunks
// (delta = 0, log-sum-exp = +inf there, which makes every decode weight of a padding token exactly zero)
// -------------------------------------------------------------------------------------------------
// One block per (8 tokens, batch row), 16 heads at a time: dY and y of a token lie head by head behind one another, so a block
// streams them in long runs with two pieces of each in flight per thread, eight blocks to an SM; its results, which lie token by
// token, go through shared memory into rows of 8.  B=4 N=4096 H=16 D=128, 134 MB to read, us with the launch: 31; 35 with 16
// tokens and four pieces (its grid is 1.7 waves), 33 with 4 tokens or one piece, 41 with 16 tokens and eight pieces, 41 with one
// piece and results scattered as they come.
constexpr int ST_TOK = 8, ST_HEADS = 16, ST_LOADS = 2;
__global__ void __launch_bounds__(256, 8) bwd_tc_token_stats_kernel(const __nv_bfloat16* dy, int64_t dy_sb,
                                                                  int64_t dy_sn, int64_t dy_sh,
                                                                  const __nv_bfloat16* y, int64_t y_sb,
                                                                  int64_t y_sn, int64_t y_sh, const float* lse,
                                                                  int B, int N, int H, int Dv, int npad, float* tok_l2,
                                                                  float* tok_delta, const int* fwd_gate,
                                                                  int fwd_gate_words, int* gate, int* sync) {
  pdl_begin();
  __shared__ float delta_s[ST_HEADS][ST_TOK + 1];
  if (blockIdx.x == 0) {
    // this call's gate word starts as "did any CTA of the forward find its tokens outside the numeric domain" (the forward's
    // leading word says how many words per lane it wrote; after a replay it is the word written here)
    const int words = min(B * H * fwd_gate[0], fwd_gate_words - 1);
    int raised = 0;
    for (int i = threadIdx.x; i < words; i += 256) raised |= fwd_gate[1 + i];
    raised = __syncthreads_or(raised);
    if (threadIdx.x == 0) *gate = raised ? 1 : 0;
    if (threadIdx.x < kBwdSyncWords) sync[threadIdx.x] = 0;
  }
  // Dv / 8 threads per (token, head) row (8 or 16, a divisor of the warp size), one 16-byte piece of dY and of y each
  const int tpr = Dv >> 3, rows_per_pass = 256 / tpr;
  const int sub = threadIdx.x % tpr, row0 = threadIdx.x / tpr;
  const int tiles = npad / ST_TOK, b = blockIdx.x / tiles, n0 = (blockIdx.x - b * tiles) * ST_TOK;
  const __nv_bfloat16* const dy_b = dy + b * dy_sb + sub * 8;
  const __nv_bfloat16* const y_b = y + b * y_sb + sub * 8;
  for (int h0 = 0; h0 < H; h0 += ST_HEADS) {
    const int heads = min(ST_HEADS, H - h0);
    for (int r0 = row0; r0 < ST_TOK * heads; r0 += ST_LOADS * rows_per_pass) {  // (the same for all rows of a warp)
      uint4 a[ST_LOADS], c[ST_LOADS];
#pragma unroll
      for (int u = 0; u < ST_LOADS; ++u) {
        const int r = r0 + u * rows_per_pass, t = r / heads, h = h0 + (r - t * heads), n = n0 + t;
        const bool on = t < ST_TOK && n < N;
        a[u] = on ? *reinterpret_cast<const uint4*>(dy_b + (int64_t)n * dy_sn + h * dy_sh) : make_uint4(0, 0, 0, 0);
        c[u] = on ? *reinterpret_cast<const uint4*>(y_b + (int64_t)n * y_sn + h * y_sh) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < ST_LOADS; ++u) {
        float acc = (bf16_lo(a[u].x) * bf16_lo(c[u].x) + bf16_hi(a[u].x) * bf16_hi(c[u].x)) +
                    (bf16_lo(a[u].y) * bf16_lo(c[u].y) + bf16_hi(a[u].y) * bf16_hi(c[u].y)) +
                    (bf16_lo(a[u].z) * bf16_lo(c[u].z) + bf16_hi(a[u].z) * bf16_hi(c[u].z)) +
                    (bf16_lo(a[u].w) * bf16_lo(c[u].w) + bf16_hi(a[u].w) * bf16_hi(c[u].w));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
          if (o < tpr) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const int r = r0 + u * rows_per_pass, t = r / heads;
        if (sub == 0 && t < ST_TOK) delta_s[r - t * heads][t] = acc;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < heads * ST_TOK; i += 256) {
      const int h = i / ST_TOK, t = i % ST_TOK, n = n0 + t;
      const int64_t lane = (int64_t)b * H + h0 + h;
      tok_delta[lane * npad + n] = n < N ? delta_s[h][t] : 0.f;
      tok_l2[lane * npad + n] = n < N ? lse[lane * N + n] * kLog2e : INFINITY;
    }
    __syncthreads();
  }
}

// sum of the latent groups' dV partials (bf16) in fp32
__global__ void __launch_bounds__(256) bwd_tc_sum_groups_kernel(const __nv_bfloat16* part, int groups, int64_t n8,
                                                                 __nv_bfloat16* out) {
  pdl_begin();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n8) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int g = 0; g < groups; ++g) {
    const uint4 v = load_streaming(reinterpret_cast<const uint4*>(part + (int64_t)g * n8 * 8) + idx);
    acc[0] += bf16_lo(v.x); acc[1] += bf16_hi(v.x); acc[2] += bf16_lo(v.y); acc[3] += bf16_hi(v.y);
    acc[4] += bf16_lo(v.z); acc[5] += bf16_hi(v.z); acc[6] += bf16_lo(v.w); acc[7] += bf16_hi(v.w);
  }
  reinterpret_cast<uint4*>(out)[idx] = make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]),
                                                  pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
}

// dq[i] = sum over the (batch, split) partials in fixed order
__global__ void __launch_bounds__(256) bwd_tc_sum_dq_kernel(const float* part, int count, int64_t n4, void* out,
                                                             int out_dtype) {
  pdl_begin();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n4) return;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < count; s0 += 8) {  // eight loads in flight: few threads, latency is all there is
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = s0 + u < count ? load_streaming(reinterpret_cast<const float4*>(part + (int64_t)(s0 + u) * n4 * 4) + idx)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
    }
  }
  store4(out, out_dtype, idx * 4, acc.x, acc.y, acc.z, acc.w);
}

// -------------------------------------------------------------------------------------------------
// dK = scale dS^T Q per chunk, dQ = scale sum_t dS K per (lane, split of the chunks).
// One CTA per (lane, split), 6 warps: 0 TMA producer, 1 MMA issuer, 2-5 epilogue (thread = TMEM lane).
// -------------------------------------------------------------------------------------------------
constexpr int NT_GRAD = 192;

constexpr int GRAD_MAXST = 8;  // stages of a ring

// Shared memory: rings of nds dS planes ([2 t-blocks][rows m][64 t], rows = 64 for banks of at most 64 latents, else 128) and of nk K
// tiles ([DKB][128 t][64]), the latent bank (groups x [DKB][128 m][64]), two 32 x 32 tiles of dK rows per epilogue warp.  A streaming
// kernel: as many stages as fit, about two planes for a K tile.  B=4 N=4096 H=16 M=64 D=128 (200 MB, 31 us at the copy rate): 33 us; 45
// with two stages of each, planes of 128 rows whatever the bank, and dK rows stored by their threads in 16-byte pieces.
struct GradRings {
  int plane, nds, nk, smem;
};
GradRings grad_rings(int M, int dkb) {
  const int groups = (M + 127) / 128, tile = dkb * 16384, fixed = groups * tile + 16384 + 512 + 1024;
  GradRings r;
  r.plane = M <= 64 ? 16384 : 32768;
  for (r.nk = 4;; --r.nk) {
    r.nds = (232448 - fixed - r.nk * tile) / r.plane;
    if (r.nk == 2 || r.nds >= 2 * r.nk - 1) break;
  }
  if (r.nds > GRAD_MAXST) r.nds = GRAD_MAXST;
  r.smem = fixed + r.nk * tile + r.nds * r.plane;
  return r;
}

struct GradMisc {
  uint64_t q_full, ds_full[GRAD_MAXST], ds_empty[GRAD_MAXST], k_full[4], k_empty[4], dk_ready[2], dk_free[2], dq_ready;
  uint32_t tmem_base;
  volatile int abort_flag;
};
static_assert(sizeof(GradMisc) <= 512, "GradMisc");
// the next stage of a ring, and the parity of its phase
struct Stage {
  int s = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next(int n) {
    if (++s == n) s = 0, phase ^= 1;
  }
};

template <int DKB>
__global__ void __launch_bounds__(NT_GRAD, 1)
bwd_tc_grads_kernel(const __grid_constant__ CUtensorMap tm_ds, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_dk, const GradTcParams p) {
  constexpr int DK = DKB * 64;
  constexpr uint32_t TM_DK = 0, TM_DQ = 2 * DK;  // tensor-memory columns: two buffers of dK, then dQ of every group
  pdl_wait();
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int G = p.groups, plane = p.plane, nds = p.nds, nk = p.nk;
  uint8_t* const k_ring = smem + nds * plane;
  uint8_t* const q_bank = k_ring + nk * DKB * 16384;
  uint8_t* const stage = q_bank + G * DKB * 16384;
  GradMisc* misc = reinterpret_cast<GradMisc*>(stage + 16384);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lane_id = blockIdx.x, split = blockIdx.y;
  const int b = lane_id / p.H, h = lane_id % p.H;
  const int c_begin = split * p.chunks_per_split, c_end = min(p.nch, c_begin + p.chunks_per_split);
  const int ncs = max(0, c_end - c_begin);
  const uint32_t tm_cols = (2 + G) * DK <= 256 ? 256u : 512u;

  if (tid == 0) {
    mbar_init(&misc->q_full, 1);
    for (int i = 0; i < GRAD_MAXST; ++i) {
      mbar_init(&misc->ds_full[i], 1);
      mbar_init(&misc->ds_empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&misc->k_full[i], 1);
      mbar_init(&misc->k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&misc->dk_ready[i], 1);
      mbar_init(&misc->dk_free[i], 4);
    }
    mbar_init(&misc->dq_ready, 1);
    misc->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&misc->tmem_base, tm_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = misc->tmem_base;
  bool ok = true;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return tc::wait_or_abort(bar, parity, &misc->abort_flag, 1); };

  if (warp == 0) {
    if (elect_one()) {
      prefetch_tensormap(&tm_ds);
      prefetch_tensormap(&tm_k);
      mbar_arrive_expect_tx(&misc->q_full, G * DKB * 16384);
      for (int g = 0; g < G; ++g)
        for (int kb = 0; kb < DKB; ++kb)
          tma_load_3d(q_bank + (g * DKB + kb) * 16384, &tm_q, &misc->q_full, kb * 64, g * 128, h);
      Stage ks, ds;  // (a fresh ring's stages are empty: the phase before the first one counts as complete)
      for (int cc = 0; ok && cc < ncs; ++cc, ks.next(nk)) {
        const int t0 = (c_begin + cc) * C;
        if (!(ok = wait(&misc->k_empty[ks.s], ks.phase ^ 1))) break;
        mbar_arrive_expect_tx(&misc->k_full[ks.s], DKB * 16384);
        for (int kb = 0; kb < DKB; ++kb)
          tma_load_4d(k_ring + (ks.s * DKB + kb) * 16384, &tm_k, &misc->k_full[ks.s], kb * 64, h, t0, b);
        for (int gp = 0; ok && gp < 2 * G; ++gp, ds.next(nds)) {  // (group, hi | lo plane)
          const int g = gp >> 1, part = gp & 1;
          if (!(ok = wait(&misc->ds_empty[ds.s], ds.phase ^ 1))) break;
          mbar_arrive_expect_tx(&misc->ds_full[ds.s], plane);
          for (int tb = 0; tb < 2; ++tb)  // (rows beyond M read as zero)
            tma_load_4d(smem + ds.s * plane + tb * (plane >> 1), &tm_ds, &misc->ds_full[ds.s], t0 + tb * 64, g * 128, part, lane_id);
        }
      }
      pdl_trigger();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t ID_DK = make_idesc_bf16(128, DK, 1, 1);  // dS (MN-major: tokens contiguous) x Q (MN-major)
      constexpr uint32_t ID_DQ = make_idesc_bf16(128, DK, 0, 1);  // dS (K-major: rows = latents) x K tile (MN-major)
      ok = wait(&misc->q_full, 0);
      Stage ks, ds;
      for (int cc = 0; ok && cc < ncs; ++cc, ks.next(nk)) {
        const int kb = cc & 1;
        if (!(ok = wait(&misc->k_full[ks.s], ks.phase))) break;
        if (cc >= 2 && !(ok = wait(&misc->dk_free[kb], ((cc - 2) >> 1) & 1))) break;
        tc_fence_after_sync();
        const uint64_t d_k_mn = make_desc_sw128(smem_u32(k_ring + ks.s * DKB * 16384), 16384, 1024);
        for (int gp = 0; ok && gp < 2 * G; ++gp, ds.next(nds)) {  // (group, hi | lo plane): lo accumulates on top of hi
          const int g = gp >> 1;
          if (!(ok = wait(&misc->ds_full[ds.s], ds.phase))) break;
          tc_fence_after_sync();
          const uint32_t ds_addr = smem_u32(smem + ds.s * plane);
          const uint64_t d_ds_mn = make_desc_sw128(ds_addr, plane >> 1, 1024), d_ds_k = make_desc_sw128(ds_addr, 16, 1024);
          const uint64_t d_q_mn = make_desc_sw128(smem_u32(q_bank + g * DKB * 16384), 16384, 1024);
          const int rows = min(128, p.M - g * 128);
          const int ksm = (rows + 15) >> 4;
          for (int st = 0; st < ksm; ++st)  // contraction over the latents of the group
            mma_ss(tmem + TM_DK + kb * DK, mnmaj_step(d_ds_mn, st), mnmaj_step(d_q_mn, st), ID_DK, (gp > 0 || st > 0) ? 1u : 0u);
          // contraction over the tokens of the chunk.  (Planes of 64 rows: the product's upper 64 rows come from whatever lies behind
          // the block; they belong to no latent and are not read.)
#pragma unroll
          for (int st = 0; st < 8; ++st)
            mma_ss(tmem + TM_DQ + g * DK, d_ds_k + (uint64_t)(((st >> 2) * (plane >> 1) + (st & 3) * 32) >> 4), mnmaj_step(d_k_mn, st),
                   ID_DQ, (cc > 0 || (gp & 1) || st > 0) ? 1u : 0u);
          tc_commit(&misc->ds_empty[ds.s]);
        }
        if (!ok) break;
        tc_commit(&misc->dk_ready[kb]);
        tc_commit(&misc->k_empty[ks.s]);
      }
      if (ok) tc_commit(&misc->dq_ready);
    }
  } else {
    const int wq = warp & 3;  // TMEM lane quarter of this warp
    const uint32_t tl = tmem + ((uint32_t)(wq * 32) << 16);
    const int tt = wq * 32 + lane;
    for (int cc = 0; ok && cc < ncs; ++cc) {
      const int kb = cc & 1;
      if (!(ok = wait(&misc->dk_ready[kb], (cc >> 1) & 1))) break;
      tc_fence_after_sync();
#pragma unroll
      for (int half = 0; half < DK / 32; ++half) {
        uint32_t r[32];
        tmem_ld32(tl + TM_DK + kb * DK + half * 32, r);
        tmem_wait_ld();
        tmem_fence_regs(r);
        if (half == DK / 32 - 1) {
          tc_fence_before_sync();
          warp_arrive(&misc->dk_free[kb], lane);
        }
        // two 32 x 32 tiles (64-byte swizzle), stored in turn; rows beyond the sequence end are clipped
        uint8_t* const tile = stage + wq * 4096 + (half & 1) * 2048;
        if (lane == 0) bulk_wait_group_read1();
        __syncwarp();
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(r[ch * 8 + 0]) * p.scale, __uint_as_float(r[ch * 8 + 1]) * p.scale);
          v.y = pack_bf16(__uint_as_float(r[ch * 8 + 2]) * p.scale, __uint_as_float(r[ch * 8 + 3]) * p.scale);
          v.z = pack_bf16(__uint_as_float(r[ch * 8 + 4]) * p.scale, __uint_as_float(r[ch * 8 + 5]) * p.scale);
          v.w = pack_bf16(__uint_as_float(r[ch * 8 + 6]) * p.scale, __uint_as_float(r[ch * 8 + 7]) * p.scale);
          *reinterpret_cast<uint4*>(tile + lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4)) = v;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_4d(&tm_dk, tile, half * 32, h, (c_begin + cc) * C + wq * 32, b);
          bulk_commit_group();
        }
      }
    }
    if (lane == 0) bulk_wait_group0();
    // this split's part of dQ
    float* part = p.dq_part + (((int64_t)(b * p.nsplit + split) * p.H + h) * p.M) * DK;
    if (ncs > 0) ok = ok && wait(&misc->dq_ready, 0);
    tc_fence_after_sync();
    for (int g = 0; g < G; ++g) {
      const int mg = g * 128 + tt;
#pragma unroll
      for (int half = 0; half < DK / 32; ++half) {
        uint32_t r[32];
        if (ncs > 0 && ok) {
          tmem_ld32(tl + TM_DQ + g * DK + half * 32, r);
          tmem_wait_ld();
          tmem_fence_regs(r);
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) r[k] = 0u;
        }
        if (mg < p.M) {
          float4* dst = reinterpret_cast<float4*>(part + (int64_t)mg * DK + half * 32);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            dst[k] = make_float4(__uint_as_float(r[4 * k]) * p.scale, __uint_as_float(r[4 * k + 1]) * p.scale,
                                 __uint_as_float(r[4 * k + 2]) * p.scale, __uint_as_float(r[4 * k + 3]) * p.scale);
        }
      }
    }
  }
  if (!ok) {
    misc->abort_flag = 1;
    atomicOr(p.err, 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, tm_cols);
}

template <int DKB>
int launch_grads(const CUtensorMap& tds, const CUtensorMap& tk, const CUtensorMap& tq, const CUtensorMap& tdk, GradTcParams p,
                 dim3 grid, cudaStream_t stream) {
  auto kern = bwd_tc_grads_kernel<DKB>;
  const GradRings r = grad_rings(p.M, DKB);
  p.plane = r.plane; p.nds = r.nds; p.nk = r.nk;
  FLARE_CUDA_CHECK(allow_smem(kern));
  LaunchTimer timer("bwd_tc_grads_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(kern, grid, dim3(NT_GRAD), r.smem, stream, tds, tk, tq, tdk, p));
  return FLARE_OK;
}

// -------------------------------------------------------------------------------------------------
// host: plan, workspace, launch sequence
// -------------------------------------------------------------------------------------------------
bool have_saved(const flare_bwd_args_t& a);  // defined below, with the keep-buffer layout

// Sequence segments of the reverse sweep, one CTA each per (lane, latent group).  A carry-only chunk (scores, E, R, A, P
// and G, but no X, dV, dS) takes kCarryCost of a full one.
//  * lead: the CTA of a segment first walks every later chunk carry-only.  Later segments are longer so that all CTAs take
//    equally long; no second launch, no exchange, bit-identical results.  Good for two or three CTAs per lane.
//  * exchange: equal segments; a first launch takes the carries of every segment but the first, the second starts from
//    their sum.  Good when many SMs are idle.
// Every alternative is estimated in chunks of the longest SM (CTAs per SM x chunks per CTA) and the least one is taken;
// kExchangeCost stands for the second launch and the carries' way through L2.
struct SegmentPlan {
  int n;
  bool lead;
  int begin[kMaxBwdSegments + 1];
};
// B200: B=4 N=4096 H=16 M=64 D=128 (64 lanes, 2 lead segments) 583 -> 504 us a training step, stablemax B=2 N=1000 H=8
// M=64 D=64 (16 lanes, 8 segments with an exchange) 170 -> 112 us.
constexpr double kCarryCost = 0.55, kExchangeCost = 0.6;

SegmentPlan plan_segments(int64_t ctas, int nch) {
  SegmentPlan pl;
  pl.n = 1;
  pl.lead = false;
  pl.begin[0] = 0;
  pl.begin[1] = nch;
  const int64_t sms = sm_count();
  auto waves = [&](int64_t n) { return (double)((n + sms - 1) / sms); };
  double best = waves(ctas) * nch * 0.97;  // (a split has to gain more than the estimate's error)
  for (int s = 2; s <= kMaxBwdSegments && s <= nch; ++s) {
    if (ctas * s <= sms) {
      double q = 1.0;
      for (int k = 0; k < s; ++k) q *= 1.0 - kCarryCost;
      const double t = nch * kCarryCost / (1.0 - q);
      SegmentPlan c;
      c.n = s;
      c.lead = true;
      c.begin[s] = nch;
      double worst = 0.0;
      bool fits = true;
      for (int k = s - 1; k >= 0; --k) {
        const int later = nch - c.begin[k + 1];
        int len = k == 0 ? c.begin[1] : (int)(t - kCarryCost * later + 0.5);
        if (len < 1) len = 1;
        if (len > c.begin[k + 1] - k) fits = false;
        c.begin[k] = c.begin[k + 1] - len;
        const double cost = len + kCarryCost * later;
        if (cost > worst) worst = cost;
      }
      if (fits && worst < best) {
        best = worst;
        pl = c;
      }
    }
    const int len = (nch + s - 1) / s;
    if ((nch + len - 1) / len != s) continue;  // the same as a smaller number of segments
    const double cost = len * (waves(ctas * s) + kCarryCost * waves(ctas * (s - 1))) + kExchangeCost;
    if (cost < best) {
      best = cost;
      pl.n = s;
      pl.lead = false;
      for (int k = 0; k <= s; ++k) pl.begin[k] = k * len < nch ? k * len : nch;
    }
  }
  return pl;
}

struct TcBwdPlan {
  int nch, npad, groups, nsplit, chunks_per_split;
  size_t gate_words, gate_bytes;  // the call's gate word and those of the forward's replay come first
  size_t exact_bytes;  // path AUTO: scratch of the exact pass standing by (shares the space behind the gate words)
  size_t fwd_ws;  // then the forward's own scratch
  SegmentPlan seg;
  size_t off_xg, off_xc;  // carries that the segments exchange
  size_t off_y, off_lse, off_l2, off_delta, off_cu, off_cc, off_cd, off_ds, off_dqp, off_dvp, total;
};

TcBwdPlan plan_tc(const flare_bwd_args_t& a) {
  const flare_fwd_args_t& f = a.fwd;
  TcBwdPlan pl;
  memset(&pl, 0, sizeof(pl));
  pl.nch = (f.N + C - 1) / C;
  pl.npad = pl.nch * C;
  pl.groups = (f.M + 127) / 128;
  const int64_t lanes = (int64_t)f.B * f.H;
  pl.seg = plan_segments(lanes * pl.groups, pl.nch);
  int nsplit = (int)(sm_count() / (lanes > 0 ? lanes : 1));
  if (nsplit < 1) nsplit = 1;
  if (nsplit > pl.nch) nsplit = pl.nch;
  pl.chunks_per_split = (pl.nch + nsplit - 1) / nsplit;
  pl.nsplit = (pl.nch + pl.chunks_per_split - 1) / pl.chunks_per_split;
  flare_fwd_args_t probe = f;
  probe.y = const_cast<void*>(a.dy);  // any non-null pointer: "an output is wanted"
  probe.y_stride_b = a.dy_stride_b; probe.y_stride_n = a.dy_stride_n; probe.y_stride_h = a.dy_stride_h;
  probe.mask = nullptr; probe.lengths = nullptr;
  probe.lse_dec = nullptr; probe.lse_enc = nullptr;
  memset(&probe.state_in, 0, sizeof(probe.state_in));
  memset(&probe.state_out, 0, sizeof(probe.state_out));
  probe.path = FLARE_PATH_TENSOR;
  probe.keep = nullptr; probe.keep_bytes = 0;
  const bool saved = have_saved(a);
  pl.fwd_ws = saved ? 0 : align_up(flare_forward_workspace_bytes(&probe), 256);
  pl.gate_words = saved ? 1 : forward_gate_words(&probe);
  // (and the counters of the pass standing by, 256 bytes that the token statistics zero)
  pl.gate_bytes = align_up(pl.gate_words * sizeof(int), 256) + 256;
  size_t off = pl.gate_bytes + pl.fwd_ws;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += align_up(bytes, 256);
    return o;
  };
  pl.off_y = saved ? 0 : take((size_t)f.B * f.N * f.H * f.Dv * 2);
  pl.off_lse = saved ? 0 : take((size_t)lanes * f.N * 4);
  pl.off_l2 = take((size_t)lanes * pl.npad * 4);
  pl.off_delta = take((size_t)lanes * pl.npad * 4);
  pl.off_cu = saved ? 0 : take((size_t)lanes * pl.nch * f.M * f.Dv * 2);
  pl.off_cc = saved ? 0 : take((size_t)lanes * pl.nch * f.M * 4);
  pl.off_cd = saved ? 0 : take((size_t)lanes * pl.nch * f.M * 4);
  pl.off_ds = take((size_t)2 * lanes * f.M * pl.npad * 2);  // a hi and a lo row per latent
  pl.off_dqp = take((size_t)f.B * pl.nsplit * f.H * f.M * f.Dk * 4);
  pl.off_dvp = pl.groups > 1 ? take((size_t)pl.groups * f.B * f.N * f.H * f.Dv * 2) : 0;
  const size_t xrows = pl.seg.n > 1 && !pl.seg.lead ? (size_t)lanes * pl.seg.n * f.M : 0;
  pl.off_xg = xrows ? take(xrows * f.Dv * 4) : 0;
  pl.off_xc = xrows ? take(xrows * 4) : 0;
  pl.total = off;
  if (f.path == FLARE_PATH_AUTO) {
    flare_bwd_args_t ex = a;
    ex.fwd.path = FLARE_PATH_EXACT;
    pl.exact_bytes = bwd_exact_workspace_bytes(ex);
    if (pl.gate_bytes + pl.exact_bytes > pl.total) pl.total = pl.gate_bytes + pl.exact_bytes;
  }
  return pl;
}

}  // namespace

// the forward problems whose backward runs on the tensor kernels (everything but the gradient-side conditions)
static bool tc_trainable(const flare_fwd_args_t& f) {
  if (f.path == FLARE_PATH_EXACT || f.B <= 0 || f.N <= 0 || f.state_in.u != nullptr) return false;
  flare_fwd_args_t probe = f;
  if (probe.y == nullptr) probe.y = const_cast<void*>(f.k);  // any aligned non-null pointer: "an output is wanted"
  probe.mask = nullptr; probe.lengths = nullptr; probe.lse_dec = nullptr; probe.lse_enc = nullptr;
  memset(&probe.state_in, 0, sizeof(probe.state_in));
  memset(&probe.state_out, 0, sizeof(probe.state_out));
  probe.path = FLARE_PATH_TENSOR;
  if (f.mask != nullptr || f.lengths != nullptr || !prefill_tc_supported(&probe)) return false;
  const int groups = (f.M + 127) / 128;
  return (2 + groups) * f.Dk <= 512;  // tensor-memory columns of the dK / dQ kernel
}

KeepLayout keep_layout(const flare_fwd_args_t& f) {
  KeepLayout k;
  memset(&k, 0, sizeof(k));
  if (!tc_trainable(f)) return k;
  const size_t lanes = (size_t)f.B * f.H;
  k.nch = (f.N + C - 1) / C;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += align_up(bytes, 256);
    return o;
  };
  k.gate_words = forward_gate_words(&f);
  k.off_gate = take(k.gate_words * sizeof(int));
  k.off_u = take(lanes * k.nch * f.M * f.Dv * 2);
  k.off_c = take(lanes * k.nch * f.M * 4);
  k.off_d = take(lanes * k.nch * f.M * 4);
  k.total = off;
  return k;
}

// true when the caller handed over what a forward with `keep` left behind
namespace {
bool have_saved(const flare_bwd_args_t& a) {
  if (a.y == nullptr || a.lse_dec == nullptr || a.fwd.keep == nullptr) return false;
  const KeepLayout k = keep_layout(a.fwd);
  return k.total > 0 && a.fwd.keep_bytes >= k.total && (reinterpret_cast<uintptr_t>(a.fwd.keep) & 255u) == 0 &&
         (reinterpret_cast<uintptr_t>(a.y) & 15u) == 0 && (a.y_stride_b % 8) == 0 && (a.y_stride_n % 8) == 0 &&
         (a.y_stride_h % 8) == 0;
}
}  // namespace

bool bwd_tc_supported(const flare_bwd_args_t& a) {
  const flare_fwd_args_t& f = a.fwd;
  if (a.carry_b || a.carry_c || a.carry_rho || a.span_b0 || a.span_c0 || a.span_gam || a.span_rho_first || a.phase != 0)
    return false;  // spans of a longer sequence run on the exact kernels
  if (!tc_trainable(f)) return false;
  if ((reinterpret_cast<uintptr_t>(a.dy) & 15u) || (a.dy_stride_b % 8) || (a.dy_stride_n % 8) || (a.dy_stride_h % 8)) return false;
  return true;
}

size_t bwd_tc_workspace_bytes(const flare_bwd_args_t& a) { return plan_tc(a).total; }

int bwd_tc(const flare_bwd_args_t& a, cudaStream_t stream) {
  const flare_fwd_args_t& f = a.fwd;
  const TcBwdPlan pl = plan_tc(a);
  if (f.workspace == nullptr || f.workspace_bytes < pl.total || (reinterpret_cast<uintptr_t>(f.workspace) & 255u))
    return FLARE_ERR_WORKSPACE;
  char* ws = reinterpret_cast<char*>(f.workspace);
  const int64_t lanes = (int64_t)f.B * f.H;
  int* gate = reinterpret_cast<int*>(ws);
  int* sync = reinterpret_cast<int*>(ws + pl.gate_bytes - 256);
  const bool saved = have_saved(a);
  const int* fwd_gate;
  int fwd_gate_words;
  const void* y = nullptr;
  int64_t y_sb, y_sn, y_sh;
  const float* lse = nullptr;
  ChunkStates keep{nullptr, nullptr, nullptr, pl.nch};
  if (saved) {
    // (1') the training forward kept everything: its output, its log-sum-exp, the chunk states, its gate words
    const KeepLayout kl = keep_layout(f);
    char* kb = reinterpret_cast<char*>(f.keep);
    fwd_gate = reinterpret_cast<const int*>(kb + kl.off_gate);
    fwd_gate_words = (int)kl.gate_words;
    keep.u = kb + kl.off_u;
    keep.c = reinterpret_cast<float*>(kb + kl.off_c);
    keep.d = reinterpret_cast<float*>(kb + kl.off_d);
    y = a.y; y_sb = a.y_stride_b; y_sn = a.y_stride_n; y_sh = a.y_stride_h;
    lse = a.lse_dec;
  } else {
    // (1) forward on the tensor path: y, the decode log-sum-exp and the per-chunk prefix states
    fwd_gate = gate;
    fwd_gate_words = (int)pl.gate_words;
    keep.u = ws + pl.off_cu;
    keep.c = reinterpret_cast<float*>(ws + pl.off_cc);
    keep.d = reinterpret_cast<float*>(ws + pl.off_cd);
    flare_fwd_args_t fw = f;
    fw.y = ws + pl.off_y;
    fw.y_stride_b = (int64_t)f.N * f.H * f.Dv; fw.y_stride_n = (int64_t)f.H * f.Dv; fw.y_stride_h = f.Dv;
    fw.mask = nullptr; fw.lengths = nullptr;
    fw.lse_dec = reinterpret_cast<float*>(ws + pl.off_lse); fw.lse_enc = nullptr;
    fw.keep = nullptr; fw.keep_bytes = 0;
    memset(&fw.state_in, 0, sizeof(fw.state_in));
    memset(&fw.state_out, 0, sizeof(fw.state_out));
    fw.workspace = ws + pl.gate_bytes; fw.workspace_bytes = pl.fwd_ws;
    fw.path = FLARE_PATH_TENSOR;
    const int rc = forward_keep_states(&fw, keep, gate, stream);
    if (rc != FLARE_OK) return rc;
    y = fw.y; y_sb = fw.y_stride_b; y_sn = fw.y_stride_n; y_sh = fw.y_stride_h;
    lse = fw.lse_dec;
  }
  float* tok_l2 = reinterpret_cast<float*>(ws + pl.off_l2);
  float* tok_delta = reinterpret_cast<float*>(ws + pl.off_delta);
  // (2) per-token statistics
  {
    LaunchTimer timer("bwd_tc_token_stats_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(bwd_tc_token_stats_kernel, dim3((unsigned)(pl.npad / ST_TOK) * (unsigned)f.B), dim3(256), 0, stream,
                                reinterpret_cast<const __nv_bfloat16*>(a.dy), a.dy_stride_b, a.dy_stride_n, a.dy_stride_h,
                                reinterpret_cast<const __nv_bfloat16*>(y), y_sb, y_sn, y_sh, lse, f.B, f.N, f.H, f.Dv, pl.npad,
                                tok_l2, tok_delta, fwd_gate, fwd_gate_words, gate, sync));
    count_launches(1);
  }
  int* err = nullptr;
  {
    const int rc = tc_error_word(&err);
    if (rc != FLARE_OK) return rc;
  }
  // (3) reverse chunk sweep: dV and the dS plane
  const bool pack = f.M <= 64;
  CUtensorMap tk, tv, tdy, tu, tds, tdv, tdk, tq;
  {
    const uint64_t dimk[4] = {(uint64_t)f.Dk, (uint64_t)f.H, (uint64_t)f.N, (uint64_t)f.B};
    const uint64_t dimv[4] = {(uint64_t)f.Dv, (uint64_t)f.H, (uint64_t)f.N, (uint64_t)f.B};
    const uint32_t box[4] = {64, 1, 128, 1};
    const int64_t strk[3] = {f.k_stride_h, f.k_stride_n, f.k_stride_b};
    const int64_t strv[3] = {f.v_stride_h, f.v_stride_n, f.v_stride_b};
    const int64_t strd[3] = {a.dy_stride_h, a.dy_stride_n, a.dy_stride_b};
    const uint64_t dimu[4] = {(uint64_t)f.Dv, (uint64_t)f.M, (uint64_t)pl.nch, (uint64_t)lanes};
    const int64_t stru[3] = {f.Dv, (int64_t)f.M * f.Dv, (int64_t)pl.nch * f.M * f.Dv};
    const uint32_t boxu[4] = {64, pack ? 64u : 128u, 1, 1};
    const uint64_t dims[4] = {(uint64_t)pl.npad, (uint64_t)f.M, 2, (uint64_t)lanes};
    const int64_t strs[3] = {pl.npad, (int64_t)f.M * pl.npad, 2 * (int64_t)f.M * pl.npad};
    const uint32_t boxs[4] = {64, pack ? 64u : 128u, 1, 1};
    // dV rows, or with several latent groups their dense partials
    void* const dv = pl.groups > 1 ? static_cast<void*>(ws + pl.off_dvp) : a.dv;
    const uint64_t dimdv[4] = {(uint64_t)f.Dv, (uint64_t)f.H, (uint64_t)f.N, (uint64_t)f.B * pl.groups};
    const int64_t strdv[3] = {f.Dv, (int64_t)f.H * f.Dv, (int64_t)f.N * f.H * f.Dv};
    const int64_t strdk[3] = {f.Dk, (int64_t)f.H * f.Dk, (int64_t)f.N * f.H * f.Dk};
    const uint32_t boxdv[4] = {32, 1, 32, 1};
    const uint64_t dimq[3] = {(uint64_t)f.Dk, (uint64_t)f.M, (uint64_t)f.H};
    const int64_t strq[2] = {f.q_stride_m, f.q_stride_h};
    const uint32_t boxq[3] = {64, 128, 1};
    if (!tc::make_map_bf16(&tk, f.k, 4, dimk, strk, box) || !tc::make_map_bf16(&tv, f.v, 4, dimv, strv, box) ||
        !tc::make_map_bf16(&tdy, a.dy, 4, dimv, strd, box) || !tc::make_map_bf16(&tu, keep.u, 4, dimu, stru, boxu) ||
        !tc::make_map_bf16(&tds, ws + pl.off_ds, 4, dims, strs, boxs) ||
        !tc::make_map_bf16(&tdk, a.dk, 4, dimk, strdk, boxdv, CU_TENSOR_MAP_SWIZZLE_64B) ||
        !tc::make_map_bf16(&tdv, dv, 4, dimdv, strdv, boxdv, CU_TENSOR_MAP_SWIZZLE_64B) || !tc::make_map_bf16(&tq, f.q, 3, dimq, strq, boxq)) {
      set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (backward operands)");
      return FLARE_ERR_CUDA;
    }
  }
  {
    BwdTcParams p;
    memset(&p, 0, sizeof(p));
    p.q = f.q; p.q_stride_h = f.q_stride_h; p.q_stride_m = f.q_stride_m;
    p.N = f.N; p.H = f.H; p.M = f.M; p.nch = pl.nch; p.npad = pl.npad; p.block = f.block_size;
    p.scale = f.scale; p.power = f.power;
    p.chunk_c = keep.c; p.chunk_d = keep.d; p.tok_l2 = tok_l2; p.tok_delta = tok_delta;
    p.err = err;
    p.gate = gate;
    p.trace = trace_buffer();
    const int mode = f.variant == FLARE_STABLEMAX ? 2 : (f.block_size > 1 ? 1 : 0);
    p.nseg = pl.seg.n;
    memcpy(p.seg_begin, pl.seg.begin, sizeof(p.seg_begin));
    p.lead = pl.seg.lead ? 1 : 0;
    auto sweep = [&](int seg_first, int emit_only) -> int {
      p.seg_first = seg_first;
      p.emit_only = emit_only;
      const dim3 grid((unsigned)lanes, pl.groups, pl.seg.n - seg_first);
      count_launches(1);
      const auto launch = f.Dk == 128   ? (pack ? launch_bwd_tc_unit<4> : launch_bwd_tc_unit<1>)
                          : f.Dv == 128 ? (pack ? launch_bwd_tc_unit<5> : launch_bwd_tc_unit<2>)
                                        : (pack ? launch_bwd_tc_unit<3> : launch_bwd_tc_unit<0>);
      return launch(mode, tk, tv, tdy, tu, tds, tdv, p, grid, stream);
    };
    int rc = FLARE_OK;
    if (pl.seg.n > 1 && !pl.seg.lead) {
      p.xg = reinterpret_cast<float*>(ws + pl.off_xg);
      p.xc = reinterpret_cast<float*>(ws + pl.off_xc);
      rc = sweep(1, 1);
      if (rc != FLARE_OK) return rc;
    }
    rc = sweep(0, 0);
    if (rc != FLARE_OK) return rc;
    if (pl.groups > 1) {
      const int64_t n8 = (int64_t)f.B * f.N * f.H * f.Dv / 8;
      LaunchTimer timer("bwd_tc_sum_groups_kernel", stream);
      FLARE_CUDA_CHECK(launch_pdl(bwd_tc_sum_groups_kernel, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, stream,
                                  reinterpret_cast<const __nv_bfloat16*>(ws + pl.off_dvp), pl.groups, n8,
                                  reinterpret_cast<__nv_bfloat16*>(a.dv)));
      count_launches(1);
    }
  }
  // (4) dK and dQ from the dS plane
  {
    GradTcParams g;
    memset(&g, 0, sizeof(g));
    g.H = f.H; g.M = f.M; g.nch = pl.nch; g.groups = pl.groups;
    g.nsplit = pl.nsplit; g.chunks_per_split = pl.chunks_per_split; g.scale = f.scale;
    g.dq_part = reinterpret_cast<float*>(ws + pl.off_dqp);
    g.err = err;
    const dim3 grid((unsigned)lanes, pl.nsplit, 1);
    const int rc = f.Dk == 128 ? launch_grads<2>(tds, tk, tq, tdk, g, grid, stream) : launch_grads<1>(tds, tk, tq, tdk, g, grid, stream);
    if (rc != FLARE_OK) return rc;
    const int64_t n4 = (int64_t)f.H * f.M * f.Dk / 4;
    LaunchTimer timer("bwd_tc_sum_dq_kernel", stream);
    FLARE_CUDA_CHECK(launch_pdl(bwd_tc_sum_dq_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, g.dq_part,
                                f.B * pl.nsplit, n4, a.dq, a.dq_dtype));
    count_launches(2);
  }
  // (5) path AUTO: the exact pass stands by.  Its kernel looks at the gate word and returns at once unless the tensor
  // kernels above found the inputs outside their numeric domain, in which case it rewrites dq, dk, dv.
  if (f.path == FLARE_PATH_AUTO) {
    flare_bwd_args_t ex = a;
    ex.fwd.path = FLARE_PATH_EXACT;
    ex.fwd.workspace = ws + pl.gate_bytes;
    ex.fwd.workspace_bytes = pl.total - pl.gate_bytes;
    const int rc = bwd_exact(ex, stream, gate, sync);
    if (rc != FLARE_OK) return rc;
  }
  return FLARE_OK;
}

#endif  // FLARE_BT_UNIT

}  // namespace flare
