// Tensor-core (tcgen05 + TMEM + TMA) backward pass (see bwd_tc.cu).
#pragma once
#include "flare_common.cuh"

namespace flare {

// Per-chunk prefix states kept by the tensor-core forward for the backward pass (chunks of 128 tokens over the
// whole sequence): u bf16 [lanes][nch][M][Dv], c / d fp32 [lanes][nch][M].
struct ChunkStates {
  void* u;
  float *c, *d;
  int nch;
};

// Layout of flare_fwd_args_t::keep for a problem (all offsets in bytes; total == 0: the problem keeps nothing).  It depends on
// the sizes alone: the forward that fills it and the backward that reads it may run under different instance choices.
struct KeepLayout {
  size_t off_gate, off_u, off_c, off_d, total;
  size_t gate_words;
  int nch;
};
KeepLayout keep_layout(const flare_fwd_args_t& f);

// true when flare_backward takes the tensor-core kernels for this problem
bool bwd_tc_supported(const flare_bwd_args_t& a);
size_t bwd_tc_workspace_bytes(const flare_bwd_args_t& a);
int bwd_tc(const flare_bwd_args_t& a, cudaStream_t stream);

// Forward on the tensor path that also writes y, the decode log-sum-exp and the per-chunk prefix states
// (defined with the forward dispatch).
// `gate` (may be null): forward_gate_words() ints, of which the kernels write 1 + lanes * gate[0] (see TcParams::gate).
int forward_keep_states(const flare_fwd_args_t* a, const ChunkStates& keep, int* gate, cudaStream_t stream);
// room for the gate words of any forward of these sizes on the tensor path: one leading word and the CTAs' words
size_t forward_gate_words(const flare_fwd_args_t* a);
// diagnostic buffer set with flare_set_trace_buffer (null in normal use)
long long* trace_buffer();
// kernels launched so far by the current forward / backward call of this thread (measurement hook)
void count_launches(int n);

}  // namespace flare
