// The exact backward standing by behind the tensor-core one, as ONE kernel instead of nine: in a call that stays inside the
// tensor kernels' numeric domain each of the nine only cost its launch (B200: 25 of 112 us of a training step at B=2 N=1000 H=8
// M=64 D=64, stablemax: 112 -> 95 us with one).
//
// The nine kernels' CTAs are tasks, handed out one after another, phase by phase, by a counter.  A task of a phase begins when
// all tasks of the phase before are done, whose number another counter holds.  Every task handed out belongs to a CTA that
// is running, and waits only for tasks handed out before it, so the waits end whatever number of CTAs is resident (no
// cooperative launch, which would want the whole GPU at once); they are bounded all the same: a CTA that sees no task of the phase
// before it end for kPatience gives up, and so do the others with it.
//
// A call that is redone takes as long as with the nine kernels, 0.98 to 1.03 times over six shapes of M = 32 .. 256 (B=4 N=2048 H=16
// M=64 D=128 5.36 and 5.27 ms, B=1 N=8192 H=8 M=128 D=128 16.7 and 16.6), but where a walk of many latents leaves one CTA per SM to
// the phases that had several: M=256 D=64 B=8 N=2048 H=16 19.0 -> 20.9 ms, M=512 11.2 -> 11.8.  The launches saved for the
// calls that are not redone weigh more.
#include "bwd_cta.cuh"
#include "fold_device.cuh"
#include "walk_cta.cuh"

namespace flare {

namespace {

// ns; one task at most walks a lane, a few us for each of its tokens: longer than any task that fits the GPU's memory takes
constexpr uint64_t kPatience = 20000000000ull;

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <int MM_MAX, int DD>
__global__ void __launch_bounds__(NT, (MM_MAX * DD <= 32) ? 2 : 1) bwd_standby_kernel(const __grid_constant__ StandbyParams p) {
  pdl_begin();
  if (*p.gate == 0) return;
  // the last 16 bytes of the dynamic shared memory (a static variable would not fit beside the most that may be asked for)
  extern __shared__ __align__(16) float smem_raw[];
  uint32_t smem_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(smem_bytes));
  volatile int* const word = reinterpret_cast<volatile int*>(reinterpret_cast<uint8_t*>(smem_raw) + smem_bytes - 16);
  int phase = 0, first = 0;  // phase of this CTA's next task, number of its first task
  for (;;) {
    __syncthreads();  // everyone is done with the task before (shared memory, ticket)
    if (threadIdx.x == 0) word[0] = atomicAdd(p.sync, 1);
    __syncthreads();
    const int ticket = word[0];
    for (; phase < kStandbyPhases; ++phase) {
      const int n = p.nx[phase] * p.ny[phase] * p.nz[phase];
      if (ticket < first + n) break;
      first += n;
    }
    if (phase == kStandbyPhases) return;
    if (threadIdx.x == 0) {
      // phases end in their order, so the last one before this with tasks says it all
      int before = phase - 1, want = 0;
      for (; before >= 0; --before) {
        want = p.nx[before] * p.ny[before] * p.nz[before];
        if (want > 0) break;
      }
      bool ok = true;
      if (before >= 0) {
        int seen = -1;
        uint64_t since = 0;
        for (;;) {
          const int done = load_acquire(p.sync + 1 + before);
          if (done >= want) break;
          if (done != seen) {
            seen = done;
            since = now_ns();
          }
          ok = now_ns() - since < kPatience && load_acquire(p.sync + 1 + kStandbyPhases) == 0;
          if (!ok) break;
          __nanosleep(128);
        }
      }
      word[1] = ok;
    }
    __syncthreads();
    __threadfence();
    if (!word[1]) {
      if (threadIdx.x == 0) {
        atomicOr(p.sync + 1 + kStandbyPhases, 1);
        atomicOr(p.err, 1);
      }
      return;
    }
    const int i = ticket - first;
    const uint3 blk = make_uint3(i % p.nx[phase], i / p.nx[phase] % p.ny[phase], i / (p.nx[phase] * p.ny[phase]));
    switch (phase) {
      case 0: walk_cta<MM_MAX, DD>(p.walk, blk); break;
      case 1: {
        const int m = blk.y * NW + (threadIdx.x >> 5);
        if (m < p.fold.M) fold::fold_row(p.fold, blk.x, m, threadIdx.x & 31);
        break;
      }
      case 2: replay_cta<MM_MAX, DD>(p.bwd, blk); break;
      case 3: carry_cta(p.carry, blk); break;
      case 4: scan_element(p.scan, (int64_t)blk.x * NT + threadIdx.x); break;
      case 5: reverse_cta<MM_MAX, DD>(p.bwd, blk); break;
      case 6: rows_cta(p.rows, blk); break;
      case 7: lat_cta(p.lat, blk); break;
      default: sum_element(p.sum, (int64_t)blk.x * NT + threadIdx.x); break;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(p.sync + 1 + phase, 1);
  }
}

template <int MM_MAX, int DD>
int launch_one(const StandbyParams& p, size_t smem, cudaStream_t stream) {
  auto kern = bwd_standby_kernel<MM_MAX, DD>;
  FLARE_CUDA_CHECK(allow_smem(kern));
  int most = 1;  // as many CTAs as the widest phase has tasks, two per SM at most
  for (int i = 0; i < kStandbyPhases; ++i) {
    const int64_t n = (int64_t)p.nx[i] * p.ny[i] * p.nz[i];
    if (n > most) most = n < 2 * sm_count() ? (int)n : 2 * sm_count();
  }
  LaunchTimer timer("bwd_standby_kernel", stream);
  FLARE_CUDA_CHECK(launch_pdl(kern, dim3((unsigned)most), dim3(NT), smem + 16, stream, p));
  return FLARE_OK;
}

}  // namespace

template <>
int launch_bwd_standby<FLARE_WALK_MM>(const StandbyParams& p, int dd, size_t smem, cudaStream_t stream) {
  constexpr int MM_MAX = FLARE_WALK_MM;
  if (dd == 1) return launch_one<MM_MAX, 1>(p, smem, stream);
  if (dd == 2) {
    if constexpr (MM_MAX * 2 <= 64) return launch_one<MM_MAX, 2>(p, smem, stream);
  }
  if (dd == 4) {
    if constexpr (MM_MAX * 4 <= 64) return launch_one<MM_MAX, 4>(p, smem, stream);
  }
  return FLARE_ERR_UNSUPPORTED;
}

}  // namespace flare
