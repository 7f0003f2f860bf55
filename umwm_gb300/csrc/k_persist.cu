// Persistent substep kernel: the inner dynamic-dts loop of umwm_run
// (umwm_top.F90:97-150) for every member of a model in one cooperative
// launch.  Each CTA loops over substeps; within a substep it takes the
// stages in order (forcing interpolation, the dts pre-pass,
// dts, the integration, propagation + refraction + stress, the screen line),
// working through the stage's tiles grid-stride, with a grid-wide barrier
// between stages.  The stage bodies are those of the per-stage kernels
// (src_body.cuh, adv_body.cuh, misc_body.cuh); the propagation reads E*
// with coherent loads, since the same launch wrote it.  The loop ends when no
// member is left inside the dtg or the armed substep budget is spent.
//
// Every barrier wait is bounded (a globaltimer limit); a wait that runs out
// sets Global::bar_err and its CTA returns, and so does every CTA at its next
// barrier, so the launch always ends and the host reports UMWM_ERR_TIMEOUT.
// All CTAs are co-resident (cooperative launch, grid sized from the occupancy
// of this kernel), which is what the barrier needs.
#include <algorithm>

#include "adv_body.cuh"
#include "kernels.hpp"
#include "misc_body.cuh"
#include "src_body.cuh"

namespace umwm {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier over `expected` CTAs with a bounded wait.  Returns false
// (in every thread of the CTA) when this or an earlier wait gave up.
__device__ __forceinline__ bool grid_barrier(Global* g, unsigned expected, unsigned long long limit_ns, int* ok_s) {
  __syncthreads();  // this CTA's stage work is done
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile unsigned* genp = &g->bar_gen;
    const unsigned gen = *genp;
    __threadfence();  // release this CTA's writes before arriving
    if (atomicAdd(&g->bar_count, 1u) == expected - 1) {
      atomicExch(&g->bar_count, 0u);
      __threadfence();
      atomicAdd(&g->bar_gen, 1u);
    } else {
      const unsigned long long t0 = globaltimer_ns();
      while (*genp == gen) {
        if (globaltimer_ns() - t0 > limit_ns) {
          atomicExch(&g->bar_err, 1);
          ok = 0;
          break;
        }
        __nanosleep(100);
      }
    }
    __threadfence();  // acquire the other CTAs' writes
    *ok_s = ok && *(volatile int*)&g->bar_err == 0;
  }
  __syncthreads();
  return *ok_s != 0;
}

// The forcing interpolation of every member still inside the dtg, PREP_U
// points per thread with their loads first (prep_points).  One point per
// thread: more overlap their latencies, but their registers cost the
// propagation, which shares the budget, more than that saves.
#ifndef UMWM_PERSIST_PREP_U
#define UMWM_PERSIST_PREP_U 1
#endif
__device__ __forceinline__ void forcing_stage(const Params& prm, const Ptrs& P, int nb, int compute_rot) {
  constexpr int U = UMWM_PERSIST_PREP_U;
  for (int m = 0; m < prm.nmem; ++m) {
    const Member& M = prm.mem[m];
    Ctl* ctl = M.ctl;
    if (ctl->done) continue;
    bool cur = false;
    for (int i = blockIdx.x * 128 + threadIdx.x; i < M.NM; i += U * nb * 128)
      cur |= prep_points<U>(prm, P, M, ctl, i, nb * 128, compute_rot);
    set_anycurrent(ctl, cur);
  }
}

// dynamic shared memory of the stages, one after another: the propagation's
// level sums and rows in flight, the integration's cos(wdir - th) and rows in
// flight per warp
template <int NP>
static size_t persist_smem(int om) {
  return sizeof(float) * std::max(adv_red_floats(om) + 4 * adv_ring_floats<NP>(), 4 * (NP * 32 + integ_ring_floats<NP>()));
}

template <int NP, bool CURV>
#ifndef UMWM_PERSIST_MINB
#define UMWM_PERSIST_MINB 4  // resident CTAs per SM
#endif
__global__ void __launch_bounds__(128, UMWM_PERSIST_MINB)
    k_persist(const Params prm, const Ptrs P, unsigned expected, unsigned long long limit_ns) {
  extern __shared__ __align__(128) float dsm[];
  __shared__ float phys_s[4 * 64], scr[2][256];
  __shared__ int ok_s;
  __shared__ float4 dirs_s[NP / 4 * DIR_ROWS], cw[NP / 4 * 32];
  dir_fill<NP>(prm, reinterpret_cast<float*>(dirs_s));
  __syncthreads();
  const uint32_t dirs = adv_smem_u32(dirs_s);
  constexpr int NG = NP / integ_dirs<NP>();
  const int nvb = prm.Ntot / 32;  // blocks of 32 points
  const int warp = threadIdx.x >> 5;
  const int nb = gridDim.x;
  const int compute_rot = prm.currents;
  Global* gl = P.glob;
  // each barrier ends a stage; block 0 books the stage's time
  unsigned long long t_last = globaltimer_ns();
  auto bar_s = [&](int stage) {
    const bool ok = grid_barrier(gl, expected, limit_ns, &ok_s);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const unsigned long long t = globaltimer_ns();
      gl->stage_ns[stage] += t - t_last;
      t_last = t;
    }
    return ok;
  };
  const int budget = gl->budget;  // armed before the launch (k_loop_arm)
  for (int it = 0; it < budget; ++it) {
    forcing_stage(prm, P, nb, compute_rot);
    if (!bar_s(0)) return;
    for (int v = blockIdx.x; v < nvb; v += nb) {
      phys_body<NP, 0>(prm, P, compute_rot, v, dirs, cw, phys_s, nullptr, 0u);
      __syncthreads();  // the next block reuses the maxima
    }
    if (!bar_s(2)) return;
    if (blockIdx.x == 0) dts_body(prm, P, compute_rot, 0);
    if (!bar_s(3)) return;
    for (int u = blockIdx.x * 4 + warp; u < nvb * NG; u += nb * 4) 
      integ_body<NP, false>(prm, P, dirs, reinterpret_cast<float4*>(dsm) + warp * (NP / 4 * 32),
                     dsm + 4 * NP * 32 + warp * integ_ring_floats<NP>(), u / NG, u % NG, 1);
    if (!bar_s(4)) return;
    for (int v = blockIdx.x; v < nvb; v += nb) {
      advect_body<NP, CURV, false, true, false>(prm, P, v, dirs, cw, dsm, dsm + adv_red_floats(prm.O));
      __syncthreads();  // the next block reuses the sums
    }
    if (!bar_s(5)) return;
    for (int m = blockIdx.x; m < prm.nmem; m += nb) {
      screen_member<256>(prm, P, prm.mem[m], scr[0], scr[1]);
      __syncthreads();  // the next member reuses the sums
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) gl->iters += 1;
    if (!bar_s(6)) return;
    // not_done was set by this substep's dts, two barriers ago
    if (*(volatile int*)&gl->not_done == 0) break;
  }
}

// reset of the barrier before a launch
__global__ void k_persist_arm(Global* g) {
  g->bar_count = 0;
  g->bar_gen = 0;
  g->bar_err = 0;
}

template <int NP, bool CURV>
static cudaError_t launch_persist_t(const Params& prm, const Ptrs& P, int stall_test, cudaStream_t st) {
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = persist_smem<NP>(prm.O);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_persist<NP, CURV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)persist_smem<NP>(MAX_OM));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_persist<NP, CURV>, 128, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const unsigned grid = (unsigned)std::max(1, std::min(nsm * per_sm, prm.Ntot / 32));
  // the barrier expects one CTA more than launched when the stall test is
  // armed: every wait then runs out after 20 ms
  const unsigned expected = grid + (stall_test ? 1u : 0u);
  const unsigned long long limit_ns = stall_test ? 20000000ull : 2000000000ull;
  k_persist_arm<<<1, 1, 0, st>>>(P.glob);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  void* args[] = {(void*)&prm, (void*)&P, (void*)&expected, (void*)&limit_ns};
  return cudaLaunchCooperativeKernel((const void*)k_persist<NP, CURV>, dim3(grid), dim3(128), args, smem, st);
}

// (The kernel has a split of its own; that the others' agree is asked as it was
// when they were mappings that rounded differently.)
bool persist_supported(const Params& prm) {
  return prm.P == 36 && prm.groups4 == prm.groups4_phys && prm.groups4 == prm.adv_groups4;
}

cudaError_t launch_persist(const Params& prm, const Ptrs& P, int stall_test, cudaStream_t st) {
  if (!persist_supported(prm)) return cudaErrorInvalidConfiguration;
  const bool curv = prm.curvilinear != 0;
  return curv ? launch_persist_t<36, true>(prm, P, stall_test, st) : launch_persist_t<36, false>(prm, P, stall_test, st);
}

}  // namespace umwm
