// Source-term kernels: sin_d12, sds_d12, snl_d12, s_ice and source()
// (umwm_source_functions.F90:16-183, umwm_physics.F90:9-86).
//
// Lane = point: a warp holds 32 consecutive wet points (one block of the
// layout) and reads four directions of all of them per instruction.
//
// The mean-square-slope adjustment of Sds is a prefix over the levels:
//   dummy(o,p) = dummy(o-1,p) + k3dk(o-1) * sum_pp e(o-1,pp) cth2pp(pp,p),
//   cth2pp(pp,p) = cos^2(th(pp)-th(p)) dth
//                = dth/2 (1 + cos2th(pp)cos2th(p) + sin2th(pp)sin2th(p)),
// so dummy(o,.) = A + B cos2th(p) + C sin2th(p) with three sums per point
// (exact algebra; two multiply-adds per bin instead of pm).  They depend on e
// alone and are stored per level (Ptrs::MSS) by the kernel that writes e, so
// the levels are independent of one another here.
//
// Dts pre-pass: per-point max |exponent argument| -> physics_time_step and the
//   global min for dts (umwm_physics.F90:18-41); with compute_rot also the
//   global max of the rotation rate for refraction's dtr
//   (umwm_advection.F90:125-154).  A CTA owns a block; its warps share out the
//   prognostic levels.
//   Bound by the SFU (two of its operations per bin) and HBM about equally.
//   305 k points: 0.33 ms with each warp's next level staged by a bulk copy,
//   0.36 ms loading the rows itself, 0.42 ms for the kernel this replaces (a
//   point's directions over two lanes); 171 points: 12 us with 16 warps, 20 us
//   with 4 (before: 26).
// Integration: exponential integration (o <= oc), equilibrium tail (o > oc),
//   E* = (e + ef)/2 -> ES (umwm_physics.F90:61-84); ef -> EF (= E) above the
//   cut-off only: below it e stays and the propagation forms ef = 2 E* - e,
//   which saves a spectrum write per substep.  A warp takes 12 (or 8)
//   directions of a block and walks the levels downwards with the two levels
//   above in registers (Snl); small models split the levels over several
//   warps of the block's CTA.
//   Bound by issue slots and latency at 15 warps per SM (128 registers).  The
//   walk is downwards so that Snl's two levels are registers, not shared
//   memory; a level's branch (below the cut-off, above, mixed) is taken once
//   for the warp.  305 k points: 0.65 ms (before: 0.84); 171 points: 23 us in
//   five chunks, 43 us in one (before: 47).
#include <algorithm>

#include "kernels.hpp"
#include "misc_body.cuh"
#include "src_body.cuh"

namespace umwm {

// dts of the substep, and in a graph its count and the while node's condition
__device__ __forceinline__ void dts_end(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end) {
  const int left = dts_body(prm, P, compute_rot, end.first);
  if (threadIdx.x == 0 && end.in_graph) {
    Global* g = P.glob;
    g->iters += 1;
    if (g->budget > 0) g->budget -= 1;
    cudaGraphSetConditional(end.loop, (left && g->budget != 0) ? 1u : 0u);
  }
}

// END: the last block through forms dts (dts_fused); compiled in only where it
// is used, since its registers cost the other form 3% at 305 k points.
template <int NP, int W, int MINB, int TMA, bool END>
__global__ void __launch_bounds__(W * 32, MINB)
    k_phys(const Params prm, const Ptrs P, int compute_rot, const SubstepEnd end) {
  __shared__ int last;
  extern __shared__ __align__(128) float dsm[];
  __shared__ float red[W * 64];
  __shared__ float4 dirs[NP / 4 * DIR_ROWS], cw[NP / 4 * 32];
  __shared__ __align__(8) unsigned long long mbar[TMA ? 2 * W : 1];
  dir_fill<NP>(prm, reinterpret_cast<float*>(dirs));  // (phys_body's barrier)
  wait_previous(prm);
  phys_body<NP, TMA>(prm, P, compute_rot, blockIdx.x, adv_smem_u32(dirs), cw, red, dsm, adv_smem_u32(mbar));
  if constexpr (!END) return;
  // thread 0 of each block wrote the block's minimum and maximum
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&P.glob->phys_blocks, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) P.glob->phys_blocks = 0;
  dts_end(prm, P, compute_rot, end);
}
__global__ void k_dts(const Params prm, const Ptrs P, int compute_rot, const SubstepEnd end) {
  wait_previous(prm);
  dts_end(prm, P, compute_rot, end);
}

template <int NP, int W, int MINB, int TMA = 0, bool END = (W == 16)>
static cudaError_t go_phys(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end, int warps,
                           cudaStream_t st) {
  const size_t smem = TMA ? (size_t)warps * 2 * NP * 32 * sizeof(float) : 0;
  if (TMA) {
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e =
        allow_smem((const void*)k_phys<NP, W, MINB, TMA, END>, (size_t)W * 2 * NP * 32 * sizeof(float), done);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(k_phys<NP, W, MINB, TMA, END>, prm.Ntot / 32, warps * 32, smem, st, prm, P, compute_rot, end);
}

// prm.groups4_phys: 16 warps per block (8 where the blocks are more than one
// per SM) instead of 4.  prm.phys_tma (36 directions): the staged form; 0: the
// form that loads its rows itself, with prm.minb_phys the resident CTAs its
// register budget is sized for.
template <int NP>
static cudaError_t launch_phys_np(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end,
                                  cudaStream_t st) {
  if (prm.groups4_phys) return go_phys<NP, 16, 1>(prm, P, compute_rot, end, prm.Ntot / 32 <= prm.nsm ? 16 : 8, st);
  if constexpr (NP == 36) {
    if (prm.phys_tma && end.fused) return go_phys<NP, 4, 5, 1, true>(prm, P, compute_rot, end, 4, st);
    if (prm.phys_tma) return go_phys<NP, 4, 5, 1>(prm, P, compute_rot, end, 4, st);
    if (prm.minb_phys == 5) return go_phys<NP, 4, 5>(prm, P, compute_rot, end, 4, st);
    if (prm.minb_phys == 7) return go_phys<NP, 4, 7>(prm, P, compute_rot, end, 4, st);
  }
  return go_phys<NP, 4, 6>(prm, P, compute_rot, end, 4, st);
}

// The integration: NG direction groups x nc level chunks of one block per CTA.
template <int NP, int WMAX, int MINB>
__global__ void __launch_bounds__(WMAX * 32, MINB) k_integ(const Params prm, const Ptrs P, int nc) {
  // cos(wdir - th) per level chunk: the chunks' warps then need no barrier
  constexpr int NG = NP / integ_dirs<NP>(), NC = WMAX / NG;
  extern __shared__ __align__(128) float dsm[];
  __shared__ float4 dirs[NP / 4 * DIR_ROWS], cw[NC * NP / 4 * 32];
  dir_fill<NP>(prm, reinterpret_cast<float*>(dirs));
  __syncthreads();
  const int w = threadIdx.x >> 5;
  wait_previous(prm);
  integ_body<NP, MINB == 1>(prm, P, adv_smem_u32(dirs), cw + (w / NG) * (NP / 4 * 32), dsm + w * integ_ring_floats<NP>(),
                 blockIdx.x, w, nc);
}

template <int NP, int WMAX, int MINB>
static cudaError_t go_integ(const Params& prm, const Ptrs& P, int nc, cudaStream_t st) {
  constexpr size_t warp = integ_ring_floats<NP>() * sizeof(float);
  const int warps = nc * (NP / integ_dirs<NP>());
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = allow_smem((const void*)k_integ<NP, WMAX, MINB>, WMAX * warp, done);
  if (e != cudaSuccess) return e;
  return launch_chained(k_integ<NP, WMAX, MINB>, prm.Ntot / 32, 32 * warps, warps * warp, st, prm, P, nc);
}

// prm.groups4: the levels of a block in several chunks (small models: the
// walk over all levels is the time of the kernel there).  Else the register
// budget of 15 warps per SM (128 registers), or of 18 where the
// blocks then fit one wave instead of two.  prm.minb_integ 3, 5: 12, 18 warps.
template <int NP>
static cudaError_t launch_integ_np(const Params& prm, const Ptrs& P, cudaStream_t st) {
  constexpr int NG = NP / integ_dirs<NP>(), C15 = std::max(1, 15 / NG), C18 = std::max(1, 18 / NG);
  const int blocks = prm.Ntot / 32;
  if (prm.groups4) {
    const int nc = std::min(blocks <= 2 * prm.nsm ? 16 / NG : 2, prm.O / 4);
    if (nc > 1) return go_integ<NP, 16, 1>(prm, P, nc, st);
  }
  if (NP == 36 && prm.minb_integ == 3) return go_integ<NP, NG, 4>(prm, P, 1, st);
  if (prm.minb_integ == 5 || (blocks > C15 * prm.nsm && blocks <= C18 * prm.nsm))
    return go_integ<NP, NG, C18>(prm, P, 1, st);
  return go_integ<NP, NG, C15>(prm, P, 1, st);
}

#define UMWM_ALL_NP(F, ...)                      \
  switch (prm.P) {                               \
    case 8: return F<8>(__VA_ARGS__);            \
    case 12: return F<12>(__VA_ARGS__);          \
    case 16: return F<16>(__VA_ARGS__);          \
    case 24: return F<24>(__VA_ARGS__);          \
    case 32: return F<32>(__VA_ARGS__);          \
    case 36: return F<36>(__VA_ARGS__);          \
    case 48: return F<48>(__VA_ARGS__);          \
    default: return cudaErrorInvalidConfiguration; \
  }

cudaError_t launch_source_phys(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end,
                               cudaStream_t st) {
  UMWM_ALL_NP(launch_phys_np, prm, P, compute_rot, end, st)
}
cudaError_t launch_dts(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end, cudaStream_t st) {
  return launch_chained(k_dts, 1, 128, 0, st, prm, P, compute_rot, end);
}
cudaError_t launch_source_integ(const Params& prm, const Ptrs& P, cudaStream_t st) {
  UMWM_ALL_NP(launch_integ_np, prm, P, st)
}

bool supported_pm(int pm) {
  const int h = pm / 2;
  return pm % 4 == 0 && (h == 4 || h == 6 || h == 8 || h == 12 || h == 16 || h == 18 || h == 24);
}

}  // namespace umwm
