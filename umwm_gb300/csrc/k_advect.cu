// Propagation, refraction, e = ef and stress('atm') in one pass
// (umwm_advection.F90:18-180, umwm_top.F90:113-115, umwm_stress.F90:17-264).
//
// Thread mapping: a CTA owns one block of 32 consecutive points, lane = point;
// its warps share out the frequency levels, and a thread walks its point's
// whole direction row, four directions at a time.  The levels are independent
// here (the e written is not read again in this kernel), so the number of
// warps is free: it sets how many levels of a block are in flight.  Against
// the split of a point's directions over two or four lanes that this
// replaces, the tables, the per-level factors and the neighbour addresses are
// formed once per level and point, the refraction's p +- 1 are registers, and
// a block's loads do not wait for the level before.
//
// What bounds it: latency, at 12 warps per SM (154 registers; the packed
// arithmetic keeps every per-point factor in a register pair).  Each warp
// therefore has the rows of two quads ahead in flight (cp.async into a ring of
// three slots, adv_body.cuh) and the next level's rows on their way to L2.
// 4 warps per block and three CTAs per SM measured fastest where the blocks
// fill the SMs: 1.17 ms at 305 k points, against 1.38 with two CTAs of 8 warps
// and 1.23 with two of 6 (which spill or hold fewer registers), and 1.32 for
// the kernel this replaces.  With at most two blocks per SM 8 warps are faster
// (45 us against 49 at 9.6 k points; before: 97), with at most one 16 (27 us
// against 31 at 171 points; before: 66).
//
// Propagation.  cg0 > 0, so for an edge velocity cge = (cg0_i + cg0_ie) c,
// (cge + |cge|) = 2 (cg0_i + cg0_ie) max(c, 0) and (cge - |cge|) uses min(c, 0):
// per direction one side of each axis is upwind, known from the direction's
// index, so only that neighbour's row is read, unless the point's current
// blows from the other side (a flag per warp and side).
// The rotation rate is recomputed from cp0 and the currents (it depends on no
// spectral value); when the reference would reuse the rotation of an earlier
// substep (currents = .F.) the mask o <= oc of that substep is kept in oc_rot.
// The wind stress sums e*Sin*cos/sin(th)/cp over the new spectrum while it is
// in registers; the levels' sums meet in shared memory and the first warp adds
// them in the order of the levels (so the results do not depend on the number
// of warps) and finishes the drag, skin stress and ustar.
#include "kernels.hpp"
#include "adv_body.cuh"
#include "misc_body.cuh"

namespace umwm {

// k_advect: register budget for MINB resident CTAs of at most W warps per SM;
// CNT counts the non-negativity cut.
template <int NP, bool CURV, int W, int MINB, bool CNT = false>
__global__ void __launch_bounds__(W * 32, MINB) k_advect(const Params prm, const Ptrs P) {
  extern __shared__ __align__(128) float dsm[];
  __shared__ float4 dirs[NP / 4 * DIR_ROWS], cw[NP / 4 * 32];
  dir_fill<NP>(prm, reinterpret_cast<float*>(dirs));  // (advect_body's barrier)
  wait_previous(prm);
  advect_body<NP, CURV, CNT, false, (MINB > 2)>(prm, P, blockIdx.x, adv_smem_u32(dirs), cw, dsm, dsm + adv_red_floats(prm.O));
  // the block of a member's print point (its first block without one) writes
  // the member's screen line and counts the substep; a kernel of its own took
  // 8 to 14 us a substep, this 0 to 2 us
  const Member& M = prm.mem[prm.tile_mem[(blockIdx.x * 32) / TILE]];
  if ((M.iip >= 0 ? M.iip : M.off) >> 5 == blockIdx.x) {
    __syncthreads();  // this block's spectrum and stress are written
    screen_member<256>(prm, P, M, dsm, dsm + 256);
  }
}

template <int NP, bool CURV, int W, int MINB, bool CNT = false>
static cudaError_t go(const Params& prm, const Ptrs& P, int warps, cudaStream_t st) {
  const size_t smem = (adv_red_floats(prm.O) + (size_t)warps * adv_ring_floats<NP>()) * sizeof(float);
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = allow_smem((const void*)k_advect<NP, CURV, W, MINB, CNT>,
                                   (adv_red_floats(MAX_OM) + (size_t)W * adv_ring_floats<NP>()) * sizeof(float), done);
  if (e != cudaSuccess) return e;
  return launch_chained(k_advect<NP, CURV, W, MINB, CNT>, prm.Ntot / 32, warps * 32, smem, st, prm, P);
}

// prm.adv_groups4: 16 warps per block (8 where the blocks are more than one
// per SM) instead of 4.  prm.minb_adv 4, 5 (36 directions): 8, 6 warps, two
// CTAs per SM.
template <int NP, bool CURV>
static cudaError_t launch_np(const Params& prm, const Ptrs& P, cudaStream_t st) {
  if constexpr (NP == 36) {
    if (prm.count_cut) return go<NP, CURV, 4, 3, true>(prm, P, 4, st);
    if (!prm.adv_groups4 && prm.minb_adv == 5) return go<NP, CURV, 6, 2>(prm, P, 6, st);
    if (!prm.adv_groups4 && prm.minb_adv == 4) return go<NP, CURV, 8, 2>(prm, P, 8, st);
  }
  if (prm.adv_groups4)
    return prm.Ntot / 32 <= prm.nsm ? go<NP, CURV, 16, 1>(prm, P, 16, st) : go<NP, CURV, 8, 2>(prm, P, 8, st);
  return go<NP, CURV, 4, 3>(prm, P, 4, st);
}

cudaError_t launch_advect(const Params& prm, const Ptrs& P, cudaStream_t st) {
  const bool curv = prm.curvilinear != 0;
  switch (prm.P) {
#define CASE(X) \
  case X: return curv ? launch_np<X, true>(prm, P, st) : launch_np<X, false>(prm, P, st);
    CASE(8) CASE(12) CASE(16) CASE(24) CASE(32) CASE(36) CASE(48)
#undef CASE
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace umwm
