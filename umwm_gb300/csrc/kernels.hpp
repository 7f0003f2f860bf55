// Launchers of the GB300 UMWM kernels (all on one stream).
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "dev.cuh"

namespace umwm {

// Lets kernel f take `bytes` of dynamic shared memory on the current device
// (once per kernel and device; done: the devices it has been set on).
inline cudaError_t allow_smem(const void* f, size_t bytes, std::atomic<unsigned long long>& done) {
  int d = 0;
  cudaError_t e = cudaGetDevice(&d);
  if (e != cudaSuccess || (d < 64 && (done.load(std::memory_order_relaxed) >> d & 1))) return e;
  e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && d < 64) done.fetch_or(1ull << d, std::memory_order_relaxed);
  return e;
}

// Launch of a substep's kernel behind another one on the stream: its blocks may
// start while the last of the kernel before are at work, up to
// wait_previous(), so that the launch and the kernel's set-up are off
// the chain of a substep's kernels.
template <typename... K, typename... A>
cudaError_t launch_chained(void (*f)(K...), int grid, int block, size_t smem, cudaStream_t st, const A&... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, f, a...);
}

bool supported_pm(int pm);
cudaError_t launch_prep(const Params& prm, const Ptrs& P, int compute_rot, int max_nm, cudaStream_t st);
// What follows the dts pre-pass's last block: dts, dtr and sumt of every
// member, and in a graph the count of the substep and the condition of its
// while node (another substep while a member is inside the dtg and the budget
// lasts).
struct SubstepEnd {
  int first;      // the reference's 'first'
  int fused;      // the pre-pass's last block does it, not launch_dts
  int in_graph;   // loop is the graph's while node
  cudaGraphConditionalHandle loop;
};
// The pre-pass does it itself in the split for small models and in the staged
// form on grids of at most four blocks of 32 points per SM: the ticket each
// block takes lengthens the pre-pass by 1 to 2 us there
// (171 to 17 k points), a launch of its own is 6 to 7 us.  On larger grids
// every wave of blocks waits for its tickets: +5 us at 32 k points, +8 at 86 k
// and +32 of 331 at 305 k.
inline bool dts_fused(const Params& prm) {
  return prm.groups4_phys || (prm.P == 36 && prm.phys_tma && prm.Ntot / 32 <= 4 * prm.nsm);
}
cudaError_t launch_dts(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end, cudaStream_t st);
cudaError_t launch_source_phys(const Params& prm, const Ptrs& P, int compute_rot, const SubstepEnd& end,
                               cudaStream_t st);
cudaError_t launch_source_integ(const Params& prm, const Ptrs& P, cudaStream_t st);
cudaError_t launch_advect(const Params& prm, const Ptrs& P, cudaStream_t st);
cudaError_t launch_diag(const Params& prm, const Ptrs& P, cudaStream_t st);
cudaError_t launch_stokes(const Params& prm, const Ptrs& P, cudaStream_t st);
cudaError_t launch_to_ref(const Params& prm, const float* E, float* F, int off, int n, cudaStream_t st);
cudaError_t launch_from_ref(const Params& prm, const float* F, float* E, int off, int n, cudaStream_t st);
// the mss prefix of the points [off, off + padded) (whole blocks) from e
cudaError_t launch_mss(const Params& prm, const Ptrs& P, int off, int padded, cudaStream_t st);
cudaError_t launch_begin_dtg(const Params& prm, cudaStream_t st);
cudaError_t launch_stress_ocn(const Params& prm, const Ptrs& P, cudaStream_t st);
cudaError_t launch_loop_arm(Global* g, int budget, cudaStream_t st);
cudaError_t launch_count_nonfinite(const float* a, size_t n, int* count, cudaStream_t st);
cudaError_t launch_fill(float* a, size_t n, float v, cudaStream_t st);
// persistent substep kernel (k_persist.cu): up to Global::budget substeps
// (armed by launch_loop_arm) of every member in one cooperative launch;
// Global::iters counts them, bar_err marks a barrier wait that ran out
// (stall_test: one CTA more is expected than launched, so every wait runs
// out after 20 ms)
bool persist_supported(const Params& prm);
cudaError_t launch_persist(const Params& prm, const Ptrs& P, int stall_test, cudaStream_t st);

}  // namespace umwm
