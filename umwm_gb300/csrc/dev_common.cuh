// Device helpers shared by the kernel translation units.
#pragma once
#include <cuda_runtime.h>

#include "dev.cuh"

namespace umwm {

__device__ __forceinline__ unsigned enc_ord_d(float x) {
  unsigned u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float dec_ord_d(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// sheltering_coare35, umwm_sheltering.F90:49-79
__device__ __forceinline__ float shelter_coare35(float w) {
  const float x1 = 15.f, x2 = 33.f, x3 = 60.f, y1 = 0.10f, y2 = 0.09f, y3 = 0.06f;
  const float intercept = 0.04f, curvature = 0.65f, decay = 1.6f;
  float slope1 = (y1 - intercept) / x1;
  float slope2 = (y3 - y2) / (x3 - x2);
  float c = curvature * (slope2 - slope1) / (x2 - x1);
  float b = slope1 - 2.f * c * x1;
  float a = y1 - b * x1 - c * (x1 * x1);
  float s1 = a + b * x2 + c * (x2 * x2);
  if (w <= x1) return intercept + slope1 * w;
  if (w <= x2) return a + b * w + c * (w * w);
  return s1 * expf(-(w - x2) / (decay * w));
}

// Per-point inputs of the wind-input source term, sin_d12
// (umwm_source_functions.F90:16-82).
struct WindIn {
  float wspd, uc, vc, ustar25, shelt, c1;
  int oc;  // 1-based cut-off index; 0-based level o is prognostic when o < oc
};

// jj: global wet index; ja: its all-point index
__device__ __forceinline__ WindIn load_wind(const Params& prm, const Ptrs& P, int jj, int ja, float ustar) {
  WindIn w;
  w.wspd = P.wspd[ja];
  w.uc = P.uc[ja];
  w.vc = P.vc[ja];
  w.ustar25 = 2.5f * ustar;
  w.shelt = P.shelt[jj];
  // (1 - fice) * twopi * rhorat
  w.c1 = ((1.f - P.fice[ja]) * (2.f * 3.14159274f)) * P.rhorat[ja];
  w.oc = P.oc[jj];
  return w;
}

// all-point index of a wet (or ghost) point of member M
__device__ __forceinline__ int apt(const Member& M, int j) { return M.nmoff + (j - M.off); }

// max(x, 0) with NaN kept (max.NaN)
__device__ __forceinline__ float max_nan0(float x) {
  float r;
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// max(x, lo) with NaN kept
__device__ __forceinline__ float max_nan(float x, float lo) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(lo));
  return r;
}

// Sin of one bin from x = U cos(wdir - th) - cp0 - uc cos th - vc sin th,
// umwm_source_functions.F90:39-80, with its factors folded: the reference
// forms sin_fac |x| x, then multiplies by shelt/sin_fac where positive, by
// fieldscale1 where negative and by fieldscale2 where still negative and
// cos(wdir - th) > 0, then by (1 - fice) 2 pi rhorat and fkovg.  Here
// (x |x|) is multiplied once by the factor its sign selects (shelt, or
// sin_fac fieldscale1 [fieldscale2], prm.sin_neg1/2) and once by
// gl = (1 - fice) 2 pi rhorat fkovg of the level: the same product in
// another order (a few ulp apart), in fewer instructions.
__device__ __forceinline__ float sin_fold(const Params& prm, float shelt, float x, float cw, float gl, bool tail) {
  const float a = x * fabsf(x);
  const float f = x > 0.f ? shelt : (cw > 0.f ? prm.sin_neg2 : prm.sin_neg1);
  float s = (a * f) * gl;
  if (tail) s = fmaxf(s, 0.f);
  return s;
}

// 2^x through the SFU (ex2.approx.ftz)
__device__ __forceinline__ float ex2a(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// bulk prefetch of a contiguous, 16-byte aligned range into L2 (sizes are multiples of 16 bytes)
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// k^4 rounded once (the products' errors carried), as the host's tables have powers
__device__ __forceinline__ float pow4(float k) {
  const float h = __fmul_rn(k, k), l = fmaf(k, k, -h), q = __fmul_rn(h, h);
  return __fadd_rn(q, fmaf(2.f * h, l, fmaf(h, h, -q)));
}

// The direction constants of four directions: cos and sin of th and of 2 th,
// and the mean sin and cos over the edge to the next direction.  A CTA copies
// them to shared memory ([pm/4] of them, float4 each): the packed arithmetic
// takes register pairs, and holding pm of them over the levels (where the
// compiler puts loop-invariant constants) would cost the registers.
enum DirRow { DIR_C = 0, DIR_S, DIR_C2, DIR_S2, DIR_SH, DIR_CH, DIR_ROWS };
template <int NP>
__device__ __forceinline__ void dir_fill(const Params& prm, float* d) {  // then a CTA barrier
  for (int p = threadIdx.x; p < NP; p += blockDim.x) {
    float* r = d + (p >> 2) * (4 * DIR_ROWS) + (p & 3);
    r[4 * DIR_C] = prm.dcth[p];
    r[4 * DIR_S] = prm.dsth[p];
    r[4 * DIR_C2] = prm.dc2th[p];
    r[4 * DIR_S2] = prm.ds2th[p];
    r[4 * DIR_SH] = prm.shs[p];
    r[4 * DIR_CH] = prm.chs[p];
  }
}
// (volatile: read where it is used)
struct F2x2 {
  float2 a[2];
};
__device__ __forceinline__ F2x2 dir4(uint32_t dirs, int q, int row) {
  F2x2 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.a[0].x), "=f"(v.a[0].y), "=f"(v.a[1].x), "=f"(v.a[1].y)
               : "r"(dirs + (uint32_t)(q * DIR_ROWS + row) * 16u));
  return v;
}

// cos(wdir - th) of directions 4q0 .. 4q1 - 1 of this lane's point into shared
// memory, four directions per float4: cw[q * 32 + lane].  (Formed from the
// rounded angle as the reference does: x = U cos(wdir - th) - cp0 - ...
// cancels, and products of cos wdir and cos th round differently there.)
__device__ __forceinline__ void cw_fill(const Params& prm, float wdir, int q0, int q1, int step, float4* cw) {
  const int lane = threadIdx.x & 31;
  for (int q = q0; q < q1; q += step)
    cw[q * 32 + lane] = make_float4(cosf(wdir - prm.th[4 * q]), cosf(wdir - prm.th[4 * q + 1]),
                                    cosf(wdir - prm.th[4 * q + 2]), cosf(wdir - prm.th[4 * q + 3]));
}

// The substep's kernels are launched without waiting for the one before
// (launch_chained); each waits here, before its first load of a result, until
// that kernel has completed and its results are visible.  (Every result is
// read behind the branch on the member's flags, themselves read after this.)
// A kernel of at most one block per SM lets the next one's blocks onto the SMs
// as soon as its own are all there.  A larger one does not: the blocks that
// come early crowd the SMs that are done first (13 k points 7.53 ms per 40
// substeps without chaining, 7.85 with every kernel starting early, 7.37 so).
__device__ __forceinline__ void let_next_start(const Params& prm) {
  if (gridDim.x <= prm.nsm) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_previous(const Params& prm) {
  let_next_start(prm);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Copies to shared memory behind the thread's back (16 bytes through L2 only,
// 4 bytes); copy_async_wait: all of this thread's but the last N groups have landed
__device__ __forceinline__ void copy_async16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two directions' parts of a level's mss sums, e (1, cos 2th, sin 2th), even and
// odd directions apart.  Whoever writes e adds them so.
__device__ __forceinline__ void mss_add(float2 e, float2 c2, float2 s2, float2& m0, float2& m1, float2& m2) {
  m0 = __fadd2_rn(m0, e);
  m1 = __ffma2_rn(e, c2, m1);
  m2 = __ffma2_rn(e, s2, m2);
}

// The mss prefix of sum m (0: A, 1: B, 2: C) of block blk, one lane per point:
// MSS[o] = the levels' sums below o, from v[o * stride + m * 32 + lane] in
// shared memory, added in the order of the levels.
__device__ __forceinline__ void mss_prefix(const Params& prm, const Ptrs& P, int blk, int m, const float* v,
                                           int stride) {
  const int lane = threadIdx.x & 31;
  float a = 0.f;
  float* out = P.MSS + (size_t)blk * prm.O * 96 + m * 32 + lane;
#pragma unroll 4
  for (int o = 0; o < prm.O; ++o) {
    out[(size_t)o * 96] = a;
    a += v[(size_t)o * stride + m * 32 + lane];
  }
}

// stress_tail, umwm_stress.F90:300-311
__device__ __forceinline__ float stress_tail(float w, float kmax) {
  const float kcap = 1e3f, a = 0.000112f, b = -0.01451f, c = -1.0186f;
  float tail = a * (w * w) + b * w + c;
  float kpt = powf(kmax, tail);
  return (powf(kcap, tail + 1.f) - kmax * kpt) / (kpt * (tail + 1.f));
}

// 1-D bulk copies (TMA) into shared memory completing on an mbarrier, and
// the bounded wait for them (about 2 s of clock)
__device__ __forceinline__ uint32_t adv_smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void adv_mbar_init(uint32_t bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void adv_mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void adv_bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool adv_mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool adv_mbar_wait(uint32_t bar, uint32_t parity, long long limit_cycles) {
  if (adv_mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!adv_mbar_try(bar, parity))
    if (clock64() - t0 > limit_cycles) return false;
  return true;
}

}  // namespace umwm
