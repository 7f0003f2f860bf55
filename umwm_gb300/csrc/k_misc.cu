// Per-substep forcing and cut-off kernel, and the once-per-output kernels:
// diag, Stokes drift, stress('ocn') and the spectrum layout transposes.
#include <algorithm>
#include <cfloat>

#include "kernels.hpp"
#include "misc_body.cuh"

namespace umwm {

// forcinginterpolate + the global side effects at the top of sin_d12
// (umwm_forcing.F90:40-99, umwm_source_functions.F90:21-36): per unrolled
// point (land included) interpolate the 2-d forcing levels in sumt/dtg,
// clamp wspd, rhorat; per wet point the cut-off index oc and the
// sheltering coefficient (umwm_source_functions.F90:52).
__global__ void k_prep(const Params prm, const Ptrs P, int compute_rot) {
  let_next_start(prm);
  const Member& M = prm.mem[blockIdx.y];
  Ctl* ctl = M.ctl;
  if (ctl->done) return;
  bool cur = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.NM; i += gridDim.x * blockDim.x)
    cur |= prep_points<1>(prm, P, M, ctl, i, 0, compute_rot);
  set_anycurrent(ctl, cur);
}

// The once-per-interval kernels below share one mapping: a CTA owns a block of 32 points (lane = point), its MW warps take
// every MW-th frequency level and read four directions of 32 points per
// access, and the warps' partial sums meet in shared memory.  One thread per
// point walked 1332 bins in a chain of dependent loads: 94 us at 171 points
// and 543 us at 305 k for the diagnostics, 270 and 1140 us for the Stokes
// drift.  So split: 18 and 503 us, 26 and 493 us (small models wait on the
// levels' chain; at 305 k points the 1.6 GB spectrum is read at 3.2 TB/s, the
// rest being the level sums' instructions).
constexpr int MW = 8;

struct BlockPoint {
  int j, lane, w;
  bool valid;
};
// false (for the whole CTA): a block of padding
__device__ __forceinline__ bool block_point(const Member& Mb, BlockPoint& b) {
  b.lane = threadIdx.x & 31;
  b.w = threadIdx.x >> 5;
  b.j = blockIdx.x * 32 + b.lane;
  b.valid = b.j < Mb.ghost;
  return blockIdx.x * 32 < Mb.ghost;
}
// cos th and sin th, four directions each, [pm/4][2] (then a CTA barrier)
__device__ __forceinline__ void fill_cs(const Params& prm, float* cs) {
  for (int p = threadIdx.x; p < prm.P; p += blockDim.x) {
    cs[(p >> 2) * 8 + (p & 3)] = prm.cth[p];
    cs[(p >> 2) * 8 + 4 + (p & 3)] = prm.sth[p];
  }
}

// diag, umwm_physics.F90:89-205.  A level's direction sums are formed first
// and weighted by its table rows, so the sums run in another order than the
// reference's direction-outer loops; the peak keeps the reference's choice
// among equal values, the first in its (o fastest, p slowest) order.
__global__ void __launch_bounds__(MW * 32) k_diag(const Params prm, const Ptrs P) {
  enum { M0, M2, M2K, XC, YC, MX, MY, CXX, CXY, CYY, NS };
  __shared__ float part[MW][NS][32], pbest[MW][32];
  __shared__ int ppeak[MW][32];  // o * MAX_PM + p
  __shared__ float4 cs[MAX_PM / 2];
  fill_cs(prm, reinterpret_cast<float*>(cs));
  __syncthreads();
  const Member& Mb = prm.mem[prm.tile_mem[(blockIdx.x * 32) / TILE]];
  BlockPoint b;
  if (!block_point(Mb, b)) return;
  const int j = b.j, lane = b.lane, w = b.w, O = prm.O, NQ = prm.P / 4;
  const int oc = b.valid ? P.oc[j] : 0;
  float sum[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) sum[i] = 0.f;
  float best = -1.f;
  int op = 0, pp = 0;
  for (int o = w; o < O; o += MW) {
    const float* T = P.TAB + tidx(prm, o, 0, j);
    const float kdk = T[T_KDK * 32], k3dk = T[T_K3DK * 32], f2_ = prm.f[o] * prm.f[o];
    const float4* r = reinterpret_cast<const float4*>(P.E + sidx(prm, o, 0, j));
    float s0 = 0.f, sc = 0.f, ss = 0.f, scc = 0.f, scs = 0.f, sss = 0.f;
#pragma unroll 3
    for (int q = 0; q < NQ; ++q) {
      const float4 e4 = r[q * 32], c4 = cs[2 * q], n4 = cs[2 * q + 1];
      const float e[4] = {e4.x, e4.y, e4.z, e4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w}, n[4] = {n4.x, n4.y, n4.z, n4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float ec = e[i] * c[i], es = e[i] * n[i];
        s0 += e[i];
        sc += ec;
        ss += es;
        scc = fmaf(ec, c[i], scc);
        scs = fmaf(ec, n[i], scs);
        sss = fmaf(es, n[i], sss);
        const float ek = e[i] * kdk;
        const int p = 4 * q + i;
        if (ek > best || (ek == best && p < pp)) { best = ek; op = o; pp = p; }
      }
    }
    sum[M0] = fmaf(s0, kdk, sum[M0]);
    sum[M2] = fmaf(f2_ * s0, kdk, sum[M2]);
    sum[M2K] = fmaf(s0, k3dk, sum[M2K]);
    sum[XC] = fmaf(sc, kdk, sum[XC]);
    sum[YC] = fmaf(ss, kdk, sum[YC]);
    if (o < oc) {
      const float ki = kdk / T[T_CP0 * 32], kg = ki * T[T_CG0 * 32];
      sum[MX] = fmaf(sc, ki, sum[MX]);
      sum[MY] = fmaf(ss, ki, sum[MY]);
      sum[CXX] = fmaf(scc, kg, sum[CXX]);
      sum[CXY] = fmaf(scs, kg, sum[CXY]);
      sum[CYY] = fmaf(sss, kg, sum[CYY]);
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) part[w][i][lane] = sum[i];
  pbest[w][lane] = best;
  ppeak[w][lane] = op * MAX_PM + pp;
  __syncthreads();
  if (w != 0 || !b.valid) return;
  for (int v = 1; v < MW; ++v) {
#pragma unroll
    for (int i = 0; i < NS; ++i) sum[i] += part[v][i][lane];
    const float bv = pbest[v][lane];
    const int ov = ppeak[v][lane] / MAX_PM, pv = ppeak[v][lane] % MAX_PM;
    if (bv > best || (bv == best && (pv < pp || (pv == pp && ov < op)))) { best = bv; op = ov; pp = pv; }
  }
  const int ja = apt(Mb, j);
  const float rw = P.rhow[ja] * prm.dthg, m0 = sum[M0], m2k = sum[M2K];
  P.mwp[j] = sqrtf(m0 / (sum[M2] + FLT_MIN));
  P.momx[j] = sum[MX] * rw; P.momy[j] = sum[MY] * rw;
  P.cgmxx[j] = sum[CXX] * rw; P.cgmxy[j] = sum[CXY] * rw; P.cgmyy[j] = sum[CYY] * rw;
  P.ht[j] = 4.f * sqrtf(m0 * prm.dth);
  P.mwd[j] = atan2f(sum[YC], sum[XC]);
  P.mss[j] = m2k * prm.dth;
  P.mwl[j] = 2.f * 3.14159274f * sqrtf(m0 / (m2k + FLT_MIN));
  P.dwd[j] = prm.th[pp];
  P.dwl[j] = 2.f * 3.14159274f / P.TAB[tidx(prm, op, T_K, j)];
  P.dwp[j] = 1.f / prm.f[op];
  const float c0 = P.TAB[tidx(prm, op, T_CP0, j)], g0 = P.TAB[tidx(prm, op, T_CG0, j)];
  P.dcp0[j] = c0; P.dcg0[j] = g0;
  const float uc = P.uc[ja], vc = P.vc[ja];
  P.dcp[j] = c0 + uc * prm.cth[pp] + vc * prm.sth[pp];
  P.dcg[j] = g0 + uc * prm.cth[pp] + vc * prm.sth[pp];
}

// stokes_drift, umwm_stokes.F90:55-128: util recomputed from k, d and cg0
// instead of stored (it would be om*im*lm floats).  The warps first share out
// the levels (direction sums times the depth-independent factors, to shared
// memory: [om][4][32]), then the depths, with the depth-dependent
// exponentials through ex2 (cosh(x) = (2^(x log2 e) + 2^(-x log2 e)) / 2, which
// has no cancellation; sinh(kd), which has, stays sinhf); the first warp then
// finds the e-folding depth from the profile ([lm][32]).
__global__ void __launch_bounds__(MW * 32) k_stokes(const Params prm, const Ptrs P) {
  extern __shared__ float sh[];
  __shared__ float4 cs[MAX_PM / 2];
  fill_cs(prm, reinterpret_cast<float*>(cs));
  __syncthreads();
  const Member& Mb = prm.mem[prm.tile_mem[(blockIdx.x * 32) / TILE]];
  BlockPoint b;
  if (!block_point(Mb, b)) return;
  const int j = b.j, lane = b.lane, w = b.w, O = prm.O, NQ = prm.P / 4, ldN = prm.ldN, lm = prm.lm;
  float* const um_s = sh + O * 128;
  const float d = P.d[j];
  const float twopi = 2.f * 3.14159274f, log2e = 1.44269504f;
  for (int o = w; o < O; o += MW) {
    const float* T = P.TAB + tidx(prm, o, 0, j);
    const float4* r = reinterpret_cast<const float4*>(P.E + sidx(prm, o, 0, j));
    float x = 0.f, y = 0.f;
#pragma unroll 3
    for (int q = 0; q < NQ; ++q) {
      const float4 e = r[q * 32], c = cs[2 * q], n = cs[2 * q + 1];
      x += e.x * c.x + e.y * c.y + e.z * c.z + e.w * c.w;
      y += e.x * n.x + e.y * n.y + e.z * n.z + e.w * n.w;
    }
    const float kk = T[T_K * 32], kd = kk * d;
    const float a = ((twopi * prm.f[o]) * (kk * kk)) * (prm.dom[o] / fabsf(T[T_CG0 * 32])) * prm.dth;
    const float s = sinhf(kd);
    float* q4 = sh + o * 128 + lane;
    q4[0] = a * x;
    q4[32] = a * y;
    q4[64] = 2.f * kk * log2e;
    q4[96] = kd > 50.f ? -1.f : 1.f / (s * s);  // -1: deep water at every depth
  }
  __syncthreads();
  for (int l = w; l < lm; l += MW) {
    const float dep = prm.depth[l];
    float su = 0.f, sv = 0.f;
    if (!(fabsf(dep) > d)) {
#pragma unroll 4
      for (int o = 0; o < O; ++o) {
        const float* q4 = sh + o * 128 + lane;
        const float k2l = q4[64], is2 = q4[96], t = k2l * (dep + d);
        // |2 k (z + d)| > 50 or k d > 50: the deep-water profile
        const bool deep = is2 < 0.f || fabsf(t) > 50.f * log2e;
        const float u = deep ? 2.f * ex2a(k2l * dep) : (0.5f * (ex2a(t) + ex2a(-t))) * is2;
        su = fmaf(u, q4[0], su);
        sv = fmaf(u, q4[32], sv);
      }
    }
    if (b.valid) {
      P.us[(size_t)l * ldN + j] = su;
      P.vs[(size_t)l * ldN + j] = sv;
    }
    um_s[l * 32 + lane] = sqrtf(su * su + sv * sv);
  }
  __syncthreads();
  if (w != 0 || !b.valid) return;
  float ds = 0.f;
  const float um1 = lm > 0 ? um_s[lane] : 0.f, ust_ef = um1 * prm.eulerinv;
  float prev = um1;
  for (int l = 1; l < lm && um1 != 0.f; ++l) {
    const float um = um_s[l * 32 + lane];
    if (um < ust_ef) {
      ds = (fabsf(prev - ust_ef) * prm.depth[l] + fabsf(um - ust_ef) * prm.depth[l - 1]) / (prev - um);
      break;
    }
    prev = um;
  }
  P.ds[j] = -ds;
}

// Reference order F(om,pm,im) (o fastest) <-> the blocked device layout, one
// CTA per 32 wet points (from `off`, which need not start a block) and four
// directions: reads of 16 bytes per point and level, rows of 4 om floats per
// point on the reference's side, turned through shared memory.
template <bool TO_REF>
__global__ void __launch_bounds__(256) k_ref(const Params prm, float* __restrict__ E, float* __restrict__ F, int off,
                                             int n) {
  extern __shared__ float tile[];  // [32][4 om + 1]
  const int O = prm.O, pitch = 4 * O + 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int j0 = blockIdx.x * 32, p = blockIdx.y * 4;
  const int cnt = min(32, n - j0);
  auto ref_side = [&](bool out) {  // a warp per point
    for (int i = w; i < cnt; i += nw) {
      float* f = F + ((size_t)(j0 + i) * prm.P + p) * O;
      for (int c = lane; c < 4 * O; c += 32) {
        if (out) f[c] = tile[i * pitch + c];
        else tile[i * pitch + c] = f[c];
      }
    }
  };
  auto dev_side = [&](bool out) {  // a warp per level, lane = point
    for (int o = w; o < O; o += nw) {
      if (lane >= cnt) continue;
      float4* e = reinterpret_cast<float4*>(E + sidx(prm, o, p, off + j0 + lane));
      float* t = tile + lane * pitch + o;
      if (out) {
        *e = make_float4(t[0], t[O], t[2 * O], t[3 * O]);
      } else {
        const float4 v = *e;
        t[0] = v.x; t[O] = v.y; t[2 * O] = v.z; t[3 * O] = v.w;
      }
    }
  };
  if (TO_REF) dev_side(false);
  else ref_side(false);
  __syncthreads();
  if (TO_REF) ref_side(true);
  else dev_side(true);
}

// The mss prefix (Ptrs::MSS) of blocks [b0, b0 + gridDim.x) from e: after a
// state was set; the propagation keeps it from then on.  A level's directions
// are added as the propagation adds them (mss_add), so that a run goes on from
// its own state, handed back, with the same bits.
__global__ void __launch_bounds__(128) k_mss(const Params prm, const Ptrs P, int b0) {
  __shared__ float v[MAX_OM * 96];
  const int blk = b0 + blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int j = blk * 32 + lane;
  for (int o = w; o < prm.O; o += nw) {
    const float4* r = reinterpret_cast<const float4*>(P.E + sidx(prm, o, 0, j));
    float2 m0 = f2(0.f), m1 = m0, m2 = m0;
    for (int q = 0; q < prm.P / 4; ++q) {
      const float4 e4 = r[q * 32];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        mss_add(h ? make_float2(e4.z, e4.w) : make_float2(e4.x, e4.y),
                make_float2(prm.dc2th[4 * q + 2 * h], prm.dc2th[4 * q + 2 * h + 1]),
                make_float2(prm.ds2th[4 * q + 2 * h], prm.ds2th[4 * q + 2 * h + 1]), m0, m1, m2);
    }
    const float hk = P.TAB[tidx(prm, o, T_K3DK, j)] * (0.5f * prm.dth);
    v[o * 96 + lane] = hk * (m0.x + m0.y);
    if (prm.ice_possible) P.ehs[((size_t)blk * prm.O + o) * 32 + lane] = P.TAB[tidx(prm, o, T_KDK, j)] * (m0.x + m0.y);
    v[o * 96 + 32 + lane] = hk * (m1.x + m1.y);
    v[o * 96 + 64 + lane] = hk * (m2.x + m2.y);
  }
  __syncthreads();
  if (w < 3) mss_prefix(prm, P, blk, w, v, 96);
}

// start of a dtg: sumt = 0 and no member done (umwm_top.F90:88)
__global__ void k_begin_dtg(const Params prm) {
  for (int m = threadIdx.x; m < prm.nmem; m += blockDim.x) {
    Ctl& c = *prm.mem[m].ctl;
    c.sumt = 0.f;
    c.done = 0;
  }
}

// stress('ocn'), umwm_stress.F90:34-214: per wet point, from the current
// spectrum and the source terms the last substep of the dtg kept (Sin, Sds
// after cothkd, Snl, and the ustar of its sdt).  A level's direction sums
// (e, e Sds, Snl and e Sin times cos th and sin th; e Sin split by the three
// form-drag classes) are formed first and weighted by the level's factors.
__global__ void __launch_bounds__(MW * 32) k_stress_ocn(const Params prm, const Ptrs P) {
  enum { TOPX, TOPY, BOTX, BOTY, SNLX, SNLY, EOX, EOY, EAX, EAY, F1X, F1Y, F2X, F2Y, F3X, F3Y, TX, TY, NS };
  __shared__ float part[MW][NS][32];
  __shared__ float4 cs[MAX_PM / 2], cw[MAX_PM / 4 * 32];
  fill_cs(prm, reinterpret_cast<float*>(cs));
  const Member& M = prm.mem[prm.tile_mem[(blockIdx.x * 32) / TILE]];
  BlockPoint b;
  if (!block_point(M, b)) return;
  const int j = b.j, lane = b.lane, w = b.w, O = prm.O, NQ = prm.P / 4;
  const int jj = b.valid ? j : M.ghost, ja = apt(M, jj), oc = b.valid ? P.oc[j] : 0;
  cw_fill(prm, P.wdir[ja], w, NQ, MW, cw);
  __syncthreads();
  const float sdtc = (prm.sdt_fac * sqrtf(P.rhorat[ja])) * P.src_ust[jj];
  float sum[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) sum[i] = 0.f;
  for (int o = w; o < O; o += MW) {
    const float* T = P.TAB + tidx(prm, o, 0, j);
    const float cp0 = T[T_CP0 * 32], icp = 1.f / cp0, kdk = T[T_KDK * 32], kk = T[T_K * 32];
    const float sdt = sdtc * kk, sdv = T[T_SDV * 32], sbf = T[T_SBF * 32];
    // downshifting weights at levels o >= 3 (1-based)
    float wm = 0.f, wl = 0.f;
    if (o >= 2) {
      const float i1 = 1.f / T[(T_CP0 - T_COUNT) * 32], i2 = 1.f / T[(T_CP0 - 2 * T_COUNT) * 32];
      wm = prm.bf1 * cp0 * i1 + prm.bf2 * cp0 * i2;
      wl = prm.bf1 * (1.f - cp0 * i1) + prm.bf2 * (1.f - cp0 * i2);
    }
    const size_t a0 = sidx(prm, o, 0, j);
    float ex = 0, ey = 0, dx = 0, dy = 0, nx = 0, ny = 0, g1x = 0, g1y = 0, g2x = 0, g2y = 0, g3x = 0, g3y = 0;
    for (int q = 0; q < NQ; ++q) {
      auto row = [&](const float* f) { return *reinterpret_cast<const float4*>(f + a0 + q * 128); };
      const float4 e4 = row(P.E), i4 = row(P.src_sin), d4 = row(P.src_sds), n4 = row(P.src_snl);
      const float4 c4 = cs[2 * q], s4 = cs[2 * q + 1], w4 = cw[q * 32 + lane];
      const float e[4] = {e4.x, e4.y, e4.z, e4.w}, si[4] = {i4.x, i4.y, i4.z, i4.w}, sd[4] = {d4.x, d4.y, d4.z, d4.w};
      const float sn[4] = {n4.x, n4.y, n4.z, n4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
      const float cwv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float ed = e[i] * sd[i], ei = e[i] * si[i];
        ex = fmaf(e[i], c[i], ex); ey = fmaf(e[i], s[i], ey);
        dx = fmaf(ed, c[i], dx); dy = fmaf(ed, s[i], dy);
        nx = fmaf(sn[i], c[i], nx); ny = fmaf(sn[i], s[i], ny);
        if (si[i] > 0.f) {
          g1x = fmaf(ei, c[i], g1x); g1y = fmaf(ei, s[i], g1y);
        } else if (cwv[i] < 0.f) {
          g2x = fmaf(ei, c[i], g2x); g2y = fmaf(ei, s[i], g2y);
        } else {
          g3x = fmaf(ei, c[i], g3x); g3y = fmaf(ei, s[i], g3y);
        }
      }
    }
    const float ux = (dx + ex * (sdt + sdv) - nx * wm) * icp, uy = (dy + ey * (sdt + sdv) - ny * wm) * icp;
    sum[TOPX] += ux * kdk; sum[TOPY] += uy * kdk;
    sum[BOTX] += ex * sbf * icp * kdk; sum[BOTY] += ey * sbf * icp * kdk;
    if (o >= 2 && o < oc) {
      sum[SNLX] += nx * wl * icp * kdk; sum[SNLY] += ny * wl * icp * kdk;
    }
    sum[EOX] += (dx - nx * wm) * kdk; sum[EOY] += (dy - ny * wm) * kdk;
    sum[EAX] += (g1x + g2x + g3x) * kdk; sum[EAY] += (g1y + g2y + g3y) * kdk;
    const float ki = icp * kdk;
    sum[F1X] += g1x * ki; sum[F1Y] += g1y * ki;
    sum[F2X] += g2x * ki; sum[F2Y] += g2y * ki;
    sum[F3X] += g3x * ki; sum[F3Y] += g3y * ki;
    if (o == O - 1) {
      sum[TX] = ux * kk;
      sum[TY] = uy * kk;
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) part[w][i][lane] = sum[i];
  __syncthreads();
  if (w != 0 || !b.valid) return;
  for (int v = 1; v < MW; ++v)
#pragma unroll
    for (int i = 0; i < NS; ++i) sum[i] += part[v][i][lane];
  const float rg = P.rhow[ja] * prm.dthg;
  const float tl = stress_tail(P.wspd[ja], P.TAB[tidx(prm, O - 1, T_K, j)]);
  const float tailx = sum[TX] * tl * rg, taily = sum[TY] * tl * rg;
  const size_t L = (size_t)prm.ldN;
  float* out = P.ocn;
  out[OCN_TAUX_TOP * L + j] = sum[TOPX] * rg + tailx + P.taux_skin[j];
  out[OCN_TAUY_TOP * L + j] = sum[TOPY] * rg + taily + P.tauy_skin[j];
  out[OCN_TAUX_BOT * L + j] = sum[BOTX] * rg;
  out[OCN_TAUY_BOT * L + j] = sum[BOTY] * rg;
  out[OCN_TAUX_SNL * L + j] = sum[SNLX] * rg;
  out[OCN_TAUY_SNL * L + j] = sum[SNLY] * rg;
  out[OCN_EPSX_OCN * L + j] = sum[EOX] * rg;
  out[OCN_EPSY_OCN * L + j] = sum[EOY] * rg;
  out[OCN_EPSX_ATM * L + j] = sum[EAX] * rg;
  out[OCN_EPSY_ATM * L + j] = sum[EAY] * rg;
  out[OCN_TAILX * L + j] = tailx;
  out[OCN_TAILY * L + j] = taily;
  out[OCN_TAUX1 * L + j] = sum[F1X] * rg;
  out[OCN_TAUY1 * L + j] = sum[F1Y] * rg;
  out[OCN_TAUX2 * L + j] = sum[F2X] * rg;
  out[OCN_TAUY2 * L + j] = sum[F2Y] * rg;
  out[OCN_TAUX3 * L + j] = sum[F3X] * rg;
  out[OCN_TAUY3 * L + j] = sum[F3Y] * rg;
}

// Graph-driven inner loop: arm before the graph launch; each substep's dts
// counts it and sets the while node's condition.
__global__ void k_loop_arm(Global* g, int budget) {
  g->budget = budget;
  g->iters = 0;
}

// Count the NaN/Inf values of a[0..n) into *count (option "check_finite").
__global__ void k_count_nonfinite(const float* __restrict__ a, size_t n, int* count) {
  int bad = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    bad += isfinite(a[i]) ? 0 : 1;
  bad = __syncthreads_count(bad > 0);
  if (threadIdx.x == 0 && bad) atomicAdd(count, bad);
}

__global__ void k_fill(float* a, size_t n, float v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) a[i] = v;
}

static int grid_for(long n, int block) {
  long g = (n + block - 1) / block;
  if (g > 152L * 32) g = 152L * 32;
  return (int)(g < 1 ? 1 : g);
}

cudaError_t launch_prep(const Params& prm, const Ptrs& P, int compute_rot, int max_nm, cudaStream_t st) {
  dim3 grid(grid_for(max_nm, 256), prm.nmem);
  k_prep<<<grid, 256, 0, st>>>(prm, P, compute_rot);
  return cudaGetLastError();
}
cudaError_t launch_diag(const Params& prm, const Ptrs& P, cudaStream_t st) {
  k_diag<<<prm.Ntot / 32, MW * 32, 0, st>>>(prm, P);
  return cudaGetLastError();
}
cudaError_t launch_stokes(const Params& prm, const Ptrs& P, cudaStream_t st) {
  // at most 64 levels x 512 + 100 depths x 128 bytes
  k_stokes<<<prm.Ntot / 32, MW * 32, (size_t)(prm.O * 128 + prm.lm * 32) * sizeof(float), st>>>(prm, P);
  return cudaGetLastError();
}
template <bool TO_REF>
static cudaError_t launch_ref(const Params& prm, float* E, float* F, int off, int n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const dim3 grid((n + 31) / 32, prm.P / 4);
  k_ref<TO_REF><<<grid, 256, (size_t)32 * (4 * prm.O + 1) * sizeof(float), st>>>(prm, E, F, off, n);
  return cudaGetLastError();
}
cudaError_t launch_to_ref(const Params& prm, const float* E, float* F, int off, int n, cudaStream_t st) {
  return launch_ref<true>(prm, const_cast<float*>(E), F, off, n, st);
}
cudaError_t launch_from_ref(const Params& prm, const float* F, float* E, int off, int n, cudaStream_t st) {
  return launch_ref<false>(prm, E, const_cast<float*>(F), off, n, st);
}
cudaError_t launch_mss(const Params& prm, const Ptrs& P, int off, int padded, cudaStream_t st) {
  k_mss<<<padded / 32, 128, 0, st>>>(prm, P, off / 32);
  return cudaGetLastError();
}
cudaError_t launch_begin_dtg(const Params& prm, cudaStream_t st) {
  k_begin_dtg<<<1, 256, 0, st>>>(prm);
  return cudaGetLastError();
}
cudaError_t launch_stress_ocn(const Params& prm, const Ptrs& P, cudaStream_t st) {
  k_stress_ocn<<<prm.Ntot / 32, MW * 32, 0, st>>>(prm, P);
  return cudaGetLastError();
}
cudaError_t launch_loop_arm(Global* g, int budget, cudaStream_t st) {
  k_loop_arm<<<1, 1, 0, st>>>(g, budget);
  return cudaGetLastError();
}
cudaError_t launch_count_nonfinite(const float* a, size_t n, int* count, cudaStream_t st) {
  k_count_nonfinite<<<grid_for((long)std::min<size_t>(n, 1u << 30), 256), 256, 0, st>>>(a, n, count);
  return cudaGetLastError();
}
cudaError_t launch_fill(float* a, size_t n, float v, cudaStream_t st) {
  k_fill<<<grid_for((long)std::min<size_t>(n, 1u << 30), 256), 256, 0, st>>>(a, n, v);
  return cudaGetLastError();
}

}  // namespace umwm
