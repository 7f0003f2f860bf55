// Device bodies of the source-term kernels (see k_source.cu for the thread
// mapping), shared by the per-stage kernels and the persistent substep kernel.
#pragma once
#include <type_traits>

#include "dev_common.cuh"

namespace umwm {

__device__ __forceinline__ float lg2a(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The inputs of a point that every level uses, and the level's factors formed
// from them and the tables.
struct SrcPoint {
  WindIn wi;
  float wdir, sdtc, sv;
  int oc;
};
__device__ __forceinline__ SrcPoint src_point(const Params& prm, const Ptrs& P, const Member& Mb, int j, bool valid) {
  SrcPoint s;
  const int jj = valid ? j : Mb.ghost, ja = apt(Mb, jj);
  const float ustar = P.ustar[jj];
  s.wi = load_wind(prm, P, jj, ja, ustar);
  s.wdir = P.wdir[ja];
  s.sdtc = (prm.sdt_fac * sqrtf(P.rhorat[ja])) * ustar;
  s.sv = prm.ice_possible ? P.sice_v[jj] : 0.f;
  s.oc = valid ? s.wi.oc : 0;  // padding points have no prognostic level
  return s;
}

// Sds of two directions, sA (1 + mss_fac chi)^2 (e k4)^sds_power
// (umwm_source_functions.F90:99-103) with the level's factors in the
// exponent: 2^(p log2 e + lsk), lsk = p log2 k4 + log2 sA; chi = A + B cos 2th + C sin 2th.
__device__ __forceinline__ float2 sds2(const Params& prm, float2 e, float2 A, float2 B, float2 C, float2 c2, float2 s2,
                                       float2 lsk) {
  const float2 chi = __ffma2_rn(C, s2, __ffma2_rn(B, c2, A));
  const float2 t = __ffma2_rn(make_float2(prm.mss_fac, prm.mss_fac), chi, make_float2(1.f, 1.f));
  const float2 x = __ffma2_rn(make_float2(prm.sds_power, prm.sds_power), make_float2(lg2a(e.x), lg2a(e.y)), lsk);
  return __fmul2_rn(__fmul2_rn(t, t), make_float2(ex2a(x.x), ex2a(x.y)));
}

// Sin of two directions (see sin_fold) with cw = cos(wdir - th).
__device__ __forceinline__ float2 sin2(const Params& prm, const WindIn& wi, float2 U, float2 ncp, float2 cw, float2 c,
                                       float2 s, float2 gl) {
  const float2 x = __ffma2_rn(f2(-wi.vc), s, __ffma2_rn(f2(-wi.uc), c, __ffma2_rn(U, cw, ncp)));
  const float2 f = make_float2(x.x > 0.f ? wi.shelt : (cw.x > 0.f ? prm.sin_neg2 : prm.sin_neg1),
                               x.y > 0.f ? wi.shelt : (cw.y > 0.f ? prm.sin_neg2 : prm.sin_neg1));
  return __fmul2_rn(__fmul2_rn(make_float2(x.x * fabsf(x.x), x.y * fabsf(x.y)), f), gl);
}

// ---- the dts pre-pass ---------------------------------------------------------
// Block blk of 32 points, lane = point; the CTA's warps share out the levels
// (independent of one another, the mss prefix being stored per level).  Only
// the prognostic levels o < oc count.  red: [warps][2][32] floats.
// TMA: the own e rows come from shared memory, staged by bulk copies into two
// buffers per warp.
template <int NP, int TMA>
__device__ __forceinline__ void phys_body(const Params& prm, const Ptrs& P, int compute_rot, int blk, uint32_t dirs,
                                          float4* cw, float* red, float* stage, uint32_t mbar) {
  constexpr int NQ = NP / 4, GQ = NQ % 3 == 0 ? 3 : 2;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const Member& Mb = prm.mem[prm.tile_mem[(blk * 32) / TILE]];
  Ctl* ctl = Mb.ctl;
  const int N = Mb.ghost;
  if (ctl->done || blk * 32 >= N) return;  // the member sits the substep out, or a block of padding
  const int j = blk * 32 + lane;
  const bool valid = j < N;
  const int jj = valid ? j : N;
  const SrcPoint s = src_point(prm, P, Mb, j, valid);
  const int OP = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(s.oc, 0));
  constexpr unsigned lstride = NP * 32, tstride = T_COUNT * 32;  // from level to level
  const size_t rb = (size_t)blk * prm.O * lstride, tb = (size_t)blk * prm.O * tstride;

  // rotation rate (umwm_advection.F90:125-139): 0.5 ((dcx sin th + dvc) odx -
  // (dcy cos th + duc) ody) = ps sin th + pc cos th + p0
  size_t tE = 0, tW = 0, tN = 0, tS = 0;
  float odx = 0.f, ody = 0.f, p0 = 0.f;
  if (compute_rot) {
    auto toff = [&](int i) { return tidx(prm, 0, T_CP0, i); };
    tE = toff(P.ie[jj]); tW = toff(P.iw[jj]); tN = toff(P.in[jj]); tS = toff(P.is[jj]);
    odx = P.oneovdx[jj]; ody = P.oneovdy[jj];
    p0 = 0.5f * ((P.vc[P.iie[jj]] - P.vc[P.iiw[jj]]) * odx - (P.uc[P.iin[jj]] - P.uc[P.iis[jj]]) * ody);
  }

  const int PFD = prm.pf_phys;
  auto pf = [&](int o) {
    if (o < OP && lane == 0) {
      bulk_prefetch_l2(P.E + o * lstride + rb, NP * 128);
      bulk_prefetch_l2(P.TAB + o * tstride + tb + T_SRC0 * 32, T_SRC_ROWS * 128);
    }
  };
  const uint32_t bar = mbar + 16u * w;
  float* const buf = TMA ? stage + (size_t)w * 2 * (NP * 32) : nullptr;
  auto issue = [&](int o, int b) {  // one lane
    if (o >= OP) return;
    adv_mbar_expect(bar + 8u * b, NP * 128);
    adv_bulk_copy(adv_smem_u32(buf + b * (NP * 32)), P.E + o * lstride + rb, NP * 128, bar + 8u * b);
  };
  if (TMA) {
    if (lane == 0) {
      adv_mbar_init(bar);
      adv_mbar_init(bar + 8u);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      issue(w, 0);
    }
    __syncwarp();
  } else {
    for (int i = 1; i < PFD; ++i) pf(w + i * nw);
  }

  cw_fill(prm, s.wdir, w, NQ, nw, cw);
  __syncthreads();
  const float4* const cwl = cw + lane;
  float mx = 0.f, rmx = 0.f;
  for (int o = w, it = 0; o < OP; o += nw, ++it) {
    if (!TMA) pf(o + PFD * nw);
    const int b = it & 1;
    if (TMA) {
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(o + nw, b ^ 1);
      }
      const bool ok = adv_mbar_wait(bar + 8u * b, (it >> 1) & 1, 4000000000LL);
      if (!__all_sync(0xffffffffu, ok)) {  // an error flag and a bounded drain of the other copy instead of a hang
        if (lane == 0) {
          atomicOr(&ctl->err, 2);
          if (o + nw < OP) adv_mbar_wait(bar + 8u * (b ^ 1), ((it + 1) >> 1) & 1, 400000000LL);
        }
        break;
      }
    }
    const float* row = TMA ? buf + b * (NP * 32) + lane * 4 : P.E + o * lstride + rb + lane * 4;
    const float* T = P.TAB + o * tstride + tb + lane;
    const float* M3 = P.MSS + ((size_t)blk * prm.O + o) * 96 + lane;
    const float kk = __ldg(T + T_K * 32), cp0 = __ldg(T + T_CP0 * 32);
    const float U = fmaf(s.wi.ustar25, __ldg(T + T_LOGL2Z * 32), s.wi.wspd);
    const float cs = __fmul_rn(__ldg(T + T_COTHKD * 32), 1.f - (__ldg(T + T_BF1R * 32) + __ldg(T + T_BF2R * 32)));
    float sink = __fadd_rn(fmaf(s.sdtc, kk, __ldg(T + T_SBF * 32)), __ldg(T + T_SDV * 32));
    if (s.sv != 0.f) sink = fmaf(-2.f * __ldg(T + T_CG0 * 32), s.sv, sink);
    const float2 A = f2(M3[0]), B = f2(M3[32]), C = f2(M3[64]);
    const float2 lsk = f2(fmaf(prm.sds_power, lg2a(pow4(kk)), lg2a(prm.twopisds_fac * prm.f[o])));
    const float2 U2 = f2(U), ncp = f2(-cp0);
    const float2 gl = f2(__fmul_rn(s.wi.c1, __ldg(T + T_FKOVG * 32))), ncs = f2(-cs), nsk = f2(-sink);
    float m = 0.f;
    // GQ quads at a time, the next ones' loads ahead of this one's arithmetic
    float4 nx[GQ];
#pragma unroll
    for (int i = 0; i < GQ; ++i) nx[i] = *reinterpret_cast<const float4*>(row + i * 128);
#pragma unroll 1
    for (int q0 = 0; q0 < NQ; q0 += GQ) {
      float4 e4[GQ];
#pragma unroll
      for (int i = 0; i < GQ; ++i) e4[i] = nx[i];
      if (q0 + GQ < NQ) {
#pragma unroll
        for (int i = 0; i < GQ; ++i) nx[i] = *reinterpret_cast<const float4*>(row + (q0 + GQ + i) * 128);
      }
#pragma unroll
      for (int i = 0; i < GQ; ++i) {
        const int q = q0 + i;
        const float4 cq = cwl[q * 32];
        const F2x2 dc = dir4(dirs, q, DIR_C), ds = dir4(dirs, q, DIR_S), dc2 = dir4(dirs, q, DIR_C2), ds2 = dir4(dirs, q, DIR_S2);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 e = h ? make_float2(e4[i].z, e4[i].w) : make_float2(e4[i].x, e4[i].y);
          const float2 sds = sds2(prm, e, A, B, C, dc2.a[h], ds2.a[h], lsk);
          const float2 si = sin2(prm, s.wi, U2, ncp, h ? make_float2(cq.z, cq.w) : make_float2(cq.x, cq.y), dc.a[h], ds.a[h], gl);
          const float2 a = __ffma2_rn(sds, ncs, __fadd2_rn(si, nsk));
          m = fmaxf(m, fmaxf(fabsf(a.x), fabsf(a.y)));
        }
      }
    }
    if (o < s.oc) mx = fmaxf(mx, m);
    if (compute_rot) {
      const float* CP = P.TAB + o * tstride;
      const float ps = 0.5f * ((__ldg(CP + tE) - __ldg(CP + tW)) * odx);
      const float pc = -0.5f * ((__ldg(CP + tN) - __ldg(CP + tS)) * ody);
      // no direction exceeds |ps| + |pc| + p0: the directions are looked at
      // only where that could raise some point's maximum
      if (__any_sync(0xffffffffu, o < s.oc && !((fabsf(ps) + fabsf(pc) + p0) * 1.0001f <= rmx))) {
        float r = 0.f;
#pragma unroll 1
        for (int q = 0; q < NQ; ++q) {
          const F2x2 dc = dir4(dirs, q, DIR_C), ds = dir4(dirs, q, DIR_S);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 v = __ffma2_rn(f2(ps), ds.a[h], __ffma2_rn(f2(pc), dc.a[h], f2(p0)));
            r = fmaxf(r, fmaxf(v.x, v.y));
          }
        }
        if (o < s.oc) rmx = fmaxf(rmx, r);
      }
    }
    if (TMA) __syncwarp();  // every lane is done with this buffer
  }
  red[w * 64 + lane] = mx;
  red[w * 64 + 32 + lane] = rmx;
  __syncthreads();
  if (w != 0) return;
  for (int i = 1; i < nw; ++i) {
    mx = fmaxf(mx, red[i * 64 + lane]);
    rmx = fmaxf(rmx, red[i * 64 + 32 + lane]);
  }
  const float ph = prm.explim / mx;
  if (valid) P.phys[j] = ph;
  float bm = valid ? ph : __int_as_float(0x7f800000);
  float rm = valid ? rmx : 0.f;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    bm = fminf(bm, __shfl_xor_sync(0xffffffffu, bm, d));
    rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, d));
  }
  if (lane == 0) {
    atomicMin(&ctl->minphys_enc, enc_ord_d(bm));
    if (compute_rot) atomicMax(&ctl->maxrot_enc, enc_ord_d(rm));
  }
}

// ---- the integration ----------------------------------------------------------
// One warp's unit of work: block blk of 32 points (lane = point), direction
// group g of D = NP/NG directions, levels [a, b).  The levels are walked
// downwards: Snl at level o needs Sds e at o+1 and o+2, which are the two
// levels before (kept in registers; a unit that does not start at the top
// forms them first).  A level's rows are copied to shared memory while the
// level before is at work: read in place, half of a warp's time went by waiting
// for them (756 -> 692 us at 305 k points, 384 -> 357 at 144 k, and 650 and 340
// with the prefetch to L2 two levels ahead; three stages instead of two give no
// more).  EARLY: the e rows go to registers at the start
// of a level (the forms of one CTA per SM: 45 us against 47 at 10 k points),
// else a quad at a time, which spills less (713 against 691).  SAVE: this
// substep also stores its source terms for stress('ocn').
template <int NP>
__host__ __device__ constexpr int integ_dirs() { return NP % 12 == 0 ? 12 : 8; }

// A level's rows, copied to shared memory during the level before: the warp's e
// rows, the tables (IT_*) and the mss prefix, two stages per warp
enum { IT_K, IT_CP0, IT_COTHKD, IT_LOGL2Z, IT_SDV, IT_FKOVG, IT_BF1R, IT_BF2R, IT_SBF, IT_CG0, IT_A, IT_B, IT_C, IT_ROWS };
template <int NP>
__host__ __device__ constexpr size_t integ_stage_floats() { return (size_t)(integ_dirs<NP>() + IT_ROWS) * 32; }
template <int NP>
__host__ __device__ constexpr size_t integ_ring_floats() { return 2 * integ_stage_floats<NP>(); }

template <int NP, bool SAVE, bool EARLY>
__device__ __forceinline__ void integ_unit(const Params& prm, const Ptrs& P, const Member& Mb, const Ctl* ctl, int blk,
                                           uint32_t dirs, float4* cw, float* ring, int g, int a, int b, bool chunked) {
  constexpr int D = integ_dirs<NP>(), DQ = D / 4;
  constexpr size_t SF = integ_stage_floats<NP>();
  const int lane = threadIdx.x & 31;
  const int O = prm.O, N = Mb.ghost;
  const int j = blk * 32 + lane;
  const bool inside = j < N;
  const bool valid = inside && (!P.fb_pt || P.fb_pt[j]);
  const SrcPoint s = src_point(prm, P, Mb, j, inside);
  if (SAVE && valid && g == 0 && a == 0) P.src_ust[j] = P.ustar[j];  // the ustar of this substep's sdt
  const float dts = ctl->dts, dtsl2 = dts * 1.44269504f;  // dts log2(e)
  cw_fill(prm, s.wdir, g * DQ, (g + 1) * DQ, 1, cw);  // own directions only: no barrier
  const float4* const cwl = cw + g * DQ * 32 + lane;
  constexpr unsigned lstride = NP * 32, tstride = T_COUNT * 32;  // from level to level
  const size_t rb = (size_t)blk * O * lstride + (size_t)g * (D * 32) + lane * 4;
  const size_t tb = (size_t)blk * O * tstride;
  const int ocw = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(s.oc, 0));  // the block's highest cut-off
  const int top = min(b + 1, O - 1);
  const uint32_t dg = dirs + (uint32_t)(g * DQ * DIR_ROWS) * 16u;  // the group's direction constants

  const int PFD = prm.pf_integ;
  auto pf = [&](int o) {
    if (o >= a && lane == 0) {
      bulk_prefetch_l2(P.E + o * lstride + rb, D * 128);
      if (g == 0) {
        bulk_prefetch_l2(P.TAB + o * tstride + tb + T_SRC0 * 32, T_SRC_ROWS * 128);
        if (!EARLY) bulk_prefetch_l2(P.MSS + ((size_t)blk * O + o) * 96, 384);
      }
    }
  };
  for (int i = 1; i < PFD; ++i) pf(top - i);

  const bool icy = __any_sync(0xffffffffu, s.sv != 0.f);
  const uint32_t rg = adv_smem_u32(ring);
  auto stage = [&](int o) {
    const uint32_t d = rg + (uint32_t)((o & 1) * SF) * 4u;
    const float* row = P.E + o * lstride + rb;
#pragma unroll
    for (int q = 0; q < DQ; ++q) copy_async16(d + q * 512 + lane * 16, row + q * 128);
    const float* T = P.TAB + o * tstride + tb + lane;
    const float* M3 = P.MSS + ((size_t)blk * prm.O + o) * 96 + lane;
    const uint32_t t = d + D * 128 + lane * 4;
    auto row4 = [&](int i, const float* src) { copy_async4(t + i * 128, src); };
    row4(IT_K, T + T_K * 32), row4(IT_CP0, T + T_CP0 * 32), row4(IT_COTHKD, T + T_COTHKD * 32);
    row4(IT_LOGL2Z, T + T_LOGL2Z * 32), row4(IT_SDV, T + T_SDV * 32), row4(IT_FKOVG, T + T_FKOVG * 32);
    row4(IT_BF1R, T + T_BF1R * 32), row4(IT_BF2R, T + T_BF2R * 32), row4(IT_SBF, T + T_SBF * 32);
    if (icy) row4(IT_CG0, T + T_CG0 * 32);
    row4(IT_A, M3), row4(IT_B, M3 + 32), row4(IT_C, M3 + 64);
    copy_async_commit();
  };
  stage(top);

  float2 d1[D / 2], d2[D / 2];  // Sds e at o+1, o+2
#pragma unroll
  for (int i = 0; i < D / 2; ++i) d1[i] = d2[i] = f2(0.f);
  for (int o = top; o >= a; --o) {
    // the levels above b - 1 are another warp's to overwrite (ef above the
    // cut-off goes to e's place): every warp of the block has read its two
    // before any writes
    if (chunked && o == b - 1) __syncthreads();
    pf(o - PFD);
    copy_async_wait<0>();  // this level's rows have landed
    const float* const sp = ring + (o & 1) * SF;
    auto erow = [&](int q) { return *reinterpret_cast<const float4*>(sp + q * 128 + lane * 4); };
    float4 e4e[DQ];
    if (EARLY) {
#pragma unroll
      for (int q = 0; q < DQ; ++q) e4e[q] = erow(q);
    }
    const float* const T = sp + D * 32 + lane;
    const float kk = T[IT_K * 32], cp0 = T[IT_CP0 * 32];
    const float coth = T[IT_COTHKD * 32];
    const float U = fmaf(s.wi.ustar25, T[IT_LOGL2Z * 32], s.wi.wspd);
    const float2 A = f2(T[IT_A * 32]), B = f2(T[IT_B * 32]), C = f2(T[IT_C * 32]);
    // (the contractions are written out: the kernels that share this body are
    // to give the same bits)
    const float k4 = pow4(kk), sdv = T[IT_SDV * 32];
    const float sA = prm.twopisds_fac * prm.f[o];
    const float2 U2 = f2(U), ncp = f2(-cp0);
    const float2 gl = f2(__fmul_rn(s.wi.c1, T[IT_FKOVG * 32]));
    const float sice = s.sv != 0.f ? __fmul_rn(2.f * T[IT_CG0 * 32], s.sv) : 0.f;
    const float sdt = __fmul_rn(s.sdtc, kk);
    const bool prog = o < s.oc, write = o < b && valid;
    float* ES = P.ES + o * lstride + rb;
    const size_t so = o * lstride + rb;
    // Sds is needed at the prognostic levels and at the two above them (Snl)
    const bool needs = SAVE || o < ocw + 2;
    const float2 lsk = f2(fmaf(prm.sds_power, lg2a(k4), lg2a(sA)));
    const float2 b1 = f2(T[IT_BF1R * 32]), b2 = f2(T[IT_BF2R * 32]);
    const float2 nsk = f2(__fsub_rn(sice, __fadd_rn(__fadd_rn(T[IT_SBF * 32], sdt), sdv)));
    // equilibrium above the cut-off, umwm_physics.F90:73-82: ef = (num / (sA t^2
    // coth))^(1/p) / k^4 as 2^((log2 num - 2 log2 t) / p + lt0)
    const float2 lt0 = f2(-fmaf(prm.inv_sds_power, lg2a(sA * coth), lg2a(k4)));
    const float2 ntail = f2(__fsub_rn(__fsub_rn(sice, sdt), sdv));
    if (o > a) stage(o - 1);
    // One quad: PR some, TL some points of the warp prognostic, above their
    // cut-off; SD: Sds is formed
    auto quad = [&](auto PR, auto TL, auto SD, int q) {
      constexpr bool pr = decltype(PR)::value, tl = decltype(TL)::value, sdn = decltype(SD)::value;
      const float4 cq = cwl[q * 32], e4 = EARLY ? e4e[q] : erow(q);
      const F2x2 dc = dir4(dg, q, DIR_C), ds = dir4(dg, q, DIR_S);
      F2x2 dc2, ds2;
      if (tl || sdn) dc2 = dir4(dg, q, DIR_C2), ds2 = dir4(dg, q, DIR_S2);
      float2 es[2], ef[2], sv1[2], sv2[2], sv3[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = 2 * q + h;
        const float2 e = h ? make_float2(e4.z, e4.w) : make_float2(e4.x, e4.y);
        const float2 cw2 = h ? make_float2(cq.z, cq.w) : make_float2(cq.x, cq.y);
        float2 sds = f2(0.f), de = f2(0.f), snl = f2(0.f);
        if (sdn) {
          sds = sds2(prm, e, A, B, C, dc2.a[h], ds2.a[h], lsk);
          de = __fmul2_rn(sds, e);
        }
        const float2 si = sin2(prm, s.wi, U2, ncp, cw2, dc.a[h], ds.a[h], gl);
        if (pr) {
          snl = __ffma2_rn(f2(-prm.snl_fac), de, __ffma2_rn(b2, d2[i], __fmul2_rn(b1, d1[i])));
          // the level's sinks summed once: S = Sin - Sds coth - (sbf + sdt + sdv - sice)
          const float2 S = __fadd2_rn(__ffma2_rn(sds, f2(-coth), si), nsk);
          const float2 x = __fmul2_rn(f2(dtsl2), S);
          ef[h] = __ffma2_rn(e, make_float2(ex2a(x.x), ex2a(x.y)), __fmul2_rn(f2(dts), snl));
        }
        const float2 sp = make_float2(fmaxf(si.x, 0.f), fmaxf(si.y, 0.f));
        if (tl) {
          const float2 num = __fadd2_rn(sp, ntail);
          const float2 chi = __ffma2_rn(C, ds2.a[h], __ffma2_rn(B, dc2.a[h], A));
          const float2 t = __ffma2_rn(f2(prm.mss_fac), chi, f2(1.f));
          const float2 x = __ffma2_rn(f2(prm.inv_sds_power),
                                      __ffma2_rn(f2(-2.f), make_float2(lg2a(t.x), lg2a(t.y)),
                                                 make_float2(lg2a(num.x), lg2a(num.y))), lt0);
          const float2 et = make_float2(num.x >= 0.f ? ex2a(x.x) : 0.f, num.y >= 0.f ? ex2a(x.y) : 0.f);
          ef[h] = pr ? make_float2(prog ? ef[h].x : et.x, prog ? ef[h].y : et.y) : et;
        }
        es[h] = __fmul2_rn(f2(0.5f), __fadd2_rn(e, ef[h]));
        if (SAVE) {
          sv1[h] = prog ? si : sp;
          sv2[h] = __fmul2_rn(sds, f2(coth));
          sv3[h] = prog ? snl : f2(0.f);  // zero above the cut-off
        }
        d2[i] = d1[i];
        d1[i] = de;
      }
      if (write) {
        *reinterpret_cast<float4*>(ES + q * 128) = make_float4(es[0].x, es[0].y, es[1].x, es[1].y);
        // above the cut-off ef goes to e's place; below it e stays and the
        // propagation forms ef = 2 E* - e
        if (tl && !(pr && prog))
          *reinterpret_cast<float4*>(P.EF + so + q * 128) = make_float4(ef[0].x, ef[0].y, ef[1].x, ef[1].y);
        if (SAVE) {
          *reinterpret_cast<float4*>(P.src_sin + so + q * 128) = make_float4(sv1[0].x, sv1[0].y, sv1[1].x, sv1[1].y);
          *reinterpret_cast<float4*>(P.src_sds + so + q * 128) = make_float4(sv2[0].x, sv2[0].y, sv2[1].x, sv2[1].y);
          *reinterpret_cast<float4*>(P.src_snl + so + q * 128) = make_float4(sv3[0].x, sv3[0].y, sv3[1].x, sv3[1].y);
        }
      }
    };
    // (the branches are on the warp's points together: most levels are below
    // every point's cut-off or above)
    using Y = std::true_type;
    using Nn = std::false_type;
    const bool anyp = __any_sync(0xffffffffu, prog), anyt = !__all_sync(0xffffffffu, prog);
    if (!anyt) {
#pragma unroll
      for (int q = 0; q < DQ; ++q) quad(Y{}, Nn{}, Y{}, q);
    } else if (anyp) {
#pragma unroll
      for (int q = 0; q < DQ; ++q) quad(Y{}, Y{}, Y{}, q);
    } else if (needs) {
#pragma unroll
      for (int q = 0; q < DQ; ++q) quad(Nn{}, Y{}, Y{}, q);
    } else {
#pragma unroll
      for (int q = 0; q < DQ; ++q) quad(Nn{}, Y{}, Nn{}, q);
    }
  }
}

// Warp `w` of block blk's NG x nc warps: direction group fastest (a block's
// tables are then shared through L1), then level chunk.  A CTA (or, with
// nc = 1, any warp) runs it; with nc > 1 every warp of the CTA belongs to the
// one block.  cw: NP/4 x 32 float4 of this chunk's warps; ring: integ_ring_floats
// of this warp.
template <int NP, bool EARLY>
__device__ __forceinline__ void integ_body(const Params& prm, const Ptrs& P, uint32_t dirs, float4* cw, float* ring, int blk, int w,
                                           int nc) {
  constexpr int NG = NP / integ_dirs<NP>();
  const int g = w % NG, c = w / NG;
  const int tile = (blk * 32) / TILE;
  const Member& Mb = prm.mem[prm.tile_mem[tile]];
  const Ctl* ctl = Mb.ctl;
  // members that have finished the current dtg sit the substep out
  if (!ctl->running || blk * 32 >= Mb.ghost) return;
  if (P.fb_tile && !P.fb_tile[tile]) return;  // surrogate fallback: flagged tiles only
  const int a = prm.O * c / nc, b = prm.O * (c + 1) / nc;
  // the last substep of a step that computes stress('ocn') or writes output
  // keeps its source terms, and so does the model's first substep (its
  // spectrum output)
  if (P.src_sin && (ctl->done || ctl->first) && P.glob->save_src)
    integ_unit<NP, true, EARLY>(prm, P, Mb, ctl, blk, dirs, cw, ring, g, a, b, nc > 1);
  else
    integ_unit<NP, false, EARLY>(prm, P, Mb, ctl, blk, dirs, cw, ring, g, a, b, nc > 1);
}

}  // namespace umwm
