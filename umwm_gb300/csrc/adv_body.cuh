// Device body of the propagation/refraction/stress kernel (see k_advect.cu),
// shared by the per-stage kernel and the persistent substep kernel.
#pragma once
#include "dev_common.cuh"

namespace umwm {

// The levels' sums of a CTA's 32 points: per level x and y of the form-stress
// integrand times k dk and the three mss sums, and the top level's stress sums
// without k dk: [om][5][32] + [2][32] floats of dynamic shared memory.
__host__ __device__ constexpr size_t adv_red_floats(int om) { return (size_t)(5 * om + 2) * 32; }

// Rows in flight: each warp copies the rows of ADV_S - 1 quads ahead of the
// one it works on into shared memory (cp.async, each lane its own point's), a
// ring of ADV_S slots of six rows (E* of the point and its four neighbours, e),
// and as many rows through which the warp's points pass one another their E*:
// a north or south neighbour is mostly the next point of the same block, and
// only the others are copied.  ADV_S divides the row's quads, so that a quad's
// slot is a constant.
template <int NP>
__host__ __device__ constexpr int adv_stages() { return (NP / 4) % 3 == 0 ? 3 : 2; }
template <int NP>
__host__ __device__ constexpr size_t adv_ring_floats() { return (size_t)adv_stages<NP>() * 7 * 128; }  // per warp

template <bool COH>
__device__ __forceinline__ void adv_copy16(uint32_t dst, const float* src) {
  if (COH) copy_async16(dst, src);
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float4 adv_lds(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}

__device__ __forceinline__ void adv_sts(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// The body of k_advect for the 32-point block `blk` (the kernel's block
// index, or a persistent CTA's current block).  Lane = point; each of the
// CTA's warps takes every nw-th frequency level and walks its whole direction
// row, four directions at a time.  CNT: also count the bins whose negative ef
// is cut to 0 (option "count_cut"; a separate instance so that the plain one
// carries no counter).  COH: E* is read through L2 only, for a persistent
// kernel in which the same launch wrote it.  red, ring: shared memory (adv_red_floats, adv_ring_floats per warp).
template <int NP, bool CURV, bool CNT, bool COH, bool AHEAD>
__device__ __forceinline__ void advect_body(const Params& prm, const Ptrs& P, int blk, uint32_t dirs, float4* cw,
                                            float* red, float* ring) {
  constexpr int NQ = NP / 4, S = adv_stages<NP>();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int O = prm.O;
  const Member& Mb = prm.mem[prm.tile_mem[(blk * 32) / TILE]];
  const Ctl* ctl = Mb.ctl;
  const int N = Mb.ghost;
  // the member has finished the current dtg, or the block is all padding
  if (!ctl->running || blk * 32 >= N) return;
  const int j = blk * 32 + lane;
  const bool valid = j < N;
  const int jj = valid ? j : N;
  const int ja = apt(Mb, jj);

  const float dta = ctl->dta, dtr = ctl->dtr;
  const bool zerocur = ctl->zerocurrents != 0;
  const int ie = P.ie[jj], iw = P.iw[jj], in = P.in[jj], is = P.is[jj];
  const int oc = valid ? P.oc[jj] : 0, ocr = P.oc_rot[jj];
  const bool ice = P.fice[ja] > prm.fice_uth;
  const float oneovar = P.oneovar[jj], dxn = P.dxn[jj], dxs = P.dxs[jj], dye = P.dye[jj], dyw = P.dyw[jj];
  const float odx = P.oneovdx[jj], ody = P.oneovdy[jj];
  const float ustar = P.ustar[jj];
  const WindIn wi = load_wind(prm, P, jj, ja, ustar);
  const float wdir = P.wdir[ja];
  cw_fill(prm, wdir, w, NQ, nw, cw);
  __syncthreads();
  const float4* const cwl = cw + lane;

  // current advection, umwm_advection.F90:62-82, folded per point into five
  // coefficients of E* at the point and its neighbours
  float F0 = 0.f, kE = 0.f, kW = 0.f, kN = 0.f, kS = 0.f;
  const float uci = wi.uc, vci = wi.vc;
  const float ucn = P.uc[P.iin[jj]], ucs = P.uc[P.iis[jj]];
  const float vce = P.vc[P.iie[jj]], vcw = P.vc[P.iiw[jj]];
  if (!zerocur) {
    const float uce = P.uc[P.iie[jj]], ucw = P.uc[P.iiw[jj]], vcn = P.vc[P.iin[jj]], vcs = P.vc[P.iis[jj]];
    const float ue = uci + uce, uw = uci + ucw, vn = vci + vcn, vs = vci + vcs;
    const float feup = (ue + fabsf(ue)) * dye, fwdn = (uw - fabsf(uw)) * dyw;
    const float fnup = (vn + fabsf(vn)) * dxn, fsdn = (vs - fabsf(vs)) * dxs;
    kE = (ue - fabsf(ue)) * dye; kW = -(uw + fabsf(uw)) * dyw;
    kN = (vn - fabsf(vn)) * dxn; kS = -(vs + fabsf(vs)) * dxs;
    F0 = feup - fwdn + fnup - fsdn;
  }
  // A neighbour's row is read where a direction of the four is upwind of it,
  // and where some lane's current blows from it
  const bool uE = CURV || __any_sync(0xffffffffu, kE != 0.f), uW = CURV || __any_sync(0xffffffffu, kW != 0.f);
  const bool uN = CURV || __any_sync(0xffffffffu, kN != 0.f), uS = CURV || __any_sync(0xffffffffu, kS != 0.f);
  const float c0 = (0.5f * (vce - vcw)) * odx - (0.5f * (ucn - ucs)) * ody;
  const float ccv = CURV ? cosf(P.curv[jj]) : 1.f, scv = CURV ? sinf(P.curv[jj]) : 0.f;

  // rows of the point and its neighbours at level 0; from level to level a
  // block's rows are lstride apart
  constexpr unsigned lstride = NP * 32, tstride = T_COUNT * 32;
  auto off = [&](int i) { return sidx(prm, 0, 0, i); };
  const size_t rb = (size_t)blk * O * lstride, tb = (size_t)blk * O * tstride;
  const float *const nE = P.ES + off(ie), *const nW = P.ES + off(iw), *const nN = P.ES + off(in), *const nS = P.ES + off(is);
  const float *const tO = P.TAB + tidx(prm, 0, 0, j);
  const float *const tE = P.TAB + tidx(prm, 0, 0, ie), *const tW = P.TAB + tidx(prm, 0, 0, iw);
  const float *const tN = P.TAB + tidx(prm, 0, 0, in), *const tS = P.TAB + tidx(prm, 0, 0, is);
  // stress_vector_integral divides by cp0 of the previous unrolled point
  // (assumed-shape dummy with lower bound 1 over cp0(:,0:im)),
  // umwm_stress.F90:401, :495-513; the member's first point uses its ghost
  const int jprev = (jj == Mb.off || jj >= N) ? N : jj - 1;
  const float* const tV = P.TAB + tidx(prm, 0, T_CP0, jprev);
  const float dtaq = 0.25f * dta * oneovar;
  const float dtrq = dtr * prm.oneovdth;
  const int ocw = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(oc, 0));
  unsigned ncut = 0;  // bins of this lane whose negative ef was cut (CNT)

  // the block's E*, e and table rows prm.pf_adv of this warp's levels ahead
  // go to L2 in the background (E* is read only below the block's highest
  // cut-off)
  const int PFD = prm.pf_adv;
  auto pf = [&](int o) {
    if (o < O && lane == 0) {
      const size_t b = rb + o * lstride;
      if (o < ocw) bulk_prefetch_l2(P.ES + b, NP * 128);
      bulk_prefetch_l2(P.EF + b, NP * 128);
      bulk_prefetch_l2(P.TAB + tb + o * tstride, T_ADV_ROWS * 128);
    }
  };
  for (int i = 1; i < PFD; ++i) pf(w + i * nw);

  // copies of quad q of level o into its slot: the point's e and neighbours'
  // E*, and the point's E* one quad on (the refraction looks one direction
  // ahead; after the last quad, the first of this warp's next level)
  const uint32_t rg = adv_smem_u32(ring + w * adv_ring_floats<NP>()) + lane * 16;
  const uint32_t xg = rg + S * 3072u;  // the exchanged rows
  // north and south neighbours in this block: where their E* is exchanged
  const bool bN = (in >> 5) == blk, bS = (is >> 5) == blk;
  const uint32_t aN = bN ? xg + (uint32_t)((in & 31) - lane) * 16u : rg + 2048u;
  const uint32_t aS = bS ? xg + (uint32_t)((is & 31) - lane) * 16u : rg + 2560u;
  const uint32_t dN = bN ? 512u : 3072u, dS = bS ? 512u : 3072u;  // from slot to slot
  const size_t ro = rb + lane * 4;
  auto issue = [&](int o, int q) {
    const uint32_t d = rg + (uint32_t)(q % S) * 3072u;
    const unsigned a = o * lstride + q * 128;
    if (o < O) {
      constexpr int H = NP / 2;
      const int p = 4 * q;
      adv_copy16<COH>(d + 512, P.EF + ro + a);
      if (o < ocw) {
        if (CURV || p < H / 2 || p + 3 >= H + H / 2 || uE) adv_copy16<COH>(d + 1024, nE + a);
        if (CURV || (p + 3 >= H / 2 && p < H + H / 2) || uW) adv_copy16<COH>(d + 1536, nW + a);
        if ((CURV || p < H || uN) && !bN) adv_copy16<COH>(d + 2048, nN + a);
        if ((CURV || p + 3 >= H || uS) && !bS) adv_copy16<COH>(d + 2560, nS + a);
        if (q + 1 < NQ) adv_copy16<COH>(d, P.ES + ro + a + 128);
        else if (o + nw < ocw) adv_copy16<COH>(d, P.ES + ro + (o + nw) * lstride);
      }
    }
    copy_async_commit();
  };
  auto lde = [](const float* a) { return COH ? __ldcg(a) : __ldg(a); };
#pragma unroll
  for (int i = 0; i < S - 1; ++i) issue(w, i);
  float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);  // E* of the quad at hand
  float elast = 0.f;                             // E* of the level's last direction
  if (w < ocw) {
    const float* r = P.ES + ro + w * lstride;
    cur = COH ? __ldcg(reinterpret_cast<const float4*>(r)) : __ldg(reinterpret_cast<const float4*>(r));
    elast = lde(r + poff(NP - 1));
  }

  // AHEAD: a level's table values, read during the last quad of the level
  // before (their latency was a sixth of the kernel's stalls: 1176 -> 1152 us
  // at 305 k points, 511 -> 498 at 144 k); the forms of 128 registers read
  // them in place, since the 15 registers would spill there
  struct { float cp0, kdk, fkovg, k3, l2z, cpv, cg, cgE, cgW, cgN, cgS, cpE, cpW, cpN, cpS; } T;
  auto tab = [&](int o) {
    if (o >= O) return;
    const unsigned to = o * tstride;
    T.cp0 = __ldg(tO + to + T_CP0 * 32), T.kdk = __ldg(tO + to + T_KDK * 32);
    T.fkovg = __ldg(tO + to + T_FKOVG * 32), T.k3 = __ldg(tO + to + T_K3DK * 32);
    T.l2z = __ldg(tO + to + T_LOGL2Z * 32), T.cpv = __ldg(tV + to);
    if (o < ocw) {
      T.cg = __ldg(tO + to + T_CG0 * 32);
      T.cgE = __ldg(tE + to + T_CG0 * 32), T.cgW = __ldg(tW + to + T_CG0 * 32);
      T.cgN = __ldg(tN + to + T_CG0 * 32), T.cgS = __ldg(tS + to + T_CG0 * 32);
      T.cpE = __ldg(tE + to + T_CP0 * 32), T.cpW = __ldg(tW + to + T_CP0 * 32);
      T.cpN = __ldg(tN + to + T_CP0 * 32), T.cpS = __ldg(tS + to + T_CP0 * 32);
    }
  };
  if (AHEAD) tab(w);
  for (int o = w; o < O; o += nw) {
    pf(o + PFD * nw);
    const unsigned lo = o * lstride, to = o * tstride;
    auto tv = [&](float ahead, const float* t) { return AHEAD ? ahead : __ldg(t + to); };
    float* const Eo = P.E + ro + lo;
    const bool prog = o < oc, refr = prog && o < ocr;
    const bool anyp = o < ocw, anyr = __any_sync(0xffffffffu, refr);
    const float cp0 = tv(T.cp0, tO + T_CP0 * 32), kdk = tv(T.kdk, tO + T_KDK * 32);
    const float fkovg = tv(T.fkovg, tO + T_FKOVG * 32), hk = tv(T.k3, tO + T_K3DK * 32) * (0.5f * prm.dth);
    const float U = fmaf(wi.ustar25, tv(T.l2z, tO + T_LOGL2Z * 32), wi.wspd);
    const float icp = 1.f / tv(T.cpv, tV);
    const float2 U2 = f2(U), ncp = f2(-cp0), nuc = f2(-uci), nvc = f2(-vci);
    // above the cut-off Sin is cut at 0 (the NaN-keeping maximum with -inf keeps it below)
    const float slo = prog ? __int_as_float(0xff800000) : 0.f;
    float DE = 0.f, DW = 0.f, DN = 0.f, DS = 0.f, alc = 0.f, bec = 0.f;
    if (anyp) {
      const float cgi = tv(T.cg, tO + T_CG0 * 32);
      DE = 2.f * (cgi + tv(T.cgE, tE + T_CG0 * 32)) * dye;
      DW = 2.f * (cgi + tv(T.cgW, tW + T_CG0 * 32)) * dyw;
      DN = 2.f * (cgi + tv(T.cgN, tN + T_CG0 * 32)) * dxn;
      DS = 2.f * (cgi + tv(T.cgS, tS + T_CG0 * 32)) * dxs;
    }
    if (anyr) {
      const float gx = 0.5f * (tv(T.cpE, tE + T_CP0 * 32) - tv(T.cpW, tW + T_CP0 * 32));
      const float gy = 0.5f * (tv(T.cpN, tN + T_CP0 * 32) - tv(T.cpS, tS + T_CP0 * 32));
      alc = gx * odx;
      bec = -(gy * ody);
    }
    // the rotation rate of the edge between directions p and p + 1 (the mean of
    // the two directions' rates, from the edge's mean sin and cos) and the flux
    // through it, max(rl, 0) e(p) + min(rl, 0) e(p+1) = rl e(upwind side);
    // each direction takes F(p) - F(p-1)
    const float2 al2 = make_float2(alc, alc), be2 = make_float2(bec, bec), c02 = make_float2(c0, c0);
    const float dtl = refr ? -dtrq : 0.f;
    float fprev = 0.f, efirst;  // flux of the edge before direction 0, E* of direction 0
    float2 tx2 = make_float2(0.f, 0.f), ty2 = tx2, m0 = tx2, m1 = tx2, m2 = tx2;
    efirst = cur.x;
    if (anyr) {
      const float rl = fmaf(alc, prm.shs[NP - 1], fmaf(bec, prm.chs[NP - 1], c0));
      fprev = rl * (rl > 0.f ? elast : efirst);
    }
    if (o + nw < ocw) elast = lde(P.ES + ro + lo + nw * lstride + poff(NP - 1));  // the next level's
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int p = 4 * q;
      if (AHEAD && q + 1 == NQ) tab(o + nw);
      copy_async_wait<S - 2>();  // this quad's rows have landed
      const uint32_t d = rg + (uint32_t)(q % S) * 3072u;
      float4 ef4 = adv_lds(d + 512);  // e below the cut-off, ef above
      float2 ef[2] = {make_float2(ef4.x, ef4.y), make_float2(ef4.z, ef4.w)};
      const F2x2 dc = dir4(dirs, q, DIR_C), ds = dir4(dirs, q, DIR_S);
      float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
      if (anyp) {
        // th(p) = (p - (pm + 1) / 2) dth: sin th < 0 for p < pm/2, cos th < 0
        // for p < pm/4 and p >= 3 pm/4 (setup_params checks it)
        constexpr int H = NP / 2;
        const bool qE = CURV || p < H / 2 || p + 3 >= H + H / 2, qW = CURV || (p + 3 >= H / 2 && p < H + H / 2);
        const bool qN = CURV || p < H, qS = CURV || p + 3 >= H;
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 fe = (qE || uE) ? adv_lds(d + 1024) : z4, fw = (qW || uW) ? adv_lds(d + 1536) : z4;
        adv_sts(xg + (q % S) * 512u, cur);
        __syncwarp();  // (three slots, or two with an even row: a slot is rewritten two barriers on)
        const float4 fn = (qN || uN) ? adv_lds(aN + (q % S) * dN) : z4, fs = (qS || uS) ? adv_lds(aS + (q % S) * dS) : z4;
        nxt = adv_lds(d);
        const float enext = q + 1 < NQ ? nxt.x : efirst;
        const F2x2 dsh = dir4(dirs, q, DIR_SH), dch = dir4(dirs, q, DIR_CH);
        const float2 es[2] = {make_float2(cur.x, cur.y), make_float2(cur.z, cur.w)};
        const float2 er[2] = {make_float2(cur.y, cur.z), make_float2(cur.w, enext)};
        const float2 ee[2] = {make_float2(fe.x, fe.y), make_float2(fe.z, fe.w)};
        const float2 ew[2] = {make_float2(fw.x, fw.y), make_float2(fw.z, fw.w)};
        const float2 en[2] = {make_float2(fn.x, fn.y), make_float2(fn.z, fn.w)};
        const float2 eS[2] = {make_float2(fs.x, fs.y), make_float2(fs.z, fs.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = p + 2 * h;
          // ef = 2 E* - e (the integration left e in place and wrote E* = (e + ef)/2)
          float2 r = __ffma2_rn(ef[h], f2(-1.f), __fadd2_rn(es[h], es[h]));
          // ---- propagation, umwm_advection.F90:30-97: one upwind side per
          // direction and axis, cos th (D_E e_E - D_W e0) where cos th < 0,
          // cos th (D_E e0 - D_W e_W) where > 0, the same for sin th, N and S
          float2 f;
          const float2 c = dc.a[h], s = ds.a[h];
          if constexpr (!CURV) {
            auto cneg = [&](int p_) { return p_ < H / 2 || p_ >= H + H / 2; };
            const float2 ea = make_float2(cneg(k) ? ee[h].x : es[h].x, cneg(k + 1) ? ee[h].y : es[h].y);
            const float2 eb = make_float2(cneg(k) ? es[h].x : ew[h].x, cneg(k + 1) ? es[h].y : ew[h].y);
            const float2 na = make_float2(k < H ? en[h].x : es[h].x, k + 1 < H ? en[h].y : es[h].y);
            const float2 nb = make_float2(k < H ? es[h].x : eS[h].x, k + 1 < H ? es[h].y : eS[h].y);
            const float2 u = __ffma2_rn(make_float2(-DW, -DW), eb, __fmul2_rn(make_float2(DE, DE), ea));
            const float2 v = __ffma2_rn(make_float2(-DS, -DS), nb, __fmul2_rn(make_float2(DN, DN), na));
            f = __ffma2_rn(s, v, __fmul2_rn(c, u));
          } else {  // curvilinear: the directions turned by the grid's curvature
            const float2 cv = make_float2(ccv, ccv), sv = make_float2(scv, scv);
            const float2 cc = __ffma2_rn(make_float2(-scv, -scv), s, __fmul2_rn(cv, c));
            const float2 sc = __ffma2_rn(sv, c, __fmul2_rn(cv, s));
            const float2 cp = make_float2(fmaxf(cc.x, 0.f), fmaxf(cc.y, 0.f)), cm = make_float2(fminf(cc.x, 0.f), fminf(cc.y, 0.f));
            const float2 sp = make_float2(fmaxf(sc.x, 0.f), fmaxf(sc.y, 0.f)), sm = make_float2(fminf(sc.x, 0.f), fminf(sc.y, 0.f));
            f = __fmul2_rn(make_float2(DE, DE), __ffma2_rn(cm, ee[h], __fmul2_rn(cp, es[h])));
            f = __ffma2_rn(make_float2(-DW, -DW), __ffma2_rn(cm, es[h], __fmul2_rn(cp, ew[h])), f);
            f = __ffma2_rn(make_float2(DN, DN), __ffma2_rn(sm, en[h], __fmul2_rn(sp, es[h])), f);
            f = __ffma2_rn(make_float2(-DS, -DS), __ffma2_rn(sm, es[h], __fmul2_rn(sp, eS[h])), f);
          }
          if (!zerocur) {
            f = __ffma2_rn(make_float2(F0, F0), es[h], f);
            f = __ffma2_rn(make_float2(kE, kE), ee[h], f);
            f = __ffma2_rn(make_float2(kW, kW), ew[h], f);
            f = __ffma2_rn(make_float2(kN, kN), en[h], f);
            f = __ffma2_rn(make_float2(kS, kS), eS[h], f);
          }
          r = __ffma2_rn(make_float2(-dtaq, -dtaq), f, r);
          // ---- refraction, umwm_advection.F90:122-178
          if (anyr) {
            const float2 rl = __ffma2_rn(al2, dsh.a[h], __ffma2_rn(be2, dch.a[h], c02));
            const float2 up = make_float2(rl.x > 0.f ? es[h].x : er[h].x, rl.y > 0.f ? es[h].y : er[h].y);
            const float2 fk = __fmul2_rn(rl, up);
            const float2 d = __ffma2_rn(make_float2(fprev, fk.x), f2(-1.f), fk);
            r = __ffma2_rn(make_float2(dtl, dtl), d, r);
            fprev = fk.y;
          }
          // sea ice above fice_uth: propagation and refraction leave ef = 0
          // (umwm_advection.F90:89-97, :170-178)
          if (ice) r = make_float2(0.f, 0.f);
          if (prog) ef[h] = r;
        }
      }
      // the slot before this one is free: the rows of S - 1 quads on
      if (q + S - 1 < NQ) issue(o, q + S - 1);
      else issue(o + nw, q + S - 1 - NQ);
      cur = nxt;
      // ---- e = ef with negatives cut to 0 (NaN stays NaN): the explicit Snl
      // term can leave a tiny negative ef, and a negative e makes the next
      // step's (e k^4)^sds_power NaN (the oracle cuts them at the same point)
      if (CNT) ncut += valid ? (ef[0].x < 0.f) + (ef[0].y < 0.f) + (ef[1].x < 0.f) + (ef[1].y < 0.f) : 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) ef[h] = make_float2(max_nan0(ef[h].x), max_nan0(ef[h].y));
      // above the cut-off e = ef is in place (EF aliases E)
      if (prog) *reinterpret_cast<float4*>(Eo + q * 128) = make_float4(ef[0].x, ef[0].y, ef[1].x, ef[1].y);
      const F2x2 dc2 = dir4(dirs, q, DIR_C2), ds2 = dir4(dirs, q, DIR_S2);
      const float4 cq = cwl[q * 32];
      // ---- the form-stress integrand with the new spectrum.  Sin without the
      // level's factor gl = c1 fkovg (>= 0), which multiplies the level's sums
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 c = dc.a[h], s = ds.a[h];
        const float2 cv = h ? make_float2(cq.z, cq.w) : make_float2(cq.x, cq.y);
        const float2 x = __ffma2_rn(nvc, s, __ffma2_rn(nuc, c, __ffma2_rn(U2, cv, ncp)));
        const float2 a = make_float2(x.x * fabsf(x.x), x.y * fabsf(x.y));
        const float2 g = make_float2(x.x > 0.f ? wi.shelt : (cv.x > 0.f ? prm.sin_neg2 : prm.sin_neg1),
                                     x.y > 0.f ? wi.shelt : (cv.y > 0.f ? prm.sin_neg2 : prm.sin_neg1));
        float2 sd = __fmul2_rn(a, g);
        sd = make_float2(max_nan(sd.x, slo), max_nan(sd.y, slo));
        const float2 es2 = __fmul2_rn(ef[h], sd);
        tx2 = __ffma2_rn(es2, c, tx2);
        ty2 = __ffma2_rn(es2, s, ty2);
        // the mss sums of the new spectrum (the source terms' prefix)
        mss_add(ef[h], dc2.a[h], ds2.a[h], m0, m1, m2);
      }
    }
    const float lf = icp * (wi.c1 * fkovg);
    const float tx = (tx2.x + tx2.y) * lf, ty = (ty2.x + ty2.y) * lf;
    float* rl_ = red + (size_t)o * 160 + lane;
    rl_[0] = tx * kdk;
    rl_[32] = ty * kdk;
    rl_[64] = hk * (m0.x + m0.y);
    if (prm.ice_possible) P.ehs[((size_t)blk * O + o) * 32 + lane] = kdk * (m0.x + m0.y);
    rl_[96] = hk * (m1.x + m1.y);
    rl_[128] = hk * (m2.x + m2.y);
    if (o == O - 1) {
      red[(size_t)O * 160 + lane] = tx;
      red[(size_t)O * 160 + 32 + lane] = ty;
    }
  }
  if (CNT) {
    const unsigned c = __reduce_add_sync(0xffffffffu, ncut);
    if (lane == 0 && c) atomicAdd(&P.glob->cut_count, (unsigned long long)c);
  }
  __syncthreads();
  if (w >= 1 && w <= 3) {  // the mss prefix of one of the three sums
    mss_prefix(prm, P, blk, w - 1, red + 64, 160);
    return;
  }
  if (w != 0 || !valid) return;
  // the sums over the levels, in their order whatever the number of warps
  float sx = 0.f, sy = 0.f, dsx = 0.f, dsy = 0.f;
#pragma unroll 4
  for (int o = 0; o < O; ++o) {
    const float tx = red[(size_t)o * 160 + lane], ty = red[(size_t)o * 160 + 32 + lane];
    sx += tx;
    sy += ty;
    if (o >= oc - 1) {
      dsx += tx;
      dsy += ty;
    }
  }
  const float txom = red[(size_t)O * 160 + lane], tyom = red[(size_t)O * 160 + 32 + lane];
  // ---- stress('atm') per point, umwm_stress.F90:216-262
  const float rhow = P.rhow[ja], rhoa = P.rhoa[ja], wspd = wi.wspd;
  const float kom = __ldg(tO + (O - 1) * tstride + T_K * 32);
  const float tl = stress_tail(wspd, kom);
  const float tax = txom * kom * tl * rhow * prm.dthg;
  const float tay = tyom * kom * tl * rhow * prm.dthg;
  const float tfx = sx * rhow * prm.dthg + tax;
  const float tfy = sy * rhow * prm.dthg + tay;
  P.tailatmx[j] = tax; P.tailatmy[j] = tay;
  P.taux_form[j] = tfx; P.tauy_form[j] = tfy;
  P.taux_diag[j] = dsx * rhow * prm.dthg;
  P.tauy_diag[j] = dsy * rhow * prm.dthg;
  const float us1 = prm.lm > 0 ? P.us[j] : 0.f, vs1 = prm.lm > 0 ? P.vs[j] : 0.f;
  const float urel = wspd * cosf(wdir) - (uci + us1);
  const float vrel = wspd * sinf(wdir) - (vci + vs1);
  const float wrel = sqrtf(urel * urel + vrel * vrel);
  const float drel = atan2f(vrel, urel);
  const float cdf = sqrtf(tfx * tfx + tfy * tfy) / (rhoa * (wspd * wspd));
  float z0 = 1e-3f, usk = 0.f;
  for (int n = 0; n < 6; ++n) {  // friction_velocity_skin, :275-298
    usk = prm.kappa * wrel / logf(prm.z / z0);
    z0 = 0.132f * prm.nu_air / usk;
  }
  float cds = (usk * usk) / (wspd * wspd);
  cds = cds * (1.f + 2.f * cds / (cds + cdf + 1.17549435e-38f)) / 3.f;
  if (cds > 1e-2f) cds = 1e-2f;
  const float tsx = rhoa * cds * (wrel * wrel) * cosf(drel);
  const float tsy = rhoa * cds * (wrel * wrel) * sinf(drel);
  P.taux_skin[j] = tsx; P.tauy_skin[j] = tsy;
  const float tx = tfx + tsx, ty = tfy + tsy;
  P.taux[j] = tx; P.tauy[j] = ty;
  const float tm = sqrtf(tx * tx + ty * ty);
  P.cd[j] = tm / (rhoa * (wspd * wspd));
  P.ustar[j] = sqrtf(tm / rhoa);
}

}  // namespace umwm
