// Device-side definitions shared by the GB300 UMWM kernels.
//
// One model is an ensemble of members (a single domain is a one-member
// ensemble).  Member m owns the wet indices [off, off + N) of a common index
// space, then its own ghost point at off + N (the reference's aliased land
// neighbour iistart-1), padded to a multiple of 64 points so that every CTA
// tile belongs to one member.  The index space is grouped in NB blocks of 32
// consecutive points (ldN = 32 NB):
//   spectrum arrays E, ES (= E* after the source half-step), EF:
//       [j/32][o][p/4][32][4]: a 32-point block's whole spectrum is one
//       contiguous region of O*P*128 bytes, one frequency of it P*128 bytes;
//       within that four directions of a point are 16 consecutive bytes, so a
//       warp (lane = point) reads four directions of 32 points as one 512-byte
//       access, a thread gets its direction pairs in register pairs, and every
//       direction offset is a compile-time immediate.  The blocks in flight
//       and their neighbours lie in a window of memory that few large pages
//       cover, whichever levels their warps are at
//   per-(o,i) tables TAB: [j/32][o][table][32], tables T_* below
//   mss prefix MSS: [j/32][o][3][32], the sums A, B, C over the levels below o
//       of k^3 dk dth/2 sum_p e (1, cos 2th, sin 2th); kept with E by whoever
//       writes E (the propagation, and k_mss after a state is set)
//   per-point arrays: [ldN]; all-point (land included) arrays: [imm]
#pragma once
#include <cstdint>

namespace umwm {

constexpr int MAX_OM = 64;
constexpr int MAX_PM = 72;
constexpr int MAX_LM = 100;

// per-(o,i) table rows (stored per frequency o, then table, then point)
enum TableRow {
  T_CG0 = 0,    // group velocity cg0 (ghost = min)   umwm_init.F90:1494, :1653-1656
  T_KDK,        // k dk                               :1505
  T_K3DK,       // k^3 dk                             :1506
  T_CP0,        // phase speed cp0 (ghost = min)      :1493, :1653-1656
  T_LOGL2Z,     // log(l2/z), capped                  :1530-1533
  T_FKOVG,      // f k / g                            :1507
  T_K,          // wavenumber k                       :1473
  T_SBF,        // bottom friction+percolation        :1510-1511
  T_SDV,        // viscous dissipation                :1512
  T_COTHKD,     // coth(0.2 kd)                       :1508
  T_BF1R,       // Snl weight to o+1                  :1523
  T_BF2R,       // Snl weight to o+2                  :1524
  T_COUNT
};
// rows 0 .. T_FKOVG: all the propagation and stress read; rows T_CP0 .. T_BF2R:
// what the source terms read (k^4 is formed from k)
constexpr int T_ADV_ROWS = T_FKOVG + 1;
constexpr int T_SRC0 = T_CP0, T_SRC_ROWS = T_BF2R + 1 - T_CP0;

constexpr int TILE = 64;  // wet points of a tile (a member's points start on a tile boundary)

// default levels ahead the spectral kernels prefetch the spectrum (and table)
// rows into L2 (Params::pf_*, tunable).  The integration copies a level's rows
// one level ahead, so the prefetch has to be two ahead to come before the copy:
// 692 us with one, 650 with two, 644 with three at 305 k points, 181, 176 and
// 176 at 86 k.  The propagation, 1.5 times as many rows in flight, loses with
// more than one (305 k points 1153, 1162 and 1255 us; 86 k 280, 289 and 313);
// the dts pre-pass is staged and prefetches only in its other form (two).
#ifndef UMWM_PF_DIST_PHYS
#define UMWM_PF_DIST_PHYS 2
#endif
#ifndef UMWM_PF_DIST_INTEG
#define UMWM_PF_DIST_INTEG 2
#endif
#ifndef UMWM_PF_DIST_ADV
#define UMWM_PF_DIST_ADV 1
#endif

// Direction counts with the small-model split of the levels over more warps
// (options "direction_groups" and the like, value 4) and with direction
// constants from a quarter turn.
__host__ __device__ constexpr bool quarter_groups(int pm) {
  return pm % 4 == 0 && (pm / 4 == 4 || pm / 4 == 6 || pm / 4 == 8 || pm / 4 == 9 || pm / 4 == 12);
}

struct Ctl;
struct Member;

struct Params {
  int Ntot, ldN, NB, O, P, NMtot, lm;
  int nmem;              // members
  int nsm;               // SMs of the device
  int ntiles;            // CTA tiles of TILE points over the whole index space
  const Member* mem;     // [nmem]
  const int* tile_mem;   // member of each tile [ntiles]
  float g, explim, sin_fac, fieldscale1, fieldscale2, twopisds_fac, sds_power, inv_sds_power, mss_fac, snl_fac,
      sdt_fac, z, nu_air, kappa, fprog, dth, dthg, oneovdth, dtg, fice_lth, fice_uth, eulerinv, rhow0;
  float bf1, bf2;  // downshifting weights (umwm_init.F90:1290-1294)
  // Sin factors of negative x (sin_fold): sin_fac fieldscale1, and with
  // fieldscale2 where cos(wdir - th) > 0 (umwm_source_functions.F90:60-67)
  float sin_neg1, sin_neg2;
  float gustiness;      // wind gust amplitude (umwm_forcing.F90:49-61)
  unsigned gust_seed;   // seed of the gust draws (option "gust_seed")
  int winds, currents, air_density, water_density, seaice, restart, curvilinear, isglobal;
  int ice_possible;  // fice can exceed fice_lth somewhere
  int groups4;       // the integration splits a block's levels over more warps (option "direction_groups" 4)
  int groups4_phys;  // the dts pre-pass does (options "direction_groups", "phys_groups")
  int adv_groups4;   // the propagation kernel does (options "direction_groups", "advect_groups")
  // Launch configuration of the three spectral kernels, chosen by the
  // autotuner or the options: the resident CTAs per SM their register budget
  // is sized for (__launch_bounds__ instances) and how many frequency levels
  // ahead they prefetch the spectrum and table rows into L2.  Results do not
  // depend on these.
  int minb_phys, minb_integ, minb_adv;
  int pf_phys, pf_integ, pf_adv;
  int count_cut;     // the propagation counts the bins its non-negativity cut changes (Global::cut_count)
  int adv_tma;       // option "advect_tma" (no effect: the propagation stages its rows in every form)
  int phys_tma;      // the dts pre-pass stages its rows with bulk copies (option "phys_tma")
  float f[MAX_OM], dom[MAX_OM];
  float th[MAX_PM], cth[MAX_PM], sth[MAX_PM], c2th[MAX_PM], s2th[MAX_PM];
  // The spectral kernels' direction constants: those of the directions of a
  // quarter (or half) turn, turned exactly to the others, so that opposite
  // directions (and, with quarters, perpendicular ones) have the same rounding;
  // and the mean sin and cos over the edge between p and p+1
  float dcth[MAX_PM], dsth[MAX_PM], dc2th[MAX_PM], ds2th[MAX_PM], shs[MAX_PM], chs[MAX_PM];
  float depth[MAX_LM];
};

// Device-resident control block of the inner (dynamic-dts) loop, one per member.
// What every block reads, what every block may update, and the flag of the
// forcing kernel lie on lines of their own: in one line, the loads of 12 k
// warps waited behind as many stores of the flag (66 to 85 us for the forcing
// of 305 k points with currents; 29 so, with one store per block).
struct Ctl {
  float sumt, dts, dta, dtr, dtr_temp;
  int zerocurrents;       // latched for propagation of this substep
  int first;              // reference's 'first' (first substep of the first run)
  int compute_rot;        // rotation recomputed this substep
  int done;               // sumt >= dtg: the member has finished the current dtg
  int running;            // the member takes part in the current substep
  int substep;            // substeps since initialize
  int err;                // error flags (bit 0: timeout)
  int log_count;
  alignas(128) unsigned minphys_enc;  // ordered encoding of min_i(explim/max|arg|)
  unsigned maxrot_enc;                // ordered encoding of max rotation flux
  alignas(128) int anycurrent;  // set by the forcing kernel when a wet current is non-zero
};

// Per-member ranges, scalars and pointers.
struct Member {
  int off, N, ghost;       // wet indices [off, off+N), ghost point off+N
  int nmoff, NM, mm, nm;   // all-point range [nmoff, nmoff+NM) and 2-d grid
  int iip;                 // index of the screen point, -1 if none
  float dtamin;
  Ctl* ctl;
  double* log;             // screen lines, 8 per substep
  int log_cap;
  const int *mi, *ni;      // 1-based (m, n) of each all-point index (member-local, [NM])
  // forcing levels (mm*nm, Fortran order): b = n, f = n+1
  const float *uwb, *uwf, *vwb, *vwf, *ucb, *ucf, *vcb, *vcf, *rhoab, *rhoaf, *rhowb, *rhowf, *ficeb, *ficef;
};

// control shared by all members (one per model)
struct Global {
  int not_done;            // members still inside the current dtg after this substep
  int budget;              // substeps the graph-driven inner loop may still run (-1: no limit)
  int iters;               // substeps the graph-driven inner loop ran since it was armed
  int nonfinite;           // non-finite values found by the last finite check
  int save_src;            // the last substep of this dtg keeps its source terms (for stress('ocn'))
  unsigned phys_blocks;    // blocks of the dts pre-pass that are through (back at 0 after it)
  unsigned long long cut_count;  // bins whose negative ef the propagation cut to 0 (option "count_cut")
  // grid barrier of the persistent substep kernel: arrivals, generation,
  // and the error flag a timed-out wait sets (reset before each launch)
  unsigned bar_count, bar_gen;
  int bar_err;
  // time block 0 of the persistent kernel spent in each stage, up to and
  // including the barrier that ends it (globaltimer ns, accumulated over
  // launches until read): forcing, (none), dts pre-pass, dts, integration,
  // propagation, screen
  unsigned long long stage_ns[8];
};

struct Ptrs {
  float *E, *ES, *EF;  // spectrum arrays (EF aliases E: each bin is read and then overwritten by one thread)
  const float* TAB;     // [NB][O][T_COUNT][32]
  float* MSS;           // [NB][O][3][32]
  // wet-point arrays [ldN]
  const int *ie, *iw, *in, *is;      // aliased neighbours (global index; the member's ghost for land)
  const int *iie, *iiw, *iin, *iis;  // true neighbours (global all-point index)
  const float *oneovar, *oneovdx, *oneovdy, *dxn, *dxs, *dye, *dyw, *d, *curv;
  int* oc;
  int* oc_rot;      // oc at the last rotation computation
  float* ustar;
  float* cd;
  float *taux, *tauy, *taux_form, *tauy_form, *taux_skin, *tauy_skin, *taux_diag, *tauy_diag, *tailatmx,
      *tailatmy;
  float* shelt;
  float* fcutoff;
  float* phys;      // physics_time_step
  float* sice_v;    // per-point sea-ice attenuation factor (0 when no ice)
  float* ehs;       // models with sea ice: a level's sum of e times k dk, [NB][O][32], kept with MSS
  // all-point arrays, member m at [nmoff, nmoff+NM) (land included; wet
  // points first, in the member's unrolled order)
  float *wspd, *wdir, *uc, *vc, *rhoa, *rhow, *rhorat, *fice;
  // Stokes drift [lm][ldN] and e-folding depth
  float *us, *vs, *ds;
  // diagnostics [ldN]
  float *ht, *mwp, *mwd, *mss, *mwl, *dwd, *dwl, *dwp, *dcp0, *dcp, *dcg0, *dcg, *momx, *momy, *cgmxx, *cgmxy,
      *cgmyy;
  Global* glob;
  // surrogate fallback (null otherwise): the source integration runs only
  // tiles with fb_tile[t] != 0 and writes only points with fb_pt[j] != 0
  const int* fb_tile;
  const unsigned char* fb_pt;
  // source terms of the last substep of a dtg, kept for stress('ocn') when
  // Global::save_src is set (null when not allocated): Sin, Sds after the
  // cothkd factor, Snl (spectrum layout) and the ustar they used [ldN]
  float *src_sin, *src_sds, *src_snl, *src_ust;
  float* ocn;  // stress('ocn') outputs, OCN_COUNT arrays of [ldN]
};

// stress('ocn') outputs (umwm_stress.F90:34-214), in this order in Ptrs::ocn
enum OcnField {
  OCN_TAUX_TOP = 0, OCN_TAUY_TOP, OCN_TAUX_BOT, OCN_TAUY_BOT, OCN_TAUX_SNL, OCN_TAUY_SNL, OCN_EPSX_OCN,
  OCN_EPSY_OCN, OCN_EPSX_ATM, OCN_EPSY_ATM, OCN_TAILX, OCN_TAILY, OCN_TAUX1, OCN_TAUY1, OCN_TAUX2, OCN_TAUY2,
  OCN_TAUX3, OCN_TAUY3, OCN_COUNT
};

// Wind gust draws, umwm_forcing.F90:49-56.  The reference fills gustu and
// gustv with Fortran random_number once per substep; here draw number
// (substep, cell, component) is a function of those three and a seed, so a
// run is reproducible and the oracle makes the same draws: the SplitMix64
// finaliser (Steele, Lea and Flood, 2014) of the seed and substep keys a
// second finalising of the cell index (column-major over the 2-d grid, as
// random_number fills an array) and the component (0: u, 1: v); its top
// 24 bits are the uniform draw in [0, 1).
__host__ __device__ inline uint64_t splitmix64_mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__host__ __device__ inline float gust_uniform(unsigned seed, unsigned substep, unsigned cell, unsigned comp) {
  const uint64_t key = splitmix64_mix(((uint64_t)seed << 32) | substep);
  const uint64_t z = splitmix64_mix(key ^ (((uint64_t)cell << 1) | comp));
  return (float)(z >> 40) * (1.f / 16777216.f);
}

// element offsets in the blocked layouts
__host__ __device__ inline size_t sidx(const Params& prm, int o, int p, int j) {
  return ((size_t)(j >> 5) * prm.O + o) * prm.P * 32 + (p >> 2) * 128 + (j & 31) * 4 + (p & 3);
}
__host__ __device__ inline size_t tidx(const Params& prm, int o, int t, int j) {
  return (((size_t)(j >> 5) * prm.O + o) * T_COUNT + t) * 32 + (j & 31);
}
// offset of direction p from direction 0 of the same bin row
__host__ __device__ constexpr int poff(int p) { return (p >> 2) * 128 + (p & 3); }

}  // namespace umwm
