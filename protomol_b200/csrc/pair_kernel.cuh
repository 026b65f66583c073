// The fused nonbonded pair kernel: Lennard-Jones and Coulomb with
// ProtoMol's switching functions (OneAtomPair / OneAtomPairTwo,
// force/OneAtomPairTwo.h:30-100) and the Ewald real-space term
// (NonbondedFullEwaldSystemForce::realTerm, .h:753-858), over the
// cluster-pair list (8 x 4 atom tiles, one pair per lane, each unordered
// pair listed once).
//
// Arithmetic:
//   * forces: the kernel precision Real (FP32 in the mixed mode) from
//     hi/lo-split FP64 coordinates; pairs whose FP32 distance lies within a
//     relative band of a cutoff are re-tested with the reference's exact
//     FP64 arithmetic, so the accepted pair set is the reference's;
//   * energies and virial: only when requested (ProtoMol's energies are
//     observed at output steps), and then in FP64 from the FP64 wrapped
//     coordinates (in mixed precision by a kernel of their own,
//     k_pairs_e64), because FP32 rounding of large cancelling pair energies
//     alone leaves a relative error near 1e-5 on the Ewald real-space sum;
//   * Cn switching: its polynomial in (r - rc) has large alternating
//     coefficients (switch/CnSwitchingFunction.cpp:9-23), so it is evaluated
//     in FP64 in every mode.
#pragma once

#include "pm_device.cuh"

namespace pmgpu {

template <typename Real>
struct PairArgs {
  Box box;
  int n;
  int ntypes;
  int mask;
  SwitchDev<Real> lj_sw, coul_sw;
  SwitchDev<double> lj_sw64, coul_sw64;
  int lj_modify, coul_modify;
  // rough-test cutoffs^2 (FP64 exact and the kernel-precision band)
  double lj_cut2, coul_cut2, ew_cut2, max_cut2;
  Real lj_lo, lj_hi, coul_lo, coul_hi, ew_lo, ew_hi, max_lo, max_hi;
  int same_cut;          // all active terms share one cutoff
  int minimal_image;     // LJ / Coulomb cutoff terms only for the minimal image
  Real half_edge[3];
  Real alpha, a2pi;
  double alpha64, a2pi64;
  int exact_erf;
  Real csf;  // coulomb scaling factor
  double csf64;
  int cap;              // tiles per row
  int nclusters;        // 8-atom i clusters (kRowParts tile rows each)
  int splits;           // warps per i cluster
  int shares, group;    // batched FP32 tile kernel: a cluster's shares of tiles
                        // and how many a warp takes
  const int *sorted;
  const double *pos;     // raw positions (exact re-test)
  const int *excl_start, *excl_partner, *excl_class;
  const uint2 *tiles;
  const unsigned *tmod;  // modified masks of flagged tiles
  const uint2 *jlanes;   // j-lane entries (force-only kernel)
  const float4 *ewtab;   // Ewald real-space force table (null: analytic)
  const int *jl_count;   // entries per row
  const int *tile_count;
  const float4 *xhi, *xlo;
  const double4 *xw;
  const int *type;
  const float4 *lj32;
  const double4 *lj64;
  long long *fslot;      // 3 planes of ns: forces by list slot (added to the
                         // atoms' forces by k_slot_forces)
  int ns;                // slots (plane stride of fslot)
  long long *acc;
  long long *pairbuf;
  long long pairbuf_cap;
  long long *paircount;
  int count_pairs;       // accumulate the accepted-pair count
  int same_sw;           // both cutoff terms take one switch (the same constants)
};

// Relative band around a cutoff^2 in which a squared distance formed from
// the wrapped FP64 coordinates does not decide.  Its error is that of the
// raw coordinates: 4e-14 of r^2 for atoms at 1e3 A, 3e-11 at 1e6 A; one pair
// in 1e8 takes the exact test needlessly.
constexpr double kBand64 = 1.0e-8;

// Exact FP64 squared distance of the image in hand, formed the way the
// reference forms it: the minimal difference (PeriodicBoundaryConditions.h:
// 72-110) plus a lattice vector (NonbondedFullEwaldSystemForce.h:790-805;
// for orthogonal boxes lattice components are exactly e_c * k_c).  d is the
// kernel's own difference, used only to pick the lattice vector.
template <typename Real>
__device__ __forceinline__ double exact_r2(const PairArgs<Real> &a, int oi, int oj,
                                           double dx, double dy, double dz) {
  double mx, my, mz;
  double r2 = box_mindiff(a.box, a.pos[3 * oi], a.pos[3 * oi + 1], a.pos[3 * oi + 2],
                          a.pos[3 * oj], a.pos[3 * oj + 1], a.pos[3 * oj + 2], mx, my, mz);
  if (!a.box.periodic) return r2;
  double kx = rint((dx - mx) * a.box.er[0]);
  double ky = rint((dy - my) * a.box.er[1]);
  double kz = rint((dz - mz) * a.box.er[2]);
  if (kx == 0.0 && ky == 0.0 && kz == 0.0) return r2;
  return xnorm2(xadd(mx, xmul(a.box.e[0], kx)), xadd(my, xmul(a.box.e[1], ky)),
                xadd(mz, xmul(a.box.e[2], kz)));
}

__device__ __forceinline__ float fast_exp(float x) { return __expf(x); }
__device__ __forceinline__ double fast_exp(double x) { return exp(x); }

// Value and derivative of a run-time switch; sv and sd keep them for a
// second term under the same switch (known = 1).
template <typename Real>
__device__ __forceinline__ void apply_switch(const SwitchDev<Real> &sw,
                                             const SwitchDev<double> &sw64, Real r2,
                                             Real &ff, Real &en, Real &sv, Real &sd, int known) {
  if (known) {
    ff = ff * sv - en * sd;
    en = en * sv;
    return;
  }
  // the Cn and CmpCnCn polynomials cancel in FP32: evaluated in FP64
  if (sizeof(Real) == 4 && (sw.kind == PMGPU_SW_CN || sw.kind == PMGPU_SW_CMPCNCN)) {
    double v64, d64;
    switch_eval<double>(sw64, (double)r2, v64, d64);
    sv = (Real)v64;
    sd = (Real)d64;
  } else {
    switch_eval<Real>(sw, r2, sv, sd);
  }
  ff = ff * sv - en * sd;
  en = en * sv;
}

// Compile-time description of a j-lane force-only kernel's switching
// functions and erfc variant (-1: the term has no switch), so that the
// per-pair arithmetic of the common configurations carries no run-time
// dispatch.
template <int LJK, int CK, int EXACT>
struct PairSpec {
  static constexpr int lj = LJK, coul = CK, exact = EXACT;
};

// Per-pair flags of an accepted pair: which terms are inside their cutoff,
// and whether the pair is a modified (scaled 1-4) one.
constexpr int kQLJ = 1, kQCoul = 2, kQEwald = 4, kQModified = 8;

// Pair force, energies of one accepted pair (the terms' arithmetic of
// OneAtomPairTwo::doOneAtomPair, force/OneAtomPairTwo.h:55-100).
// Returns f with F_i -= d * f.
template <typename Real, int TERMS>
__device__ __forceinline__ Real pair_force(const PairArgs<Real> &a, const Real *ljrow, Real r2,
                                           Real qq, int tj, int flags, Real &en_lj,
                                           Real &en_c) {
  const bool modified = flags & kQModified;
  const Real rinv = rsqrt_nr(r2);
  const Real rinv2 = rinv * rinv;
  Real f = 0, sv = 1, sd = 0;
  int known = 0;
  if ((TERMS & TERM_LJ) && (flags & kQLJ)) {
    Real A, B;
    if (sizeof(Real) == 4) {
      float4 p = __ldg(reinterpret_cast<const float4 *>(ljrow) + tj);
      A = modified ? p.z : p.x;
      B = modified ? p.w : p.y;
    } else {
      double4 p = reinterpret_cast<const double4 *>(ljrow)[tj];
      A = modified ? p.z : p.x;
      B = modified ? p.w : p.y;
    }
    // LennardJonesForce::operator() (force/LennardJonesForce.h:28-60)
    Real r6 = rinv2 * rinv2 * rinv2;
    Real r6B = B * r6;
    Real r12A = A * r6 * r6;
    Real en = r12A - r6B;
    Real ff = (Real(12) * r12A - Real(6) * r6B) * rinv2;
    if (a.lj_modify) apply_switch<Real>(a.lj_sw, a.lj_sw64, r2, ff, en, sv, sd, 0);
    known = a.same_sw;
    en_lj += en;
    f += ff;
  }
  if (modified) qq *= a.csf;
  if ((TERMS & TERM_COUL) && (flags & kQCoul)) {
    // CoulombForce::operator() (force/CoulombForce.h:29-40)
    Real en = qq * rinv;
    Real ff = en * rinv2;
    if (a.coul_modify) apply_switch<Real>(a.coul_sw, a.coul_sw64, r2, ff, en, sv, sd, known);
    en_c += en;
    f += ff;
  }
  if ((TERMS & TERM_EWALD) && (flags & kQEwald)) {
    // NonbondedFullEwaldSystemForce::realTerm (:820-842)
    Real r = r2 * rinv;
    Real ar = a.alpha * r;
    Real ee = qq * fast_exp(-ar * ar);
    Real en;
    if (!a.exact_erf)
      en = poly5_fast<Real>(ar) * ee * rinv;  // A&S erfc (MathUtilities.cpp:39-49)
    else
      en = qq * erfc(ar) * rinv;  // USE_EWALD_EXACT_ERF: C library erfc
    f += (en + a.a2pi * ee) * rinv2;
    en_c += en;
  }
  return f;
}

// Switch of a force-only specialised kernel, without branches: the value
// and derivative of every region are formed and the region's selected
// (C2SwitchingFunction.h:42-52, C1SwitchingFunction.h:41-50).  rinv is
// 1/sqrt(r2).
template <typename Real, int KIND>
__device__ __forceinline__ void switch_fast(const SwitchDev<Real> &sw, Real r2, Real rinv,
                                            Real &ff, Real en) {
  if (KIND == PMGPU_SW_C2) {
    // the polynomial is 1 with zero slope at the switch-on distance and 0
    // with zero slope at the cutoff, so r^2 clamped into [rs^2, rc^2] gives
    // every region's value and derivative (to rounding) without selects
    const Real r2c = fmin(fmax(r2, sw.switchon2), sw.cutoff2);
    const Real c2 = sw.cutoff2 - r2c;
    const Real c4 = c2 * (sw.s2 + Real(2) * r2c);
    const Real val = sw.s1 * (c2 * c4);
    const Real der = sw.s3 * (c2 * c2 - c4);
    ff = ff * val - en * der;
  } else if (KIND == PMGPU_SW_C1) {
    const Real d = r2 * rinv;
    const bool off = r2 > sw.cutoff2;
    const Real val = off ? Real(0) : Real(1) - d * (sw.c1a - r2 * sw.c1b);
    const Real der = off ? Real(0) : -sw.c1a * rinv + d * sw.c1c;
    ff = ff * val - en * der;
  }
}

// Pair force of the force-only specialised kernels: every term inside its
// (common) cutoff, no energies, no branches.  Same arithmetic as
// pair_force.  p holds the pair's LJ table entry (A, B, A14, B14).
template <typename Real, int TERMS, typename SPEC, bool MOD, typename P4>
__device__ __forceinline__ Real pair_force_p(const PairArgs<Real> &a, const P4 &p, Real r2,
                                             Real qq, bool modified) {
  const Real rinv = rsqrt_nr(r2);
  const Real rinv2 = rinv * rinv;
  Real f = 0;
  if (TERMS & TERM_LJ) {
    const Real A = MOD && modified ? p.z : p.x;
    const Real B = MOD && modified ? p.w : p.y;
    const Real r6 = rinv2 * rinv2 * rinv2;
    const Real r6B = B * r6;
    const Real r12A = A * r6 * r6;
    Real ff = (Real(12) * r12A - Real(6) * r6B) * rinv2;
    switch_fast<Real, SPEC::lj>(a.lj_sw, r2, rinv, ff, r12A - r6B);
    f += ff;
  }
  if (MOD) qq = modified ? qq * a.csf : qq;
  if (TERMS & TERM_COUL) {
    const Real en = qq * rinv;
    Real ff = en * rinv2;
    switch_fast<Real, SPEC::coul>(a.coul_sw, r2, rinv, ff, en);
    f += ff;
  }
  if (TERMS & TERM_EWALD) {
    const Real ar = a.alpha * (r2 * rinv);
    const Real ee = qq * fast_exp(-ar * ar);
    const Real en = SPEC::exact == 0 ? poly5_fast<Real>(ar) * ee * rinv : qq * erfc(ar) * rinv;
    f += (en + a.a2pi * ee) * rinv2;
  }
  return f;
}

// pair_force_p of the LJ + Ewald real force-only kernel with the Ewald
// factor read from the force table (kEwTabN cubics in shared memory): no
// square root, exponential or erfc per pair.  r2 must lie in the table's
// range [2^kEwTabLoExp, 2^(kEwTabLoExp + kEwTabOctaves)); others read the
// nearest end interval (the callers keep them out of the accepted pairs).
template <typename SPEC>
__device__ __forceinline__ float pair_force_tab(const PairArgs<float> &a, const float4 &p,
                                                float r2, float qq, bool modified,
                                                const float4 *s_ew) {
  const float rinv2 = __fdividef(1.f, r2);
  const float A = modified ? p.z : p.x;
  const float B = modified ? p.w : p.y;
  const float r6 = rinv2 * rinv2 * rinv2;
  const float r6B = B * r6;
  const float r12A = A * r6 * r6;
  float ff = (12.f * r12A - 6.f * r6B) * rinv2;
  switch_fast<float, SPEC::lj>(a.lj_sw, r2, 0.f, ff, r12A - r6B);
  qq = modified ? qq * a.csf : qq;
  const unsigned bits = __float_as_uint(r2);
  const int idx = min(max((int)(bits >> (23 - kEwTabSubBits)) - (int)kEwTabBase, 0), kEwTabN - 1);
  const float t =
      __uint_as_float(((bits << kEwTabSubBits) & 0x007FFFFFu) | 0x3F800000u) - 1.f;
  const float4 c = s_ew[idx];
  return fmaf(qq, fmaf(t, fmaf(t, fmaf(t, c.w, c.z), c.y), c.x), ff);
}

// Registers: the force-only FP32 kernels are held to 64 so four blocks fit
// per SM; the record and FP64 variants get more.
template <typename Real, int MODE>
struct PairOccupancy {
  static constexpr int warps = MODE == PAIR_FORCE && sizeof(Real) == 4 ? 32 : 16;
  static constexpr int blocks = warps / kPairWarps;
};

// Sum of (x, y, z) over the 8 lanes that share lane >> 3, transposed: on
// return lane l holds component (l & 3) of its group's sum (x, y, z, 0).
// Four shuffles instead of nine.
template <typename Real>
__device__ __forceinline__ Real group8_sum3(Real x, Real y, Real z, int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
  // xor 1: even lanes keep (x, z), odd lanes keep (y, 0)
  const Real k0 = b0 ? y : x, s0 = b0 ? x : y;
  const Real k1 = b0 ? Real(0) : z, s1 = b0 ? z : Real(0);
  const Real r0 = k0 + __shfl_xor_sync(0xffffffffu, s0, 1);
  const Real r1 = k1 + __shfl_xor_sync(0xffffffffu, s1, 1);
  // xor 2: lanes with bit 1 clear keep r0, the others r1
  Real v = (b1 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, b1 ? r0 : r1, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  return v;
}

__device__ __forceinline__ long long fixed_force(float v) {
  return __float2ll_rn(v * 4294967296.0f);  // exact scaling by 2^32
}
__device__ __forceinline__ long long fixed_force(double v) { return to_fixed(v, kForceScale); }

// The energies and virial of a block's pairs into the accumulators: v holds
// a lane's LJ energy, Coulomb (and Ewald) energy and the virial's upper
// triangle.  Summed over the block in FP64 and rounded to fixed point once a
// block (once a warp would leave an error growing with the splits).  Every
// thread of the block calls it.
template <int TERMS, bool VIRIAL, int WARPS>
__device__ __forceinline__ void block_energies(long long *acc, const double (&v)[8]) {
  constexpr int N = VIRIAL ? 8 : 2;
  __shared__ double s_e[WARPS][N];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < N; q++) {
    const double t = warp_sum(v[q]);
    if (lane == 0) s_e[wib][q] = t;
  }
  __syncthreads();
  const int q = threadIdx.x;
  if (q >= N) return;
  double t = 0.0;
  for (int w = 0; w < WARPS; w++) t += s_e[w][q];
  const long long fixed = to_fixed(t, kEnergyScale);
  if (q == 0) {
    if (TERMS & TERM_LJ) red_add(&acc[ACC_LJ], fixed);
  } else if (q == 1) {
    if (TERMS & (TERM_COUL | TERM_EWALD)) red_add(&acc[ACC_COULOMB], fixed);
  } else {
    const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    for (int k = 0; k < 9; k++)
      if (map[k] == q - 2) red_add(&acc[ACC_VIRIAL + k], fixed);
  }
}

// One warp per (8-atom i cluster, contiguous share of its tiles).  Lane
// l holds pair (i atom l & 7, j atom l >> 3) of every 8 x 4 tile, so a
// tile's 32 pairs are evaluated at once with no compaction.  The list holds
// each unordered pair once, so the pair force goes to both atoms: i's
// share accumulates in the lane over the warp's tiles, j's share is summed
// over the 8 lanes of the same j atom and added with one fixed-point
// atomic per component.  Energies and virial count every pair once.
// Pairs are accepted by the cutoff tests of the reference (with the exact
// FP64 re-test near a cutoff); the tile mask carries the list's exclusion
// and modified (scaled 1-4) status.
//
// SHARES (FP32, batched launches): a warp takes `group` of the `shares` that
// the single-system launch gives a warp each, and rounds its i sums to fixed
// point share by share, so it leaves the same forces with fewer warps.
template <typename Real, int TERMS, int MODE, bool SHARES>
__device__ __forceinline__ void pairs_body(const PairArgs<Real> &a, Blk blk) {
  constexpr bool MIXED = sizeof(Real) == 4;
  // (in mixed precision energies come from k_pairs_e64)
  constexpr bool ENERGY = !MIXED && (MODE == PAIR_ENERGY || MODE == PAIR_VIRIAL);
  constexpr bool VIRIAL = !MIXED && MODE == PAIR_VIRIAL;
  constexpr bool RECORD = MODE == PAIR_RECORD;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int il = lane & 7, jl = lane >> 3;
  const unsigned lanebit = 1u << lane;  // this lane's bit of a tile mask
  double Elj = 0, Ec = 0;
  Real vxx = 0, vxy = 0, vxz = 0, vyy = 0, vyz = 0, vzz = 0;
  int npairs = 0;
  // this warp's work item (i cluster, share of its tiles)
  const int wib = threadIdx.x >> 5, gw = blk.x * kPairWarps + wib;
  const bool item = gw < a.nclusters * a.splits;
  const int ci = item ? gw / a.splits : 0, sp = gw - ci * a.splits;
  // the cluster's tiles are its kRowParts rows read one after the other;
  // this warp takes tiles [t0, t1) of that sequence
  static_assert(kRowParts == 4, "one int4 of row counts per cluster");
  const int4 c4 = *reinterpret_cast<const int4 *>(a.tile_count + kRowParts * ci);
  const int cnt = item ? c4.x + c4.y + c4.z + c4.w : 0;
  const int t0 = SHARES ? (int)((long long)cnt * (sp * a.group) / a.shares)
                        : (int)((long long)cnt * sp / a.splits);
  const int t1 = SHARES ? (int)((long long)cnt * min((sp + 1) * a.group, a.shares) / a.shares)
                        : (int)((long long)cnt * (sp + 1) / a.splits);
  const int islot = 8 * ci + il;
  const int oi = a.sorted[islot];
  Real fx = 0, fy = 0, fz = 0;
  // an i component's sum over the 4 j lanes of each i atom: lane (il, jl)
  // ends with component jl (x, y, z, none) of i atom il
  auto i_sum = [&]() {
    const bool b0 = jl & 1, b1 = jl & 2;
    const Real r0 = (b0 ? fy : fx) + __shfl_xor_sync(kAll, b0 ? fx : fy, 8);
    const Real r1 = (b0 ? Real(0) : fz) + __shfl_xor_sync(kAll, b0 ? fz : Real(0), 8);
    return (b1 ? r1 : r0) + __shfl_xor_sync(kAll, b1 ? r0 : r1, 16);
  };
  // this warp's i sums in fixed point, of the shares done (SHARES)
  __shared__ long long s_i[SHARES ? kPairWarps : 1][24];
  if (SHARES && jl < 3) s_i[wib][lane] = 0;
  if (t1 > t0) {
  const double4 wi = a.xw[islot];  // the FP64 kernel only
  Real xi_h[3], xi_l[3];
  Real qi;
  int ti;
  if (MIXED) {
    const float4 h = a.xhi[islot], l = a.xlo[islot];
    xi_h[0] = h.x; xi_h[1] = h.y; xi_h[2] = h.z; qi = h.w;
    xi_l[0] = l.x; xi_l[1] = l.y; xi_l[2] = l.z; ti = __float_as_int(l.w);
  } else {
    xi_h[0] = wi.x; xi_h[1] = wi.y; xi_h[2] = wi.z; qi = wi.w;
    xi_l[0] = xi_l[1] = xi_l[2] = Real(0);
    ti = oi >= 0 ? a.type[oi] : 0;
  }
  const Real *ljrow = MIXED ? reinterpret_cast<const Real *>(a.lj32 + ti * a.ntypes)
                            : reinterpret_cast<const Real *>(a.lj64 + ti * a.ntypes);
  // i as seen from the tile's image of j (d = xj - (xi - s L))
  int cur = kZeroShift;
  Real xs_h[3] = {xi_h[0], xi_h[1], xi_h[2]};
  Real xs_l[3] = {xi_l[0], xi_l[1], xi_l[2]};
  constexpr int kAllTerms = ((TERMS & TERM_LJ) ? kQLJ : 0) | ((TERMS & TERM_COUL) ? kQCoul : 0) |
                            ((TERMS & TERM_EWALD) ? kQEwald : 0);
  // tile t0 is index kb of row part p; the warp walks the parts in order
  int p = 0, kb = t0, rowlen = c4.x;
  while (kb >= rowlen) {
    kb -= rowlen;
    p++;
    rowlen = p == 1 ? c4.y : (p == 2 ? c4.z : c4.w);
  }
  // tb: the end of the share tile tc is in (this warp's only one without
  // SHARES)
  int tc = t0, tb = t1;
  unsigned share = SHARES ? sp * a.group : 0;
  while (tc < t1) {
    if (SHARES) {
      while ((tb = (int)((unsigned)cnt * (share + 1u) / (unsigned)a.shares)) == tc) share++;
    }
    const size_t row0 = (size_t)(kRowParts * ci + p) * a.cap;
    const uint2 *row = a.tiles + row0;
    const int ke = min(rowlen, kb + (tb - tc));
    tc += ke - kb;
  for (int k = kb; k < ke; k++) {
    const uint2 t2 = __ldg(row + k);
    const uint3 tile = make_uint3(t2.x, t2.y,
                                  (t2.x & kModFlag) ? __ldg(a.tmod + row0 + k) : 0u);
    const int hj = (int)(tile.x & kJMask);
    const int sh = (int)((tile.x >> kShiftBits) & kShiftMask);
    if (__any_sync(kAll, sh != cur)) {  // tiles are grouped by image
      const int sx = (sh & 3) - 1, sy = ((sh >> 2) & 3) - 1, sz = ((sh >> 4) & 3) - 1;
      // reloaded rather than held in registers through the loop
      const double4 w = a.xw[islot];
      const double xs64[3] = {w.x - sx * a.box.e[0], w.y - sy * a.box.e[1],
                              w.z - sz * a.box.e[2]};
      for (int c = 0; c < 3; c++) {
        if (MIXED) {
          const float h = (float)xs64[c];
          xs_h[c] = h;
          xs_l[c] = (float)(xs64[c] - (double)h);
        } else {
          xs_h[c] = xs64[c];
        }
      }
      cur = sh;
    }
    const int jslot = 4 * hj + jl;
    const bool live = (tile.y & lanebit) != 0u;
    Real dx, dy, dz, qj;
    int tj = 0;
    if (MIXED) {
      const float4 h = a.xhi[jslot], l = a.xlo[jslot];
      dx = (h.x - xs_h[0]) + (l.x - xs_l[0]);
      dy = (h.y - xs_h[1]) + (l.y - xs_l[1]);
      dz = (h.z - xs_h[2]) + (l.z - xs_l[2]);
      qj = h.w;
      tj = __float_as_int(l.w);
    } else {
      const double4 wj = a.xw[jslot];
      dx = wj.x - xs_h[0];
      dy = wj.y - xs_h[1];
      dz = wj.z - xs_h[2];
      qj = wj.w;
    }
    const Real r2 = dx * dx + dy * dy + dz * dz;
    int flags = 0;
    bool band = false;
    if (live && a.same_cut) {  // every term shares one cutoff
      if (r2 <= a.max_lo) flags = kAllTerms;
      else band = r2 <= a.max_hi;
    } else if (live) {
      if (TERMS & TERM_LJ) {
        if (r2 <= a.lj_lo) flags |= kQLJ;
        else band |= r2 <= a.lj_hi;
      }
      if (TERMS & TERM_COUL) {
        if (r2 <= a.coul_lo) flags |= kQCoul;
        else band |= r2 <= a.coul_hi;
      }
      if (TERMS & TERM_EWALD) {
        if (r2 <= a.ew_lo) flags |= kQEwald;
        else band |= r2 <= a.ew_hi;
      }
    }
    // pairs within a rounding band of a cutoff take the reference's exact
    // FP64 test (rare: a real branch)
    if (__any_sync(kAll, band)) {
      if (band) {
        const double r2x = exact_r2(a, oi, a.sorted[jslot], (double)dx, (double)dy, (double)dz);
        if ((TERMS & TERM_LJ) && r2 > a.lj_lo && r2x <= a.lj_cut2) flags |= kQLJ;
        if ((TERMS & TERM_COUL) && r2 > a.coul_lo && r2x <= a.coul_cut2) flags |= kQCoul;
        if ((TERMS & TERM_EWALD) && r2 > a.ew_lo && r2x <= a.ew_cut2) flags |= kQEwald;
      }
    }
    // boxes below twice the cutoff: cutoff terms take the minimal image only
    // (Ewald real space sums every image, NonbondedFullEwaldSystemForce.h:790)
    if ((TERMS & (TERM_LJ | TERM_COUL)) && a.minimal_image && (flags & (kQLJ | kQCoul)) &&
        !(fabs(dx) <= a.half_edge[0] && fabs(dy) <= a.half_edge[1] &&
          fabs(dz) <= a.half_edge[2]))
      flags &= ~(kQLJ | kQCoul);
    Real jx = 0, jy = 0, jz = 0;
    if (flags) {
      if ((tile.z >> lane) & 1u) flags |= kQModified;
      if (!MIXED) tj = a.type[a.sorted[jslot]];
      Real en_lj = 0, en_c = 0;
      const Real f = pair_force<Real, TERMS>(a, ljrow, r2, qi * qj, tj, flags, en_lj, en_c);
      jx = dx * f;
      jy = dy * f;
      jz = dz * f;
      fx -= jx;
      fy -= jy;
      fz -= jz;
      npairs++;
      if (ENERGY) {
        Elj += (double)en_lj;
        Ec += (double)en_c;
      }
      if (VIRIAL) {
        // addVirial(fij, d) with fij = d * f
        vxx += dx * jx; vxy += dx * jy; vxz += dx * jz;
        vyy += dy * jy; vyz += dy * jz; vzz += dz * jz;
      }
      if (RECORD) {
        const int oj = a.sorted[jslot];
        if (oi != oj) {
          long long slot = atomicAdd((unsigned long long *)a.paircount, 1ull);
          if (slot < a.pairbuf_cap)
            a.pairbuf[slot] = ((long long)min(oi, oj) << 32) | (unsigned)max(oi, oj);
        }
      }
    }
    // j's share: summed over its 8 lanes, one atomic per component
    {
      const unsigned act = __ballot_sync(kAll, flags != 0);
      const Real js = group8_sum3<Real>(jx, jy, jz, lane);
      long long *dst = a.fslot + il * a.ns + jslot;
      const long long v = fixed_force(js);
      if (il < 3 && ((act >> (8 * jl)) & 0xFFu)) red_add(dst, v);
    }
  }
    kb = ke;
    if (SHARES && tc == tb) {
      const Real v = i_sum();
      if (jl < 3) s_i[wib][lane] += fixed_force(v);
      fx = fy = fz = 0;
    }
    if (tc < t1 && kb == rowlen) {  // next non-empty row part
      do {
        p++;
        rowlen = __ldg(a.tile_count + kRowParts * ci + p);
      } while (rowlen == 0);
      kb = 0;
    }
  }
  }  // tiles
  const Real isum = SHARES ? Real(0) : i_sum();
  if constexpr (MIXED) {
    if (jl < 3 && oi >= 0 && t1 > t0)
      red_add(&a.fslot[jl * a.ns + islot], SHARES ? s_i[wib][lane] : fixed_force(isum));
  } else {
    // in FP64 the rounding to fixed point is the forces' only error: the
    // block's warps of one cluster add up first, so that an atom's i share is
    // rounded once a block, not once a warp
    __shared__ double s_f[kPairWarps][24];
    __shared__ int s_ci[kPairWarps];
    if (jl < 3) s_f[wib][lane] = isum;
    if (lane == 0) s_ci[wib] = item ? ci : -1;
    __syncthreads();
    if (item && (wib == 0 || s_ci[wib - 1] != ci) && lane < 24) {
      double t[kPairWarps];
#pragma unroll
      for (int w = 0; w < kPairWarps; w++) t[w] = s_ci[w] == ci ? s_f[w][lane] : 0.0;
#pragma unroll
      for (int o = kPairWarps / 2; o > 0; o >>= 1)
#pragma unroll
        for (int w = 0; w < o; w++) t[w] += t[w + o];
      const double f = t[0];
      const int slot = 8 * ci + (lane & 7);
      if (f != 0.0 && a.sorted[slot] >= 0)
        red_add(&a.fslot[(lane >> 3) * a.ns + slot], fixed_force(f));
    }
  }
  if (ENERGY || a.count_pairs) {
    int np = warp_sum(npairs);
    if (lane == 0) red_add(&a.acc[ACC_PAIRS], (long long)np);
  }
  if constexpr (ENERGY) {
    const double v[8] = {Elj,         Ec,          (double)vxx, (double)vxy,
                         (double)vxz, (double)vyy, (double)vyz, (double)vzz};
    block_energies<TERMS, VIRIAL, kPairWarps>(a.acc, v);
  }
}

template <typename Real, int TERMS, int MODE>
__global__ void __launch_bounds__(kPairWarps * 32, PairOccupancy<Real, MODE>::blocks)
    k_pairs(PairArgs<Real> a) {
  pairs_body<Real, TERMS, MODE, false>(a, own_blk());
}

template <typename Real, int TERMS, int MODE>
__global__ void __launch_bounds__(kPairWarps * 32, PairOccupancy<Real, MODE>::blocks)
    k_pairs_batch(const PairArgs<Real> *__restrict__ tab, const int *__restrict__ first, int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(PairArgs<Real>)];
  const int m = batch_member(first, nm, blockIdx.x);
  pairs_body<Real, TERMS, MODE, true>(batch_args_shared(tab, m, raw), batch_blk(first, m));
}

// ---------------------------------------------------------------------------
// Force-only FP32 pair kernel of the inner MD steps, j atoms on the lanes.
//
// A warp takes the tiles of its work item (one 8-atom i cluster, a
// contiguous share of its tiles) eight at a time: lane l holds j atom l & 3
// of tile l >> 2 of the batch and evaluates its pairs with the cluster's 8
// i atoms one after another, the i atoms broadcast from shared memory.  A
// lane's j force is complete after those eight pairs and goes out with one
// fixed-point atomic per component.  The i forces stay in registers (8
// atoms x 3 components per lane) over all the tiles of the item and are
// summed over the lanes once, at its end, by transposed butterflies
// (warp_tsum8).  Against one pair per lane per tile (k_pairs) this leaves
// out the per-tile image bookkeeping, the per-tile j-force reduction and the
// tile-wide votes: the work per tile is the pair arithmetic and a few loads.
//
// Coordinates: FP32 vectors from the cluster's first atom, formed in FP64
// from the wrapped FP64 positions with the j atom's periodic image added in
// FP64, so each distance carries one FP32 rounding of vectors no longer
// than the reach plus the cluster extent.  Pairs within the relative band
// of the cutoff take the reference's exact FP64 test after the batch's
// pairs (rare), so the accepted set is the reference's.
constexpr int kJlWarps = 8;
constexpr int kJlMaxTypes = 16;  // a cluster's LJ pairs staged in shared memory up to this many types
constexpr int kJlMaxSplits = 16;  // warps one i cluster's tiles may be divided over
constexpr float kEwTabMin = 1.0f / (1 << -kEwTabLoExp);  // the table's lowest r^2

// The eight pairs of one lane's j atom with the cluster's i atoms (mi: the
// pairs of the list's interaction mask); unmodified pairs of the table form
// take jl_pairs8_x2.
template <int TERMS, typename SPEC, bool MOD, bool TAB>
__device__ __forceinline__ void jl_pairs8(const PairArgs<float> &a, const float4 *s_ew,
                                          const float4 *xi, const int *ti, float rjx, float rjy,
                                          float rjz, float qj, int tj, unsigned mi, unsigned mm,
                                          float2 (&fi)[4][3], float &fjx, float &fjy, float &fjz,
                                          unsigned &band, int &npairs) {
#pragma unroll
  for (int il = 0; il < 8; il++) {
    const float4 x = xi[il];
    const float dx = rjx - x.x, dy = rjy - x.y, dz = rjz - x.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    const bool on = (mi >> il) & 1u;
    // (table form: pairs closer than the table's range take the exact path)
    const bool act = on && r2 <= a.max_lo && (!TAB || r2 >= kEwTabMin);
    band |= (on && !act && r2 <= a.max_hi) ? (1u << il) : 0u;
    npairs += act;
    const float rr = act ? r2 : 1.f;
    const float4 p = __ldg(a.lj32 + ti[il] + tj);
    float f;
    if constexpr (TAB)
      f = pair_force_tab<SPEC>(a, p, rr, x.w * qj, (mm >> il) & 1u, s_ew);
    else
      f = pair_force_p<float, TERMS, SPEC, MOD>(a, p, rr, x.w * qj, MOD && ((mm >> il) & 1u));
    f = act ? f : 0.f;
    fjx = fmaf(dx, f, fjx);
    fjy = fmaf(dy, f, fjy);
    fjz = fmaf(dz, f, fjz);
    float2 *fp = fi[il >> 1];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float d = c == 0 ? dx : (c == 1 ? dy : dz);
      if (il & 1) fp[c].y = fmaf(-d, f, fp[c].y);
      else fp[c].x = fmaf(-d, f, fp[c].x);
    }
  }
}

// The j atoms' records of one warp step, staged by cp.async: the FP64
// wrapped position and charge, and the type.
struct JlStage {
  double4 w[32];
  int t[32];
};

// A warp's shared memory: its cluster's atoms from the reference point, one
// by one (xi: position, charge) and by twos for the packed pair arithmetic
// (xy: x0, x1, y0, y1; zq: z0, z1, q0, q1; ljp[k][t]: jl_lj_pair of the two
// atoms with j type t), and the j-atom records of two warp steps.
template <bool LJP>
struct JlWarp {
  float4 xi[8], xy[4], zq[4];
  float4 ljp[LJP ? 4 : 1][LJP ? kJlMaxTypes : 1];
  double wc[4];  // reference point (FP64)
  int ti[8];     // i type * ntypes
  int oi[8];     // i atom (-1: padding)
  JlStage js[2];
};
template <bool SMEM_LJ, bool TAB>
struct JlSmem {
  float4 ew[TAB ? kEwTabN : 1];
  JlWarp<SMEM_LJ && TAB> w[kJlWarps];
};

// 12 A and -6 B of two i atoms against one j type, times the C2 switch's
// factor s1.
__device__ __forceinline__ float4 jl_lj_pair(const float4 &p0, const float4 &p1, float s1) {
  const float a = 12.f * s1, b = -6.f * s1;
  return make_float4(a * p0.x, a * p1.x, b * p0.y, b * p1.y);
}

// The unmodified pairs of one lane's j atom with the cluster's 8 i atoms,
// LJ C2 + Ewald table form, two i atoms at a time in packed FP32 (fma, mul
// and add on register pairs: one issue slot for two results).  The kernel
// is issue-bound, and packing halves the distance, Lennard-Jones, switch
// and force-sum instructions; the reciprocal, the cutoff test and the table
// lookup stay scalar.  A pair's distance bits less the table's first
// (u) give the cutoff test, the table's range test and its index at once;
// pairs outside read the table's last interval and are dropped by a select.
// Warp instructions of a launch 33.2 -> 25.3 M on 23,550 atoms, 46.4 -> 40.4
// us (caches warm; 22.5 M with the two warps a cluster it takes now);
// 49,998 atoms 83.6 -> 70.7 us.  What is left is the
// per-entry work (decode, FP64 image shift, staging, three 64-bit force
// atomics) and the latency of 24 warps an SM.
// (d = xi - xj here.)  fj gets the sum of f d, i.e. minus the force on j.
template <bool SMEM_LJ>
__device__ __forceinline__ void jl_pairs8_x2(const PairArgs<float> &a, const float4 *s_ew,
                                             const JlWarp<SMEM_LJ> &W, float rjx, float rjy,
                                             float rjz, float qj, int tj, unsigned mi,
                                             unsigned umax, float2 (&fi)[4][3], float2 (&fj)[3],
                                             bool &band) {
  constexpr unsigned kBase = kEwTabBase << (23 - kEwTabSubBits);
  const float2 nx = make_float2(-rjx, -rjx), ny = make_float2(-rjy, -rjy),
               nz = make_float2(-rjz, -rjz), q2 = make_float2(qj, qj);
  const float2 ncut = make_float2(-a.lj_sw.cutoff2, -a.lj_sw.cutoff2),
               s2 = make_float2(a.lj_sw.s2, a.lj_sw.s2), m3 = make_float2(-1.f / 3.f, -1.f / 3.f);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float4 xy = W.xy[k], zq = W.zq[k];
    const float2 dx = add2(make_float2(xy.x, xy.y), nx),
                 dy = add2(make_float2(xy.z, xy.w), ny),
                 dz = add2(make_float2(zq.x, zq.y), nz);
    const float2 r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
    // LJ times the switch's factor s1: 12 A r^-12 and -6 B r^-6
    float4 ab;
    if constexpr (SMEM_LJ) {
      ab = W.ljp[k][tj];
    } else {
      const float4 p0 = __ldg(a.lj32 + W.ti[2 * k] + tj), p1 = __ldg(a.lj32 + W.ti[2 * k + 1] + tj);
      ab = jl_lj_pair(p0, p1, a.lj_sw.s1);
    }
    const float2 i2 = make_float2(rcp_fast(r2.x), rcp_fast(r2.y));
    const float2 r6 = mul2(mul2(i2, i2), i2);
    const float2 nb = mul2(make_float2(ab.z, ab.w), r6);
    const float2 a12 = mul2(mul2(make_float2(ab.x, ab.y), r6), r6);
    const float2 sum = add2(a12, nb);
    // C2 switch on r^2 clamped into [rs^2, rc^2] (switch_fast), with
    // c = r^2 - rc^2 and w = rc^2 - 3 rs^2 + 2 r^2
    const float2 rc = make_float2(fminf(fmaxf(r2.x, a.lj_sw.switchon2), a.lj_sw.cutoff2),
                                  fminf(fmaxf(r2.y, a.lj_sw.switchon2), a.lj_sw.cutoff2));
    const float2 c = add2(rc, ncut);
    const float2 cw = mul2(c, add2(add2(rc, rc), s2));
    // (s1 is in the parameters; the derivative's factor s3 is 4 s1, and
    // sum + nb is 12 times the energy)
    const float2 der = mul2(m3, fma2(c, c, cw));
    const float2 lj = fma2(mul2(sum, i2), mul2(c, cw),
                                 mul2(add2(sum, nb), der));
    const float2 qq = mul2(make_float2(zq.z, zq.w), q2);
    float2 f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float rr = h ? r2.y : r2.x;
      const unsigned u = __float_as_uint(rr) - kBase;
      const bool on = (mi >> (2 * k + h)) & 1u;
      const bool act = on && u <= umax;
      band |= on && !act && rr <= a.max_hi;
      const float4 t4 = s_ew[min(u >> (23 - kEwTabSubBits), (unsigned)kEwTabN - 1u)];
      const float t =
          __uint_as_float(((u << kEwTabSubBits) & 0x007FFFFFu) | 0x3F800000u) - 1.f;
      const float g = fmaf(t, fmaf(t, fmaf(t, t4.w, t4.z), t4.y), t4.x);
      const float v = fmaf(h ? qq.y : qq.x, g, h ? lj.y : lj.x);
      (h ? f.y : f.x) = act ? v : 0.f;
    }
    fj[0] = fma2(dx, f, fj[0]);
    fj[1] = fma2(dy, f, fj[1]);
    fj[2] = fma2(dz, f, fj[2]);
    fi[k][0] = fma2(dx, f, fi[k][0]);
    fi[k][1] = fma2(dy, f, fi[k][1]);
    fi[k][2] = fma2(dz, f, fi[k][2]);
  }
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

extern __shared__ __align__(16) unsigned char jl_smem[];

template <int TERMS, typename SPEC, bool SMEM_LJ, bool TAB>
__device__ __forceinline__ void pairs_jl_body(const PairArgs<float> &a, Blk blk) {
  constexpr unsigned kAll = 0xffffffffu;
  JlSmem<SMEM_LJ, TAB> &S = *reinterpret_cast<JlSmem<SMEM_LJ, TAB> *>(jl_smem);
  const float4 *s_ew = S.ew;
  if (TAB) {
    for (int k = threadIdx.x; k < kEwTabN; k += blockDim.x) S.ew[k] = __ldg(a.ewtab + k);
    __syncthreads();
  }
  // the largest accepted r^2, as table position (see jl_pairs8_x2)
  const unsigned umax =
      __float_as_uint(a.max_lo) - (kEwTabBase << (23 - kEwTabSubBits));
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  auto &W = S.w[wib];
  int npairs = 0;
  const int nitems = a.nclusters * a.splits;
  const size_t rowcap = 4 * (size_t)a.cap;  // entries per row
  for (int gw = blk.x * kJlWarps + wib; gw < nitems; gw += blk.n * kJlWarps) {
    const int ci = gw / a.splits, sp = gw - ci * a.splits;
    static_assert(kRowParts == 4, "one int4 of row counts per cluster");
    const int4 c4 = *reinterpret_cast<const int4 *>(a.jl_count + kRowParts * ci);
    const int p1 = c4.x, p2 = p1 + c4.y, p3 = p2 + c4.z, cnt = p3 + c4.w;
    const int t0 = (int)((long long)cnt * sp / a.splits);
    const int t1 = (int)((long long)cnt * (sp + 1) / a.splits);
    if (t1 <= t0) continue;
    __syncwarp();  // the previous item's reads of this warp's staging are done
    if (lane < 8) {
      const int islot = 8 * ci + lane;
      const double4 w0 = a.xw[8 * ci];  // a cluster with entries has an atom in its first slot
      const double4 wi = a.xw[islot];
      const int oi = a.sorted[islot];
      const float4 x = make_float4((float)(wi.x - w0.x), (float)(wi.y - w0.y),
                                   (float)(wi.z - w0.z), (float)wi.w);
      W.xi[lane] = x;
      if (TAB) {
        float *xy = &W.xy[lane >> 1].x + (lane & 1), *zq = &W.zq[lane >> 1].x + (lane & 1);
        xy[0] = x.x;
        xy[2] = x.y;
        zq[0] = x.z;
        zq[2] = x.w;
      }
      W.ti[lane] = (oi >= 0 ? __float_as_int(__ldg(&a.xlo[islot].w)) : 0) * a.ntypes;
      W.oi[lane] = oi;
      if (lane < 3) W.wc[lane] = lane == 0 ? w0.x : (lane == 1 ? w0.y : w0.z);
    }
    __syncwarp();
    if constexpr (TAB && SMEM_LJ) {
      for (int k = lane; k < 4 * a.ntypes; k += 32) {
        const int c = k / a.ntypes, t = k - c * a.ntypes;
        const float4 p0 = __ldg(a.lj32 + W.ti[2 * c] + t), p1 = __ldg(a.lj32 + W.ti[2 * c + 1] + t);
        W.ljp[c][t] = jl_lj_pair(p0, p1, a.lj_sw.s1);
      }
      __syncwarp();
    }
    const float4 *xi = W.xi;
    const int *ti = W.ti;
    float2 fi[4][3];
#pragma unroll
    for (int k = 0; k < 4; k++) fi[k][0] = fi[k][1] = fi[k][2] = make_float2(0.f, 0.f);
    // Software pipeline over the warp steps (32 entries each): the entries
    // of step k + 2 are loaded into registers and the j atoms' records of
    // step k + 1 are copied into this lane's shared-memory slot (cp.async)
    // while step k computes, so the dependent loads (entry, then the j
    // atom's record) are in flight during a whole step.  A lane reads only
    // the slot it copied itself.
    auto entry_at = [&](int idx) -> uint2 {
      if (idx >= t1) return make_uint2(0u, 0u);  // mask 0: no entry
      const int p = (idx >= p1) + (idx >= p2) + (idx >= p3);
      const int off = idx - (p == 0 ? 0 : (p == 1 ? p1 : (p == 2 ? p2 : p3)));
      return __ldg(a.jlanes + (size_t)(kRowParts * ci + p) * rowcap + off);
    };
    auto stage = [&](uint2 e, int buf) {
      if (e.y & 0xFFu) {
        const int js = (int)(e.x & kJSlotMask);
        JlStage &g = W.js[buf];
        cp_async16(&g.w[lane], &a.xw[js]);
        cp_async16(reinterpret_cast<char *>(&g.w[lane]) + 16,
                   reinterpret_cast<const char *>(&a.xw[js]) + 16);
        cp_async4(&g.t[lane], &a.xlo[js].w);
      }
      cp_async_commit();
    };
    uint2 ecur = entry_at(t0 + lane), enext = entry_at(t0 + 32 + lane);
    stage(ecur, 0);
    for (int b0 = t0, k = 0; b0 < t1; b0 += 32, k++) {
      stage(enext, (k + 1) & 1);
      const uint2 enext2 = entry_at(b0 + 64 + lane);
      cp_async_wait<1>();  // this step's copies have landed
      unsigned mi = ecur.y & 0xFFu, mm = (ecur.y >> 8) & 0xFFu;
      const int jslot = (int)(ecur.x & kJSlotMask);
      int tj = 0;
      float rjx = 0.f, rjy = 0.f, rjz = 0.f, qj = 0.f;
      if (mi) {
        const JlStage &g = W.js[k & 1];
        const double4 wj = g.w[lane];
        // the j atom in the entry's image (d = xj + s L - xi), from the
        // reference point; the image offsets are exact (-L, 0 or L)
        const int sh = (int)(ecur.x >> kJSlotBits);
        const int sx = sh & 3, sy = (sh >> 2) & 3, sz = (sh >> 4) & 3;
        const double ox = sx == 1 ? 0.0 : (sx == 0 ? -a.box.e[0] : a.box.e[0]);
        const double oy = sy == 1 ? 0.0 : (sy == 0 ? -a.box.e[1] : a.box.e[1]);
        const double oz = sz == 1 ? 0.0 : (sz == 0 ? -a.box.e[2] : a.box.e[2]);
        rjx = (float)((wj.x + ox) - W.wc[0]);
        rjy = (float)((wj.y + oy) - W.wc[1]);
        rjz = (float)((wj.z + oz) - W.wc[2]);
        qj = (float)wj.w;
        tj = g.t[lane];
      }
      ecur = enext;
      enext = enext2;
      float fjx = 0.f, fjy = 0.f, fjz = 0.f;
      unsigned band = 0u;
      // modified (scaled 1-4) pairs are rare: batches without any take the
      // path without their selects
      const bool mod = __any_sync(kAll, mm != 0u);
      if (mod) {
        jl_pairs8<TERMS, SPEC, true, TAB>(a, s_ew, xi, ti, rjx, rjy, rjz, qj, tj, mi, mm, fi, fjx,
                                          fjy, fjz, band, npairs);
      } else if constexpr (TAB) {
        float2 fj[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        bool any = false;
        jl_pairs8_x2<SMEM_LJ>(a, s_ew, W, rjx, rjy, rjz, qj, tj, mi, umax, fi, fj, any);
        fjx = -(fj[0].x + fj[0].y);
        fjy = -(fj[1].x + fj[1].y);
        fjz = -(fj[2].x + fj[2].y);
        // which pairs need the exact test and, when pairs are counted, which
        // were accepted (the packed arithmetic's rounding): counting must not
        // change the arithmetic of the forces
        if (any || a.count_pairs)
          for (int il = 0; il < 8; il++) {
            const float4 x = xi[il];
            const float dx = x.x - rjx, dy = x.y - rjy, dz = x.z - rjz;
            const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
            const bool act =
                __float_as_uint(r2) - (kEwTabBase << (23 - kEwTabSubBits)) <= umax;
            if (!((mi >> il) & 1u)) continue;
            npairs += act;
            if (!act && r2 <= a.max_hi) band |= 1u << il;
          }
      } else {
        jl_pairs8<TERMS, SPEC, false, TAB>(a, s_ew, xi, ti, rjx, rjy, rjz, qj, tj, mi, mm, fi,
                                           fjx, fjy, fjz, band, npairs);
      }
      // pairs within the rounding band of the cutoff: the exact FP64 test
      // (rare; their i forces go out as atomics, so this path keeps none of
      // the register-held sums live)
      if (__any_sync(kAll, band != 0u)) {
        const int oj = band ? a.sorted[jslot] : -1;
        while (band) {
          const int il = __ffs(band) - 1;
          band &= band - 1u;
          const float4 x = xi[il];
          const float dx = rjx - x.x, dy = rjy - x.y, dz = rjz - x.z;
          const float r2 = dx * dx + dy * dy + dz * dz;
          if (exact_r2(a, W.oi[il], oj, (double)dx, (double)dy, (double)dz) > a.max_cut2)
            continue;
          const float4 p = __ldg(a.lj32 + ti[il] + tj);
          const float f = pair_force_p<float, TERMS, SPEC, true>(a, p, r2, x.w * qj,
                                                                 (mm >> il) & 1u);
          fjx = fmaf(dx, f, fjx);
          fjy = fmaf(dy, f, fjy);
          fjz = fmaf(dz, f, fjz);
          long long *di = a.fslot + 8 * ci + il;
          red_add(di, fixed_force(-dx * f));
          red_add(di + a.ns, fixed_force(-dy * f));
          red_add(di + 2 * (size_t)a.ns, fixed_force(-dz * f));
          npairs++;
        }
      }
      if (mi) {
        long long *dst = a.fslot + jslot;
        red_add(dst, fixed_force(fjx));
        red_add(dst + a.ns, fixed_force(fjy));
        red_add(dst + 2 * (size_t)a.ns, fixed_force(fjz));
      }
    }
    cp_async_wait<0>();  // no copy of this item is left in flight
    // the i forces summed over the lanes: lane l ends with the totals of i
    // atom (l >> 2) & 7 and writes component l & 3
    float sum[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = k & 1 ? fi[k >> 1][c].y : fi[k >> 1][c].x;
      sum[c] = warp_tsum8(v, lane);
    }
    const int il = (lane >> 2) & 7, comp = lane & 3;
    if (comp < 3 && W.oi[il] >= 0)
      red_add(&a.fslot[(size_t)comp * a.ns + 8 * ci + il],
              fixed_force(comp == 0 ? sum[0] : (comp == 1 ? sum[1] : sum[2])));
  }
  if (a.count_pairs) {
    const int np = warp_sum(npairs);
    if (lane == 0) red_add(&a.acc[ACC_PAIRS], (long long)np);
  }
}

template <int TERMS, typename SPEC, bool SMEM_LJ, bool TAB>
__global__ void __launch_bounds__(kJlWarps * 32, 3) k_pairs_jl(PairArgs<float> a) {
  pairs_jl_body<TERMS, SPEC, SMEM_LJ, TAB>(a, own_blk());
}

template <int TERMS, typename SPEC, bool SMEM_LJ, bool TAB>
__global__ void __launch_bounds__(kJlWarps * 32, 3)
    k_pairs_jl_batch(const PairArgs<float> *__restrict__ tab, const int *__restrict__ first,
                     int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(PairArgs<float>)];
  const int m = batch_member(first, nm, blockIdx.x);
  pairs_jl_body<TERMS, SPEC, SMEM_LJ, TAB>(batch_args_shared(tab, m, raw),
                                           batch_blk(first, m));
}

// ---------------------------------------------------------------------------
// FP64 energies (and virial) of the mixed-precision path, j atoms on the
// lanes, accepted pairs compacted.
//
// A warp takes an (i cluster, share of its j-lane entries) item as
// k_pairs_jl does.  Per 32 entries each lane tests its j atom against the
// cluster's 8 i atoms (FP64 squared distances, the reference's exact test
// within a rounding band of a cutoff) and appends the accepted pairs to the
// warp's queue in shared memory; whole batches of 32 queued pairs are then
// evaluated, one per lane.  A third of the tested pairs lie inside the
// cutoff, so the FP64 terms (a square root, an exponential, the switches)
// run on full warps instead of a third of their lanes, and the reciprocal
// and the square root share one Newton iteration.  FP64 issue bounds the
// kernel.  Against one pair per lane of a tile with run-time switches:
// 49,998 atoms, LJ C2 + Ewald, energies: 488 -> 157 us; 648 atoms, LJ C2 +
// Coulomb C1: 37 -> 10 us; 12,000 atoms, Cn at 10 A, energies and virial:
// 650 us with the forces -> 117 us, and 115 us for the forces.
constexpr int kE64Warps = 8;
constexpr int kE64Queue = 32 + 256;  // pairs left over + pairs of one warp step
template <bool VIRIAL>
struct E64Queue {
  double r2[kE64Queue], qq[kE64Queue];
  double d[VIRIAL ? 3 : 1][VIRIAL ? kE64Queue : 1];
  uint2 code[kE64Queue];  // LJ table index; kQ* flags
};
template <bool VIRIAL>
struct E64Warp {
  E64Queue<VIRIAL> q;
  double4 wi[8];  // the cluster's atoms
  int ti[8], oi[8];
};

// 1 / sqrt(x) in FP64: the hardware's 20-bit estimate and two Newton steps
// y += y (1 - x y^2) / 2, each of which doubles the correct bits; within two
// units in the last place for normal x.
__device__ __forceinline__ double rsqrt_newton(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x * y, y, 1.0);
  y = fma(0.5 * y, e, y);
  e = fma(-x * y, y, 1.0);
  return fma(0.5 * y, e, y);
}
// 1 / x the same way, y += y (1 - x y).
__device__ __forceinline__ double rcp_newton(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// Value and, when DER, derivative over the distance of switch KIND at an
// accepted pair (r2 within the cutoff), 1/r at hand.
template <int KIND, bool DER>
__device__ __forceinline__ void switch64(const SwitchDev<double> &w, double r2, double rinv,
                                         double &val, double &der) {
  der = 0.0;
  val = 1.0;
  if (KIND == PMGPU_SW_C2) {
    if (r2 >= w.switchon2) {
      const double c2 = w.cutoff2 - r2, c4 = c2 * (w.s2 + 2.0 * r2);
      val = w.s1 * (c2 * c4);
      if (DER) der = w.s3 * (c2 * c2 - c4);
    }
  } else if (KIND == PMGPU_SW_C1) {
    const double d = r2 * rinv;
    val = 1.0 - d * (w.c1a - r2 * w.c1b);
    if (DER) der = -w.c1a * rinv + d * w.c1c;
  } else if (KIND < 0) {
    switch_eval<double>(w, r2, val, der);
  }
}

template <int TERMS, bool VIRIAL, int LJK, int CK>
__device__ __forceinline__ void pairs_e64_body(const PairArgs<float> &a, Blk blk,
                                               E64Warp<VIRIAL> *warps) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  E64Warp<VIRIAL> &W = warps[wib];
  constexpr int kAllTerms = ((TERMS & TERM_LJ) ? kQLJ : 0) | ((TERMS & TERM_COUL) ? kQCoul : 0) |
                            ((TERMS & TERM_EWALD) ? kQEwald : 0);
  double Elj = 0, Ec = 0, V[6] = {0, 0, 0, 0, 0, 0};
  int npairs = 0, queued = 0;  // (queued: the same in every lane)

  // energies of the queued pair k
  auto evaluate = [&](int k) {
    const double r2 = W.q.r2[k];
    double qq = W.q.qq[k];
    const uint2 code = W.q.code[k];
    const bool modified = code.y & kQModified;
    const double rinv = rsqrt_newton(r2), rr2 = rinv * rinv;
    double f = 0.0;
    if ((TERMS & TERM_LJ) && (code.y & kQLJ)) {
      const double2 *tab = reinterpret_cast<const double2 *>(a.lj64 + code.x);
      const double2 p = __ldg(tab + (modified ? 1 : 0));  // A, B or A14, B14
      const double r6 = rr2 * rr2 * rr2, r6B = p.y * r6, r12A = p.x * r6 * r6;
      double en = r12A - r6B, ff = VIRIAL ? (12.0 * r12A - 6.0 * r6B) * rr2 : 0.0;
      if (LJK >= 0 || a.lj_modify) {
        double sv, sd;
        switch64<LJK, VIRIAL>(a.lj_sw64, r2, rinv, sv, sd);
        if (VIRIAL) ff = ff * sv - en * sd;
        en *= sv;
      }
      Elj += en;
      f += ff;
    }
    if (modified) qq *= a.csf64;
    if ((TERMS & TERM_COUL) && (code.y & kQCoul)) {
      double en = qq * rinv, ff = VIRIAL ? en * rr2 : 0.0;
      if (CK >= 0 || a.coul_modify) {
        double sv, sd;
        switch64<CK, VIRIAL>(a.coul_sw64, r2, rinv, sv, sd);
        if (VIRIAL) ff = ff * sv - en * sd;
        en *= sv;
      }
      Ec += en;
      f += ff;
    }
    if ((TERMS & TERM_EWALD) && (code.y & kQEwald)) {
      const double ar = a.alpha64 * (r2 * rinv), ee = qq * exp(-ar * ar);
      double en;
      if (!a.exact_erf) {
        // A&S 7.1.26 (MathUtilities.cpp:39-49), as poly5
        const double t = rcp_newton(1.0 + 0.3275911 * ar);
        en = t * (0.254829592 +
                  t * (-0.284496736 +
                       t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * ee * rinv;
      } else {
        en = qq * erfc(ar) * rinv;
      }
      Ec += en;
      if (VIRIAL) f += (en + a.a2pi64 * ee) * rr2;
    }
    if constexpr (VIRIAL) {
      // addVirial(fij, d) with fij = d * f (each pair is listed once)
      const double x = W.q.d[0][k], y = W.q.d[1][k], z = W.q.d[2][k];
      const double fx = x * f, fy = y * f;
      V[0] += x * fx; V[1] += y * fx; V[2] += z * fx;
      V[3] += y * fy; V[4] += z * fy; V[5] += z * (z * f);
    }
    npairs++;
  };

  const int nitems = a.nclusters * a.splits;
  const size_t rowcap = 4 * (size_t)a.cap;
  for (int gw = blk.x * kE64Warps + wib; gw < nitems; gw += blk.n * kE64Warps) {
    const int ci = gw / a.splits, sp = gw - ci * a.splits;
    const int4 c4 = *reinterpret_cast<const int4 *>(a.jl_count + kRowParts * ci);
    const int p1 = c4.x, p2 = p1 + c4.y, p3 = p2 + c4.z, cnt = p3 + c4.w;
    const int t0 = (int)((long long)cnt * sp / a.splits);
    const int t1 = (int)((long long)cnt * (sp + 1) / a.splits);
    if (t1 <= t0) continue;
    __syncwarp();  // the previous item's reads of the cluster are done
    if (lane < 8) {
      const int islot = 8 * ci + lane, oi = a.sorted[islot];
      W.wi[lane] = a.xw[islot];
      W.ti[lane] = (oi >= 0 ? __float_as_int(__ldg(&a.xlo[islot].w)) : 0) * a.ntypes;
      W.oi[lane] = oi;
    }
    __syncwarp();
    auto entry_at = [&](int idx) -> uint2 {
      if (idx >= t1) return make_uint2(0u, 0u);  // mask 0: no entry
      const int p = (idx >= p1) + (idx >= p2) + (idx >= p3);
      const int off = idx - (p == 0 ? 0 : (p == 1 ? p1 : (p == 2 ? p2 : p3)));
      return __ldg(a.jlanes + (size_t)(kRowParts * ci + p) * rowcap + off);
    };
    // the next step's entry and j record are loaded while this one runs
    uint2 next = entry_at(t0 + lane);
    double4 wnext = make_double4(0, 0, 0, 0);
    int tnext = 0;
    auto fetch = [&]() {
      if (next.y & 0xFFu) {
        const int js = (int)(next.x & kJSlotMask);
        wnext = a.xw[js];
        tnext = __float_as_int(__ldg(&a.xlo[js].w));
      }
    };
    fetch();
    for (int b0 = t0; b0 < t1; b0 += 32) {
      const uint2 e = next;
      const double4 wj = wnext;
      const int tj = tnext;
      next = entry_at(b0 + 32 + lane);
      fetch();
      const unsigned mi = e.y & 0xFFu, mm = (e.y >> 8) & 0xFFu;
      // the j atom in the entry's image (d = xj + s L - xi)
      const int sh = (int)(e.x >> kJSlotBits);
      const double jx = wj.x + ((sh & 3) - 1) * a.box.e[0];
      const double jy = wj.y + (((sh >> 2) & 3) - 1) * a.box.e[1];
      const double jz = wj.z + (((sh >> 4) & 3) - 1) * a.box.e[2];
      // accepted pairs of this lane and, when the terms' cutoffs differ or
      // only the minimal image counts, each one's terms (4 bits a pair)
      unsigned acc = 0u, terms = 0u;
#pragma unroll
      for (int il = 0; il < 8; il++) {
        const double4 wi = W.wi[il];
        const double dx = jx - wi.x, dy = jy - wi.y, dz = jz - wi.z;
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (!((mi >> il) & 1u) || r2 > a.max_cut2 * (1.0 + kBand64)) continue;
        int flags = 0;
        bool band = false;
        if (a.same_cut) {
          if (r2 <= a.max_cut2 * (1.0 - kBand64)) flags = kAllTerms;
          else band = true;
        } else {
          if (TERMS & TERM_LJ) {
            if (r2 <= a.lj_cut2 * (1.0 - kBand64)) flags |= kQLJ;
            else band |= r2 <= a.lj_cut2 * (1.0 + kBand64);
          }
          if (TERMS & TERM_COUL) {
            if (r2 <= a.coul_cut2 * (1.0 - kBand64)) flags |= kQCoul;
            else band |= r2 <= a.coul_cut2 * (1.0 + kBand64);
          }
          if (TERMS & TERM_EWALD) {
            if (r2 <= a.ew_cut2 * (1.0 - kBand64)) flags |= kQEwald;
            else band |= r2 <= a.ew_cut2 * (1.0 + kBand64);
          }
        }
        if (band) {  // rare: the reference's own arithmetic decides
          const double x = exact_r2(a, W.oi[il], a.sorted[e.x & kJSlotMask], dx, dy, dz);
          if ((TERMS & TERM_LJ) && x <= a.lj_cut2) flags |= kQLJ;
          if ((TERMS & TERM_COUL) && x <= a.coul_cut2) flags |= kQCoul;
          if ((TERMS & TERM_EWALD) && x <= a.ew_cut2) flags |= kQEwald;
        }
        // boxes below twice the cutoff: cutoff terms take the minimal image
        if ((TERMS & (TERM_LJ | TERM_COUL)) && a.minimal_image &&
            !(fabs(dx) <= a.box.H2[0] && fabs(dy) <= a.box.H2[1] && fabs(dz) <= a.box.H2[2]))
          flags &= ~(kQLJ | kQCoul);
        if (flags) {
          acc |= 1u << il;
          terms |= (unsigned)flags << (4 * il);
        }
      }
      // this lane's place in the queue: an exclusive scan of the counts
      const int n = __popc(acc);
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += t;
      }
      int at = queued + incl - n;
      queued += __shfl_sync(kAll, incl, 31);
      while (acc) {
        const int il = __ffs(acc) - 1;
        acc &= acc - 1u;
        const double4 wi = W.wi[il];
        const double dx = jx - wi.x, dy = jy - wi.y, dz = jz - wi.z;
        W.q.r2[at] = dx * dx + dy * dy + dz * dz;
        W.q.qq[at] = wi.w * wj.w;
        if constexpr (VIRIAL) {
          W.q.d[0][at] = dx;
          W.q.d[1][at] = dy;
          W.q.d[2][at] = dz;
        }
        W.q.code[at] = make_uint2((unsigned)(W.ti[il] + tj),
                                  ((terms >> (4 * il)) & 7u) | (((mm >> il) & 1u) ? kQModified : 0));
        at++;
      }
      __syncwarp();
      while (queued >= 32) {
        queued -= 32;
        evaluate(queued + lane);
      }
      __syncwarp();  // the next step appends after the reads
    }
  }
  if (lane < queued) evaluate(lane);
  const int np = warp_sum(npairs);
  if (lane == 0) red_add(&a.acc[ACC_PAIRS], (long long)np);
  const double v[8] = {Elj, Ec, V[0], V[1], V[2], V[3], V[4], V[5]};
  block_energies<TERMS, VIRIAL, kE64Warps>(a.acc, v);
}

extern __shared__ __align__(16) unsigned char e64_smem[];

template <int TERMS, bool VIRIAL, int LJK, int CK>
__global__ void __launch_bounds__(kE64Warps * 32, 2) k_pairs_e64(PairArgs<float> a) {
  pairs_e64_body<TERMS, VIRIAL, LJK, CK>(a, own_blk(),
                                         reinterpret_cast<E64Warp<VIRIAL> *>(e64_smem));
}
template <int TERMS, bool VIRIAL, int LJK, int CK>
__global__ void __launch_bounds__(kE64Warps * 32, 2)
    k_pairs_e64_batch(const PairArgs<float> *__restrict__ tab, const int *__restrict__ first,
                      int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(PairArgs<float>)];
  const int m = batch_member(first, nm, blockIdx.x);
  pairs_e64_body<TERMS, VIRIAL, LJK, CK>(batch_args_shared(tab, m, raw), batch_blk(first, m),
                                         reinterpret_cast<E64Warp<VIRIAL> *>(e64_smem));
}

// Adds the forces accumulated by list slot into the atoms' forces and
// clears the slot buffer for the next launch.
struct SlotArgs {
  int ns, n;
  const int *sorted;
  long long *fslot, *force;
};
__device__ __forceinline__ void slot_forces_body(const SlotArgs &A, Blk b) {
  const int ns = A.ns, n = A.n;
  const int *__restrict__ sorted = A.sorted;
  long long *__restrict__ fslot = A.fslot;
  long long *__restrict__ force = A.force;
  const int s = b.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  const int i = sorted[s];
  if (i < 0) return;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const long long v = fslot[(size_t)c * ns + s];
    if (v) {
      red_add(&force[(size_t)c * n + i], v);
      fslot[(size_t)c * ns + s] = 0;
    }
  }
}
__global__ void k_slot_forces(SlotArgs a) {
  pdl_wait();  // the predecessor's writes are visible from here on
  slot_forces_body(a, own_blk());
}
__global__ void k_slot_forces_batch(const SlotArgs *__restrict__ tab, const int *__restrict__ first,
                                    int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  slot_forces_body(tab[m], batch_blk(first, m));
}

}  // namespace pmgpu
