// kernels_mol.cu -- per-molecule solute-solvent energies, fused with the binning.
//
// For every placement of the batch and solvent molecule (a "slot" of the frame's spatially
// sorted order):
//   recip   sum over its sites of q * sum_{c1,c2,c3} theta theta theta phi(g - c)
//           (recpcal_energy, recpcal.F90:451-502), phi being the solute's PME potential;
//   real    LJ (4 switch forms) + q q erfc(beta r) / r against every solute site within
//           the cutoffs (get_pair_energy_block, realcal.F90:585-784), entered only when
//           the molecule is inside the solute's bounding sphere + cutoff, so the cell
//           list of the reference (realcal.F90:373-582) is not needed;
//   resid   -pi Q_u Q_j / (beta^2 V) (residual_ene, engproc.F90:859-869);
// then the total u = real + (resid + recip) (get_uv_energy, engproc.F90:736-753) is binned
// exactly as getiduv/binsearch do (engproc.F90:927-1020), with integer keys, into the
// placement's histogram (insdst, engproc.F90:813-830).  Per-species sum/min/max go to
// per-block partials reduced in a fixed tree, so every result is run-to-run deterministic.
//
// Mixed path: the gather, then a thread per molecule and up to 8 placements; fixed-point
// positions, FP32 pair terms and grid gather, float-float totals, block histograms in shared
// memory.  FP64 path: 4 or 16 threads per molecule and placement, everything in FP64 with the
// reference's formulas, counts straight into the batch's histograms.
#include <cub/device/device_radix_sort.cuh>

#include "async_copy.cuh"
#include "engine.cuh"

namespace ermod {

struct LjK {  // switching constants (realcal.F90:629-642, 888-904)
  float lw2, up2, lw3, up3, lw6, up6, repA, repB, repC, attA, attB, attC, lw, up, ele2, den3;
};
// the same in FP64 (the FP64 path, and the mixed path's FP64 pair terms)
struct LjK64 {
  double lw2, up2, lw3, up3, lw6, up6, repA, repB, repC, attA, attB, attC, lw, up, ele2;
};

struct MolArgs {
  // frame, slot order
  const int4* site_pos;
  const float4* site_rec;
  const int* site_grid;
  const double* site_x;
  const double* site_w;
  const double* site_q;
  const int* slot_mol;
  const int* slot_site;
  const int* slot_species;
  const double* slot_qmol;
  const float* frame_scal;
  const int* mol_to_k;
  int slvmax, nummol;
  int max_mol_sites;  // of the solvent molecules
  // LJ tables
  const double* ljene;
  const double* ljlensq;
  const float* ljene_f;
  const float* ljlensq_f;
  int T;
  int ldb;  // interleave stride of the mixed potential grids (placements per grid point)
  // energy coordinate
  const long long* uvkey;
  const int* uvkey_f;  // 32-bit keys of the edges rounded down to floats (FP32 totals)
  const int* spec;  // [numslv][3]
  int numslv, ermax, soln, mbin_mode;  // mbin_mode: 0 off, 1 error, 2 flag only
  int hist_global;  // finish kernel: histogram atomics straight into global memory (large ermax)
  // interaction parameters
  FrameGeom g;
  int ljswitch;
  double elecut, lwljcut, upljcut, screen;
  // FP32 constants of the mixed kernels, computed on the host
  float fxf[3];    // fixed-point unit per axis (box length / 2^32)
  float screen_f;  // Ewald beta
  float rc_f;      // max(elecut, upljcut)
  float fx_scale_f;  // finish kernel: 2^bits of the fixed-point sums of FP32 pair terms
  float reach2_f;    // finish kernel: the larger squared cutoff of LJ and Coulomb
  int bare;        // cltype 0: bare Coulomb within elecut (no cutoff when non-periodic), no reciprocal space
                   // or residual
  LjK k32;         // LJ switching constants
  LjK64 k64;
  double resid_fac;  // pi / screen^2 / volume
  // batch
  BatchArgs a;
  int ntile;
  DevStatus* status;
};

namespace {

template <typename T>
__device__ __forceinline__ T lj_low(int sw, const LjK& k, T eps, T sg2, T dist) {
  const T invr2 = sg2 / dist;
  const T invr6 = invr2 * invr2 * invr2;
  if (sw <= 1) return T(4) * eps * invr6 * (invr6 - T(1));
  const T s6 = sg2 * sg2 * sg2;
  if (sw == 2) {
    const T vdwa = invr6 * invr6 - s6 * s6 / (T(k.lw6) * T(k.up6));
    const T vdwb = invr6 - s6 / (T(k.lw3) * T(k.up3));
    return T(4) * eps * (vdwa - vdwb);
  }
  const T vdwa = invr6 * invr6 - s6 * s6 * T(k.repC);
  const T vdwb = invr6 - s6 * T(k.attC);
  return T(4) * eps * (vdwa - vdwb);
}

template <typename T>
__device__ __forceinline__ T lj_switch(int sw, const LjK& k, T eps, T sg2, T dist) {
  const T invr2 = sg2 / dist;
  const T invr6 = invr2 * invr2 * invr2;
  if (sw == 0) {
    const T dd = dist - T(k.up2), den = T(k.up2) - T(k.lw2);
    return T(4) * eps * invr6 * (invr6 - T(1)) * (T(2) * dist + T(k.up2) - T(3) * T(k.lw2)) * (dd * dd) /
           (den * den * den);
  }
  if (sw == 1) {
    const T swfac = (sqrt(dist) - T(k.lw)) / (T(k.up) - T(k.lw));
    const T s3 = swfac * swfac * swfac, s4 = s3 * swfac, s5 = s4 * swfac;
    return T(4) * eps * invr6 * (invr6 - T(1)) * (T(1) - T(10) * s3 + T(15) * s4 - T(6) * s5);
  }
  const T s6 = sg2 * sg2 * sg2;
  if (sw == 2) {
    const T invr3 = sqrt(invr6), s3 = sqrt(s6);
    const T a = invr6 - s6 / T(k.up6), b = invr3 - s3 / T(k.up3);
    const T vdwa = T(k.up6) / (T(k.up6) - T(k.lw6)) * (a * a);
    const T vdwb = T(k.up3) / (T(k.up3) - T(k.lw3)) * (b * b);
    return T(4) * eps * (vdwa - vdwb);
  }
  const T swfac = sqrt(dist) - T(k.lw);
  const T f3 = swfac * swfac * swfac, f4 = f3 * swfac;
  const T vdwa = invr6 * invr6 - s6 * s6 * (T(k.repA) * f3 + T(k.repB) * f4 + T(k.repC));
  const T vdwb = invr6 - s6 * (T(k.attA) * f3 + T(k.attB) * f4 + T(k.attC));
  return T(4) * eps * (vdwa - vdwb);
}

__device__ __forceinline__ double lj_low64(int sw, const LjK64& k, double eps, double sg2, double dist) {
  const double invr2 = sg2 / dist;
  const double invr6 = invr2 * invr2 * invr2;
  if (sw <= 1) return 4.0 * eps * invr6 * (invr6 - 1.0);
  const double s6 = sg2 * sg2 * sg2;
  if (sw == 2) {
    const double vdwa = invr6 * invr6 - s6 * s6 / (k.lw6 * k.up6);
    const double vdwb = invr6 - s6 / (k.lw3 * k.up3);
    return 4.0 * eps * (vdwa - vdwb);
  }
  const double vdwa = invr6 * invr6 - s6 * s6 * k.repC;
  const double vdwb = invr6 - s6 * k.attC;
  return 4.0 * eps * (vdwa - vdwb);
}

__device__ __forceinline__ double lj_switch64(int sw, const LjK64& k, double eps, double sg2, double dist) {
  const double invr2 = sg2 / dist;
  const double invr6 = invr2 * invr2 * invr2;
  if (sw == 0) {
    const double dd = dist - k.up2, den = k.up2 - k.lw2;
    return 4.0 * eps * invr6 * (invr6 - 1.0) * (2.0 * dist + k.up2 - 3.0 * k.lw2) * (dd * dd) / (den * den * den);
  }
  if (sw == 1) {
    const double swfac = (sqrt(dist) - k.lw) / (k.up - k.lw);
    const double s3 = swfac * swfac * swfac, s4 = s3 * swfac, s5 = s4 * swfac;
    return 4.0 * eps * invr6 * (invr6 - 1.0) * (1.0 - 10.0 * s3 + 15.0 * s4 - 6.0 * s5);
  }
  const double s6 = sg2 * sg2 * sg2;
  if (sw == 2) {
    const double invr3 = sqrt(invr6), s3 = sqrt(s6);
    const double a = invr6 - s6 / k.up6, b = invr3 - s3 / k.up3;
    const double vdwa = k.up6 / (k.up6 - k.lw6) * (a * a);
    const double vdwb = k.up3 / (k.up3 - k.lw3) * (b * b);
    return 4.0 * eps * (vdwa - vdwb);
  }
  const double swfac = sqrt(dist) - k.lw;
  const double f3 = swfac * swfac * swfac, f4 = f3 * swfac;
  const double vdwa = invr6 * invr6 - s6 * s6 * (k.repA * f3 + k.repB * f4 + k.repC);
  const double vdwb = invr6 - s6 * (k.attA * f3 + k.attB * f4 + k.attC);
  return 4.0 * eps * (vdwa - vdwb);
}

__host__ __device__ __forceinline__ void gmx_params(int pw, double lw, double up, double& A, double& B, double& C) {
  const double df = up - lw;
  double upp2 = 1.0, upp = 1.0;
  for (int i = 0; i < pw + 2; ++i) upp2 *= up;
  for (int i = 0; i < pw; ++i) upp *= up;
  A = -(double)pw * ((double)(pw + 4) * up - (double)(pw + 1) * lw) / (upp2 * (df * df)) / 3.0;
  B = (double)pw * ((double)(pw + 3) * up - (double)(pw + 1) * lw) / (upp2 * (df * df * df)) / 4.0;
  C = 1.0 / upp - A * (df * df * df) - B * (df * df * df * df);
}

__host__ __device__ __forceinline__ LjK64 make_k64(const MolArgs& A) {
  LjK64 k;
  k.lw = A.lwljcut;
  k.up = A.upljcut;
  k.lw2 = A.lwljcut * A.lwljcut;
  k.up2 = A.upljcut * A.upljcut;
  k.lw3 = A.lwljcut * A.lwljcut * A.lwljcut;
  k.up3 = A.upljcut * A.upljcut * A.upljcut;
  k.lw6 = k.lw3 * k.lw3;
  k.up6 = k.up3 * k.up3;
  gmx_params(12, A.lwljcut, A.upljcut, k.repA, k.repB, k.repC);
  gmx_params(6, A.lwljcut, A.upljcut, k.attA, k.attB, k.attC);
  k.ele2 = A.elecut * A.elecut;
  return k;
}

__host__ __device__ __forceinline__ LjK to_f32(const LjK64& d) {
  LjK k;
  k.lw2 = (float)d.lw2; k.up2 = (float)d.up2; k.lw3 = (float)d.lw3; k.up3 = (float)d.up3;
  k.lw6 = (float)d.lw6; k.up6 = (float)d.up6; k.repA = (float)d.repA; k.repB = (float)d.repB;
  k.repC = (float)d.repC; k.attA = (float)d.attA; k.attB = (float)d.attB; k.attC = (float)d.attC;
  k.lw = (float)d.lw; k.up = (float)d.up; k.ele2 = (float)d.ele2; k.den3 = 0.f;
  return k;
}

__device__ __forceinline__ int wrapi(int x, int K) {
  if (x < 0) x += K;
  if (x >= K) x -= K;
  return x;
}

__device__ __forceinline__ double key_to_double(long long k) {
  k = k ^ ((k >> 63) & 0x7fffffffffffffffll);
  return __longlong_as_double(k);
}


// getiduv / binsearch for one molecule: returns the status code (0 = binned) and ret,
// the count of edges strictly below u (bin = sp_off + ret - 1).
__device__ __forceinline__ int bin_molecule(const MolArgs& A, double u, int species, int sp_off, int sp_n,
                                            int sp_soft, int& ret) {
  ret = 0;
  if (species < 1 || species > A.numslv) return ERMOD_E_ENG_CNS;
  if (u != u) return ERMOD_E_ENG_MIN;
  const long long ku = ordered_key(u);
  const long long* keys = A.uvkey + sp_off;
  int lo = 0, hi = sp_n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(keys + mid) < ku)
      lo = mid + 1;
    else
      hi = mid;
  }
  ret = lo;
  if (ret <= 0) return ERMOD_E_ENG_MIN;
  if (A.soln && ret > sp_soft) return ERMOD_E_ENG_SFT;
  if (ret == sp_n && u < 1.0e3 && A.mbin_mode != 0) {
    if (A.mbin_mode == 1) return ERMOD_W_MBIN;
    atomicOr(&A.status->mbin_hit, 1);
  }
  return 0;
}

// warp-aggregated shared-memory histogram increment
__device__ __forceinline__ void hist_add(int* h, int bin) {
  const unsigned am = __activemask();
  const unsigned peers = __match_any_sync(am, bin);
  const int leader = __ffs(peers) - 1;
  if ((threadIdx.x & 31) == leader) atomicAdd(&h[bin], __popc(peers));
}

// FP32 pair terms larger than these (kcal/mol) are recomputed in FP64.  Below them an
// FP32 term is within a few units in the last place (the LJ term's sigma^12 amplifies the
// distance's rounding 6-fold; erfcf is within 4 ulp), 5e-6 kcal/mol at most; above them the
// FP32 rounding, and the fixed-point quantisation of the displacement (2.3e-8 A at
// L = 99.5 A), would grow with the term up to the 1e10 kcal/mol of overlapping pairs.
constexpr float kFp64Lj = 8.0f;
constexpr float kFp64Coulomb = 16.0f;
constexpr int kPairLj = 1, kPairCoulomb = 2;  // the parts of a pair evaluated in FP64

// parts of one solute-solvent site pair in FP64, as the FP64 path computes them: minimum
// image of the FP64 wrapped coordinates (realcal.F90:202-209), LJ with the switch form
// (realcal.F90:686-770) and the screened or bare Coulomb term (realcal.F90:771-782, 245)
__device__ __forceinline__ double pair_fp64(const MolArgs& A, int idx, const double* __restrict__ ux, double qu,
                                         int tu, int parts) {
  double dist = 0.0;
  for (int i = 0; i < 3; ++i) {
    const double h = 0.5 * A.g.L[i];
    const double x = fabs(A.site_x[3 * (size_t)idx + i] - ux[i]);
    const double d = A.g.periodic ? h - fabs(h - x) : x;
    dist += d * d;
  }
  const int tv = A.site_pos[idx].w;
  double e = 0.0;
  const double ljeps = A.ljene[tv + A.T * tu];
  if ((parts & kPairLj) && ljeps > 0) {
    const double sg2 = A.ljlensq[tv + A.T * tu];
    if (dist <= A.k64.lw2)
      e += lj_low64(A.ljswitch, A.k64, ljeps, sg2, dist);
    else if (dist <= A.k64.up2)
      e += lj_switch64(A.ljswitch, A.k64, ljeps, sg2, dist);
  }
  if (parts & kPairCoulomb) {
    if (A.bare) {
      if (dist < A.k64.ele2) e += qu * A.site_q[idx] / sqrt(dist);
    } else if (dist <= A.k64.ele2) {
      const double r = sqrt(dist);
      e += qu * A.site_q[idx] * (1.0 - erf(A.screen * r)) / r;
    }
  }
  return e;
}

// ---- the finish kernel's real-space pass -------------------------------------------------
// Its FP64 pairs are gathered in a list per block; more than that many and each item's thread
// finds its own again.
constexpr int kBigList = 1024;
// a pair: near item (11 bits: at most 8 placements of 256 molecules), solute site (8 bits), site
// of the solvent molecule within a window of 8,192 (13 bits); the pass takes larger molecules
// window by window
constexpr int kSiteWindowBits = 13;
constexpr int kListWindows = 64;  // windows that a listed pair's byte holds beside its FP64 parts
__device__ __forceinline__ unsigned pair_key(int near, int su, int s) {
  return ((unsigned)near << 21) | ((unsigned)su << kSiteWindowBits) | (unsigned)s;
}
// Solutes of at least this many sites take the stage that drops an item's solute sites too far
// from the whole molecule.  256 insertions of 36 sites into 2,000 waters: 309 us without it, 243
// with it (4,000 of them 13.3 and 12.5 ms); 12 sites into 33,000 waters the same; 6 sites into
// 4,000 waters, two thirds of whose items pass, 1% slower with it.
constexpr int kTwoStageSites = 16;
constexpr int kPairQueue = 64;  // entries waiting in one of a warp's two queues: at most 31 + 32
// the pass's scratch (ints): the list (values, pairs, their order as 16 bits, their FP64 parts as
// bytes), the warps' queues, the fixed-point sums of the near items, the molecules' first
// sites, and the list of near (molecule, placement) items (16 bits)
__host__ __device__ constexpr int finish_scratch_ints(int G, bool two) {  // for the larger tile, 256
  return 2 * kBigList + kBigList + kBigList / 2 + kBigList / 4 + (two ? 2 : 1) * 8 * kPairQueue + 2 * 256 * G + 256 +
         G * 256 / 2;
}
// the dynamic shared memory of the finish kernel before its edge keys: the block
// histograms (when in shared memory) or the real-space pass's scratch, whichever is larger
__host__ __device__ constexpr int finish_region_ints(int G, bool two, int ermax, int hist_global) {
  const int h = hist_global ? 0 : G * ermax;
  return h > finish_scratch_ints(G, two) ? h : finish_scratch_ints(G, two);
}

// its dynamic shared memory in bytes, and an upper bound of its static one (the totals of 256 molecules)
constexpr size_t finish_smem(int G, bool two, int ermax, int hist_global) {
  return sizeof(int) * ((size_t)finish_region_ints(G, two, ermax, hist_global) + ermax);
}
constexpr size_t finish_static_smem(int G) { return 2112 * (size_t)G + 512; }
constexpr size_t kMaxSmem = 227 * 1024;  // per block

__device__ __forceinline__ float pair_r2(const MolArgs& A, const int4& vp, const int4& up) {
  const float ex = (float)(int)((unsigned)vp.x - (unsigned)up.x) * A.fxf[0];
  const float ey = (float)(int)((unsigned)vp.y - (unsigned)up.y) * A.fxf[1];
  const float ez = (float)(int)((unsigned)vp.z - (unsigned)up.z) * A.fxf[2];
  return ex * ex + ey * ey + ez * ez;
}

// a squared distance in FP32 above this is beyond r2 in FP64 too (the fixed-point and FP32
// roundings are below 1e-6 of it)
__device__ __forceinline__ float margin_r2(float r2) { return r2 * 1.0001f + 1e-3f; }

// the FP32 terms of one pair at squared distance r2: LJ (0 beyond its cutoff) and screened or
// bare Coulomb; returns the parts too large for FP32 (above kFp64Lj / kFp64Coulomb in
// magnitude, or not finite: the comparisons are false for NaN and inf)
__device__ __forceinline__ int pair_fp32(const MolArgs& A, const int4& vp, const int4& up, float qu, float qv, float r2,
                                         float& elj, float& eco) {
  const LjK& k32 = A.k32;
  elj = 0.f;
  eco = 0.f;
  const float ljeps = A.ljene_f[vp.w + A.T * up.w];
  if (ljeps > 0.f) {
    const float sg2 = A.ljlensq_f[vp.w + A.T * up.w];
    if (r2 <= k32.lw2)
      elj = lj_low<float>(A.ljswitch, k32, ljeps, sg2, r2);
    else if (r2 <= k32.up2)
      elj = lj_switch<float>(A.ljswitch, k32, ljeps, sg2, r2);
  }
  if (A.bare) {
    if (r2 < k32.ele2) eco = qu * qv / sqrtf(r2);  // realcal_bare
  } else if (r2 <= k32.ele2) {
    const float r = sqrtf(r2);
    eco = qu * qv * erfcf(A.screen_f * r) / r;
  }
  return (fabsf(elj) <= kFp64Lj ? 0 : kPairLj) | (fabsf(eco) <= kFp64Coulomb ? 0 : kPairCoulomb);
}

// Sums of FP32 terms as integers of 1 / A.fx_scale_f kcal/mol: exact additions, so that the sum does
// not depend on the order in which a block's threads add.  A pair adds an LJ and a Coulomb term, at
// most kFixedTerm together.  Two words, the low one's carry passed on, while they leave the unit at
// 2^-48 kcal/mol or finer for every pair of the largest molecule with a solute (1,365 pairs; 2^-53 for
// water and 12 sites); three words of 2^-58 beyond.  (Float-float sums hold 48 bits.  With a unit of 2^-44
// for water the small terms of distant pairs lost theirs; adding them costs 1% of this kernel at 36
// solute sites, 4.98 -> 5.04 ms of 4,000 insertions into 2,000 waters.)
constexpr float kFixedTerm = kFp64Lj + kFp64Coulomb;
constexpr int kFixedNarrowBits = 48, kFixedWideBits = 58;
static_assert(kFixedTerm < 32.f, "a pair's terms in 63 bits at kFixedWideBits");
__device__ __forceinline__ void fixed_add(unsigned* lo, unsigned* hi, long long v) {
  const unsigned l = (unsigned)v, old = atomicAdd(lo, l);
  atomicAdd(hi, (unsigned)((unsigned long long)v >> 32) + (old + l < old ? 1u : 0u));
}
__device__ __forceinline__ void fixed_add_wide(unsigned* lo, unsigned* hi, unsigned* top, long long v) {
  const unsigned l = (unsigned)v, old = atomicAdd(lo, l), c = old + l < old ? 1u : 0u;
  const unsigned m = (unsigned)((unsigned long long)v >> 32), mc = m + c, oldm = atomicAdd(hi, mc);
  const unsigned t = (v < 0 ? ~0u : 0u) + (mc < m || oldm + mc < oldm ? 1u : 0u);
  if (t) atomicAdd(top, t);
}
__device__ __forceinline__ ff fixed_to_ff(unsigned lo, unsigned hi, float unit) {
  const long long v = (long long)(((unsigned long long)hi << 32) | lo);
  const float h = __ll2float_rn(v);
  return ff{h * unit, __ll2float_rn(v - __float2ll_rn(h)) * unit};
}
// three words: the magnitude's upper and lower 64 bits as doubles (rounded at 53 bits)
__device__ __noinline__ ff fixed_to_ff_wide(unsigned lo, unsigned hi, unsigned top, float unit) {
  unsigned long long v = ((unsigned long long)hi << 32) | lo;
  const bool neg = (int)top < 0;
  if (neg) {
    v = ~v + 1ull;
    top = ~top + (v == 0ull ? 1u : 0u);
  }
  const double x = fma((double)top, 18446744073709551616.0, (double)v) * (double)unit;
  return ff_from_double(neg ? -x : x);
}

constexpr long long kKeyPosInf = 0x7ff0000000000000ll;
constexpr long long kKeyNegInf = (long long)0x800fffffffffffffull;  // ordered key of -inf

// The plain FP64 path: T = 4 TY threads per (solvent molecule, placement).  FP64 runs at 2
// FMA per clock and SM on GB300, a warp instruction taking as long with one active lane as
// with 32, so the work is laid out for full lanes.  Reciprocal part: thread t of a molecule
// takes the stencil columns c1 = t mod 4, + 4, .. (four consecutive doubles of a grid row side
// by side in a warp's load, and 21 FP64 instructions per site instead of 148 for the plain
// triple loop) and the stencil rows c2 = t / 4, + TY, ...  Real space: the warp tests its near
// molecules' pairs, 32 at a time, in FP32 (with a margin: the FP64 distances decide), and
// evaluates those that pass on full warps out of a queue; a molecule's values are added by a
// segmented scan over the queue's order, which is the order of its pairs.  (Each thread
// evaluating its share of all pairs in FP64, half of them beyond the cutoffs, 21.5 of 32 lanes
// active: the FP64 pipe 87% busy for 534 us per 64 placements of 4,000 waters and 801 us per 16
// of 33,000.  200 insertions into 4,000 waters 4.54 -> 3.78 ms, 32 into 33,000 6.23 -> 5.36 ms.)  TY = 1 in reference mode, where the batch fills the GPU; TY = 4 for
// a solution-mode frame of few molecules, whose latency is one molecule's serial chain (mol64_ty).
constexpr int kMol64Threads = 256;
constexpr int kQueue64 = 64;  // pairs waiting in a warp's queue: at most 31 + 32
template <int P, int TY>
__global__ void __launch_bounds__(kMol64Threads) mol_energy_kernel(MolArgs A) {
  constexpr int T = 4 * TY, kMols = kMol64Threads / T, kWarps = kMol64Threads / 32, kWarpMols = 32 / T;
  __shared__ int2 squeue[kWarps][kQueue64];  // {molecule of the warp | solute site << 8, site of the molecule}
  __shared__ double sreal[kMols];
  const int tile = blockIdx.x, b = blockIdx.y;
  const BatchArgs& a = A.a;
  const int sub = threadIdx.x % T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = tile * kMols + threadIdx.x / T;
  const bool valid = m < A.slvmax;
  int k = -1, s0 = 0, ns = 0, species = 0;
  if (valid) {
    k = A.slot_mol[m];
    s0 = A.slot_site[m];
    ns = A.slot_site[m + 1] - s0;
    species = A.slot_species[m];
  }
  const FrameGeom& g = A.g;
  const int K1 = g.K[0], K2 = g.K[1], K3 = g.K[2];
  const int tg = a.tagslt[b] - 1;
  const int kskip = (tg >= 0 && tg < A.nummol) ? A.mol_to_k[tg] : -2;
  // a placement rejected by check_mol_configuration has no molecule (engproc.F90:690-691)
  const bool active = valid && (k != kskip) && !(a.skip && a.skip[b]);
  double recip = 0.0;
  // ---- reciprocal part ----
  if (active && !A.bare) {  // bare Coulomb: no reciprocal part
    const double* phi = a.phi64 + (size_t)b * K1 * K2 * K3;
    for (int s = 0; s < ns; ++s) {
      const int idx = s0 + s;
      const double* w = A.site_w + (size_t)idx * 3 * P;
      const int gp = A.site_grid[idx];
      const int g1 = gp & 1023, g2 = (gp >> 10) & 1023, g3 = (gp >> 20) & 1023;
      double w3[P];
      int z[P];
#pragma unroll
      for (int c3 = 0; c3 < P; ++c3) {
        w3[c3] = w[2 * P + c3];
        z[c3] = wrapi(g3 - c3, K3);
      }
      double site = 0.0;
#pragma unroll
      for (int c1 = sub & 3; c1 < P; c1 += 4) {
        const double* col = phi + wrapi(g1 - c1, K1);
        double line = 0.0;
#pragma unroll
        for (int c2 = sub >> 2; c2 < P; c2 += TY) {
          const double* row = col + (size_t)wrapi(g2 - c2, K2) * K1;
          double t = 0.0;
#pragma unroll
          for (int c3 = 0; c3 < P; ++c3) t = fma(w3[c3], row[(size_t)z[c3] * K1 * K2], t);
          line = fma(w[P + c2], t, line);
        }
        site = fma(w[c1], line, site);
      }
      recip = fma(A.site_q[idx], site, recip);
    }
  }
#pragma unroll
  for (int o = 1; o < T; o <<= 1) recip += __shfl_xor_sync(0xffffffffu, recip, o);  // the T threads' parts
  // ---- real space (every lane of the warp takes part) ----
  const int nu = a.u_nsite[b];
  const size_t ub = (size_t)b * kMaxSoluteSites;
  const float rcut = A.rc_f + a.u_radius[b] + A.frame_scal[0];
  const bool near = active && nu > 0 && !(pair_r2(A, A.site_pos[s0], a.u_pos[ub]) > margin_r2(rcut * rcut));
  if (sub == 0) sreal[threadIdx.x / T] = 0.0;
  __syncwarp();
  unsigned nearm = __ballot_sync(0xffffffffu, near && sub == 0);
  if (nearm) {
    const float reach2 = margin_r2(A.reach2_f);
    int2* queue = squeue[warp];
    int nq = 0;  // warp-uniform
    // the first n pairs of the warp's queue, one per lane; the others move up
    auto evaluate = [&](int n) {
      __syncwarp();
      const bool on = lane < n;
      const int2 e = on ? queue[lane] : make_int2(kWarpMols, 0);
      const int mw = e.x & 0xff, su = e.x >> 8;  // mw = kWarpMols: no pair
      const int site = __shfl_sync(0xffffffffu, s0, (mw * T) & 31) + e.y;
      double v = 0.0;
      if (on)
        v = pair_fp64(A, site, a.u_x + (ub + su) * 3, a.u_q[ub + su], a.u_pos[ub + su].w, kPairLj | kPairCoulomb);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {  // inclusive scan within each molecule's run of lanes
        const double up = __shfl_up_sync(0xffffffffu, v, o);
        const int mo = __shfl_up_sync(0xffffffffu, mw, o);
        if (lane >= o && mo == mw) v += up;
      }
      const int next = __shfl_down_sync(0xffffffffu, mw, 1);
      if (on && (lane == n - 1 || next != mw)) sreal[warp * kWarpMols + mw] += v;
      const int2 rest = lane < nq - n ? queue[n + lane] : make_int2(0, 0);
      __syncwarp();
      if (lane < nq - n) queue[lane] = rest;
      __syncwarp();
      nq -= n;
    };
    const unsigned magic = nu > 1 ? (unsigned)((0x100000000ull + nu - 1) / nu) : 0u;
    for (; nearm; nearm &= nearm - 1) {
      const int owner = __ffs(nearm) - 1, mw = owner / T;
      const int is0 = __shfl_sync(0xffffffffu, s0, owner), ins = __shfl_sync(0xffffffffu, ns, owner);
      // pairs with the solute site fastest (32 x nu pairs, whole solvent sites, at a time keep
      // the division's operand small)
      for (int sb = 0; sb < ins; sb += 32) {
        const int npair = min(32, ins - sb) * nu;
        for (int p0 = 0; p0 < npair; p0 += 32) {
          const int p = p0 + lane;
          const int ds = nu > 1 ? (int)__umulhi((unsigned)p, magic) : p, s = sb + ds, su = p - ds * nu;
          const bool in = p < npair && !(pair_r2(A, A.site_pos[is0 + s], a.u_pos[ub + su]) > reach2);
          const unsigned mask = __ballot_sync(0xffffffffu, in);
          if (in) queue[nq + __popc(mask & ((1u << lane) - 1u))] = make_int2(mw | su << 8, s);
          nq += __popc(mask);
          if (nq >= 32) evaluate(32);
        }
      }
    }
    if (nq > 0) evaluate(nq);
    __syncwarp();
  }
  const bool mine = active && sub == 0;
  double u = 0.0;
  if (valid && sub == 0) {
    if (active) {
      // residual_ene + assembly (engproc.F90:741-752); bare Coulomb has no such term (factor 0)
      const double epcl = A.resid_fac * a.u_qmol[b] * A.slot_qmol[m];
      u = sreal[threadIdx.x / T] + (recip - epcl);
      // ---- getiduv / binsearch ----
      int sp_off = 0, sp_n = 1, sp_soft = 1, ret = 0;
      if (species >= 1 && species <= A.numslv) {
        sp_off = A.spec[3 * (species - 1)];
        sp_n = A.spec[3 * (species - 1) + 1];
        sp_soft = A.spec[3 * (species - 1) + 2];
      }
      const int code = bin_molecule(A, u, species, sp_off, sp_n, sp_soft, ret);
      if (code)
        atomicMin(&A.status->err_key, make_err_key(a.b0 + b, k + 1, code));
      else
        hist_add(a.hist + (size_t)b * A.ermax, sp_off + ret - 1);
    }
    if (a.uvengy_out) a.uvengy_out[(size_t)(a.b0 + b) * (A.slvmax + 1) + k + 1] = u;
  }
  // per-species partials {sum, min, max} of this block: fixed trees over the warps, then the
  // warps in order
  __shared__ double wsum[kWarps];
  __shared__ long long wmin[kWarps], wmax[kWarps];
  for (int sp = 1; sp <= A.numslv; ++sp) {
    const bool take = mine && species == sp;
    double s = take ? u : 0.0;
    long long mn = take ? ordered_key(u) : kKeyPosInf, mx = take ? ordered_key(u) : kKeyNegInf;
    for (int o = 16; o >= T; o >>= 1) {  // only a molecule's first lane has values
      s += __shfl_xor_sync(0xffffffffu, s, o);
      mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
      wsum[warp] = s;
      wmin[warp] = mn;
      wmax[warp] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kWarps; ++w) {
        s += wsum[w];
        mn = min(mn, wmin[w]);
        mx = max(mx, wmax[w]);
      }
      double* pt = a.part + (((size_t)b * A.ntile + tile) * A.numslv + (sp - 1)) * 3;
      pt[0] = s;
      pt[1] = key_to_double(mn);
      pt[2] = key_to_double(mx);
    }
    __syncthreads();
  }
}


// ---- TMA + mbarrier helpers (inline PTX, sm_90+ forms, valid on sm_103a) -------------

// Mixed path, step 1 -- gather by bricks.  CTA per (kBrickX x kBrickY x kBrickZ brick of the
// PME grid, run of placement groups of 4).  One TMA box copy per group brings the
// brick's stencil halo of the group's interleaved potential grids into shared memory as
// [z][y][x][4], in gather_stages(P) buffers so that the next groups' copies are in flight
// while this one is used; each thread takes a site of the brick (its B-spline weights
// computed once for all groups, FP32 stable recursion) and accumulates
// q theta theta theta phi for the four placements with one 16-byte shared load per
// stencil point.  Bound by those loads (66% of the shared-memory wavefronts, a launch of 256
// placements at 96^3 in 340 us); 160-thread CTAs, three to an SM, measured 2% slower.
constexpr int kGatherThreads = 256;
// halo buffers (TMA copies in flight) per gather CTA: two for order 4, whose halos leave an SM room
// for two CTAs of them; one for orders 6 and 8, where two buffers of 57 and 83 KB would leave it a
// single CTA, and another CTA hides the copies better (1,024 insertions of 33,000 waters: order 6
// 11.44 ms with two buffers, 10.62 with one; order 8 16.20 and 15.65)
constexpr int gather_stages(int P) { return P <= 4 ? 2 : 1; }

template <int P>
__device__ __forceinline__ void site_setup(int site, const float4* __restrict__ site_rec,
                                           const int* __restrict__ site_grid, int K1, int K2, int K3, int ox,
                                           int oy, int oz, int BX, float (&w1)[P], float (&w2)[P],
                                           float (&w3)[P], int& base, float& q) {
  constexpr int BY = kBrickY + P - 1;
  const float4 rec = site_rec[site];
  const int gp = site_grid[site];
  bspline_w<P>(rec.x, w1);
  bspline_w<P>(rec.y, w2);
  bspline_w<P>(rec.z, w3);
  int g1 = gp & 1023, g2 = (gp >> 10) & 1023, g3 = (gp >> 20) & 1023;
  if (g1 >= K1) g1 -= K1;
  if (g2 >= K2) g2 -= K2;
  if (g3 >= K3) g3 -= K3;
  base = ((g3 - oz) * BY + (g2 - oy)) * BX + (g1 - ox);  // stencil c covers l0 - c
  q = rec.w;
}

template <int P>
__device__ __forceinline__ float4 site_stencil(const float4* __restrict__ halo, int base, int BX,
                                               const float (&w1)[P], const float (&w2)[P], const float (&w3)[P]) {
  constexpr int BY = kBrickY + P - 1;
  constexpr int U3 = P <= 4 ? P : 1;  // higher orders: keep the register footprint bounded
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll U3
  for (int c3 = 0; c3 < P; ++c3) {
#pragma unroll
    for (int c2 = 0; c2 < P; ++c2) {
      const float w32 = w3[c3] * w2[c2];
      const float4* row = halo + base - (c3 * BY + c2) * BX;
#pragma unroll
      for (int c1 = 0; c1 < P; ++c1) {
        const float w = w32 * w1[c1];
        const float4 v = row[-c1];
        acc.x = fmaf(w, v.x, acc.x);
        acc.y = fmaf(w, v.y, acc.y);
        acc.z = fmaf(w, v.z, acc.z);
        acc.w = fmaf(w, v.w, acc.w);
      }
    }
  }
  return acc;
}

template <int P>
__global__ void __launch_bounds__(kGatherThreads) gather_tma_kernel(
    const __grid_constant__ CUtensorMap tmap, int nb, int groups_per_cta, const float4* __restrict__ site_rec,
    const int* __restrict__ site_grid, const int* __restrict__ brick_site, const int* __restrict__ brick_start,
    int K1, int K2, int K3, int nbx, int nby, int BX, int ldb, float* __restrict__ site_e, DevStatus* status) {
  constexpr int BY = kBrickY + P - 1, BZ = kBrickZ + P - 1, kStages = gather_stages(P);
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long bar[kStages];
  const int npt = BZ * BY * BX;
  // kStages halo buffers [z][y][x] of float4 (the four placements of a group),
  // 128-byte aligned; group g lands in buffer (g - g_begin) % kStages
  float4* halo_base = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  const int hstride = (npt + 7) & ~7;  // float4 elements, a multiple of 128 bytes
  const int brick = blockIdx.x;
  const int bx = brick % nbx, by = (brick / nbx) % nby, bz = brick / (nbx * nby);
  const int g_begin = blockIdx.y * groups_per_cta;
  const int g_end = min((nb + 3) / 4, g_begin + groups_per_cta);
  const uint32_t box_bytes = (uint32_t)(npt * sizeof(float4));
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) mbar_init(&bar[i], 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  __syncthreads();
  // padded coordinates: the halo of brick (bx, by, bz) starts at (kBrickX bx,
  // kBrickY by, kBrickZ bz), four floats (the group's placements) per x
  if (threadIdx.x == 0) {
    for (int g = g_begin; g < min(g_end, g_begin + kStages); ++g) {
      const int st = g - g_begin;
      mbar_expect_tx(&bar[st], box_bytes);
      tma_load_4d(halo_base + (size_t)st * hstride, &tmap, 4 * bx * kBrickX, by * kBrickY, bz * kBrickZ, g, &bar[st]);
    }
  }
  const int h = P - 1;
  const int ox = bx * kBrickX - h, oy = by * kBrickY - h, oz = bz * kBrickZ - h;
  const int s_begin = brick_start[brick], s_end = brick_start[brick + 1];
  const int n = s_end - s_begin;
  // Site-to-thread map.  A 16-byte shared load is served 8 lanes at a time, and the
  // 8 lanes are conflict free when their halo indices differ mod 8; every stencil
  // point shifts all lanes' indices by the same offset.  So the brick's sites are
  // bucketed by (stencil base index mod 8), and lane t takes entry t / 8 of bucket t % 8.
  // Bricks with more sites than threads keep the plain order.
  __shared__ int sbucket[8][kGatherThreads / 8];
  __shared__ int scnt[8];
  __shared__ int sovf[kGatherThreads];
  __shared__ int novf;
  const bool bucketed = n <= (int)blockDim.x;
  int site0 = -1;
  if (bucketed) {
    if (threadIdx.x < 8) scnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) novf = 0;
    __syncthreads();
    if ((int)threadIdx.x < n) {
      const int site = brick_site[s_begin + threadIdx.x];
      const int gp = site_grid[site];
      int g1 = gp & 1023, g2 = (gp >> 10) & 1023, g3 = (gp >> 20) & 1023;
      if (g1 >= K1) g1 -= K1;
      if (g2 >= K2) g2 -= K2;
      if (g3 >= K3) g3 -= K3;
      const int r = ((((g3 - oz) * BY + (g2 - oy)) * BX + (g1 - ox)) & 7);
      const int pos = atomicAdd(&scnt[r], 1);
      if (pos < (int)(kGatherThreads / 8))
        sbucket[r][pos] = site;
      else
        sovf[atomicAdd(&novf, 1)] = site;
    }
    __syncthreads();
    const int r = threadIdx.x & 7, k = threadIdx.x >> 3;
    if (k < scnt[r] && k < (int)(kGatherThreads / 8)) site0 = sbucket[r][k];
  } else if ((int)threadIdx.x < n) {
    site0 = brick_site[s_begin + threadIdx.x];
  }
  // this thread's site, set up once for every group
  float w1[P], w2[P], w3[P];
  int base = 0;
  float q = 0.f;
  if (site0 >= 0) site_setup<P>(site0, site_rec, site_grid, K1, K2, K3, ox, oy, oz, BX, w1, w2, w3, base, q);
  const int n_extra = bucketed ? novf : max(0, n - (int)blockDim.x);
  for (int g = g_begin; g < g_end; ++g) {
    const int slot = (g - g_begin) % kStages;
    const uint32_t parity = (uint32_t)(((g - g_begin) / kStages) & 1);
    bool ok = false;
    for (long it = 0; it < kWaitLimit; ++it)
      if (mbar_try_wait(&bar[slot], parity)) {
        ok = true;
        break;
      }
    if (!__syncthreads_and(ok)) {  // flag, let the other copies in flight land (bounded), leave
      if (threadIdx.x == 0) atomicOr(&status->range_fault, 2);
      for (int g2 = g + 1; g2 < min(g_end, g + kStages); ++g2) {
        const int s2 = (g2 - g_begin) % kStages;
        const uint32_t p2 = (uint32_t)(((g2 - g_begin) / kStages) & 1);
        for (long it = 0; it < kWaitLimit; ++it)
          if (mbar_try_wait(&bar[s2], p2)) break;
      }
      return;
    }
    const float4* halo = halo_base + (size_t)slot * hstride;
    const int b0 = 4 * g;
    if (site0 >= 0) {
      const float4 acc = site_stencil<P>(halo, base, BX, w1, w2, w3);
      *reinterpret_cast<float4*>(site_e + (size_t)site0 * ldb + b0) =
          make_float4(q * acc.x, q * acc.y, q * acc.z, q * acc.w);
    }
    for (int i = threadIdx.x; i < n_extra; i += blockDim.x) {  // bucket overflow / crowded bricks
      const int site = bucketed ? sovf[i] : brick_site[s_begin + blockDim.x + i];
      float v1[P], v2[P], v3[P];
      int bs;
      float qs;
      site_setup<P>(site, site_rec, site_grid, K1, K2, K3, ox, oy, oz, BX, v1, v2, v3, bs, qs);
      const float4 acc = site_stencil<P>(halo, bs, BX, v1, v2, v3);
      *reinterpret_cast<float4*>(site_e + (size_t)site * ldb + b0) =
          make_float4(qs * acc.x, qs * acc.y, qs * acc.z, qs * acc.w);
    }
    __syncthreads();  // halo[slot] consumed: the copy of group g + kStages may land in it
    if (threadIdx.x == 0 && g + kStages < g_end) {
      fence_proxy_async_smem();
      mbar_expect_tx(&bar[slot], box_bytes);
      tma_load_4d(halo_base + (size_t)slot * hstride, &tmap, 4 * bx * kBrickX, by * kBrickY, bz * kBrickZ,
                  g + kStages, &bar[slot]);
    }
  }
}


// The number of a species' edges e below u = hi + lo, given pos, the number of edges
// whose float keys rd(e) lie below key32(hi) (kk: the species' float keys, uvkey: its
// FP64 edges as ordered keys).  The two counts can differ only for an edge within one
// float step of hi; such an edge is compared exactly in FP64 (e - hi is exact there, and
// lo is a float), so the bin is the one the FP64 value hi + lo takes against the FP64
// edges (getiduv/binsearch, engproc.F90:927-1020).
// (The FP64 comparisons sit in a function of their own, called only for a total that near
// an edge: inline, the compiler would issue them predicated for every molecule, and an
// FP64 instruction costs GB300 about 64 times an FP32 one even when no lane executes it.)
__device__ __noinline__ int exact_count_near(const long long* __restrict__ uvkey, const int* kk, int n, int pos,
                                            int khi, float hi, float lo) {
  while (pos > 0 && kk[pos - 1] >= khi - 2) {  // counted, but maybe not below u
    if (key_to_double(__ldg(uvkey + pos - 1)) - (double)hi < (double)lo) break;
    --pos;
  }
  while (pos < n && kk[pos] <= khi + 2) {  // not counted, but maybe below u
    if (!(key_to_double(__ldg(uvkey + pos)) - (double)hi < (double)lo)) break;
    ++pos;
  }
  return pos;
}
__device__ __forceinline__ int exact_count(const long long* __restrict__ uvkey, const int* kk, int n, int pos,
                                           int khi, float hi, float lo) {
  const bool near = (pos > 0 && kk[pos - 1] >= khi - 2) || (pos < n && kk[pos] <= khi + 2);
  return near ? exact_count_near(uvkey, kk, n, pos, khi, hi, lo) : pos;
}

// the finish kernel's per-species partials of its block (see mol_finish_kernel)
template <int G, int TILE, bool kSum>
__device__ __forceinline__ void species_partials(const MolArgs& A, const BatchArgs& a, const float (*su)[TILE],
                                                 const float (*sul)[TILE], const unsigned char* sspec, int g0, int ng,
                                                 int tile) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int pr = warp; pr < ng * A.numslv; pr += blockDim.x / 32) {
    const int j = pr / A.numslv, sp = pr % A.numslv + 1;
    long long mn = kFfKeyNone, mx = kFfKeyNoneMax;
    double s = 0.0;
    for (int t = lane; t < TILE; t += 32) {
      const float v = su[j][t];
      if (sspec[t] == sp && v == v) {
        const float lo = sul[j][t];
        if (kSum) s += (double)v + (double)lo;
        const long long key = ff_key(v, lo);
        mn = min(mn, key);
        mx = max(mx, key);
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      if (kSum) s += __shfl_down_sync(0xffffffffu, s, off);
      mn = min(mn, __shfl_down_sync(0xffffffffu, mn, off));
      mx = max(mx, __shfl_down_sync(0xffffffffu, mx, off));
    }
    if (lane == 0) {
      double* pt = a.part + (((size_t)(g0 + j) * A.ntile + tile) * A.numslv + (sp - 1)) * 3;
      pt[0] = s;
      reinterpret_cast<long long*>(pt)[1] = mn;  // kFfKeyNone: no molecule of the species
      reinterpret_cast<long long*>(pt)[2] = mx;
    }
  }
}

// Mixed path, step 2 -- per molecule x G placements: float-float sums of the site terms
// and of the real-space pair terms, the residual, then the G bin searches in lockstep
// (binary lifting over the float keys of the edges staged in shared memory, finished
// exactly against the FP64 edges), histograms and per-species partials.
//
// The real-space pass: the block's (molecule, placement) items within the solute's bounding
// sphere + cutoff are compacted into a list (2% of the 33,000-water box's molecules).  A thread
// takes an item and a solute site; for large solutes, those whose first molecule site lies
// within the cutoff and the largest molecule's radius -- a sixth at 36 sites -- go through a
// queue per warp to the test of each of the molecule's sites, and the pairs within the cutoffs
// through another one to the evaluation, so that each stage, several times as long as the one
// before, runs on full warps.  The terms are added as fixed-point integers, in any order.  (A
// few threads per item, each walking its pairs: 19 of 32 lanes active, 438 us for 256
// insertions of a 36-site solute into 2,000 waters, now 243; 12 sites into 33,000 waters 340,
// now 294.)
//
// Four blocks per SM (64 registers): 2-3% faster over a whole run than three of 80.
// TILE: molecules per block of 256 threads.  16 or 64 in solution mode, where a frame's one placement
// makes few blocks and the real-space pass, the FP64 pairs of the first shell above all, takes
// all 256 threads.
// kTwo: the stage before the pairs' test, for solutes of many sites (kTwoStageSites).
// kWide: the sums of the pair terms take three words (fixed_add_wide); a parameter, so that the usual
// kernels keep their registers.
template <int G, int TILE, bool kTwo, bool kWide>
__global__ void __launch_bounds__(256, 4) mol_finish_kernel(MolArgs A, const float* __restrict__ site_e) {
  extern __shared__ __align__(16) int smem_dyn[];
  // [G][ermax] block histograms, or none when they would not fit beside other blocks: the
  // molecules' counts then go to the batch histograms in global memory (warp-aggregated).
  // Before the histograms are zeroed, the same region holds the real-space pass's scratch
  // (finish_scratch_ints ints).
  int* smem_hist = A.hist_global ? nullptr : smem_dyn;
  int* skeys = smem_dyn + finish_region_ints(G, kTwo, A.ermax, A.hist_global);  // [ermax] 32-bit edge keys
  double* sval = reinterpret_cast<double*>(smem_dyn);                           // [kBigList] FP64 values of the list
  unsigned* sbig = reinterpret_cast<unsigned*>(sval + kBigList);                // [kBigList] the list's pairs
  unsigned short* sorder = reinterpret_cast<unsigned short*>(sbig + kBigList);  // [kBigList] in the pairs' order
  unsigned char* sparts = reinterpret_cast<unsigned char*>(sorder + kBigList);  // [kBigList] the parts left out
  unsigned* squeue = reinterpret_cast<unsigned*>(sparts + kBigList);            // [1 or 2][8][kPairQueue]
  unsigned* sfix = squeue + (kTwo ? 16 : 8) * kPairQueue;                                    // [2][G * 256] sums, low and high words
  [[maybe_unused]] unsigned* stop = reinterpret_cast<unsigned*>(sval);                           // [G * 256] their third ones, read before sval is written
  int* ss0 = reinterpret_cast<int*>(sfix + 2 * 256 * G);                        // [256] first sites
  unsigned short* snear = reinterpret_cast<unsigned short*>(ss0 + 256);         // [G * 256] molecule | placement << 8
  __shared__ int swarp[8];
  __shared__ int snlist, snu;    // pairs in the FP64 list; the placements' most solute sites
  __shared__ float su[G][TILE];   // totals, hi part (NaN: no molecule)
  __shared__ float sul[G][TILE];  // totals, lo part
  __shared__ float sres[G];      // residual factor x solute charge of the G placements
  __shared__ float srcut[G];     // bounding-sphere cutoff of the real-space sum
  __shared__ int skskip[G];      // slot of the solute molecule itself (not a solvent)
  __shared__ int srej[G];        // placement rejected by check_mol_configuration
  __shared__ int4 supos[G];      // first solute site (fixed point)
  __shared__ unsigned char sspec[TILE];
  const int tile = blockIdx.y;
  const int g0 = blockIdx.x * G;
  const BatchArgs& a = A.a;
  const int ng = min(G, a.nb - g0);
  const bool mine = TILE == 256 || threadIdx.x < TILE;
  const int m = tile * TILE + threadIdx.x;
  const bool valid = mine && m < A.slvmax;
  for (int i = threadIdx.x; i < A.ermax; i += blockDim.x) skeys[i] = A.uvkey_f[i];
  if (threadIdx.x < ng) {
    const int b = g0 + threadIdx.x;
    sres[threadIdx.x] = (float)(A.resid_fac * a.u_qmol[b]);
    srcut[threadIdx.x] = A.rc_f + a.u_radius[b] + A.frame_scal[0];
    const int tg = a.tagslt[b] - 1;
    skskip[threadIdx.x] = (tg >= 0 && tg < A.nummol) ? A.mol_to_k[tg] : -2;
    srej[threadIdx.x] = (a.skip && a.skip[b]) ? 1 : 0;
    supos[threadIdx.x] = a.u_pos[(size_t)b * kMaxSoluteSites];
  }
  int k = -1, s0 = 0, ns = 0, species = 0;
  // residual_ene's molecular charge: the term pi Q_u Q_v / (beta^2 V) is below 1e-2 kcal/mol
  // for unit charges in these boxes, so its FP32 product is exact to 1e-9 kcal/mol
  float qmol = 0.f;
  if (valid) {
    k = A.slot_mol[m];
    s0 = A.slot_site[m];
    ns = A.slot_site[m + 1] - s0;
    species = A.slot_species[m];
    qmol = (float)A.slot_qmol[m];
  }
  const bool spec_ok = valid && species >= 1 && species <= A.numslv;
  if (mine) sspec[threadIdx.x] = (unsigned char)(spec_ok ? species : 0);
  const int ldb = A.ldb;
  int sp_off = 0, sp_n = 1, sp_soft = 1;
  if (spec_ok) {
    sp_off = A.spec[3 * (species - 1)];
    sp_n = A.spec[3 * (species - 1) + 1];
    sp_soft = A.spec[3 * (species - 1) + 2];
  }
  __syncthreads();  // sres staged
  // ---- totals of the G placements, as float-float numbers.  First the site terms: the G
  // placements' terms of a site are G consecutive floats (16-byte loads when G, g0 and ldb
  // are multiples of 4).  The totals then wait in su (hi) and sul (lo) until the bin search;
  // the real-space pass adds to them ----
  unsigned actm = 0u;   // placements whose total is a solvent molecule's energy
  unsigned nearm = 0u;  // of those, the ones within reach of the solute
  {
    ff rs[G];
#pragma unroll
    for (int j = 0; j < G; ++j) rs[j] = ff{0.f, 0.f};
    if (valid) {
      for (int s = 0; s < (A.bare ? 0 : ns); ++s) {
        const float* row = site_e + (size_t)(s0 + s) * ldb + g0;
        if (G % 4 == 0 && ng == G) {
#pragma unroll
          for (int j4 = 0; j4 + 4 <= G; j4 += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(row + j4));
            rs[j4] = ff_add(rs[j4], v.x);
            rs[j4 + 1] = ff_add(rs[j4 + 1], v.y);
            rs[j4 + 2] = ff_add(rs[j4 + 2], v.z);
            rs[j4 + 3] = ff_add(rs[j4 + 3], v.w);
          }
        } else {
#pragma unroll
          for (int j = 0; j < G; ++j)
            if (j < ng) rs[j] = ff_add(rs[j], __ldg(row + j));
        }
      }
    }
    const int4 p0 = valid ? A.site_pos[s0] : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const bool on = j < ng && valid && k != skskip[j] && !srej[j];
      if (on) {
        actm |= 1u << j;
        const int4 u0 = supos[j];
        const float dx = (float)(int)((unsigned)p0.x - (unsigned)u0.x) * A.fxf[0];
        const float dy = (float)(int)((unsigned)p0.y - (unsigned)u0.y) * A.fxf[1];
        const float dz = (float)(int)((unsigned)p0.z - (unsigned)u0.z) * A.fxf[2];
        if (!(dx * dx + dy * dy + dz * dz > srcut[j] * srcut[j])) nearm |= 1u << j;
      }
      // residual_ene (engproc.F90:859-869)
      const ff t = on ? ff_add(rs[j], -sres[j] * qmol) : ff{0.f, 0.f};
      if (mine) {
        su[j][threadIdx.x] = t.hi;
        sul[j][threadIdx.x] = t.lo;
      }
    }
  }
  // ---- real space: get_uv_energy (engproc.F90:736-753) adds it to residual + recip ----
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int near0, nnear;  // this thread's first entry of the block's near list; its length
  {
    const int cnt = __popc(nearm);
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) swarp[wid] = incl;
    ss0[threadIdx.x] = s0;
    __syncthreads();
    near0 = incl - cnt;
    nnear = 0;
    for (int w2 = 0; w2 < 8; ++w2) {
      if (w2 < wid) near0 += swarp[w2];
      nnear += swarp[w2];
    }
    for (unsigned q = nearm; q; q &= q - 1) snear[near0++] = (unsigned short)(threadIdx.x | ((__ffs(q) - 1) << 8));
    for (int i = threadIdx.x; i < nnear; i += 256) {
      sfix[i] = sfix[256 * G + i] = 0u;
      if constexpr (kWide) stop[i] = 0u;
    }
    if (threadIdx.x == 0) {
      snlist = 0;
      snu = 0;
      for (int j = 0; j < ng; ++j) snu = max(snu, a.u_nsite[g0 + j]);
    }
    __syncthreads();
  }
  if (nnear > 0) {  // block-uniform
    const int nu_max = snu;
    const unsigned magic = nu_max > 1 ? (unsigned)((0x100000000ull + nu_max - 1) / nu_max) : 0u;
    const float scale = A.fx_scale_f, reach2 = A.reach2_f;
    // beyond this a molecule's first site is too far from a solute site for any pair of the two
    const float mol_reach = sqrtf(reach2) + A.frame_scal[0], mol_reach2 = margin_r2(mol_reach * mol_reach);
    unsigned* queue = squeue + wid * kPairQueue;
    [[maybe_unused]] unsigned* cand = queue + 8 * kPairQueue;
    int nq = 0;  // warp-uniform
    int win = 0;  // the window of 8,192 molecule sites that the queue's pairs lie in (block-uniform)
    // the last n pairs of the warp's queue, one per lane
    auto evaluate = [&](int n) {
      __syncwarp();
      if (lane < n) {
        const unsigned key = queue[nq - n + lane];
        const int near = key >> 21, su_ = (key >> 13) & 0xff, s = (int)(key & 0x1fff) + (win << kSiteWindowBits);
        const int nr = snear[near], site = ss0[nr & 0xff] + s;
        const size_t us = (size_t)(g0 + (nr >> 8)) * kMaxSoluteSites + su_;
        const int4 vp = A.site_pos[site], up = a.u_pos[us];
        float elj, eco;
        const int parts = pair_fp32(A, vp, up, a.u_qf[us], A.site_rec[site].w, pair_r2(A, vp, up), elj, eco);
        long long v = 0;
        if (!(parts & kPairLj)) v = __float2ll_rn(elj * scale);
        if (!(parts & kPairCoulomb)) v += __float2ll_rn(eco * scale);
        if (v != 0) {
          if constexpr (kWide)
            fixed_add_wide(sfix + near, sfix + 256 * G + near, stop + near, v);
          else
            fixed_add(sfix + near, sfix + 256 * G + near, v);
        }
        if (parts) {
          // (a window that the byte cannot hold: the items' threads find all their own again)
          const int q = win < kListWindows ? atomicAdd(&snlist, 1) : atomicMax(&snlist, kBigList + 1);
          if (q < kBigList && win < kListWindows) {
            sbig[q] = key;
            sparts[q] = (unsigned char)(parts | win << 2);
          }
        }
      }
      __syncwarp();
      nq -= n;
    };
    const int total = nnear * nu_max;
    for (int wbase = 0; wbase < A.max_mol_sites; wbase += 1 << kSiteWindowBits, ++win) {
      int nc = 0;  // candidates waiting: at most 31 + 32 (warp-uniform)
      for (int task0 = wid * 32;; task0 += 256) {
        const bool more = task0 < total;  // warp-uniform
        bool on = false;                  // the lane's candidate
        unsigned key = 0u;
        if (more) {
          const int task = task0 + lane;
          const int near = nu_max > 1 ? (int)__umulhi((unsigned)task, magic) : task, su_ = task - near * nu_max;
          key = pair_key(near, su_, 0);
          if (near < nnear) {
            const int nr = snear[near], b = g0 + (nr >> 8);
            on = su_ < a.u_nsite[b];
            if (kTwo && on)
              on = !(pair_r2(A, A.site_pos[ss0[nr & 0xff]], a.u_pos[(size_t)b * kMaxSoluteSites + su_]) > mol_reach2);
          }
        }
        if constexpr (kTwo) {  // wait for 32 of them
          const unsigned m = __ballot_sync(0xffffffffu, on);
          if (on) cand[nc + __popc(m & ((1u << lane) - 1u))] = key;
          nc += __popc(m);
          if (more && nc < 32) continue;
          const int n = min(nc, 32);
          __syncwarp();
          on = lane < n;
          if (on) key = cand[nc - n + lane];
          __syncwarp();
          nc -= n;
        }
        int is0 = 0, ins = 0;
        int4 up = make_int4(0, 0, 0, 0);
        if (on) {
          const int nr = snear[key >> 21];
          is0 = ss0[nr & 0xff] + wbase;
          ins = min(A.slot_site[tile * TILE + (nr & 0xff) + 1] - is0, 1 << kSiteWindowBits);
          up = a.u_pos[(size_t)(g0 + (nr >> 8)) * kMaxSoluteSites + ((key >> kSiteWindowBits) & 0xff)];
        }
        for (int s = 0; __any_sync(0xffffffffu, s < ins); ++s) {
          const bool in = s < ins && pair_r2(A, A.site_pos[is0 + s], up) <= reach2;
          const unsigned m = __ballot_sync(0xffffffffu, in);
          if (in) queue[nq + __popc(m & ((1u << lane) - 1u))] = key | (unsigned)s;
          nq += __popc(m);
          if (nq >= 32) evaluate(32);
        }
        if (!more) break;
      }
      if (nq > 0) evaluate(nq);
    }
    __syncthreads();
    auto add_sums = [&] {
      for (int near = threadIdx.x; near < nnear; near += 256) {
        const int t = snear[near] & 0xff, j = snear[near] >> 8;
        const unsigned lo = sfix[near], hi = sfix[256 * G + near];
        ff r;
        if constexpr (kWide)
          r = fixed_to_ff_wide(lo, hi, stop[near], 1.f / scale);
        else
          r = fixed_to_ff(lo, hi, 1.f / scale);
        const ff x = ff_add2(ff{su[j][t], sul[j][t]}, r);
        su[j][t] = x.hi;
        sul[j][t] = x.lo;
      }
      __syncthreads();
    };
    static_assert(sizeof(unsigned) * 256 * G <= sizeof(double) * kBigList, "the third words in sval's place");
    if constexpr (kWide) add_sums();  // before sval takes the third words' place
    // FP64 pass over the listed pair parts (overlapping pairs, left out of the FP32 sums): one
    // per thread, so that every FP64 instruction runs on full warps; an item's values are added
    // in the order of its pairs (solute site, molecule site), by the thread of the first
    const int nlist = snlist;
    if (nlist <= kBigList) {
      for (int q = threadIdx.x; q < nlist; q += 256) {
        const unsigned key = sbig[q];
        int rank = 0;
        for (int i = 0; i < nlist; ++i) rank += sbig[i] < key || (sbig[i] == key && sparts[i] < sparts[q]) ? 1 : 0;
        sorder[rank] = (unsigned short)q;
        const int nr = snear[key >> 21];
        const size_t us = (size_t)(g0 + (nr >> 8)) * kMaxSoluteSites + ((key >> 13) & 0xff);
        const int s = (int)(key & 0x1fff) + ((sparts[q] >> 2) << kSiteWindowBits);
        sval[q] = pair_fp64(A, ss0[nr & 0xff] + s, a.u_x + us * 3, a.u_q[us], a.u_pos[us].w, sparts[q] & 3);
      }
      __syncthreads();
    }
    if constexpr (!kWide) add_sums();
    if (nlist <= kBigList) {
      for (int r = threadIdx.x; r < nlist; r += 256) {
        const unsigned near = sbig[sorder[r]] >> 21;
        if (r > 0 && sbig[sorder[r - 1]] >> 21 == near) continue;
        const int t = snear[near] & 0xff, j = snear[near] >> 8;
        ff x{su[j][t], sul[j][t]};
        for (int i = r; i < nlist && sbig[sorder[i]] >> 21 == near; ++i) x = ff_add2(x, ff_from_double(sval[sorder[i]]));
        su[j][t] = x.hi;
        sul[j][t] = x.lo;
      }
    } else {  // more than the list holds: each item's pairs again, in the same order
      for (int near = threadIdx.x; near < nnear; near += 256) {
        const int t = snear[near] & 0xff, j = snear[near] >> 8, b = g0 + j;
        const int is0 = ss0[t], ins = A.slot_site[tile * TILE + t + 1] - is0, nu = a.u_nsite[b];
        const size_t ub = (size_t)b * kMaxSoluteSites;
        ff x{su[j][t], sul[j][t]};
        for (int u = 0; u < nu; ++u)
          for (int s = 0; s < ins; ++s) {
            const int4 vp = A.site_pos[is0 + s], up = a.u_pos[ub + u];
            const float r2 = pair_r2(A, vp, up);
            if (!(r2 <= reach2)) continue;
            float elj, eco;
            const int parts = pair_fp32(A, vp, up, a.u_qf[ub + u], A.site_rec[is0 + s].w, r2, elj, eco);
            if (parts)
              x = ff_add2(x, ff_from_double(pair_fp64(A, is0 + s, a.u_x + (ub + u) * 3, a.u_q[ub + u], up.w, parts)));
          }
        su[j][t] = x.hi;
        sul[j][t] = x.lo;
      }
    }
  }
  __syncthreads();  // the totals are complete and the scratch is free: the histograms may take the region
  if (!A.hist_global)
    for (int i = threadIdx.x; i < G * A.ermax; i += blockDim.x) smem_hist[i] = 0;
  int ku[G];     // ordered key of the total's hi part
  float ulo[G];  // the total's lo part
#pragma unroll
  for (int j = 0; j < G; ++j) {
    ku[j] = mine ? ordered_key32(su[j][threadIdx.x]) : 0;
    ulo[j] = mine ? sul[j][threadIdx.x] : 0.f;
  }
  if (valid && a.uvengy_out) {
#pragma unroll
    for (int j = 0; j < G; ++j) {
      if (j >= ng) break;
      a.uvengy_out[(size_t)(a.b0 + g0 + j) * (A.slvmax + 1) + k + 1] =
          (actm & (1u << j)) ? (double)key32_to_float(ku[j]) + (double)ulo[j] : 0.0;
    }
  }
  __syncthreads();  // histograms zeroed, keys staged
  // ---- getiduv / binsearch for all G at once: pos = #edges whose float keys lie below
  // the key of the total's hi part ----
  int pos[G];
#pragma unroll
  for (int j = 0; j < G; ++j) pos[j] = 0;
  int step = 1;
  while ((step << 1) <= sp_n) step <<= 1;
  const int* kk = skeys + sp_off;
  for (; step > 0; step >>= 1) {
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int q = pos[j] + step;
      if (q <= sp_n && kk[q - 1] < ku[j]) pos[j] = q;
    }
  }
#pragma unroll
  for (int j = 0; j < G; ++j) {
    float hv = __uint_as_float(0x7fc00000u);  // NaN marks "no molecule"
    float lv = 0.f;
    if (actm & (1u << j)) {
      const float v = key32_to_float(ku[j]), lo = ulo[j];
      int ret = pos[j];
      int code = 0;
      if (!spec_ok) {
        code = ERMOD_E_ENG_CNS;
      } else if (v != v) {
        code = ERMOD_E_ENG_MIN;
      } else {
        ret = exact_count(A.uvkey + sp_off, kk, sp_n, ret, ku[j], v, lo);
        if (ret <= 0)
          code = ERMOD_E_ENG_MIN;
        else if (A.soln && ret > sp_soft)
          code = ERMOD_E_ENG_SFT;
        else if (ret == sp_n && (v < 1.0e3f || (v == 1.0e3f && lo < 0.f)) && A.mbin_mode != 0) {
          if (A.mbin_mode == 1)
            code = ERMOD_W_MBIN;
          else
            atomicOr(&A.status->mbin_hit, 1);
        }
      }
      if (code)
        atomicMin(&A.status->err_key, make_err_key(a.b0 + g0 + j, k + 1, code));
      else
        hist_add(A.hist_global ? a.hist + (size_t)(g0 + j) * A.ermax : smem_hist + j * A.ermax, sp_off + ret - 1);
      if (a.mol_bin) a.mol_bin[(size_t)(g0 + j) * A.slvmax + m] = code ? A.ermax : sp_off + ret - 1;
      hv = v;
      lv = lo;
    } else if (a.mol_bin && valid && j < ng) {
      a.mol_bin[(size_t)(g0 + j) * A.slvmax + m] = A.ermax;
    }
    if (mine) {
      su[j][threadIdx.x] = hv;
      sul[j][threadIdx.x] = lv;
    }
  }
  __syncthreads();
  // per-species {sum, min, max} of the block: one warp per (placement, species),
  // fixed lane order and a fixed shuffle tree; min and max as ordered keys of the
  // float-float totals (decoded by the reduce kernel), so that no FP64 instruction issues
  // here unless the species sums are wanted -- they are flceng (engproc.F90:822-825),
  // needed for slnuv (solution mode) and when the caller asks for flceng
  if (A.soln || a.flceng_out != nullptr)
    species_partials<G, TILE, true>(A, a, su, sul, sspec, g0, ng, tile);
  else
    species_partials<G, TILE, false>(A, a, su, sul, sspec, g0, ng, tile);
  if (A.hist_global) return;
  for (int j = 0; j < ng; ++j) {
    const int* h = smem_hist + j * A.ermax;
    int* out = a.hist + (size_t)(g0 + j) * A.ermax;
    for (int i = threadIdx.x; i < A.ermax; i += blockDim.x) {
      const int c = h[i];
      if (c) atomicAdd(out + i, c);
    }
  }
}

template <int TY>
cudaError_t launch_mol64(Engine& e, const MolArgs& A) {
  const dim3 grid(A.ntile, A.a.nb);
  switch (e.P_order) {
    case 4:
      mol_energy_kernel<4, TY><<<grid, kMol64Threads, 0, A.a.stream>>>(A);
      break;
    case 6:
      mol_energy_kernel<6, TY><<<grid, kMol64Threads, 0, A.a.stream>>>(A);
      break;
    case 8:
      mol_energy_kernel<8, TY><<<grid, kMol64Threads, 0, A.a.stream>>>(A);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

// bits below the binary point that two words leave the sums of the largest molecule's pairs with the
// largest solute (the device API may name any molecule as one): their sum stays below 2^63 units
static int fixed_bits(const Engine& e) {
  const double most = (double)kFixedTerm * e.max_mol_sites *
                      std::min(kMaxSoluteSites, std::max(e.max_mol_sites, e.max_solute_sites));
  return 63 - (std::ilogb(most) + 1);
}
static bool fixed_wide(const Engine& e) { return fixed_bits(e) < kFixedNarrowBits; }

static MolArgs make_mol_args(Engine& e, const BatchArgs& a) {
  MolArgs A{};
  A.site_pos = e.d_site_pos;
  A.site_rec = e.d_site_rec;
  A.site_grid = e.d_site_grid;
  A.site_x = e.d_site_x;
  A.site_w = e.d_site_w;
  A.site_q = e.d_site_q;
  A.slot_mol = e.d_slot_mol;
  A.slot_site = e.d_slot_site;
  A.slot_species = e.d_slot_species;
  A.slot_qmol = e.d_slot_qmol;
  A.frame_scal = e.d_frame_scal;
  A.mol_to_k = e.d_mol_to_k;
  A.slvmax = e.slvmax;
  A.nummol = e.nummol;
  A.max_mol_sites = e.max_mol_sites;
  A.ljene = e.d_ljene;
  A.ljlensq = e.d_ljlensq;
  A.ljene_f = e.d_ljene_f;
  A.ljlensq_f = e.d_ljlensq_f;
  A.T = e.ljtype_max;
  A.ldb = e.Bmax;
  A.uvkey = e.d_uvkey;
  A.uvkey_f = e.d_uvkey_f;
  A.spec = e.d_spec;
  A.numslv = e.numslv;
  A.ermax = e.ermax;
  A.soln = (e.P.slttype == 1) ? 1 : 0;
  A.mbin_mode = e.warn_bin_firsttime ? (e.P.force_calculation ? 2 : 1) : 0;
  A.g = e.geom;
  A.ljswitch = e.P.ljswitch;
  // non-periodic: the Coulomb cutoff is infinite (realcal.F90:174)
  A.elecut = e.geom.periodic ? e.P.elecut : HUGE_VAL;
  A.lwljcut = e.P.lwljcut;
  A.upljcut = e.P.upljcut;
  A.screen = e.P.screen;
  A.bare = (e.P.cltype == 0) ? 1 : 0;
  A.resid_fac = A.bare ? 0.0 : kPi / e.P.screen / e.P.screen / e.geom.volume;
  for (int i = 0; i < 3; ++i) A.fxf[i] = (float)e.geom.fx_scale[i];
  A.screen_f = (float)e.P.screen;
  A.rc_f = (float)std::max(A.elecut, e.P.upljcut);
  A.k64 = make_k64(A);
  A.k32 = to_f32(A.k64);
  A.reach2_f = std::max(A.k32.up2, A.k32.ele2);
  A.fx_scale_f = std::ldexp(1.f, fixed_wide(e) ? kFixedWideBits : fixed_bits(e));
  A.a = a;
  A.ntile = e.ntile;
  A.status = e.d_status;
  return A;
}

// step 1 of the mixed path: gather by bricks (TMA-staged halos, double-buffered over
// placement groups) into a.site_e
cudaError_t launch_gather(Engine& e, const BatchArgs& a) {
  cudaError_t err = cudaSuccess;
  const int ngroups = (a.nb + 3) / 4;
  // groups per CTA: 16 (site set-up and the first copies' latency paid once for them), 8 where 16
  // would leave fewer than four rounds of the two CTAs an SM holds
  int gpc = std::min(ngroups, 16);
  if ((long long)e.nbricks * ((ngroups + gpc - 1) / gpc) < 8LL * e.num_sm) gpc = std::min(ngroups, 8);
  dim3 g1(e.nbricks, (ngroups + gpc - 1) / gpc);
  const int K1 = e.geom.K[0], K2 = e.geom.K[1], K3 = e.geom.K[2];
  const size_t npt = (size_t)e.gbox[0] * e.gbox[1] * e.gbox[2];
  const size_t hstride = (npt + 7) & ~(size_t)7;  // as in the kernel: 128-byte aligned halos
  const size_t sh = 128 + gather_stages(e.P_order) * hstride * sizeof(float4);
#define ERMOD_GATHER(PP)                                                                                        \
  if (e.P_order == PP) {                                                                                        \
    static SmemAttr attr;                                                                                       \
    if ((err = attr.ensure(gather_tma_kernel<PP>, sh)) != cudaSuccess) return err;                              \
    gather_tma_kernel<PP><<<g1, kGatherThreads, sh, a.stream>>>(                                                \
        e.phi_tmap[a.slot], a.nb, gpc, e.d_site_rec, e.d_site_grid, e.d_brick_site, e.d_brick_start, K1, K2, K3,  \
        e.nbrick[0], e.nbrick[1], e.gbox[0], e.Bmax, a.site_e, e.d_status);                                     \
  }
  ERMOD_GATHER(4)
  ERMOD_GATHER(6)
  ERMOD_GATHER(8)
#undef ERMOD_GATHER
  e.count_launch();
  return cudaGetLastError();
}

// the FP64 path's threads per molecule, 4 TY: a solution-mode call holds one placement (or
// one per solute molecule), so its molecules are split further while that still leaves the
// GPU room; fixed for a context, so that a placement's sums do not depend on its batch
static int mol64_ty(const Engine& e) { return e.P.slttype == 1 && e.slvmax < 512 * e.num_sm ? 4 : 1; }
// molecules per block of the molecule kernels: the FP64 path's as above; the mixed path's 256, or
// in solution mode 16 while that gives at most a block per SM (a droplet of 300 molecules, a frame
// of which makes hundreds of FP64 pairs: 145 -> 137 us; 1,000 waters 172.4 -> 171.5; at 8,000 no
// faster than 64), then 64 while that leaves few
int mol_tile(const Engine& e) {
  if (!e.mixed) return kMol64Threads / (4 * mol64_ty(e));
  if (e.P.slttype != 1 || e.P.finish_group != 0 || e.slvmax >= 64 * 3 * e.num_sm) return 256;
  return e.slvmax <= 16 * e.num_sm ? 16 : 64;
}

// placements per molecule-energy block: the caller's choice (4 or 8), else 4, halved while the
// launch has fewer than 1.5 blocks per SM (2,000 waters, 36 sites, batches of 64: 26.6 ms of
// 4,000 insertions with 128 blocks of 4, 22.2 with 256 of 2, 22.1 with 512 of 1; with 256 or
// more blocks of 4 -- 4,000 waters -- fewer placements per block are no faster, and at 33,000
// waters 2 cost 5%).  A molecule's energy does not depend on the split.
static int finish_group(const Engine& e, int nb) {
  int G = e.G;
  if (e.P.finish_group != 0) return G;
  if (e.tile < 256) return 1;
  while (G > 1 && 2LL * e.ntile * ((nb + G - 1) / G) < 3LL * e.num_sm) G /= 2;
  return G;
}

cudaError_t launch_mol_energy(Engine& e, const BatchArgs& a) {
  MolArgs A = make_mol_args(e, a);
  e.count_launch();
  cudaError_t err = cudaSuccess;
  if (!e.mixed) return mol64_ty(e) == 4 ? launch_mol64<4>(e, A) : launch_mol64<1>(e, A);
  int G = finish_group(e, a.nb);
  bool two = e.tile == 256 && e.max_solute_sites >= kTwoStageSites;
  // block histograms in shared memory up to 64 KB (three blocks per SM fit); beyond that, and
  // for the few molecules of a small tile, the counts go straight to global memory
  A.hist_global = (e.tile < 256 || (size_t)G * e.ermax * sizeof(int) > 64 * 1024) ? 1 : 0;
  // the keys of a coordinate of tens of thousands of bins may leave no room for the scratch of G
  // placements (48,788 bins leave it for 4): one placement and one stage need the least, up to 52,268
  if (finish_smem(G, two, e.ermax, A.hist_global) + finish_static_smem(G) > kMaxSmem) {
    G = 1;
    two = false;
  }
  if (e.P.cltype != 0 && (err = launch_gather(e, a)) != cudaSuccess) return err;
  if (a.phases) {
    e.phase_end_on(a.stream);
    e.phase_begin_on(PH_MOL, a.stream);
  }
  // step 2: per-molecule totals and binning (histograms + edge keys in shared memory)
  const size_t smem_f = finish_smem(G, two, e.ermax, A.hist_global);
  dim3 g2((a.nb + G - 1) / G, e.ntile);
#define ERMOD_FINISH(GG, TILE, TWO, WIDE)                                                                       \
  if (G == GG && e.tile == TILE && two == TWO && wide == WIDE) {                                               \
    static SmemAttr attr;                                                                                      \
    if ((err = attr.ensure(mol_finish_kernel<GG, TILE, TWO, WIDE>, smem_f)) != cudaSuccess) return err;        \
    mol_finish_kernel<GG, TILE, TWO, WIDE><<<g2, 256, smem_f, a.stream>>>(A, a.site_e);                        \
  }
#define ERMOD_FINISH_ALL(WIDE)        \
  ERMOD_FINISH(1, 16, false, WIDE)    \
  ERMOD_FINISH(1, 64, false, WIDE)    \
  ERMOD_FINISH(1, 256, false, WIDE)   \
  ERMOD_FINISH(2, 256, false, WIDE)   \
  ERMOD_FINISH(4, 256, false, WIDE)   \
  ERMOD_FINISH(8, 256, false, WIDE)   \
  ERMOD_FINISH(1, 256, true, WIDE)    \
  ERMOD_FINISH(2, 256, true, WIDE)    \
  ERMOD_FINISH(4, 256, true, WIDE)    \
  ERMOD_FINISH(8, 256, true, WIDE)
  const bool wide = fixed_wide(e);
  ERMOD_FINISH_ALL(false)
  ERMOD_FINISH_ALL(true)
#undef ERMOD_FINISH_ALL
#undef ERMOD_FINISH
  e.count_launch();
  return cudaGetLastError();
}


// ---- adjoint mode -------------------------------------------------------------------
//
// For a placement b of the differentiated solute and every solvent molecule k, the
// derivatives of u_k = real(k) + residual(k) + recip(k) (get_uv_energy,
// engproc.F90:662-756) with respect to each solute site's charge q_s (topology units),
// LJ epsilon eps_s and LJ sigma sigma_s:
//   du/dq_s     = sum_t q_t erfc(beta r)/r (r <= elecut) + sum_t q_t phi_s(r_t) - pi Q_k/(beta^2 V)
//   du/deps_s   = sum_t LJ_st / (2 eps_s)                       (eps_st = sqrt(eps_s eps_t))
//   du/dsigma_s = sum_t 4 eps_st (6 vdwa - 3 vdwb)/sigma_st^2 * d(sigma_st^2)/d(sigma_s)
// where phi_s is the PME potential of a unit charge on site s (computed by the mixed
// kernels as a batch of single-site "placements") and LJ_st = 4 eps_st (vdwa - vdwb) in
// every switching form (realcal.F90:686-770), vdwa ~ sigma^12 and vdwb ~ sigma^6.  Each
// molecule's derivatives (FP32) are then summed per energy bin of u_k in FP64, in a fixed
// order (molecules stably sorted by bin), times the placement's weight engnmfc.
namespace {

__device__ __forceinline__ void lj_parts_f(int sw, const LjK& k, float x, float r2, float& vdwa, float& vdwb) {
  const float invr2 = x / r2;
  const float invr6 = invr2 * invr2 * invr2;
  const float s6 = x * x * x;
  if (r2 <= k.lw2) {
    if (sw <= 1) {
      vdwa = invr6 * invr6;
      vdwb = invr6;
    } else if (sw == 2) {
      vdwa = invr6 * invr6 - s6 * s6 / (k.lw6 * k.up6);
      vdwb = invr6 - s6 / (k.lw3 * k.up3);
    } else {
      vdwa = invr6 * invr6 - s6 * s6 * k.repC;
      vdwb = invr6 - s6 * k.attC;
    }
    return;
  }
  if (sw == 0) {
    const float dd = r2 - k.up2, den = k.up2 - k.lw2;
    const float f = (2.f * r2 + k.up2 - 3.f * k.lw2) * (dd * dd) / (den * den * den);
    vdwa = invr6 * invr6 * f;
    vdwb = invr6 * f;
  } else if (sw == 1) {
    const float t = (sqrtf(r2) - k.lw) / (k.up - k.lw);
    const float t3 = t * t * t, t4 = t3 * t, t5 = t4 * t;
    const float f = 1.f - 10.f * t3 + 15.f * t4 - 6.f * t5;
    vdwa = invr6 * invr6 * f;
    vdwb = invr6 * f;
  } else if (sw == 2) {
    const float invr3 = sqrtf(invr6), s3 = sqrtf(s6);
    const float a = invr6 - s6 / k.up6, b = invr3 - s3 / k.up3;
    vdwa = k.up6 / (k.up6 - k.lw6) * (a * a);
    vdwb = k.up3 / (k.up3 - k.lw3) * (b * b);
  } else {
    const float f = sqrtf(r2) - k.lw;
    const float f3 = f * f * f, f4 = f3 * f;
    vdwa = invr6 * invr6 - s6 * s6 * (k.repA * f3 + k.repB * f4 + k.repC);
    vdwb = invr6 - s6 * (k.attA * f3 + k.attB * f4 + k.attC);
  }
}

struct AdjArgs {
  int b;          // placement within the batch
  int s_begin;    // first solute site of this chunk of unit-charge potentials
  int nchunk;     // sites in the chunk
  int nsu;        // solute sites: 3 nsu parameters
  int adj_mol;    // 1-based molecule whose placements are differentiated
  int cmbrule;
  int first;      // first chunk: also writes the bin keys
  const float* site_e_ps;  // [nsite][ldb] q_t phi_s(r_t) of the chunk's sites
  const int* mol_bin;      // [slvmax] bins of placement b's molecules, slot order (ermax: none)
  const float2* par;       // [nsu] {eps_s, sigma_s}
  float* du;               // [slvmax][3 nsu]
  int* key;                // [slvmax] global bin, or ermax to leave the molecule out
  int* val;                // [slvmax] slot index
};

// A thread per (molecule, site of the chunk), sites fastest: a molecule's site terms and its
// derivatives are then consecutive words, and a solution-mode frame's few thousand molecules
// fill the GPU (a thread per molecule walking the sites: 39 us of latency for 8,000 waters and
// 16 sites, 32 CTAs).
__global__ void __launch_bounds__(256) adjoint_mol_kernel(MolArgs A, AdjArgs J) {
  const long long task = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int m = (int)(task / J.nchunk), j = (int)(task - (long long)m * J.nchunk);
  if (m >= A.slvmax) return;
  const BatchArgs& a = A.a;
  const int b = J.b;
  const int k = A.slot_mol[m];
  const int s0 = A.slot_site[m];
  const int ns = A.slot_site[m + 1] - s0;
  const int species = A.slot_species[m];
  const int tg = a.tagslt[b] - 1;
  const int kskip = (tg >= 0 && tg < A.nummol) ? A.mol_to_k[tg] : -2;
  bool take = (tg + 1 == J.adj_mol) && (k != kskip) && species >= 1 && species <= A.numslv &&
              !(a.skip && a.skip[b]);
  if (J.first && j == 0) {
    // the molecule's bin as the finish kernel found it (ermax: not binned)
    const int key = take ? J.mol_bin[m] : A.ermax;
    J.key[m] = key;
    J.val[m] = m;
  }
  if (!take) return;
  const size_t ub = (size_t)b * kMaxSoluteSites;
  const int P = 3 * J.nsu;
  const float fx = A.fxf[0], fy = A.fxf[1], fz = A.fxf[2];
  const LjK& k32 = A.k32;
  const float beta = A.screen_f;
  const float rq = (float)A.resid_fac * (float)A.slot_qmol[m];
  // the molecule is near the solute when its first site lies within the solute's
  // bounding sphere plus the cutoff (the finish kernel's test)
  const int4 p0 = A.site_pos[s0];
  const int4 q0 = a.u_pos[ub];
  const float dx0 = (float)(int)((unsigned)p0.x - (unsigned)q0.x) * fx;
  const float dy0 = (float)(int)((unsigned)p0.y - (unsigned)q0.y) * fy;
  const float dz0 = (float)(int)((unsigned)p0.z - (unsigned)q0.z) * fz;
  const float rcut = A.rc_f + a.u_radius[b] + A.frame_scal[0];
  const bool near = dx0 * dx0 + dy0 * dy0 + dz0 * dz0 <= rcut * rcut;
  const int s = J.s_begin + j;
  float dq = -rq, deps = 0.f, dsig = 0.f;
  for (int t = 0; t < ns; ++t) dq += J.site_e_ps[(size_t)(s0 + t) * A.ldb + j];
  if (near) {
    const int4 up = a.u_pos[ub + s];
    const float2 par = J.par[s];
    for (int t = 0; t < ns; ++t) {
      const int4 vp = A.site_pos[s0 + t];
      const float ex = (float)(int)((unsigned)vp.x - (unsigned)up.x) * fx;
      const float ey = (float)(int)((unsigned)vp.y - (unsigned)up.y) * fy;
      const float ez = (float)(int)((unsigned)vp.z - (unsigned)up.z) * fz;
      const float r2 = ex * ex + ey * ey + ez * ez;
      const float ljeps = A.ljene_f[vp.w + A.T * up.w];
      if (ljeps > 0.f && r2 <= k32.up2) {
        const float x = A.ljlensq_f[vp.w + A.T * up.w];
        float va, vb;
        lj_parts_f(A.ljswitch, k32, x, r2, va, vb);
        if (par.x > 0.f) deps += 4.f * ljeps * (va - vb) / (2.f * par.x);
        const float dldx = 4.f * ljeps * (6.f * va - 3.f * vb) / x;
        const float dxds = (J.cmbrule == 0) ? sqrtf(x) : (par.y > 0.f ? x / par.y : 0.f);
        dsig += dldx * dxds;
      }
      if (r2 <= k32.ele2) {
        const float r = sqrtf(r2);
        dq += A.site_rec[s0 + t].w * erfcf(beta * r) / r;
      }
    }
  }
  float* o = J.du + (size_t)m * P + 3 * s;
  o[0] = dq;
  o[1] = deps;
  o[2] = dsig;
}

// the chunk's unit-charge single-site placements: site s_begin + j of placement b
__global__ void adjoint_pseudo_kernel(const float2* __restrict__ bvec, int b, int s_begin, int Kmax, int* nsite,
                                      float* qf, float2* ps_bvec) {
  const int j = blockIdx.x;
  if (threadIdx.x == 0) {
    nsite[j] = 1;
    qf[(size_t)j * kMaxSoluteSites] = 1.f;
  }
  const float2* src = bvec + ((size_t)b * kMaxSoluteSites + s_begin + j) * 3 * Kmax;
  float2* dst = ps_bvec + (size_t)j * kMaxSoluteSites * 3 * Kmax;
  for (int i = threadIdx.x; i < 3 * Kmax; i += blockDim.x) dst[i] = src[i];
}

__global__ void adjoint_bounds_kernel(const int* __restrict__ key, int n, int ermax, int* seg_b, int* seg_e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int kk = key[i];
  if (kk >= ermax) return;
  if (i == 0 || key[i - 1] != kk) seg_b[kk] = i;
  if (i == n - 1 || key[i + 1] != kk) seg_e[kk] = i + 1;
}

// one CTA per bin, one thread per parameter: FP64 sums in the sorted (bin, slot) order
__global__ void adjoint_reduce_kernel(const int* __restrict__ val, const float* __restrict__ du, int P,
                                      const int* __restrict__ seg_b, const int* __restrict__ seg_e,
                                      const double* __restrict__ engnmfc, int b, int ermax, double* grad,
                                      double* wsum) {
  const int bin = blockIdx.x;
  const int i0 = seg_b[bin], i1 = seg_e[bin];
  if (i0 >= i1) return;
  const double w = engnmfc[b];
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    double acc = 0.0;
    for (int i = i0; i < i1; ++i) acc += (double)du[(size_t)val[i] * P + p];
    grad[(size_t)p * ermax + bin] += w * acc;
  }
  if (threadIdx.x == 0) wsum[bin] += w * (double)(i1 - i0);
}

// The same sums without a sort: CTA per bin, which lists its molecules in slot order from the
// keys, 4,096 at a time, and adds their derivatives, a thread per parameter (at most kAdjPar
// of each).  Every CTA reads every key: n ermax of them cost less than the sort's six launches
// until kAdjDirect (8,000 molecules and 1,396 bins, a third of it: 27 us against 23 for the sums of
// sorted molecules and 40 for the sort and the bounds; the rest is the fullest bin's chain of FP64
// additions, whose order is the slots').  An adjoint frame of that size 454 -> 372 us with the
// derivatives' kernel split over the sites.
// a float as a double by integer operations (exact): the conversion instruction is the FP64 pipe's,
// 64 clocks of a scheduler for a warp, as long as the addition that it feeds
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f), mag = u & 0x7fffffffu;
  if (mag - 1u < 0x007fffffu || mag >= 0x7f800000u) return (double)f;  // subnormal, infinite or NaN
  const unsigned hi = (u & 0x80000000u) | (mag == 0u ? 0u : (mag >> 3) + 0x38000000u);
  return __hiloint2double((int)hi, (int)(u << 29));
}
constexpr int kAdjThreads = 256, kAdjWindow = 4096;
constexpr int kAdjPar = (3 * kMaxSoluteSites + kAdjThreads - 1) / kAdjThreads;
constexpr long long kAdjDirect = 1ll << 25;
__global__ void __launch_bounds__(kAdjThreads) adjoint_bins_kernel(const int* __restrict__ key, int n,
                                                                   const float* __restrict__ du, int P,
                                                                   const double* __restrict__ engnmfc, int b, int ermax,
                                                                   double* grad, double* wsum) {
  constexpr int kWarps = kAdjThreads / 32, kPer = kAdjWindow / kAdjThreads;
  __shared__ int list[kAdjWindow];
  __shared__ int wcount[kWarps];
  const int bin = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc[kAdjPar];
#pragma unroll
  for (int i = 0; i < kAdjPar; ++i) acc[i] = 0.0;
  int count = 0;
  for (int w0 = 0; w0 < n; w0 += kAdjWindow) {
    unsigned m[kPer];
    int own = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {  // the warp's keys in order: 32 kPer consecutive ones
      const int at = w0 + (warp * kPer + i) * 32 + lane;
      m[i] = __ballot_sync(0xffffffffu, at < n && __ldg(key + min(at, n - 1)) == bin);
      own += __popc(m[i]);
    }
    if (lane == 0) wcount[warp] = own;
    if (!__syncthreads_or(own)) continue;  // most bins hold few molecules
    int at = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) at += wcount[w];
      total += wcount[w];
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (m[i] >> lane & 1u) list[at + __popc(m[i] & ((1u << lane) - 1u))] = w0 + (warp * kPer + i) * 32 + lane;
      at += __popc(m[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kAdjPar; ++i) {
      const int p = threadIdx.x + i * kAdjThreads;
      if (p >= P) break;
      for (int q = 0; q < total; q += 16) {  // 16 loads in flight; the adds in slot order
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = q + k < total ? du[(size_t)list[q + k] * P + p] : 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k)
          if (q + k < total) acc[i] += widen(v[k]);
      }
    }
    count += total;
    __syncthreads();  // the list is used again
  }
  if (count == 0) return;
  const double w = engnmfc[b];
#pragma unroll
  for (int i = 0; i < kAdjPar; ++i) {
    const int p = threadIdx.x + i * kAdjThreads;
    if (p < P) grad[(size_t)p * ermax + bin] += w * acc[i];
  }
  if (threadIdx.x == 0) wsum[bin] += w * (double)count;
}

int key_bits(int ermax) {
  int bits = 1;
  while ((1 << bits) <= ermax) ++bits;
  return bits;
}

}  // namespace

size_t adjoint_cub_bytes(int n) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (int*)nullptr, (int*)nullptr, (int*)nullptr, (int*)nullptr, n);
  return bytes;
}

cudaError_t launch_adjoint(Engine& e, const BatchArgs& a, cudaStream_t s) {
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const int n = e.slvmax;
  const int P = 3 * e.adj_ns;
  const int chunk = e.Bmax;
  int* key = e.d_adj_key;
  int* val = key + n;
  int* key_s = val + n;
  int* val_s = key_s + n;
  for (int b = 0; b < a.nb; ++b) {
    for (int s0 = 0; s0 < e.adj_ns; s0 += chunk) {
      const int nch = std::min(chunk, e.adj_ns - s0);
      adjoint_pseudo_kernel<<<nch, 128, 0, s>>>(a.u_bvec, b, s0, e.Kmax(), e.d_ps_nsite, e.d_ps_qf, e.d_ps_bvec);
      e.count_launch();
      BatchArgs pa = a;  // unit charges on single sites, this slot's grids and site terms
      pa.nb = nch;
      pa.u_nsite = e.d_ps_nsite;
      pa.u_qf = e.d_ps_qf;
      pa.u_bvec = e.d_ps_bvec;
      pa.self_part = e.d_ps_self;
      pa.stream = s;
      pa.phases = 0;
      if ((err = launch_pme_mixed(e, pa)) != cudaSuccess) return err;
      if ((err = launch_gather(e, pa)) != cudaSuccess) return err;
      MolArgs A = make_mol_args(e, a);
      AdjArgs J{};
      J.b = b;
      J.s_begin = s0;
      J.nchunk = nch;
      J.nsu = e.adj_ns;
      J.adj_mol = e.adj_mol;
      J.cmbrule = e.adj_cmbrule;
      J.first = (s0 == 0);
      J.site_e_ps = a.site_e;
      J.mol_bin = a.mol_bin + (size_t)b * n;
      J.par = e.d_adj_par;
      J.du = e.d_adj_du;
      J.key = key;
      J.val = val;
      adjoint_mol_kernel<<<(unsigned)(((long long)n * nch + 255) / 256), 256, 0, s>>>(A, J);
      e.count_launch();
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    if ((long long)n * e.ermax <= kAdjDirect) {
      adjoint_bins_kernel<<<e.ermax, kAdjThreads, 0, s>>>(key, n, e.d_adj_du, P, a.engnmfc, b, e.ermax, e.d_adj_grad,
                                                          e.d_adj_w);
      e.count_launch();
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
      continue;
    }
    size_t bytes = e.adj_cub_bytes;
    err = cub::DeviceRadixSort::SortPairs(e.d_adj_cub, bytes, key, key_s, val, val_s, n, 0, key_bits(e.ermax), s);
    if (err != cudaSuccess) return err;
    if ((err = cudaMemsetAsync(e.d_adj_seg, 0, sizeof(int) * 2 * (size_t)e.ermax, s)) != cudaSuccess) return err;
    adjoint_bounds_kernel<<<(n + 255) / 256, 256, 0, s>>>(key_s, n, e.ermax, e.d_adj_seg, e.d_adj_seg + e.ermax);
    adjoint_reduce_kernel<<<e.ermax, 64, 0, s>>>(val_s, e.d_adj_du, P, e.d_adj_seg, e.d_adj_seg + e.ermax, a.engnmfc,
                                                 b, e.ermax, e.d_adj_grad, e.d_adj_w);
    e.count_launch(2);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
  }
  return cudaSuccess;
}

}  // namespace ermod
