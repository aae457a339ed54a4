// kernels_accum.cu -- update_histogram's accumulation (engproc.F90:758-856).
//
//   accumulate    one CTA per batch: solute self energy u0 (engproc.F90:711-733), its
//                 weight engnmfc (wgtslf / volcorrect, engproc.F90:772-796,871-887),
//                 engnorm/engsmpl/avslf, eself, minuv/maxuv, flceng and slnuv, and
//                 edens += engnmfc * insdst.  Every FP64 sum runs in placement order, as
//                 in the reference's sequential loop, so results are bit-reproducible.
//                 A batch in which any molecule failed a bin check is not accumulated.
//   ecorr_digits, ecorr_mma   the ecorr update (engproc.F90:841-853) of the placements
//                 buffered in the ring as exact integer matrix products; the kernels below
//                 take what these do not (short rings, exact counts, weights too far apart).
//   ecorr_ff      the same sum by a walk of the placements in float-float registers.
//   ring_compact  per placement, the ascending list of occupied bins (bin, count).
//   ecorr_rows    ecorr(iduvp, iduv) += engnmfc * insdst(iduv) * insdst(iduvp)
//                 (engproc.F90:841-853) for the placements buffered in the ring: each
//                 CTA owns a few rows of the matrix in shared memory and walks the
//                 placements in order, touching only occupied (row, column) pairs; an
//                 exact int64 mirror sum insdst(i) insdst(j) is kept beside it.
#include <mutex>

#include "engine.cuh"

namespace ermod {

namespace {

struct AccArgs {
  BatchArgs a;
  int ntile, numslv, ermax, esmax, nself;
  int selfcal, wgtslf, soln, estype, rigid, mbin_mode;
  double temp, volume, volfac;  // volfac = pi Qtot^2 / beta^2 / V / 2 (volcorrect)
  double screen;                // residual_ene(slt, slt) = -(pi Q Q / beta / beta / V) / 2
  double stat_weight_system;
  int bare;      // cltype 0: no reciprocal self energy, no residual, volcorrect without its factor
  int ff_keys;   // the tile partials' min and max are ordered float-float keys (mixed path)
  double* scal;  // {engnorm, engsmpl, avslf, voffset, voffset_init, usreal, usreal_valid}
  double* edens;
  double* eself;
  double* slnuv;
  double* minuv;
  double* maxuv;
  const long long* eskey;
  int* ring_valid;  // [nb] entries of this batch in the ring
  double* ring_w;
  int slvmax;
  double* u0;      // [nb] solute self energies of the batch
  int* self_bin;   // [nb] eself bin (0-based) or -1
  DevStatus* status;
  // intermediate-state extension (solution mode), null when off
  const unsigned char* zmask;  // [ermax] 1 where the reference-solvent density is zero
  double* edintm;              // [ermax]
  double* uvintm;              // [numslv]
  double* iscal;               // {soln_total, soln_intm, norm_intm}
};

constexpr int kAccThreads = 256;
constexpr int kMaxBatch = 512;

// How many of the batch's placements are accumulated, given the call's first error.  Mixed
// path: none when the error lies in this batch or an earlier one.  FP64 path: those before
// the failing placement, as the reference's loop accumulates them.  Errors of later batches
// (already running on the other stream) do not count.  The answer cannot change between the
// accumulation kernels of a batch: the earlier batches' kernels are complete by then and the
// error key only decreases.
__device__ __forceinline__ int batch_accepted(const AccArgs& A) {
  const volatile unsigned long long* ek = &A.status->err_key;
  const unsigned long long k = *ek;
  if (k == kNoError) return A.a.nb;
  const long long before = (long long)(k >> 36) - A.a.b0;
  if (before >= A.a.nb) return A.a.nb;
  return (A.ff_keys || before <= 0) ? 0 : (int)before;
}

// fixed-order warp sum: lane t adds elements t, t + 32, ... in order, then a fixed tree
__device__ __forceinline__ double warp_sum_fixed(const double* x, int n, int stride) {
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < n; i += 32) s += x[(size_t)i * stride];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__device__ __forceinline__ void warp_min_max(double& mn, double& mx) {
  for (int o = 16; o > 0; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
}

// one placement, by one CTA: self energy u0, the self-energy bin check, and the per-species
// tile partials reduced to flceng / min / max (written to tile slot 0).  A warp per sum (the
// self energy's partials, then each species): their block-wide trees took 9 us a launch
__device__ void reduce_placement(const AccArgs& A, int b) {
  const BatchArgs& a = A.a;
  __shared__ double self_sum;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  for (int item = warp; item <= A.numslv; item += nwarp) {
    if (item == 0) {
      const double s = A.bare ? 0.0 : warp_sum_fixed(a.self_part + (size_t)b * A.nself, A.nself, 1);
      if (lane == 0) self_sum = s;
      continue;
    }
    const int sp = item - 1;
    double* base = a.part + ((size_t)b * A.ntile * A.numslv + sp) * 3;
    const int stride = A.numslv * 3;
    const double s = warp_sum_fixed(base, A.ntile, stride);
    double mn = INFINITY, mx = -INFINITY;
    for (int t = lane; t < A.ntile; t += 32) {
      const double* pt = base + (size_t)t * stride;
      if (A.ff_keys) {
        mn = fmin(mn, ff_key_to_double(reinterpret_cast<const long long*>(pt)[1]));
        mx = fmax(mx, ff_key_to_double(reinterpret_cast<const long long*>(pt)[2]));
      } else {
        mn = fmin(mn, pt[1]);
        mx = fmax(mx, pt[2]);
      }
    }
    warp_min_max(mn, mx);  // (every lane has read tile slot 0 before lane 0 overwrites it)
    if (lane == 0) {
      base[0] = s;
      base[1] = mn;
      base[2] = mx;
      if (a.flceng_out) a.flceng_out[(size_t)(a.b0 + b) * A.numslv + sp] = s;
    }
  }
  __syncthreads();
  const double self = self_sum;
  if (threadIdx.x == 0 && a.skip && a.skip[b]) {  // rejected by check_mol_configuration
    A.u0[b] = 0.0;
    A.self_bin[b] = -1;
    if (a.uvengy_out) a.uvengy_out[(size_t)(a.b0 + b) * (A.slvmax + 1)] = 0.0;
  } else if (threadIdx.x == 0) {
    double usreal;
    if (A.rigid)
      usreal = (A.scal[6] != 0.0) ? A.scal[5] : a.u_usreal[0];
    else
      usreal = a.u_usreal[b];
    const double qm = a.u_qmol[b];
    double epcl = A.bare ? 0.0 : kPi * qm * qm / A.screen / A.screen / A.volume;
    epcl = epcl / 2.0;
    const double residual = -epcl;
    double u0 = self;
    u0 = u0 + usreal + residual;  // uvengy(0) = uvengy(0) + pairep + residual
    A.u0[b] = u0;
    A.self_bin[b] = -1;
    if (a.uvengy_out) a.uvengy_out[(size_t)(a.b0 + b) * (A.slvmax + 1)] = u0;
    if (A.selfcal) {  // getiduv(0, uvengy(0))
      int code = 0, ret = 0;
      if (u0 != u0) {
        code = ERMOD_E_ENG_MIN;
      } else {
        const long long ku = ordered_key(u0);
        int lo = 0, hi = A.esmax;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (A.eskey[mid] < ku)
            lo = mid + 1;
          else
            hi = mid;
        }
        ret = lo;
        if (ret <= 0)
          code = ERMOD_E_ENG_MIN;
        else if (ret == A.esmax && u0 < 1.0e3 && A.mbin_mode != 0) {
          if (A.mbin_mode == 1)
            code = ERMOD_W_MBIN;
          else
            atomicOr(&A.status->mbin_hit, 1);
        }
      }
      if (code)
        atomicMin(&A.status->err_key, make_err_key(a.b0 + b, 0, code));
      else
        A.self_bin[b] = ret - 1;
    }
  }
}

__global__ void __launch_bounds__(kAccThreads) reduce_kernel(AccArgs A) { reduce_placement(A, blockIdx.x); }

// the batch's weights and scalar sums, by one CTA; every thread returns the number of
// placements accumulated
__device__ int accumulate_scalars(const AccArgs& A) {
  const BatchArgs& a = A.a;
  __shared__ double sw[kMaxBatch];
  __shared__ double stw[kMaxBatch];
  __shared__ double su0[kMaxBatch];
  __shared__ int sbin[kMaxBatch];
  __shared__ unsigned char srej[kMaxBatch];  // rejected by the configuration check
  __shared__ int accepted;
  __shared__ double s_voffset;
  for (int b = threadIdx.x; b < a.nb; b += blockDim.x) srej[b] = (a.skip && a.skip[b]) ? 1 : 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nb = accepted = batch_accepted(A);
    if (nb > 0 && A.wgtslf && A.scal[4] == 0.0) {
      // voffset from the first placement ever accumulated (update_histogram,
      // engproc.F90:779-783); rejected placements never reach it
      int first = 0;
      while (first < nb && srej[first]) ++first;
      if (first < nb) {
        A.scal[3] = A.u0[first];
        A.scal[4] = 1.0;
      }
    }
    if (nb > 0 && A.rigid && A.scal[6] == 0.0) {
      A.scal[5] = a.u_usreal[0];
      __threadfence();  // place_prep of a batch on another stream may see the flag
      A.scal[6] = 1.0;
    }
    s_voffset = A.scal[3];
  }
  __syncthreads();
  const int nb = accepted;
  for (int b = nb + threadIdx.x; b < a.nb; b += blockDim.x) {
    a.engnmfc[b] = 0.0;
    A.ring_valid[b] = 0;
  }
  if (nb == 0) return 0;
  // weights (parallel); u0 and the eself bins staged for the ordered sums
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    su0[b] = A.u0[b];
    sbin[b] = A.self_bin[b];
    if (srej[b]) {  // the loop's skipcond (engproc.F90:389-390): no update_histogram
      sw[b] = 0.0;
      stw[b] = 0.0;
      a.engnmfc[b] = 0.0;
      A.ring_w[b] = 0.0;
      A.ring_valid[b] = 0;
      continue;
    }
    double engnmfc;
    if (!A.wgtslf) {
      engnmfc = 1.0;
    } else {
      const double factor = su0[b] - s_voffset;
      engnmfc = A.soln ? exp(factor / A.temp) : exp(-factor / A.temp);
    }
    double total_weight = A.stat_weight_system * (a.stat_weight_solute ? a.stat_weight_solute[b] : 1.0);
    if (A.estype == 2) {
      total_weight = total_weight * A.volume;
      total_weight = total_weight * exp(A.volfac / A.temp);
    }
    engnmfc = engnmfc * total_weight;
    sw[b] = engnmfc;
    stw[b] = total_weight;
    a.engnmfc[b] = engnmfc;
    A.ring_w[b] = engnmfc;
    A.ring_valid[b] = 1;
  }
  __syncthreads();
  // ordered scalar sums (placement order, as the reference's loop), a warp's first thread each:
  // serial chains of FP64 adds, whose inputs are the shared weights (0 for a rejected
  // placement, which leaves a sum as it is).  256 placements, one thread for everything: 69 us
  if (threadIdx.x == 0 || threadIdx.x == 32) {
    const double* x = threadIdx.x == 0 ? sw : stw;
    double* to = A.scal + (threadIdx.x == 0 ? 0 : 2);  // engnorm, avslf
    double v = *to;
#pragma unroll 8
    for (int b = 0; b < nb; ++b) v = v + x[b];
    *to = v;
  } else if (threadIdx.x == 64 && A.selfcal) {
    for (int b = 0; b < nb; ++b)
      if (!srej[b]) A.eself[sbin[b]] += sw[b];
  } else if (threadIdx.x == 96) {
    int kept = 0;
    for (int b = 0; b < nb; ++b) kept += srej[b] ? 0 : 1;
    A.scal[1] += (double)kept;  // engsmpl: ones, exact in any order
  }
  // per species a warp: min/max over the batch, slnuv in placement order (species -1: the
  // solute self energies)
  for (int sp = (int)(threadIdx.x >> 5) - 1; sp < A.numslv; sp += blockDim.x >> 5) {
    const int lane = threadIdx.x & 31;
    double mn = INFINITY, mx = -INFINITY;
    for (int b = lane; b < nb; b += 32) {
      const double* pt = a.part + ((size_t)b * A.ntile * A.numslv + max(sp, 0)) * 3;
      if (sp < 0 && srej[b]) continue;
      mn = fmin(mn, sp < 0 ? su0[b] : pt[1]);
      mx = fmax(mx, sp < 0 ? su0[b] : pt[2]);
    }
    warp_min_max(mn, mx);
    if (lane == 0) {
      A.minuv[sp + 1] = fmin(A.minuv[sp + 1], mn);
      A.maxuv[sp + 1] = fmax(A.maxuv[sp + 1], mx);
      if (A.soln && sp >= 0) {
        double sl = A.slnuv[sp];
        for (int b = 0; b < nb; ++b)
          if (!srej[b]) sl = sl + a.part[((size_t)b * A.ntile * A.numslv + sp) * 3] * sw[b];
        A.slnuv[sp] = sl;
      }
    }
  }
  __syncthreads();
  if (!A.zmask) return nb;  // edens: accumulate_bins
  // edens += engnmfc * insdst, placements in order
  for (int i = threadIdx.x; i < A.ermax; i += blockDim.x) {
    double e = A.edens[i];
    bool touched = false;
    for (int b = 0; b < nb; ++b) {
      const int c = a.hist[(size_t)b * A.ermax + i];
      if (c) {
        e = e + sw[b] * (double)c;
        touched = true;
      }
    }
    if (touched) A.edens[i] = e;
  }
  // intermediate state (extensions/Intermediate/engproc.F90, update_histogram hunk):
  // a placement belongs to it when none of its occupied bins has zero density in the
  // reference solvent; its weight, histogram and flceng then accumulate separately
  if (A.zmask) {
    __shared__ unsigned char sout[kMaxBatch];
    for (int b = 0; b < nb; ++b) {
      int out = 0;
      for (int i = threadIdx.x; i < A.ermax; i += blockDim.x)
        if (A.zmask[i] && a.hist[(size_t)b * A.ermax + i] > 0) out = 1;
      out = __syncthreads_or(out);
      if (threadIdx.x == 0) sout[b] = (unsigned char)out;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double tot = A.iscal[0], in = A.iscal[1], nrm = A.iscal[2];
      for (int b = 0; b < nb; ++b) {
        if (srej[b]) continue;
        tot = tot + sw[b];
        if (!sout[b]) {
          in = in + sw[b];
          nrm = nrm + sw[b];
        }
      }
      A.iscal[0] = tot;
      A.iscal[1] = in;
      A.iscal[2] = nrm;
    }
    for (int i = threadIdx.x; i < A.ermax; i += blockDim.x) {
      double e = A.edintm[i];
      for (int b = 0; b < nb; ++b) {
        const int c = a.hist[(size_t)b * A.ermax + i];
        if (c > 0 && !sout[b]) e = e + sw[b] * (double)c;
      }
      A.edintm[i] = e;
    }
    for (int sp = threadIdx.x; sp < A.numslv; sp += blockDim.x) {
      double u = A.uvintm[sp];
      for (int b = 0; b < nb; ++b)
        if (!sout[b]) u = u + a.part[((size_t)b * A.ntile * A.numslv + sp) * 3] * sw[b];
      A.uvintm[sp] = u;
    }
  }
  return nb;
}

__global__ void __launch_bounds__(kAccThreads) accumulate_kernel(AccArgs A) { accumulate_scalars(A); }

// edens(i) += engnmfc * insdst(i) (engproc.F90:836-838) by one thread, the batch's placements
// in order (so the FP64 sums are those of the reference's loop); the intermediate-state mode
// does this inside accumulate_scalars instead.  A serial chain of FMAs; the counts of the next
// kBinAhead placements load while it runs, and a warp whose bins are all empty skips theirs.
constexpr int kBinAhead = 16;
__device__ __forceinline__ void accumulate_bin(const AccArgs& A, int i, int nb, const double* sw) {
  const int* h = A.a.hist + i;
  const size_t E = (size_t)A.ermax;
  double e = A.edens[i];
  int touched = 0;
  int next[kBinAhead];
#pragma unroll
  for (int u = 0; u < kBinAhead; ++u) next[u] = u < nb ? h[(size_t)u * E] : 0;
  for (int b = 0; b < nb; b += kBinAhead) {
    int c[kBinAhead], any = 0;
#pragma unroll
    for (int u = 0; u < kBinAhead; ++u) {
      c[u] = next[u];
      any |= c[u];
      next[u] = b + kBinAhead + u < nb ? h[(size_t)(b + kBinAhead + u) * E] : 0;
    }
    if (any) {
      touched = 1;
#pragma unroll
      for (int u = 0; u < kBinAhead; ++u)
        if (c[u]) e = fma(sw[b + u], (double)c[u], e);
    }
  }
  if (touched) A.edens[i] = e;
}

// one warp per block: the FP64 pipe takes 16 clocks per warp instruction and SM, so the bins
// are spread over the SMs (256 placements of 1,396 bins: 40 us in blocks of 128)
constexpr int kBinThreads = 32;
__global__ void __launch_bounds__(kBinThreads) accumulate_bins_kernel(AccArgs A) {
  const int nb = batch_accepted(A);
  if (nb <= 0) return;  // the batch was not accumulated (an error)
  __shared__ double sw[kMaxBatch];
  for (int b = threadIdx.x; b < nb; b += blockDim.x) sw[b] = A.a.engnmfc[b];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < A.ermax) accumulate_bin(A, i, nb, sw);
}

// A batch of one or two placements (a solution-mode frame): the three steps in one launch
constexpr int kSmallBatch = 2;
constexpr int kSmallThreads = 512;
__global__ void __launch_bounds__(kSmallThreads) accumulate_small_kernel(AccArgs A) {
  for (int b = 0; b < A.a.nb; ++b) reduce_placement(A, b);
  __syncthreads();
  const int nb = accumulate_scalars(A);
  if (nb == 0 || A.zmask) return;
  __syncthreads();
  double w[kSmallBatch];
#pragma unroll
  for (int b = 0; b < kSmallBatch; ++b) w[b] = b < nb ? A.a.engnmfc[b] : 0.0;
  for (int i = threadIdx.x; i < A.ermax; i += blockDim.x) {
    int c[kSmallBatch];
#pragma unroll
    for (int b = 0; b < kSmallBatch; ++b) c[b] = b < nb ? A.a.hist[(size_t)b * A.ermax + i] : 0;
    if (!(c[0] | c[1])) continue;
    double e = A.edens[i];
#pragma unroll
    for (int b = 0; b < kSmallBatch; ++b)
      if (c[b]) e = fma(w[b], (double)c[b], e);
    A.edens[i] = e;
  }
}
static_assert(kSmallBatch == 2, "the counts of two placements tested together");

// occupied-bin list per ring entry: entries (bin << 0) with counts beside them
__global__ void __launch_bounds__(256) ring_compact_kernel(const int* __restrict__ hist, const int* __restrict__ valid,
                                                         int ermax, const int* __restrict__ mma,
                                                         int* __restrict__ nz_bin, int* __restrict__ nz_cnt,
                                                         int* __restrict__ nnz) {
  if (mma && *mma) return;  // summed by the matrix kernels
  const int p = blockIdx.x;
  const int* h = hist + (size_t)p * ermax;
  __shared__ int scan[256];
  const int per = (ermax + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = min(ermax, lo + per);
  int cnt = 0;
  if (valid[p])
    for (int i = lo; i < hi; ++i) cnt += (h[i] != 0);
  scan[threadIdx.x] = cnt;
  __syncthreads();
  for (int off = 1; off < blockDim.x; off <<= 1) {  // inclusive Hillis-Steele scan
    const int v = (threadIdx.x >= off) ? scan[threadIdx.x - off] : 0;
    __syncthreads();
    scan[threadIdx.x] += v;
    __syncthreads();
  }
  int pos = scan[threadIdx.x] - cnt;
  if (valid[p])
    for (int i = lo; i < hi; ++i)
      if (h[i]) {
        nz_bin[(size_t)p * ermax + pos] = i;
        nz_cnt[(size_t)p * ermax + pos] = h[i];
        ++pos;
      }
  if (threadIdx.x == blockDim.x - 1) nnz[p] = valid[p] ? scan[threadIdx.x] : 0;
}

__global__ void __launch_bounds__(256) ecorr_rows_kernel(const int* __restrict__ hist, const int* __restrict__ nz_bin,
                                                       const int* __restrict__ nz_cnt, const int* __restrict__ nnz,
                                                       const double* __restrict__ w, int nring, int ermax, int R,
                                                       const int* __restrict__ mma, double* __restrict__ ecorr,
                                                       long long* __restrict__ ecorr_n) {
  if (mma && *mma) return;  // summed by the matrix kernels
  extern __shared__ double srow[];  // [R][ermax] (+ [R][ermax] int64 mirror)
  long long* srow_n = reinterpret_cast<long long*>(srow + (size_t)R * ermax);
  const int row0 = blockIdx.x * R;
  const int nrow = min(R, ermax - row0);
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int t = threadIdx.x; t < nring * nrow; t += blockDim.x) {
    const int p = t / nrow, r = t % nrow;
    if (nnz[p] > 0 && hist[(size_t)p * ermax + row0 + r] != 0) any = 1;
  }
  __syncthreads();
  if (!any) return;
  for (int t = threadIdx.x; t < nrow * ermax; t += blockDim.x) {
    srow[t] = ecorr[(size_t)row0 * ermax + t];
    if (ecorr_n) srow_n[t] = ecorr_n[(size_t)row0 * ermax + t];
  }
  __syncthreads();
  for (int p = 0; p < nring; ++p) {
    const int n = nnz[p];
    if (n == 0) continue;
    const int* bins = nz_bin + (size_t)p * ermax;
    const int* cnts = nz_cnt + (size_t)p * ermax;
    for (int r = 0; r < nrow; ++r) {
      const int ci = hist[(size_t)p * ermax + row0 + r];
      if (ci == 0) continue;
      const double wi = w[p] * (double)ci;
      double* row = srow + (size_t)r * ermax;
      long long* rown = srow_n + (size_t)r * ermax;
      for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int j = bins[t];
        const int cj = cnts[t];
        row[j] = row[j] + wi * (double)cj;
        if (ecorr_n) rown[j] += (long long)ci * (long long)cj;
      }
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < nrow * ermax; t += blockDim.x) {
    ecorr[(size_t)row0 * ermax + t] = srow[t];
    if (ecorr_n) ecorr_n[(size_t)row0 * ermax + t] = srow_n[t];
  }
}

// the dynamic shared memory of ecorr_rows_kernel, shared by the FP64 flush and the
// no-allocation entry point: one record, so that a caller needing less never lowers the
// size another caller has set
SmemAttr& ecorr_rows_attr() {
  static SmemAttr attr;
  return attr;
}

// what the flush's kernels need to know of the ring
struct RingInfo {
  int nact;  // active bins
  int emax;  // binary exponent of the largest weight: w = f 2^emax, f in [1/2, 1)
  int mma;   // 1: the matrix kernels sum this flush, 0: the walk (weights or bins out of their range)
};


// Mixed path flush, same sum as ecorr_rows_kernel.  A CTA owns kEcRows rows and 256
// columns of the matrix; thread t owns one column and keeps the flush's contribution
// to its kEcRows entries in registers as float-float pairs (exact products by fma,
// TwoSum additions: ~44 significant bits), walking the ring's placements in order.
// No two threads share an entry, so the walk needs no barrier and its loads pipeline;
// the pairs are added to the FP64 matrix once per flush.  The row coefficients
// hist[p][row0 + r] of every placement are staged in shared memory with a bit mask of
// the nonzero ones.
constexpr int kEcRows = 8;

__device__ __forceinline__ void ff_add_prod(float& hi, float& lo, float wh, float wl, float c) {
  const float p = wh * c;
  float pe = fmaf(wh, c, -p);  // exact low part of wh * c
  pe = fmaf(wl, c, pe);
  const float s = hi + p;  // TwoSum(hi, p)
  const float bb = s - hi;
  const float err = (hi - (s - bb)) + (p - bb);
  lo += err + pe;
  hi = s;
}

// The rows and columns walked are the flush's active bins only (act[0 .. *nact): the bins
// some placement of the ring occupies, in increasing order), so a coordinate of thousands
// of bins costs what its occupied part costs; an inactive row or column has no
// contribution, so the sums are those of the walk over every bin.  The matrix is
// symmetric: only entries on or above the diagonal (column index >= row index in act) are
// summed, and each is added at (row, column) and (column, row), so that both halves get
// the same value from one sum.
template <bool COUNT>
__global__ void __launch_bounds__(256, 2) ecorr_ff_kernel(const int* __restrict__ hist, const int* __restrict__ valid,
                                                        const double* __restrict__ w, int nring, int ermax,
                                                        const int* __restrict__ act, const RingInfo* __restrict__ info,
                                                        double* __restrict__ ecorr, long long* __restrict__ ecorr_n) {
  extern __shared__ float2 sdyn2[];
  float2* sa = sdyn2;  // [nring][kEcRows]: w_p * hist[p][row r's bin] as a float-float pair
  unsigned* smask = reinterpret_cast<unsigned*>(sa + (size_t)nring * kEcRows);  // [nring]
  int* sci = reinterpret_cast<int*>(smask + nring);  // [nring][kEcRows] counts (count mirror only)
  if (info->mma) return;  // summed by the matrix kernels
  const int nact = info->nact;
  const int row0 = blockIdx.y * kEcRows;
  if (row0 >= nact) return;  // the grid covers every bin; the active ones come first
  if ((int)(blockIdx.x * blockDim.x + blockDim.x) <= row0) return;  // all below the diagonal
  const int nrow = min(kEcRows, nact - row0);
  int rbin[kEcRows];
#pragma unroll
  for (int r = 0; r < kEcRows; ++r) rbin[r] = act[row0 + min(r, nrow - 1)];
  const int jj = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = jj < nact ? act[jj] : ermax;  // this thread's column (ermax: none)
  for (int p = threadIdx.x; p < nring; p += blockDim.x) {
    unsigned m = 0;
    const bool ok = valid[p] != 0;
    const double wd = w[p];
    const float wh = (float)wd;
    const float wl = (float)(wd - (double)wh);
    for (int r = 0; r < kEcRows; ++r) {
      const int c = (ok && r < nrow) ? hist[(size_t)p * ermax + rbin[r]] : 0;
      // w * c as a float-float pair (c < 2^24 is exact in FP32; the high product is
      // split exactly by fma)
      const float fc = (float)c;
      const float ah = wh * fc;
      const float al = fmaf(wl, fc, fmaf(wh, fc, -ah));
      sa[p * kEcRows + r] = make_float2(ah, al);
      if (COUNT) sci[p * kEcRows + r] = c;
      if (c) m |= 1u << r;
    }
    smask[p] = m;
  }
  __syncthreads();
  if (j >= ermax || jj < row0) return;
  // rows r <= jj - row0 of this column are on or above the diagonal
  const unsigned rows_on = (jj - row0 >= kEcRows - 1) ? 0xffu : ((2u << (jj - row0)) - 1u);
  float hi[kEcRows], lo[kEcRows];
  long long cn[COUNT ? kEcRows : 1];
#pragma unroll
  for (int r = 0; r < kEcRows; ++r) {
    hi[r] = 0.f;
    lo[r] = 0.f;
    if (COUNT) cn[r] = 0;
  }
  bool any = false;
  constexpr int U = 4;  // loads in flight per thread
  for (int p0 = 0; p0 < nring; p0 += U) {
    int cj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = p0 + u;
      cj[u] = (p < nring && smask[p]) ? __ldg(hist + (size_t)p * ermax + j) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (cj[u] == 0) continue;
      const int p = p0 + u;
      any = true;
      const unsigned m = smask[p] & rows_on;
      const float c = (float)cj[u];
      const float2* ap = sa + p * kEcRows;
#pragma unroll
      for (int r = 0; r < kEcRows; ++r) {
        if (m & (1u << r)) {
          const float2 a = ap[r];
          ff_add_prod(hi[r], lo[r], a.x, a.y, c);
          if (COUNT) cn[r] += (long long)sci[p * kEcRows + r] * (long long)cj[u];
        }
      }
    }
  }
  if (!any) return;
#pragma unroll
  for (int r = 0; r < kEcRows; ++r) {
    if (r >= nrow) break;
    const size_t at = (size_t)rbin[r] * ermax + j, ta = (size_t)j * ermax + rbin[r];
    if (hi[r] != 0.f || lo[r] != 0.f) {
      const double v = (double)hi[r] + (double)lo[r];
      ecorr[at] = ecorr[at] + v;
      if (ta != at) ecorr[ta] = ecorr[ta] + v;
    }
    if (COUNT && cn[r] != 0) {
      ecorr_n[at] += cn[r];
      if (ta != at) ecorr_n[ta] += cn[r];
    }
  }
}

// The flush's active bins: top[i] = the largest count of bin i over the ring's valid placements
// (top zeroed first; 0: no placement occupies it).  CTA per (256 bins, 32 placements): the 32
// loads of a thread are independent and in flight together.
constexpr int kActivePlacements = 32;
__global__ void __launch_bounds__(256) ring_active_kernel(const int* __restrict__ hist, const int* __restrict__ valid,
                                                        int nring, int ermax, int* __restrict__ top) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int p0 = blockIdx.y * kActivePlacements;
  if (i >= ermax) return;
  int c[kActivePlacements];
#pragma unroll
  for (int u = 0; u < kActivePlacements; ++u) {
    const int p = p0 + u;
    c[u] = (p < nring && valid[p]) ? __ldg(hist + (size_t)p * ermax + i) : 0;
  }
  int most = 0;
#pragma unroll
  for (int u = 0; u < kActivePlacements; ++u) most = max(most, c[u]);
  if (most) atomicMax(&top[i], most);
}

// act[0 .. nact) = the active bins in increasing order, atop their largest counts, and whether
// the matrix kernels may sum the flush: at most max_bins active bins and positive finite weights
// whose exponents differ by at most spread (one CTA, chunks of 1024)
__global__ void __launch_bounds__(1024) ring_active_list_kernel(const int* __restrict__ top, int ermax,
                                                              const int* __restrict__ valid,
                                                              const double* __restrict__ w, int nring, int max_bins,
                                                              int spread, int all, int* __restrict__ act,
                                                              int* __restrict__ atop, RingInfo* __restrict__ info) {
  __shared__ int warp_sum[32];
  __shared__ int s_max, s_min, s_bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    s_max = -100000;
    s_min = 100000;
    s_bad = 0;
  }
  __syncthreads();
  int base = 0;
  for (int c0 = 0; c0 < ermax; c0 += 1024) {
    const int i = c0 + (int)threadIdx.x;
    const int t = i < ermax ? (all ? 1 : top[i]) : 0;
    const unsigned m = __ballot_sync(0xffffffffu, t != 0);
    if (lane == 0) warp_sum[warp] = __popc(m);
    __syncthreads();
    int before = __popc(m & ((1u << lane) - 1u)), total = 0;
    for (int k = 0; k < 32; ++k) {
      if (k < warp) before += warp_sum[k];
      total += warp_sum[k];
    }
    if (t) {
      act[base + before] = i;
      atop[base + before] = t;
      if (t >= 1 << 24) s_bad = 1;  // more digits than the planes hold
    }
    __syncthreads();  // warp_sum read by every thread before the next chunk overwrites it
    base += total;
  }
  int emx = -100000, emn = 100000;
  for (int p = threadIdx.x; p < nring; p += 1024) {
    if (!valid[p]) continue;
    const double x = w[p];
    if (x == 0.0) continue;
    if (!(x > 0.0) || isinf(x)) {
      s_bad = 1;
      continue;
    }
    const int e = ilogb(x) + 1;
    emx = max(emx, e);
    emn = min(emn, e);
  }
  atomicMax(&s_max, emx);
  atomicMin(&s_min, emn);
  __syncthreads();
  if (threadIdx.x == 0) {
    info->nact = base;
    info->emax = s_max;
    info->mma = (!all && !s_bad && base <= max_bins && s_max >= s_min && s_max - s_min <= spread) ? 1 : 0;
  }
}

// ---- the flush as exact integer matrix products ------------------------------------------
// ecorr(i, j) += sum_p w_p h_p(i) h_p(j), a product of (bins x placements) matrices.  With the
// weights as integers m_p = w_p 2^(T - emax) (T = 60, FP64 path 63: a weight whose exponent is
// within the spread of the largest, 12 or 10, keeps 48 bits, as the walk's float-float pairs hold
// it, or all 53), m_p h_p(i) is cut into 7-bit digits and h_p(j) into 8-bit ones: their bf16
// values are exact, and the FP32 sums of 512 products of two digits are integers below 2^24,
// exact too.  So mma.sync adds the digit planes without error, and each entry is rounded once
// per 35 bits of planes when they are joined.  512 placements, with the two kernels before: 168 ->
// 97 us for 4,000 waters, 294 -> 130 us for 33,000 (float-float sums by the walk below); FP64
// path, 64 placements of 4,000 waters 253 -> 45 us.
constexpr int kMmaK = 512;         // placements per pass (a longer ring takes several)
constexpr int kMmaBins = 2048;     // active bins, at most
constexpr int kMaxADigits = 13;    // 7-bit digits of m h: T + 24 bits of a count
constexpr int kMaxBDigits = 3;     // 8-bit digits of a count below 2^24
constexpr int kMmaMinRing = 48;    // placements in the ring for the matrix kernels to pay

__device__ __forceinline__ int bit_length(int x) { return 32 - __clz(x); }
__device__ __forceinline__ int a_digits(int T, int top) { return (T + 1 + bit_length(top) + 6) / 7; }
__device__ __forceinline__ int b_digits(int top) { return (bit_length(top) + 7) / 8; }
// the largest count of 16 active bins from block ib on (by a whole warp)
__device__ __forceinline__ int block_top(const int* atop, int nact, int ib) {
  const int i = 16 * ib + (threadIdx.x & 15);
  return max(1, __reduce_max_sync(0xffffffffu, i < nact ? atop[i] : 0));
}

// the digits in the order of mma.m16n8k16's fragments: [plane][block of 16 bins][block of 16
// placements][lane][8].  A warp per block of 16 x 16: lane (g, t) = (lane / 4, lane % 4) holds
// bins g and g + 8 and placements 2 t, 2 t + 1, + 8 of it.
__global__ void __launch_bounds__(256) ecorr_digits_kernel(const int* __restrict__ hist, const int* __restrict__ valid,
                                                         const double* __restrict__ w, int p0, int n, int ermax, int T,
                                                         int nbins, const int* __restrict__ act,
                                                         const int* __restrict__ atop, const RingInfo* __restrict__ info,
                                                         uint4* __restrict__ A, uint4* __restrict__ B) {
  const RingInfo I = *info;
  const int ib = blockIdx.x, kb = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int nkb = (n + 15) / 16;
  if (!I.mma || 16 * ib >= I.nact || kb >= nkb) return;
  const int g = lane >> 2, t = lane & 3;
  const int top = block_top(atop, I.nact, ib);
  const int na = a_digits(T, top), nb = b_digits(top);
  unsigned long long lo[8], hi[8];
  int h[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {  // e = 4 (placement + 8) + 2 (bin + 8) + (placement + 1)
    const int i = 16 * ib + g + ((e >> 1) & 1) * 8, k = 16 * kb + 2 * t + (e & 1) + (e >> 2) * 8;
    const int p = p0 + k;
    h[e] = (k < n && i < I.nact && valid[p]) ? __ldg(hist + (size_t)p * ermax + act[i]) : 0;
    unsigned long long m = 0;
    if (h[e]) m = (unsigned long long)__double2ull_rn(ldexp(w[p], T - I.emax));
    lo[e] = m * (unsigned long long)h[e];
    hi[e] = __umul64hi(m, (unsigned long long)h[e]);
  }
  auto bf = [](unsigned a, unsigned b) {  // two digits below 256 as bf16, exactly
    return (__float_as_uint((float)a) >> 16) | (__float_as_uint((float)b) & 0xffff0000u);
  };
  const size_t nib = (size_t)nbins / 16, at = ((size_t)ib * (kMmaK / 16) + kb) * 32 + lane;
  const size_t plane = nib * (kMmaK / 16) * 32;
  for (int l = 0; l < na; ++l) {
    unsigned d[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      d[e] = (unsigned)lo[e] & 127u;
      lo[e] = (lo[e] >> 7) | (hi[e] << 57);
      hi[e] >>= 7;
    }
    A[l * plane + at] = make_uint4(bf(d[0], d[1]), bf(d[2], d[3]), bf(d[4], d[5]), bf(d[6], d[7]));
  }
  for (int m = 0; m < nb; ++m) {
    unsigned d[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) d[e] = ((unsigned)h[e] >> (8 * m)) & 255u;
    // as the second operand: bins g (then g + 8), for each the placements and those + 8
    B[m * plane + at] = make_uint4(bf(d[0], d[1]), bf(d[4], d[5]), bf(d[2], d[3]), bf(d[6], d[7]));
  }
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4& a, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
      "%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// CTA per 32 x 32 active bins on or above the diagonal.  The digit planes' products come from
// fragments in L2; a warp takes five planes, joined as 64-bit integers, and a quarter of the
// placements, so that the loads' latency is paid a few times over and not once per plane and
// round (one warp per tile: twice the time); the warps' integers are added exactly and joined
// in FP64.  Bound by that latency still: two CTAs to an SM take 68 us a flush of 512 placements
// of 4,000 waters, one with more loads in flight per warp 120.  Each entry is added at both mirrored positions.
constexpr int kMmaWarps = 8, kMmaParts = 4;
__global__ void __launch_bounds__(32 * kMmaWarps, 2) ecorr_mma_kernel(const uint4* __restrict__ A,
                                                                 const uint4* __restrict__ B, int n, int ermax, int T,
                                                                 int nbins, const int* __restrict__ act,
                                                                 const int* __restrict__ atop,
                                                                 const RingInfo* __restrict__ info,
                                                                 double* __restrict__ ecorr) {
  extern __shared__ long long sq[];  // [kMmaWarps][32 entries of a lane][32 lanes]
  const RingInfo I = *info;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  if (!I.mma || c0 < r0 || r0 >= I.nact || c0 >= I.nact) return;
  const int nkb = (n + 15) / 16;
  const int nblk = (I.nact + 15) / 16;  // blocks of 16 bins written
  const int rb = r0 / 16, cb = c0 / 16;
  const bool r1 = rb + 1 < nblk, c1 = cb + 1 < nblk;
  const size_t row = (size_t)(kMmaK / 16) * 32, plane = (size_t)(nbins / 16) * row;
  // a block's planes beyond its own digits were not written: each block has its own count
  const int top0 = block_top(atop, I.nact, rb), top1 = block_top(atop, I.nact, rb + 1);
  const int cop0 = block_top(atop, I.nact, cb), cop1 = block_top(atop, I.nact, cb + 1);
  const int na0 = a_digits(T, top0), na1 = r1 ? a_digits(T, top1) : 0, na = max(na0, na1);
  const int nb0 = b_digits(cop0), nb1 = c1 ? b_digits(cop1) : 0;
  const int part = warp % kMmaParts, half = warp / kMmaParts;
  const int nround = (na + 9) / 10;  // two groups of five planes at a time
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  double S[4] = {0.0, 0.0, 0.0, 0.0};  // the entries, all digits of the second operand joined
  for (int m = max(nb0, nb1) - 1; m >= 0; --m) {
    double R[4] = {0.0, 0.0, 0.0, 0.0};
    for (int round = nround - 1; round >= 0; --round) {
      const int l0 = 10 * round + 5 * half;
      long long q[2][4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) q[i][j][e] = 0;
      for (int l = min(l0 + 4, na - 1); l >= l0; --l) {
        float c[2][4][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) c[i][j][e] = 0.f;
        const uint4* a = A + l * plane + rb * row + lane;
        const uint4* b = B + m * plane + cb * row + lane;
#pragma unroll 2
        for (int kb = part; kb < nkb; kb += kMmaParts) {
          const uint4 a0 = l < na0 ? __ldg(a + kb * 32) : zero, a1 = l < na1 ? __ldg(a + row + kb * 32) : zero;
          const uint4 b0 = m < nb0 ? __ldg(b + kb * 32) : zero, b1 = m < nb1 ? __ldg(b + row + kb * 32) : zero;
          mma_bf16(c[0][0], a0, b0.x, b0.y);
          mma_bf16(c[0][1], a0, b0.z, b0.w);
          mma_bf16(c[0][2], a0, b1.x, b1.y);
          mma_bf16(c[0][3], a0, b1.z, b1.w);
          mma_bf16(c[1][0], a1, b0.x, b0.y);
          mma_bf16(c[1][1], a1, b0.z, b0.w);
          mma_bf16(c[1][2], a1, b1.x, b1.y);
          mma_bf16(c[1][3], a1, b1.z, b1.w);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) q[i][j][e] = q[i][j][e] * 128 + __float2int_rn(c[i][j][e]);
      }
      __syncthreads();  // the round before has been read
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) sq[(warp * 32 + i * 16 + j * 4 + e) * 32 + lane] = q[i][j][e];
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int at = warp + 8 * u;  // entry of each lane
        long long lo = 0, hi = 0;
#pragma unroll
        for (int p = 0; p < kMmaParts; ++p) {
          lo += sq[(p * 32 + at) * 32 + lane];
          hi += sq[((p + kMmaParts) * 32 + at) * 32 + lane];
        }
        R[u] = fma(fma(R[u], 34359738368.0, (double)hi), 34359738368.0, (double)lo);  // 2^35 per five planes
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) S[u] = fma(S[u], 256.0, R[u]);
  }
  // (weights below 1e-304 have no unit in a double: their entries are scaled by ldexp)
  const int ex = I.emax - T;
  const double unit = ldexp(1.0, ex);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    // entry (i, j, e) of the fragments: row 16 i + lane / 4 (+ 8 for e >= 2), column 8 j + 2 (lane % 4) + (e & 1)
    const int at = warp + 8 * u, i = at >> 4, j = (at >> 2) & 3, e = at & 3;
    const int ri = r0 + 16 * i + (lane >> 2) + (e >> 1) * 8, ci = c0 + 8 * j + 2 * (lane & 3) + (e & 1);
    if (ci < ri || ci >= I.nact || S[u] == 0.0) continue;
    const double v = unit > 0.0 ? S[u] * unit : ldexp(S[u], ex);
    const size_t br = act[ri], bc = act[ci];
    // one addition per entry and launch: an atomic one only so that no thread waits for it
    atomicAdd(ecorr + br * ermax + bc, v);
    if (br != bc) atomicAdd(ecorr + bc * ermax + br, v);
  }
}

// Coordinates of at most this many bins walk every bin in ecorr_ff_kernel: on the 33,000-water
// workload (1,396 bins, about 900 of them active in a flush) the gathered walk over the active
// ones was slower than the contiguous walk over all.
constexpr int kActiveMinBins = 2048;

size_t mma_bins(int ermax) { return ((size_t)std::min(ermax, kMmaBins) + 63) / 64 * 64; }

}  // namespace

int accumulate_max_batch() { return kMaxBatch; }

cudaError_t launch_accumulate(Engine& e, const BatchArgs& a, cudaStream_t s) {
  AccArgs A{};
  A.a = a;
  A.ntile = e.ntile;
  A.numslv = e.numslv;
  A.ermax = e.ermax;
  A.esmax = e.esmax;
  A.nself = e.mixed ? spectrum_partials(e) : spectrum64_partials(e);
  A.selfcal = e.P.selfcal;
  A.wgtslf = e.P.wgtslf;
  A.soln = e.P.slttype == 1;
  A.estype = e.P.estype;
  A.rigid = e.P.slttype == 2;
  A.mbin_mode = e.warn_bin_firsttime ? (e.P.force_calculation ? 2 : 1) : 0;
  A.temp = e.P.temp;
  A.volume = e.geom.volume;
  A.bare = (e.P.cltype == 0) ? 1 : 0;
  A.ff_keys = e.mixed ? 1 : 0;
  A.volfac = A.bare ? 0.0  // volcorrect multiplies by the volume only (engproc.F90:871-887)
                    : kPi * (e.total_charge_phys * e.total_charge_phys) / (e.P.screen * e.P.screen) / e.geom.volume / 2.0;
  A.screen = e.P.screen;
  A.stat_weight_system = e.stat_weight_system;
  A.scal = e.d_scal;
  A.edens = e.d_edens;
  A.eself = e.d_eself;
  A.slnuv = e.d_slnuv;
  A.minuv = e.d_minuv;
  A.maxuv = e.d_maxuv;
  A.eskey = e.d_eskey;
  A.ring_valid = e.d_ring_valid + e.ring_off + e.ring_fill;
  A.ring_w = e.d_ring_w + e.ring_off + e.ring_fill;
  A.slvmax = e.slvmax;
  A.u0 = a.u0;
  A.self_bin = a.self_bin;
  A.status = e.d_status;
  if (e.d_int_mask) {
    A.zmask = e.d_int_mask;
    A.edintm = e.d_edintm;
    A.uvintm = e.d_edintm + e.ermax;
    A.iscal = e.d_edintm + e.ermax + e.numslv;
  }
  if (a.nb <= kSmallBatch) {
    accumulate_small_kernel<<<1, kSmallThreads, 0, s>>>(A);
    e.count_launch();
    return cudaGetLastError();
  }
  reduce_kernel<<<a.nb, kAccThreads, 0, s>>>(A);
  accumulate_kernel<<<1, kAccThreads, 0, s>>>(A);
  e.count_launch(2);
  if (!A.zmask) {
    accumulate_bins_kernel<<<(e.ermax + kBinThreads - 1) / kBinThreads, kBinThreads, 0, s>>>(A);
    e.count_launch();
  }
  return cudaGetLastError();
}

size_t ecorr_digits_bytes(int ermax) {
  return sizeof(uint4) * mma_bins(ermax) / 16 * (kMmaK / 16) * 32 * (kMaxADigits + kMaxBDigits);
}
size_t ecorr_scratch_ints(int ermax) { return 3 * (size_t)ermax + sizeof(RingInfo) / sizeof(int); }

cudaError_t launch_ecorr_flush(Engine& e, cudaStream_t s) {
  if (e.ring_fill == 0) return cudaSuccess;
  const int n = e.ring_fill;
  const bool count = e.d_ecorr_n != nullptr;
  const int* hist = e.d_ring_hist + (size_t)e.ring_off * e.ermax;
  const int* valid = e.d_ring_valid + e.ring_off;
  const double* w = e.d_ring_w + e.ring_off;
  int* top = e.d_ring_act;              // [ermax] largest counts
  int* act = top + e.ermax;             // [ermax] the active bins
  int* atop = act + e.ermax;            // [ermax] their largest counts
  RingInfo* info = reinterpret_cast<RingInfo*>(atop + e.ermax);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  // the matrix kernels, unless the flush is short or the exact counts are wanted too; the walk
  // below them returns at once when they have summed the flush
  const bool mma = !count && n >= kMmaMinRing;
  if (mma || (e.mixed && e.ermax > kActiveMinBins)) {
    if ((err = cudaMemsetAsync(top, 0, sizeof(int) * e.ermax, s)) != cudaSuccess) return err;
    ring_active_kernel<<<dim3((e.ermax + 255) / 256, (n + kActivePlacements - 1) / kActivePlacements), 256, 0, s>>>(
        hist, valid, n, e.ermax, top);
    e.count_launch();
  }
  // (every bin walked on a short coordinate: the list costs more than the bins it could leave out)
  const int all = !mma && e.ermax <= kActiveMinBins;
  const int T = e.mixed ? 60 : 63, spread = e.mixed ? 12 : 10;
  if (mma || e.mixed) {
    ring_active_list_kernel<<<1, 1024, 0, s>>>(top, e.ermax, valid, w, n, mma ? kMmaBins : -1, spread, all, act, atop,
                                             info);
    e.count_launch();
  }
  if (mma) {
    const int nbins = (int)mma_bins(e.ermax);
    constexpr size_t smem_q = sizeof(long long) * kMmaWarps * 32 * 32;
    static SmemAttr attr_q;
    if ((err = attr_q.ensure(ecorr_mma_kernel, smem_q)) != cudaSuccess) return err;
    uint4* A = reinterpret_cast<uint4*>(e.d_ring_digits);
    uint4* B = A + (size_t)nbins / 16 * (kMmaK / 16) * 32 * kMaxADigits;
    for (int p0 = 0; p0 < n; p0 += kMmaK) {
      const int np = std::min(kMmaK, n - p0);
      ecorr_digits_kernel<<<dim3(nbins / 16, (np + 127) / 128), 256, 0, s>>>(hist, valid, w, p0, np, e.ermax, T, nbins,
                                                                            act, atop, info, A, B);
      ecorr_mma_kernel<<<dim3(nbins / 32, nbins / 32), 32 * kMmaWarps, smem_q, s>>>(A, B, np, e.ermax, T, nbins, act, atop, info,
                                                                   e.d_ecorr);
      e.count_launch(2);
    }
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
  }
  if (e.mixed) {
    const size_t smem =
        (size_t)n * (kEcRows * sizeof(float2) + sizeof(unsigned) + (count ? kEcRows * sizeof(int) : 0));
    void (*kern)(const int*, const int*, const double*, int, int, const int*, const RingInfo*, double*, long long*) =
        count ? ecorr_ff_kernel<true> : ecorr_ff_kernel<false>;
    static SmemAttr attr_ff[2];  // per instantiation; the size set only ever grows
    if ((err = attr_ff[count ? 1 : 0].ensure(kern, smem)) != cudaSuccess) return err;
    dim3 grid((e.ermax + 255) / 256, (e.ermax + kEcRows - 1) / kEcRows);
    kern<<<grid, 256, smem, s>>>(hist, valid, w, n, e.ermax, act, info, e.d_ecorr, e.d_ecorr_n);
    e.count_launch();
    return cudaGetLastError();
  }
  int* nz_bin = e.d_ring_nz;
  int* nz_cnt = e.d_ring_nz + (size_t)e.ring_cap * e.ermax;
  ring_compact_kernel<<<n, 256, 0, s>>>(hist, valid, e.ermax, mma ? &info->mma : nullptr, nz_bin, nz_cnt, e.d_ring_nnz);
  e.count_launch();
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  const size_t per_row = (size_t)e.ermax * (sizeof(double) + (e.d_ecorr_n ? sizeof(long long) : 0));
  int R = (int)std::max<size_t>(1, std::min<size_t>(8, (96 * 1024) / per_row));
  const size_t smem = per_row * R;
  if ((err = ecorr_rows_attr().ensure(ecorr_rows_kernel, smem)) != cudaSuccess) return err;
  const int nblk = (e.ermax + R - 1) / R;
  ecorr_rows_kernel<<<nblk, 256, smem, s>>>(hist, nz_bin, nz_cnt, e.d_ring_nnz, w, n, e.ermax, R,
                                            mma ? &info->mma : nullptr, e.d_ecorr, e.d_ecorr_n);
  e.count_launch();
  return cudaGetLastError();
}


// ---- ecorr from caller-owned histograms, with no allocation -----------------------
//
// Some hosts cannot let a library allocate device memory in the middle of their step:
// an MD engine that has sized its memory pool to the whole card, or one that keeps
// other streams busy on the same device, where cudaFree would synchronise the device
// and stall them.  ermod_ecorr_add_noalloc serves such hosts.  Its only scratch (the
// occupied-bin lists that ring_compact_kernel builds for the ring) lives in one fixed
// file-scope device array, so a call allocates nothing.

namespace {

constexpr size_t kNoAllocEntries = (size_t)kNoAllocMaxEntries;  // 8 MiB of (bin, count) lists
constexpr int kNoAllocMaxDevices = 64;

// [kNoAllocEntries] bins, [kNoAllocEntries] counts, [kNoAllocMaxPlace] list lengths.
// Shared by every call on a device: calls that overlap on the GPU race on it.
static __device__ __align__(256) int g_noalloc_scratch[2 * kNoAllocEntries + kNoAllocMaxPlace];

std::mutex g_noalloc_mu;
int* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// ring_compact_kernel for caller histograms: every placement is valid, the lists go to
// the fixed scratch.  Each list length is written for every placement and each list
// entry below it, so nothing in the scratch has to start at zero.
__global__ void __launch_bounds__(256) compact_noalloc_kernel(const int* __restrict__ hist, int ermax,
                                                              int* __restrict__ nz_bin, int* __restrict__ nz_cnt,
                                                              int* __restrict__ nnz) {
  const int p = blockIdx.x;
  const int* h = hist + (size_t)p * ermax;
  __shared__ int scan[256];
  const int per = (ermax + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = min(ermax, lo + per);
  int cnt = 0;
  for (int i = lo; i < hi; ++i) cnt += (h[i] != 0);
  scan[threadIdx.x] = cnt;
  __syncthreads();
  for (int off = 1; off < blockDim.x; off <<= 1) {
    const int v = (threadIdx.x >= off) ? scan[threadIdx.x - off] : 0;
    __syncthreads();
    scan[threadIdx.x] += v;
    __syncthreads();
  }
  int pos = scan[threadIdx.x] - cnt;
  for (int i = lo; i < hi; ++i)
    if (h[i]) {
      nz_bin[(size_t)p * ermax + pos] = i;
      nz_cnt[(size_t)p * ermax + pos] = h[i];
      ++pos;
    }
  if (threadIdx.x == blockDim.x - 1) nnz[p] = scan[threadIdx.x];
}

// the scratch address on the current device, looked up once per device
cudaError_t noalloc_scratch(int** out) {
  int dev = -1;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    int* p = nullptr;
    err = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
    if (err != cudaSuccess) return err;
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace

cudaError_t launch_ecorr_noalloc(const int* hist, const double* weight, int nplace, int ermax, double* ecorr,
                                 long long* ecorr_count, cudaStream_t s) {
  int* scratch = nullptr;
  cudaError_t err = noalloc_scratch(&scratch);
  if (err != cudaSuccess) return err;
  int* nz_bin = scratch;
  int* nz_cnt = scratch + kNoAllocEntries;
  int* nnz = scratch + 2 * kNoAllocEntries;
  compact_noalloc_kernel<<<nplace, 256, 0, s>>>(hist, ermax, nz_bin, nz_cnt, nnz);
  err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const size_t per_row = (size_t)ermax * (sizeof(double) + (ecorr_count ? sizeof(long long) : 0));
  const int R = (int)std::max<size_t>(1, std::min<size_t>(8, (96 * 1024) / per_row));
  const size_t smem = per_row * R;
  err = ecorr_rows_attr().ensure(ecorr_rows_kernel, smem);
  if (err != cudaSuccess) return err;
  ecorr_rows_kernel<<<(ermax + R - 1) / R, 256, smem, s>>>(hist, nz_bin, nz_cnt, nnz, weight, nplace, ermax, R,
                                                           nullptr, ecorr, ecorr_count);
  return cudaGetLastError();
}

}  // namespace ermod
