// kernels_place.cu -- per-placement solute preparation and the plain FP64 PME path.
//
//   place_prep    solute sites of every placement in a batch: wrapped FP64 and
//                 fixed-point coordinates, calc_spline_molecule (recpcal.F90:408-442,
//                 FP64 weights on both paths),
//                 realcal_self (realcal.F90:284-328, FP64) and the 1-D structure-factor
//                 vectors
//                     b_{s,a}(k) = sum_c theta_{s,a,c} exp(-2 pi i k (g_{s,a} - c) / K_a);
//                 (the mixed path's spectrum and transforms are in kernels_fft.cu);
//   spectrum64    the plain FP64 path's spectrum engfac S(k) from those vectors, with the
//                 self energy; its inverse transforms are in kernels_fft64.cu.
#include "engine.cuh"

namespace ermod {

namespace {

__host__ __device__ __forceinline__ double ipow_d(double x, int e) {
  double r = 1.0;
  bool first = true;
  while (e > 0) {
    if (e & 1) {
      r = first ? x : r * x;
      first = false;
    }
    e >>= 1;
    if (e) x = x * x;
  }
  return r;
}

struct Coef {
  double c[kMaxSplineOrder + 1];
  int order;
  double screen;
};

__device__ __forceinline__ double spline_value(const Coef& s, double rst) {  // spline.F90:47-59
  double f = 0.0;
  if ((rst > 0.0) && (rst < (double)s.order)) {
    const int k = (int)rst;
    for (int i = 0; i <= k; ++i) f = f + s.c[i] * ipow_d(rst - (double)i, s.order - 1);
  }
  return f;
}

struct PrepArgs {
  BatchArgs a;
  const double* solxyz;   // [nb][S][3] raw solute coordinates of this batch, or null (use frame)
  const double* sitepos;  // frame raw coordinates
  const int* mbi0;        // [nummol+1] 0-based
  const double* charge;
  const int* ljtype;
  const double* mol_qmol_all;  // [nummol]
  const double2* twiddle64;    // [K1+K2+K3] exp(-2 pi i m / K)
  FrameGeom g;
  Coef sc;
  int mixed;
  int self_mode;  // 0: none, 1: all placements, 2: only placement 0 of the batch
  int nummol;
  int bare;  // cltype 0
  unsigned mK[3];  // ceil(2^32 / d): n / d = umulhi(n, m) for n d < 2^32
  unsigned mKh[3];  // the same for K / 2 + 1
  const double* usreal_known;  // rigid solutes: nonzero once the context holds realcal_self's value
  DevStatus* status;
};

__device__ __forceinline__ void wrap_coord(const double* v, double x0raw, const FrameGeom& g, double out[3]) {
  for (int i = 0; i < 3; ++i) out[i] = v[i] - g.L[i] * floor(g.invL[i] * v[i]);
  out[1] = out[1] - g.L[1] * floor(g.invL[1] * out[1]);
  const double x0 = x0raw - g.L[0] * floor(g.invL[0] * x0raw);
  const double x0b = x0 - g.L[0] * floor(g.invL[0] * x0);
  out[0] = out[0] - g.L[0] * floor(g.invL[0] * x0b);
}

// 1-D structure factors of one axis of one placement's solute: FP64 weights
// (calc_spline_molecule on the raw coordinates) and twiddles; the mixed path rounds them to
// FP32 once at the end, so that their errors are independent roundings.  Half of the range is
// computed, the other half is its conjugate
__device__ void structure_factors(const PrepArgs& A, int b, int atom0, int ns, int ax) {
  __shared__ double th[kMaxSoluteSites * kMaxSplineOrder];
  __shared__ int sgrd[kMaxSoluteSites];
  const BatchArgs& a = A.a;
  const FrameGeom& g = A.g;
  const int P = A.sc.order, K = g.K[ax];
  for (int t = threadIdx.x; t < ns * P; t += blockDim.x) {
    const int s = t / P, spi = t - s * P;
    const double* raw = A.solxyz ? A.solxyz + ((size_t)b * ns + s) * 3 : A.sitepos + 3 * (size_t)(atom0 + s);
    double factor = g.invcl[ax + 0] * raw[0] + g.invcl[ax + 3] * raw[1] + g.invcl[ax + 6] * raw[2];
    factor = factor - floor(factor);
    const double f2 = factor * (double)K;
    const int rci = (int)f2;
    th[t] = spline_value(A.sc, f2 - (double)(rci - spi));
    if (spi == 0) sgrd[s] = rci;
  }
  __syncthreads();
  const int Kmax = max(g.K[0], max(g.K[1], g.K[2]));
  const double2* tw = A.twiddle64 + (ax == 0 ? 0 : (ax == 1 ? g.K[0] : g.K[0] + g.K[1]));
  const unsigned mk = A.mK[ax], mh = A.mKh[ax];
  const int Kh = K / 2 + 1;
  for (int t = threadIdx.x; t < ns * Kh; t += blockDim.x) {
    const int s = (int)__umulhi((unsigned)t, mh), k = t - s * Kh;
    const int grd = sgrd[s];
    double re = 0.0, im = 0.0;
    for (int c = 0; c < P; ++c) {
      int gc = grd - c;  // in (-P, K)
      if (gc < 0) gc += K;
      const unsigned x = (unsigned)(k * gc);  // < K^2 <= 10^6
      const int mm = (int)(x - __umulhi(x, mk) * (unsigned)K);
      const double2 w = tw[mm];
      re = fma(th[s * P + c], w.x, re);
      im = fma(th[s * P + c], w.y, im);
    }
    const size_t row = (((size_t)b * kMaxSoluteSites + s) * 3 + ax) * Kmax;
    const bool two = k > 0 && 2 * k < K;  // K - k is another point
    if (A.mixed) {
      const float2 v = make_float2((float)re, (float)im);
      a.u_bvec[row + k] = v;
      if (two) a.u_bvec[row + K - k] = make_float2(v.x, -v.y);
    } else {
      a.u_bvec64[row + k] = make_double2(re, im);
      if (two) a.u_bvec64[row + K - k] = make_double2(re, -im);
    }
  }
}

// Four blocks per placement of the batch: the structure factors of each axis, and the rest
// (coordinates, charges, bounding radius, realcal_self), so that a single placement's FP64
// chains run side by side and on four SMs' FP64 pipes (one block, one thread per site for the
// weights: 24 us for 6 sites at 32^3, on a solution-mode frame's critical path).
__global__ void __launch_bounds__(256) place_prep_kernel(PrepArgs A) {
  const int b = blockIdx.x;
  const int part = A.bare ? 3 : (int)blockIdx.y;
  const BatchArgs& a = A.a;
  const FrameGeom& g = A.g;
  const int mol = a.tagslt[b] - 1;
  // device-side inputs are checked here, not trusted
  const int atom0 = (mol < 0 || mol >= A.nummol) ? 0 : A.mbi0[mol];
  const int ns = (mol < 0 || mol >= A.nummol) ? 0 : A.mbi0[mol + 1] - atom0;
  if (ns < 1 || ns > kMaxSoluteSites) {
    if (part == 3 && threadIdx.x == 0) {
      atomicOr(&A.status->range_fault, 1);
      a.u_nsite[b] = 0;
    }
    return;
  }
  if (part < 3) {
    structure_factors(A, b, atom0, ns, part);
    return;
  }
  __shared__ double sx[kMaxSoluteSites][3];
  __shared__ double red[256];
  for (int s = threadIdx.x; s < ns; s += blockDim.x) {
    const double* raw = A.solxyz ? A.solxyz + ((size_t)b * ns + s) * 3 : A.sitepos + 3 * (size_t)(atom0 + s);
    double w[3];
    const bool is_atom1 = (A.solxyz == nullptr) && (atom0 + s == 0);
    if (!g.periodic) {  // non-periodic: coordinates as they are, within the fixed-point reach
      for (int i = 0; i < 3; ++i) {
        w[i] = raw[i];
        if (!(fabs(raw[i]) < g.reach)) atomicOr(&A.status->range_fault, 4);
      }
    } else if (is_atom1) {  // atom 1 itself takes the first-pass x shift of its own x
      for (int i = 0; i < 3; ++i) w[i] = raw[i] - g.L[i] * floor(g.invL[i] * raw[i]);
      w[1] = w[1] - g.L[1] * floor(g.invL[1] * w[1]);
      w[0] = w[0] - g.L[0] * floor(g.invL[0] * w[0]);
    } else {
      wrap_coord(raw, A.sitepos[0], g, w);
    }
    const size_t us = (size_t)b * kMaxSoluteSites + s;
    for (int i = 0; i < 3; ++i) {
      a.u_x[us * 3 + i] = w[i];
      sx[s][i] = w[i];
    }
    unsigned int X[3];
    for (int i = 0; i < 3; ++i) X[i] = (unsigned int)(unsigned long long)llrint(w[i] * g.invL[i] * 4294967296.0);
    a.u_pos[us] = make_int4((int)X[0], (int)X[1], (int)X[2], A.ljtype[atom0 + s]);
    a.u_q[us] = A.charge[atom0 + s];
    a.u_qf[us] = (float)A.charge[atom0 + s];
  }
  if (threadIdx.x == 0) {
    a.u_nsite[b] = ns;
    a.u_qmol[b] = A.mol_qmol_all[mol];
  }
  // bounding radius about site 1 (minimum image; FP32, padded to stay conservative)
  __shared__ int rmax_bits;
  if (threadIdx.x == 0) rmax_bits = 0;
  __syncthreads();
  for (int s = 1 + threadIdx.x; s < ns; s += blockDim.x) {
    float r2 = 0.f;
    for (int i = 0; i < 3; ++i) {
      const float h = 0.5f * (float)g.L[i];
      const float d = h - fabsf(h - fabsf((float)(sx[s][i] - sx[0][i])));
      r2 += d * d;
    }
    atomicMax(&rmax_bits, __float_as_int(sqrtf(r2)));  // nonnegative floats order as ints
  }
  __syncthreads();
  if (threadIdx.x == 0) a.u_radius[b] = __int_as_float(rmax_bits) * 1.0001f + 1e-4f;
  // realcal_self (realcal.F90:284-328), fixed-order block reduction.  A rigid solute's is taken
  // from the context's first placement (the accumulation keeps it), so that later batches' blocks
  // are spared the longest chain of the kernel; it is read here only as a flag
  const bool need_self =
      (A.self_mode == 1) || (A.self_mode == 2 && b == 0 && *(const volatile double*)A.usreal_known == 0.0);
  if (need_self && A.bare) {  // realcal_self returns 0 for bare Coulomb (realcal.F90:294)
    if (threadIdx.x == 0) a.u_usreal[b] = 0.0;
    return;
  }
  if (need_self) {
    double acc = 0.0;
    for (int is = threadIdx.x; is < ns; is += blockDim.x) {  // the diagonal gives the atoms' residuals
      const double qi = A.charge[atom0 + is];
      acc += -qi * qi * A.sc.screen / sqrt(kPi);
    }
    // every pair once, as (is, is + d mod ns), d up to ns / 2 (half of the last row when ns is
    // even), so that no lane idles through an erf
    const int half = ns / 2;
    for (int t = threadIdx.x; t < ns * half; t += blockDim.x) {
      const int d = t / ns + 1, is = t - (d - 1) * ns;
      if (2 * d == ns && is >= half) continue;
      const int js = is + d < ns ? is + d : is + d - ns;
      double d2 = 0.0;
      for (int i = 0; i < 3; ++i) {
        const double h = 0.5 * g.L[i];
        const double x = h - fabs(h - fabs(sx[is][i] - sx[js][i]));
        d2 += x * x;
      }
      const double rst = sqrt(d2);
      acc += -A.charge[atom0 + is] * A.charge[atom0 + js] * erf(A.sc.screen * rst) / rst;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
      if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
      __syncthreads();
    }
    if (threadIdx.x == 0) a.u_usreal[b] = red[0];
  }
}

// ---- FP64 path ----------------------------------------------------------------------
struct Spec64Args {
  const double2* bvec;  // [nb][S][3][Kmax]
  const double* u_q;    // [nb][S]
  const int* u_nsite;
  const double* engfac;  // [K3][K2][H]
  double2* spec;         // [nb][K3][K2][H]
  double* self_part;     // [nb][spectrum64_partials]
  int K1, K2, K3, H, Kmax;
  int groups;  // groups of the threads' k3 pairs per CTA
};

// The FP64 spectrum engfac(k) S(k), S = sum_s q_s b1_s(k1) b2_s(k2) b3_s(k3): exactly the R2C
// transform of the spread charges (recpcal.F90:357-384) without the K^3 grid, the spread and
// the forward transform, and with the self energy 0.5 sum_k engfac |S|^2 (recpcal.F90:385-394)
// in the same pass.
//
// Bound by the FP64 pipe (2 FMA per clock and SM), so k3 and K3 - k3 are computed together:
// b3(K3 - k3) is the conjugate of b3(k3) = c + i s, so with the site's p = q b1 b2,
// A = sum p c and B = sum p s (real times complex, 2 FMA each) give S(k3) = A + i B and
// S(K3 - k3) = A - i B: half of the 4 FMA per point and site that each point takes by itself.
// Pair 0 holds the real b3(0) and b3(K3 / 2) (the latter 0 for odd K3): S(0) = A, S(K3 / 2) = B.
// CTA per (k2, groups x 4 pairs, placement), a thread per k1 and 4 pairs (one in solution mode,
// whose single placement waits for each warp's chain); p and the pairs'
// factors of 16 sites at a time in shared memory.  200 insertions on 48^3 (6 sites) 4.83 -> 4.54
// ms, 32 on 96^3 (12 sites) 6.78 -> 6.16 ms against a thread per point.
constexpr int kSpecPairsMost = 4;  // k3 pairs per thread, in reference mode
constexpr int kSpecSites = 16;  // sites staged at a time
constexpr int kSpec64Threads = 512;
template <int kSpecPairs>
__global__ void __launch_bounds__(kSpec64Threads) spectrum64_kernel(Spec64Args A) {
  extern __shared__ double2 sc[];
  double2* sp = sc;                      // [kSpecSites][H]: q_s b1_s(k1) b2_s(k2)
  double2* sd = sc + kSpecSites * A.H;   // [kSpecSites][groups * kSpecPairs]: the pairs' (c, s)
  const int k2 = blockIdx.x, b = blockIdx.z;
  const int npair = (A.K3 + 1) / 2, width = A.groups * kSpecPairs, pair0 = blockIdx.y * width;
  const int ns = A.u_nsite[b];
  const bool even = (A.K1 % 2) == 0, even3 = (A.K3 % 2) == 0;
  const double2* bv = A.bvec + (size_t)b * kMaxSoluteSites * 3 * A.Kmax;
  const int ntask = A.groups * A.H;
  double self = 0.0;
  for (int t0 = 0; t0 < ntask; t0 += blockDim.x) {  // one round unless H is above the CTA's size
    const int t = t0 + (int)threadIdx.x;
    const int gr = t / A.H, k1 = t - gr * A.H;
    const int pa = pair0 + gr * kSpecPairs;
    const bool on = t < ntask && pa < npair;
    double2 a[kSpecPairs], c[kSpecPairs];
#pragma unroll
    for (int i = 0; i < kSpecPairs; ++i) a[i] = c[i] = make_double2(0.0, 0.0);
    for (int s0 = 0; s0 < ns; s0 += kSpecSites) {
      const int n = min(kSpecSites, ns - s0);
      __syncthreads();
      for (int i = threadIdx.x; i < n * A.H; i += blockDim.x) {
        const int s = i / A.H, k = i - s * A.H;
        const double2* row = bv + (size_t)(s0 + s) * 3 * A.Kmax;
        const double q = A.u_q[(size_t)b * kMaxSoluteSites + s0 + s];
        const double2 b2 = row[A.Kmax + k2], b1 = row[k];
        const double x = q * b2.x, y = q * b2.y;
        sp[s * A.H + k] = make_double2(x * b1.x - y * b1.y, x * b1.y + y * b1.x);
      }
      for (int i = threadIdx.x; i < n * width; i += blockDim.x) {
        const int s = i / width, p = pair0 + i - s * width;
        const double2* row = bv + (size_t)(s0 + s) * 3 * A.Kmax + 2 * A.Kmax;
        double2 v = make_double2(0.0, 0.0);
        if (p == 0)
          v = make_double2(row[0].x, even3 ? row[A.K3 / 2].x : 0.0);
        else if (p < npair)
          v = row[p];
        sd[s * width + p - pair0] = v;
      }
      __syncthreads();
      if (on) {
        const double2* d = sd + gr * kSpecPairs;
        for (int s = 0; s < n; ++s) {
          const double2 p = sp[s * A.H + k1];
#pragma unroll
          for (int i = 0; i < kSpecPairs; ++i) {
            const double2 v = d[s * width + i];
            a[i].x = fma(p.x, v.x, a[i].x);
            a[i].y = fma(p.y, v.x, a[i].y);
            c[i].x = fma(p.x, v.y, c[i].x);
            c[i].y = fma(p.y, v.y, c[i].y);
          }
        }
      }
    }
    if (on) {
      const double w = (k1 == 0 || (even && k1 == A.H - 1)) ? 0.5 : 1.0;
      double own = 0.0;  // the thread's points share the weight
      auto put = [&](double2* to, double f, double2 x) {
        const double2 y = make_double2(f * x.x, f * x.y);
        own = fma(y.y, x.y, fma(y.x, x.x, own));
        *to = y;
      };
      const size_t plane = (size_t)A.K2 * A.H, at0 = (size_t)k2 * A.H + k1;
      double2* out = A.spec + (size_t)b * A.K3 * plane + at0;
#pragma unroll
      for (int i = 0; i < kSpecPairs; ++i) {
        const int p = pa + i;
        if (p >= npair) break;
        const int lo = p, hi = p == 0 ? A.K3 / 2 : A.K3 - p;  // odd K3: pair 0 has no upper point
        const double2 x = p == 0 ? a[i] : make_double2(a[i].x - c[i].y, a[i].y + c[i].x);
        const double2 y = p == 0 ? c[i] : make_double2(a[i].x + c[i].y, a[i].y - c[i].x);
        put(out + (size_t)lo * plane, A.engfac[(size_t)lo * plane + at0], x);
        if (p > 0 || even3) put(out + (size_t)hi * plane, A.engfac[(size_t)hi * plane + at0], y);
      }
      self = fma(w, own, self);
    }
  }
  __shared__ double red[kSpec64Threads / 32];
  for (int o = 16; o > 0; o >>= 1) self += __shfl_xor_sync(0xffffffffu, self, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = self;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) self += red[w];
    A.self_part[((size_t)b * gridDim.y + blockIdx.y) * A.K2 + k2] = self;
  }
}

// Pairs per thread and groups of them per CTA, fixed for a context, so that a placement's self
// energy does not depend on its batch.  Solution mode: 4 groups of one pair (32^3, 6 sites: 14.8 us
// with one group of 4 pairs); otherwise the groups of the least FP64 work in whole warps, 16 FMA per
// thread and site and 4 per staged p (at 96^3 2 x 320 threads of 6 groups; the staging is then
// 5% of the work).
int spec64_pairs(const Engine& e) { return e.P.slttype == 1 ? 1 : kSpecPairsMost; }
int spec64_groups(const Engine& e) {
  const int H = e.H(), all = ((e.geom.K[2] + 1) / 2 + kSpecPairsMost - 1) / kSpecPairsMost;
  if (e.P.slttype == 1) return 4;
  int best = 1;
  long long cost = 0;
  for (int g = 1; g <= all && (g == 1 || g * H <= kSpec64Threads); ++g) {
    const long long parts = (all + g - 1) / g;
    const long long c = parts * (16LL * ((g * H + 31) / 32) + 4LL * ((H + 31) / 32));
    if (g == 1 || c < cost) {
      cost = c;
      best = g;
    }
  }
  return best;
}
int spec64_parts(const Engine& e) {
  const int width = spec64_groups(e) * spec64_pairs(e);
  return ((e.geom.K[2] + 1) / 2 + width - 1) / width;
}

Coef make_coef(int order, double screen) {
  Coef s{};
  s.order = order;
  for (int i = 0; i <= order; ++i) {
    double factor = 1.0;
    for (int k = 1; k <= i; ++k) factor = factor * (double)k;
    for (int k = 1; k <= order - i; ++k) factor = factor * (double)k;
    factor = (double)order / factor;
    if (i % 2 == 1) factor = -factor;
    s.c[i] = factor;
  }
  s.screen = screen;
  return s;
}

}  // namespace

// self-energy partials per placement of the mixed path: one per k2 (the pme_a CTA of
// (k2, placement) writes self_part[b][k2])
int spectrum_partials(const Engine& e) { return e.geom.K[1]; }

cudaError_t launch_place_prep(Engine& e, const BatchArgs& a, const double* sol_xyz, int self_mode, cudaStream_t s) {
  PrepArgs A{};
  A.a = a;
  A.solxyz = sol_xyz;
  A.sitepos = e.d_sitepos;
  A.mbi0 = e.d_mbi0;
  A.charge = e.d_charge;
  A.ljtype = e.d_ljtype;
  A.mol_qmol_all = e.d_qmol_all;
  A.twiddle64 = e.d_twiddle64;
  A.g = e.geom;
  A.sc = make_coef(e.P_order, e.P.screen);
  A.mixed = e.mixed ? 1 : 0;
  A.self_mode = self_mode;
  A.bare = (e.P.cltype == 0) ? 1 : 0;
  A.nummol = e.nummol;
  A.status = e.d_status;
  auto magic = [](unsigned d) { return (unsigned)((0x100000000ull + d - 1) / d); };
  for (int i = 0; i < 3; ++i) {
    A.mK[i] = magic((unsigned)e.geom.K[i]);
    A.mKh[i] = magic((unsigned)(e.geom.K[i] / 2 + 1));
  }
  A.usreal_known = e.d_scal + 6;
  place_prep_kernel<<<dim3(a.nb, A.bare ? 1 : 4), 256, 0, s>>>(A);
  e.count_launch();
  return cudaGetLastError();
}

int spectrum64_partials(const Engine& e) { return e.geom.K[1] * spec64_parts(e); }

cudaError_t launch_spectrum64(Engine& e, const BatchArgs& a) {
  Spec64Args A{};
  A.bvec = a.u_bvec64;
  A.u_q = a.u_q;
  A.u_nsite = a.u_nsite;
  A.engfac = e.d_engfac;
  A.spec = a.spec64;
  A.self_part = a.self_part;
  A.K1 = e.geom.K[0];
  A.K2 = e.geom.K[1];
  A.K3 = e.geom.K[2];
  A.H = e.H();
  A.Kmax = e.Kmax();
  A.groups = spec64_groups(e);
  const int pairs = spec64_pairs(e);
  void (*kern)(Spec64Args) = pairs == 1 ? spectrum64_kernel<1> : spectrum64_kernel<kSpecPairsMost>;
  const size_t smem = sizeof(double2) * kSpecSites * (A.H + A.groups * pairs);
  static SmemAttr attr1, attr4;
  cudaError_t err = (pairs == 1 ? attr1 : attr4).ensure(kern, smem);
  if (err != cudaSuccess) return err;
  const dim3 grid(A.K2, spec64_parts(e), a.nb);
  const int nthr = std::min(kSpec64Threads, (A.groups * A.H + 31) / 32 * 32);
  kern<<<grid, nthr, smem, a.stream>>>(A);
  e.count_launch();
  return cudaGetLastError();
}

}  // namespace ermod
