// kernels_fft64.cu -- the plain FP64 path's inverse transforms (unnormalised, sign +1): the
// spectra [b][k3][k2][k1] of a batch along k3, then k2, in place, then complex to real along k1
// into the potential grids [b][z][y][x] (recpcal_prepare_solute's C2R, recpcal.F90:397-402).
//
// Bound by the FP64 pipe, which takes a warp's instruction every 16 clocks of an SM: the passes
// use radices up to 16 (96 points: 12 x 8, 2,100 instructions where 5 N log2 N
// counts 3,160), and two real rows share one complex transform.  Integer work and
// shared memory hide behind it, so one kernel serves every length with factors 2, 3 and 5 (others
// take cuFFT).  16 placements at 96^3: 293, 314 and 346 us (the first two at 85% of the FP64 pipe's
// rate), cuFFT's three kernels 333, 333 and 834; 64 at 48^3 440 us and 594.
#include "dft.cuh"
#include "engine.cuh"

namespace ermod {

namespace {

constexpr int kThreads64 = 128;

// one Stockham pass of radix R over n transforms of length N, A -> B: element i of transform c at
// c cs + i es.  COLS: consecutive threads take consecutive transforms, else consecutive elements.
// put(B, c, i, value) stores.
template <int R, bool COLS, class Get, class Put>
__device__ __forceinline__ void pass64(int N, int Ns, int n, const double2* tw, Get get, Put put) {
  const int NR = N / R, step = N / (Ns * R);
  for (int t = threadIdx.x; t < n * NR; t += kThreads64) {
    const int c = COLS ? t % n : t / NR, j = COLS ? t / n : t % NR;
    const int jq = j / Ns, k = j - jq * Ns;
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = get(c, j + r * NR);
    if (k > 0) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[r * k * step]);
    }
    Dft<R>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) put(c, jq * Ns * R + k + r * Ns, v[r]);
  }
}

template <bool COLS, class Get, class Put>
__device__ __forceinline__ void run_pass64(int R, int N, int Ns, int n, const double2* tw, Get get, Put put) {
#define ERMOD_PASS64(RR) \
  case RR: pass64<RR, COLS>(N, Ns, n, tw, get, put); break;
  switch (R) {
    ERMOD_PASS64(2)
    ERMOD_PASS64(3)
    ERMOD_PASS64(4)
    ERMOD_PASS64(5)
    ERMOD_PASS64(6)
    ERMOD_PASS64(8)
    ERMOD_PASS64(9)
    ERMOD_PASS64(10)
    ERMOD_PASS64(12)
    ERMOD_PASS64(15)
    ERMOD_PASS64(16)
    default: break;
  }
#undef ERMOD_PASS64
}

__device__ __forceinline__ void stage_twiddles(const double2* __restrict__ table, int N, double2* tw) {
  for (int i = threadIdx.x; i < N; i += kThreads64) {
    const double2 t = table[i];  // exp(-2 pi i m / N), conjugated for the inverse
    tw[i] = make_double2(t.x, -t.y);
  }
}

// ncol columns of N elements es apart, the columns' first elements consecutive; blockIdx.y counts
// blocks of such columns, dist elements apart.  C columns per CTA, in place.
__global__ void __launch_bounds__(kThreads64, 4) fft64_columns_kernel(double2* data, const double2* __restrict__ table,
                                                                   FftPlan p, int ncol, size_t es, size_t dist,
                                                                   int C) {
  extern __shared__ double2 sm64[];
  const int N = p.n;
  double2* tw = sm64;         // [N]
  double2* A = sm64 + N;      // [N][C]
  double2* B = A + (size_t)N * C;  // the same, with more than two passes
  const int c0 = blockIdx.x * C, n = min(C, ncol - c0);
  double2* g = data + blockIdx.y * dist + c0;
  stage_twiddles(table, N, tw);
  for (int i = 0; i < p.npass; ++i) {
    __syncthreads();
    const bool first = i == 0, last = i == p.npass - 1;
    const double2* src = first ? g : ((i & 1) ? A : B);
    double2* dst = last ? g : ((i & 1) ? B : A);
    const size_t ies = first ? es : (size_t)C, oes = last ? es : (size_t)C;
    // (a single pass reads and writes each column with one thread)
    run_pass64<true>(
        p.r[i], N, p.ns[i], n, tw, [&](int c, int e) { return src[c + e * ies]; },
        [&](int c, int e, double2 v) { dst[c + e * oes] = v; });
  }
}

// nrow half spectra of H = K / 2 + 1 points to nrow real rows of K, P pairs of rows per CTA: the
// rows of a pair are one complex transform Z = X_0 + i X_1, Hermitian-completed
__global__ void __launch_bounds__(kThreads64, 4) fft64_rows_kernel(const double2* __restrict__ spec, double* __restrict__ out,
                                                                const double2* __restrict__ table, FftPlan p, int H,
                                                                long long nrow, int P) {
  extern __shared__ double2 sm64[];
  const int N = p.n, RS = N | 1;
  double2* tw = sm64;                   // [N]
  double2* rows = sm64 + N;             // [2 P][H]; later passes' second buffer
  double2* A = rows + (size_t)2 * P * max(H, (RS + 1) / 2);  // [P][RS]
  const long long r0 = (long long)blockIdx.x * 2 * P;
  const int nr = (int)min((long long)2 * P, nrow - r0), n = (nr + 1) / 2;
  stage_twiddles(table, N, tw);
  const double2* g = spec + r0 * H;
  for (int i = threadIdx.x; i < nr * H; i += kThreads64) rows[i] = g[i];
  double* o = out + r0 * N;
  for (int i = 0; i < p.npass; ++i) {
    __syncthreads();
    const bool first = i == 0, last = i == p.npass - 1;
    double2* W = (i & 1) ? rows : A;        // this pass's output
    const double2* src = (i & 1) ? A : rows;
    auto load = [&](int c, int e) {
      if (!first) return src[c * RS + e];
      const bool lo = e < H;
      const int k = lo ? e : N - e;
      double2 x = rows[2 * c * H + k];
      double2 y = 2 * c + 1 < nr ? rows[(2 * c + 1) * H + k] : make_double2(0.0, 0.0);
      if (!lo) {
        x.y = -x.y;
        y.y = -y.y;
      }
      if (e == 0 || 2 * e == N) x.y = y.y = 0.0;  // self-conjugate points
      return make_double2(x.x - y.y, x.y + y.x);
    };
    auto store = [&](int c, int e, double2 v) {
      if (!last) {
        W[c * RS + e] = v;
        return;
      }
      o[(size_t)2 * c * N + e] = v.x;
      if (2 * c + 1 < nr) o[(size_t)(2 * c + 1) * N + e] = v.y;
    };
    run_pass64<false>(p.r[i], N, p.ns[i], n, tw, load, store);
  }
}

// The plan of a length: the two radices nearest each other where there are such (the general plan
// takes the largest first).  They cost the same instructions, and a pass lasts as long as one
// warp's radix where a single placement leaves the GPU idle: 64 clocks an instruction.
bool plan64(int n, FftPlan& p) {
  if (!fft_plan(n, p)) return false;
  for (int a : {12, 10, 9, 8, 6, 5, 4})
    for (int b : {12, 10, 9, 8, 6, 5, 4})
      if (a >= b && a * b == n) {
        p.npass = 2;
        p.r[0] = a;
        p.r[1] = b;
        p.ns[0] = 1;
        p.ns[1] = a;
      }
  return true;
}

// the most items (at most `most`) whose shared memory stays within a quarter of an SM's, halved
// while the launch has too few CTAs for the GPU (never below `least`)
int items_per_cta(const Engine& e, long long items, size_t bytes_each, int most, int least) {
  int c = (int)std::max<size_t>(1, std::min<size_t>(most, (size_t)54 * 1024 / bytes_each));
  while (c > least && items / c < 2LL * e.num_sm) c = (c + 1) / 2;
  return c;
}

}  // namespace

bool fft64_fits(int K1, int K2, int K3) {
  FftPlan p;
  return fft_plan(K1, p) && fft_plan(K2, p) && fft_plan(K3, p);
}

cudaError_t launch_fft64(Engine& e, const BatchArgs& a) {
  const int K1 = e.geom.K[0], K2 = e.geom.K[1], K3 = e.geom.K[2], H = e.H();
  FftPlan p1, p2, p3;
  if (!plan64(K1, p1) || !plan64(K2, p2) || !plan64(K3, p3)) return cudaErrorInvalidValue;
  static SmemAttr attr_c, attr_r;
  cudaError_t err;
  auto columns = [&](const FftPlan& p, const double2* table, int ncol, size_t es, size_t dist, int blocks) {
    const int nbuf = p.npass > 2 ? 2 : 1;
    int C = items_per_cta(e, (long long)ncol * blocks, sizeof(double2) * p.n * nbuf, 32, 8);
    C = (ncol + (ncol + C - 1) / C - 1) / ((ncol + C - 1) / C);  // even shares
    const size_t smem = sizeof(double2) * ((size_t)p.n + (size_t)p.n * C * nbuf);
    if ((err = attr_c.ensure(fft64_columns_kernel, smem)) != cudaSuccess) return err;
    fft64_columns_kernel<<<dim3((ncol + C - 1) / C, blocks), kThreads64, smem, a.stream>>>(a.spec64, table, p, ncol, es,
                                                                                          dist, C);
    e.count_launch();
    return cudaGetLastError();
  };
  const size_t plane = (size_t)K2 * H;
  if ((err = columns(p3, e.d_twiddle64 + K1 + K2, K2 * H, plane, K3 * plane, a.nb)) != cudaSuccess) return err;
  if ((err = columns(p2, e.d_twiddle64 + K1, H, H, plane, a.nb * K3)) != cudaSuccess) return err;
  const long long nrow = (long long)a.nb * K3 * K2;
  const int RS = K1 | 1;
  const size_t each = sizeof(double2) * (2 * (size_t)std::max(H, (RS + 1) / 2) + RS);
  const int P = items_per_cta(e, (nrow + 1) / 2, each, 16, 4);
  const size_t smem = sizeof(double2) * K1 + each * P;
  if ((err = attr_r.ensure(fft64_rows_kernel, smem)) != cudaSuccess) return err;
  fft64_rows_kernel<<<(unsigned)((nrow + 2 * P - 1) / (2 * P)), kThreads64, smem, a.stream>>>(a.spec64, a.phi64,
                                                                                            e.d_twiddle64, p1, H, nrow,
                                                                                            P);
  e.count_launch();
  return cudaGetLastError();
}

}  // namespace ermod
