// Longstaff-Schwartz fit of the Bermudans of a plan on the GPU: the policy (exercise decision) and the
// continuation regressions that the fused kernel's AMC terms evaluate.
//
// It follows the reference's compile-time fit (fitAmc, src/gpu/fused_exposure.cpp:103-156, with
// PolynomialRegression, src/core/regression.cpp:29-98): backwards over the exercise dates, a masked
// (in-the-money) regression of the deflated realised value on the standardised short-rate state, the
// exercise rule "exercise value > 0 and > regression", and on every date with an exercise ahead an
// unmasked regression of the value of the policy from the next exercise on.  The degree falls back as the
// reference's does (degenerate regressor, too few samples) and the ridge is 1e-12 n.
//
// B200 layout.  The chain over the exercises is serial: each policy needs the realised values that the later ones leave.  A
// regression is two passes over the paths (moments, then the Gram and right-hand side of the standardised design), each over
// the whole GPU for all Bermudans at once: grid (path chunks, regressions), a partial per CTA, and the regression's last CTA
// adds the partials in chunk order (so the fit is deterministic) and solves the normal equations by an FP64 Cholesky
// factorisation.  The exercise update of a policy is part of the next one's first pass.  The realised values after each
// exercise are kept, so the continuation regressions of every date, which nothing waits for, run after the chain in two
// launches.  The Gram of a one-dimensional monomial basis is a handful of power moments, an FP64 CUDA-core reduction: the
// work per path is ~30 flops against 12-20 bytes read.
// One netting set of 4 Bermudans, 200,000 paths, 40 dates, fit without the simulation: 4.1 ms in one cluster of 8 CTAs per
// Bermudan, date by date; here 0.66 ms, of it the chain's 19 launches 0.40.  Two regressors, 3 Bermudans, 50,000 paths:
// 5.0 ms and 0.77 ms.
#include "zk_device.cuh"
#include "zk_kernels.h"

namespace zk {

namespace {

constexpr int kFitThreads = 256;
constexpr int kFitWarps = kFitThreads / 32;
constexpr int kMoments2 = 6;     // count, sum x, sum x^2, sum s, sum s^2, sum y (one regressor: count, sum x, sum x^2, sum y)
constexpr int kGram1 = 14;       // 10 Gram entries (lower triangle, degree 3) + 4 right-hand sides
// The two-regressor basis: its Gram entries are the mixed moments sum z^a w^b, a + b <= 6 (28 of them, where the
// lower triangle of 10 functions has 55 entries), plus the 10 right-hand sides: one pass of 38 sums.
constexpr int kMom2 = 28, kGram2 = kMom2 + 10;
static_assert(kGram2 <= kFitSums, "a partial holds the sums");

struct FitSmem {
  double warpBuf[kFitWarps][kGram2];
  double tot[kGram2];
  bool last;
};

// Sums V values over the CTA (a fixed shuffle tree per warp, then the warps in order) into the item's partial of this
// chunk; the item's last CTA to arrive adds the partials in chunk order into s.tot and returns true.
template <int V>
__device__ __forceinline__ bool itemSum(double (&v)[V], FitSmem& s, double* __restrict__ part, uint32_t* __restrict__ counter) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_xor_sync(0xFFFFFFFFu, v[i], off);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < V; ++i) s.warpBuf[warp][i] = v[i];
  __syncthreads();
  double* item = part + static_cast<size_t>(blockIdx.y) * gridDim.x * kFitSums;
  if (threadIdx.x < V) {
    double t = 0.0;
    for (int w = 0; w < kFitWarps; ++w) t += s.warpBuf[w][threadIdx.x];
    item[static_cast<size_t>(blockIdx.x) * kFitSums + threadIdx.x] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s.last = atomicAdd(counter + blockIdx.y, 1u) + 1u == gridDim.x;
    if (s.last) counter[blockIdx.y] = 0;  // for the next launch
  }
  __syncthreads();
  if (!s.last) return false;
  __threadfence();
  for (int i = warp; i < V; i += kFitWarps) {  // a warp per sum: lanes over the chunks, then a fixed tree
    double t = 0.0;
    for (uint32_t c = lane; c < gridDim.x; c += 32) t += __ldcg(item + static_cast<size_t>(c) * kFitSums + i);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
    if (lane == 0) s.tot[i] = t;
  }
  __syncthreads();
  return true;
}

// z^0 .. z^d by repeated multiplication, as the reference's design rows.
__device__ __forceinline__ void powers(double z, int d, double (&pw)[4]) {
  pw[0] = 1.0;
#pragma unroll
  for (int i = 1; i < 4; ++i) pw[i] = i <= d ? pw[i - 1] * z : 0.0;
}

// A fitted record f (kFitOut doubles): center, scale, c0..c3 and at [kFitOut - 1] the degree; two regressors: cx, sx, cs, ss,
// c0..c9 and the degree (-1: no sample, predicts 0).
__device__ __forceinline__ double predict(const double* f, double x) {
  const double z = (x - f[0]) / f[1];
  const int d = static_cast<int>(f[kFitOut - 1]);
  double v = 0.0;
  for (int i = d; i >= 0; --i) v = v * z + f[2 + i];
  return v;
}

// ---- the two-regressor basis (this library's extension: the reference regresses on x alone) ----

// The co-terminal swap rate of a path from its short rate, over the slot's bonds in plan order (as the fused
// kernel forms it: annuity and float leg each summed term by term, then their ratio).
__device__ __forceinline__ double swapRateOf(const double4* __restrict__ b, uint2 range, double x) {
  double ann = 0.0, flt = 0.0;
  for (uint32_t i = 0; i < range.y; ++i) {
    const double4 q = b[range.x + i];
    const double v = q.y * (q.z * exp(-q.w * x));
    if (q.x == 13.0) ann += v;
    else flt += v;
  }
  return ann != 0.0 ? flt / ann : 0.0;
}

// The graded monomials 1, z, w, z^2, z w, w^2, z^3, z^2 w, z w^2, w^3: the exponents of z and w of function i.
__host__ __device__ constexpr int powZ(int i) { return i == 1 || i == 4 || i == 8 ? 1 : i == 3 || i == 7 ? 2 : i == 6 ? 3 : 0; }
__host__ __device__ constexpr int powW(int i) { return i == 2 || i == 4 || i == 7 ? 1 : i == 5 || i == 8 ? 2 : i == 9 ? 3 : 0; }
// Index of the moment sum z^a w^b (a + b <= 6) among the 28.
__host__ __device__ constexpr int moment2(int a, int b) { return a * 7 - a * (a - 1) / 2 + b; }

__device__ __forceinline__ int basisCount2(int d) { return d <= 0 ? 1 : d == 1 ? 3 : d == 2 ? 6 : 10; }

__device__ __forceinline__ double predict2(const double* res, double x, double s) {
  const int d = static_cast<int>(res[kFitOut - 1]);
  if (d < 0) return 0.0;
  const double z = (x - res[0]) / res[1], w = (s - res[2]) / res[3];
  const double m[10] = {1.0, z, w, z * z, z * w, w * w, z * z * z, z * z * w, z * w * w, w * w * w};
  const int count = basisCount2(d);
  double v = 0.0;
#pragma unroll
  for (int i = 0; i < 10; ++i)
    if (i < count) v += res[4 + i] * m[i];
  return v;
}

// The normal equations A c = b of k functions by FP64 Cholesky, A = L L^T, L y = b, L^T c = y, by one warp: lane i holds
// row i of A (its lower triangle is read) and b_i, and ends with c_i.  False when A is not positive definite.  (By one
// thread, with the matrix in local memory, it was most of a policy's 26 us second pass.)
template <int K>
__device__ bool solveWarp(double (&a)[K], double& b, int k) {
  const int lane = threadIdx.x & 31;
  auto from = [](double v, int src) { return __shfl_sync(0xFFFFFFFFu, v, src); };
  bool ok = true;
#pragma unroll
  for (int m = 0; m < K; ++m) {
    if (m >= k) break;
    double d = from(a[m], m);
    if (!(d > 0.0)) ok = false, d = 1.0;
    const double root = sqrt(d);
    a[m] = lane == m ? root : a[m] / root;  // column m of L (rows above are not read)
#pragma unroll
    for (int j = m + 1; j < K; ++j) {
      const double l = from(a[m], j);
      if (lane >= j) a[j] -= a[m] * l;
    }
  }
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (j >= k) break;
    const double y = from(b, j) / from(a[j], j);
    if (lane == j) b = y;
    else if (lane > j) b -= a[j] * y;
  }
#pragma unroll
  for (int j = K - 1; j >= 0; --j) {
    if (j >= k) continue;
    const double c = from(b, j) / from(a[j], j);
    if (lane == j) b = c;
#pragma unroll
    for (int i = 0; i < j; ++i) {
      const double l = from(a[i], j);
      if (lane == i) b -= l * c;
    }
  }
  return ok;
}

// center, scale and degree of a one-regressor fit of n samples from their moments, and at degree 0 the mean y: the record f.
__device__ __forceinline__ void standardise1(double n, double sx, double sxx, double sy, int degree, double* f) {
  int d = degree;
  f[0] = 0.0, f[1] = 1.0;
  for (int i = 2; i < 6; ++i) f[i] = 0.0;
  if (n == 0.0) {
    d = 0;  // no sample: the regression predicts 0
  } else {
    f[0] = sx / n;
    const double var = sxx / n - f[0] * f[0];
    f[1] = sqrt(var > 0.0 ? var : 0.0);
    if (f[1] < 1e-12 * fmax(1.0, fabs(f[0]))) d = 0;
    if (n < 2.0 * (d + 1)) d = n >= 4.0 ? static_cast<int>(n) / 2 - 1 : 0;
    if (d == 0) f[1] = 1.0, f[2] = sy / n;
  }
  f[kFitOut - 1] = static_cast<double>(d);
}

// The one-regressor coefficients of degree d from the Gram's lower triangle and the right-hand sides, by one warp into
// c[0..3]; the ridge is 1e-12 n.
__device__ __forceinline__ bool solve1(const double* gram, const double* rhs, int d, double* c) {
  const int lane = threadIdx.x & 31;
  double a[4], b = lane <= d ? rhs[lane & 3] : 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = lane < 4 && j <= lane ? gram[lane * (lane + 1) / 2 + j] : 0.0;
    if (j == lane) a[j] += 1e-12 * gram[0];
  }
  const bool ok = solveWarp(a, b, d + 1);
  if (lane < 4) c[lane] = lane <= d ? b : 0.0;
  return ok;
}

// First pass of the regressions `items`: the realised values after the policy `prev` (its exercise rule "E > 0 and E >
// regression": realised = D E), then the moments of the included paths; the item's last CTA writes center, scale and degree
// (and at degree 0 the mean) into the record.  Two regressors: each included path's co-terminal swap rate (its bonds'
// exponentials) into the item's row of swap rates, which the second pass and the next policy's update read.
template <typename R, bool TwoD>
__global__ void __launch_bounds__(kFitThreads) fitMomentsKernel(const FitItem* __restrict__ items, const FitData<R> F) {
  __shared__ FitSmem s;
  const FitItem I = items[blockIdx.y];
  const uint32_t nP = F.nP, per = (nP + gridDim.x - 1) / gridDim.x, p1 = min((blockIdx.x + 1) * per, nP);
  const R* X = F.x + static_cast<size_t>(I.date) * nP;
  const R* D = F.D + static_cast<size_t>(I.date) * nP;
  const R* E = I.eRow != kNoRow ? F.E + static_cast<size_t>(I.eRow) * nP : nullptr;
  const R* pX = F.x + static_cast<size_t>(I.prevDate) * nP;
  const R* pD = F.D + static_cast<size_t>(I.prevDate) * nP;
  const R* pE = F.E + static_cast<size_t>(I.prevERow) * nP;
  const double* pf = F.fit + static_cast<size_t>(I.prevSlot) * kFitOut;
  const double* in = I.realisedIn != kNoRow ? F.realised + static_cast<size_t>(I.realisedIn) * nP : nullptr;
  double* out = I.prevSlot != kNoRow ? F.realised + static_cast<size_t>(I.realisedOut) * nP : nullptr;
  double* sw = TwoD && I.twoD ? F.swap + static_cast<size_t>(I.swapRow) * nP : nullptr;
  const double* pSw = TwoD && I.twoD ? F.swap + static_cast<size_t>(I.prevSwapRow) * nP : nullptr;
  double m[kMoments2] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (uint32_t p = blockIdx.x * per + threadIdx.x; p < p1; p += kFitThreads) {
    double r = in ? in[p] : 0.0;
    if (out) {
      const double e = static_cast<double>(pE[p]);
      if (e > 0.0) {
        const double xp = static_cast<double>(pX[p]), c = TwoD && I.twoD ? predict2(pf, xp, pSw[p]) : predict(pf, xp);
        if (e > c) r = static_cast<double>(pD[p]) * e;
      }
      out[p] = r;
    }
    if (I.slot == kNoRow || (E && !(E[p] > R(0)))) continue;
    const double x = static_cast<double>(X[p]), y = r / static_cast<double>(D[p]);
    if (TwoD && I.twoD) {
      const double w = swapRateOf(F.bonds, I.bonds, x);
      sw[p] = w;
      m[0] += 1.0, m[1] += x, m[2] += x * x, m[3] += w, m[4] += w * w, m[5] += y;
    } else {
      m[0] += 1.0, m[1] += x, m[2] += x * x, m[3] += y;
    }
  }
  if (I.slot == kNoRow) return;  // the update after the first exercise alone
  if (!itemSum(m, s, F.part, F.counter) || threadIdx.x != 0) return;
  double f[kFitOut] = {};
  const double n = s.tot[0];
  int d = static_cast<int>(I.degree);
  if (TwoD && I.twoD) {
    // Standardised regressors, degree 0 when either is degenerate, lower while the samples are fewer than twice the basis.
    f[1] = f[3] = 1.0;
    if (n == 0.0) {
      d = -1;
    } else {
      f[0] = s.tot[1] / n, f[2] = s.tot[3] / n;
      const double vx = s.tot[2] / n - f[0] * f[0], vs = s.tot[4] / n - f[2] * f[2];
      f[1] = sqrt(vx > 0.0 ? vx : 0.0), f[3] = sqrt(vs > 0.0 ? vs : 0.0);
      if (f[1] < 1e-12 * fmax(1.0, fabs(f[0])) || f[3] < 1e-12 * fmax(1.0, fabs(f[2]))) d = 0;
      while (d > 0 && n < 2.0 * basisCount2(d)) --d;
      if (d == 0) f[0] = f[2] = 0.0, f[1] = f[3] = 1.0, f[4] = s.tot[5] / n;
    }
    f[kFitOut - 1] = static_cast<double>(d);
  } else {
    standardise1(n, s.tot[1], s.tot[2], s.tot[3], d, f);
  }
  double* dst = F.fit + static_cast<size_t>(I.slot) * kFitOut;
  for (int i = 0; i < kFitOut; ++i) dst[i] = f[i];
}

// Second pass: Gram and right-hand side of the standardised design, and the solution.  The ridge is 1e-12 n; with two
// regressors 1e-6 n: in a one-factor model the swap rate is a smooth function of the short rate, the graded Gram's condition
// number reaches 1e17, and 1e-6 n keeps the predictions stable to the summation order (~1e-11) at a negligible bias where
// the data are well conditioned.
template <typename R, bool TwoD>
__global__ void __launch_bounds__(kFitThreads) fitGramKernel(const FitItem* __restrict__ items, const FitData<R> F) {
  __shared__ FitSmem s;
  const FitItem I = items[blockIdx.y];
  const uint32_t nP = F.nP, per = (nP + gridDim.x - 1) / gridDim.x, p0 = blockIdx.x * per + threadIdx.x, p1 = min((blockIdx.x + 1) * per, nP);
  const R* X = F.x + static_cast<size_t>(I.date) * nP;
  const R* D = F.D + static_cast<size_t>(I.date) * nP;
  const R* E = I.eRow != kNoRow ? F.E + static_cast<size_t>(I.eRow) * nP : nullptr;
  // The realised values this regression explains: those its first pass formed, or read.
  const uint32_t row = I.prevSlot != kNoRow ? I.realisedOut : I.realisedIn;
  const double* rz = row != kNoRow ? F.realised + static_cast<size_t>(row) * nP : nullptr;
  double* f = F.fit + static_cast<size_t>(I.slot) * kFitOut;
  const int d = static_cast<int>(f[kFitOut - 1]);
  if (d <= 0) return;
  if (TwoD && I.twoD) {
    const double* sw = F.swap + static_cast<size_t>(I.swapRow) * nP;
    const double cx = f[0], sx = f[1], cs = f[2], ss = f[3];
    // The moments sum z^a w^b (a + b <= 6) and sum z^a w^b y over the basis' exponents, one pass.
    double g[kGram2];
#pragma unroll
    for (int i = 0; i < kGram2; ++i) g[i] = 0.0;
    for (uint32_t p = p0; p < p1; p += kFitThreads) {
      if (E && !(E[p] > R(0))) continue;
      const double z = (static_cast<double>(X[p]) - cx) / sx, w = (sw[p] - cs) / ss;
      const double y = (rz ? rz[p] : 0.0) / static_cast<double>(D[p]);
      double zp[7], wp[7];
      zp[0] = wp[0] = 1.0;
#pragma unroll
      for (int i = 1; i < 7; ++i) zp[i] = zp[i - 1] * z, wp[i] = wp[i - 1] * w;
#pragma unroll
      for (int a = 0; a <= 6; ++a)
#pragma unroll
        for (int b = 0; a + b <= 6; ++b) g[moment2(a, b)] += zp[a] * wp[b];
#pragma unroll
      for (int i = 0; i < 10; ++i) g[kMom2 + i] += zp[powZ(i)] * wp[powW(i)] * y;  // the right-hand sides
    }
    if (!itemSum(g, s, F.part, F.counter) || threadIdx.x >= 32) return;
    const int lane = threadIdx.x, count = basisCount2(d);
    double a[10], b = lane < count ? s.tot[kMom2 + lane] : 0.0;
#pragma unroll
    for (int j = 0; j < 10; ++j) {
      a[j] = lane < 10 ? s.tot[moment2(powZ(lane) + powZ(j), powW(lane) + powW(j))] : 0.0;
      if (j == lane) a[j] += 1e-6 * s.tot[0];  // sum z^0 w^0: the sample count
    }
    if (!solveWarp(a, b, count) && lane == 0) atomicExch(F.err, kDevBadTerm);
    if (lane < 10) f[4 + lane] = lane < count ? b : 0.0;
  } else {
    const double center = f[0], scale = f[1];
    double g[kGram1];
#pragma unroll
    for (int i = 0; i < kGram1; ++i) g[i] = 0.0;
    for (uint32_t p = p0; p < p1; p += kFitThreads) {
      if (E && !(E[p] > R(0))) continue;
      double pw[4];
      powers((static_cast<double>(X[p]) - center) / scale, d, pw);
      const double y = (rz ? rz[p] : 0.0) / static_cast<double>(D[p]);
      int k = 0;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b <= a; ++b) g[k++] += pw[a] * pw[b];
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) g[10 + a] += pw[a] * y;
    }
    if (!itemSum(g, s, F.part, F.counter) || threadIdx.x >= 32) return;
    if (!solve1(s.tot, s.tot + 10, d, f + 2) && threadIdx.x == 0) atomicExch(F.err, kDevBadTerm);
  }
}

// The continuation regressions of one date for up to kFitShared Bermudans (one regressor, one degree): every path is
// included, so x's moments and the Gram are the same for all of them, and a path's standardised powers and 1 / D are formed
// once.  Pass 1 (gram = false): the moments; pass 2: Gram and right-hand sides, and the solutions.
template <typename R, bool kGram>
__global__ void __launch_bounds__(kFitThreads) fitDateKernel(const FitDate* __restrict__ items, const FitData<R> F) {
  __shared__ FitSmem s;
  constexpr int V = kGram ? 10 + 4 * kFitShared : 3 + kFitShared;
  const FitDate I = items[blockIdx.y];
  const uint32_t nP = F.nP, per = (nP + gridDim.x - 1) / gridDim.x, p1 = min((blockIdx.x + 1) * per, nP);
  const R* X = F.x + static_cast<size_t>(I.date) * nP;
  const R* D = F.D + static_cast<size_t>(I.date) * nP;
  const double* rz[kFitShared];
#pragma unroll
  for (int q = 0; q < kFitShared; ++q)
    rz[q] = q < static_cast<int>(I.count) ? F.realised + static_cast<size_t>(I.realisedIn[q]) * nP : nullptr;
  const double* f0 = F.fit + static_cast<size_t>(I.slot[0]) * kFitOut;
  const int d = kGram ? static_cast<int>(f0[kFitOut - 1]) : 0;
  if (kGram && d <= 0) return;
  const double center = kGram ? f0[0] : 0.0, inv = kGram ? 1.0 / f0[1] : 0.0;
  double g[V];
#pragma unroll
  for (int i = 0; i < V; ++i) g[i] = 0.0;
#pragma unroll 2
  for (uint32_t p = blockIdx.x * per + threadIdx.x; p < p1; p += kFitThreads) {
    const double x = static_cast<double>(X[p]), over = 1.0 / static_cast<double>(D[p]);
    double y[kFitShared];
#pragma unroll
    for (int q = 0; q < kFitShared; ++q) y[q] = q < static_cast<int>(I.count) ? rz[q][p] * over : 0.0;
    if constexpr (kGram) {
      double pw[4];
      powers((x - center) * inv, d, pw);
      int k = 0;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b <= a; ++b) g[k++] += pw[a] * pw[b];
      }
#pragma unroll
      for (int q = 0; q < kFitShared; ++q)
#pragma unroll
        for (int a = 0; a < 4; ++a) g[10 + 4 * q + a] += pw[a] * y[q];
    } else {
      g[0] += 1.0, g[1] += x, g[2] += x * x;
#pragma unroll
      for (int q = 0; q < kFitShared; ++q) g[3 + q] += y[q];
    }
  }
  const uint32_t q = threadIdx.x >> 5;  // a warp per Bermudan
  if (!itemSum(g, s, F.part, F.counter) || q >= I.count) return;
  double* f = F.fit + static_cast<size_t>(I.slot[q]) * kFitOut;
  if constexpr (kGram) {
    if (!solve1(s.tot, s.tot + 10 + 4 * q, d, f + 2) && (threadIdx.x & 31u) == 0) atomicExch(F.err, kDevBadTerm);
  } else if ((threadIdx.x & 31u) == 0) {
    standardise1(s.tot[0], s.tot[1], s.tot[2], s.tot[3 + q], static_cast<int>(I.degree), f);
  }
}

}  // namespace

template <typename R>
cudaError_t launchFit(const FitItem* items, uint32_t numItems, uint32_t chunks, bool gram, bool twoD, const FitData<R>& F, cudaStream_t stream) {
  if (numItems == 0) return cudaSuccess;
  if (numItems > 65535u || chunks == 0 || (twoD && (!F.bonds || !F.swap))) return cudaErrorInvalidValue;
  const dim3 grid(chunks, numItems);
  if (gram) {
    if (twoD) fitGramKernel<R, true><<<grid, kFitThreads, 0, stream>>>(items, F);
    else fitGramKernel<R, false><<<grid, kFitThreads, 0, stream>>>(items, F);
  } else {
    if (twoD) fitMomentsKernel<R, true><<<grid, kFitThreads, 0, stream>>>(items, F);
    else fitMomentsKernel<R, false><<<grid, kFitThreads, 0, stream>>>(items, F);
  }
  return cudaGetLastError();
}

template <typename R>
cudaError_t launchFitDates(const FitDate* items, uint32_t numItems, uint32_t chunks, const FitData<R>& F, cudaStream_t stream) {
  if (numItems == 0) return cudaSuccess;
  if (numItems > 65535u || chunks == 0) return cudaErrorInvalidValue;
  const dim3 grid(chunks, numItems);
  fitDateKernel<R, false><<<grid, kFitThreads, 0, stream>>>(items, F);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  fitDateKernel<R, true><<<grid, kFitThreads, 0, stream>>>(items, F);
  return cudaGetLastError();
}

template cudaError_t launchFitDates<float>(const FitDate*, uint32_t, uint32_t, const FitData<float>&, cudaStream_t);
template cudaError_t launchFitDates<double>(const FitDate*, uint32_t, uint32_t, const FitData<double>&, cudaStream_t);
template cudaError_t launchFit<float>(const FitItem*, uint32_t, uint32_t, bool, bool, const FitData<float>&, cudaStream_t);
template cudaError_t launchFit<double>(const FitItem*, uint32_t, uint32_t, bool, bool, const FitData<double>&, cudaStream_t);

}  // namespace zk
