// The exposure kernels: risk-factor simulation, then revalue -> net -> collateralise -> reduce.
//
// They execute the reference's plan semantics (the fused-exposure WGSL kernel,
// src/gpu/fused_kernels.cpp:224-530, and its CPU mirror simulatePath,
// src/gpu/fused_reference.cpp:198-422), organised for a B200 and for books of many netting sets:
//
//   simulateKernel   producer warps draw the counter-based normals and correlate them, ahead of the warps that
//                    step Hull-White, the lognormal assets and the CIR++ intensities once per date (simulateWalkKernel:
//                    a thread does all of a path or pair, where those fill the GPU), writing the factor state (x, D, S,
//                    Q; lnS and y when probes read them) path-major to HBM.
//                    Every netting set of the launch reuses it: the reference re-simulates per plan.
//                    Only factors are stored, never the paths x dates x trades value cube.
//   revalueKernel    one CTA per (tile of kTile paths, netting set).  CTA ids run tile-major, so the
//                    netting sets of one tile execute together and its factor slice stays in L2.
//                    Each thread revalues its path date by date from the netting set's merged term
//                    table (warp-uniform loads, served to all 32 lanes by one L1 broadcast), applies
//                    the CSA with the margin-call look-back kept in a shared-memory ring, writes the
//                    reporting-date rows and reduces the 8 (+5 per trade) statistics of the date with a
//                    warp reduce-scatter (9 shuffles) and one cross-warp pass per 128-path group into
//                    per-group partials, which the reduce kernel sums in path order: the results are
//                    deterministic and the same for every tile shape.
#include <algorithm>

#include "zk_device.cuh"
#include "zk_kernels.h"

namespace zk {

namespace {

// Lane l ends with the warp sum of statistic statSlotOfLane(l).  The lanes are combined as a binary tree over
// neighbours (xor 1, then 2, 4, 8, 16: the first three halve the 8 values, the last two complete the sums), so
// a statistic's sum over the warp's paths has the same tree whether a lane holds one path or the in-thread sum
// of 2 or 4 adjacent paths: the partials do not depend on the tile shape.
template <typename R>
__device__ __forceinline__ R warpReduceScatter8(const R (&v)[8], uint32_t lane) {
  const bool b0 = lane & 1u, b1 = lane & 2u, b2 = lane & 4u;
  R a[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const R send = b0 ? v[i] : v[i + 4];
    const R keep = b0 ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 1);
  }
  R b[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const R send = b1 ? a[i] : a[i + 2];
    const R keep = b1 ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2);
  }
  R c = (b2 ? b[1] : b[0]) + __shfl_xor_sync(0xFFFFFFFFu, b2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xFFFFFFFFu, c, 8);
  c += __shfl_xor_sync(0xFFFFFFFFu, c, 16);
  return c;
}

__device__ __forceinline__ uint32_t statSlotOfLane(uint32_t lane) {
  return (lane & 1u) * 4u + ((lane >> 1) & 1u) * 2u + ((lane >> 2) & 1u);
}

template <typename R>
__device__ __forceinline__ R sel4(const R (&a)[4], uint32_t i) {
  return i == 0 ? a[0] : i == 1 ? a[1] : i == 2 ? a[2] : a[3];
}

template <typename R>
__device__ __forceinline__ void add4(R (&a)[4], uint32_t i, R v) {
  if (i == 0) a[0] += v;
  else if (i == 1) a[1] += v;
  else if (i == 2) a[2] += v;
  else a[3] += v;
}

template <typename R>
__device__ __forceinline__ void set4(R (&a)[4], uint32_t i, R v) {
  if (i == 0) a[0] = v;
  else if (i == 1) a[1] = v;
  else if (i == 2) a[2] = v;
  else a[3] = v;
}

// One term record (8 values) with warp-uniform vector loads through the read-only path.
__device__ __forceinline__ void loadTerm(const float* t, float (&r)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(t));
  const float4 b = __ldg(reinterpret_cast<const float4*>(t) + 1);
  r[0] = a.x, r[1] = a.y, r[2] = a.z, r[3] = a.w, r[4] = b.x, r[5] = b.y, r[6] = b.z, r[7] = b.w;
}
__device__ __forceinline__ void loadTerm(const double* t, double (&r)[8]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(t) + k);
    r[2 * k] = v.x, r[2 * k + 1] = v.y;
  }
}

// Whether the record at lowered unit u (of a run ending at `end`) is a two-regressor policy / continuation record:
// the next record an extension (kBermExt); then its two extension records into e1, e2.
template <typename R>
__device__ __forceinline__ bool twoRegressors(const R* table, uint32_t u, uint32_t end, R (&e1)[8], R (&e2)[8]) {
  if (u + 2 >= end || (asUint(table[4 * (u + 2)]) & 15u) != kBermExt) return false;
  loadTerm(table + 4 * (u + 2), e1);
  loadTerm(table + 4 * (u + 4), e2);
  return true;
}

// The co-terminal swap rate from its float leg and annuity (0 without an annuity).
template <typename R>
__device__ __forceinline__ R swapRate(R flt, R ann) {
  return ann != R(0) ? flt / ann : R(0);
}

constexpr int kSimWarps = 8, kSimThreads = 32 * kSimWarps;  // warps and threads per CTA of the simulate kernel

// The simulate kernel's shared memory (values of R): a ring of two buffers of `dates` dates, each date `slots` values of the
// CTA's streams, then, with `table`, the Brownian-bridge coefficients [nT][substeps - 1][2].  `need` normals are read
// per date.
struct SimLayout {
  uint32_t need, slots, dates;
  bool table;
};

// The drivers of one (stream, date) into its ring column, slot m at col[m * cols]: the correlated drivers w_0 .. w_{nCorr-1},
// the independent normals of the integrated rates, and per credit the Brownian increments of its sub-steps (the last one
// after all normals, slot need + c).  The Box-Muller pairs are independent of one another, so they overlap.
template <typename R, uint32_t cols>
__device__ __forceinline__ void drawDate(const ScenarioArgs<R>& sc, const SimLayout& L, uint32_t stream, uint32_t j, uint32_t injectedStream,
                                         const R* bridge, R* col) {
  const uint32_t nB = sc.substeps - 1;
  if (sc.normals) {
    for (uint32_t m = 0; m < L.need; ++m)
      col[m * cols] = sc.normals[(static_cast<size_t>(j - 1) * sc.nNormals + m) * sc.nStreams + injectedStream];
  } else {
#pragma unroll 4
    for (uint32_t q = 0; 2 * q < L.need; ++q) {
      R z0, z1;
      gauss2(stream, j, q, z0, z1);
      col[2 * q * cols] = z0;
      if (2 * q + 1 < L.need) col[(2 * q + 1) * cols] = z1;
    }
  }
  // Correlated drivers: each padded Cholesky row as two 4-term dot products (as the reference).
  R z[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) z[k] = static_cast<uint32_t>(k) < sc.nCorr ? col[k * cols] : R(0);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (static_cast<uint32_t>(i) < sc.nCorr) {
      const R* row = sc.chol + i * kChol;
      const R d0 = fma(row[3], z[3], fma(row[2], z[2], fma(row[0], z[0], row[1] * z[1])));
      const R d1 = fma(row[7], z[7], fma(row[6], z[6], fma(row[4], z[4], row[5] * z[5])));
      col[i * cols] = d0 + d1;
    }
  if (sc.nC == 0) return;
  const R dt = __ldg(sc.steps + static_cast<size_t>(j) * sc.stepStride + 6), h = dt / static_cast<R>(sc.substeps);
  const R* bj = bridge + static_cast<size_t>(j) * nB * 2;
  for (uint32_t c = 0; c < sc.nC; ++c) {
    R* zc = col + (sc.nCorr + 1 + sc.nF + c * nB) * cols;
    R rem = rsqrt_(dt) * col[(1 + sc.nA + c) * cols], remT = dt;
    for (uint32_t s = 0; s < nB; ++s) {
      const R a = L.table ? bj[2 * s] : h / remT;
      const R b = L.table ? bj[2 * s + 1] : rsqrt_(fmax(h * (remT - h) / remT, R(0)));
      const R dW = fma(a, rem, b * zc[s * cols]);
      zc[s * cols] = dW;
      rem -= dW;
      remT -= h;
    }
    col[(L.need + c) * cols] = rem;
  }
}

}  // namespace

// A thread's PPT adjacent paths in one 8- or 16-byte access (p aligned to PPT values).
template <typename R, int PPT>
__device__ __forceinline__ void ldPaths(const R* p, R (&v)[PPT]) {
  if constexpr (PPT == 1) {
    v[0] = __ldg(p);
  } else if constexpr (sizeof(R) == 4 && PPT == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    v[0] = t.x, v[1] = t.y;
  } else if constexpr (sizeof(R) == 4 && PPT == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
#pragma unroll
    for (int q = 0; q < PPT; q += 2) {
      const double2 t = __ldg(reinterpret_cast<const double2*>(p) + q / 2);
      v[q] = t.x, v[q + 1] = t.y;
    }
  }
}
template <typename R, int PPT>
__device__ __forceinline__ void stPaths(R* p, const R (&v)[PPT]) {
  if constexpr (PPT == 1) {
    p[0] = v[0];
  } else if constexpr (sizeof(R) == 4 && PPT == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  } else if constexpr (sizeof(R) == 4 && PPT == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int q = 0; q < PPT; q += 2) reinterpret_cast<double2*>(p)[q / 2] = make_double2(v[q], v[q + 1]);
  }
}

namespace {

// The Brownian-bridge coefficients of the CIR sub-steps, the same for every path: the CTA computes them once.
template <typename R>
__device__ __forceinline__ void bridgeTable(const ScenarioArgs<R>& sc, R* bridge) {
  const uint32_t nB = sc.substeps - 1;
  for (uint32_t jj = threadIdx.x + 1; jj < sc.nT; jj += blockDim.x) {
    const R dt = sc.steps[static_cast<size_t>(jj) * sc.stepStride + 6], h = dt / static_cast<R>(sc.substeps);
    R remT = dt;
    for (uint32_t q = 0; q < nB; ++q) {
      bridge[(static_cast<size_t>(jj) * nB + q) * 2] = h / remT;
      bridge[(static_cast<size_t>(jj) * nB + q) * 2 + 1] = rsqrt_(fmax(h * (remT - h) / remT, R(0)));
      remT -= h;
    }
  }
  __syncthreads();
}

// The rates and assets of a thread's PPL paths.  The deflator's exponent -sum of the integrated short rate accumulates in
// double precision in both modes (the reference's kernel sums it in single precision, fused_kernels.cpp:250-253);
// D = exp(lnD) is then taken in R.
template <typename R, int PPL>
struct RateState {
  R x[PPL], D[PPL], S[4][PPL], lnS[4][PPL], xf[2][PPL];  // xf: stochastic foreign short-rate states of assets 0 and 1
  double lnD[PPL];
  __device__ __forceinline__ explicit RateState(const ScenarioArgs<R>& sc) {
#pragma unroll
    for (int i = 0; i < PPL; ++i) {
      x[i] = R(0), D[i] = R(1), lnD[i] = 0.0, xf[0][i] = xf[1][i] = R(0);
#pragma unroll
      for (int a = 0; a < 4; ++a) S[a][i] = sc.spots[a], lnS[a][i] = R(0);
    }
  }
};

// One date's step, from the drivers at buf[m * cols].
template <typename R, int PPL, uint32_t cols>
__device__ __forceinline__ void stepRates(const ScenarioArgs<R>& sc, uint32_t j, const R* buf, const R (&sign)[PPL], RateState<R, PPL>& st) {
  const R* step = sc.steps + static_cast<size_t>(j) * sc.stepStride;
  const R s0 = __ldg(step), s1 = __ldg(step + 1), s2 = __ldg(step + 2), s3 = __ldg(step + 3), s4 = __ldg(step + 4), s5 = __ldg(step + 5);
  const R w0 = buf[0], zI = buf[sc.nCorr * cols];
  R integratedRate[PPL], carry[4][PPL];
#pragma unroll
  for (int i = 0; i < PPL; ++i) {
    const R w = sign[i] * w0, z = sign[i] * zI;
    integratedRate[i] = fma(s3, z, fma(st.x[i], s5, s2 * w)) + s4;
    st.x[i] = fma(st.x[i], s0, s1 * w);
    st.lnD[i] -= static_cast<double>(integratedRate[i]);
    st.D[i] = rexp(static_cast<R>(st.lnD[i]));
  }
  // Stochastic foreign rates: the exact Hull-White step of x_f (with its quanto drift) and of its integral, on
  // driver 1 + nA + nC + f and the independent normal nCorr + 1 + f; the asset's carry is then the simulated
  // integral of r_f instead of the deterministic one.
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int i = 0; i < PPL; ++i) carry[a][i] = __ldg(step + 8 + a);
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    if (static_cast<uint32_t>(f) < sc.nF) {
      const R* fs = step + kStepStride + 8 * f;
      const R wf0 = buf[(1 + sc.nA + sc.nC + f) * cols], zf0 = buf[(sc.nCorr + 1 + f) * cols];
#pragma unroll
      for (int i = 0; i < PPL; ++i) {
        const R wf = sign[i] * wf0, zf = sign[i] * zf0;
        carry[f][i] = fma(__ldg(fs + 3), zf, fma(st.xf[f][i], __ldg(fs + 5), __ldg(fs + 2) * wf)) + __ldg(fs + 4) + __ldg(fs + 7);
        st.xf[f][i] = fma(st.xf[f][i], __ldg(fs), __ldg(fs + 1) * wf) + __ldg(fs + 6);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    if (static_cast<uint32_t>(a) < sc.nA) {
      const R drift = __ldg(step + 16 + a), vol = __ldg(step + 12 + a), wa = buf[(1 + a) * cols];
#pragma unroll
      for (int i = 0; i < PPL; ++i) {
        st.lnS[a][i] = st.lnS[a][i] + fma(vol, sign[i] * wa, integratedRate[i] - carry[a][i] - drift);
        st.S[a][i] = sc.spots[a] * rexp(st.lnS[a][i]);
      }
    }
  }
}

template <typename R, int PPL, typename Put>
__device__ __forceinline__ void writeRates(const ScenarioArgs<R>& sc, const CubeArgs<R>& cb, uint32_t j, const RateState<R, PPL>& st, const Put& put) {
  put(0, j, st.x);
  put(1, j, st.D);
#pragma unroll
  for (int a = 0; a < 4; ++a)
    if (static_cast<uint32_t>(a) < sc.nA) put(cb.fS + a, j, st.S[a]);
#pragma unroll
  for (int f = 0; f < 2; ++f)
    if (static_cast<uint32_t>(f) < sc.nF) put(cb.fXf + f, j, st.xf[f]);
  if (cb.probes)
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if (static_cast<uint32_t>(a) < sc.nA) put(cb.fLnS + a, j, st.lnS[a]);
}

// One CIR++ intensity of a thread's PPL paths, and where a date's drivers hold its increments (values from the column's first).
template <typename R, int PPL>
struct CreditState {
  R y[PPL], Y[PPL], Q[PPL], kappa, theta, xi;
  uint32_t at, last;
  __device__ __forceinline__ CreditState(const ScenarioArgs<R>& sc, const SimLayout& L, uint32_t c, uint32_t cols)
      : kappa(sc.cir[4 * c]), theta(sc.cir[4 * c + 1]), xi(sc.cir[4 * c + 2]),
        at((sc.nCorr + 1 + sc.nF + c * (sc.substeps - 1)) * cols), last((L.need + c) * cols) {
#pragma unroll
    for (int i = 0; i < PPL; ++i) y[i] = sc.cir[4 * c + 3], Y[i] = R(0), Q[i] = R(1);
  }
};

template <typename R, int PPL, uint32_t cols>
__device__ __forceinline__ void stepCredit(const ScenarioArgs<R>& sc, uint32_t c, uint32_t j, const R* buf, const R (&sign)[PPL],
                                           CreditState<R, PPL>& st) {
  const uint32_t nB = sc.substeps - 1;
  const R* step = sc.steps + static_cast<size_t>(j) * sc.stepStride;
  const R h = __ldg(step + 6) / static_cast<R>(sc.substeps), shift = __ldg(step + 20 + c);
  auto subStep = [&](R dW0) {
#pragma unroll
    for (int i = 0; i < PPL; ++i) {
      const R dW = sign[i] * dW0, yp = fmax(st.y[i], R(0));
      const R yn = fma(st.xi * rsqrt_(yp), dW, fma(st.kappa * (st.theta - yp), h, st.y[i]));
      st.Y[i] = fma(R(0.5) * (yp + fmax(yn, R(0))), h, st.Y[i]);
      st.y[i] = yn;
    }
  };
#pragma unroll 4
  for (uint32_t s = 0; s < nB; ++s) subStep(buf[st.at + s * cols]);
  subStep(buf[st.last]);
#pragma unroll
  for (int i = 0; i < PPL; ++i) st.Q[i] = rexp(-st.Y[i] - shift);
}

template <typename R, int PPL, typename Put>
__device__ __forceinline__ void writeCredit(const CubeArgs<R>& cb, uint32_t c, uint32_t j, const CreditState<R, PPL>& st, const Put& put) {
  put(cb.fQ + c, j, st.Q);
  if (cb.probes) put(cb.fY + c, j, st.y);
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Risk factors of every path and date (the transitions of the reference's ScenarioGenerator:
// hull_white.cpp:40-68, lognormal_asset.cpp:17-22, cir_intensity.cpp:49-66, in the statement order
// of the reference kernel; the fused multiply-adds are written out so that every shape rounds alike).
//
// Only the states are serial in the dates; the normals and everything linear in them (correlation, Brownian bridge) are
// not, and they are most of the work.  So a CTA takes `cols` normal streams with eight warps: one steps the rates and the
// assets, one per credit steps its CIR++ intensity, and the others produce the drivers of several dates ahead into a
// shared-memory ring.  An antithetic pair's drivers differ by their sign only (exactly, rounding being symmetric), so
// they are produced once per pair: with 32 streams a lane steps both paths of its stream (PPL = 2: two independent
// chains of the CIR++ sub-steps' square roots, which bind), with 16 streams adjacent lanes share one and a producer pass
// covers two dates.  Without pairs a stream is a path.
// Against one thread that draws and steps a path: 389 us at 2,000 paths x 121 dates, 4 factors, and 1,159 us at 100,000 x 169,
// 6 factors; 16 streams take 80 and 991 us, 32 take 108 and 735.
template <typename R, int PPL, uint32_t cols>
__global__ void __launch_bounds__(kSimThreads, sizeof(R) == 4 ? 4 : 2) simulateKernel(const ScenarioArgs<R> sc, const CubeArgs<R> cb,
                                                                                     const SimLayout L) {
  extern __shared__ __align__(16) unsigned char simRaw[];
  R* ring = reinterpret_cast<R*>(simRaw);
  const uint32_t bufLen = L.dates * L.slots * cols;
  R* bridge = ring + 2 * static_cast<size_t>(bufLen);
  // bridgeTable in line: as a call it costs the credits' loops 3%.
  const uint32_t nB = sc.substeps - 1, nP = sc.nP, nT = sc.nT;
  if (L.table) {
    for (uint32_t jj = threadIdx.x + 1; jj < nT; jj += blockDim.x) {
      const R dt = sc.steps[static_cast<size_t>(jj) * sc.stepStride + 6], h = dt / static_cast<R>(sc.substeps);
      R remT = dt;
      for (uint32_t q = 0; q < nB; ++q) {
        bridge[(static_cast<size_t>(jj) * nB + q) * 2] = h / remT;
        bridge[(static_cast<size_t>(jj) * nB + q) * 2 + 1] = rsqrt_(fmax(h * (remT - h) / remT, R(0)));
        remT -= h;
      }
    }
    __syncthreads();
  }
  // The roles rotate with the CTA over the warps, so that the resident CTAs load the four schedulers alike.
  const uint32_t lane = threadIdx.x & 31u, role = ((threadIdx.x >> 5) + blockIdx.x) & (kSimWarps - 1u);
  const uint32_t numProducers = kSimWarps - 1 - sc.nC;
  const uint32_t blocks = nT > 1 ? (nT - 1 + L.dates - 1) / L.dates : 0u;  // ring buffers, dates 1 .. nT - 1
  // This lane's first path p0 (with PPL = 2, p0 + 1 is the antithetic one) and its stream's column; lanes past the last
  // path repeat it and write nothing.
  const uint32_t p0 = (blockIdx.x * 32u + lane) * PPL, col = cols == 16u ? lane >> 1u : lane;
  auto planPath = [&](uint32_t p) { return sc.pathMap ? sc.pathMap[min(p, nP - 1)] : min(p, nP - 1); };

  if (role > sc.nC) {
    // ================================ producers ================================
    constexpr uint32_t perPass = 32u / cols;  // dates of a producer warp's pass
    const uint32_t mine = lane & (cols - 1u), sub = lane / cols;
    const uint32_t po = planPath(cols == 16u ? blockIdx.x * 32u + 2u * mine : p0);
    const uint32_t pathStream = sc.antithetic ? po >> 1u : po;
    const uint32_t injectedStream = sc.nStreams > 0 ? min(pathStream, sc.nStreams - 1) : 0u;
    const uint32_t stream = pcg(pcg(sc.seed) ^ pcg(pathStream + 0x9E3779B9u));
    for (uint32_t b = 0; b <= blocks; ++b) {
      if (b < blocks)
        for (uint32_t d = (role - 1 - sc.nC) * perPass + sub; d < L.dates; d += numProducers * perPass) {
          const uint32_t j = 1 + b * L.dates + d;
          if (j < nT) drawDate<R, cols>(sc, L, stream, j, injectedStream, bridge, ring + (b & 1u) * bufLen + d * L.slots * cols + mine);
        }
      __syncthreads();
    }
    return;
  }

  // ================================ the states ================================
  const uint32_t po = planPath(p0);
  R sign[PPL];
#pragma unroll
  for (int i = 0; i < PPL; ++i) sign[i] = PPL == 2 ? (i == 0 ? R(1) : R(-1)) : sc.antithetic && (po & 1u) ? R(-1) : R(1);
  const bool vec = PPL == 2 && nP % 2u == 0u;  // a lane's pair of paths in one store
  auto put = [&](uint32_t field, uint32_t j, const R (&v)[PPL]) {
    R* dst = cb.data + (static_cast<size_t>(field) * nT + j) * nP + p0;
    if (vec) {
      if (p0 < nP) stPaths<R, PPL>(dst, v);
    } else {
#pragma unroll
      for (int i = 0; i < PPL; ++i)
        if (p0 + i < nP) dst[i] = v[i];
    }
  };
  if (role == 0) {
    RateState<R, PPL> st(sc);
    writeRates<R, PPL>(sc, cb, 0, st, put);
    for (uint32_t b = 0; b <= blocks; ++b) {
      if (b > 0) {
        const uint32_t j0 = 1 + (b - 1) * L.dates, j1 = min(j0 + L.dates, nT);
        const R* buf = ring + ((b - 1) & 1u) * bufLen + col;
#pragma unroll 1
        for (uint32_t j = j0; j < j1; ++j, buf += L.slots * cols) {
          stepRates<R, PPL, cols>(sc, j, buf, sign, st);
          writeRates<R, PPL>(sc, cb, j, st, put);
        }
      }
      __syncthreads();
    }
    return;
  }
  const uint32_t c = role - 1;  // this warp's credit
  CreditState<R, PPL> st(sc, L, c, cols);
  writeCredit<R, PPL>(cb, c, 0, st, put);
  for (uint32_t b = 0; b <= blocks; ++b) {
    if (b > 0) {
      const uint32_t j0 = 1 + (b - 1) * L.dates, j1 = min(j0 + L.dates, nT);
      const R* buf = ring + ((b - 1) & 1u) * bufLen + col;
#pragma unroll 1
      for (uint32_t j = j0; j < j1; ++j, buf += L.slots * cols) {
        stepCredit<R, PPL, cols>(sc, c, j, buf, sign, st);
        writeCredit<R, PPL>(cb, c, j, st, put);
      }
    }
    __syncthreads();
  }
}

// The same states by threads that each draw and step their PPL paths (2: an antithetic pair) date after date: where the paths
// alone fill the GPU it is the faster one (launchSimulate has the rule and the times).  Its working set is a thread's drivers
// of one date; what binds it is the issue of the normals and exponentials.
template <typename R, int PPL>
__global__ void __launch_bounds__(kSimThreads) simulateWalkKernel(const ScenarioArgs<R> sc, const CubeArgs<R> cb, const SimLayout L) {
  extern __shared__ __align__(16) unsigned char simRaw[];
  R* col = reinterpret_cast<R*>(simRaw) + threadIdx.x;
  R* bridge = reinterpret_cast<R*>(simRaw) + static_cast<size_t>(L.slots) * kSimThreads;
  if (L.table) bridgeTable(sc, bridge);
  const uint32_t nP = sc.nP, p0 = (blockIdx.x * kSimThreads + threadIdx.x) * PPL;
  if (p0 >= nP) return;
  const uint32_t po = sc.pathMap ? sc.pathMap[p0] : p0, pathStream = sc.antithetic ? po >> 1u : po;
  const uint32_t injectedStream = sc.nStreams > 0 ? min(pathStream, sc.nStreams - 1) : 0u;
  const uint32_t stream = pcg(pcg(sc.seed) ^ pcg(pathStream + 0x9E3779B9u));
  R sign[PPL];
#pragma unroll
  for (int i = 0; i < PPL; ++i) sign[i] = PPL == 2 ? (i == 0 ? R(1) : R(-1)) : sc.antithetic && (po & 1u) ? R(-1) : R(1);
  auto put = [&](uint32_t field, uint32_t j, const R (&v)[PPL]) {
    R* dst = cb.data + (static_cast<size_t>(field) * sc.nT + j) * nP + p0;
    if (PPL == 2 && nP % 2u == 0u) {
      stPaths<R, PPL>(dst, v);
    } else {
#pragma unroll
      for (int i = 0; i < PPL; ++i)
        if (p0 + i < nP) dst[i] = v[i];
    }
  };
  RateState<R, PPL> st(sc);
  CreditState<R, PPL> cr[2] = {CreditState<R, PPL>(sc, L, 0, kSimThreads), CreditState<R, PPL>(sc, L, 1, kSimThreads)};
  for (uint32_t j = 0; j < sc.nT; ++j) {
    if (j > 0) {
      drawDate<R, kSimThreads>(sc, L, stream, j, injectedStream, bridge, col);
      stepRates<R, PPL, kSimThreads>(sc, j, col, sign, st);
    }
    writeRates<R, PPL>(sc, cb, j, st, put);
#pragma unroll
    for (uint32_t c = 0; c < 2; ++c)
      if (c < sc.nC) {
        if (j > 0) stepCredit<R, PPL, kSimThreads>(sc, c, j, col, sign, cr[c]);
        writeCredit<R, PPL>(cb, c, j, cr[c], put);
      }
  }
}

// ---------------------------------------------------------------------------------------------
// The exponential of a lowered term: 2^(b x) with b = -B log2 e in single precision, e^(b x) with b = -B
// in double (lowerTerms, capi.cu).
__device__ __forceinline__ float termExp(float b, float x) { return ex2(b * x); }
__device__ __forceinline__ double termExp(double b, double x) { return exp(b * x); }

template <typename R> struct Vec4;
template <> struct Vec4<float> { using T = float4; };
template <> struct Vec4<double> { using T = double4; };
__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ double4 ld4(const double* p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// Prefetches into L1 the 128-byte lines of one date's lowered terms, one line per thread of the CTA:
// the next date's block arrives while the current date computes.
__device__ __forceinline__ void prefetchL1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(p)));
}
template <typename R>
__device__ __forceinline__ void prefetchDate(uint32_t begin, uint32_t end, const R* table, uint32_t tid) {
  const size_t b = static_cast<size_t>(begin) * 4 * sizeof(R), e = static_cast<size_t>(end) * 4 * sizeof(R);
  const uint32_t lines = e > b ? static_cast<uint32_t>((e - 1) / 128 - b / 128 + 1) : 0u;
  if (tid < lines) prefetchL1(reinterpret_cast<const char*>(table) + (b / 128 + tid) * 128);
}

template <typename R, int PPT>
__device__ __forceinline__ R pick4(const R (&a)[4][PPT], uint32_t k, int i) {
  return k == 0 ? a[0][i] : k == 1 ? a[1][i] : k == 2 ? a[2][i] : a[3][i];
}

// A product never fused into an addition and an addition never fused with a product: what two kernels compute alike rounds
// alike, however the compiler arranges each.
__device__ __forceinline__ float mulRn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulRn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float addRn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double addRn(double a, double b) { return __dadd_rn(a, b); }

// The fixing that a generic record (c, A, B) sets from its date's short rate.
template <typename R>
__device__ __forceinline__ R genericFixing(R c, R A, R B, R x) {
  return (A * fastExp(-B * x) - R(1)) / c;
}

// a e + b f with one product fused, the same one in every kernel (left to the compiler, the walk and the split differed in
// double precision).
__device__ __forceinline__ float bondPair(float a, float e, float b, float f) { return fmaf(a, e, b * f); }
__device__ __forceinline__ double bondPair(double a, double e, double b, double f) { return fma(b, f, a * e); }

// The netting set's value on date j of a thread's PPT paths (value), from the date's lowered runs [d0, d1), and the
// fixings and exercise states the date sets.  state: the fixings [slot][PPT][kTile]; the exercise index of Bermudan b
// (-1: not exercised) in bytes exS[b][PPT][kTile] when exBytes, else in registers ex.  kGiven: the decisions are those
// of decideKernel (A.exIndex), not taken here.
template <typename R, int PPT, bool kPerTrade, bool kSink, bool kLean, bool kGiven>
__device__ __forceinline__ void revalueDate(const NsArgs<R>& A, const CubeArgs<R>& cb, const R* const (&cubeP)[PPT], const uint4 d0,
                                            const uint4 d1, const uint32_t j, const uint32_t tid, const uint32_t (&pth)[PPT],
                                            const bool (&act)[PPT], const R (&x)[PPT], const R (&D)[PPT], const R (&S)[4][PPT],
                                            const R (&xf)[2][PPT], const R guardJ, R* state, R* vtBuf, signed char* exS,
                                            const bool exBytes, R (&ex)[4][PPT], R (&value)[PPT]) {
  const R* __restrict__ table = A.table;
  R* __restrict__ expo = A.expo;
  const uint32_t nP = cb.nP;
  const size_t fieldStride = static_cast<size_t>(cb.nT) * nP;
  const bool manyBerm = !kLean && exBytes;
  const uint32_t nTr = kPerTrade ? min(A.nTr, static_cast<uint32_t>(kMaxTradeGroups)) : 0u;
  auto fix = [&](uint32_t slot, int i) -> R& { return state[(slot * PPT + i) * kTile + tid]; };
  auto vt = [&](uint32_t g, int i) -> R& { return vtBuf[(g * PPT + i) * kTile + tid]; };
  auto cube = [&](uint32_t field, uint32_t jj, int i) { return cubeP[i][field * fieldStride + static_cast<size_t>(jj) * nP]; };
  auto xfOf = [&](uint32_t a, int i) { return kGiven ? (a == 0 ? xf[0][i] : xf[1][i]) : cube(cb.fXf + a, j, i); };
  auto exOf = [&](uint32_t b, int i) -> R {
    return manyBerm ? static_cast<R>(exS[(b * PPT + i) * kTile + tid]) : pick4<R, PPT>(ex, b, i);
  };
  R ev[4][PPT];
  R annS[PPT], fltS[PPT];  // the co-terminal swap of the next two-regressor record: annuity, float leg
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    value[i] = R(0), annS[i] = R(0), fltS[i] = R(0);
#pragma unroll
    for (int b = 0; b < 4; ++b) ev[b][i] = R(0);
  }
  using R4 = typename Vec4<R>::T;
  for (uint32_t u = d0.x; u < d0.y; ++u) {  // running floating coupons
    const R4 r = ld4(table + 4 * u);
    const uint32_t slot = asUint(r.w);
#pragma unroll
    for (int i = 0; i < PPT; ++i) value[i] = fma(fma(r.x, fix(slot, i), r.y), termExp(r.z, x[i]), value[i]);
  }
#pragma unroll 2
  for (uint32_t u = d0.y; u < d0.z; ++u) {  // bonds, two per record
    const R4 r = ld4(table + 4 * u);
#pragma unroll
    for (int i = 0; i < PPT; ++i) value[i] += bondPair(r.x, termExp(r.y, x[i]), r.z, termExp(r.w, x[i]));
  }
  for (uint32_t u = d0.z; u < d0.w; ++u) {  // asset forwards: (c, A, asset)
    const R4 r = ld4(table + 4 * u);
    const uint32_t a = asUint(r.z) & 3u;
#pragma unroll
    for (int i = 0; i < PPT; ++i) value[i] = fma(r.x * pick4<R, PPT>(S, a, i), r.y, value[i]);
  }
  if (kPerTrade && A.nTr > 0)
    for (uint32_t g = 0; g < kMaxTradeGroups; ++g)
#pragma unroll
      for (int i = 0; i < PPT; ++i) vt(g, i) = R(0);
  for (uint32_t u = d0.w; u < d1.x; u += 2) {  // generic terms: the reference's records
    R rec[8];
    loadTerm(table + 4 * u, rec);
    const uint32_t code = asUint(rec[0]), slot = asUint(rec[1]);
    const uint32_t kind = code & 15u, bm = bermudanOf(code, A.manyBerm != 0), extra = code >> 12u;
    const uint32_t grp = min((code >> 4u) & 15u, 15u);
    if (!kLean && kind == kBermBond && slot >= kBlockMark) {
      // A block of nb bonds of Bermudan bm (the lowering's run of its kBermBond records): each counts on a path
      // that exercised at or before the bond's exercise index; a warp with no such path skips the block.
      const uint32_t nb = slot - kBlockMark;
      R exi[PPT];
      bool live = false;
#pragma unroll
      for (int i = 0; i < PPT; ++i) exi[i] = exOf(bm, i), live = live || (exi[i] >= R(0) && exi[i] <= rec[2]);
      if (__any_sync(0xFFFFFFFFu, live))
        for (uint32_t q = 0; q < nb; ++q) {
          const R4 b = ld4(table + 4 * (u + 2 + q));
          const R nBq = -b.z;
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            R term = R(0);
            if (exi[i] >= R(0) && exi[i] <= b.w) term = b.x * (b.y * fastExp(nBq * x[i]));
            if (kPerTrade && A.nTr > 0) vt(grp, i) += term;
            else value[i] = addRn(value[i], term);
          }
        }
      u += 2 * ((nb + 1) / 2);
      continue;
    }
    const R c = rec[2], nB = -rec[4];
    R term[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) term[i] = R(0);
    switch (kind) {
      case kBond:
#pragma unroll
        for (int i = 0; i < PPT; ++i) term[i] = c * (rec[3] * fastExp(nB * x[i]));
        break;
      case kFixedFloat:
#pragma unroll
        for (int i = 0; i < PPT; ++i) term[i] = (c * fix(slot, i) + rec[5]) * (rec[3] * fastExp(nB * x[i]));
        break;
      case kAsset:
#pragma unroll
        for (int i = 0; i < PPT; ++i) term[i] = c * pick4<R, PPT>(S, slot & 3u, i) * rec[3];
        break;
      case kSetFixing:
#pragma unroll
        for (int i = 0; i < PPT; ++i) fix(slot, i) = genericFixing(c, rec[3], rec[4], x[i]);
        break;
      case kOption: {
        const R p3 = rec[7];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
          const R b0 = rec[3] * fastExp(nB * x[i]);
          term[i] = c * black(pick4<R, PPT>(S, slot & 3u, i) * rec[5] / b0, rec[6], fabs(p3), b0, p3 > R(0));
        }
        break;
      }
      case kForeignForward: {  // c S P_f(t, T | x_f), P_f = A_f e^{-B_f x_f}: the foreign bond of the asset's currency
        const uint32_t a = min(extra, 1u);
#pragma unroll
        for (int i = 0; i < PPT; ++i) term[i] = c * pick4<R, PPT>(S, a, i) * (rec[3] * fastExp(-rec[1] * xfOf(a, i)));
        break;
      }
      case kForeignOption: {  // Black on S P_f(t, T | x_f) / P(t, T | x)
        const uint32_t a = min(extra, 1u);
        const R p3 = rec[7];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
          const R b0 = rec[3] * fastExp(nB * x[i]);
          const R q = rec[5] * fastExp(-rec[1] * xfOf(a, i));
          term[i] = c * black(pick4<R, PPT>(S, a, i) * q / b0, rec[6], fabs(p3), b0, p3 > R(0));
        }
        break;
      }
      default:
        if constexpr (!kLean) switch (kind) {  // the AMC and probe terms (absent from lean launches)
        case kBermExercise:
          if constexpr (kGiven) break;
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            const R v = c * (rec[3] * fastExp(nB * x[i]));
            if (manyBerm || bm == 0) ev[0][i] += v;  // with many Bermudans, one running value: its policy follows
            else if (bm == 1) ev[1][i] += v;
            else if (bm == 2) ev[2][i] += v;
            else ev[3][i] += v;
          }
          break;
        case kBermAnnuity:
#pragma unroll
          for (int i = 0; i < PPT; ++i) annS[i] += c * (rec[3] * fastExp(nB * x[i]));
          break;
        case kBermCoterm:
#pragma unroll
          for (int i = 0; i < PPT; ++i) fltS[i] += c * (rec[3] * fastExp(nB * x[i]));
          break;
        case kBermExt:
          break;  // read with its policy or continuation record
        case kBermDecide: {
          if constexpr (kGiven) {
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
              annS[i] = R(0), fltS[i] = R(0);
              if (act[i] && A.exIndex[static_cast<size_t>(bm) * nP + pth[i]] == static_cast<int>(extra))
                exS[(bm * PPT + i) * kTile + tid] = static_cast<signed char>(extra);
            }
            break;
          }
          R e1[8], e2[8];
          const bool twoD = twoRegressors(table, u, d1.x, e1, e2);
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            const R e = manyBerm ? ev[0][i] : pick4<R, PPT>(ev, bm, i);
            if (manyBerm) ev[0][i] = R(0);
            const R cont = twoD ? amcPoly2(rec, e1, e2, x[i], swapRate(fltS[i], annS[i])) : amcPoly(rec, x[i]);
            annS[i] = R(0), fltS[i] = R(0);
            if (kSink) {
              if (act[i]) A.sinkEx[static_cast<size_t>(A.sinkRowOfBermudan[bm] + extra) * nP + pth[i]] = e;
            } else if (exOf(bm, i) < R(0)) {
              // the exact-decision check: the rule's margins are e (against 0) and e - cont
              if (act[i] && (fabs(e) <= guardJ || fabs(e - cont) <= guardJ)) flagPath(A.flags, pth[i]);
              if (e > R(0) && e > cont) {
                const R v = static_cast<R>(extra);
                if (manyBerm) exS[(bm * PPT + i) * kTile + tid] = static_cast<signed char>(extra);
                else if (bm == 0) ex[0][i] = v;
                else if (bm == 1) ex[1][i] = v;
                else if (bm == 2) ex[2][i] = v;
                else ex[3][i] = v;
              }
            }
          }
          break;
        }
        case kBermContinue: {
          R e1[8], e2[8];
          const bool twoD = twoRegressors(table, u, d1.x, e1, e2);
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            const R cont = twoD ? amcPoly2(rec, e1, e2, x[i], swapRate(fltS[i], annS[i])) : amcPoly(rec, x[i]);
            annS[i] = R(0), fltS[i] = R(0);
            if (exOf(bm, i) < R(0)) term[i] = rec[1] * fmax(cont, R(0));
          }
          break;
        }
        case kBermBond:
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            const R e = exOf(bm, i);
            if (e >= R(0) && e <= static_cast<R>(extra)) term[i] = c * (rec[3] * fastExp(nB * x[i]));
          }
          break;
        case kProbe: {
          const uint32_t what = slot & 15u, ix = min(slot >> 4u, 3u), ic = min(ix, 1u);
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            R q;
            switch (what) {
              case 0: q = x[i]; break;
              case 1: q = D[i]; break;
              case 2: q = pick4<R, PPT>(S, ix, i); break;
              case 3: q = ix < cb.nA ? cube(cb.fLnS + ix, j, i) : R(0); break;
              case 4: q = ic < cb.nC ? cube(cb.fY + ic, j, i) : R(0); break;
              case 5: q = ic < cb.nC ? cube(cb.fQ + ic, j, i) : R(1); break;
              case 6: q = D[i] * pick4<R, PPT>(S, ix, i); break;
              default: q = D[i] * (rec[3] * fastExp(nB * x[i]));
            }
            if (!kSink && act[i]) expo[static_cast<size_t>(static_cast<uint32_t>(rec[5])) * nP + pth[i]] = q + c;
          }
          break;
        }
        default:  // kBermFloat
#pragma unroll
          for (int i = 0; i < PPT; ++i) {
            const R e = exOf(bm, i);
            if (e >= R(0) && e <= static_cast<R>(extra)) term[i] = (c * fix(slot, i) + rec[5]) * (rec[3] * fastExp(nB * x[i]));
          }
        }
    }
    if (kPerTrade && A.nTr > 0) {
#pragma unroll
      for (int i = 0; i < PPT; ++i) vt(grp, i) += term[i];
    } else {
#pragma unroll
      for (int i = 0; i < PPT; ++i) value[i] = kLean ? value[i] + term[i] : addRn(value[i], term[i]);
    }
  }
  for (uint32_t u = d1.x; u < d1.y; ++u) {  // fixings, after every use of the previous fixing
    const R4 r = ld4(table + 4 * u);
    const uint32_t slot = asUint(r.w);
#pragma unroll
    for (int i = 0; i < PPT; ++i) fix(slot, i) = (r.x * termExp(r.y, x[i]) - R(1)) * r.z;
  }
  for (uint32_t g = 0; g < nTr; ++g)
#pragma unroll
    for (int i = 0; i < PPT; ++i) value[i] += vt(g, i);
}

// Resident CTAs per SM the lean variants are compiled for (register budget 65536 / (128 x blocks)).  The
// shared-memory state of a netting set with many swap slots allows 6 CTAs of 2-path threads; netting sets
// with little state (kSmallState: at most kSmallStateWords words per path) fit 8, and their variant is
// compiled for 8 (64 registers).
template <int PPT, bool kLean, bool kSmallState = false>
constexpr int revalueMinBlocks() {
  return !kLean ? 1 : PPT == 1 ? 8 : PPT == 2 ? (kSmallState ? 8 : 6) : (kSmallState ? 4 : 3);
}

// Each thread owns PPT paths (p, p + kTile, ...): every term record, kind decode, date descriptor and
// statistics reduction is shared by PPT paths, and their independent exponentials keep the SFU busy.
// kCash: every netting set of the launch has a cash CSA whose margin calls look back at most one date and writes
// none of the optional value, exposure, collateral or change rows, so the collateral code is that case alone (no
// securities price, no shared-memory ring) and the optional rows are compiled out.
template <typename R, int PPT, bool kPerTrade, bool kSink, bool kLean, bool kSmallState = false, bool kCash = false>
__global__ void __launch_bounds__(kTile, (revalueMinBlocks<PPT, kLean, kSmallState>())) revalueKernel(const CubeArgs<R> cb, const NsArgs<R>* __restrict__ nsArgs,
                                                        uint32_t numNs) {
  extern __shared__ __align__(16) unsigned char smemRaw[];
  __shared__ NsArgs<R> sA;
  R* vtBuf = reinterpret_cast<R*>(smemRaw);                        // [16][PPT][kTile] per-trade values
  R* state = vtBuf + (kPerTrade ? kMaxTradeGroups * PPT * kTile : 0);  // fixings [nSlots][PPT][kTile] | ring

  const uint32_t n = blockIdx.x % numNs, tile = blockIdx.x / numNs;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) sA = nsArgs[n];
  __syncthreads();
  const NsArgs<R>& A = sA;  // read from shared memory: no global reloads after the stores below
  const uint4* __restrict__ dates = reinterpret_cast<const uint4*>(A.dates);
  const R* __restrict__ table = A.table;
  R* __restrict__ expo = A.expo;
  const uint32_t nP = cb.nP, nT = cb.nT;
  // Lean launches hold only plans with the netting set's 8 statistics per date (no per-trade ones).
  const uint32_t nSlots = A.nSlots, ringLen = kCash ? 2u : A.ring, nS = kLean ? static_cast<uint32_t>(kStatsPerDate) : A.nS;
  const uint32_t ctype = kCash ? 0u : A.ctype;
  const bool hasCsa = kCash || A.hasCsa != 0, usesAssets = A.usesAssets != 0;
  R* __restrict__ const rowEP = expo + static_cast<size_t>(A.rowEP) * nP;
  const bool moreRows = !kCash && (A.rowDV != kNoRow || A.rowE != kNoRow || A.rowV != kNoRow || A.rowC != kNoRow);
  uint32_t pth[PPT], pp[PPT];
  bool act[PPT];
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    pth[i] = tile * (kTile * PPT) + tid * PPT + i;  // a thread's paths are adjacent
    act[i] = pth[i] < nP;
    // Threads past the last path read valid paths and contribute nothing: the last PPT paths when nP is a
    // multiple of PPT (an aligned group, read as one vector), else the last path.
    pp[i] = act[i] ? pth[i] : nP % PPT == 0 ? nP - PPT + i : nP - 1;
  }
  auto fix = [&](uint32_t slot, int i) -> R& { return state[(slot * PPT + i) * kTile + tid]; };
  auto ring = [&](uint32_t r, int i) -> R& { return state[((nSlots + r) * PPT + i) * kTile + tid]; };
  // More than 4 Bermudans (non-lean launches only): each path's exercise index of Bermudan b is a byte of shared
  // memory after the fixings and the margin ring, [b][PPT][kTile], -1 while not exercised.
  const bool manyBerm = !kLean && A.manyBerm != 0;
  signed char* exS = reinterpret_cast<signed char*>(
      state + static_cast<size_t>(nSlots + (hasCsa ? ringLen * (ctype != 0 ? 2u : 1u) : 0u)) * PPT * kTile);
  if (manyBerm)
    for (uint32_t b = 0; b < A.nBerm; ++b)
#pragma unroll
      for (int i = 0; i < PPT; ++i) exS[(b * PPT + i) * kTile + tid] = -1;
  auto vt = [&](uint32_t g, int i) -> R& { return vtBuf[(g * PPT + i) * kTile + tid]; };
  for (uint32_t s = 0; s < nSlots; ++s)
#pragma unroll
    for (int i = 0; i < PPT; ++i) fix(s, i) = R(0);
  const uint32_t nTr = kPerTrade ? min(A.nTr, static_cast<uint32_t>(kMaxTradeGroups)) : 0u;
  const uint32_t fQ = A.cpty < cb.nC ? cb.fQ + A.cpty : 0xFFFFFFFFu;
  // Factor loads: per path a base pointer, per date an offset j * nP, per field a stride nT * nP.
  const size_t fieldStride = static_cast<size_t>(nT) * nP;
  const R* cubeP[PPT];
#pragma unroll
  for (int i = 0; i < PPT; ++i) cubeP[i] = cb.data + pp[i];
  auto cube = [&](uint32_t field, uint32_t j, int i) { return cubeP[i][field * fieldStride + static_cast<size_t>(j) * nP]; };

  R held[PPT], prevDE[PPT], prevQ[PPT], prevRV[PPT], ex[4][PPT], noXf[2][PPT];  // noXf: the terms read x_f from the cube
#pragma unroll
  for (int i = 0; i < PPT; ++i) noXf[0][i] = noXf[1][i] = R(0);
  // The exercise index (-1: not exercised) of Bermudan b on the thread's path i.
  auto exOf = [&](uint32_t b, int i) -> R {
    return manyBerm ? static_cast<R>(exS[(b * PPT + i) * kTile + tid]) : pick4<R, PPT>(ex, b, i);
  };
  // Look-back of at most one date (the margin-call dates t - MPR sit on the grid): the previous date's value
  // and collateral price in registers instead of the shared-memory ring.
  const bool shortLook = kCash || ringLen <= 2;
  R vPrev[PPT], pPrev[PPT];
#pragma unroll
  for (int i = 0; i < PPT; ++i) vPrev[i] = R(0), pPrev[i] = R(1);
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    held[i] = R(0), prevDE[i] = R(0), prevQ[i] = R(1), prevRV[i] = R(0);
#pragma unroll
    for (int b = 0; b < 4; ++b) ex[b][i] = R(-1);  // exercise index of each Bermudan, -1 if not exercised
  }
  uint32_t ringPos = 0;

  // Software pipeline: the factors and the date descriptor of date j + 1 load while date j computes.
  R nx[PPT], nD[PPT], nQ[PPT], nS4[4][PPT];
  const size_t qOff = fQ != 0xFFFFFFFFu ? fQ * fieldStride : 0, sOff = static_cast<size_t>(cb.fS) * fieldStride;
  // With nP a multiple of PPT a thread's paths are all live or all past the end, and their factors are one
  // vector access per field (past the end: the last PPT paths).
  const bool vecPaths = PPT > 1 && nP % PPT == 0;
  auto loadFactors = [&](uint32_t j) {
    const size_t off = static_cast<size_t>(j) * nP;
    if (vecPaths) {
      const R* c = cubeP[0] + off;
      ldPaths<R, PPT>(c, nx);
      ldPaths<R, PPT>(c + fieldStride, nD);
      if (fQ != 0xFFFFFFFFu) {
        ldPaths<R, PPT>(c + qOff, nQ);
      } else {
#pragma unroll
        for (int i = 0; i < PPT; ++i) nQ[i] = R(1);
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        if (usesAssets && static_cast<uint32_t>(a) < cb.nA) {
          ldPaths<R, PPT>(c + sOff + a * fieldStride, nS4[a]);
        } else {
#pragma unroll
          for (int i = 0; i < PPT; ++i) nS4[a][i] = R(0);
        }
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      const R* c = cubeP[i] + off;
      nx[i] = __ldg(c), nD[i] = __ldg(c + fieldStride), nQ[i] = fQ != 0xFFFFFFFFu ? __ldg(c + qOff) : R(1);
#pragma unroll
      for (int a = 0; a < 4; ++a)
        nS4[a][i] = usesAssets && static_cast<uint32_t>(a) < cb.nA ? __ldg(c + sOff + a * fieldStride) : R(0);
    }
  };
  loadFactors(0);
  uint4 nd0 = __ldg(dates), nd1 = __ldg(dates + 1);
  // The block of the date after next is prefetched one date ahead of use.
  uint32_t fBeg = nT > 1 ? __ldg(A.dates + 8) : 0u, fEnd = nT > 1 ? __ldg(A.dates + 13) : 0u;
  prefetchDate<R>(nd0.x, nd1.y, table, tid);

  for (uint32_t j = 0; j < nT; ++j) {
    R x[PPT], D[PPT], Q[PPT], S[4][PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      x[i] = nx[i], D[i] = nD[i], Q[i] = nQ[i];
#pragma unroll
      for (int a = 0; a < 4; ++a) S[a][i] = nS4[a][i];
    }
    const uint4 d0 = nd0, d1 = nd1;
    const R guardJ = A.flags ? A.guard[j] : R(-1);  // < 0: no check
    if (j + 1 < nT) {
      loadFactors(j + 1);
      nd0 = __ldg(dates + 2 * (j + 1)), nd1 = __ldg(dates + 2 * (j + 1) + 1);
      prefetchDate<R>(fBeg, fEnd, table, tid);
      if (j + 2 < nT) {
        fBeg = __ldg(A.dates + 8 * (j + 2)), fEnd = __ldg(A.dates + 8 * (j + 2) + 5);
      }
    }
    if (kSink && n == 0)
#pragma unroll
      for (int i = 0; i < PPT; ++i)
        if (act[i]) {
          A.sinkX[static_cast<size_t>(j) * nP + pth[i]] = x[i];
          A.sinkD[static_cast<size_t>(j) * nP + pth[i]] = D[i];
        }

    R value[PPT];
    revalueDate<R, PPT, kPerTrade, kSink, kLean, false>(A, cb, cubeP, d0, d1, j, tid, pth, act, x, D, S, noXf, guardJ, state, vtBuf, exS,
                                                        manyBerm, ex, value);
    if (kSink) continue;

    // ---- CSA: collateral called on the value at t - MPR (collateral.cpp:10-47) ----
    R e[PPT], ep[PPT], en[PPT];
    const uint32_t callJ = d1.z, rs = d1.w;
    // Ring slots without a modulo: ringPos = j mod ringLen, advanced by one per date; the margin-call date
    // lies j - callJ < ringLen dates back.
    const uint32_t lag = j - callJ, callPos = ringPos >= lag ? ringPos - lag : ringPos + ringLen - lag;
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      R collateral = R(0);
      if (hasCsa) {
        R price = R(1);
        if (ctype == 1) price = A.steps[static_cast<size_t>(j) * A.stepStride + 22] * rexp(-A.steps[static_cast<size_t>(j) * A.stepStride + 23] * x[i]);
        else if (ctype == 2) price = pick4<R, PPT>(S, min(A.casset, 3u), i);
        R vc, pc = price;
        if (shortLook) {
          vc = callJ != j ? vPrev[i] : value[i];
          if (callJ != j) pc = pPrev[i];
          vPrev[i] = value[i], pPrev[i] = price;
        } else {
          ring(ringPos, i) = value[i];
          if (ctype != 0) ring(ringLen + ringPos, i) = price;
          vc = callJ != j ? ring(callPos, i) : value[i];
          if (ctype != 0 && callJ != j) pc = ring(ringLen + callPos, i);
        }
        R required = R(0);
        if (vc > A.hc) required += vc - A.hc;
        if (A.hb >= R(0) && -vc > A.hb) required -= -vc - A.hb;
        // The call rule |required - held| >= MTA; the exact-decision check flags the path when its margin
        // | |required - held| - MTA | is within the date's guard.
        if (ctype == 0) {  // cash: one unit is worth one, no division
          const R gap = fabs(required - held[i]);
          if (j > 0 && act[i] && fabs(gap - A.mta) <= guardJ) flagPath(A.flags, pth[i]);
          if (j == 0 || gap >= A.mta) held[i] = required;
          collateral = held[i] + A.ia;
        } else {
          const R keep = A.keepHaircut;
          const R gap = fabs(required - held[i] * keep * pc);
          if (j > 0 && act[i] && fabs(gap - A.mta) <= guardJ) flagPath(A.flags, pth[i]);
          if (j == 0 || gap >= A.mta) held[i] = required / (keep * pc);
          collateral = held[i] * price + A.ia;
        }
      }
      e[i] = value[i] - collateral, ep[i] = fmax(e[i], R(0)), en[i] = fmin(e[i], R(0));
      if (act[i] && rs > 0) {
        const size_t k = rs - 1, pi = pth[i], at = k * nP + pi;
        if (!vecPaths) rowEP[at] = ep[i];
        if (moreRows) {
          if (A.rowDV != kNoRow) expo[(A.rowDV + k) * nP + pi] = rs == 1 ? R(0) : fabs(value[i] - prevRV[i]);
          if (A.rowE != kNoRow) expo[(A.rowE + k) * nP + pi] = e[i];
          if (A.rowV != kNoRow) expo[(A.rowV + k) * nP + pi] = value[i];
          if (A.rowC != kNoRow) expo[(A.rowC + k) * nP + pi] = collateral;
        }
        if (!kLean && A.rowGross != kNoRow) {
          R gross = R(0);
          for (uint32_t g = 0; g < nTr; ++g) gross += fmax(vt(g, i), R(0));
          expo[(A.rowGross + k) * nP + pi] = gross;
        }
        if (!kLean && A.rowTrades != kNoRow)
          for (uint32_t g = 0; g < nTr; ++g) expo[(A.rowTrades + g * A.nR + k) * nP + pi] = vt(g, i);
      }
      if (!kLean && !kSink && rs > 0 && A.imState && act[i]) {  // the start of this path's inner paths
        R* st = A.imState + static_cast<size_t>(rs - 1) * A.imWords * nP + pth[i];
        st[0] = value[i];
#pragma unroll
        for (int b = 0; b < 4; ++b) st[static_cast<size_t>(1 + b) * nP] = pick4<R, PPT>(ex, b, i);
        for (uint32_t q = 0; q < nSlots; ++q) st[static_cast<size_t>(5 + q) * nP] = fix(q, i);
      }
      if (!kLean && act[i] && A.rowEx != kNoRow)
        for (uint32_t b = 0; b < (manyBerm ? A.nBerm : min(A.nBerm, 4u)); ++b) {
          const R v = exOf(b, i);
          expo[(A.rowEx + b) * static_cast<size_t>(nP) + pth[i]] = v < R(0) ? R(-1) : v;
        }
    }
    if (vecPaths && act[0] && rs > 0) stPaths<R, PPT>(rowEP + static_cast<size_t>(rs - 1) * nP + pth[0], ep);
    R cvaInc[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      cvaInc[i] = R(0);
      if (rs > 0) {
        prevRV[i] = value[i];
        const R de = D[i] * ep[i];
        if (j > 0) cvaInc[i] = R(0.5) * (prevDE[i] + de) * (prevQ[i] - Q[i]);
        prevDE[i] = de;
        prevQ[i] = Q[i];
      }
    }

    // ---- statistics of this date: the netting set's 8, then kTradeStats per trade, summed per warp over its
    // 32 PPT adjacent paths as a binary tree (a thread's adjacent paths first, then the lanes) into one partial
    // per warp: no block barrier.  The reduce kernel completes each 128-path group's tree from 4, 2 or 1 warp
    // partials, so the group sums and their bits do not depend on the tile shape ----
    const uint32_t unit = tile * kWarps + warp;
    const bool unitLive = unit * (32u * PPT) < nP;
    for (uint32_t q = 0; q < nS; q += 8) {
      R w8[PPT][8];
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
#pragma unroll
        for (int c = 0; c < 8; ++c) w8[i][c] = R(0);
        if (act[i]) {
          if (q == 0) {
            w8[i][0] = e[i], w8[i][1] = ep[i], w8[i][2] = en[i], w8[i][3] = D[i] * ep[i], w8[i][4] = D[i] * en[i];
            w8[i][5] = cvaInc[i], w8[i][6] = Q[i], w8[i][7] = D[i];
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint32_t k = q + c - kStatsPerDate, g = k / kTradeStats;
              if (q + c < nS && g < nTr) w8[i][c] = tradeStat<R>(k % kTradeStats, vt(g, i), value[i], D[i]);
            }
          }
        }
      }
      R v8[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if constexpr (PPT == 1) v8[c] = w8[0][c];
        else if constexpr (PPT == 2) v8[c] = w8[0][c] + w8[1][c];
        else v8[c] = (w8[0][c] + w8[1][c]) + (w8[2][c] + w8[3][c]);
      }
      const R s = warpReduceScatter8(v8, lane);
      const uint32_t c = statSlotOfLane(lane);
      if (lane < 8u && unitLive && q + c < nS) A.partials[(static_cast<size_t>(unit) * nT + j) * nS + q + c] = s;
    }
    ringPos = ringPos + 1 == ringLen ? 0u : ringPos + 1;
  }
}

// ---------------------------------------------------------------------------------------------
// The same revaluation split over the dates.  revalueKernel walks every date of a (path tile, netting set) in one CTA: a
// launch of few paths, or of netting sets of very different sizes, leaves most of the GPU idle or waiting for the
// largest.  What is serial in the dates is little: a fixing needs its own date's short rate only, an exercise decision
// its own date's state and whether an earlier one was taken, the collateral one comparison per date.  So
//   decideKernel  per (paths, Bermudan): the exercise date chosen, from the exercise dates' records alone;
//   valueKernel   per (path tile, netting set, run of dates): the netted values, into A.vals [date][path];
//   settleKernel  per (32 paths, netting set): the collateral walk over the dates by one warp, then rows and statistics of
//                 the dates by all eight.
// Same arithmetic per date as revalueKernel (revalueDate), same statistics tree: the same results.
// Revaluation before and after (us): 2,000 paths x 121 dates of 3 trades 146 and 20, 10,000 x 61 of 20 swaps 203 and 31, 12
// netting sets of 119 trades at 33,333 paths x 169 dates 1,497 and 1,077, 24 + 24 netting sets with 40
// Bermudans among 800 trades at 65,536 x 241 66,061 and 28,457.
// kSink: the AMC state pass, which keeps the exercise values (A.sinkEx) instead of deciding on them.
template <typename R, bool kSink>
__global__ void __launch_bounds__(kTile) decideKernel(const CubeArgs<R> cb, const NsArgs<R>* __restrict__ nsArgs,
                                                      const DecideJob* __restrict__ jobs, const R* __restrict__ table) {
  const DecideJob J = jobs[blockIdx.y];
  const NsArgs<R>& A = nsArgs[J.ns];
  const uint32_t nP = cb.nP, p = blockIdx.x * kTile + threadIdx.x;
  if (p >= nP) return;
  const bool many = A.manyBerm != 0;
  R x = R(0), ev = R(0), ann = R(0), flt = R(0), guardJ = R(-1), ex = R(-1);
  for (uint32_t u = J.begin; u < J.end; u += 2) {
    R rec[8];
    loadTerm(table + 4 * u, rec);
    const uint32_t code = asUint(rec[0]), kind = code & 15u;
    if (kind == kBond) {  // the records of date rec[1] follow
      const uint32_t j = asUint(rec[1]);
      x = __ldg(cb.data + static_cast<size_t>(j) * nP + p);
      ev = ann = flt = R(0);
      guardJ = A.flags ? A.guard[j] : R(-1);
      continue;
    }
    if (kind == kBermDecide) {
      if constexpr (kSink) {
        A.sinkEx[static_cast<size_t>(A.sinkRowOfBermudan[J.berm] + (code >> 12u)) * nP + p] = ev;
        if (many) ev = R(0);
        continue;
      }
      R e1[8], e2[8];
      const bool twoD = twoRegressors(table, u, J.end, e1, e2);
      const R cont = twoD ? amcPoly2(rec, e1, e2, x, swapRate(flt, ann)) : amcPoly(rec, x);
      ann = flt = R(0);
      if (ex < R(0)) {
        if (fabs(ev) <= guardJ || fabs(ev - cont) <= guardJ) flagPath(A.flags, p);
        if (ev > R(0) && ev > cont) ex = static_cast<R>(code >> 12u);
      }
      if (many) ev = R(0);
    } else if (kind != kBermExt) {
      const R v = rec[2] * (rec[3] * fastExp(-rec[4] * x));
      if (kind == kBermExercise) ev += v;
      else if (kind == kBermAnnuity) ann += v;
      else flt += v;
    }
  }
  if constexpr (kSink) return;
  A.exIndex[static_cast<size_t>(J.berm) * nP + p] = static_cast<signed char>(ex);
  if (A.rowEx != kNoRow && (many || J.berm < 4u)) A.expo[(A.rowEx + J.berm) * static_cast<size_t>(nP) + p] = ex;
}

template <typename R, int PPT, bool kLean>
__global__ void __launch_bounds__(kTile, (sizeof(R) == 8 ? 4 : kLean ? 8 : 6)) valueKernel(
    const CubeArgs<R> cb, const NsArgs<R>* __restrict__ nsArgs, const ValueItem* __restrict__ items, const uint2* __restrict__ pre,
    const uint8_t* __restrict__ exFirst, uint32_t pathBegin, uint32_t slabPaths) {
  extern __shared__ __align__(16) unsigned char smemRaw[];
  __shared__ NsArgs<R> sA;
  R* state = reinterpret_cast<R*>(smemRaw);
  const ValueItem I = items[blockIdx.y];
  const uint32_t tid = threadIdx.x;
  if (tid < sizeof(NsArgs<R>) / 4) reinterpret_cast<uint32_t*>(&sA)[tid] = reinterpret_cast<const uint32_t*>(nsArgs + I.ns)[tid];
  __syncthreads();
  const NsArgs<R>& A = sA;
  const uint32_t nP = cb.nP, nT = cb.nT, nSlots = A.nSlots, last = min(pathBegin + slabPaths, nP);
  uint32_t pth[PPT], pp[PPT];
  bool act[PPT];
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    pth[i] = pathBegin + (blockIdx.x * kTile + tid) * PPT + i;
    act[i] = pth[i] < last;
    pp[i] = act[i] ? pth[i] : nP % PPT == 0 ? nP - PPT + i : nP - 1;
  }
  const size_t fieldStride = static_cast<size_t>(nT) * nP;
  const R* cubeP[PPT];
#pragma unroll
  for (int i = 0; i < PPT; ++i) cubeP[i] = cb.data + pp[i];
  const bool vecPaths = PPT > 1 && nP % PPT == 0;
  auto load = [&](size_t at, R (&v)[PPT]) {
    if (vecPaths) {
      ldPaths<R, PPT>(cubeP[0] + at, v);
    } else {
#pragma unroll
      for (int i = 0; i < PPT; ++i) v[i] = __ldg(cubeP[i] + at);
    }
  };
  // The fixings that the run's first dates read, each from its own date's short rate; fixings never set are zero.
  for (uint32_t q = 0; q < nSlots; ++q)
#pragma unroll
    for (int i = 0; i < PPT; ++i) state[(q * PPT + i) * kTile + tid] = R(0);
  for (uint32_t q = I.preBegin; q < I.preEnd; ++q) {
    const uint2 f = __ldg(pre + q);  // fixing record, date
    const auto r = ld4(A.table + 4 * static_cast<size_t>(f.x));
    R x[PPT];
    load(static_cast<size_t>(f.y & ~kGenericFixing) * nP, x);
    if (f.y & kGenericFixing) {  // (code, slot, c, A), (B, ...)
      const R B = __ldg(A.table + 4 * static_cast<size_t>(f.x) + 4);
#pragma unroll
      for (int i = 0; i < PPT; ++i) state[(asUint(r.y) * PPT + i) * kTile + tid] = genericFixing(r.z, r.w, B, x[i]);
      continue;
    }
#pragma unroll
    for (int i = 0; i < PPT; ++i) state[(asUint(r.w) * PPT + i) * kTile + tid] = (r.x * termExp(r.y, x[i]) - R(1)) * r.z;
  }
  signed char* exS = reinterpret_cast<signed char*>(state + static_cast<size_t>(nSlots) * PPT * kTile);
  if constexpr (!kLean)
    for (uint32_t b = 0; b < A.nBerm; ++b) {
      const int e0 = exFirst[I.exAt + b];  // exercises decided before the run
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int e = A.exIndex[static_cast<size_t>(b) * nP + pp[i]];
        exS[(b * PPT + i) * kTile + tid] = static_cast<signed char>(e < e0 ? e : -1);
      }
    }
  const uint4* __restrict__ dates = reinterpret_cast<const uint4*>(A.dates);
  const size_t sOff = static_cast<size_t>(cb.fS) * fieldStride, fOff = static_cast<size_t>(cb.fXf) * fieldStride;
  R nx[PPT], nD[PPT], nS4[4][PPT], nXf[2][PPT];
  auto loadFactors = [&](uint32_t j) {
    const size_t off = static_cast<size_t>(j) * nP;
    load(off, nx);
    if constexpr (!kLean) load(off + fieldStride, nD);  // probes
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if (A.usesAssets && static_cast<uint32_t>(a) < cb.nA) load(off + sOff + a * fieldStride, nS4[a]);
#pragma unroll
    for (int a = 0; a < 2; ++a)
      if (A.usesForeign && static_cast<uint32_t>(a) < cb.nF) load(off + fOff + a * fieldStride, nXf[a]);
  };
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    nD[i] = R(0);
#pragma unroll
    for (int a = 0; a < 4; ++a) nS4[a][i] = R(0);
    nXf[0][i] = nXf[1][i] = R(0);
  }
  loadFactors(I.j0);
  uint4 nd0 = __ldg(dates + 2 * I.j0), nd1 = __ldg(dates + 2 * I.j0 + 1);
  for (uint32_t j = I.j0; j < I.j1; ++j) {
    R x[PPT], D[PPT], S[4][PPT], xf[2][PPT], ex[4][PPT], value[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      x[i] = nx[i], D[i] = nD[i], xf[0][i] = nXf[0][i], xf[1][i] = nXf[1][i];
#pragma unroll
      for (int a = 0; a < 4; ++a) S[a][i] = nS4[a][i], ex[a][i] = R(-1);
    }
    const uint4 d0 = nd0, d1 = nd1;
    if (j + 1 < I.j1) {
      loadFactors(j + 1);
      nd0 = __ldg(dates + 2 * (j + 1)), nd1 = __ldg(dates + 2 * (j + 1) + 1);
      prefetchDate<R>(nd0.x, nd1.y, A.table, tid);
    }
    revalueDate<R, PPT, false, false, kLean, true>(A, cb, cubeP, d0, d1, j, tid, pth, act, x, D, S, xf, R(-1), state, nullptr, exS, true, ex,
                                                   value);
    R* dst = A.vals + static_cast<size_t>(j) * slabPaths + (pth[0] - pathBegin);
    if (vecPaths && slabPaths % PPT == 0) {
      if (act[0]) stPaths<R, PPT>(dst, value);
    } else {
#pragma unroll
      for (int i = 0; i < PPT; ++i)
        if (act[i]) dst[i] = value[i];
    }
    if (!kLean && A.imState && d1.w > 0) {  // the start of the paths' inner paths
#pragma unroll
      for (int i = 0; i < PPT; ++i)
        if (act[i]) {
          R* st = A.imState + static_cast<size_t>(d1.w - 1) * A.imWords * nP + pth[i];
          st[0] = value[i];
#pragma unroll
          for (uint32_t b = 0; b < 4; ++b)
            st[static_cast<size_t>(1 + b) * nP] = b < A.nBerm ? static_cast<R>(exS[(b * PPT + i) * kTile + tid]) : R(-1);
          for (uint32_t q = 0; q < nSlots; ++q) st[static_cast<size_t>(5 + q) * nP] = state[(q * PPT + i) * kTile + tid];
        }
    }
  }
}

constexpr uint32_t kSettleThreads = 256, kSettleWarps = kSettleThreads / 32;

// What a CTA of settleKernel holds of kDates dates and its 32 V paths; rows padded so that a column's walk over the paths
// by one thread per date meets no bank conflict.
template <typename R, int V>
struct SettleSmem {
  static constexpr uint32_t kDates = sizeof(R) * V == 4 ? 64 : 32, kRow = 32 * V + 1;
  R v[kDates][kRow];  // values, then exposures e
  R c[kDates][kRow];  // required collateral, then collateral, then D max(e, 0); the sums' parts with d
  R d[kDates][kRow];  // deflators
  R q[kDates][kRow];  // the counterparty's survival
  R lastDE[32 * V], lastQ[32 * V];  // D max(e, 0) and Q of the last reporting date before them
  uint32_t call[kDates], slot[kDates], prev[kDates];  // margin-call date, reporting slot, previous reporting date (kNoRow: none)
};

// V: paths per lane, 32 apart (a row's address and loop are shared by them).
template <typename R, int V>
__global__ void __launch_bounds__(kSettleThreads) settleKernel(const CubeArgs<R> cb, const NsArgs<R>* __restrict__ nsArgs, uint32_t pathBegin,
                                                               uint32_t slabPaths) {
  extern __shared__ __align__(16) unsigned char smemRaw[];
  __shared__ NsArgs<R> sA;
  SettleSmem<R, V>& s = *reinterpret_cast<SettleSmem<R, V>*>(smemRaw);
  constexpr uint32_t kDates = SettleSmem<R, V>::kDates, kGroups = kSettleThreads / kDates, kPer = 32 * V / kGroups;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid < sizeof(NsArgs<R>) / 4) reinterpret_cast<uint32_t*>(&sA)[tid] = reinterpret_cast<const uint32_t*>(nsArgs + blockIdx.y)[tid];
  if (tid < 32 * V) s.lastDE[tid] = R(0), s.lastQ[tid] = R(1);
  __syncthreads();
  const NsArgs<R>& A = sA;
  const uint32_t nP = cb.nP, nT = cb.nT, first = pathBegin + blockIdx.x * 32u * V;
  const uint32_t live = min(32u * V, min(pathBegin + slabPaths, nP) - first);  // the CTA's paths
  const bool hasCsa = A.hasCsa != 0, hasQ = A.cpty < cb.nC;
  const uint32_t unit = first / (32u * V);
  uint32_t at[V];  // the lane's paths from `first`; past the last path they repeat it and write nothing
#pragma unroll
  for (int i = 0; i < V; ++i) at[i] = min(lane + 32u * i, live - 1);
  const R* __restrict__ vals = A.vals + (first - pathBegin);
  const size_t fieldStride = static_cast<size_t>(nT) * nP;
  const R* __restrict__ cube = cb.data + first;
  const size_t qOff = hasQ ? (cb.fQ + A.cpty) * fieldStride : 0;
  R held[V];
#pragma unroll
  for (int i = 0; i < V; ++i) held[i] = R(0);
  uint32_t lastRep = kNoRow;
  for (uint32_t j0 = 0; j0 < nT; j0 += kDates) {
    const uint32_t n = min(kDates, nT - j0);
#pragma unroll 4
    for (uint32_t k = warp; k < n; k += kSettleWarps) {
      const R* pv = vals + static_cast<size_t>(j0 + k) * slabPaths;
      const R* pd = cube + fieldStride + static_cast<size_t>(j0 + k) * nP;
      const R* pq = cube + qOff + static_cast<size_t>(j0 + k) * nP;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        s.v[k][lane + 32 * i] = __ldg(pv + at[i]);
        s.d[k][lane + 32 * i] = __ldg(pd + at[i]);
        s.q[k][lane + 32 * i] = hasQ ? __ldg(pq + at[i]) : R(1);
      }
    }
    if (tid < n) {
      const uint2 w = __ldg(reinterpret_cast<const uint2*>(A.dates + 8 * static_cast<size_t>(j0 + tid) + 6));
      s.call[tid] = w.x, s.slot[tid] = w.y;
    }
    __syncthreads();
    if (tid < n) {
      uint32_t k = tid;
      while (k > 0 && s.slot[k - 1] == 0) --k;
      s.prev[tid] = k > 0 ? j0 + k - 1 : lastRep;
    }
    // ---- CSA: collateral called on the value at t - MPR (collateral.cpp:10-47) ----
    if (hasCsa) {
      for (uint32_t k = warp; k < n; k += kSettleWarps) {
        const uint32_t callJ = s.call[k];
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const R vc = callJ >= j0 ? s.v[callJ - j0][lane + 32 * i] : __ldg(vals + static_cast<size_t>(callJ) * slabPaths + at[i]);
          R required = R(0);
          if (vc > A.hc) required += vc - A.hc;
          if (A.hb >= R(0) && -vc > A.hb) required -= -vc - A.hb;
          s.c[k][lane + 32 * i] = required;
        }
      }
      __syncthreads();
      if (warp == 0) {  // the one serial step: the collateral held, date by date
        if (A.ctype == 0 && !A.flags) {  // cash: one unit is worth one, no division
          const R mta = A.mta, ia = A.ia;
#pragma unroll 8
          for (uint32_t k = 0; k < n; ++k)
#pragma unroll
            for (int i = 0; i < V; ++i) {
              const R required = s.c[k][lane + 32 * i];
              if (j0 + k == 0 || fabs(required - held[i]) >= mta) held[i] = required;
              s.c[k][lane + 32 * i] = held[i] + ia;
            }
        } else {
          auto price = [&](uint32_t j, uint32_t p) -> R {
            if (A.ctype == 1) {
              const R* st = A.steps + static_cast<size_t>(j) * A.stepStride;
              return st[22] * rexp(-st[23] * __ldg(cube + static_cast<size_t>(j) * nP + p));
            }
            return A.ctype == 2 ? __ldg(cube + (cb.fS + min(A.casset, 3u)) * fieldStride + static_cast<size_t>(j) * nP + p) : R(1);
          };
          for (uint32_t k = 0; k < n; ++k)
#pragma unroll
            for (int i = 0; i < V; ++i) {
              const uint32_t j = j0 + k, callJ = s.call[k];
              const R guardJ = A.flags ? A.guard[j] : R(-1);  // < 0: no check
              const R required = s.c[k][lane + 32 * i], pj = price(j, at[i]), pCall = callJ != j ? price(callJ, at[i]) : pj;
              const R gap = A.ctype == 0 ? fabs(required - held[i]) : fabs(required - held[i] * A.keepHaircut * pCall);
              if (j > 0 && lane + 32 * i < live && fabs(gap - A.mta) <= guardJ) flagPath(A.flags, first + lane + 32 * i);
              if (j == 0 || gap >= A.mta) held[i] = A.ctype == 0 ? required : required / (A.keepHaircut * pCall);
              s.c[k][lane + 32 * i] = held[i] * pj + A.ia;
            }
        }
      }
    }
    __syncthreads();
    // ---- exposures and the reporting dates' rows ----
    for (uint32_t k = warp; k < n; k += kSettleWarps) {
      const uint32_t rs = s.slot[k];
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const uint32_t col = lane + 32 * i;
        const R value = s.v[k][col], collateral = hasCsa ? s.c[k][col] : R(0), e = value - collateral, ep = fmax(e, R(0));
        s.v[k][col] = e;
        s.c[k][col] = mulRn(s.d[k][col], ep);
        if (rs > 0 && col < live) {
          const size_t row = static_cast<size_t>(rs - 1) * nP + first + col;
          A.expo[static_cast<size_t>(A.rowEP) * nP + row] = ep;
          if (A.moreRows) {
            if (A.rowDV != kNoRow) {
              const R before = s.prev[k] != kNoRow ? __ldg(vals + static_cast<size_t>(s.prev[k]) * slabPaths + col) : R(0);
              A.expo[static_cast<size_t>(A.rowDV) * nP + row] = rs == 1 ? R(0) : fabs(value - before);
            }
            if (A.rowE != kNoRow) A.expo[static_cast<size_t>(A.rowE) * nP + row] = e;
            if (A.rowV != kNoRow) A.expo[static_cast<size_t>(A.rowV) * nP + row] = value;
            if (A.rowC != kNoRow) A.expo[static_cast<size_t>(A.rowC) * nP + row] = collateral;
            if (A.rowGross != kNoRow) A.expo[static_cast<size_t>(A.rowGross) * nP + row] = R(0);  // no trade groups here
          }
        }
      }
    }
    __syncthreads();
    // ---- the 8 statistics of each date: a thread sums kPer adjacent paths of one date as a binary tree, then the groups
    // are added as one: revalueKernel's tree over the paths, and its roundings ----
    const uint32_t k = tid % kDates, g = tid / kDates;
    R sum[8];
    if (k < n) {
      const bool rep = s.slot[k] > 0 && j0 + k > 0;
      const uint32_t pk = s.prev[k];
      const bool inside = pk != kNoRow && pk >= j0;  // else the last reporting date before these, or none (DE 0, Q 1)
      const R* prevDE = inside ? s.c[pk - j0] : s.lastDE;
      const R* prevQ = inside ? s.q[pk - j0] : s.lastQ;
      R level[4][8];  // the sums of 1, 2, 4 paths that wait for their neighbour
#pragma unroll
      for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t i = g * kPer + u;
        R t[8] = {R(0), R(0), R(0), R(0), R(0), R(0), R(0), R(0)};
        if (i < live) {
          const R e = s.v[k][i], D = s.d[k][i], Q = s.q[k][i], ep = fmax(e, R(0)), en = fmin(e, R(0));
          t[0] = e, t[1] = ep, t[2] = en, t[3] = s.c[k][i], t[4] = mulRn(D, en), t[6] = Q, t[7] = D;
          if (rep) t[5] = mulRn(R(0.5) * (prevDE[i] + t[3]), prevQ[i] - Q);
        }
        uint32_t l = 0;
#pragma unroll
        for (uint32_t w = u; w & 1u; w >>= 1, ++l)
#pragma unroll
          for (int c = 0; c < 8; ++c) t[c] = level[l][c] + t[c];
#pragma unroll
        for (int c = 0; c < 8; ++c) level[l][c] = t[c];
        if (u + 1 == kPer)
#pragma unroll
          for (int c = 0; c < 8; ++c) sum[c] = t[c];
      }
    }
    // The last reporting date so far, for the next dates.
    uint32_t rep = n;
    while (rep > 0 && s.slot[rep - 1] == 0) --rep;
    const R de = rep > 0 && tid < 32 * V ? s.c[rep - 1][tid] : R(0), q = rep > 0 && tid < 32 * V ? s.q[rep - 1][tid] : R(0);
    __syncthreads();
    if (rep > 0 && tid < 32 * V) s.lastDE[tid] = de, s.lastQ[tid] = q;
    if (rep > 0) lastRep = j0 + rep - 1;
    R* part = &s.c[0][0];  // [kGroups][8][kDates + 1], over c and d
    static_assert(sizeof(R) * kGroups * 8 * (kDates + 1) <= sizeof(s.c) + sizeof(s.d), "the parts fit");
    if (k < n)
#pragma unroll
      for (int c = 0; c < 8; ++c) part[(g * 8 + c) * (kDates + 1) + k] = sum[c];
    __syncthreads();
    for (uint32_t o = tid; o < n * 8; o += kSettleThreads) {
      const R* mine = part + (o % 8) * (kDates + 1) + o / 8;
      auto of = [&](uint32_t h) { return mine[h * 8 * (kDates + 1)]; };
      R t = (of(0) + of(1)) + (of(2) + of(3));
      if constexpr (kGroups == 8) t = t + ((of(4) + of(5)) + (of(6) + of(7)));
      A.partials[(static_cast<size_t>(unit) * nT + j0 + o / 8) * A.nS + o % 8] = t;
    }
    if (A.nS > 8)
      for (uint32_t o = tid; o < n * (A.nS - 8); o += kSettleThreads)
        A.partials[(static_cast<size_t>(unit) * nT + j0 + o / (A.nS - 8)) * A.nS + 8 + o % (A.nS - 8)] = R(0);
    __syncthreads();  // before the next dates overwrite the shared memory
  }
}

// ---------------------------------------------------------------------------------------------
// Nested Monte Carlo for the conditional initial margin (the reference's innerStep / innerValue and the
// inner loop of simulatePath: fused_reference.cpp:108-196, 356-393).  The reference runs the nInner inner
// paths of an outer path one after the other inside the path's thread; here one warp takes one
// (reporting slot, outer path) and its lanes run inner paths lane, lane + 32, ... side by side: every lane of
// the warp steps the same dates, so the date's records are warp-uniform broadcasts, and the grid holds
// nR x nP warps instead of nP threads.

// One inner path's exact step to date jj on its own stream: the outer step's short rate and asset levels
// with the inner normals (the intensity enters no value and is not stepped).  Pairs past the normals the
// Cholesky rows and the integrated rate read stay zero; the Cholesky factor is zero there.
template <typename R>
__device__ __forceinline__ void innerStep(const ImArgs<R>& M, uint32_t jj, uint32_t stream, R sign, R& x, R (&lnS)[4],
                                          R (&S)[4]) {
  R z[8];
  const uint32_t pairs = M.nCorr / 2 + 1;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    z[2 * k] = z[2 * k + 1] = R(0);
    if (static_cast<uint32_t>(k) < pairs) {
      gauss2(stream, jj, static_cast<uint32_t>(k), z[2 * k], z[2 * k + 1]);
      z[2 * k] *= sign, z[2 * k + 1] *= sign;
    }
  }
  R w[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const R* row = M.model + 4 + i * kChol;
    const R d0 = __ldg(row) * z[0] + __ldg(row + 1) * z[1] + __ldg(row + 2) * z[2] + __ldg(row + 3) * z[3];
    const R d1 = __ldg(row + 4) * z[4] + __ldg(row + 5) * z[5] + __ldg(row + 6) * z[6] + __ldg(row + 7) * z[7];
    w[i] = d0 + d1;
  }
  R zc = R(0);  // the independent normal of the integrated rate, z[nCorr]
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (static_cast<uint32_t>(k) == M.nCorr) zc = z[k];
  const R* st = M.steps + static_cast<size_t>(jj) * kStepStride;
  const R integrated = x * __ldg(st + 5) + __ldg(st + 2) * w[0] + __ldg(st + 3) * zc + __ldg(st + 4);
  x = x * __ldg(st) + __ldg(st + 1) * w[0];
#pragma unroll
  for (int a = 0; a < 4; ++a)
    if (static_cast<uint32_t>(a) < M.nA) {
      lnS[a] = lnS[a] + (integrated - __ldg(st + 8 + a) - __ldg(st + 16 + a) + __ldg(st + 12 + a) * w[1 + a]);
      S[a] = __ldg(M.model + a) * rexp(lnS[a]);
    }
}

// The netting set's value on date jj of one inner path, from the date's lowered runs (the outer kernel's
// order: floating coupons, bonds, asset forwards, generic records, fixings); no trade groups, no probes.
// fix points at the lane's fixings, fixing s at fix[s * 32].
template <typename R>
__device__ R innerDateValue(const ImArgs<R>& M, uint32_t jj, R x, const R (&S)[4], R* fix, R (&ex)[4]) {
  using R4 = typename Vec4<R>::T;
  const uint4* dates = reinterpret_cast<const uint4*>(M.dates);
  const uint4 d0 = __ldg(dates + 2 * jj), d1 = __ldg(dates + 2 * jj + 1);
  const R* table = M.table;
  R value = R(0), ev[4] = {R(0), R(0), R(0), R(0)};
  for (uint32_t u = d0.x; u < d0.y; ++u) {
    const R4 r = ld4(table + 4 * u);
    value += (r.x * fix[asUint(r.w) * 32u] + r.y) * termExp(r.z, x);
  }
  for (uint32_t u = d0.y; u < d0.z; ++u) {
    const R4 r = ld4(table + 4 * u);
    value += r.x * termExp(r.y, x) + r.z * termExp(r.w, x);
  }
  for (uint32_t u = d0.z; u < d0.w; ++u) {
    const R4 r = ld4(table + 4 * u);
    value += r.x * sel4(S, asUint(r.z) & 3u) * r.y;
  }
  for (uint32_t u = d0.w; u < d1.x; u += 2) {
    R rec[8];
    loadTerm(table + 4 * u, rec);
    const uint32_t code = asUint(rec[0]), slot = asUint(rec[1]);
    const uint32_t kind = code & 15u, bm = min((code >> 8u) & 15u, 3u), extra = code >> 12u;
    if (kind == kBermBond && slot >= kBlockMark) {  // a block of the Bermudan's bonds (see the outer kernel)
      const uint32_t nb = slot - kBlockMark;
      const R e = sel4(ex, bm);
      if (e >= R(0) && e <= rec[2])
        for (uint32_t q = 0; q < nb; ++q) {
          const R4 b = ld4(table + 4 * (u + 2 + q));
          if (e <= b.w) value += b.x * (b.y * fastExp(-b.z * x));
        }
      u += 2 * ((nb + 1) / 2);
      continue;
    }
    const R c = rec[2];
    switch (kind) {
      case kBond: value += c * (rec[3] * fastExp(-rec[4] * x)); break;
      case kFixedFloat: value += (c * fix[slot * 32u] + rec[5]) * (rec[3] * fastExp(-rec[4] * x)); break;
      case kAsset: value += c * sel4(S, slot & 3u) * rec[3]; break;
      case kSetFixing: fix[slot * 32u] = (rec[3] * fastExp(-rec[4] * x) - R(1)) / c; break;
      case kOption: {
        const R b0 = rec[3] * fastExp(-rec[4] * x);
        value += c * black(sel4(S, slot & 3u) * rec[5] / b0, rec[6], fabs(rec[7]), b0, rec[7] > R(0));
        break;
      }
      case kBermExercise: add4(ev, bm, c * (rec[3] * fastExp(-rec[4] * x))); break;
      case kBermDecide:
        if (sel4(ex, bm) < R(0) && sel4(ev, bm) > R(0) && sel4(ev, bm) > amcPoly(rec, x)) set4(ex, bm, static_cast<R>(extra));
        break;
      case kBermContinue:
        if (sel4(ex, bm) < R(0)) value += rec[1] * fmax(amcPoly(rec, x), R(0));
        break;
      case kBermBond: {
        const R e = sel4(ex, bm);
        if (e >= R(0) && e <= static_cast<R>(extra)) value += c * (rec[3] * fastExp(-rec[4] * x));
        break;
      }
      case kBermFloat: {
        const R e = sel4(ex, bm);
        if (e >= R(0) && e <= static_cast<R>(extra)) value += (c * fix[slot * 32u] + rec[5]) * (rec[3] * fastExp(-rec[4] * x));
        break;
      }
      default: break;  // probes write rows of the outer path only
    }
  }
  for (uint32_t u = d1.x; u < d1.y; ++u) {
    const R4 r = ld4(table + 4 * u);
    fix[asUint(r.w) * 32u] = (r.x * termExp(r.y, x) - R(1)) * r.z;
  }
  return value;
}

constexpr int kImWarps = 4;

// One warp per (reporting slot r, outer path p), item r * nP + p.  Each lane keeps the 16 largest of its
// samples |V_inner(target) - V| in descending order (the reference's insertion, which never admits a NaN);
// 16 rounds of a warp maximum over the lanes' heads then give the 16 largest of all nInner samples, the
// same multiset as the reference's single list, and the quantile interpolates between two of them.
template <typename R>
__global__ void __launch_bounds__(kImWarps * 32) nestedImKernel(const ImArgs<R> M) {
  extern __shared__ __align__(16) unsigned char smemRaw[];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  R* fixIn = reinterpret_cast<R*>(smemRaw) + static_cast<size_t>(warp) * M.nSlots * 33u;  // [nSlots][32] inner
  R* fixOut = fixIn + M.nSlots * 32u;                                                     // [nSlots] outer
  const uint64_t item = static_cast<uint64_t>(blockIdx.x) * kImWarps + warp;
  if (item >= static_cast<uint64_t>(M.nR) * M.nP) return;  // warp-uniform; no block barrier below
  const uint32_t r = static_cast<uint32_t>(item / M.nP), p = static_cast<uint32_t>(item % M.nP);
  const uint32_t j = __ldg(M.slots + 2 * r), target = __ldg(M.slots + 2 * r + 1);
  if (j == kNoRow) return;  // a reporting slot on no date: the outer kernel writes no row for it either
  R* out = M.expo + static_cast<size_t>(M.rowIm + r) * M.nP + p;
  if (target == kNoRow) {
    if (lane == 0) *out = R(0);
    return;
  }
  const size_t nP = M.nP, fs = static_cast<size_t>(M.nT) * nP;
  const R* os = M.state + static_cast<size_t>(r) * (5 + M.nSlots) * nP + p;
  const R value = os[0];
  R ex0[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) ex0[b] = os[(1 + b) * nP];
  for (uint32_t q = lane; q < M.nSlots; q += 32) fixOut[q] = os[(5 + q) * nP];
  __syncwarp();
  const R x0 = M.cube[static_cast<size_t>(j) * nP + p];
  R lnS0[4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
    lnS0[a] = static_cast<uint32_t>(a) < M.nA ? M.cube[(M.fLnS + a) * fs + static_cast<size_t>(j) * nP + p] : R(0);
  const uint32_t pathStream = M.anti ? p >> 1u : p;
  const uint32_t stream = pcg(pcg(M.seed) ^ pcg(pathStream + 0x9E3779B9u));

  R top[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) top[k] = R(0);
  for (uint32_t i = lane; i < M.nInner; i += 32) {
    R x = x0, lnS[4], S[4], ex[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) lnS[a] = lnS0[a], S[a] = R(0), ex[a] = ex0[a];
    for (uint32_t q = 0; q < M.nSlots; ++q) fixIn[q * 32u + lane] = fixOut[q];
    const uint32_t istream = pcg(stream ^ pcg(0x85EBCA6Bu + (i >> 1u) * 0x9E3779B9u + j));
    const R isign = (i & 1u) ? R(-1) : R(1);
    R vi = value;
    for (uint32_t jj = j + 1; jj <= target; ++jj) {
      innerStep(M, jj, istream, isign, x, lnS, S);
      vi = innerDateValue(M, jj, x, S, fixIn + lane, ex);
    }
    R cur = fabs(vi - value);
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (cur > top[k]) {
        const R t = top[k];
        top[k] = cur, cur = t;
      }
  }
  const R rank = M.level * static_cast<R>(M.nInner - 1);
  const uint32_t k = static_cast<uint32_t>(floor(rank));
  const uint32_t hi = min(M.nInner - 1 - k, 15u);
  R ok = R(0), ok1 = R(0);
  for (uint32_t round = 0; round <= hi; ++round) {
    R m = top[0];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, d));
    if (round + 1 == hi) ok1 = m;
    if (round == hi) ok = m;
    const uint32_t owner = __ffs(__ballot_sync(0xFFFFFFFFu, top[0] == m)) - 1;
    if (lane == owner) {
#pragma unroll
      for (int q = 0; q < 15; ++q) top[q] = top[q + 1];
      top[15] = R(0);
    }
  }
  if (hi == 0) ok1 = ok;
  if (lane == 0) *out = ok + (rank - static_cast<R>(k)) * (ok1 - ok);
}

template <typename R>
cudaError_t launchNestedIm(const ImArgs<R>& M, cudaStream_t stream) {
  const uint64_t items = static_cast<uint64_t>(M.nR) * M.nP;
  if (items == 0 || M.nInner == 0) return cudaSuccess;
  const uint64_t blocks = (items + kImWarps - 1) / kImWarps;
  if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
  const size_t smem = static_cast<size_t>(kImWarps) * M.nSlots * 33u * sizeof(R);
  nestedImKernel<R><<<static_cast<uint32_t>(blocks), kImWarps * 32, smem, stream>>>(M);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
template <typename R>
cudaError_t launchSimulate(const ScenarioArgs<R>& sc, const CubeArgs<R>& cb, cudaStream_t stream) {
  SimLayout L{};
  // Adjacent paths share a stream with opposite signs (a re-run of chosen paths does not keep pairs together).  16
  // streams per CTA while they run in one wave (four CTAs per SM: 18,944 paths; 94 us against 120 at 10,000 paths, but
  // 217 against 178 at 33,333), 32 beyond.
  const bool paired = sc.antithetic && !sc.pathMap, small = paired && sc.nP <= 148u * 4u * 32u;
  const uint32_t cols = small ? 16 : 32;
  L.need = sc.nCorr + 1 + sc.nF + sc.nC * (sc.substeps - 1);
  L.slots = (L.need + sc.nC) | 1u;  // odd: the two dates of a 16-stream pass fall on different banks
  // A pass of each producer warp per buffer, two with short dates, as far as 96 KB hold two buffers.
  const uint32_t perPass = 32 / cols, round = (kSimWarps - 1 - sc.nC) * perPass;
  const size_t date = static_cast<size_t>(L.slots) * cols * sizeof(R);
  L.dates = L.slots <= 8 ? 2 * round : round;
  L.dates = std::min(L.dates, std::max(static_cast<uint32_t>(96 * 1024 / (2 * date)), 1u));
  // Threads that draw and step for themselves once they fill the GPU: the ring's stepping warps hold 64 paths (32 unpaired) of
  // a CTA's 256 threads, and each credit adds a stepping warp.  Ring against threads in us, 61 dates: unpaired, no assets nor
  // credits 73 / 76 at 33,333 paths, 185 / 96 at 100,000, 1,558 / 668 at a million; pairs, two stochastic FX rates and a credit
  // of 8 sub-steps 282 / 329 at 100,000, 547 / 462 at 200,000, 2,623 / 1,966 at a million; the same in double precision 769 /
  // 731 (whole calls) at 65,536; two credits of 4 sub-steps unpaired 650 / 677 at 200,000, 1,642 / 1,512 at 500,000, of one 392 /
  // 330 at 200,000.
  const uint32_t threads = paired ? (sc.nP + 1) / 2 : sc.nP;
  const uint32_t chains = sc.substeps <= 2 ? sc.nC : sc.nC == 2 ? 12u : 2u * sc.nC;  // several sub-steps: the credits' chains bind
  const bool walk = threads >= (2u + chains) * 148u * (sizeof(R) == 4 ? 128u : 64u);
  size_t smem = walk ? static_cast<size_t>(L.slots) * kSimThreads * sizeof(R) : 2 * L.dates * date;
  const size_t table = static_cast<size_t>(sc.nT) * (sc.substeps - 1) * 2 * sizeof(R);
  L.table = sc.nC > 0 && sc.substeps > 1 && table <= 32 * 1024;
  if (L.table) smem += table;
  auto go = [&](auto kernel, uint32_t paths) {
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      if (e != cudaSuccess) return e;
    }
    kernel<<<(sc.nP + paths - 1) / paths, kSimThreads, smem, stream>>>(sc, cb, L);
    return cudaGetLastError();
  };
  if (walk) return paired ? go(simulateWalkKernel<R, 2>, 2 * kSimThreads) : go(simulateWalkKernel<R, 1>, kSimThreads);
  return small ? go(simulateKernel<R, 1, 16>, 32) : paired ? go(simulateKernel<R, 2, 32>, 64) : go(simulateKernel<R, 1, 32>, 32);
}

size_t revalueSmemBytes(size_t stateWordsMax, bool perTrade, bool f64, int ppt) {
  const size_t r = f64 ? 8 : 4;
  return ((perTrade ? kMaxTradeGroups * ppt * kTile : 0) + stateWordsMax * ppt * kTile) * r;
}

namespace {
template <typename R, int PPT>
cudaError_t launchRevaluePPT(const CubeArgs<R>& cb, const NsArgs<R>* nsArgs, uint32_t numNs, uint32_t numTiles, size_t stateWordsMax,
                             bool perTrade, bool sink, bool lean, bool smallState, bool cash, cudaStream_t stream) {
  const size_t smem = revalueSmemBytes(stateWordsMax, perTrade, sizeof(R) == 8, PPT);
  const uint64_t blocks = static_cast<uint64_t>(numTiles) * numNs;
  if (blocks == 0) return cudaSuccess;
  if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
  auto go = [&](auto kernel) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kernel<<<static_cast<uint32_t>(blocks), kTile, smem, stream>>>(cb, nsArgs, numNs);
    return cudaGetLastError();
  };
  if (sink) return go(revalueKernel<R, PPT, false, true, false>);
  if (perTrade) return go(revalueKernel<R, PPT, true, false, false>);
  if (lean && smallState && stateWordsMax <= static_cast<size_t>(kSmallStateWords) && sizeof(R) == 4 && PPT > 1)
    return cash ? go(revalueKernel<R, PPT, false, false, true, true, true>) : go(revalueKernel<R, PPT, false, false, true, true>);
  if (lean) return cash ? go(revalueKernel<R, PPT, false, false, true, false, true>) : go(revalueKernel<R, PPT, false, false, true>);
  return go(revalueKernel<R, PPT, false, false, false>);
}
}  // namespace

template <typename R>
cudaError_t launchRevalue(const CubeArgs<R>& cb, const NsArgs<R>* nsArgs, uint32_t numNs, uint32_t numTiles, size_t stateWordsMax,
                          bool perTrade, bool sink, bool lean, int ppt, cudaStream_t stream, bool smallState, bool cash) {
  switch (ppt) {
    case 1: return launchRevaluePPT<R, 1>(cb, nsArgs, numNs, numTiles, stateWordsMax, perTrade, sink, lean, smallState, cash, stream);
    case 2: return launchRevaluePPT<R, 2>(cb, nsArgs, numNs, numTiles, stateWordsMax, perTrade, sink, lean, smallState, cash, stream);
    case 4:
      if (sizeof(R) == 4) return launchRevaluePPT<R, 4>(cb, nsArgs, numNs, numTiles, stateWordsMax, perTrade, sink, lean, smallState, cash, stream);
      return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
}

template <typename R>
cudaError_t launchSplit(const CubeArgs<R>& cb, const NsArgs<R>* nsArgs, uint32_t numNs, const SplitArgs<R>& sp, cudaStream_t stream) {
  if (numNs == 0 || sp.numItems == 0) return cudaSuccess;
  if (numNs > 65535u || sp.numItems > 65535u || sp.numDecides > 65535u) return cudaErrorInvalidConfiguration;
  if (sp.numDecides > 0) {
    decideKernel<R, false><<<dim3((cb.nP + kTile - 1) / kTile, sp.numDecides), kTile, 0, stream>>>(cb, nsArgs, sp.decides, sp.decideTable);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  auto value = [&](auto kernel, bool lean, uint32_t at, uint32_t n) {
    const uint32_t items = lean ? sp.numItems - sp.numFull : sp.numFull, tile = static_cast<uint32_t>(kTile * sp.ppt);
    if (items == 0) return cudaSuccess;
    const size_t smem = (sp.slotsMax[lean] * sizeof(R) + (lean ? 0u : sp.bermsMax)) * tile;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kernel<<<dim3((n + tile - 1) / tile, items), kTile, smem, stream>>>(cb, nsArgs, sp.items + (lean ? sp.numFull : 0u), sp.pre, sp.exFirst, at,
                                                                        sp.slabPaths);
    return cudaGetLastError();
  };
  auto settle = [&](auto kernel, size_t smem, uint32_t paths, uint32_t at, uint32_t n) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kernel<<<dim3((n + paths - 1) / paths, numNs), kSettleThreads, smem, stream>>>(cb, nsArgs, at, sp.slabPaths);
    return cudaGetLastError();
  };
  for (uint32_t at = 0; at < cb.nP; at += sp.slabPaths) {
    const uint32_t n = std::min(sp.slabPaths, cb.nP - at);
    cudaError_t e = sp.ppt == 1 ? value(valueKernel<R, 1, false>, false, at, n) : value(valueKernel<R, 2, false>, false, at, n);
    if (e == cudaSuccess) e = sp.ppt == 1 ? value(valueKernel<R, 1, true>, true, at, n) : value(valueKernel<R, 2, true>, true, at, n);
    if (e == cudaSuccess) e = sp.settlePaths == 32 ? settle(settleKernel<R, 1>, sizeof(SettleSmem<R, 1>), 32u, at, n)
                                                   : settle(settleKernel<R, 2>, sizeof(SettleSmem<R, 2>), 64u, at, n);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template <typename R>
cudaError_t launchExerciseValues(const CubeArgs<R>& cb, const NsArgs<R>* nsArgs, const DecideJob* jobs, uint32_t numJobs, const R* table,
                                 cudaStream_t stream) {
  if (numJobs == 0) return cudaSuccess;
  if (numJobs > 65535u) return cudaErrorInvalidConfiguration;
  decideKernel<R, true><<<dim3((cb.nP + kTile - 1) / kTile, numJobs), kTile, 0, stream>>>(cb, nsArgs, jobs, table);
  return cudaGetLastError();
}
template cudaError_t launchExerciseValues<float>(const CubeArgs<float>&, const NsArgs<float>*, const DecideJob*, uint32_t, const float*,
                                                 cudaStream_t);
template cudaError_t launchExerciseValues<double>(const CubeArgs<double>&, const NsArgs<double>*, const DecideJob*, uint32_t, const double*,
                                                  cudaStream_t);
template cudaError_t launchSplit<float>(const CubeArgs<float>&, const NsArgs<float>*, uint32_t, const SplitArgs<float>&, cudaStream_t);
template cudaError_t launchSplit<double>(const CubeArgs<double>&, const NsArgs<double>*, uint32_t, const SplitArgs<double>&, cudaStream_t);
template cudaError_t launchNestedIm<float>(const ImArgs<float>&, cudaStream_t);
template cudaError_t launchNestedIm<double>(const ImArgs<double>&, cudaStream_t);
template cudaError_t launchSimulate<float>(const ScenarioArgs<float>&, const CubeArgs<float>&, cudaStream_t);
template cudaError_t launchSimulate<double>(const ScenarioArgs<double>&, const CubeArgs<double>&, cudaStream_t);
template cudaError_t launchRevalue<float>(const CubeArgs<float>&, const NsArgs<float>*, uint32_t, uint32_t, size_t, bool, bool, bool,
                                          int, cudaStream_t, bool, bool);
template cudaError_t launchRevalue<double>(const CubeArgs<double>&, const NsArgs<double>*, uint32_t, uint32_t, size_t, bool, bool, bool,
                                           int, cudaStream_t, bool, bool);

}  // namespace zk
