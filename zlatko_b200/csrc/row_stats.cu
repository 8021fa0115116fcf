// reduce-partials and row statistics (the reference's second and third kernels,
// src/gpu/fused_kernels.cpp:538-563 and :565-771; CPU mirror finishFused,
// src/gpu/fused_reference.cpp:468-607).
//
// reduce: the per-tile partials of each (date, statistic) in tile order, in 32 segments of compensated double-precision
// sums added in order, so the result depends neither on scheduling nor on the launch's other plans.
//
// row statistics: one CTA per request.  Quantiles are the *exact* empirical quantile interpolated
// between order statistics k = floor(p (n - 1)) and k + 1, as ccr::quantile does
// (include/ccr/core/math.hpp:39-47), found without sorting the row.  Rows of 8K values or more: a 1/16 sample says in
// which window of values the ranks lie, and one pass counts the values under it and keeps those in it, among which a radix
// selection finds them.  Shorter rows, and rows whose window misses or overflows: a min/max pass, a 4096-bin
// histogram pass that locates the bins of ranks k and k + 1, then either one pass that reads the
// maximum of k's bin and the minimum of k+1's bin (different bins) or a gather of k's bin into
// shared memory and a radix selection there (same bin; narrowed again if the bin holds more than
// kCap values).  The reference's histogram kernel interpolates inside the final bin instead and
// agrees with the exact quantile to about 5e-8 (README.md:182).
#include <cfloat>

#include "zk_device.cuh"
#include "zk_kernels.h"

namespace zk {

namespace {

constexpr int kRowThreads = 256;
constexpr int kRowWarps = kRowThreads / 32;
constexpr int kBins = 4096;
constexpr int kCap = 4096;
constexpr int kMaxRounds = 16;
constexpr int kHistBins = 3072;  // the reference's histogram-request limit (kPfeBins)
constexpr int kPool = 8192;      // values kept from the window the sample points at
// A window of the sample holds about 16 times its values in the row, give or take a few hundred, spread over the warps'
// shares of kPool: the pass is made where it expects to keep at most this many.  (With a pool of half the size, and the pass
// made whether it fitted or not, 97.5% of a million paths took 1.96 ms in four netting sets and 0.55 now, 99% of two million
// 3.10 and 0.96, a median of 500,000 in twelve 4.18 and 3.95.)
constexpr uint32_t kWindowKept = 7000;

template <typename R>
struct RowSmem {
  union {  // the histogram is read up to the choice of the bins; the candidates are gathered after it
    uint32_t hist[kBins];
    R cand[kCap];
    R pool[kPool];
  };
  alignas(8) uint32_t digits[264];
  double dsum[kRowWarps];
  R rmin[kRowWarps], rmax[kRowWarps];
  uint32_t candCount;
  uint32_t usum[kRowWarps], ukept[kRowWarps];
  uint32_t pick[5];
  double flo[kMaxRounds], finvw[kMaxRounds];
  uint32_t fb0[kMaxRounds], fb1[kMaxRounds];
};

__device__ __forceinline__ double blockSum(double v, double* scratch) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kRowWarps; ++w) s += scratch[w];
  __syncthreads();
  return s;  // valid in thread 0
}

// Bin 0 holds the row's minimum, the dominant duplicate of exposure rows (exact zeros): instead of counting it value
// by value, its count is the values binned less the other bins' counts, summed here over the CTA.
__device__ __forceinline__ void fillBinZero(uint32_t* hist, uint32_t binned, uint32_t* scratch) {
  uint32_t v = 0;
  for (uint32_t b = threadIdx.x; b < static_cast<uint32_t>(kBins); b += kRowThreads)
    if (b != 0) v += hist[b];
  v = __reduce_add_sync(0xFFFFFFFFu, v);
  if ((threadIdx.x & 31u) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kRowWarps; ++w) t += scratch[w];
    hist[0] = binned - t;
  }
  __syncthreads();
}

template <typename R>
__device__ __forceinline__ void blockMinMax(R& lo, R& hi, R* smin, R* smax) {
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) smin[warp] = lo, smax[warp] = hi;
  __syncthreads();
  lo = smin[0], hi = smax[0];
  for (int w = 1; w < kRowWarps; ++w) lo = fmin(lo, smin[w]), hi = fmax(hi, smax[w]);
  __syncthreads();
}

// The bin of a value over a range starting at lo, `scale` bins per unit: any non-decreasing map of the values to the
// bins serves the rank search, as long as every pass of a round uses the same one.  Double rows: floor((v - lo)
// scale) in double.  Single-precision rows: (v - lo) scale in float, clamped, rounded to an integer by adding 2^23
// (an FMA-pipe add and an integer subtract instead of two conversions per value); scaleOf gives the float scale.
__device__ __forceinline__ uint32_t binOf(double v, double lo, double scale) {
  const double f = (v - lo) * scale;
  const uint32_t b = f <= 0.0 ? 0u : (f >= static_cast<double>(kBins) ? static_cast<uint32_t>(kBins) : static_cast<uint32_t>(f));
  return min(b, static_cast<uint32_t>(kBins - 1));
}
__device__ __forceinline__ uint32_t binOf(float v, double lo, double scale) {
  const float f = fminf(fmaxf((v - static_cast<float>(lo)) * static_cast<float>(scale), 0.0f), static_cast<float>(kBins - 1));
  return __float_as_uint(f + 8388608.0f) - 0x4B000000u;
}
template <typename R>
__device__ __forceinline__ double scaleOf(R lo, R hi) {
  const double sc = static_cast<double>(kBins) / (static_cast<double>(hi) - static_cast<double>(lo));
  return sizeof(R) == 4 ? static_cast<double>(static_cast<float>(sc)) : sc;
}

template <typename R>
__device__ __forceinline__ bool passes(const RowSmem<R>& s, int rounds, R v) {
  for (int r = 0; r < rounds; ++r) {
    const uint32_t b = binOf(v, s.flo[r], s.finvw[r]);
    if (b < s.fb0[r] || b > s.fb1[r]) return false;
  }
  return true;
}

// The 16-byte vectors of a row: the first aligned value and the number of whole vectors after it.
template <typename R>
struct RowVectors {
  uint32_t head, count;
};
template <typename R>
__device__ __forceinline__ RowVectors<R> vectorsOf(const R* X, uint32_t nP) {
  constexpr uint32_t kVec = 16 / sizeof(R);
  const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(X) / sizeof(R)) % kVec, head = min((kVec - off) % kVec, nP);
  return {head, (nP - head) / kVec};
}

// Calls f(v, valid) for every value of the row, through max(x, 0) when pos, 16 bytes per load; the values before the first
// aligned one and after the last whole vector (rows of an odd number of paths start anywhere) one by one.
template <typename R, typename F>
__device__ __forceinline__ void forEachValue(const R* X, uint32_t nP, bool pos, F&& f) {
  const uint32_t tid = threadIdx.x;
  auto fix = [&](R x) { return pos ? fmax(x, R(0)) : x; };
  constexpr uint32_t kVec = 16 / sizeof(R);
  const RowVectors<R> V = vectorsOf(X, nP);
  const R* body = X + V.head;
#pragma unroll 4
  for (uint32_t base = 0; base < V.count; base += kRowThreads) {
    const uint32_t i = base + tid;
    const bool ok = i < V.count;
    if constexpr (sizeof(R) == 4) {
      const float4 q = ok ? __ldg(reinterpret_cast<const float4*>(body) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      f(fix(q.x), ok), f(fix(q.y), ok), f(fix(q.z), ok), f(fix(q.w), ok);
    } else {
      const double2 q = ok ? __ldg(reinterpret_cast<const double2*>(body) + i) : make_double2(0.0, 0.0);
      f(fix(q.x), ok), f(fix(q.y), ok);
    }
  }
  const uint32_t tail = V.head + V.count * kVec, loose = V.head + (nP - tail);
  if (tid < loose) f(fix(__ldg(X + (tid < V.head ? tid : tail + tid - V.head))), true);
}

// Values of the row (through max(x, 0) when pos) below `from` counted, and those in [from, to] kept: each warp appends to its
// own kPoolWarp slots by ballots (an atomic with its returned position stalls the warp at nearly every vector).  Returns
// this thread's count below; `kept` the warp's values in the window, more than kPoolWarp when they did not fit.
constexpr uint32_t kPoolWarp = kPool / kRowWarps;
template <typename R>
__device__ __forceinline__ uint32_t windowPass(const R* X, uint32_t nP, bool pos, R from, R to, R* pool, uint32_t& kept) {
  constexpr uint32_t kVec = 16 / sizeof(R), kDeep = 4;
  const uint32_t tid = threadIdx.x, below = (1u << (tid & 31u)) - 1u;
  const RowVectors<R> V = vectorsOf(X, nP);
  const R* body = X + V.head;
  R* mine = pool + (tid >> 5) * kPoolWarp;
  uint32_t under = 0, n = 0;
  auto take = [&](const R (&v)[kVec], bool ok) {
    bool in[kVec], any = false;
#pragma unroll
    for (uint32_t e = 0; e < kVec; ++e) {
      const R x = pos ? fmax(v[e], R(0)) : v[e];
      const bool up = x >= from;  // a NaN ranks below, as in the rounds' bin 0
      under += ok && !up ? 1u : 0u;
      in[e] = ok && up && x <= to, any = any || in[e];
    }
    if (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
      for (uint32_t e = 0; e < kVec; ++e) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, in[e]), at = n + __popc(m & below);
        if (in[e] && at < kPoolWarp) mine[at] = pos ? fmax(v[e], R(0)) : v[e];
        n += __popc(m);
      }
    }
  };
  auto load = [&](uint32_t i, R (&v)[kVec]) {
    if constexpr (sizeof(R) == 4) {
      const float4 q = i < V.count ? __ldg(reinterpret_cast<const float4*>(body) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
      const double2 q = i < V.count ? __ldg(reinterpret_cast<const double2*>(body) + i) : make_double2(0.0, 0.0);
      v[0] = q.x, v[1] = q.y;
    }
  };
  for (uint32_t base = 0; base < V.count; base += kRowThreads * kDeep) {
    R v[kDeep][kVec];
#pragma unroll
    for (uint32_t d = 0; d < kDeep; ++d) load(base + d * kRowThreads + tid, v[d]);
#pragma unroll
    for (uint32_t d = 0; d < kDeep; ++d) take(v[d], base + d * kRowThreads + tid < V.count);
  }
  // the values outside the whole vectors, fewer than eight: the first warp's
  const uint32_t tail = V.head + V.count * kVec, loose = V.head + (nP - tail);
  if (tid < 32) {
    R v[kVec] = {};
    if (tid < loose) v[0] = __ldg(X + (tid < V.head ? tid : tail + tid - V.head));
    const uint32_t before = under;
    const R x = pos ? fmax(v[0], R(0)) : v[0];
    const bool ok = tid < loose, up = x >= from, in = ok && up && x <= to;
    under = before + (ok && !up ? 1u : 0u);
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, in), at = n + __popc(m & below);
    if (in && at < kPoolWarp) mine[at] = x;
    n += __popc(m);
  }
  kept = n;
  return under;
}

// A quantile's histogram needs a range, not the row's exact extremes: values outside it fall into the end bins,
// and the ranks are still located exactly.  On long rows the range is the minimum and maximum of a sample,
// every 16th block of 32 vectors (512 bytes, one 16-byte load per lane of a warp), about 1/16 of the row.
constexpr uint32_t kSampleStride = 16;
constexpr uint32_t kSampleMinVectors = 2048;  // rows of 8K floats or 4K doubles and more

template <typename R>
__device__ __forceinline__ bool canSample(const R* X, uint32_t nP) {
  return vectorsOf(X, nP).count >= kSampleMinVectors;
}

template <typename R>
__device__ __forceinline__ void sampleMinMax(const R* X, uint32_t nP, bool pos, R& lo, R& hi) {
  const RowVectors<R> V = vectorsOf(X, nP);
  const uint32_t blocks = V.count / 32, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  X += V.head;
  auto take = [&](R x) {
    x = pos ? fmax(x, R(0)) : x;
    lo = fmin(lo, x), hi = fmax(hi, x);
  };
#pragma unroll 4
  for (uint32_t b = warp * kSampleStride; b < blocks; b += kRowWarps * kSampleStride) {
    const uint32_t i = b * 32 + lane;
    if constexpr (sizeof(R) == 4) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(X) + i);
      take(q.x), take(q.y), take(q.z), take(q.w);
    } else {
      const double2 q = __ldg(reinterpret_cast<const double2*>(X) + i);
      take(q.x), take(q.y);
    }
  }
}

// The histogram of the same sample as sampleMinMax over the bins of (dlo, invw), bin 0's votes per warp as in the
// full pass; returns the number of values sampled.
template <typename R>
__device__ __forceinline__ uint32_t sampleHistogram(const R* X, uint32_t nP, bool pos, double dlo, double invw, uint32_t* hist) {
  constexpr uint32_t kVec = 16 / sizeof(R);
  const RowVectors<R> V = vectorsOf(X, nP);
  const uint32_t blocks = V.count / 32, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  X += V.head;
  auto put = [&](R x) {  // bin 0 is filled afterwards (fillBinZero)
    x = pos ? fmax(x, R(0)) : x;
    const uint32_t b = binOf(x, dlo, invw);
    if (b != 0) atomicAdd(&hist[b], 1u);
  };
#pragma unroll 4
  for (uint32_t b = warp * kSampleStride; b < blocks; b += kRowWarps * kSampleStride) {
    const uint32_t i = b * 32 + lane;
    if constexpr (sizeof(R) == 4) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(X) + i);
      put(q.x), put(q.y), put(q.z), put(q.w);
    } else {
      const double2 q = __ldg(reinterpret_cast<const double2*>(X) + i);
      put(q.x), put(q.y);
    }
  }
  return (blocks + kSampleStride - 1) / kSampleStride * 32u * kVec;
}

// The bins of ranks k and k1 >= k among the candidates counted in s.hist, `below` values ranking under bin 0:
// pick = {bin of k, bin of k1, values under k's bin, count of k's bin, values up to k1's bin}, as a walk over the bins in
// order would find them.  One warp: lane l owns bins [128 l, 128 l + 128) (read skewed by l, free of bank conflicts), a
// warp scan of the lanes' counts finds the lane holding each rank, and that lane walks its own bins.
template <typename R>
__device__ __forceinline__ void locateRanks(RowSmem<R>& s, uint32_t below, uint32_t k, uint32_t k1, uint32_t lane) {
  constexpr uint32_t kPer = kBins / 32;
  uint32_t own = 0;
  for (uint32_t j = 0; j < kPer; ++j) own += s.hist[lane * kPer + ((j + lane) & (kPer - 1))];
  uint32_t incl = own;
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += v;
  }
  const uint32_t start = below + incl - own;  // values under this lane's first bin
  const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, below + incl > k), m1 = __ballot_sync(0xFFFFFFFFu, below + incl > k1);
  const uint32_t l0 = m0 ? __ffs(m0) - 1 : 31u, l1 = m1 ? __ffs(m1) - 1 : 31u;
  auto walk = [&](uint32_t r, uint32_t& bin, uint32_t& under) {
    uint32_t cum = start;
    bin = lane * kPer + kPer - 1, under = cum;
    for (uint32_t b = lane * kPer; b < lane * kPer + kPer; ++b) {
      const uint32_t c = s.hist[b];
      if (cum + c > r) {
        bin = b, under = cum;
        return;
      }
      cum += c;
    }
  };
  if (lane == l0) {
    uint32_t b0, under0;
    walk(k, b0, under0);
    if (!m0) b0 = kBins - 1, under0 = below;  // no rank k among the candidates (cannot happen): the last bin
    s.pick[0] = b0, s.pick[2] = under0, s.pick[3] = s.hist[b0];
  }
  if (lane == l1) {
    uint32_t b1, under1;
    walk(k1, b1, under1);
    if (!m1) b1 = kBins - 1;
    s.pick[1] = b1, s.pick[4] = under1 + s.hist[b1];
  }
}

__device__ __forceinline__ uint32_t orderKey(float v) { return floatKey(v); }
__device__ __forceinline__ unsigned long long orderKey(double v) { return doubleKey(v); }
__device__ __forceinline__ float fromKey(uint32_t k) { return keyFloat(k); }
__device__ __forceinline__ double fromKey(unsigned long long k) { return keyDouble(k); }

// The values of ranks r and r1 (r or r + 1, below n) among n values, by their order-preserving integer keys (each(f) calls
// f(value) for this thread's share of the values):
// a radix selection of 8 bits a pass finds rank r's value, and the next one is that value again or the least above it.  (A
// bitonic sort of 2,048 values took 66 barriers and 45 us, four passes take 4.)  scratch: 256 + 8 words; every thread gets
// both values.
template <typename R, typename Each>
__device__ __forceinline__ void selectRanks(Each&& each, uint32_t n, uint32_t r, uint32_t r1, uint32_t* scratch, R& v, R& v1) {
  using Key = decltype(orderKey(R(0)));
  constexpr int kBits = 8 * static_cast<int>(sizeof(R));
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  static_assert(kRowThreads == 256, "a thread per digit");
  Key prefix = 0, mask = 0;
  uint32_t rank = r, same = n;  // rank among the values with the prefix; how many those are
  for (int shift = kBits - 8; shift >= 0; shift -= 8) {
    scratch[tid] = 0;
    __syncthreads();
    each([&](R x) {
      const Key key = orderKey(x);
      if ((key & mask) == prefix) atomicAdd(&scratch[static_cast<uint32_t>(key >> shift) & 255u], 1u);
    });
    __syncthreads();
    // The digit whose running count passes the rank: each thread scans its digit's count over the CTA.
    const uint32_t own = scratch[tid];
    uint32_t incl = own;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();  // scratch has been read
    if (lane == 31) scratch[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; ++w) before += scratch[w];
    const uint32_t lo = before + incl - own;
    if (own > 0 && lo <= rank && rank < lo + own) scratch[16] = tid, scratch[17] = lo, scratch[18] = own;
    __syncthreads();
    prefix |= static_cast<Key>(scratch[16]) << shift, mask |= static_cast<Key>(255) << shift;
    rank -= scratch[17], same = scratch[18];
    __syncthreads();
  }
  v = fromKey(prefix);
  v1 = v;
  if (r1 == r || rank + 1 < same) return;  // rank r + 1 is the same value
  // The least value above: its key minimum over the CTA, two words for a double's.
  Key best = ~static_cast<Key>(0);
  each([&](R x) {
    const Key key = orderKey(x);
    if (key > prefix && key < best) best = key;
  });
#pragma unroll
  for (uint32_t o = 16; o > 0; o >>= 1) {
    const Key t = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    best = t < best ? t : best;
  }
  Key* keys = reinterpret_cast<Key*>(scratch);
  if (lane == 0) keys[warp] = best;
  __syncthreads();
  for (uint32_t w = 0; w < static_cast<uint32_t>(kRowWarps); ++w) best = keys[w] < best ? keys[w] : best;
  v1 = fromKey(best);
  __syncthreads();
}

template <typename R>
__global__ void __launch_bounds__(kRowThreads, 6) rowStatsKernel(const RowJob<R>* __restrict__ jobs, uint32_t* __restrict__ err,
                                                                 uint32_t maxRounds) {
  extern __shared__ __align__(16) unsigned char raw[];
  RowSmem<R>& s = *reinterpret_cast<RowSmem<R>*>(raw);
  const RowJob<R> J = jobs[blockIdx.x];
  const R* rq = J.request;
  const uint32_t op = static_cast<uint32_t>(rq[0]), row = static_cast<uint32_t>(rq[1]), row2 = static_cast<uint32_t>(rq[2]);
  const uint32_t count = static_cast<uint32_t>(rq[3]);
  const size_t outAt = static_cast<size_t>(rq[7]);
  const uint32_t nP = J.nP, tid = threadIdx.x;
  const R* X = J.expo + static_cast<size_t>(row) * nP;
  R* out = J.out + outAt;

  if (op == 4) {  // samples: the first `count` paths
    for (uint32_t i = tid; i < count && i < nP; i += kRowThreads) out[i] = X[i];
    return;
  }
  if (op != 0 && op != 5 && op != 7) {  // means, in double precision
    const R* Y = J.expo + static_cast<size_t>(row2) * nP;
    double acc = 0.0;
    if (op == 1 || op == 2 || op == 3) {
      forEachValue(X, nP, false, [&](R x, bool ok) {
        const R f = op == 2 ? fmax(x, R(0)) : op == 3 ? fmin(x, R(0)) : x;
        if (ok) acc += static_cast<double>(f);
      });
    } else {
      for (uint32_t i = tid; i < nP; i += kRowThreads) {
        const R x = X[i];
        R f = x;
        switch (op) {
          case 6: f = x * Y[i]; break;
          case 8: f = fmax(x, R(0)) * Y[i]; break;
          case 9: f = fmin(x, R(0)) * Y[i]; break;
          default: break;
        }
        acc += static_cast<double>(f);
      }
    }
    const double total = blockSum(acc, s.dsum);
    if (tid == 0) out[0] = static_cast<R>(total / static_cast<double>(nP));
    return;
  }

  const bool pos = op == 7;
  R lo = R(INFINITY), hi = R(-INFINITY);
  // Quantiles of long rows take their first histogram's range from a sample (the row is then read twice, not
  // three times); a histogram request reports its range, and a sample without spread proves nothing, so those
  // read the whole row for its exact minimum and maximum.
  bool sampled = false;
  if (op != 5 && canSample(X, nP)) {
    sampleMinMax(X, nP, pos, lo, hi);
    blockMinMax(lo, hi, s.rmin, s.rmax);
    sampled = lo < hi;
  }
  if (!sampled) {
    lo = R(INFINITY), hi = R(-INFINITY);
    forEachValue(X, nP, pos, [&](R v, bool ok) {
      if (ok) lo = fmin(lo, v), hi = fmax(hi, v);
    });
    blockMinMax(lo, hi, s.rmin, s.rmax);
  }

  if (op == 5) {  // histogram of `count` bins on [lo, hi] (the request's range unless lo == hi there)
    if (rq[5] != rq[6]) lo = rq[5], hi = rq[6];
    const R span = fmax(hi - lo, R(1e-30));
    const uint32_t nb = min(count, static_cast<uint32_t>(kHistBins));
    for (uint32_t b = tid; b < nb; b += kRowThreads) s.hist[b] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < nP; i += kRowThreads) {
      const R f = fmax((X[i] - lo) / span, R(0)) * static_cast<R>(nb);
      const uint32_t b = min(f >= R(4294967295.0) ? 0xFFFFFFFFu : static_cast<uint32_t>(f), nb - 1);
      atomicAdd(&s.hist[b], 1u);
    }
    __syncthreads();
    for (uint32_t b = tid; b < nb; b += kRowThreads) out[b] = static_cast<R>(s.hist[b]);
    if (tid == 0) out[nb] = lo, out[nb + 1] = hi;
    return;
  }

  // Exact interpolated quantile (ccr::quantile): ranks k and k1 = min(k + 1, n - 1).
  const double h = static_cast<double>(rq[4]) * static_cast<double>(nP - 1);
  const uint32_t k = min(static_cast<uint32_t>(floor(h)), nP - 1), k1 = min(k + 1, nP - 1);
  const double frac = h - static_cast<double>(k);
  if (!(lo < hi)) {
    if (tid == 0) out[0] = lo;
    return;
  }
  uint32_t below = 0, binned = nP;  // the values each round bins: the row, then the previous round's bin
  int rounds = 0;
  R vk = lo, vk1 = lo;
  bool done = false;
  // On a sampled row the sample's own histogram says where ranks k, k1 lie to within the sample's rank error: one pass
  // counts the row's values under the bins of sample ranks k_s -+ (3 sd + 4) and keeps the values in them, and when the
  // ranks fall among those (the counts prove it) they are selected there.  No histogram of the row: a shared-memory
  // atomic per value had bound the pass (100 netting sets, 121 rows each of 250,000 paths: 5.05 ms, 33,333 odd paths x 12
  // 282 us; now 3.97 ms and 156 us).  A window too full for the pool (a median of many paths, equal values) would waste the
  // pass, 4 to 20% of such a row: the sample's count says so beforehand.  Else the rounds below.
  if (sampled) {
    const double dlo0 = static_cast<double>(lo), invw0 = scaleOf(lo, hi);
    for (uint32_t b = tid; b < kBins; b += kRowThreads) s.hist[b] = 0;
    __syncthreads();
    const uint32_t ns = sampleHistogram(X, nP, pos, dlo0, invw0, s.hist);
    __syncthreads();
    fillBinZero(s.hist, ns, s.usum);
    const double q = static_cast<double>(k) / static_cast<double>(nP), ks = q * static_cast<double>(ns);
    const double sd = sqrt(static_cast<double>(ns) * q * (1.0 - q)) * 3.0 + 4.0;
    const uint32_t rlo = static_cast<uint32_t>(fmax(ks - sd, 0.0)), rhi = static_cast<uint32_t>(fmin(ks + sd + 1.0, ns - 1.0));
    if (tid < 32) locateRanks(s, 0u, rlo, rhi, tid);
    __syncthreads();
    const uint32_t winLo = s.pick[0], winHi = s.pick[1], sampledIn = s.pick[4] - s.pick[2];
    if (static_cast<uint64_t>(sampledIn) * nP <= static_cast<uint64_t>(kWindowKept) * ns) {
      // The window's edges as values, half a bin outside the bins' centres (the ends open): any edges serve, the counts decide.
      const R from = winLo == 0 ? R(-INFINITY) : static_cast<R>(dlo0 + (static_cast<double>(winLo) - 0.5) / invw0);
      const R to = winHi + 1 >= static_cast<uint32_t>(kBins) ? R(INFINITY) : static_cast<R>(dlo0 + (static_cast<double>(winHi) + (sizeof(R) == 4 ? 0.5 : 1.0)) / invw0);
      uint32_t kept;
      uint32_t under = windowPass(X, nP, pos, from, to, s.pool, kept);
      under = __reduce_add_sync(0xFFFFFFFFu, under);
      if ((tid & 31u) == 0) s.usum[tid >> 5] = under, s.ukept[tid >> 5] = kept;
      __syncthreads();
      uint32_t total = 0;
      bool fit = true;
      under = 0;
      for (int w = 0; w < kRowWarps; ++w) fit = fit && s.ukept[w] <= kPoolWarp, under += s.usum[w], total += s.ukept[w];
      if (fit && under <= k && k1 - under < total) {  // the ranks are among the kept values
        selectRanks([&](auto&& f) {  // each warp its own
          for (uint32_t i = tid & 31u; i < kept; i += 32) f(s.pool[(tid >> 5) * kPoolWarp + i]);
        }, total, k - under, k1 - under, s.digits, vk, vk1);
        done = true;
      }
      __syncthreads();
    }
  }
  while (!done) {
    if (rounds >= static_cast<int>(maxRounds)) {
      if (tid == 0) atomicExch(err, kDevBadTerm), out[0] = R(NAN);
      return;
    }
    // Range of the current candidates (round 0: the whole row, already known).
    if (rounds > 0) {
      lo = R(INFINITY), hi = R(-INFINITY);
      forEachValue(X, nP, pos, [&](R v, bool ok) {
        if (ok && passes(s, rounds, v)) lo = fmin(lo, v), hi = fmax(hi, v);
      });
      blockMinMax(lo, hi, s.rmin, s.rmax);
      if (!(lo < hi)) {  // every candidate has the same value
        vk = lo, vk1 = lo;
        break;
      }
    }
    const double dlo = static_cast<double>(lo), invw = scaleOf(lo, hi);
    for (uint32_t b = tid; b < kBins; b += kRowThreads) s.hist[b] = 0;
    __syncthreads();
    forEachValue(X, nP, pos, [&](R x, bool ok) {
      const bool in = ok && passes(s, rounds, x);
      const uint32_t b = binOf(x, dlo, invw);
      if (in && b != 0) atomicAdd(&s.hist[b], 1u);  // bin 0 is filled afterwards (fillBinZero)
    });
    __syncthreads();
    fillBinZero(s.hist, binned, s.usum);
    if (tid < 32) locateRanks(s, below, k, k1, tid);
    __syncthreads();
    const uint32_t b0 = s.pick[0], b1 = s.pick[1], below0 = s.pick[2], c0 = s.pick[3];
    if (b0 != b1) {
      // k is the largest value of bin b0, k + 1 the smallest of bin b1.
      R mx = R(-INFINITY), mn = R(INFINITY);
      forEachValue(X, nP, pos, [&](R v, bool ok) {
        if (!ok || !passes(s, rounds, v)) return;
        const uint32_t b = binOf(v, dlo, invw);
        if (b == b0) mx = fmax(mx, v);
        if (b == b1) mn = fmin(mn, v);
      });
      blockMinMax(mn, mx, s.rmin, s.rmax);  // block minimum of mn, block maximum of mx
      vk = mx, vk1 = mn;
      done = true;
    } else if (c0 <= static_cast<uint32_t>(kCap)) {
      if (tid == 0) s.candCount = 0;
      __syncthreads();
      forEachValue(X, nP, pos, [&](R v, bool ok) {
        if (ok && passes(s, rounds, v) && binOf(v, dlo, invw) == b0) s.cand[atomicAdd(&s.candCount, 1u)] = v;
      });
      __syncthreads();
      const uint32_t n = s.candCount;
      selectRanks([&](auto&& f) {
        for (uint32_t i = tid; i < n; i += kRowThreads) f(s.cand[i]);
      }, n, k - below0, min(k1 - below0, n - 1), s.digits, vk, vk1);
      done = true;
    } else {
      if (tid == 0) s.flo[rounds] = dlo, s.finvw[rounds] = invw, s.fb0[rounds] = b0, s.fb1[rounds] = b0;
      __syncthreads();
      below = below0, binned = c0;
      ++rounds;
    }
  }
  if (tid == 0) {
    const double a = static_cast<double>(vk), b = static_cast<double>(vk1);
    out[0] = static_cast<R>(a + frac * (b - a));
  }
}

// Partials come one per warp of the revalue kernel: the sum over its 32 ppt adjacent paths.  A 128-path group's
// sum completes the binary tree of the warp sums ((w0 + w1) + (w2 + w3) for one path per thread, w0 + w1 for
// two, w0 for four), absent warps past the last path counting as 0, so it has the same bits for every tile
// shape; the groups are then summed in path order with a compensated double sum.
//
// One CTA per 32 columns (date, statistic), the groups in kSegs consecutive segments, each a compensated sum of its own with
// four groups' loads in flight; the segments are added in order, compensated too.  Always kSegs of them, so that a plan's
// sums do not depend on what else is in the launch; kWarps warps share them.  (One thread walked all groups
// of a column: 129 us for 12 netting sets at 33,333 paths and 1,155 us for 100 at
// 250,000; now 18 and 889.)
constexpr int kSegs = 32;
template <typename R, int PPT, int kWarps>
__global__ void __launch_bounds__(32 * kWarps) reduceKernel(const ReduceJob<R>* __restrict__ jobs) {
  __shared__ double segSum[kSegs][32], segComp[kSegs][32];
  const ReduceJob<R> J = jobs[blockIdx.y];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, i = blockIdx.x * 32u + lane;
  if (blockIdx.x * 32u >= J.n) return;
  // A job with pad 1 or 2 has partials of 32 or 64 paths whatever the batch's shape (the basis kernel's: 64).
  const uint32_t ppt = J.pad == 1u || J.pad == 2u ? J.pad : static_cast<uint32_t>(PPT);
  const uint32_t units = 4 / ppt, unitPaths = 32 * ppt, col = min(i, J.n - 1);
  const uint32_t count = (J.nP + unitPaths - 1) / unitPaths;  // partials
  const R* __restrict__ P = J.partials + col;
  auto unit = [&](uint32_t u) { return u < count ? __ldg(P + static_cast<size_t>(u) * J.n) : R(0); };
#pragma unroll 1
  for (uint32_t seg = warp * (kSegs / kWarps); seg < (warp + 1) * (kSegs / kWarps); ++seg) {
    double sum = 0.0, comp = 0.0;
    const uint32_t t0 = static_cast<uint32_t>(static_cast<uint64_t>(J.numTiles) * seg / kSegs);
    const uint32_t t1 = static_cast<uint32_t>(static_cast<uint64_t>(J.numTiles) * (seg + 1) / kSegs);
#pragma unroll 4
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t u = t * units;
      R g;
      if (ppt == 1) g = (unit(u) + unit(u + 1)) + (unit(u + 2) + unit(u + 3));
      else if (ppt == 2) g = unit(u) + unit(u + 1);
      else g = unit(u);
      const double yv = static_cast<double>(g) - comp;
      const double tv = sum + yv;
      comp = (tv - sum) - yv;
      sum = tv;
    }
    // An infinite last group leaves the sum infinite and its compensation NaN, which no later group takes up.
    segSum[seg][lane] = sum, segComp[seg][lane] = seg == kSegs - 1 && isinf(sum) ? 0.0 : comp;
  }
  __syncthreads();
  if (warp != 0 || i >= J.n) return;
  double sum = segSum[0][lane], comp = segComp[0][lane];
  for (int s = 1; s < kSegs; ++s) {  // sum - comp is the segment's sum to more than double precision
    const double yv = (segSum[s][lane] - segComp[s][lane]) - comp;
    const double tv = sum + yv;
    comp = (tv - sum) - yv;
    sum = tv;
  }
  J.sums[i] = static_cast<R>(sum / static_cast<double>(J.nP));
}

}  // namespace

template <typename R>
cudaError_t launchReduce(const ReduceJob<R>* jobs, uint32_t numJobs, uint32_t maxN, int ppt, cudaStream_t stream) {
  if (numJobs == 0 || maxN == 0) return cudaSuccess;
  const dim3 grid((maxN + 31) / 32, numJobs);
  // 32 warps, a segment each, where the columns alone leave the GPU idle, 8 where they fill it.
  const bool few = static_cast<uint64_t>(grid.x) * grid.y < 148u * 8u;
  auto go = [&](auto kernel, int warps) { kernel<<<grid, 32 * warps, 0, stream>>>(jobs); };
  switch (ppt) {
    case 1: few ? go(reduceKernel<R, 1, 32>, 32) : go(reduceKernel<R, 1, 8>, 8); break;
    case 2: few ? go(reduceKernel<R, 2, 32>, 32) : go(reduceKernel<R, 2, 8>, 8); break;
    case 4: few ? go(reduceKernel<R, 4, 32>, 32) : go(reduceKernel<R, 4, 8>, 8); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <typename R>
cudaError_t launchRowStats(const RowJob<R>* jobs, uint32_t numJobs, uint32_t* err, cudaStream_t stream, uint32_t maxRounds) {
  if (numJobs == 0) return cudaSuccess;
  maxRounds = maxRounds < static_cast<uint32_t>(kMaxRounds) ? maxRounds : static_cast<uint32_t>(kMaxRounds);
  const size_t smem = sizeof(RowSmem<R>);
  cudaError_t e = cudaFuncSetAttribute(rowStatsKernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  rowStatsKernel<R><<<numJobs, kRowThreads, smem, stream>>>(jobs, err, maxRounds);
  return cudaGetLastError();
}

// The exact-decision check's patch: dst[r][map[q]] = src[r][q] (rounded to single precision) for every row r and
// re-run path q.  One thread per element; map holds distinct paths below nP.
__global__ void scatterRowsKernel(const double* __restrict__ src, uint32_t m, const uint32_t* __restrict__ map, uint32_t rows,
                                  float* __restrict__ dst, uint32_t nP) {
  const uint64_t k = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= static_cast<uint64_t>(rows) * m) return;
  const uint32_t r = static_cast<uint32_t>(k / m), q = static_cast<uint32_t>(k % m);
  dst[static_cast<size_t>(r) * nP + map[q]] = static_cast<float>(src[static_cast<size_t>(r) * m + q]);
}

cudaError_t launchScatterRows(const double* src, uint32_t m, const uint32_t* map, uint32_t rows, float* dst, uint32_t nP,
                              cudaStream_t stream) {
  const uint64_t n = static_cast<uint64_t>(rows) * m;
  if (n == 0) return cudaSuccess;
  scatterRowsKernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(src, m, map, rows, dst, nP);
  return cudaGetLastError();
}

template cudaError_t launchReduce<float>(const ReduceJob<float>*, uint32_t, uint32_t, int, cudaStream_t);
template cudaError_t launchReduce<double>(const ReduceJob<double>*, uint32_t, uint32_t, int, cudaStream_t);
template cudaError_t launchRowStats<float>(const RowJob<float>*, uint32_t, uint32_t*, cudaStream_t, uint32_t);
template cudaError_t launchRowStats<double>(const RowJob<double>*, uint32_t, uint32_t*, cudaStream_t, uint32_t);

}  // namespace zk
