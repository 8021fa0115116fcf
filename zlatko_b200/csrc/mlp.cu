// The surrogate's tensor-core kernels: a BF16 GEMM with FP32 accumulation in TMEM (tcgen05.mma, operands
// staged in shared memory in the canonical K-major layout, one elected thread issuing the MMAs), with the
// epilogues a multilayer perceptron needs (bias, SiLU, BF16 activations row-major and transposed, the
// pre-activations, FP32 output or accumulation).  Forward and backward passes of the MLP are chains of it:
//
//   forward   Z = H W^T + b, H' = silu(Z)                       A = H [batch][in],  B = W [out][in]
//   backward  dH = dZ W                                          A = dZ [batch][out], B = W^T [in][out]
//             dW = dZ^T H                                        A = dZ^T [out][batch], B = H^T [in][batch]
//             (weightGradKernel: the batch split over CTAs, the bias gradients from the same tiles)
//
// so every product is "A B^T" with both operands K-major, and the epilogue writes the transposed copies the
// next product reads.
#include <cuda_bf16.h>

#include "umma.cuh"
#include "zk_kernels.h"

namespace zk {

namespace {

constexpr int kGemmThreads = 256;  // the epilogue takes a row's columns with two threads
constexpr uint32_t kGemmBK = 64;
constexpr uint32_t kWaitLimit = 1u << 26;  // polls of an MMA-completion barrier before the kernel gives up

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) gemmKernel(const GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* sA = sm;                       // 128 x 64 bf16, canonical K-major
  unsigned char* sB = sm + 128 * kGemmBK * 2;   // BN x 64 bf16
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tslot;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const uint32_t m0 = blockIdx.x * 128u, n0 = blockIdx.y * BN, K = g.K;
  if (warp == 0) umma::alloc(&tslot, 128);
  if (tid == 0) mbarInit(&bar, 1);
  umma::fenceBeforeSync();
  __syncthreads();
  umma::fenceAfterSync();
  const uint32_t tmem = tslot;
  constexpr uint32_t idesc = umma::idescBf16(128, BN);
  uint32_t phase = 0;
  bool ok = true, pending = false;
  for (uint32_t k0 = 0; k0 < K && ok; k0 += kGemmBK) {
    const uint32_t kw = min(kGemmBK, K - k0), groups = kw >> 3;
    for (uint32_t v = tid; v < 128u * groups; v += kGemmThreads) {
      const uint32_t r = v / groups, kg = v % groups;
      umma::cpAsync16(sA + umma::kMajorOffset(r, kg * 8, 128), g.A + static_cast<size_t>(m0 + r) * K + k0 + kg * 8);
    }
    for (uint32_t v = tid; v < BN * groups; v += kGemmThreads) {
      const uint32_t r = v / groups, kg = v % groups;
      umma::cpAsync16(sB + umma::kMajorOffset(r, kg * 8, BN), g.B + static_cast<size_t>(n0 + r) * K + k0 + kg * 8);
    }
    umma::cpAsyncCommit();
    umma::cpAsyncWaitAll();
    umma::fenceAsyncShared();
    __syncthreads();
    if (tid == 0) {
      umma::fenceAfterSync();
      for (uint32_t i = 0; i < kw / 16; ++i) {
        const uint64_t da = umma::desc(umma::smem(sA) + i * 2 * 128 * 16, 128 * 16, 128);
        const uint64_t db = umma::desc(umma::smem(sB) + i * 2 * BN * 16, BN * 16, 128);
        umma::mma(tmem, da, db, idesc, k0 > 0 || i > 0);
      }
      umma::commit(&bar);
    }
    // The MMAs read sA / sB: the next chunk may overwrite them only once they have completed.  The vote keeps
    // every thread on the same path if one poll gives up.
    const bool done = mbarWait(&bar, phase, kWaitLimit);
    ok = __syncthreads_and(done) != 0;
    pending = !ok;
    phase ^= 1u;
  }
  if (!ok) {
    if (tid == 0) atomicExch(g.err, kDevTimeout);
    if (pending) mbarWait(&bar, phase ^ 1u, kWaitLimit);  // the MMAs in flight, before the TMEM goes away
  } else {
    umma::fenceAfterSync();
    const uint32_t row = m0 + (warp & 3u) * 32 + lane;  // a warp reads the 32 TMEM lanes of its number mod 4
    const uint32_t taddr = tmem + (((warp & 3u) * 32u) << 16);
#pragma unroll 1
    for (uint32_t c = 16 * (warp >> 2); c < BN; c += 32) {
      float v[16];
      umma::ld16(taddr + c, v);
      // A thread holds 16 adjacent columns of its row: the bf16 inputs and outputs move as two 16-byte accesses each.
      const size_t at0 = static_cast<size_t>(row) * g.N + n0 + c;  // 32-byte aligned: N and n0 + c are multiples of 16
      __align__(16) __nv_bfloat16 zb[16], hb[16], gb[16];
      if (g.gradOf) {
        reinterpret_cast<uint4*>(gb)[0] = __ldg(reinterpret_cast<const uint4*>(g.gradOf + at0));
        reinterpret_cast<uint4*>(gb)[1] = __ldg(reinterpret_cast<const uint4*>(g.gradOf + at0) + 1);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint32_t n = n0 + c + j;
        float z = v[j] + (g.bias ? __ldg(g.bias + n) : 0.0f);
        if (g.gradOf) z *= umma::siluGrad(__bfloat162float(gb[j]));
        if (g.C) g.C[at0 + j] = z;
        const float h = g.act ? umma::silu(z) : z;
        zb[j] = __float2bfloat16_rn(z);
        hb[j] = __float2bfloat16_rn(h);
        if (g.HT) g.HT[static_cast<size_t>(n) * g.M + row] = hb[j];
      }
      if (g.Z) {
        reinterpret_cast<uint4*>(g.Z + at0)[0] = reinterpret_cast<const uint4*>(zb)[0];
        reinterpret_cast<uint4*>(g.Z + at0)[1] = reinterpret_cast<const uint4*>(zb)[1];
      }
      if (g.H) {
        reinterpret_cast<uint4*>(g.H + at0)[0] = reinterpret_cast<const uint4*>(hb)[0];
        reinterpret_cast<uint4*>(g.H + at0)[1] = reinterpret_cast<const uint4*>(hb)[1];
      }
    }
  }
  umma::fenceBeforeSync();
  __syncthreads();
  if (warp == 0) umma::dealloc(tmem, 128);
}

// The weight and bias gradients of the three hidden layers over a batch: layer blockIdx.y's dW = dZ^T H (A = dZ^T, B = H^T,
// both K-major over the batch's rows) and db, the rows of A summed.  One CTA per (rows [k0, k1), layer), four 64-row chunks in
// flight; the parts are summed in order by sumPartsKernel.  128 x N is a single tile: with the whole batch in one CTA and no
// overlap the three products and three column sums of 8,192 rows took 1.0 ms; in 32 parts (two blocks of rows each) they take
// 15 us.
constexpr uint32_t kGradStages = 4;
__global__ void __launch_bounds__(kGemmThreads) weightGradKernel(const WeightGradArgs G) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) uint64_t bars[kGradStages];
  __shared__ uint32_t tslot;
  constexpr uint32_t kTile = 128 * kGemmBK * 2;  // bytes of a 128 x 64 chunk
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const WeightGradLayer Y = G.layer[blockIdx.y];
  const uint32_t k0 = blockIdx.x * G.perPart, k1 = min(k0 + G.perPart, G.rows), chunks = (k1 - k0) / kGemmBK;
  if (warp == 0) umma::alloc(&tslot, 128);
  if (tid == 0)
    for (uint32_t i = 0; i < kGradStages; ++i) mbarInit(&bars[i], 1);
  umma::fenceBeforeSync();
  __syncthreads();
  umma::fenceAfterSync();
  const uint32_t tmem = tslot, idesc = Y.N == 128 ? umma::idescBf16(128, 128) : umma::idescBf16(128, 16);
  auto load = [&](uint32_t c) {  // chunk c into its stage; a group of its own even past the last chunk
    if (c < chunks) {
      unsigned char* a = sm + (c % kGradStages) * 2 * kTile;
      const uint32_t k = k0 + c * kGemmBK;
      for (uint32_t v = tid; v < 128u * 8u; v += kGemmThreads)
        umma::cpAsync16(a + umma::kMajorOffset(v >> 3, (v & 7u) * 8, 128), Y.dZT + static_cast<size_t>(v >> 3) * G.rows + k + (v & 7u) * 8);
      for (uint32_t v = tid; v < Y.N * 8u; v += kGemmThreads)
        umma::cpAsync16(a + kTile + umma::kMajorOffset(v >> 3, (v & 7u) * 8, Y.N), Y.HT + static_cast<size_t>(v >> 3) * G.rows + k + (v & 7u) * 8);
    }
    umma::cpAsyncCommit();
  };
  float db = 0.0f;
  bool ok = true;
  int issued = -1;
  bool done = true;
  for (uint32_t c = 0; c + 1 < kGradStages; ++c) load(c);
  for (uint32_t c = 0; c < chunks; ++c) {
    umma::cpAsyncWait<kGradStages - 2>();  // this thread's part of chunk c has landed
    umma::fenceAsyncShared();
    ok = __syncthreads_and(done) != 0;  // every thread's; the bias sums have read chunk c - 1; one path if a poll gave up
    if (!ok) break;
    const unsigned char* a = sm + (c % kGradStages) * 2 * kTile;
    if (tid == 0) {
      umma::fenceAfterSync();
      for (uint32_t i = 0; i < kGemmBK / 16; ++i) {
        const uint64_t da = umma::desc(umma::smem(a) + i * 2 * 128 * 16, 128 * 16, 128);
        const uint64_t dh = umma::desc(umma::smem(a + kTile) + i * 2 * Y.N * 16, Y.N * 16, 128);
        umma::mma(tmem, da, dh, idesc, c > 0 || i > 0);
      }
      umma::commit(&bars[c % kGradStages]);
    }
    issued = static_cast<int>(c);
    // The next load overwrites the stage of chunk c - 1: once its MMAs have read it.
    if (c > 0 && c + kGradStages - 1 < chunks) done = mbarWait(&bars[(c - 1) % kGradStages], ((c - 1) / kGradStages) & 1u, kWaitLimit);
    if (done) load(c + kGradStages - 1);
    if (tid < 128)
#pragma unroll
      for (uint32_t q = 0; q < 8; ++q) {
        const uint4 v = *reinterpret_cast<const uint4*>(a + umma::kMajorOffset(tid, q * 8, 128));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) db += __uint_as_float(w[e] << 16), db += __uint_as_float(w[e] & 0xFFFF0000u);
      }
  }
  if (issued >= 0) {  // the last MMAs issued: all of them, in order
    done = mbarWait(&bars[issued % kGradStages], (static_cast<uint32_t>(issued) / kGradStages) & 1u, kWaitLimit);
    ok = __syncthreads_and(done && ok) != 0;
  }
  if (!ok) {
    if (tid == 0) atomicExch(G.err, kDevTimeout);
    umma::cpAsyncWaitAll();
  } else {
    umma::fenceAfterSync();
    float* part = G.part + static_cast<size_t>(blockIdx.x) * G.partStride;
    const uint32_t row = (warp & 3u) * 32 + lane, taddr = tmem + (((warp & 3u) * 32u) << 16);
#pragma unroll 1
    for (uint32_t c = 16 * (warp >> 2); c < Y.N; c += 32) {
      float v[16];
      umma::ld16(taddr + c, v);
      float4* dst = reinterpret_cast<float4*>(part + Y.offW + row * Y.N + c);
#pragma unroll
      for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
    if (tid < 128) part[Y.offB + tid] = db;
  }
  umma::fenceBeforeSync();
  __syncthreads();
  if (warp == 0) umma::dealloc(tmem, 128);
}

// out[c] = sum over the parts of part[p][c], in order.
__global__ void sumPartsKernel(const float* __restrict__ part, uint32_t parts, uint32_t n, uint32_t stride, float* __restrict__ out) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  float s = 0.0f;
#pragma unroll 8
  for (uint32_t p = 0; p < parts; ++p) s += __ldg(part + static_cast<size_t>(p) * stride + c);
  out[c] = s;
}

template <int BN>
cudaError_t launchGemmBN(const GemmArgs& g, cudaStream_t s) {
  const size_t smemBytes = (128 + BN) * kGemmBK * 2;
  // At least 55 KB per CTA (56 KB with the 1 KB the SM reserves per CTA) keeps at most four CTAs on an SM,
  // 4 x 128 TMEM columns, so an allocation never waits on another CTA; 58 KB allowed only three.
  const size_t dyn = smemBytes < 55 * 1024 ? 55 * 1024 : smemBytes;
  cudaError_t e = cudaFuncSetAttribute(gemmKernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn));
  if (e != cudaSuccess) return e;
  gemmKernel<BN><<<dim3(g.M / 128, g.N / BN), kGemmThreads, dyn, s>>>(g);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launchGemm(const GemmArgs& g, cudaStream_t s) {
  if (g.M == 0 || g.N == 0 || g.K == 0) return cudaSuccess;
  if (g.M % 128 || g.N % 16 || g.K % 16) return cudaErrorInvalidValue;
  if (g.N % 128 == 0) return launchGemmBN<128>(g, s);
  if (g.N % 64 == 0) return launchGemmBN<64>(g, s);
  if (g.N % 32 == 0) return launchGemmBN<32>(g, s);
  return launchGemmBN<16>(g, s);
}

cudaError_t launchWeightGrads(const WeightGradArgs& G, uint32_t parts, float* out, uint32_t n, cudaStream_t s) {
  if (G.rows % 128 || G.perPart % 128 || parts == 0) return cudaErrorInvalidValue;
  constexpr int dyn = kGradStages * 2 * 128 * kGemmBK * 2;  // 128 KB: one CTA on an SM
  cudaError_t e = cudaFuncSetAttribute(weightGradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
  if (e != cudaSuccess) return e;
  weightGradKernel<<<dim3(parts, 3), kGemmThreads, dyn, s>>>(G);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  sumPartsKernel<<<(n + 127) / 128, 128, 0, s>>>(G.part, parts, n, G.partStride, out);
  return cudaGetLastError();
}

}  // namespace zk
