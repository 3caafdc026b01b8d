// FP32 GEMM tiles: each element of C is the reference's sequential FFMA chain
// over k, restarted every KC = 384 and merged in order
// (src/gemm_kernel-inl.h:72, 161-224), so the result is the reference's bits.
//
// Bound: the FP32 pipe. The tensor cores have no IEEE FP32 chain, so the
// products run as packed FMAs (two adjacent rows of C per instruction), with
// 8 x 8 elements a thread and 64 x 32 a warp: 4 shared-memory reads of 16
// bytes feed 32 packed FMAs per k. Operand slabs of 16 k go through a
// three-stage cp.async ring, transposed on the way in if the operand is
// contiguous in k.
#include <algorithm>

#include "device.cuh"
#include "internal.h"

namespace hb {
namespace {

constexpr int kF32Kc = 384, kF32Kb = 16, kF32Stages = 3;
static_assert(kF32Kc % kF32Kb == 0, "a slab lies in one KC chunk");

template <int WM, int WN>
struct F32Tile {
  static constexpr int kBM = 64 * WM, kBN = 32 * WN, kThreads = 32 * WM * WN;
  static constexpr int kSA = kBM + 4, kSB = kBN + 4;  // row strides (floats)
  static constexpr int kStage = kF32Kb * (kSA + kSB);  // floats
  static constexpr int kSmem = kF32Stages * kStage * static_cast<int>(sizeof(float));
};

// A copy of n (4 or 16) bytes global -> shared; none of them are read (zeros
// are written) unless in.
template <int N>
__device__ __forceinline__ void CpAsyncF32(float* dst, const float* src, bool in) {
  if constexpr (N == 16) {
    CpAsync16(dst, src, in ? 16 : 0);
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                 :
                 : "r"(SmemAddr(dst)), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
  }
}

// One slab of an operand: s[q * LD + x] = op(x0 + x, k0 + q) for x < B and
// q < 16, zero outside (extent, k). xs, qs: the strides of x and q in memory.
// vec: x is contiguous and every group of four x (x0 + x a multiple of 4) is
// 16-byte aligned.
template <int B, int LD, int Threads>
__device__ __forceinline__ void LoadSlab(float* s, const float* p, long long xs, long long qs,
                                         int x0, int k0, int extent, int k, bool vec) {
  if (vec) {
#pragma unroll
    for (int l = 0; l < B * kF32Kb / 4 / Threads; ++l) {
      const int idx = threadIdx.x + l * Threads;
      const int x = idx % (B / 4) * 4, q = idx / (B / 4);
      float* dst = s + q * LD + x;
      const bool row = k0 + q < k;
      if (x0 + x + 3 < extent || !row) {
        const float* src = p + (x0 + x) + (k0 + q) * qs;
        CpAsyncF32<16>(dst, row ? src : p, row);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool in = x0 + x + e < extent;
          CpAsyncF32<4>(dst + e, in ? p + (x0 + x + e) + (k0 + q) * qs : p, in);
        }
      }
    }
    return;
  }
  const bool along_x = xs == 1;
#pragma unroll
  for (int l = 0; l < B * kF32Kb / Threads; ++l) {
    const int idx = threadIdx.x + l * Threads;
    const int x = along_x ? idx % B : idx / kF32Kb, q = along_x ? idx / B : idx % kF32Kb;
    const bool in = x0 + x < extent && k0 + q < k;
    CpAsyncF32<4>(s + q * LD + x, in ? p + (x0 + x) * xs + (k0 + q) * qs : p, in);
  }
}

__device__ __forceinline__ unsigned long long Pack2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
// Two IEEE FMAs (round to nearest) at once.
__device__ __forceinline__ void Fma2(unsigned long long& d, unsigned long long a,
                                     unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// Whether C(i, j) lies in a micro-tile of the reference's AVX-512 float
// kernel (MR 32, NR 12, MC 128, NC 4080) that crosses the diagonal: those
// tiles merge as alpha*acc + beta*C with two roundings (src/gemm-inl.h:93-130;
// src/gemm_kernel-inl.h:64-74).
__device__ __forceinline__ bool CrossingTileF32(int part, int m, int n, int i, int j) {
  constexpr int MR = 32, NR = 12, MC = 128, NC = 4080;
  const int i0 = i / MR * MR, mr = min(MR, min(MC - i0 % MC, m - i0));
  const int jc = j / NC * NC, j0 = jc + (j - jc) / NR * NR;
  const int nr = min(NR, min(NC, n - jc) - (j0 - jc));
  if (part == kLower) return !(i0 > j0 + nr - 1);
  return !(i0 + mr - 1 < j0);
}

template <int WM, int WN, bool kPart>
__global__ void __launch_bounds__(F32Tile<WM, WN>::kThreads, 512 / F32Tile<WM, WN>::kThreads)
    SgemmTileKernel(int m, int n, int k, float alpha, View<float> a, View<float> b, float beta,
                    float* c, long long ldc, int part, int veca, int vecb, const int* guard) {
  using Cfg = F32Tile<WM, WN>;
  constexpr int BM = Cfg::kBM, BN = Cfg::kBN, SA = Cfg::kSA, SB = Cfg::kSB;
  if (guard != nullptr && *guard != 0) return;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  // A tile wholly outside the triangle has nothing to do.
  if (kPart && (part == kLower ? m0 + BM - 1 < n0 : m0 > n0 + BN - 1)) return;
  extern __shared__ __align__(16) float f32_smem[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // This thread's rows: row0 + {0..3} and row0 + 32 + {0..3}; its columns
  // likewise with 16.
  const int row0 = warp % WM * 64 + lane % 8 * 4, col0 = warp / WM * 32 + lane / 8 * 4;
  const int slabs = (k + kF32Kb - 1) / kF32Kb;
  const auto load = [&](int slab) {
    if (slab < slabs) {
      float* sa = f32_smem + slab % kF32Stages * Cfg::kStage;
      LoadSlab<BM, SA, Cfg::kThreads>(sa, a.data, a.rs, a.cs, m0, slab * kF32Kb, m, k, veca);
      LoadSlab<BN, SB, Cfg::kThreads>(sa + kF32Kb * SA, b.data, b.cs, b.rs, n0, slab * kF32Kb,
                                      n, k, vecb);
    }
    CpAsyncCommit();
  };
  unsigned long long acc[4][8];  // row pairs x columns
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[r][j] = 0ull;
#pragma unroll
  for (int s = 0; s < kF32Stages - 1; ++s) load(s);
  for (int slab = 0; slab < slabs; ++slab) {
    CpAsyncWait<kF32Stages - 2>();
    __syncthreads();  // the slab is in place; the slab before it is read
    load(slab + kF32Stages - 1);
    const float* sa = f32_smem + slab % kF32Stages * Cfg::kStage + row0;
    const float* sb = f32_smem + slab % kF32Stages * Cfg::kStage + kF32Kb * SA + col0;
    const auto step = [&](int q) {
      const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(sa + q * SA);
      const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(sa + q * SA + 32);
      const float4 b0 = *reinterpret_cast<const float4*>(sb + q * SB);
      const float4 b1 = *reinterpret_cast<const float4*>(sb + q * SB + 16);
      const unsigned long long av[4] = {a0.x, a0.y, a1.x, a1.y};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned long long bb = Pack2(bv[j], bv[j]);
#pragma unroll
        for (int r = 0; r < 4; ++r) Fma2(acc[r][j], av[r], bb);
      }
    };
    const int k0 = slab * kF32Kb;
    if (k0 + kF32Kb <= k) {
#pragma unroll 8
      for (int q = 0; q < kF32Kb; ++q) step(q);
    } else {  // the padding is not multiplied: -0 + 0 would be +0
      for (int q = 0; q < k - k0; ++q) step(q);
    }
    if ((k0 + kF32Kb) % kF32Kc != 0 && slab + 1 < slabs) continue;
    // The chunk's end: merge into C, two columns' loads in flight at a time.
    const bool first = k0 < kF32Kc;
    const bool reads = !(first && beta == 0.f);
#pragma unroll
    for (int jj = 0; jj < 8; jj += 2) {
      const int i0 = m0 + row0, j0 = n0 + col0 + jj / 4 * 16 + jj % 4;
      float* cp = c + i0 + j0 * ldc;
      float cv[2][8];
#pragma unroll
      for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int di = e / 4 * 32 + e % 4;
          cv[d][e] = reads && i0 + di < m && j0 + d < n ? cp[di + d * ldc] : 0.f;
        }
#pragma unroll
      for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int di = e / 4 * 32 + e % 4;
          const unsigned long long pair = acc[e / 4 * 2 + e % 4 / 2][jj + d];
          const float r =
              alpha * __uint_as_float(static_cast<unsigned>(e % 2 == 0 ? pair : pair >> 32));
          float v;
          if (!first || beta == 1.f) v = r + cv[d][e];
          else if (beta == 0.f) v = r;
          else if (kPart && CrossingTileF32(part, m, n, i0 + di, j0 + d)) v = r + beta * cv[d][e];
          else v = fmaf(cv[d][e], beta, r);
          const bool in = !kPart || (part == kLower ? i0 + di >= j0 + d : i0 + di <= j0 + d);
          if (in && i0 + di < m && j0 + d < n) cp[di + d * ldc] = v;
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[r][j] = 0ull;
  }
}

template <int WM, int WN, bool kPart>
void LaunchTile(int m, int n, int k, float alpha, View<float> a, View<float> b, float beta,
                float* c, int ldc, Part part) {
  using Cfg = F32Tile<WM, WN>;
  static const cudaError_t attr =
      cudaFuncSetAttribute(SgemmTileKernel<WM, WN, kPart>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  if (Failed(attr, "sgemm attributes")) return;
  const auto aligned = [](const float* p, long long stride) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && stride % 4 == 0;
  };
  const int veca = a.rs == 1 && aligned(a.data, a.cs), vecb = b.cs == 1 && aligned(b.data, b.rs);
  const dim3 grid((m + Cfg::kBM - 1) / Cfg::kBM, (n + Cfg::kBN - 1) / Cfg::kBN);
  SgemmTileKernel<WM, WN, kPart><<<grid, Cfg::kThreads, Cfg::kSmem, Ctx().stream>>>(
      m, n, k, alpha, a, b, beta, c, ldc, static_cast<int>(part), veca, vecb, Ctx().guard);
  CountLaunch();
  LaunchFailed("sgemm tile");
}

}  // namespace

void SgemmTiles(int m, int n, int k, float alpha, View<float> a, View<float> b, float beta,
                float* c, int ldc, Part part) {
  const long long big = static_cast<long long>((m + 127) / 128) * ((n + 127) / 128);
  if (big >= Ctx().num_sms)
    part == kAll ? LaunchTile<2, 4, false>(m, n, k, alpha, a, b, beta, c, ldc, part)
                 : LaunchTile<2, 4, true>(m, n, k, alpha, a, b, beta, c, ldc, part);
  else
    part == kAll ? LaunchTile<1, 2, false>(m, n, k, alpha, a, b, beta, c, ldc, part)
                 : LaunchTile<1, 2, true>(m, n, k, alpha, a, b, beta, c, ldc, part);
}

}  // namespace hb
