// FP32 GEMM tiles: each element of C is the reference's sequential FFMA chain
// over k, restarted every KC = 384 and merged in order
// (src/gemm_kernel-inl.h:72, 161-224), so the result is the reference's bits.
//
// Bound: the FP32 pipe. The tensor cores have no IEEE FP32 chain, so the
// products run as packed FMAs (two adjacent rows of C per instruction), with
// 8 x 8 elements a thread and 64 x 32 a warp: 4 shared-memory reads of 16
// bytes feed 32 packed FMAs per k. Operand slabs of 16 k go through a
// three-stage cp.async ring, transposed on the way in if the operand is
// contiguous in k. 3001 x 2047 x 2500 NT: 4.08 ms with 4 x 4 elements a thread and
// no pipelining, 0.90 ms (34 TFLOP/s of the 71.8 measured) so; 3000^3 NN 6.9 -> 1.45.
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

// How an operand's slabs are copied: groups of four x (x contiguous and
// 16-byte aligned), single x (contiguous), single q (q contiguous; transposed on
// the way in).
enum SlabMode : int { kSlabVec = 0, kSlabX = 1, kSlabQ = 2 };

// One operand's slabs: s[q * LD + x] = op(x0 + x, k0 + q) for x < B and
// q < 16, zero outside. A thread's first element is fixed and the steps between
// its elements are constants, so a slab costs a pointer and one address a copy.
template <int Mode, int B, int LD, int Threads>
struct SlabLoader {
  static constexpr int kPer = Mode == kSlabVec ? 4 : 1;
  static constexpr int kCopies = B * kF32Kb / Threads / kPer;
  static constexpr int kDx = Mode == kSlabQ ? Threads / kF32Kb : 0;
  static constexpr int kDq = Mode == kSlabQ ? 0 : Threads * kPer / B;
  const float* p;  // this thread's first element of the next slab
  int left;        // elements of the operand from its first x on

  static __device__ __forceinline__ int X() {
    return Mode == kSlabQ ? threadIdx.x / kF32Kb : threadIdx.x % (B / kPer) * kPer;
  }
  static __device__ __forceinline__ int Q() {
    return Mode == kSlabQ ? threadIdx.x % kF32Kb : threadIdx.x / (B / kPer);
  }
  __device__ __forceinline__ SlabLoader(const float* data, long long ld, int x0, int n)
      : p(Mode == kSlabQ ? data + (x0 + X()) * ld + Q() : data + (x0 + X()) + Q() * ld),
        left(n - x0 - X()) {}
  // kend: rows of the slab that exist (16 but for the last). `safe` is an
  // address for copies that read nothing.
  __device__ __forceinline__ void Load(float* s, int kend, long long ld, const float* safe) {
    float* dst = s + Q() * LD + X();
#pragma unroll
    for (int l = 0; l < kCopies; ++l) {
      const float* src = p + (Mode == kSlabQ ? l * kDx * ld : l * kDq * ld);
      float* to = dst + l * (kDq * LD + kDx);
      const bool row = Q() + l * kDq < kend;
      if constexpr (Mode == kSlabVec) {
        if (left >= 4) {
          CpAsyncF32<16>(to, row ? src : safe, row);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            CpAsyncF32<4>(to + e, row && e < left ? src + e : safe, row && e < left);
        }
      } else {
        const bool in = row && l * kDx < left;
        CpAsyncF32<4>(to, in ? src : safe, in);
      }
    }
    p += Mode == kSlabQ ? kF32Kb : kF32Kb * ld;
  }
};

__device__ __forceinline__ unsigned long long Swap2(unsigned long long v) {
  unsigned long long r;
  asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tmov.b64 %0, {hi, lo};\n\t}"
      : "=l"(r)
      : "l"(v));
  return r;
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

template <int WM, int WN, bool kPart, int ModeA, int ModeB>
__global__ void __launch_bounds__(F32Tile<WM, WN>::kThreads, 512 / F32Tile<WM, WN>::kThreads)
    SgemmTileKernel(int m, int n, int k, float alpha, const float* a, long long lda,
                    const float* b, long long ldb, float beta, float* c, long long ldc, int part,
                    Guard guard) {
  using Cfg = F32Tile<WM, WN>;
  constexpr int BM = Cfg::kBM, BN = Cfg::kBN, SA = Cfg::kSA, SB = Cfg::kSB;
  if (guard.Stops()) return;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  // A tile wholly outside the triangle has nothing to do.
  if (kPart && (part == kLower ? m0 + BM - 1 < n0 : m0 > n0 + BN - 1)) return;
  extern __shared__ __align__(16) float f32_smem[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // This thread's rows: row0 + {0..3} and row0 + 32 + {0..3}; its columns
  // likewise with 16.
  const int row0 = warp % WM * 64 + lane % 8 * 4, col0 = warp / WM * 32 + lane / 8 * 4;
  const int slabs = (k + kF32Kb - 1) / kF32Kb;
  SlabLoader<ModeA, BM, SA, Cfg::kThreads> la(a, lda, m0, m);
  SlabLoader<ModeB, BN, SB, Cfg::kThreads> lb(b, ldb, n0, n);
  const auto load = [&](int slab) {
    if (slab < slabs) {
      float* sa = f32_smem + slab % kF32Stages * Cfg::kStage;
      la.Load(sa, k - slab * kF32Kb, lda, a);
      lb.Load(sa + kF32Kb * SA, k - slab * kF32Kb, ldb, b);
    }
    CpAsyncCommit();
  };
  // acc[r][j], rows 2 r and 2 r + 1 of the thread's: the first with column j,
  // the second with column j ^ 1, so that a packed FMA takes B's columns as
  // they lie or swapped.
  unsigned long long acc[4][8];
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
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(sb + q * SB);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(sb + q * SB + 16);
      const unsigned long long av[4] = {a0.x, a0.y, a1.x, a1.y};
      const unsigned long long bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned long long swapped = Swap2(bv[j]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          Fma2(acc[r][2 * j], av[r], bv[j]);
          Fma2(acc[r][2 * j + 1], av[r], swapped);
        }
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
          const unsigned long long pair = acc[e / 4 * 2 + e % 4 / 2][(jj + d) ^ (e % 2)];
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

struct TileCall {
  int m, n, k;
  float alpha;
  View<float> a, b;
  float beta;
  float* c;
  int ldc;
  Part part;
};

template <int WM, int WN, bool kPart, int ModeA, int ModeB>
void LaunchModes(const TileCall& t) {
  using Cfg = F32Tile<WM, WN>;
  static PerDevice<cudaError_t> attr;
  const auto set = [] {
    return cudaFuncSetAttribute(SgemmTileKernel<WM, WN, kPart, ModeA, ModeB>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  };
  if (Failed(attr.Get(set), "sgemm attributes")) return;
  const dim3 grid((t.m + Cfg::kBM - 1) / Cfg::kBM, (t.n + Cfg::kBN - 1) / Cfg::kBN);
  SgemmTileKernel<WM, WN, kPart, ModeA, ModeB>
      <<<grid, Cfg::kThreads, Cfg::kSmem, Ctx().stream>>>(
          t.m, t.n, t.k, t.alpha, t.a.data, t.a.ld(), t.b.data, t.b.ld(), t.beta, t.c, t.ldc,
          static_cast<int>(t.part), Ctx().guard);
  CountLaunch();
  LaunchFailed("sgemm tile");
}

// The copy mode of an operand whose x has stride xs and whose q has stride qs.
int ModeOf(const float* p, long long xs, long long qs) {
  if (xs != 1) return kSlabQ;
  return reinterpret_cast<uintptr_t>(p) % 16 == 0 && qs % 4 == 0 ? kSlabVec : kSlabX;
}

template <int WM, int WN, bool kPart, int ModeA>
void LaunchModeA(const TileCall& t, int mode_b) {
  if (mode_b == kSlabVec) LaunchModes<WM, WN, kPart, ModeA, kSlabVec>(t);
  else if (mode_b == kSlabX) LaunchModes<WM, WN, kPart, ModeA, kSlabX>(t);
  else LaunchModes<WM, WN, kPart, ModeA, kSlabQ>(t);
}

template <int WM, int WN, bool kPart>
void LaunchTile(const TileCall& t) {
  const int ma = ModeOf(t.a.data, t.a.rs, t.a.cs), mb = ModeOf(t.b.data, t.b.cs, t.b.rs);
  if (ma == kSlabVec) LaunchModeA<WM, WN, kPart, kSlabVec>(t, mb);
  else if (ma == kSlabX) LaunchModeA<WM, WN, kPart, kSlabX>(t, mb);
  else LaunchModeA<WM, WN, kPart, kSlabQ>(t, mb);
}

}  // namespace

void SgemmTiles(int m, int n, int k, float alpha, View<float> a, View<float> b, float beta,
                float* c, int ldc, Part part) {
  const TileCall t = {m, n, k, alpha, a, b, beta, c, ldc, part};
  // 128 x 128 tiles once they fill the SMs; else 128 x 64 (1024^3: 113 us against
  // 158 with either of the others, 500^3: 70 against 86), else 64 x 64.
  const long long rows = (m + 127) / 128;
  if (rows * ((n + 127) / 128) >= Ctx().num_sms)
    part == kAll ? LaunchTile<2, 4, false>(t) : LaunchTile<2, 4, true>(t);
  else if (rows * ((n + 63) / 64) >= 24)
    part == kAll ? LaunchTile<2, 2, false>(t) : LaunchTile<2, 2, true>(t);
  else
    part == kAll ? LaunchTile<1, 2, false>(t) : LaunchTile<1, 2, true>(t);
}

}  // namespace hb
