// Level-3 routines around the GEMM kernels: the FP32 TRMM product (FFMA on the CUDA
// cores, the reference's FP32 order with KC = 384), the recursive TRSM with
// its base substitution kernel, SYRK, and the reference-semantics wrappers
// (argument-independent quick returns and alpha scaling).
#include <algorithm>
#include <cstdio>
#include <utility>

#include "device.cuh"
#include "internal.h"
#include "lane_solve.cuh"

namespace hb {
namespace {

// ---------------------------------------------------------------------------
// FP32 GEMM with a triangular operand (TRMM; the other products are in
// gemm_f32.cu): 64 x 64 tile per 256-thread CTA, 4 x 4 outputs per thread, each a
// sequential FFMA chain over k restarted every 384 (src/gemm_kernel-inl.h:72).
constexpr int kSB = 64, kSK = 16;

// k range [*kb, *ke) the reference multiplies for C(i, j) when an operand is
// triangular: NonZeroRange of the AVX-512 float micro-tile (MR 32, NR 12,
// MC 128, NC 4080) holding C(i, j) (src/gemm-inl.h:62-85). Row tiles start at
// multiples of 32 (MC is a multiple of MR), column tiles at multiples of 12
// within NC blocks.
__device__ __forceinline__ void TriRangeF(int tri, int m, int n, int k, int i, int j, int* kb,
                                          int* ke) {
  *kb = 0;
  *ke = k;
  if (tri == kTriALower || tri == kTriAUpper) {
    const int i0 = i & ~31, mr = min(32, m - i0);
    if (tri == kTriALower) *ke = min(k, i0 + mr);
    else *kb = i0;
  } else if (tri == kTriBLower || tri == kTriBUpper) {
    constexpr int NR = 12, NC = 4080;
    const int jc = j / NC * NC, jr = (j - jc) / NR * NR;
    const int nr = min(NR, min(NC, n - jc) - jr);
    if (tri == kTriBLower) *kb = jc + jr;
    else *ke = min(k, jc + jr + nr);
  }
}

// `tri` (TRMM): each element's chain runs over its micro-tile's k range only,
// and a chunk outside that range leaves the element unmerged, as the
// reference skips the micro-tile (src/gemm-inl.h:202-209).
__global__ void __launch_bounds__(256)
    SgemmKernel(int m, int n, int k, float alpha, View<float> a, View<float> b,
                float beta, float* c, long long ldc, int tri, Guard guard) {
  if (guard.Stops()) return;
  __shared__ float sa[kSK][kSB + 4];
  __shared__ float sb[kSK][kSB + 4];
  const int m0 = blockIdx.x * kSB, n0 = blockIdx.y * kSB;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4] = {}, cacc[4][4] = {};
  const int kchunk = 384;
  // Row- and column-dependent bounds of the elements' k ranges (tri).
  int rkb[4], rke[4], ckb[4], cke[4];
  const int tri_a = (tri == kTriALower || tri == kTriAUpper) ? tri : kTriNone;
  const int tri_b = (tri == kTriBLower || tri == kTriBUpper) ? tri : kTriNone;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    TriRangeF(tri_a, m, n, k, m0 + tx + 16 * r, 0, &rkb[r], &rke[r]);
    TriRangeF(tri_b, m, n, k, 0, n0 + ty + 16 * r, &ckb[r], &cke[r]);
  }
  for (int k0 = 0; k0 < k; k0 += kSK) {
    for (int idx = threadIdx.x; idx < kSK * kSB; idx += 256) {
      const int kk = idx / kSB, mm = idx % kSB;
      const int gi = m0 + mm, gk = k0 + kk;
      sa[kk][mm] = (gi < m && gk < k) ? a.data[gi * a.rs + gk * a.cs] : 0.f;
      const int gj = n0 + mm;
      sb[kk][mm] = (gj < n && gk < k) ? b.data[gk * b.rs + gj * b.cs] : 0.f;
    }
    __syncthreads();
    const int kend = min(kSK, k - k0);
    for (int kk = 0; kk < kend; ++kk) {
      float av[4], bv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) av[r] = sa[kk][tx + 16 * r];
#pragma unroll
      for (int q = 0; q < 4; ++q) bv[q] = sb[kk][ty + 16 * q];
      const int kg = k0 + kk;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (kg >= max(rkb[r], ckb[q]) && kg < min(rke[r], cke[q]))
            acc[r][q] = fmaf(av[r], bv[q], acc[r][q]);
      if ((kg + 1) % kchunk == 0 || kg + 1 == k) {
        const bool first = kg < kchunk;
        const int c_lo = kg / kchunk * kchunk, c_hi = kg + 1;
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = m0 + tx + 16 * r, j = n0 + ty + 16 * q;
            const float rr = alpha * acc[r][q];
            if (!first && max(max(rkb[r], ckb[q]), c_lo) >= min(min(rke[r], cke[q]), c_hi)) {
              // Outside the element's k range: not merged.
            } else if (first) {
              if (i < m && j < n) {
                if (beta == 0.f) {
                  cacc[r][q] = rr;
                } else {
                  const float cin = c[i + j * ldc];
                  if (beta == 1.f) {
                    cacc[r][q] = rr + cin;
                  } else {
                    cacc[r][q] = fmaf(cin, beta, rr);
                  }
                }
              }
            } else {
              cacc[r][q] = rr + cacc[r][q];
            }
            acc[r][q] = 0.f;
          }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = m0 + tx + 16 * r, j = n0 + ty + 16 * q;
      if (i < m && j < n) c[i + j * ldc] = cacc[r][q];
    }
}

// ---------------------------------------------------------------------------
// TRSM base: solves X*T = B for independent rows of X (src/trsm-inl.h:107-174)
// with T (r x r, r <= 32) read from a strided view. Columns are solved in
// "solve order" s = 0..r-1 (column r-1-s for lower, s for upper):
// b_j -= x_q t(q, j) as fma(-x_q, t, b) for every solved q in that order, then
// x_j = b_j * (1/t(j, j)). Element (row, col q) of X is
// x[row * xs_row + q * xs_col].
// The recursion's node of at most 64 columns (src/trsm.cc:87-135: a base solve,
// the product, a base solve) for many rows in one launch: a CTA takes kBaseRows
// of them, two a warp. Rows that are contiguous in memory across each other
// (right side) go through shared memory, so that both sides read and write
// whole sectors.
constexpr int kBaseThreads = 256, kBaseRows = 2 * kBaseThreads / 32, kBaseW = 64;
template <typename T>
__global__ void __launch_bounds__(kBaseThreads)
    TrsmBaseKernel(View<T> tri, int lower, int unit, int r, int rows, T* x,
                   long long xs_row, long long xs_col, Guard guard) {
  if (guard.Stops()) return;
  constexpr int ld = kBaseW + 1;
  __shared__ T st[kBaseW * ld];  // st[s][u] = T(col(s), col(u)) in solve order, s < u
  __shared__ T sinv[kBaseW];
  __shared__ T xt[kBaseRows][kBaseW + 1];
  const int tid = threadIdx.x, lane = tid % 32, i0 = tid / 32 * 2;
  const int row0 = blockIdx.x * kBaseRows, n = min(kBaseRows, rows - row0);
  const bool across = xs_row == 1;
  x += row0 * xs_row;
  if (across) {
    for (int idx = tid; idx < kBaseRows * r; idx += kBaseThreads) {
      const int i = idx % kBaseRows, c = idx / kBaseRows;
      if (i < n) xt[i][c] = x[i + c * xs_col];
    }
  }
  const int w = r > 32 ? 64 : 32;
  const bool rows_fast = tri.rs == 1;
  for (int idx = tid; idx < w * w; idx += kBaseThreads) {
    const int s = rows_fast ? idx % w : idx / w, u = rows_fast ? idx / w : idx % w;
    T v = T(0);
    if (s < r && u < r && (s < u || (s == u && !unit))) {
      const int q = lower ? r - 1 - s : s, j = lower ? r - 1 - u : u;
      v = tri.data[q * tri.rs + j * tri.cs];
    }
    st[s * ld + u] = v;
    if (s == u) sinv[s] = s < r && !unit ? T(1) / v : T(1);
  }
  __syncthreads();
  // The half solved first: the leading 32 columns (upper) or the others (lower),
  // which is 32 columns' solve order from its start.
  const int f = r <= 32 ? r : (lower ? r - 32 : 32), g = r - f;
  // Column of step s, in elements from a row's first.
  const auto col = [&](int s) { return lower ? r - 1 - s : s; };
  T y[2], z[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const T* xr = across ? xt[i0 + i] : x + (i0 + i) * xs_row;
    const long long xc = across ? 1 : xs_col;
    const bool in = i0 + i < n;
    y[i] = in && lane < f ? xr[col(lane) * xc] : T(0);
    z[i] = in && lane < g ? xr[col(f + lane) * xc] : T(0);
  }
  LaneSolve<T, 2>(st, ld, sinv[lane], unit, f, y);
  if (g > 0) {
    // z -= y T: one chain an element, over the columns in memory order.
    T acc[2] = {T(0), T(0)};
#pragma unroll 4
    for (int e = 0; e < f; ++e) {
      const int q = lower ? f - 1 - e : e;
      const T t = st[q * ld + f + lane];
      acc[0] = fma(__shfl_sync(0xffffffffu, y[0], q), t, acc[0]);
      acc[1] = fma(__shfl_sync(0xffffffffu, y[1], q), t, acc[1]);
    }
    z[0] = T(-1) * acc[0] + z[0];
    z[1] = T(-1) * acc[1] + z[1];
    LaneSolve<T, 2>(st + f * ld + f, ld, sinv[min(f + lane, kBaseW - 1)], unit, g, z);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    T* xr = across ? xt[i0 + i] : x + (i0 + i) * xs_row;
    const long long xc = across ? 1 : xs_col;
    if (i0 + i >= n) continue;
    if (lane < f) xr[col(lane) * xc] = y[i];
    if (lane < g) xr[col(f + lane) * xc] = z[i];
  }
  if (across) {
    __syncthreads();
    for (int idx = tid; idx < kBaseRows * r; idx += kBaseThreads) {
      const int i = idx % kBaseRows, c = idx / kBaseRows;
      if (i < n) x[i + c * xs_col] = xt[i][c];
    }
  }
}

// The base solve (r <= 32) with one thread a row: the row in registers in solve order
// (static indices), the triangle in shared memory, two columns a pass. Bound by the
// loads once there are rows enough for the SMs; TrsmBaseKernel, a lane an element, is
// bound by its shuffles by then (right side, 32 x 400000: 312 us, 93 so).
template <typename T>
__global__ void __launch_bounds__(128)
    TrsmRowsKernel(View<T> tri, int lower, int unit, int r, int rows, T* x, long long xs_row,
                   long long xs_col, Guard guard) {
  if (guard.Stops()) return;
  __shared__ T st[32][33];  // st[s][u] = T(col(s), col(u)) in solve order, s < u
  __shared__ T sinv[32];
  for (int idx = threadIdx.x; idx < 32 * 32; idx += blockDim.x) {
    const int s = idx / 32, u = idx % 32;
    T v = T(0);
    if (s < r && u < r && (s < u || (s == u && !unit))) {
      const int q = lower ? r - 1 - s : s, j = lower ? r - 1 - u : u;
      v = tri.data[q * tri.rs + j * tri.cs];
    }
    st[s][u] = v;
    if (s == u) sinv[s] = s < r && !unit ? T(1) / v : T(1);
  }
  __syncthreads();
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  T* xr = x + row * xs_row;
  T y[32];
#pragma unroll
  for (int s = 0; s < 32; ++s)
    y[s] = s < r ? xr[(lower ? r - 1 - s : s) * xs_col] : T(0);
#pragma unroll
  for (int step = 0; step < 32; step += 2) {
    if (step >= r) break;
    T acc0 = y[step], acc1 = y[step + 1];
#pragma unroll
    for (int s = 0; s < step; ++s) {
      acc0 = fma(-y[s], st[s][step], acc0);
      acc1 = fma(-y[s], st[s][step + 1], acc1);
    }
    if (!unit) acc0 = acc0 * sinv[step];
    y[step] = acc0;
    acc1 = fma(-acc0, st[step][step + 1], acc1);
    if (!unit) acc1 = acc1 * sinv[step + 1];
    y[step + 1] = acc1;
  }
#pragma unroll
  for (int s = 0; s < 32; ++s)
    if (s < r) xr[(lower ? r - 1 - s : s) * xs_col] = y[s];
}

// Rows from which a base solve goes to TrsmRowsKernel: where its few long-running
// threads (27 us a call whatever the number of rows) meet the lanes' time. A call with
// 32 columns, lanes and rows in us: right side FP64 8000 29 and 28, 16000 34 and 27,
// FP32 12000 27 and 26; left side, whose loads are not coalesced here, FP64 12000 32
// and 30, FP32 24000 33 and 34, 32000 36 and 34.
template <typename T>
int RowsFrom(bool left) {
  if (sizeof(T) == 8) return left ? 12000 : 8000;
  return left ? 24000 : 12000;
}

// Rows from which a node of 33 to 64 columns is two such solves and a product in
// launches of their own. Lanes and launches in us: FP64 right side 64 columns 16000 52 and
// 44, 400000 733 and 250, 33 columns 16000 43 and 42; left side 32000 81 and 66, 24000
// 55 and 55 (33 columns); FP32 right side 32000 60 and 51, left side 48 columns 64000
// 88 and 82, 64 columns 100000 137 and 150, 400000 469 and 431.
template <typename T>
int SplitFrom(bool left, int r) {
  if (sizeof(T) == 8) return left ? 24000 : 16000;
  return !left ? 32000 : r <= 48 ? 64000 : 256000;
}

// A subtree of the TRSM recursion (65 to kTcRows rows of the triangle) in one
// launch. Bound by latency: up to 16 dependent base solves with an update after
// each, so all that does not depend on X is on the chip beforehand. A cluster of
// kTcCtas CTAs takes kTcRhs right-hand sides (their columns are independent): its
// CTAs hold the triangle's 16-row strips in turn (at most 180 KiB each in FP64, 196.5
// with the base triangles) in shared memory, copied once while the first base is
// solved, and the next base triangle is copied while one is solved. A base solve gives
// each warp a right-hand side, an update each warp 16 x 8 tiles of the strips its CTA
// holds; every element's chains, restarted every KC, and merges are the GEMM kernels'.
// Steps end with a cluster barrier, which is some 1.5 us less than a grid barrier; X
// goes through L2. The right side is the left side of the transposed system (each
// product's factors change places).
// 512 rows: few right-hand sides 80 us (168 as a cooperative launch over the grid),
// 64 a cluster 120 us (512 right-hand sides 140 us with 8 columns a CTA).
constexpr int kTcRows = 512, kTcThreads = 256, kTcCtas = 8, kTcRhs = 64;
constexpr int kTcStrip = 16, kTcStrips = kTcRows / kTcStrip / kTcCtas;  // a CTA's strips
constexpr int kTcLd = kTcStrip + 4;  // conflict-free fragments

template <typename T>
constexpr int kTcKc = sizeof(T) == 8 ? 256 : 384;

template <typename T>
constexpr int TcSmem() {
  // The strips' columns of the CTA that has the most: 32-row blocks below a
  // strip's own, for the strips 7, 15, 23, 31.
  constexpr int cols = 32 * (3 + 7 + 11 + 15);
  return static_cast<int>(sizeof(T)) * (cols * kTcLd + 2 * 32 * 33);
}

template <typename T>
struct TrsmClusterArgs {
  View<T> tri;  // T of T X = B
  int lower, unit, r, other;
  T* x;         // element (row, right-hand side) at row * xs + rhs * xr
  long long xs, xr;
  Guard guard;
};

__device__ __forceinline__ void TcBarrier() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}

template <typename T>
__device__ __forceinline__ void TcCopy(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(SmemAddr(dst)), "l"(src),
               "n"(sizeof(T))
               : "memory");
}

// A 16 x 8 tile of C -= A X: a(row, q) at a[q * kTcLd + row] in shared memory, x and c
// in global memory, kk terms; rows < mr and columns < nc exist.
template <typename T>
__device__ __forceinline__ void TcTile(const T* a, const T* x, T* c, long long xs, long long xr,
                                       int kk, int mr, int nc) {
  const int lane = threadIdx.x % 32, g = lane >> 2, t = lane & 3;
  T cv[4], acc[4] = {T(0), T(0), T(0), T(0)};
  bool in[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = g + (e >> 1) * 8, j = 2 * t + (e & 1);
    in[e] = i < mr && j < nc;
    cv[e] = in[e] ? __ldcg(c + i * xs + j * xr) : T(0);
  }
  if constexpr (sizeof(T) == 8) {
    constexpr int kSteps = 8;  // k8 steps whose X is in flight together
    for (int k0 = 0; k0 < kk; k0 += 8 * kSteps) {
      T fb[kSteps][2];
#pragma unroll
      for (int s = 0; s < kSteps; ++s)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = k0 + 8 * s + 4 * h + t;
          fb[s][h] = q < kk && g < nc ? __ldcg(x + q * xs + g * xr) : 0.0;
        }
#pragma unroll
      for (int s = 0; s < kSteps; ++s) {
        if (k0 + 8 * s >= kk) break;
        const int q = k0 + 8 * s + t;
        const T* fa = a + q * kTcLd + g;
        // Past kk: -0 times +0, which leaves every sum as it is.
        const bool i0 = q < kk, i1 = q + 4 < kk;
        const T a0 = i0 ? fa[0] : -0.0, a1 = i0 ? fa[8] : -0.0;
        const T a2 = i1 ? fa[4 * kTcLd] : -0.0, a3 = i1 ? fa[4 * kTcLd + 8] : -0.0;
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
            "{%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+d"(acc[0]), "+d"(acc[1]), "+d"(acc[2]), "+d"(acc[3])
            : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(fb[s][0]), "d"(fb[s][1]));
      }
    }
  } else {
    constexpr int kSteps = 16;
    for (int k0 = 0; k0 < kk; k0 += kSteps) {
      T fb[kSteps][2];
#pragma unroll
      for (int s = 0; s < kSteps; ++s)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          fb[s][h] = k0 + s < kk && 2 * t + h < nc ? __ldcg(x + (k0 + s) * xs + (2 * t + h) * xr)
                                                   : T(0);
#pragma unroll
      for (int s = 0; s < kSteps; ++s) {
        if (k0 + s >= kk) break;
        const T a0 = a[(k0 + s) * kTcLd + g], a1 = a[(k0 + s) * kTcLd + g + 8];
        acc[0] = fma(a0, fb[s][0], acc[0]);
        acc[1] = fma(a0, fb[s][1], acc[1]);
        acc[2] = fma(a1, fb[s][0], acc[2]);
        acc[3] = fma(a1, fb[s][1], acc[3]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = g + (e >> 1) * 8, j = 2 * t + (e & 1);
    if (in[e]) __stcg(c + i * xs + j * xr, T(-1) * acc[e] + cv[e]);
  }
}

template <typename T>
__global__ void __launch_bounds__(kTcThreads) TrsmClusterKernel(TrsmClusterArgs<T> p) {
  if (p.guard.Stops()) return;
  extern __shared__ __align__(16) unsigned char tc_smem[];
  T* tri[2] = {reinterpret_cast<T*>(tc_smem), reinterpret_cast<T*>(tc_smem) + 32 * 33};
  T* strips = tri[1] + 32 * 33;
  const int rank = blockIdx.x % kTcCtas, j0 = blockIdx.x / kTcCtas * kTcRhs;
  const int nrhs = min(kTcRhs, p.other - j0);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  T* x = p.x + j0 * p.xr;
  const bool rows_fast = p.tri.rs == 1;
  const int blocks = (p.r + 31) / 32;
  // Base triangle number t (in the order they are solved), in solve order:
  // st[s][u] = T(row u, column s), s <= u. A thread copies the same four (s, u) of
  // each, from the block's corner in solve order.
  const long long step_r = p.lower ? p.tri.rs : -p.tri.rs, step_c = p.lower ? p.tri.cs : -p.tri.cs;
  const int fast = threadIdx.x % 32, slow = threadIdx.x / 32;
  const auto load_base = [&](int t) {
    if (t >= blocks || rank >= nrhs) return;
    const int off = 32 * (p.lower ? t : blocks - 1 - t), n = min(32, p.r - off);
    const int corner = p.lower ? off : off + n - 1;
    const T* src = p.tri.data + corner * (p.tri.rs + p.tri.cs);
    T* st = tri[t & 1];
#pragma unroll
    for (int i = 0; i < 32; i += kTcThreads / 32) {
      const int s = rows_fast ? slow + i : fast, u = rows_fast ? fast : slow + i;
      if (s < u ? u < n : s == u && u < n && !p.unit)
        TcCopy(st + s * 33 + u, src + u * step_r + s * step_c);
    }
  };
  load_base(0);
  CpAsyncCommit();
  // This CTA's strips: number rank + kTcCtas i, its columns solved before its block.
  int at[kTcStrips], first[kTcStrips];
  int used = 0;
#pragma unroll
  for (int i = 0; i < kTcStrips; ++i) {
    const int row0 = (rank + kTcCtas * i) * kTcStrip, blk = row0 / 32;
    const int q0 = p.lower ? 0 : 32 * (blk + 1);
    const int n = row0 < p.r ? max(0, (p.lower ? 32 * blk : p.r) - q0) : 0;
    at[i] = used;
    first[i] = q0;
    T* dst = strips + used;
    used += n * kTcLd;
    for (int idx = threadIdx.x; idx < n * kTcStrip; idx += kTcThreads) {
      const int il = rows_fast ? idx % kTcStrip : idx / n, q = rows_fast ? idx / kTcStrip : idx % n;
      if (row0 + il < p.r)
        TcCopy(dst + q * kTcLd + il, p.tri.data + (row0 + il) * p.tri.rs + (q0 + q) * p.tri.cs);
    }
  }
  CpAsyncCommit();
  int s_off[8], s_r[8], s_ph[8];
  int sp = 0, base = 0;
  s_off[0] = 0;
  s_r[0] = p.r;
  s_ph[0] = 0;
  while (sp >= 0) {
    const int off = s_off[sp], rr = s_r[sp];
    if (rr <= 32) {
      if (base == 0) CpAsyncWait<1>();
      else CpAsyncWait<0>();
      __syncthreads();
      const T* st = tri[base & 1];
      load_base(++base);
      CpAsyncCommit();
      for (int j = rank + kTcCtas * warp; j < nrhs; j += kTcCtas * (kTcThreads / 32)) {
        T* e = x + (off + (p.lower ? lane : rr - 1 - lane)) * p.xs + j * p.xr;
        T y[1] = {lane < rr ? __ldcg(e) : T(0)};
        const T inv = lane < rr && !p.unit ? T(1) / st[lane * 33 + lane] : T(1);
        LaneSolve<T, 1>(st, 33, inv, p.unit, rr, y);
        if (lane < rr) __stcg(e, y[0]);
      }
      TcBarrier();
      --sp;
      continue;
    }
    const int r1 = max(32, (rr / 2) / 32 * 32), r2 = rr - r1;
    const int ph = s_ph[sp]++;
    if (ph == 2) {
      --sp;
      continue;
    }
    if (ph == 1) {
      if (base == 1) {  // the strips have arrived
        CpAsyncWait<0>();
        __syncthreads();
      }
      // The half just solved, columns [q0, q0 + kk), on the rows of the other.
      const int c0 = p.lower ? off + r1 : off, c1 = p.lower ? off + rr : off + r1;
      const int q0 = p.lower ? off : off + r1, kk = p.lower ? r1 : r2;
      const int tiles = (nrhs + 7) / 8;
      int unit = 0;
#pragma unroll
      for (int i = 0; i < kTcStrips; ++i) {
        const int row0 = (rank + kTcCtas * i) * kTcStrip;
        if (row0 < c0 || row0 >= c1) continue;
        for (int ct = 0; ct < tiles; ++ct, ++unit) {
          if (unit % (kTcThreads / 32) != warp) continue;
          T* xc = x + 8 * ct * p.xr;
          for (int k0 = 0; k0 < kk; k0 += kTcKc<T>)
            TcTile<T>(strips + at[i] + (q0 + k0 - first[i]) * kTcLd, xc + (q0 + k0) * p.xs,
                      xc + row0 * p.xs, p.xs, p.xr, min(kTcKc<T>, kk - k0), c1 - row0,
                      nrhs - 8 * ct);
        }
      }
      TcBarrier();
    }
    // ph 0: the half solved first (the leading one of a lower triangle).
    const bool leading = (ph == 0) == (p.lower != 0);
    ++sp;
    s_off[sp] = leading ? off : off + r1;
    s_r[sp] = leading ? r1 : r2;
    s_ph[sp] = 0;
  }
}

template <typename T>
bool TrsmCluster(bool left, View<T> tri, bool lower, bool unit, int r, int other, T* b, int ldb) {
  Context& ctx = Ctx();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((other + kTcRhs - 1) / kTcRhs * kTcCtas);
  cfg.blockDim = dim3(kTcThreads);
  cfg.dynamicSmemBytes = TcSmem<T>();
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kTcCtas;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  // Right-hand sides of one wave: the clusters that the GPU holds at a time (15 here, by
  // the SMs of its GPCs). A second wave takes nearly as long again, where base solves
  // and products take little more: 512 rows and 960 right-hand sides 144 us, 1024 267 us
  // in two waves and 173 as solves and products (65 rows 37, 52 and 45).
  static PerDevice<int> wave;
  const auto fit = [&cfg] {
    const void* fn = reinterpret_cast<const void*>(TrsmClusterKernel<T>);
    int clusters = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, TcSmem<T>()) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return clusters * kTcRhs;
  };
  if (other > wave.Get(fit)) return false;
  TrsmClusterArgs<T> a;
  a.tri = tri;
  if (!left) std::swap(a.tri.rs, a.tri.cs);
  a.lower = left == lower ? 1 : 0;
  a.unit = unit ? 1 : 0;
  a.r = r;
  a.other = other;
  a.x = b;
  a.xs = left ? 1 : ldb;
  a.xr = left ? ldb : 1;
  a.guard = ctx.guard;
  Failed(cudaLaunchKernelEx(&cfg, TrsmClusterKernel<T>, a), "trsm subtree");
  CountLaunch();
  return !LaunchFailed("trsm subtree");
}

template <typename T>
void LaunchGemm(int m, int n, int k, T alpha, View<T> a, View<T> b, T beta,
                T* c, int ldc);
template <>
void LaunchGemm<double>(int m, int n, int k, double alpha, View<double> a,
                        View<double> b, double beta, double* c, int ldc) {
  Dgemm(m, n, k, alpha, a, b, beta, c, ldc, kAll);
}
template <>
void LaunchGemm<float>(int m, int n, int k, float alpha, View<float> a,
                       View<float> b, float beta, float* c, int ldc) {
  Sgemm(m, n, k, alpha, a, b, beta, c, ldc, kAll);
}

// TrsmRecursive (src/trsm.cc:87-135): split at max(32, (r/2)/32*32).
template <typename T>
void TrsmRec(bool left, View<T> tri, bool lower, bool unit, int r, int other,
             T* b, int ldb) {
  if (r <= 32 || (r <= kBaseW && other < SplitFrom<T>(left, r))) {
    TrsmSolve<T>(left, tri, lower, unit, r, other, b, ldb);
    return;
  }
  if (r <= kTcRows && TrsmCluster<T>(left, tri, lower, unit, r, other, b, ldb)) return;
  const int r1 = std::max(32, (r / 2) / 32 * 32);
  const int r2 = r - r1;
  const View<T> t11 = tri;
  const View<T> t22 = tri.sub(r1, r1);
  const View<T> toff = lower ? tri.sub(r1, 0) : tri.sub(0, r1);
  const auto cm = [&](T* p) { return ColMajor<T>(p, ldb); };
  if (left) {
    T* b1 = b;
    T* b2 = b + r1;
    if (lower) {
      TrsmRec(left, t11, lower, unit, r1, other, b1, ldb);
      LaunchGemm<T>(r2, other, r1, T(-1), toff, cm(b1), T(1), b2, ldb);
      TrsmRec(left, t22, lower, unit, r2, other, b2, ldb);
    } else {
      TrsmRec(left, t22, lower, unit, r2, other, b2, ldb);
      LaunchGemm<T>(r1, other, r2, T(-1), toff, cm(b2), T(1), b1, ldb);
      TrsmRec(left, t11, lower, unit, r1, other, b1, ldb);
    }
  } else {
    T* b1 = b;
    T* b2 = b + static_cast<long long>(r1) * ldb;
    if (lower) {
      TrsmRec(left, t22, lower, unit, r2, other, b2, ldb);
      LaunchGemm<T>(other, r1, r2, T(-1), cm(b2), toff, T(1), b1, ldb);
      TrsmRec(left, t11, lower, unit, r1, other, b1, ldb);
    } else {
      TrsmRec(left, t11, lower, unit, r1, other, b1, ldb);
      LaunchGemm<T>(other, r2, r1, T(-1), cm(b1), toff, T(1), b2, ldb);
      TrsmRec(left, t22, lower, unit, r2, other, b2, ldb);
    }
  }
}

}  // namespace

void Sgemm(int m, int n, int k, float alpha, View<float> a, View<float> b,
           float beta, float* c, int ldc, Part part, Tri tri) {
  if (tri == kTriNone) {
    SgemmTiles(m, n, k, alpha, a, b, beta, c, ldc, part);
    return;
  }
  const dim3 grid((m + kSB - 1) / kSB, (n + kSB - 1) / kSB);
  SgemmKernel<<<grid, 256, 0, Ctx().stream>>>(m, n, k, alpha, a, b, beta, c, ldc,
                                              static_cast<int>(tri), Ctx().guard);
  CountLaunch();
  LaunchFailed("sgemm");
}

template <typename T>
void TrsmSolve(bool left, View<T> tri, bool lower, bool unit, int r, int other,
               T* b, int ldb) {
  if (r <= 0 || other <= 0) return;
  View<T> t = tri;
  bool lo = lower;
  long long xs_row, xs_col;
  if (left) {
    // T X = B  <=>  X^T T^T = B^T (src/trsm-inl.h:306-324): rows of X^T are
    // the columns of B.
    t.rs = tri.cs;
    t.cs = tri.rs;
    lo = !lower;
    xs_row = ldb;
    xs_col = 1;
  } else {
    xs_row = 1;
    xs_col = ldb;
  }
  if (r <= 32 && other >= RowsFrom<T>(left)) {
    TrsmRowsKernel<T><<<(other + 127) / 128, 128, 0, Ctx().stream>>>(
        t, lo ? 1 : 0, unit ? 1 : 0, r, other, b, xs_row, xs_col, Ctx().guard);
  } else {
    TrsmBaseKernel<T><<<(other + kBaseRows - 1) / kBaseRows, kBaseThreads, 0, Ctx().stream>>>(
        t, lo ? 1 : 0, unit ? 1 : 0, r, other, b, xs_row, xs_col, Ctx().guard);
  }
  CountLaunch();
  LaunchFailed("trsm base");
}
template void TrsmSolve<double>(bool, View<double>, bool, bool, int, int,
                                double*, int);
template void TrsmSolve<float>(bool, View<float>, bool, bool, int, int, float*,
                               int);

// Trsm (src/trsm.cc:137-180) after argument checks: B := alpha*B first
// (alpha != 1), zero B and return for alpha == 0, then the recursion on
// op(A) (strides swapped and triangle flipped when transposed).
template <typename T>
void TrsmFull(bool left, bool lower, bool trans, bool unit, int m, int n,
              T alpha, const T* a, int lda, T* b, int ldb) {
  if (m == 0 || n == 0) return;
  if (alpha != T(1)) ScaleMatrix<T>(m, n, alpha, b, ldb, kAll);
  if (alpha == T(0)) return;
  const View<T> tri = ColMajor<T>(a, lda, trans);
  const bool op_lower = trans ? !lower : lower;
  TrsmRec<T>(left, tri, op_lower, unit, left ? m : n, left ? n : m, b, ldb);
}
template void TrsmFull<double>(bool, bool, bool, bool, int, int, double,
                               const double*, int, double*, int);
template void TrsmFull<float>(bool, bool, bool, bool, int, int, float,
                              const float*, int, float*, int);

// Syrk (src/level3.cc:84-139; ssyrk_/dsyrk_ 410-421), real: C :=
// alpha*op(A)*op(A)^T + beta*C on one triangle, as a GEMM with a triangular C
// part (DMMA for double, the FP32 kernel for float).
template <typename T>
void SyrkFull(bool lower, bool trans, int n, int k, T alpha, const T* a, int lda, T beta,
              T* c, int ldc) {
  const Part part = lower ? kLower : kUpper;
  if (n == 0 || ((alpha == T(0) || k == 0) && beta == T(1))) return;
  if (alpha == T(0) || k == 0) {
    ScaleMatrix<T>(n, n, beta, c, ldc, part);
    return;
  }
  if constexpr (sizeof(T) == 8) {
    Dgemm(n, n, k, alpha, ColMajor<T>(a, lda, trans), ColMajor<T>(a, lda, !trans), beta, c,
          ldc, part);
  } else {
    Sgemm(n, n, k, alpha, ColMajor<T>(a, lda, trans), ColMajor<T>(a, lda, !trans), beta, c,
          ldc, part);
  }
}
template void SyrkFull<double>(bool, bool, int, int, double, const double*, int, double,
                               double*, int);
template void SyrkFull<float>(bool, bool, int, int, float, const float*, int, float, float*,
                              int);

namespace {

// A GEMM problem on the triangle `part` of C (DMMA for double, FP32 FFMA for
// float), with the reference's merge rules for tiles crossing the diagonal.
template <typename T>
void GemmPart(int m, int n, int k, T alpha, View<T> a, View<T> b, T beta, T* c, int ldc,
              Part part, Tri tri = kTriNone) {
  if constexpr (sizeof(T) == 8) {
    Dgemm(m, n, k, alpha, a, b, beta, c, ldc, part, tri);
  } else {
    Sgemm(m, n, k, alpha, a, b, beta, c, ldc, part, tri);
  }
}

// out (n x n, leading dimension ldo) := the symmetric matrix whose `lower`
// (or upper) triangle is stored in a; the other triangle of a is not read.
template <typename T>
__global__ void SymmetrizeFullKernel(int n, const T* a, long long lda, bool lower, T* out,
                                     long long ldo) {
  const long long total = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    const bool stored = lower ? i >= j : i <= j;
    out[i + j * ldo] = stored ? a[i + j * lda] : a[j + i * lda];
  }
}

// out (n x n) := the triangle `lower` of a with explicit zeros in the other
// one and ones on the diagonal when `unit` (the values the reference packs for
// a triangular operand, src/pack-inl.h:99-160); the rest of a is not read.
template <typename T>
__global__ void TriangleFullKernel(int n, const T* a, long long lda, bool lower, bool unit,
                                   T* out, long long ldo) {
  const long long total = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    T v = T(0);
    if (i == j) v = unit ? T(1) : a[i + j * lda];
    else if (lower ? i > j : i < j) v = a[i + j * lda];
    out[i + j * ldo] = v;
  }
}

int GridFor(long long total) {
  return static_cast<int>(std::min<long long>((total + 255) / 256, 8192));
}

}  // namespace

// SYMM: the reference packs the stored triangle mirrored (Structure::
// kSymmetric, src/pack-inl.h:99-160), i.e. the values of the full symmetric
// matrix; here that matrix is formed once and the plain GEMM runs on it, so
// every element's chain is the GEMM's (src/level3.cc:26-82).
template <typename T>
void SymmFull(bool left, bool lower, int m, int n, T alpha, const T* a, int lda, const T* b,
              int ldb, T beta, T* c, int ldc) {
  if (m == 0 || n == 0 || (alpha == T(0) && beta == T(1))) return;
  if (alpha == T(0)) {
    ScaleMatrix<T>(m, n, beta, c, ldc, kAll);
    return;
  }
  const int ka = left ? m : n;
  T* full = static_cast<T*>(Workspace(kWsLevel3, sizeof(T) * static_cast<size_t>(ka) * ka));
  if (full == nullptr) return;
  SymmetrizeFullKernel<T><<<GridFor(static_cast<long long>(ka) * ka), 256, 0, Ctx().stream>>>(
      ka, a, lda, lower, full, ka);
  CountLaunch();
  if (LaunchFailed("symm symmetrize")) return;
  const View<T> sym = ColMajor<T>(full, ka), gen = ColMajor<T>(b, ldb);
  GemmPart<T>(m, n, ka, alpha, left ? sym : gen, left ? gen : sym, beta, c, ldc, kAll);
}
template void SymmFull<double>(bool, bool, int, int, double, const double*, int,
                               const double*, int, double, double*, int);
template void SymmFull<float>(bool, bool, int, int, float, const float*, int, const float*,
                              int, float, float*, int);

// SYR2K: alpha op(A) op(B)^T + beta C, then + alpha op(B) op(A)^T (beta 1),
// each a GEMM problem on the uplo triangle (src/level3.cc:153-221).
template <typename T>
void Syr2kFull(bool lower, bool trans, int n, int k, T alpha, const T* a, int lda,
               const T* b, int ldb, T beta, T* c, int ldc) {
  const Part part = lower ? kLower : kUpper;
  if (n == 0 || ((alpha == T(0) || k == 0) && beta == T(1))) return;
  if (alpha == T(0) || k == 0) {
    ScaleMatrix<T>(n, n, beta, c, ldc, part);
    return;
  }
  GemmPart<T>(n, n, k, alpha, ColMajor<T>(a, lda, trans), ColMajor<T>(b, ldb, !trans), beta,
              c, ldc, part);
  GemmPart<T>(n, n, k, alpha, ColMajor<T>(b, ldb, trans), ColMajor<T>(a, lda, !trans), T(1),
              c, ldc, part);
}
template void Syr2kFull<double>(bool, bool, int, int, double, const double*, int,
                                const double*, int, double, double*, int);
template void Syr2kFull<float>(bool, bool, int, int, float, const float*, int, const float*,
                               int, float, float*, int);

// GEMMTR: op(A) (n x k) op(B) (k x n) on the uplo triangle of C
// (src/level3.cc:226-280).
template <typename T>
void GemmtrFull(bool lower, bool ta, bool tb, int n, int k, T alpha, const T* a, int lda,
                const T* b, int ldb, T beta, T* c, int ldc) {
  const Part part = lower ? kLower : kUpper;
  if (n == 0 || ((alpha == T(0) || k == 0) && beta == T(1))) return;
  if (alpha == T(0) || k == 0) {
    ScaleMatrix<T>(n, n, beta, c, ldc, part);
    return;
  }
  GemmPart<T>(n, n, k, alpha, ColMajor<T>(a, lda, ta), ColMajor<T>(b, ldb, tb), beta, c, ldc,
              part);
}
template void GemmtrFull<double>(bool, bool, bool, int, int, double, const double*, int,
                                 const double*, int, double, double*, int);
template void GemmtrFull<float>(bool, bool, bool, int, int, float, const float*, int,
                                const float*, int, float, float*, int);

// TRMM: B := alpha op(A) B (left) or alpha B op(A), computed from a copy of B
// with beta 0 (src/level3.cc:284-342). The triangle is stored out with its
// zeros and unit diagonal, and the GEMM multiplies only the k range of each
// reference micro-tile, so every element is the reference's chain.
template <typename T>
void TrmmFull(bool left, bool lower, bool trans, bool unit, int m, int n, T alpha,
              const T* a, int lda, T* b, int ldb) {
  if (m == 0 || n == 0) return;
  if (alpha == T(0)) {
    ScaleMatrix<T>(m, n, T(0), b, ldb, kAll);
    return;
  }
  const int ka = left ? m : n;
  T* tri = static_cast<T*>(Workspace(kWsLevel3, sizeof(T) * static_cast<size_t>(ka) * ka));
  if (tri == nullptr) return;
  TriangleFullKernel<T><<<GridFor(static_cast<long long>(ka) * ka), 256, 0, Ctx().stream>>>(
      ka, a, lda, lower, unit, tri, ka);
  CountLaunch();
  if (LaunchFailed("trmm triangle")) return;
  TrmmDense<T>(left, lower, trans, m, n, alpha, tri, ka, b, ldb);
}

// TRMM on a triangle already stored dense (zeros and unit diagonal written
// out), from a copy of B.
template <typename T>
void TrmmDense(bool left, bool lower, bool trans, int m, int n, T alpha, const T* tri, int ldt,
               T* b, int ldb) {
  if (m == 0 || n == 0) return;
  const int ka = left ? m : n;
  T* copy = static_cast<T*>(Workspace(kWsLevel3Copy, sizeof(T) * static_cast<size_t>(m) * n));
  if (copy == nullptr) return;
  if (Failed(cudaMemcpy2DAsync(copy, sizeof(T) * m, b, sizeof(T) * ldb, sizeof(T) * m, n,
                               cudaMemcpyDeviceToDevice, Ctx().stream),
             "trmm copy"))
    return;
  // op(A) is lower exactly when A is lower and not transposed, or upper and
  // transposed (src/api.h:133-140).
  const bool op_lower = (lower != trans);
  const View<T> t = ColMajor<T>(tri, ldt, trans), g = ColMajor<T>(copy, m);
  if (left) {
    GemmPart<T>(m, n, ka, alpha, t, g, T(0), b, ldb, kAll, op_lower ? kTriALower : kTriAUpper);
  } else {
    GemmPart<T>(m, n, ka, alpha, g, t, T(0), b, ldb, kAll, op_lower ? kTriBLower : kTriBUpper);
  }
}
template void TrmmDense<double>(bool, bool, bool, int, int, double, const double*, int,
                                double*, int);
template void TrmmDense<float>(bool, bool, bool, int, int, float, const float*, int, float*,
                               int);
template void TrmmFull<double>(bool, bool, bool, bool, int, int, double, const double*, int,
                               double*, int);
template void TrmmFull<float>(bool, bool, bool, bool, int, int, float, const float*, int,
                              float*, int);

// Gemm (src/gemm.cc:114-131) after argument checks.
template <typename T>
void GemmFull(bool ta, bool tb, int m, int n, int k, T alpha, const T* a,
              int lda, const T* b, int ldb, T beta, T* c, int ldc) {
  if (m == 0 || n == 0) return;
  if ((k == 0 || alpha == T(0)) && beta == T(1)) return;
  if (k == 0 || alpha == T(0)) {
    ScaleMatrix<T>(m, n, beta, c, ldc, kAll);
    return;
  }
  LaunchGemm<T>(m, n, k, alpha, ColMajor<T>(a, lda, ta), ColMajor<T>(b, ldb, tb),
                beta, c, ldc);
}
template void GemmFull<double>(bool, bool, int, int, int, double,
                               const double*, int, const double*, int, double,
                               double*, int);
template void GemmFull<float>(bool, bool, int, int, int, float, const float*,
                              int, const float*, int, float, float*, int);

}  // namespace hb
