// The LU panel (at most 64 columns) in one launch, and the interchanges and
// triangular solve that follow it.
//
// GetrfPanelKernel factors an m x w panel (w <= 64, m >= w) with the
// reference's recursion (src/lapack/getrf.cc:112-207: halves down to leaves of
// at most 16 columns, factor_kernels.cc:79-183) and each element's operations
// in the reference's order. It is bound by the latency of its w dependent
// pivot searches, so everything between two of them stays on the chip: a
// thread-block cluster holds the panel in shared memory, one row a thread,
// and a leaf's remaining columns in registers. Rows are never interchanged:
// each thread keeps the position its row has after the interchanges so far
// (ties of the pivot search go to the first position), and the rows go to
// their positions when the panel is written. The column loop is rolled (the
// update shifts the registers, so that the current column is always the
// first): unrolled, its instructions came from L2 once per column, which took
// longer than the column's work (dgetrf n = 4096 14.4 ms unrolled, 11.3 rolled).
// What bounds a column now is one warp's chain of instructions, some 1700 cycles at
// 256 rows: two rows a thread, with one busy warp a scheduler, made 256 x 64
// 96 us instead of 79. 4096 x 64: 400 us as leaves, interchanges, solves and
// products, 113 us so. Per column: the warps' maxima by
// redux on the bits of |x|, one block barrier, the block's candidate row sent
// to every CTA of the cluster by st.async (one one-way trip; the receiving
// mbarrier counts the bytes), and every warp picks the winner by itself.
// After a leaf, every CTA collects its pivot rows' other columns and solves
// the small triangles for itself. T is float, double or a complex element
// (Cx<float>, Cx<double>): the complex LU has the same recursion and leaves, on
// |re| + |im| and the complex AXPY, product and quotient of complex.cuh.
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "complex.cuh"
#include "device.cuh"
#include "internal.h"
#include "ref_order.cuh"

namespace hb {
namespace {

constexpr int kPanelW = 64;        // columns
constexpr int kPanelLeaf = 16;     // src/lapack/factor_kernels.h:27
// Row stride of the pivot rows: 16-byte aligned, few bank conflicts by column.
template <typename T>
constexpr int kPanelLd = kPanelW + 16 / static_cast<int>(sizeof(T));
// Rows of a CTA at most: its registers hold 16 elements a row.
template <typename T>
constexpr int kPanelThreads = sizeof(T) == 16 ? 256 : 512;
constexpr int kPanelLeast = 256;   // threads at least: the solves share all warps
constexpr int kPanelCtas = 16;
// Polls of a wait for the other CTAs' candidates, each asleep for at most 4 us
// (whatever time is asked for; spinning warps slow the others down): about a second,
// far above any real wait.
constexpr uint32_t kPanelPolls = 1u << 18;
// A limit set by hwyblas_set_leaf_wait_limit, 0: none. It counts polls that do not
// sleep, in an instantiation of its own (kSpin): chosen at run time, the two polls
// cost 8 % of a panel.
std::atomic<uint32_t> g_panel_polls{0};

template <typename R>
struct __align__(2 * sizeof(R)) Cx {
  R re, im;
};
template <typename T>
struct ElemOf {
  using Real = T;
  static constexpr bool kComplex = false;
};
template <typename R>
struct ElemOf<Cx<R>> {
  using Real = R;
  static constexpr bool kComplex = true;
};
template <typename T>
using RealOf = typename ElemOf<T>::Real;
template <typename T>
constexpr bool kWideKey = sizeof(RealOf<T>) == 8;

// The leaf's element operations (src/lapack/factor_kernels.cc:33-183).
template <typename T>
__device__ __forceinline__ T Zero() {
  if constexpr (ElemOf<T>::kComplex) return T{0, 0};
  else return T(0);
}
__device__ __forceinline__ bool IsZero(double x) { return x == 0.0; }
__device__ __forceinline__ bool IsZero(float x) { return x == 0.f; }
template <typename R>
__device__ __forceinline__ bool IsZero(Cx<R> x) {
  return x.re == R(0) && x.im == R(0);
}
template <typename T>
__device__ __forceinline__ bool IsTiny(T x) {
  if constexpr (ElemOf<T>::kComplex)
    return !ZAbsAtLeast(x.re, x.im, Sfmin<RealOf<T>>());
  else
    return !(fabs(x) >= Sfmin<T>());
}
template <typename T>
__device__ __forceinline__ T Recip(T x) {
  if constexpr (ElemOf<T>::kComplex) {
    T r;
    ZRecip(x.re, x.im, &r.re, &r.im);
    return r;
  } else {
    return T(1) / x;
  }
}
template <typename T>
__device__ __forceinline__ T Times(T x, T v) {
  if constexpr (ElemOf<T>::kComplex)
    return T{Sub(Mul(x.re, v.re), Mul(x.im, v.im)), Add(Mul(x.im, v.re), Mul(x.re, v.im))};
  else
    return x * v;
}
template <typename T>
__device__ __forceinline__ T Over(T x, T p) {
  if constexpr (ElemOf<T>::kComplex) {
    T q;
    ZDiv(x.re, x.im, p.re, p.im, &q.re, &q.im);
    return q;
  } else {
    return x / p;
  }
}
// y - u l in the AXPY rounding of a column of len elements.
template <typename T>
__device__ __forceinline__ T AxpyMinus(T y, T u, T l, int len, int lanes) {
  if constexpr (ElemOf<T>::kComplex) {
    ZAxpyRef(y.re, y.im, -u.re, -u.im, l.re, l.im, len, lanes);
    return y;
  } else {
    return Axpy(y, -u, l, len, lanes);
  }
}
// The same for a column of at least one vector.
template <typename T>
__device__ __forceinline__ T AxpyMinusLong(T y, T u, T l) {
  if constexpr (ElemOf<T>::kComplex)
    return AxpyMinus(y, u, l, 1, 0);
  else
    return fma(l, -u, y);
}
template <typename T>
__device__ __forceinline__ T Shfl(T x, int from) {
  if constexpr (ElemOf<T>::kComplex)
    return T{__shfl_sync(0xffffffffu, x.re, from), __shfl_sync(0xffffffffu, x.im, from)};
  else
    return __shfl_sync(0xffffffffu, x, from);
}
// Global elements are aligned as their real parts.
template <typename T>
__device__ __forceinline__ T LoadGlobal(const T* p) {
  if constexpr (ElemOf<T>::kComplex) {
    const RealOf<T>* r = reinterpret_cast<const RealOf<T>*>(p);
    return T{r[0], r[1]};
  } else {
    return *p;
  }
}
template <typename T>
__device__ __forceinline__ void StoreGlobal(T* p, T v) {
  if constexpr (ElemOf<T>::kComplex) {
    RealOf<T>* r = reinterpret_cast<RealOf<T>*>(p);
    r[0] = v.re;
    r[1] = v.im;
  } else {
    *p = v;
  }
}

// A CTA's candidate of one column: its key, its position after and its place
// before the interchanges, and the row from that column on. The reciprocal of
// its pivot follows in a message of its own, computed while the first is on its
// way.
template <typename T>
struct __align__(16) PanelSlot {
  unsigned long long key;
  int pos, place;
  T row[kPanelLeaf];
};

template <typename T>
struct PanelArgs {
  int m, w, R, S, lanes;  // R: rows of a CTA; S: their stride in shared memory
  T* a;
  long long lda;
  int* ipiv;
  int ipiv_add;
  int* info;
  int info_base;
  int* moves;  // count, unused, then (position, row) of every row that moved
  uint32_t polls;  // a wait's limit
  int* timeout_flag;
};

template <typename R>
__device__ __forceinline__ unsigned long long PivotKey(Cx<R> x) {
  return PivotKey(ZMag(x.re, x.im));
}

__device__ __forceinline__ uint32_t MapRank(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes to another CTA's shared memory, counted on its mbarrier.
__device__ __forceinline__ void StAsync16(uint32_t dst, ulonglong2 v, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];"
      :
      : "r"(dst), "l"(v.x), "l"(v.y), "r"(bar)
      : "memory");
}
// One value to another CTA's shared memory, counted on its mbarrier.
__device__ __forceinline__ void StAsync(uint32_t dst, double v, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
      :
      : "r"(dst), "l"(__double_as_longlong(v)), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void StAsync(uint32_t dst, float v, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
      :
      : "r"(dst), "r"(__float_as_int(v)), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void StAsync(uint32_t dst, Cx<float> v, uint32_t bar) {
  StAsync(dst, __hiloint2double(__float_as_int(v.im), __float_as_int(v.re)), bar);
}
__device__ __forceinline__ void StAsync(uint32_t dst, Cx<double> v, uint32_t bar) {
  StAsync16(dst,
            make_ulonglong2(__double_as_longlong(v.re), __double_as_longlong(v.im)), bar);
}
__device__ __forceinline__ double LoadRemote(uint32_t addr, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float LoadRemote(uint32_t addr, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
template <typename R>
__device__ __forceinline__ Cx<R> LoadRemote(uint32_t addr, Cx<R>) {
  return Cx<R>{LoadRemote(addr, R(0)), LoadRemote(addr + sizeof(R), R(0))};
}
template <bool kSpin>
__device__ __forceinline__ bool MbarTest(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (kSpin)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(SmemAddr(bar)), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(SmemAddr(bar)), "r"(parity)
        : "memory");
  return ok != 0;
}
// The wait of a panel for phase `parity`; false (and the flags set) if it gives up.
template <bool kSpin>
__device__ __forceinline__ bool PanelWait(uint64_t* bar, uint32_t parity, uint32_t limit,
                                          int* timeout_flag, int* quit) {
  for (uint32_t polls = 0; !MbarTest<kSpin>(bar, parity);) {
    if (++polls >= limit) {
      atomicExch(timeout_flag, 1);
      *quit = 1;
      return false;
    }
  }
  return true;
}
// Waits for the messages that are still on their way to a CTA that gave up: an
// mbarrier takes those of the columns of one parity, `bytes` from every CTA a
// column. sent[p]: the columns that CTA p has sent; armed: those this CTA has
// armed. The last armed column's phase is given the bytes that nobody will
// send, a later one (which the faster CTAs may have reached) is armed with the
// bytes that were sent.
__device__ void PanelDrain(uint64_t* bar, int parity, int armed, const int* sent, int P,
                           uint32_t bytes, int* timeout_flag, int* quit) {
  int c = armed > parity ? armed - 1 - ((armed - 1 - parity) & 1) : parity;
  for (;; c += 2) {
    int n = 0;
    for (int p = 0; p < P; ++p) n += sent[p] > c;
    if (n == 0) return;
    if (c >= armed) {
      MbarArriveExpectTx(bar, n * bytes);
    } else if (n < P) {
      asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(
                       SmemAddr(bar)),
                   "r"((P - n) * bytes)
                   : "memory");
    }
    if (!PanelWait<false>(bar, (c >> 1) & 1, kPanelPolls, timeout_flag, quit)) return;
  }
}
__device__ __forceinline__ void ClusterBarrier() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}

// One element global -> shared, asynchronously.
template <typename T>
__device__ __forceinline__ void CopyElement(T* dst, const T* src) {
  if constexpr (ElemOf<T>::kComplex) {
    using R = RealOf<T>;
    CopyElement(reinterpret_cast<R*>(dst), reinterpret_cast<const R*>(src));
    CopyElement(reinterpret_cast<R*>(dst) + 1, reinterpret_cast<const R*>(src) + 1);
    return;
  }
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(SmemAddr(dst)), "l"(src),
               "n"(ElemOf<T>::kComplex ? 4 : sizeof(T))
               : "memory");
}

// Solves with the unit lower triangle, N columns a warp, a lane one row: the
// solved values go round by shuffles, so that r rows are r - 1 steps and each
// element's chain runs over q ascending (src/trsm-inl.h:107-174). lrow: the
// lane's row of the triangle.
template <typename T, int N>
__device__ __forceinline__ void LaneSolve(const T* lrow, int r, T (&y)[N]) {
  const int lane = threadIdx.x % 32;
  if constexpr (ElemOf<T>::kComplex) {
    // Four chains an element from zero (src/trsm-inl.h:175-214), combined when
    // its step comes.
    using R = RealOf<T>;
    R rr[N], ir[N], ri[N], ii[N];
#pragma unroll
    for (int i = 0; i < N; ++i) rr[i] = ir[i] = ri[i] = ii[i] = R(0);
#pragma unroll 1
    for (int q = 0; q < r; ++q) {
      const T l = lrow[q];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const T v = T{Sub(y[i].re, Sub(rr[i], ii[i])), Sub(y[i].im, Add(ir[i], ri[i]))};
        const T yq = Shfl(v, q);
        if (lane == q) {
          y[i] = yq;
        } else if (lane > q) {
          rr[i] = Fma(yq.re, l.re, rr[i]);
          ir[i] = Fma(yq.im, l.re, ir[i]);
          ri[i] = Fma(yq.re, l.im, ri[i]);
          ii[i] = Fma(yq.im, l.im, ii[i]);
        }
      }
    }
  } else {
#pragma unroll 4
    for (int q = 0; q + 1 < r; ++q) {
      const T l = lrow[q];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const T yq = __shfl_sync(0xffffffffu, y[i], q);
        if (lane > q) y[i] = fma(-yq, l, y[i]);
      }
    }
  }
}

// U := L^-1 U for the n1 <= 32 pivot rows at `rows` (stride kPanelLd; L unit
// lower in their columns [0, n1), U in columns [n1, n1 + n2)).
template <typename T>
__device__ __forceinline__ void PanelSolve(T* rows, int n1, int n2) {
  constexpr int N = ElemOf<T>::kComplex ? 2 : 4;
  const int lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  T* row = rows + min(lane, n1 - 1) * kPanelLd<T>;
  for (int c = N * (threadIdx.x / 32); c < n2; c += N * nwarps) {
    T y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] = row[n1 + min(c + i, n2 - 1)];
    LaneSolve<T, N>(row, n1, y);
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (lane < n1 && c + i < n2) row[n1 + c + i] = y[i];
  }
}

// Four consecutive elements from shared memory, 16-byte loads if aligned.
template <typename T, bool kVec>
__device__ __forceinline__ void Load4Shared(const T* p, T (&v)[4]) {
  if constexpr (kVec && sizeof(T) == 8) {
    const double2 x = reinterpret_cast<const double2*>(p)[0];
    const double2 y = reinterpret_cast<const double2*>(p)[1];
    v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
  } else if constexpr (kVec) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = p[i];
  }
}

// Two rows of the trailing update: X(r, c) = -sum_q L(r, q) U(q, c) + X(r, c)
// for cw (8 or 16) columns, each sum one chain over q (alpha -1, beta 1).
template <typename T, bool kVec>
__device__ __forceinline__ void PanelUpdate(const T* l, T* x, int R, const T* u, int n1, int nc,
                                            int cw, int ra, int rb, bool ina, bool inb) {
  T acc[2][kPanelLeaf];
#pragma unroll
  for (int c = 0; c < kPanelLeaf; ++c) acc[0][c] = acc[1][c] = T(0);
#pragma unroll 2
  for (int q = 0; q < n1; ++q) {
    const T la = l[q * R + ra], lb = l[q * R + rb];
#pragma unroll
    for (int c4 = 0; c4 < kPanelLeaf / 4; ++c4) {
      if (c4 >= 2 && cw <= 8) break;
      T uv[4];
      Load4Shared<T, kVec>(u + q * kPanelLd<T> + c4 * 4, uv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[0][c4 * 4 + e] = fma(la, uv[e], acc[0][c4 * 4 + e]);
        acc[1][c4 * 4 + e] = fma(lb, uv[e], acc[1][c4 * 4 + e]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kPanelLeaf; ++c) {
    if (c >= nc) continue;
    if (ina) x[c * R + ra] = T(-1) * acc[0][c] + x[c * R + ra];
    if (inb) x[c * R + rb] = T(-1) * acc[1][c] + x[c * R + rb];
  }
}

// c + (-1) ab for ab = (rr - ii, ir + ri): the GEMM merge with alpha -1, beta 1.
template <typename R>
__device__ __forceinline__ Cx<R> MinusProduct(Cx<R> c, R rr, R ir, R ri, R ii) {
  const R re = Sub(rr, ii), im = Add(ir, ri);
  return Cx<R>{Add(Sub(Mul(re, R(-1)), Mul(im, R(0))), c.re),
               Add(Add(Mul(im, R(-1)), Mul(re, R(0))), c.im)};
}

// The complex update: four chains an element, combined as the product with
// alpha -1 and added (src/gemm_kernel-inl.h:226-428), four columns at a time.
template <typename R>
__device__ __forceinline__ void PanelUpdateComplex(const Cx<R>* l, Cx<R>* x, int S,
                                                   const Cx<R>* u, int n1, int nc, int ra,
                                                   int rb, bool ina, bool inb) {
#pragma unroll 1
  for (int c0 = 0; c0 < nc; c0 += 4) {
    R acc[2][4][4];  // rr, ir, ri, ii
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i / 16][i / 4 % 4][i % 4] = R(0);
#pragma unroll 2
    for (int q = 0; q < n1; ++q) {
      const Cx<R> lv[2] = {l[q * S + ra], l[q * S + rb]};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const Cx<R> uv = u[q * kPanelLd<Cx<R>> + c0 + c];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          acc[i][c][0] = Fma(lv[i].re, uv.re, acc[i][c][0]);
          acc[i][c][1] = Fma(lv[i].im, uv.re, acc[i][c][1]);
          acc[i][c][2] = Fma(lv[i].re, uv.im, acc[i][c][2]);
          acc[i][c][3] = Fma(lv[i].im, uv.im, acc[i][c][3]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c0 + c >= nc) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (!(i == 0 ? ina : inb)) continue;
        Cx<R>& e = x[(c0 + c) * S + (i == 0 ? ra : rb)];
        e = MinusProduct(e, acc[i][c][0], acc[i][c][1], acc[i][c][2], acc[i][c][3]);
      }
    }
  }
}

// Sixteen rows of the update on the FP64 tensor pipe (bound by instructions as FMAs:
// 32 x 32 of 256 rows took 8 us): the m16n8k8 chain runs over q ascending; past n1,
// -0 times +0 leaves every sum as it is. pos[i] >= least: row i is updated.
__device__ __forceinline__ void PanelUpdateDmma(const double* l, double* x, int S,
                                                const double* u, int n1, int n2, const int* pos,
                                                int rows, int least) {
  const int lane = threadIdx.x % 32, g = lane >> 2, t = lane & 3;
  double acc[4][4];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[b][e] = 0.0;
#pragma unroll 2
  for (int k0 = 0; k0 < n1; k0 += 8) {
    const int q0 = k0 + t, q1 = q0 + 4;
    const double* a0 = l + min(q0, n1 - 1) * S + g;
    const double* a1 = l + min(q1, n1 - 1) * S + g;
    const double f0 = q0 < n1 ? a0[0] : -0.0, f1 = q0 < n1 ? a0[8] : -0.0;
    const double f2 = q1 < n1 ? a1[0] : -0.0, f3 = q1 < n1 ? a1[8] : -0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (b * 8 >= n2) break;
      const int c = min(b * 8 + g, n2 - 1);
      const double b0 = q0 < n1 ? u[q0 * kPanelLd<double> + c] : 0.0;
      const double b1 = q1 < n1 ? u[q1 * kPanelLd<double> + c] : 0.0;
      asm volatile(
          "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
          "{%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
          : "+d"(acc[b][0]), "+d"(acc[b][1]), "+d"(acc[b][2]), "+d"(acc[b][3])
          : "d"(f0), "d"(f1), "d"(f2), "d"(f3), "d"(b0), "d"(b1));
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = g + 8 * h;
    if (i >= rows || pos[i] < least) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = b * 8 + 2 * t + e;
        if (c < n2) x[c * S + i] = -1.0 * acc[b][2 * h + e] + x[c * S + i];
      }
  }
}

// How a panel is factored: by one CTA (no clusters, messages or waits: 256 x 64 69 us,
// 74 with them compiled in), by a cluster, by a cluster whose polls do not sleep.
enum PanelMode : int { kPanelAlone = 0, kPanelCluster = 1, kPanelSpin = 2 };
template <typename T, int Mode>
__global__ void __launch_bounds__(kPanelThreads<T>) GetrfPanelKernel(PanelArgs<T> p) {
  extern __shared__ __align__(16) unsigned char panel_smem[];
  constexpr bool kCluster = Mode != kPanelAlone, kSpin = Mode == kPanelSpin;
  const int P = gridDim.x, cta = blockIdx.x, R = p.R, RS = p.S, w = p.w;
  // [2][kPanelCtas] from the CTAs, then this CTA's own.
  PanelSlot<T>* slots = reinterpret_cast<PanelSlot<T>*>(panel_smem);
  PanelSlot<T>* own = slots + 2 * kPanelCtas;
  T* prow = reinterpret_cast<T*>(own + 1);                           // [w][kPanelLd] pivot rows
  T* S = prow + w * kPanelLd<T>;                                     // [w][RS] this CTA's rows
  __shared__ T s_rinv[2][kPanelCtas];
  __shared__ unsigned long long s_wkey[2][kPanelThreads<T> / 32];
  __shared__ int s_wpos[2][kPanelThreads<T> / 32];
  __shared__ int s_place[kPanelW], s_pos[kPanelThreads<T>], s_op[7][4];
  __shared__ __align__(8) uint64_t s_bar[2], s_rbar[2];
  // s_quit: whether a wait of an even, an odd column gave up. Read behind the next
  // column's barrier, which the other column's waits come after.
  __shared__ int s_ops, s_sent[kPanelCtas], s_quit[2];
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, nwarps = blockDim.x / 32;
  const int place = cta * R + tid;
  const bool valid = tid < R && place < p.m;
  int pos = place;

  if (tid < kPanelCtas) s_sent[tid] = w;
  if (tid < 2) s_quit[tid] = 0;
  // Pivots that stay in range if the panel ends early.
  if (cta == 0 && tid < w) p.ipiv[tid] = tid + 1 + p.ipiv_add;
  if (tid == 0) {
    MbarInit(&s_bar[0], 1);
    MbarInit(&s_bar[1], 1);
    MbarInit(&s_rbar[0], 1);
    MbarInit(&s_rbar[1], 1);
    FenceBarrierInit();
    // The recursion's steps: leaves (columns c0.., n) and, between the halves
    // of a block (n1 and n2 columns), its solve and update.
    int ops = 0;
    const auto op = [&](int leaf, int c0, int n1, int n2) {
      s_op[ops][0] = leaf, s_op[ops][1] = c0, s_op[ops][2] = n1, s_op[ops][3] = n2;
      ++ops;
    };
    const auto half = [&](int c0, int n) {
      if (n <= kPanelLeaf) {
        op(1, c0, n, 0);
      } else {
        const int n1 = n / 2;
        op(1, c0, n1, 0);
        op(0, c0, n1, n - n1);
        op(1, c0 + n1, n - n1, 0);
      }
    };
    if (w <= kPanelLeaf) {
      op(1, 0, w, 0);
    } else {
      half(0, w / 2);
      op(0, 0, w / 2, w - w / 2);
      half(w / 2, w - w / 2);
    }
    s_ops = ops;
  }
  if (valid) {
    const T* src = p.a + place;
#pragma unroll 4
    for (int c = 0; c < w; ++c) CopyElement(S + c * RS + tid, src + c * p.lda);
  }
  CpAsyncCommit();
  CpAsyncWait<0>();
  // Every CTA's mbarriers are ready before any candidate is sent.
  if constexpr (kCluster) ClusterBarrier();
  else __syncthreads();

  // A wait that gives up (timed_out, a thread's own) ends the panel for its CTA at
  // the next block barrier, where all threads learn of it (alive): it arms no more
  // mbarriers and sends no more candidates, but takes part in the cluster's
  // barriers and stays until nothing is on its way to it.
  bool timed_out = false, alive = true;
  int armed = 0, sent = 0;  // columns that thread 0 has armed, that the CTA has sent
  for (int op = 0; op < s_ops; ++op) {
    const int c0 = s_op[op][1], n1 = s_op[op][2], n2 = s_op[op][3];
    if (s_op[op][0] != 0) {
      T x[kPanelLeaf];
#pragma unroll
      for (int k = 0; k < kPanelLeaf; ++k)
        x[k] = valid && k < n1 ? S[(c0 + k) * RS + tid] : Zero<T>();
#pragma unroll 1
      for (int j = 0; alive && j < n1; ++j) {
        const int jc = c0 + j, par = jc & 1;
        if (kCluster && tid == 0 && !timed_out) {
          armed = jc + 1;
          MbarArriveExpectTx(&s_bar[par], P * static_cast<uint32_t>(sizeof(PanelSlot<T>)));
          MbarArriveExpectTx(&s_rbar[par], P * static_cast<uint32_t>(sizeof(T)));
        }
        // The warp's candidate among the rows not yet taken (position >= jc). A
        // NaN at position jc wins, as the reference's search starts from it.
        unsigned long long key = valid && pos >= jc ? PivotKey(x[0]) : 0ull;
        if (valid && pos == jc && key == 0)
          key = sizeof(RealOf<T>) == 8 ? ~0ull : 0xffffffffull;
        const int wbest = WarpBest<kWideKey<T>>(key, pos);
        if (lane == wbest) {
          s_wkey[par][warp] = key;
          s_wpos[par][warp] = pos;
        }
        __syncthreads();
        const unsigned long long wkey = lane < nwarps ? s_wkey[par][lane] : 0ull;
        const int wpos = lane < nwarps ? s_wpos[par][lane] : 0x7fffffff;
        if (kCluster && s_quit[par ^ 1] != 0) {
          alive = false;
          break;
        }
        sent = jc + 1;
        // The block's, found by every warp; the warp that holds the row sends it.
        const int cbest = WarpBest<kWideKey<T>>(wkey, wpos);
        if (warp == cbest) {
          if (lane == wbest) {
            own->key = key;
            own->pos = pos;
            own->place = place;
#pragma unroll
            for (int k = 0; k < kPanelLeaf; ++k) own->row[k] = x[k];
          }
          __syncwarp();
          if constexpr (kCluster) {
            constexpr int kPieces = sizeof(PanelSlot<T>) / 16;
            const ulonglong2* src = reinterpret_cast<const ulonglong2*>(own);
            const uint32_t dst = SmemAddr(&slots[par * kPanelCtas + cta]);
            const uint32_t bar = SmemAddr(&s_bar[par]);
            for (int i = lane; i < P * kPieces; i += 32) {
              const int to = i / kPieces, e = i % kPieces;
              StAsync16(MapRank(dst + 16 * e, to), src[e], MapRank(bar, to));
            }
          }
          const T rinv = Recip(own->row[0]);
          if constexpr (kCluster) {
            if (lane < P)
              StAsync(MapRank(SmemAddr(&s_rinv[par][cta]), lane), rinv,
                      MapRank(SmemAddr(&s_rbar[par]), lane));
          } else if (lane == 0) {
            s_rinv[par][0] = rinv;
          }
        }
        int at = 2 * kPanelCtas, from = 0;  // the winner's slot
        if constexpr (kCluster) {
          timed_out =
              !PanelWait<kSpin>(&s_bar[par], (jc >> 1) & 1, p.polls, p.timeout_flag, &s_quit[par]);
          const PanelSlot<T>* slot = slots + par * kPanelCtas + lane;
          from = WarpBest<kWideKey<T>>(lane < P ? slot->key : 0ull, lane < P ? slot->pos : 0x7fffffff);
          at = par * kPanelCtas + (from & (kPanelCtas - 1));
        } else {
          __syncthreads();
        }
        const PanelSlot<T>* win = slots + at;
        const int piv = win->pos;
        const T pivot = win->row[0];
        if (tid < n1 - j) prow[jc * kPanelLd<T> + jc + tid] = win->row[tid];
        if (tid == 32 && !timed_out) {
          s_place[jc] = win->place;
          if (cta == 0) {
            p.ipiv[jc] = piv + 1 + p.ipiv_add;
            if (IsZero(pivot) && *p.info == 0) *p.info = p.info_base + jc + 1;
          }
        }
        // A zero pivot is at position jc already.
        if (pos == piv) pos = jc;
        else if (pos == jc) pos = piv;
        if (kCluster && !timed_out)
          timed_out =
              !PanelWait<kSpin>(&s_rbar[par], (jc >> 1) & 1, p.polls, p.timeout_flag, &s_quit[par]);
        if (valid && pos > jc) {
          // The column below the pivot times its reciprocal (divided if the
          // pivot is below the safe minimum, kept if it is zero), then the
          // rank-1 update of the leaf's later columns, which move up by one.
          T l = Times(x[0], s_rinv[par][from & (kPanelCtas - 1)]);
          if (IsTiny(pivot)) l = IsZero(pivot) ? x[0] : Over(x[0], pivot);
          S[jc * RS + tid] = l;
          const int len = p.m - jc - 1;
          if (len >= p.lanes) {
#pragma unroll
            for (int k = 1; k < kPanelLeaf; ++k) {
              if (k == 9 && n1 - j <= 9) break;  // no such columns
              x[k - 1] = AxpyMinusLong(x[k], win->row[k], l);
            }
          } else {
#pragma unroll
            for (int k = 1; k < kPanelLeaf; ++k)
              x[k - 1] = AxpyMinus(x[k], win->row[k], l, len, p.lanes);
          }
        }
      }
      s_pos[tid] = valid ? pos : -1;
      {
        // The rest of the leaf's pivot rows (the candidates brought their columns
        // from the pivot to the leaf's end), from the CTAs that hold them; these
        // rows change no more.
        if (__syncthreads_or(timed_out)) alive = false;
        if constexpr (kCluster) ClusterBarrier();
        for (int r = warp; alive && r < n1; r += nwarps) {
          const int from = s_place[c0 + r], owner = from / R;
          const T* row = S + (from - owner * R);
#pragma unroll
          for (int d = 0; d < kPanelW / 32; ++d) {
            const int col = lane + 32 * d;
            if (col >= w || (col >= c0 + r && col < c0 + n1)) continue;
            prow[(c0 + r) * kPanelLd<T> + col] =
                kCluster ? LoadRemote(MapRank(SmemAddr(row + col * RS), owner), Zero<T>())
                      : row[col * RS];
          }
        }
        __syncthreads();
      }
    } else if (alive) {
      T* rows = prow + c0 * kPanelLd<T> + c0;
      PanelSolve<T>(rows, n1, n2);
      __syncthreads();
      if constexpr (sizeof(T) == 8 && !ElemOf<T>::kComplex) {
        for (int r0 = warp * 16; r0 < R; r0 += nwarps * 16)
          PanelUpdateDmma(S + c0 * RS + r0, S + (c0 + n1) * RS + r0, RS, rows + n1, n1, n2,
                          s_pos + r0, R - r0, c0 + n1);
      } else {
        // Half the threads take the first cw columns of two rows each, the other
        // half the rest.
        const int cw = n2 > 16 ? 16 : 8, half = (R + 1) / 2;
        const int blk = tid >= half ? 1 : 0, ra = tid - blk * half;
        const int rb = min(ra + half, R - 1), nc = min(cw, n2 - blk * cw);
        if (ra < half && nc > 0) {
          const int cb = n1 + blk * cw;
          const bool ina = s_pos[ra] >= c0 + n1;
          const bool inb = ra + half < R && s_pos[rb] >= c0 + n1;
          if constexpr (ElemOf<T>::kComplex)
            PanelUpdateComplex(S + c0 * RS, S + (c0 + cb) * RS, RS, rows + cb, n1, nc, ra, rb, ina,
                               inb);
          else if ((c0 + cb) % (16 / static_cast<int>(sizeof(T))) == 0)
            PanelUpdate<T, true>(S + c0 * RS, S + (c0 + cb) * RS, RS, rows + cb, n1, nc, cw, ra, rb,
                                 ina, inb);
          else
            PanelUpdate<T, false>(S + c0 * RS, S + (c0 + cb) * RS, RS, rows + cb, n1, nc, cw, ra, rb,
                                  ina, inb);
        }
      }
      __syncthreads();
    }
  }
  if (alive) {
#pragma unroll 4
    for (int i = tid; i < (w - cta + P - 1) / P * kPanelW; i += blockDim.x) {
      const int r = i % kPanelW, c = cta + i / kPanelW * P;
      if (r < w) StoreGlobal(p.a + r + c * p.lda, prow[r * kPanelLd<T> + c]);
    }
    if (valid && pos >= w) {
      T* dst = p.a + pos;
#pragma unroll 8
      for (int c = 0; c < w; ++c) StoreGlobal(dst + c * p.lda, S[c * RS + tid]);
    }
    if (valid && pos != place && p.moves != nullptr) {
      const int e = atomicAdd(p.moves, 1);
      p.moves[2 + 2 * e] = pos;
      p.moves[3 + 2 * e] = place;
    }
  }
  if constexpr (kCluster) {
    if (!alive && tid < P)
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(
                       MapRank(SmemAddr(&s_sent[cta]), tid)),
                   "r"(sent)
                   : "memory");
    // No CTA exits while another may read its rows or write its counts; one whose
    // waits all ended has received every candidate sent to it.
    ClusterBarrier();
    if (!alive && tid == 0) {
      for (int par = 0; par < 2; ++par) {
        PanelDrain(&s_bar[par], par, armed, s_sent, P, sizeof(PanelSlot<T>), p.timeout_flag,
                   s_quit);
        PanelDrain(&s_rbar[par], par, armed, s_sent, P, sizeof(T), p.timeout_flag, s_quit);
      }
    }
  }
}

// Stride of a CTA's R rows in shared memory: 4 modulo 16, so that the tensor pipe's
// fragments are free of bank conflicts, and room for whole blocks of 16.
int PanelStride(int R) { return (R + 15) / 16 * 16 + 4; }

template <typename T>
size_t PanelSmem(int w, int R) {
  return (2 * kPanelCtas + 1) * sizeof(PanelSlot<T>) +
         sizeof(T) * static_cast<size_t>(w) * (kPanelLd<T> + PanelStride(R));
}

constexpr size_t kPanelSmemMax = 227 * 1024 - 4 * 1024;  // beside the static arrays

// CTAs and rows a CTA for an m x w panel; false if it does not fit a cluster
// of at most `most` CTAs.
template <typename T>
bool PanelShape(int m, int w, int most, int* ctas, int* rows) {
  int fit = kPanelThreads<T>;
  while (fit > 0 && PanelSmem<T>(w, fit) > kPanelSmemMax) fit -= 8;
  if (fit <= 0) return false;
  const int least = (m + fit - 1) / fit;
  if (least > most) return false;
  // A row a thread: about 256 rows a CTA balance the exchange (more CTAs) with
  // the updates (more rows); 160 measured 1 to 5 % slower (dgetrf n = 500 to 2500).
  const int want = std::max(least, std::min(most, (m + 255) / 256));
  *ctas = want;
  *rows = (m + want - 1) / want;
  return true;
}

// Interchanges as a list of moved rows (position, row), applied to a block of
// columns, and for the columns right of a panel the solve with its unit lower
// triangle L (jb x jb, jb <= 64): B := L^-1 P B on the panel's rows
// (src/lapack/getrf.cc:28-81, src/trsm.cc:87-135). Bound by latency: a CTA owns
// kSwapCols columns, a warp kSwapCols / 8 of them, a lane one of a column's
// rows, and the solved values go round by shuffles, so that a solve of 32
// rows is 32 steps whatever the width. 7 us for 64 columns of 500 rows, 13 us beside
// the trailing update at n = 4096; LASWP (13 us) and the solve (30 us) before.
constexpr int kSwapThreads = 256, kSwapCols = 16, kMovesMax = 2 * kPanelW;

template <typename T>
struct SwapArgs {
  int jb, left, nc;  // columns [0, left) only move; [c0, c0 + nc) are solved too
  T* a;              // row j of the matrix
  long long lda, c0;
  const T* l;        // the panel's triangle, leading dimension lda
  const int* moves;
};

template <typename T>
constexpr int SwapSmem() {
  return static_cast<int>(sizeof(T)) * (kPanelW + kSwapCols) * (kPanelW + 1);
}

template <typename T>
__global__ void __launch_bounds__(kSwapThreads) PanelSwapTrsmKernel(SwapArgs<T> p) {
  constexpr int kLd = kPanelW + 1;
  __shared__ int s_dst[kMovesMax], s_src[kMovesMax], s_top[kPanelW];
  extern __shared__ __align__(16) unsigned char swap_smem[];
  T* s_l = reinterpret_cast<T*>(swap_smem);  // [kPanelW][kLd] the triangle
  T* s_b = s_l + kPanelW * kLd;              // [kSwapCols][kLd] the columns
  const int tid = threadIdx.x, jb = p.jb;
  const int cnt = min(p.moves[0], kMovesMax);
  const int left_blocks = (p.left + kSwapCols - 1) / kSwapCols;
  const bool solve = static_cast<int>(blockIdx.x) >= left_blocks;
  const int first = (solve ? blockIdx.x - left_blocks : blockIdx.x) * kSwapCols;
  const int cols = min(kSwapCols, (solve ? p.nc : p.left) - first);
  T* b = p.a + (solve ? p.c0 + first : first) * p.lda;
  if (tid < cnt) {
    s_dst[tid] = p.moves[2 + 2 * tid];
    s_src[tid] = p.moves[3 + 2 * tid];
  }
  if (tid < kPanelW) s_top[tid] = tid;
  if (solve) {
    for (int i = tid; i < kPanelW * jb; i += kSwapThreads) {
      const int r = i % kPanelW, c = i / kPanelW;
      if (r < jb) CopyElement(s_l + r * kLd + c, p.l + r + c * p.lda);
    }
  }
  __syncthreads();
  if (solve && tid < cnt && s_dst[tid] < jb) s_top[s_dst[tid]] = s_src[tid];
  __syncthreads();
  // Every value that moves is read before any is written.
  constexpr int kPer = kMovesMax * kSwapCols / kSwapThreads;
  T v[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = (tid + i * kSwapThreads) % kMovesMax, c = (tid + i * kSwapThreads) / kMovesMax;
    if (e < cnt && c < cols && !(solve && s_dst[e] < jb))
      v[i] = LoadGlobal(b + s_src[e] + c * p.lda);
  }
  if (solve) {
    for (int i = tid; i < kPanelW * kSwapCols; i += kSwapThreads) {
      const int r = i % kPanelW, c = i / kPanelW;
      if (r < jb && c < cols) CopyElement(s_b + c * kLd + r, b + s_top[r] + c * p.lda);
      else s_b[c * kLd + r] = Zero<T>();
    }
  }
  CpAsyncCommit();
  CpAsyncWait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = (tid + i * kSwapThreads) % kMovesMax, c = (tid + i * kSwapThreads) / kMovesMax;
    if (e < cnt && c < cols && !(solve && s_dst[e] < jb))
      StoreGlobal(b + s_dst[e] + c * p.lda, v[i]);
  }
  if (!solve) return;
  // The recursion's split (src/trsm.cc:87-135): 32 rows, the product, the rest.
  const int r1 = min(jb, 32), r2 = jb - r1, lane = tid % 32, c = tid / 32 * 2;
  static_assert(kSwapCols == 2 * (kSwapThreads / 32), "two columns a warp");
  const T* l1 = s_l + min(lane, jb - 1) * kLd;
  const T* b0 = s_b + c * kLd;
  const T* b1 = b0 + kLd;
  T y[2] = {b0[lane], b1[lane]};
  LaneSolve<T, 2>(l1, r1, y);
  T z[2] = {Zero<T>(), Zero<T>()};
  if (r2 > 0) {
    const T* l2 = s_l + min(32 + lane, jb - 1) * kLd;
    z[0] = b0[32 + lane];
    z[1] = b1[32 + lane];
    if constexpr (ElemOf<T>::kComplex) {
      using R = RealOf<T>;
      R acc[2][4] = {};
#pragma unroll 2
      for (int q = 0; q < 32; ++q) {
        const T l = l2[q];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const T yq = Shfl(y[i], q);
          acc[i][0] = Fma(l.re, yq.re, acc[i][0]);
          acc[i][1] = Fma(l.im, yq.re, acc[i][1]);
          acc[i][2] = Fma(l.re, yq.im, acc[i][2]);
          acc[i][3] = Fma(l.im, yq.im, acc[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        z[i] = MinusProduct(z[i], acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
      T acc[2] = {T(0), T(0)};
#pragma unroll 4
      for (int q = 0; q < 32; ++q) {
        const T l = l2[q];
        acc[0] = fma(l, __shfl_sync(0xffffffffu, y[0], q), acc[0]);
        acc[1] = fma(l, __shfl_sync(0xffffffffu, y[1], q), acc[1]);
      }
      z[0] = T(-1) * acc[0] + z[0];
      z[1] = T(-1) * acc[1] + z[1];
    }
    LaneSolve<T, 2>(l2 + 32, r2, z);
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    if (c + d >= cols) continue;
    T* col = b + (c + d) * p.lda;
    if (lane < r1) StoreGlobal(col + lane, y[d]);
    if (lane < r2) StoreGlobal(col + 32 + lane, z[d]);
  }
}

}  // namespace

namespace {
template <typename T>
bool LaunchPanel(int m, int n, T* a, int lda, int* ipiv, int ipiv_add, int* info, int info_base,
                 int* moves) {
  Context& ctx = Ctx();
  PanelArgs<T> args;
  int ctas = 0;
  if (n < 1 || n > kPanelW || m < n) return false;
  static PerDevice<int> clusters;
  const int max_cluster = clusters.Get([] {
    const void* fn = reinterpret_cast<const void*>(GetrfPanelKernel<T, kPanelCluster>);
    for (const void* f : {fn, reinterpret_cast<const void*>(GetrfPanelKernel<T, kPanelAlone>),
                          reinterpret_cast<const void*>(GetrfPanelKernel<T, kPanelSpin>)}) {
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(kPanelSmemMax)) != cudaSuccess ||
          cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
              cudaSuccess) {
        cudaGetLastError();
        return 0;
      }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kPanelCtas);
    cfg.blockDim = dim3(kPanelThreads<T>);
    cfg.dynamicSmemBytes = kPanelSmemMax;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kPanelCtas;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int size = 0;
    if (cudaOccupancyMaxPotentialClusterSize(&size, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      size = 1;
    }
    return std::min(size, kPanelCtas);
  });
  // Beside a capped trailing update a cluster of at most 8 CTAs finds its SMs
  // in one GPC soonest; larger panels take what they need.
  if (!PanelShape<T>(m, n, std::min(max_cluster, 8), &ctas, &args.R) &&
      !PanelShape<T>(m, n, max_cluster, &ctas, &args.R))
    return false;
  args.m = m;
  args.w = n;
  args.S = PanelStride(args.R);
  args.lanes = sizeof(RealOf<T>) == 8 ? RefLanesDouble() : 2 * RefLanesDouble();
  args.a = a;
  args.lda = lda;
  args.ipiv = ipiv;
  args.ipiv_add = ipiv_add;
  args.info = info;
  args.info_base = info_base;
  args.moves = moves;
  const uint32_t limit = g_panel_polls.load(std::memory_order_relaxed);
  args.polls = limit != 0 ? limit : kPanelPolls;
  args.timeout_flag = ctx.wait_flag;
  cudaEvent_t t0 = KernelTimerStart(kFamilyLuLeaf, ctx.stream);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(std::max(kPanelLeast, (args.R + 31) / 32 * 32));
  cfg.dynamicSmemBytes = PanelSmem<T>(n, args.R);
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ctas;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const auto kernel = ctas == 1    ? GetrfPanelKernel<T, kPanelAlone>
                      : limit == 0 ? GetrfPanelKernel<T, kPanelCluster>
                                   : GetrfPanelKernel<T, kPanelSpin>;
  if (cudaLaunchKernelEx(&cfg, kernel, args) != cudaSuccess) {
    cudaGetLastError();  // not launched: the caller goes down the recursion
    if (t0 != nullptr) cudaEventDestroy(t0);
    return false;
  }
  KernelTimerStop(t0, ctx.stream);
  CountLaunch();
  return true;
}
template <typename T>
void LaunchSwapTrsm(int j, int jb, int left, int c0, int nc, T* a, int lda, const int* moves) {
  const int blocks = (left + kSwapCols - 1) / kSwapCols + (nc + kSwapCols - 1) / kSwapCols;
  if (blocks == 0) return;
  static PerDevice<cudaError_t> attr;
  const auto set = [] {
    return cudaFuncSetAttribute(PanelSwapTrsmKernel<T>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, SwapSmem<T>());
  };
  if (Failed(attr.Get(set), "panel interchanges attributes")) return;
  SwapArgs<T> args;
  args.jb = jb;
  args.left = left;
  args.nc = nc;
  args.a = a + j;
  args.lda = lda;
  args.c0 = c0;
  args.l = a + j + static_cast<long long>(j) * lda;
  args.moves = moves;
  PanelSwapTrsmKernel<T><<<blocks, kSwapThreads, SwapSmem<T>(), Ctx().stream>>>(args);
  CountLaunch();
  LaunchFailed("panel interchanges");
}
}  // namespace

void SetPanelWaitLimit(unsigned int polls) {
  g_panel_polls.store(polls, std::memory_order_relaxed);
}

template <typename T>
bool GetrfPanel(int m, int n, T* a, int lda, int* ipiv, int ipiv_add, int* info, int info_base,
                int* moves) {
  return LaunchPanel<T>(m, n, a, lda, ipiv, ipiv_add, info, info_base, moves);
}
template <typename R>
bool ZGetrfPanel(int m, int n, R* a, int lda, int* ipiv, int ipiv_add, int* info, int info_base,
                 int* moves) {
  return LaunchPanel<Cx<R>>(m, n, reinterpret_cast<Cx<R>*>(a), lda, ipiv, ipiv_add, info,
                            info_base, moves);
}
template <typename T>
void PanelSwapTrsm(int j, int jb, int left, int c0, int nc, T* a, int lda, const int* moves) {
  LaunchSwapTrsm<T>(j, jb, left, c0, nc, a, lda, moves);
}
template <typename R>
void ZPanelSwapTrsm(int j, int jb, int left, int c0, int nc, R* a, int lda, const int* moves) {
  LaunchSwapTrsm<Cx<R>>(j, jb, left, c0, nc, reinterpret_cast<Cx<R>*>(a), lda, moves);
}
template bool GetrfPanel<double>(int, int, double*, int, int*, int, int*, int, int*);
template bool GetrfPanel<float>(int, int, float*, int, int*, int, int*, int, int*);
template bool ZGetrfPanel<double>(int, int, double*, int, int*, int, int*, int, int*);
template bool ZGetrfPanel<float>(int, int, float*, int, int*, int, int*, int, int*);
template void PanelSwapTrsm<double>(int, int, int, int, int, double*, int, const int*);
template void PanelSwapTrsm<float>(int, int, int, int, int, float*, int, const int*);
template void ZPanelSwapTrsm<double>(int, int, int, int, int, double*, int, const int*);
template void ZPanelSwapTrsm<float>(int, int, int, int, int, float*, int, const int*);

}  // namespace hb
