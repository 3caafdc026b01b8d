// The triangular base solve of a warp (shared by the single-problem and the
// batched routines).
#pragma once

namespace hb {
namespace {

// N rows of X solved by a warp, lane s holding the element of step s (y): at
// step q lane q's element is final, goes round by shuffles, and every later
// lane takes its term, so each element's chain is over q ascending, as above,
// but the chains of a row run side by side. st: the triangle, row stride ld. The
// loop is rolled: unrolled for one thread a row, a launch fetched a thousand
// instructions to run each once (32 x 32 base: 10 us; 4 to 6 us so), and lanes
// along a column-major X read it coalesced.
template <bool kUnit, typename T, int N>
__device__ __forceinline__ void LaneSolveSteps(const T* st, int ld, T inv, int r, T (&y)[N]) {
  const int lane = threadIdx.x % 32;
#pragma unroll 8
  for (int q = 0; q < r; ++q) {
    const T l = st[q * ld + lane];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const T yq = __shfl_sync(0xffffffffu, kUnit ? y[i] : y[i] * inv, q);
      const T next = fma(-yq, l, y[i]);
      y[i] = lane > q ? next : !kUnit && lane == q ? yq : y[i];
    }
  }
}
template <typename T, int N>
__device__ __forceinline__ void LaneSolve(const T* st, int ld, T inv, int unit, int r, T (&y)[N]) {
  // A unit diagonal keeps the product with its reciprocal off the chain.
  if (unit) LaneSolveSteps<true, T, N>(st, ld, inv, r, y);
  else LaneSolveSteps<false, T, N>(st, ld, inv, r, y);
}

}  // namespace
}  // namespace hb
