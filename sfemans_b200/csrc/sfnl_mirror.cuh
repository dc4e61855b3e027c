// sfnl_mirror.cuh -- synthesis on the caller's grid theta_j = 2 pi j / N on the FP64 tensor cores, shared by the
// GRID products (sfnl_grid.cu) and the synthesis-only routines (sfnl_synth.cu).
//
// The grid of the reference (N = 2*m_max_pad-1, fft_parallel.F90:183; any N >= 1 here) has one symmetry for
// every N, theta_{N-j} = 2 pi - theta_j: with C_j the cosine sum and S_j the sine sum of a field at angle j,
// f_j = C_j + S_j and f_{N-j} = C_j - S_j, so nh = N/2 + 1 angles are evaluated.  For 8 points the sums of all
// modes are the contractions [8 points x m] x [m x nh] of the cosine and of the sine coefficients, run as
// mma.sync.m8n8k4.f64 tiles of 8 angles.  The matrix entries cos/sin(2 pi (n j mod N) / N) are gathered from an
// exact table of N entries in shared memory (the index advances by 4 j mod N per k-step), so no (m, N) matrix
// has to be kept in device memory and a call allocates nothing.
//
// A-fragment blocks: xs [point tile][field][k-step][cos, sin][32], lane (g, q) of a warp reading mode 4s+q of
// point g at a_frag_slot(q, g).
#pragma once
#include <cuda_runtime.h>

#include "sfnl_fold.cuh"
#include "sfnl_internal.h"

namespace sfnl {

struct MirrorGeo {
  int m, N;
  int nh;  // angles 0..nh-1 are evaluated; j and N-j are mirrors
  int NT;  // tiles of 8 angles
  int KS;  // k-steps of 4 modes
  int PT;  // 8-point tiles of a CTA's pass
};
inline MirrorGeo mirror_geo(int m, int N, int PT) { return {m, N, N / 2 + 1, (N / 2 + 8) / 8, (m + 3) / 4, PT}; }

// Warps of a CTA (2 to 8): as few as give its two phases, `n1` and `n2` equal items of `c1` and `c2` DMMAs shared
// out over the warps, the shortest time.  At m = 32 a pass of the quotient v / s has 6 synthesis and 8 analysis
// items: 8 warps leave two idle in the first phase, 6 warps would run the second one twice.
inline int mirror_warps(int n1, int c1, int n2, int c2) {
  int best = 8;
  int64_t t8 = INT64_MAX;
  for (int w = 8; w >= 2; --w) {
    const int64_t t = (int64_t)((n1 + w - 1) / w) * c1 + (int64_t)((n2 + w - 1) / w) * c2;
    if (t <= t8) {
      t8 = t;
      best = w;
    }
  }
  return best;
}

// cos and sin of 2 pi r / N: the quadrant k is taken out in integers, so that the rounded argument stays within
// pi/4 of it.
__device__ __forceinline__ void mirror_table(double *ctab, double *stab, int N) {
  for (int r = threadIdx.x; r < N; r += blockDim.x) {
    const int64_t k = (8 * (int64_t)r + N) / (2 * (int64_t)N);  // nearest quadrant boundary, 0..4
    double s, c;
    sincospi((double)(4 * (int64_t)r - k * N) / (double)(2 * (int64_t)N), &s, &c);
    ctab[r] = (k & 3) == 0 ? c : (k & 3) == 1 ? -s : (k & 3) == 2 ? -c : s;
    stab[r] = (k & 3) == 0 ? s : (k & 3) == 1 ? c : (k & 3) == 2 ? -s : -c;
  }
}

// Copies the NI fields of the 8*PT points from p0 into xs with cp.async (one group, not waited for): field f's
// cosine of mode n, point p is at in(f)[p + n*ldm(f)], its sine np further.  A thread copies two neighbouring
// points of one row for every field; v16: the rows that start 16-byte aligned (rows16).  The sine of mode 0 is
// ignored (fft_parallel.F90:241); points past np are the constant PAD: 1 for programs that divide, as a quotient of
// zeros leaves the divider's short path, for all lanes of its warp (tension tensor, m = 8, 1,701 points 16.6 -> 11.5 us).
template <int NI, int PAD, typename In, typename Ldm>
__device__ __forceinline__ void mirror_stage(double *xs, const MirrorGeo &g, In in, Ldm ldm, int64_t p0, int64_t np,
                                             int v16) {
  const int pairs = 4 * g.PT, rows = 8 * g.KS;  // rows: (mode, cos/sin)
  for (int i = threadIdx.x; i < pairs * rows; i += blockDim.x) {
    const int pr = i % pairs, row = i / pairs, c = row & 1, n = row >> 1;
    const int64_t p = p0 + 2 * pr;
    const bool live = n < g.m && !(c == 1 && n == 0);
    const bool l0 = live && p < np, l1 = live && p + 1 < np;
    double *dst = xs + ((size_t)((pr >> 2) * NI * g.KS + (n >> 2)) * 2 + c) * 32 + a_frag_slot(n & 3, (2 * pr) & 7);
#pragma unroll
    for (int f = 0; f < NI; ++f, dst += (size_t)g.KS * 64) {
      const double *src = in(f) + p + (int64_t)n * ldm(f) + (c ? np : 0);
      if (l1 && ((v16 >> c) & 1)) {
        cp_async16(dst, src);
      } else {
        const double none = PAD != 0 && row == 0 ? (double)PAD : 0.0;
        if (l0) cp_async8(dst, src); else dst[0] = none;
        if (l1) cp_async8(dst + 1, src + 1); else dst[1] = none;
      }
    }
  }
  cp_async_commit();
}

// Cosine and sine sums of PW neighbouring point tiles (first: xt) at the 8 angles of tile t:
// acc[w][f][0 cos, 1 sin][e], lane (g, q) holding point g and angle 8t + 2q + e.  ADJ: bit f set = field f is a
// cotangent (synthesised with the analysis weights).  The modes are added from the highest down: with a decaying
// spectrum the partial sums stay small until the last terms, and the quotients, whose divisor can come close to
// zero, lose less than in the other order.
template <int NI, int PW, unsigned ADJ>
__device__ __forceinline__ void mirror_synth(const double *xt, const double *ctab, const double *stab,
                                             const MirrorGeo &g, int t, double (&acc)[PW][NI][2][2]) {
  const int lane = threadIdx.x & 31, gg = lane >> 2, q = lane & 3;
  const int j = 8 * t + gg;
  int r = ((4 * (g.KS - 1) + q) * j) % g.N;
  const int dr = g.N - (4 * j) % g.N;
#pragma unroll
  for (int w = 0; w < PW; ++w)
#pragma unroll
    for (int f = 0; f < NI; ++f)
#pragma unroll
      for (int c = 0; c < 2; ++c) acc[w][f][c][0] = acc[w][f][c][1] = 0.0;
  const double *xl = xt + a_frag_slot(q, gg);
#pragma unroll 2
  for (int s = g.KS - 1; s >= 0; --s) {
    const double b[2] = {ctab[r], stab[r]};
    r += dr;
    r = r >= g.N ? r - g.N : r;
#pragma unroll
    for (int w = 0; w < PW; ++w)
#pragma unroll
      for (int f = 0; f < NI; ++f)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          double av = xl[((size_t)((w * NI + f) * g.KS + s) * 2 + c) * 32];
          if constexpr (ADJ != 0)
            if ((ADJ >> f) & 1u) av *= (s == 0 && q == 0) ? 1.0 / (double)g.N : 2.0 / (double)g.N;
          dmma(acc[w][f][c], av, b[c]);
        }
  }
}

}  // namespace sfnl
