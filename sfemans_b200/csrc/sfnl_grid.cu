// sfnl_grid.cu -- all-FP64 products on the caller's grid (SFNL_ALGO_GRID).
//
// Dense DFT on the grid the reference uses, N = 2*m_max_pad-1
// (fft_parallel.F90:183): synthesis f(theta_j) = a_0 + sum_n a_n cos(n theta_j)
// + b_n sin(n theta_j) (the c2r of :261-267 applied to the half-complex pack
// of :223-241), the pointwise program, then analysis a_n = (c_n/N) sum_j g_j
// cos(n theta_j), b_n = (2/N) sum_j g_j sin(n theta_j), n < m (the r2c, 1/N,
// 2*CONJG and truncation of :278-299).  Angles come from an exact table
// cos/sin(2 pi r / N) indexed by (n*j mod N), so the arithmetic is the same
// for every N, odd or even, dealiasing or not: with a pad too short to
// dealias it reproduces the reference's aliased result.
//
// Two kernels.  mirror_kernel takes every size whose tile fits in shared memory (with the reference's grid to m = 144
// for the cross product, 200 for the dot product, 176 for v / s, 80 for the tensors): the mirror j -> N-j of the grid is folded out and the remaining contractions run on the FP64 tensor
// cores, 8-point tiles staged with cp.async (sfnl_mirror.cuh).  grid_kernel (one warp per point, the coefficients
// broadcast from shared memory, lanes owning angles and then modes) is the fallback beyond.  This form is the
// parity anchor, and the only form of the programs that depend on the grid (the quotients and the tension
// tensor); the fast and split forms carry the throughput of the products.
#include <cuda_runtime.h>

#include "sfnl_internal.h"
#include "sfnl_mirror.cuh"
#include "sfnl_ops.cuh"

namespace sfnl {

namespace {

constexpr int kGridThreads = 128;

template <int OP>
__global__ void __launch_bounds__(kGridThreads) grid_kernel(const ProgArgs a, int warps_per_cta, int per_warp) {
  constexpr int NI = op_nin(OP), NO = op_nout(OP);
  extern __shared__ __align__(16) double smem[];
  const int N = a.N, m = a.m;
  double2 *tab = reinterpret_cast<double2 *>(smem);
  const int tab_doubles = 2 * N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *X = smem + tab_doubles + (size_t)warp * per_warp;  // NI x 2m
  double *G = X + NI * 2 * m;                                  // NO x N

  for (int r = threadIdx.x; r < N; r += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)r / (double)N, &s, &c);
    tab[r] = make_double2(c, s);
  }
  __syncthreads();
  if (warp >= warps_per_cta) return;

  const int b = blockIdx.y;
  const double invN = 1.0 / (double)N, twoN = 2.0 / (double)N;
  for (int64_t p = (int64_t)blockIdx.x * warps_per_cta + warp; p < a.np; p += (int64_t)gridDim.x * warps_per_cta) {
    // 1. stage the point's coefficients: X[f][k], k < m cos, k >= m sin.
    for (int idx = lane; idx < NI * 2 * m; idx += 32) {
      const int f = idx / (2 * m), k = idx - f * 2 * m;
      const int n = k < m ? k : k - m;
      double v = 0.0;
      if (k != m) {  // the sine of mode 0 is ignored (fft_parallel.F90:241)
        const double *src = a.in[f] + (int64_t)b * a.in_bs[f] + p + (int64_t)n * a.in_ldm[f] + (k >= m ? a.np : 0);
        v = __ldg(src);
      }
      if (op_adjoint_in(OP, f)) v *= (n == 0 ? invN : twoN);
      X[idx] = v;
    }
    __syncwarp();
    // 2. synthesis + program at the lane's angles.
    for (int j = lane; j < N; j += 32) {
      double x[NI];
#pragma unroll
      for (int f = 0; f < NI; ++f) x[f] = 0.0;
      int r = 0;  // n*j mod N
      for (int n = 0; n < m; ++n) {
        const double2 cs = tab[r];
#pragma unroll
        for (int f = 0; f < NI; ++f) x[f] = fma(X[f * 2 * m + n], cs.x, fma(X[f * 2 * m + m + n], cs.y, x[f]));
        r += j;
        if (r >= N) r -= N;
      }
      double y[NO];
      apply_op<OP>(x, y);
#pragma unroll
      for (int o = 0; o < NO; ++o) G[o * N + j] = y[o];
    }
    __syncwarp();
    // 3. analysis of the lane's modes, truncated to n < m.
    for (int n = lane; n < m; n += 32) {
      double ya[NO], yb[NO];
#pragma unroll
      for (int o = 0; o < NO; ++o) ya[o] = yb[o] = 0.0;
      int r = 0;  // n*j mod N
      for (int j = 0; j < N; ++j) {
        const double2 cs = tab[r];
#pragma unroll
        for (int o = 0; o < NO; ++o) {
          const double g = G[o * N + j];
          ya[o] = fma(g, cs.x, ya[o]);
          yb[o] = fma(g, cs.y, yb[o]);
        }
        r += n;
        if (r >= N) r -= N;
      }
      const double sc = op_adjoint_out(OP) ? 1.0 : (n == 0 ? invN : twoN);
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        double *dst = a.out[o] + (int64_t)b * a.out_bs[o] + p * a.out_ps + (int64_t)n * a.out_ldm[o];
        dst[0] = ya[o] * sc;
        dst[a.np * a.out_ps] = (n == 0) ? 0.0 : yb[o] * sc;
      }
    }
    __syncwarp();
  }
}

// The program on 8-point tiles.  Synthesis: warp items (pair of point tiles, angle tile); the lane that holds
// f_j = C + S and f_{N-j} = C - S of every field at its (point, angle) evaluates the program at both angles and
// stores P = g_j + g_{N-j} and Q = g_j - g_{N-j} in the order in which the analysis reads them as A fragments
// (P = g_j at an angle that is its own mirror).  Analysis: warp items (pair of point tiles, cos/sin, tile of 8
// modes), a_n = c_n/N sum P cos(n theta_j), b_n = 2/N sum Q sin(n theta_j).  A CTA walks over its tiles; the next
// tile's coefficients are copied while the current one is analysed.
// Measured on a B200 against one warp per point (grid_kernel), 28,000 points: v / s 0.334 -> 0.073 ms at m = 32 and
// 1.26 -> 0.22 ms at m = 64, the tension tensor 1.97 -> 0.58 ms at m = 64, c1 / c2 0.96 -> 0.10 ms.  At m = 32 the
// FP64 and DMMA pipes are busy 55 % of the time (grid_kernel waited for its shared-memory broadcasts); the rest is
// the two barriers of a pass.
template <int OP, int PW>
__global__ void __launch_bounds__(256, op_nin(OP) <= 6 ? 2 : 1) mirror_kernel(const ProgArgs a, const MirrorGeo g,
                                                                              const int vec16) {
  constexpr int NI = op_nin(OP), NO = op_nout(OP);
  constexpr unsigned ADJ = OP == OP_CROSS_VJP ? 0x1C0u : OP == OP_MHD_VJP ? 0x7E00u : 0u;
  constexpr int PAD = OP == OP_DIV || OP == OP_SVDIV || OP == OP_TENSION;
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  const int gg = lane >> 2, q = lane & 3, b = blockIdx.y;
  double *xs = smem, *ps = xs + (size_t)g.PT * NI * g.KS * 64;
  double *ctab = ps + (size_t)g.PT * NO * g.NT * 128, *stab = ctab + g.N;
  const int NU = (g.m + 7) / 8, PG = g.PT / PW;
  auto in = [&](int f) { return a.in[f] + (int64_t)b * a.in_bs[f]; };
  auto ldm = [&](int f) { return a.in_ldm[f]; };
  const int64_t tiles = (a.np + 8 * g.PT - 1) / (8 * g.PT);
  mirror_stage<NI, PAD>(xs, g, in, ldm, (int64_t)blockIdx.x * 8 * g.PT, a.np, vec16);
  mirror_table(ctab, stab, g.N);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t p0 = tile * 8 * g.PT;
    cp_async_wait_0();
    __syncthreads();
    for (int it = warp; it < PG * g.NT; it += NW) {
      const int t = it % g.NT, pg = it / g.NT;
      double acc[PW][NI][2][2];
      mirror_synth<NI, PW, ADJ>(xs + (size_t)pg * PW * NI * g.KS * 64, ctab, stab, g, t, acc);
#pragma unroll
      for (int w = 0; w < PW; ++w)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = 8 * t + 2 * q + e;
          double xp[NI], xm[NI], yp[NO], ym[NO];
#pragma unroll
          for (int f = 0; f < NI; ++f) {
            xp[f] = acc[w][f][0][e] + acc[w][f][1][e];
            xm[f] = acc[w][f][0][e] - acc[w][f][1][e];
          }
          apply_op<OP>(xp, yp);
          apply_op<OP>(xm, ym);
          double *dst = ps + ((size_t)(pg * PW + w) * NO * 2 * g.NT + t) * 64 + e * 32 + lane;
#pragma unroll
          for (int o = 0; o < NO; ++o, dst += (size_t)g.NT * 128) {
            const bool self = j == 0 || 2 * j == g.N, live = j < g.nh;
            dst[0] = !live ? 0.0 : self ? yp[o] : yp[o] + ym[o];
            dst[(size_t)g.NT * 64] = !live || self ? 0.0 : yp[o] - ym[o];
          }
        }
    }
    __syncthreads();
    if (tile + gridDim.x < tiles)
      mirror_stage<NI, PAD>(xs, g, in, ldm, (tile + gridDim.x) * 8 * g.PT, a.np, vec16);
    for (int it = warp; it < PG * 2 * NU; it += NW) {
      const int u = it % NU, c = (it / NU) & 1, pg = it / (2 * NU);
      constexpr int PC = NO * PW >= 9 ? 1 : 2;  // independent partial sums per output
      double y[PC][PW][NO][2];
#pragma unroll
      for (int i = 0; i < PC; ++i)
#pragma unroll
        for (int w = 0; w < PW; ++w)
#pragma unroll
          for (int o = 0; o < NO; ++o) y[i][w][o][0] = y[i][w][o][1] = 0.0;
      const int n8 = 8 * u + gg;  // mode of the lane's B column
      const int rn = n8 % g.N, dr = (8 * n8) % g.N;
      int r = (2 * q * n8) % g.N;
      const double *tab = c ? stab : ctab;
      const double *pa = ps + ((size_t)pg * PW * NO * 2 + c) * g.NT * 64 + lane;
#pragma unroll 2
      for (int t = 0; t < g.NT; ++t) {
        int r1 = r + rn;
        r1 = r1 >= g.N ? r1 - g.N : r1;
        const double bv[2] = {tab[r], tab[r1]};
        r += dr;
        r = r >= g.N ? r - g.N : r;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int w = 0; w < PW; ++w)
#pragma unroll
            for (int o = 0; o < NO; ++o)
              dmma(y[e % PC][w][o], pa[((size_t)(w * NO + o) * 2 * g.NT + t) * 64 + e * 32], bv[e]);
      }
#pragma unroll
      for (int w = 0; w < PW; ++w) {
        const int64_t p = p0 + 8 * (pg * PW + w) + gg;
        if (p >= a.np) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = 8 * u + 2 * q + h;
          if (n >= g.m) continue;
          const double sc = op_adjoint_out(OP) ? 1.0 : (n == 0 ? 1.0 : 2.0) / (double)g.N;
#pragma unroll
          for (int o = 0; o < NO; ++o) {
            double v = y[0][w][o][h];
#pragma unroll
            for (int i = 1; i < PC; ++i) v += y[i][w][o][h];
            a.out[o][(int64_t)b * a.out_bs[o] + p * a.out_ps + (int64_t)n * a.out_ldm[o] + (c ? a.np * a.out_ps : 0)] =
                c && n == 0 ? 0.0 : v * sc;
          }
        }
      }
    }
  }
}

template <int OP, int PW>
size_t mirror_smem(const MirrorGeo &g) {
  return sizeof(double) * (size_t)g.PT * ((size_t)op_nin(OP) * g.KS * 64 + (size_t)op_nout(OP) * g.NT * 128) +
         sizeof(double) * 2 * (size_t)g.N;
}

template <int OP, int PW>
int launch_mirror_pw(const ProgArgs &a, const MirrorGeo &g, cudaStream_t st) {
  constexpr int NI = op_nin(OP);
  int vec16 = rows16(a.np);
  for (int f = 0; f < NI; ++f)
    if ((reinterpret_cast<uintptr_t>(a.in[f]) & 15) || (a.in_ldm[f] & 1) || (a.in_bs[f] & 1)) vec16 = 0;
  const size_t smem = mirror_smem<OP, PW>(g);
  auto kern = mirror_kernel<OP, PW>;
  const int nw = mirror_warps(g.PT / PW * g.NT, 2 * NI * g.KS, g.PT / PW * 2 * ((g.m + 7) / 8), 2 * op_nout(OP) * g.NT);
  static KernelSetup setup;
  const int per_sm = setup.resident(reinterpret_cast<const void *>(kern), nw * 32, smem);
  if (per_sm < 0) return per_sm;
  const int64_t tiles = (a.np + 8 * g.PT - 1) / (8 * g.PT), cap = (int64_t)num_sms() * per_sm;
  kern<<<dim3((unsigned)(tiles < cap ? tiles : cap), (unsigned)a.batch), nw * 32, smem, st>>>(a, g, vec16);
  return check_launch("grid form");
}

// SFNL_OK / an error of the launch, or 1 when the tile does not fit in shared memory.
template <int OP>
int launch_mirror(const ProgArgs &a, cudaStream_t st) {
  constexpr size_t kTwo = 100 * 1024, kOne = 200 * 1024;  // shared memory of a CTA at two and at one CTA per SM
  constexpr int NI = op_nin(OP);
  if constexpr (NI <= 4) {
    // two point tiles share each table entry (the accumulators of up to four fields fit in 128 registers), and a
    // pass takes as many point tiles as give its warps six items
    MirrorGeo g = mirror_geo(a.m, a.N, 2);
    while (g.PT < 8 && g.PT / 2 * g.NT < 6 && 2 * mirror_smem<OP, 2>(g) <= kTwo) g.PT *= 2;
    if (mirror_smem<OP, 2>(g) <= kTwo) return launch_mirror_pw<OP, 2>(a, g, st);
  }
  MirrorGeo g = mirror_geo(a.m, a.N, 1);
  while (g.PT < 8 && g.PT * g.NT < 6 && 2 * mirror_smem<OP, 1>(g) <= kTwo) g.PT *= 2;
  if (mirror_smem<OP, 1>(g) <= kOne) return launch_mirror_pw<OP, 1>(a, g, st);
  return 1;
}

template <int OP>
int launch_grid_op(const ProgArgs &a, cudaStream_t st) {
  constexpr int NI = op_nin(OP), NO = op_nout(OP);
  if (const int rc = launch_mirror<OP>(a, st); rc <= 0) return rc;
  const int per_warp = NI * 2 * a.m + NO * a.N;  // doubles
  const size_t tab_bytes = sizeof(double) * 2 * (size_t)a.N;
  const size_t budget = 200 * 1024;
  if (tab_bytes + sizeof(double) * (size_t)per_warp > budget) return set_error(SFNL_ERR_UNSUPPORTED, "grid form: m or N too large for shared memory");
  int warps = (int)((budget - tab_bytes) / (sizeof(double) * (size_t)per_warp));
  if (warps > kGridThreads / 32) warps = kGridThreads / 32;
  const size_t smem = tab_bytes + sizeof(double) * (size_t)per_warp * warps;
  auto kern = grid_kernel<OP>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return set_error(SFNL_ERR_CUDA, "cudaFuncSetAttribute failed (grid form)");
  int64_t blocks = (a.np + warps - 1) / warps;
  const int64_t cap = (int64_t)num_sms() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  dim3 grid((unsigned)blocks, (unsigned)a.batch);
  kern<<<grid, kGridThreads, smem, st>>>(a, warps, per_warp);
  return check_launch("grid form");
}

}  // namespace

int launch_grid(const ProgArgs &a, cudaStream_t st) {
  if (a.np == 0) return SFNL_OK;
  switch (a.op) {
    case OP_CROSS: return launch_grid_op<OP_CROSS>(a, st);
    case OP_DOT: return launch_grid_op<OP_DOT>(a, st);
    case OP_PROD: return launch_grid_op<OP_PROD>(a, st);
    case OP_BUNDLE: return launch_grid_op<OP_BUNDLE>(a, st);
    case OP_CROSS_JVP: return launch_grid_op<OP_CROSS_JVP>(a, st);
    case OP_CROSS_VJP: return launch_grid_op<OP_CROSS_VJP>(a, st);
    case OP_MHD_JVP: return launch_grid_op<OP_MHD_JVP>(a, st);
    case OP_MHD_VJP: return launch_grid_op<OP_MHD_VJP>(a, st);
    case OP_DIV: return launch_grid_op<OP_DIV>(a, st);
    case OP_SVECT: return launch_grid_op<OP_SVECT>(a, st);
    case OP_SVDIV: return launch_grid_op<OP_SVDIV>(a, st);
    case OP_TENSOR: return launch_grid_op<OP_TENSOR>(a, st);
    case OP_TENSION: return launch_grid_op<OP_TENSION>(a, st);
    case OP_ADVECT: return launch_grid_op<OP_ADVECT>(a, st);
  }
  return set_error(SFNL_ERR_ARG, "unknown program");
}

}  // namespace sfnl
