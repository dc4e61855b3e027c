// sfnl_synth.cu -- synthesis-only routines on the caller's grid.
//
//   FFT_PAR_REAL     (fft_parallel.F90:28-145)     values of every field at theta_j = 2 pi j / N
//   FFT_MAX_VEL_DCL  (fft_parallel.F90:1426-1541)  max over points and angles of |v|
//
// Both evaluate f(theta) = a_0 + sum_{n<m} a_n cos(n theta) + b_n sin(n theta) (the c2r of the
// half-complex pack of :88-112, :1497-1511, whose sine of mode 0 is ignored) on the N = 2*m_max_pad-1
// angles of the reference grid.  The mirror symmetry of that grid, theta_{N-j} = 2 pi - theta_j, is
// folded out: with C_j the cosine part and S_j the sine part at angle j, f_j = C_j + S_j and
// f_{N-j} = C_j - S_j, so N/2 + 1 angles are evaluated.
//
// Two kernels.  mirror_synth_kernel takes every size whose tile fits in shared memory: 8-point tiles on the FP64
// tensor cores (sfnl_mirror.cuh).  synth_kernel (one warp per point, lanes owning angles) is the fallback beyond.
// FFT_PAR_REAL writes the angles of one field contiguously (V_out(N, nf, np), angle fastest); FFT_MAX_VEL_DCL
// reduces |v| (the first 3-vector when there are six slots, |first field| otherwise, :1527-1532) to one maximum
// per point (host entry: the points' maxima are reduced on the host) or per launch with an integer atomic max on
// the bit patterns (device entry: non-negative doubles order like their bits).
#include <cuda_runtime.h>

#include "sfnl_internal.h"
#include "sfnl_mirror.cuh"

namespace sfnl {

namespace {

constexpr int kSynthThreads = 128;

// The larger one, or a NaN that either is (fmax would drop it).
__device__ __forceinline__ double max_nan(double a, double b) { return b > a || b != b ? b : a; }

// MODE 0: grid values to out (N, nslot/2, np); 1: maximum of |v| into *vmax (atomic); 2: maximum of
// |v| of each point to out[p].
template <int MODE>
__global__ void __launch_bounds__(kSynthThreads) synth_kernel(const double *v, double *out, unsigned long long *vmax,
                                                              int64_t np, int nslot, int m, int N, int warps_per_cta) {
  constexpr bool MAXV = MODE != 0;
  extern __shared__ __align__(16) double smem[];
  const int nf = nslot / 2;
  double2 *tab = reinterpret_cast<double2 *>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *X = smem + 2 * N + (size_t)warp * nslot * m;  // X[f][0..m) cos, X[f][m..2m) sin
  for (int r = threadIdx.x; r < N; r += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)r / (double)N, &s, &c);
    tab[r] = make_double2(c, s);
  }
  __syncthreads();
  if (warp >= warps_per_cta) return;
  const int nh = N / 2 + 1;  // angles 0..nh-1 and their mirrors N-j (0, and N/2 of an even grid, are their own)
  double vm = 0.0;
  for (int64_t p = (int64_t)blockIdx.x * warps_per_cta + warp; p < np; p += (int64_t)gridDim.x * warps_per_cta) {
    for (int idx = lane; idx < nslot * m; idx += 32) {
      const int f = idx / (2 * m), k = idx - f * 2 * m;
      const int n = k < m ? k : k - m;
      // cos of mode n of field f is slot 2f, sine slot 2f+1; the sine of mode 0 is ignored
      X[idx] = (k == m) ? 0.0 : __ldg(v + p + (int64_t)np * ((k < m ? 2 * f : 2 * f + 1) + (int64_t)nslot * n));
    }
    __syncwarp();
    const int nfe = MAXV ? (nslot == 6 ? 3 : 1) : nf;  // fields that matter
    for (int j = lane; j < nh; j += 32) {
      double fp[3] = {0.0, 0.0, 0.0}, fm[3] = {0.0, 0.0, 0.0};
      for (int f = 0; f < nfe; ++f) {
        const double *xc = X + (size_t)f * 2 * m, *xs = xc + m;
        double C = 0.0, S = 0.0;
        int r = 0;  // n*j mod N
        for (int n = 0; n < m; ++n) {
          const double2 cs = tab[r];
          C = fma(xc[n], cs.x, C);
          S = fma(xs[n], cs.y, S);
          r += j;
          if (r >= N) r -= N;
        }
        if constexpr (MAXV) {
          fp[f] = C + S;
          fm[f] = C - S;
        } else {
          double *o = out + (size_t)N * (f + (int64_t)nf * p);
          o[j] = C + S;
          if (j > 0 && 2 * j != N) o[N - j] = C - S;
        }
      }
      if constexpr (MAXV) {
        const double a = sqrt(fp[0] * fp[0] + fp[1] * fp[1] + fp[2] * fp[2]);
        const double bm = sqrt(fm[0] * fm[0] + fm[1] * fm[1] + fm[2] * fm[2]);
        vm = max_nan(vm, a);
        if (j > 0) vm = max_nan(vm, bm);
      }
    }
    if constexpr (MODE == 2) {
      for (int off = 16; off > 0; off >>= 1) vm = max_nan(vm, __shfl_xor_sync(0xffffffffu, vm, off));
      if (lane == 0) out[p] = vm;
      vm = 0.0;
    }
    __syncwarp();
  }
  if constexpr (MODE == 1) {
    for (int off = 16; off > 0; off >>= 1) vm = max_nan(vm, __shfl_xor_sync(0xffffffffu, vm, off));
    if (lane == 0) atomicMax(vmax, (unsigned long long)__double_as_longlong(vm));
  }
}

// The same on 8-point tiles, NI fields at a time (blockIdx.y: field group; one group for the maxima).  Warp items
// (point tile, angle tile) hold f_j = C + S and f_{N-j} = C - S of their fields at (point, angle); the grid values
// meet in shared memory in the order of V_out, from where they are written as contiguous runs of NI*N values.
// A CTA walks over its tiles; the coefficients of the next one are copied (second buffer) while the current one is
// evaluated.  Measured on a B200 against one warp per point (synth_kernel): grid values of a 3-vector at 28,000
// points and m = 64 0.48 -> 0.072 ms, the maximum at 56,000 points and m = 32 (with its copy to the host)
// 0.411 -> 0.072 ms.
template <int MODE, int NI, int PW>
__global__ void __launch_bounds__(256, 2) mirror_synth_kernel(const double *v, double *out, unsigned long long *vmax,
                                                              int64_t np, int nslot, const MirrorGeo g,
                                                              const int vec16) {
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
  const int gg = lane >> 2, q = lane & 3, nf = nslot / 2, f0 = blockIdx.y * NI, N = g.N, pts = 8 * g.PT;
  const size_t xsz = (size_t)g.PT * NI * g.KS * 64;
  double *xs = smem, *os = xs + 2 * xsz;  // os: grid values [pts][NI][N] (MODE 0) or maxima [pts] (MODE 2)
  double *ctab = os + (MODE == 0 ? (size_t)pts * NI * N : MODE == 2 ? (size_t)pts : 0), *stab = ctab + N;
  unsigned long long *pm = reinterpret_cast<unsigned long long *>(os);
  auto in = [&](int f) { return v + (int64_t)2 * (f0 + f) * np; };
  auto ldm = [&](int) { return (int64_t)nslot * np; };
  const int64_t tiles = (np + pts - 1) / pts;
  mirror_stage<NI, 0>(xs, g, in, ldm, (int64_t)blockIdx.x * pts, np, vec16);
  mirror_table(ctab, stab, N);
  double vm = 0.0;
  int buf = 0;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
    const int64_t p0 = tile * pts;
    if constexpr (MODE == 2)
      for (int i = threadIdx.x; i < pts; i += blockDim.x) pm[i] = 0;
    cp_async_wait_0();
    __syncthreads();
    if (tile + gridDim.x < tiles)
      mirror_stage<NI, 0>(xs + (buf ^ 1) * xsz, g, in, ldm, (tile + gridDim.x) * pts, np, vec16);
    for (int it = warp; it < g.PT / PW * g.NT; it += NW) {
      const int t = it % g.NT, pg = it / g.NT;
      double acc[PW][NI][2][2];
      mirror_synth<NI, PW, 0>(xs + buf * xsz + (size_t)pg * PW * NI * g.KS * 64, ctab, stab, g, t, acc);
#pragma unroll
      for (int w = 0; w < PW; ++w) {
      const int pt = pg * PW + w;
      double pv = 0.0;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 8 * t + 2 * q + e;
        if (j >= g.nh) continue;
        double sp = 0.0, sm = 0.0;
#pragma unroll
        for (int f = 0; f < NI; ++f) {
          const double fp = acc[w][f][0][e] + acc[w][f][1][e], fm = acc[w][f][0][e] - acc[w][f][1][e];
          if constexpr (MODE == 0) {
            double *o = os + ((size_t)(8 * pt + gg) * NI + f) * N;
            o[j] = fp;
            if (j > 0 && 2 * j != N) o[N - j] = fm;
          }
          sp = fma(fp, fp, sp);
          sm = fma(fm, fm, sm);
        }
        if constexpr (MODE != 0) pv = max_nan(pv, max_nan(sp, sm));  // the root of the maximum is the maximum of the roots
      }
      if constexpr (MODE == 1) vm = max_nan(vm, pv);
      if constexpr (MODE == 2) {
        for (int off = 2; off > 0; off >>= 1) pv = max_nan(pv, __shfl_xor_sync(0xffffffffu, pv, off));
        if (q == 0) atomicMax(pm + 8 * pt + gg, (unsigned long long)__double_as_longlong(sqrt(pv)));
      }
      }
    }
    if constexpr (MODE != 1) {
      __syncthreads();
      const int live = (int)(np - p0 < pts ? np - p0 : pts);
      if constexpr (MODE == 2) {
        for (int i = threadIdx.x; i < live; i += blockDim.x) out[p0 + i] = os[i];
      } else if (nf == NI) {  // one contiguous run of all points
        double *o = out + (size_t)N * nf * p0;
        for (int i = threadIdx.x; i < live * NI * N; i += blockDim.x) o[i] = os[i];
      } else {
        for (int pt = warp; pt < live; pt += NW) {
          double *o = out + (size_t)N * (f0 + (size_t)nf * (p0 + pt));
          for (int i = lane; i < NI * N; i += 32) o[i] = os[(size_t)pt * NI * N + i];
        }
      }
      __syncthreads();  // the next tile rewrites os
    }
  }
  if constexpr (MODE == 1) {
    for (int off = 16; off > 0; off >>= 1) vm = max_nan(vm, __shfl_xor_sync(0xffffffffu, vm, off));
    if (lane == 0) atomicMax(vmax, (unsigned long long)__double_as_longlong(sqrt(vm)));
  }
}

// SFNL_OK / an error of the launch, or 1 when the tile does not fit in shared memory.
template <int MODE, int NI, int PW>
int launch_mirror_synth(const double *v, double *out, double *vmax, int64_t np, int nslot, int m, int N, int groups,
                        cudaStream_t st) {
  MirrorGeo g = mirror_geo(m, N, PW);
  auto bytes = [&](int pt) {
    const size_t per = 2 * (size_t)NI * g.KS * 64 + (MODE == 0 ? (size_t)8 * NI * N : MODE == 2 ? 8 : 0);
    return sizeof(double) * ((size_t)pt * per + 2 * (size_t)N);
  };
  if constexpr (PW == 2) {
    // two point tiles share each table entry where two CTAs of such tiles fit on an SM
    if (bytes(2) > 100 * 1024) return launch_mirror_synth<MODE, NI, 1>(v, out, vmax, np, nslot, m, N, groups, st);
  }
  if (bytes(PW) > 200 * 1024) return 1;
  while (g.PT < 8 && g.PT / PW * g.NT < 8 && bytes(2 * g.PT) <= 100 * 1024) g.PT *= 2;
  const size_t smem = bytes(g.PT);
  auto kern = mirror_synth_kernel<MODE, NI, PW>;
  const int nw = mirror_warps(g.PT / PW * g.NT, 1, 0, 0);
  static KernelSetup setup;
  const int per_sm = setup.resident(reinterpret_cast<const void *>(kern), nw * 32, smem);
  if (per_sm < 0) return per_sm;
  const int vec16 = (reinterpret_cast<uintptr_t>(v) & 15) || (nslot & 1) ? 0 : rows16(np);
  const int64_t tiles = (np + 8 * g.PT - 1) / (8 * g.PT), cap = (int64_t)num_sms() * per_sm;
  kern<<<dim3((unsigned)(tiles < cap ? tiles : cap), (unsigned)groups), nw * 32, smem, st>>>(
      v, out, reinterpret_cast<unsigned long long *>(vmax), np, nslot, g, vec16);
  return check_launch("synthesis");
}

template <int MODE>
int launch_synth(const double *v, double *out, double *vmax, int64_t np, int nslot, int m, int N, cudaStream_t st) {
  // the fields that are evaluated, three at a time where they come in threes
  const int nfe = MODE == 0 ? nslot / 2 : nslot == 6 ? 3 : 1;
  if (nfe / 3 <= 65535 && nfe % 3 == 0) {
    if (const int rc = launch_mirror_synth<MODE, 3, 2>(v, out, vmax, np, nslot, m, N, nfe / 3, st); rc <= 0) return rc;
  }
  if (nfe <= 65535) {
    if (MODE == 0 || nfe == 1)
      if (const int rc = launch_mirror_synth<MODE, 1, 2>(v, out, vmax, np, nslot, m, N, nfe, st); rc <= 0) return rc;
  }
  const size_t tab_bytes = sizeof(double) * 2 * (size_t)N, per_warp = sizeof(double) * (size_t)nslot * m;
  const size_t budget = 200 * 1024;
  if (tab_bytes + per_warp > budget) return set_error(SFNL_ERR_UNSUPPORTED, "synthesis: m or N too large for shared memory");
  int warps = (int)((budget - tab_bytes) / per_warp);
  if (warps > kSynthThreads / 32) warps = kSynthThreads / 32;
  const size_t smem = tab_bytes + per_warp * warps;
  auto kern = synth_kernel<MODE>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return set_error(SFNL_ERR_CUDA, "cudaFuncSetAttribute failed (synthesis)");
  int64_t blocks = (np + warps - 1) / warps;
  const int64_t cap = (int64_t)num_sms() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  kern<<<(unsigned)blocks, kSynthThreads, smem, st>>>(v, out, reinterpret_cast<unsigned long long *>(vmax), np, nslot,
                                                      m, N, warps);
  return check_launch("synthesis");
}

}  // namespace

int launch_real(const double *v, double *out, int64_t np, int nslot, int m, int N, cudaStream_t st) {
  if (np == 0) return SFNL_OK;
  return launch_synth<0>(v, out, nullptr, np, nslot, m, N, st);
}

// vmax: device double, not reset here (the caller zeroes it first)
int launch_max_vel(const double *v, double *vmax, int64_t np, int nslot, int m, int N, cudaStream_t st) {
  if (np == 0) return SFNL_OK;
  return launch_synth<1>(v, nullptr, vmax, np, nslot, m, N, st);
}

int launch_point_max_vel(const double *v, double *pmax, int64_t np, int nslot, int m, int N, cudaStream_t st) {
  if (np == 0) return SFNL_OK;
  return launch_synth<2>(v, pmax, nullptr, np, nslot, m, N, st);
}

}  // namespace sfnl
