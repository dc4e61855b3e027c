// sfnl_res.cu -- the FAST form at m = 65 .. 512 on residue grids of M = 64 or 128 angles, with synthesis, program and
// analysis of a residue in one kernel.
//
// On theta_j = pi(2j+1)/N with N = M R >= 3m - 2, the angles j = R i + r are phi_i + d_r, phi_i = pi(2i+1)/M and
// d_r = pi(2r + 1 - R)/N.  As in sfnl_large.cu, a field is on residue r the transform of M real coefficients to M
// angles (mode n = M q + k of y_n = z_n e^{i n d_r} is mode k with the sign (-1)^q, and the modes k and M - k meet
// in one coefficient), third-folded; a product's sums on the residues add up to its coefficients.  Any m fits with
// R = ceil((3m - 2)/M) residues (4 to 12); a larger grid than the reference's changes nothing, the product being
// alias-free on both (fft_parallel.F90:147-328).
//
//   coef_kernel   inputs -> the R residues' coefficients of every field, one pass
//   base_kernel   (linearised programs) grid values of the fields that all tangents share
//   prod_kernel   per residue, batch entry and 8-point tile: synthesis of the other fields, program, analysis
//   out_kernel    the residues' sums -> outputs, one pass
//
// The two-kernel form of sfnl_large.cu wrote every field's grid values and read them back once per three outputs; here
// only coefficients and sums cross HBM.  Both live in tile blocks, [residue][instance][tile][M rows][8 points], the
// coefficients in the order of the A fragments, so that a field's tile is one contiguous copy whatever np is.
#include <cuda_runtime.h>

#include "sfnl_fold.cuh"
#include "sfnl_internal.h"
#include "sfnl_ops.cuh"

namespace sfnl {

namespace {

// Geometry of a residue grid of M angles (64 or 128).
template <int M>
struct Res {
  static constexpr int MH = M / 2, NT = M / 32;    // folded modes, quadrant angle tiles
  static constexpr int KSE = MH / 16;              // k-steps of an even group (an odd class has twice as many)
  static constexpr int KS = tf_koff(MH, 6);        // k-steps of 4 rows
  static constexpr int TILE = KS * 32;             // doubles of one field's tile
  static constexpr int THREADS = 64 * NT;          // two warps (cosine, sine classes) per angle tile
  static constexpr int BLOCKS = 24 / (2 * NT);     // CTAs per SM: 24 warps at 80 registers
  static constexpr int XC = 2 * NT * 3 * 64, PS = 3 * 4 * NT * 64;
  static constexpr size_t SMEM = sizeof(double) * (3 * TILE + XC + PS);  // 31 or 60 KB
  static_assert(KS == 8 * KSE && tf_KS(MH, 0) == KSE && tf_KS(MH, 1) == KSE && tf_KS(MH, 2) == 2 * KSE, "row groups");
  // Row of the cosine (groups 0-2) of folded mode k in group order CE0, CE2, CO; the sine is MH rows on.
  __host__ __device__ static constexpr int row_of(int k) {
    return k & 1 ? MH / 2 + (k >> 1) : k & 2 ? MH / 4 + (k >> 2) : k >> 2;
  }
};
__device__ __forceinline__ int coef_at(int row, int g) { return (row >> 2) * 32 + a_frag_slot(row & 3, g); }

// Fields a program synthesises per batch entry (the others are the base state of a linearised program) and the first.
constexpr bool linear_op(int op) {
  return op == OP_CROSS_JVP || op == OP_CROSS_VJP || op == OP_MHD_JVP || op == OP_MHD_VJP;
}
constexpr int first_own(int op) {
  return op == OP_CROSS_JVP || op == OP_CROSS_VJP ? 6 : op == OP_MHD_JVP || op == OP_MHD_VJP ? 9 : 0;
}

struct CoefArgs {
  const double *x[kMaxIn];
  int64_t ldm[kMaxIn], bs[kMaxIn];
  int inst[kMaxIn + 1];  // first instance of each field (its batch entries follow)
  unsigned adj;          // bit f: a cotangent, which takes the analysis weights
  int nf, m, b0;         // fields; modes; first batch entry
  int64_t np, npts, tiles;
  double *C;
  const double *tw;
  double invN;
};

// Thread (point, k): Y_k and Y_{M-k} of each residue from the modes M q + k and M q + M - k (k = 0: Y_0 and Y_{M/2}
// from M q and M q + M/2); writes alpha_k - i beta_k = Y_k - conj(Y_{M-k}) (k = 0: alpha_0 = Re Y_0 and beta_{M/2} =
// -Im Y_{M/2} in the sine row of mode 0).  Residues pair as d_{R-1-r} = -d_r: one twiddle serves two.
// The block's twiddles (one k: 2 QM modes of R/2 residues) sit in shared memory and all loads are issued first; with
// both left to the loop over the modes a pass reached 1 TB/s.  k runs fastest over the blocks, so that the 64-byte pieces
// of a tile are written together (six residues of 128 angles: 519 -> 338 us for 1.8 GB).  The passes run at 5.9 and 6.1
// TB/s with six residues of 64 angles (m = 128), at 4.4 and 5.5 with twelve (m = 256).
constexpr int res_qm(int R) { return (R + 2) / 3; }  // M q + k < m needs q < QM
template <int M, int R>
__device__ __forceinline__ void load_twiddles(double2 (&tw)[res_qm(R)][2][R / 2], const double *src, int m, int k) {
  constexpr int RP = R / 2, n_tw = res_qm(R) * 2 * RP;
  for (int i = threadIdx.x; i < n_tw; i += blockDim.x) {
    const int r = i % RP, side = (i / RP) & 1, q = i / (2 * RP);
    const int n = q * M + (side == 0 ? k : k == 0 ? M / 2 : M - k);
    tw[q][side][r] = n < m ? reinterpret_cast<const double2 *>(src)[(size_t)r * m + n] : make_double2(0.0, 0.0);
  }
}
template <int M, int R>
__global__ void __launch_bounds__(128) coef_kernel(const CoefArgs a) {
  constexpr int RP = R / 2, QM = res_qm(R), MH = Res<M>::MH, TILE = Res<M>::TILE;
  __shared__ double2 tw[QM][2][RP];
  const int64_t nblk = (a.npts + blockDim.x - 1) / blockDim.x, pb = blockIdx.x / MH;
  const int inst = (int)(pb / nblk), k = blockIdx.x & (MH - 1);
  const int64_t p = (pb - inst * nblk) * blockDim.x + threadIdx.x;
  int f = 0;
  while (f + 1 < a.nf && inst >= a.inst[f + 1]) ++f;
  const double *x = a.x[f] + (int64_t)(a.b0 + inst - a.inst[f]) * a.bs[f] + p;
  const int64_t ldm = a.ldm[f];
  const bool adj = (a.adj >> f) & 1u, valid = p < a.npts;
  double av[QM][2], bv[QM][2];
#pragma unroll
  for (int q = 0; q < QM; ++q)
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int n = q * M + (side == 0 ? k : k == 0 ? MH : M - k);
      const bool live = valid && n < a.m;
      av[q][side] = live ? x[(int64_t)n * ldm] : 0.0;
      bv[q][side] = live && n > 0 ? x[(int64_t)n * ldm + a.np] : 0.0;  // the sine of mode 0 is ignored
    }
  load_twiddles<M, R>(tw, a.tw, a.m, k);
  __syncthreads();
  if (!valid) return;
  double yr[2][R], yi[2][R];
#pragma unroll
  for (int side = 0; side < 2; ++side)
#pragma unroll
    for (int r = 0; r < R; ++r) yr[side][r] = yi[side][r] = 0.0;
#pragma unroll
  for (int q = 0; q < QM; ++q) {
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const double wn = (adj ? (q == 0 && side == 0 && k == 0 ? a.invN : 2.0 * a.invN) : 1.0) * ((q & 1) ? -1.0 : 1.0);
      const double aw = av[q][side] * wn, bw = bv[q][side] * wn;
#pragma unroll
      for (int r = 0; r < RP; ++r) {
        const double2 cs = tw[q][side][r];
        const double ac = aw * cs.x, bs = bw * cs.y, as = aw * cs.y, bc = bw * cs.x;
        yr[side][r] += ac + bs;
        yi[side][r] += as - bc;
        yr[side][R - 1 - r] += ac - bs;
        yi[side][R - 1 - r] -= as + bc;
      }
      if (R & 1) {
        yr[side][RP] += aw;
        yi[side][RP] -= bw;
      }
    }
  }
  const int64_t ninst = a.inst[a.nf];
  double *c = a.C + ((int64_t)inst * a.tiles + (p >> 3)) * TILE;
  const int row = Res<M>::row_of(k), ic = coef_at(row, (int)(p & 7)), is = coef_at(row + MH, (int)(p & 7));
#pragma unroll
  for (int r = 0; r < R; ++r, c += ninst * a.tiles * TILE) {
    c[ic] = k == 0 ? yr[0][r] : yr[0][r] - yr[1][r];
    c[is] = k == 0 ? -yi[1][r] : -(yi[0][r] + yi[1][r]);
  }
}

struct OutArgs {
  const double *S;
  double *out[kMaxOut];
  int64_t ldm[kMaxOut], bs[kMaxOut];
  int nb, no, m, b0;
  int64_t npts, tiles, osin, ops;
  double w, w0;
  const double *tw;
};

// Thread (point, k): the modes M q + k and M q + M - k (k = 0: M q and M q + M/2) of one output from the R residues'
// sums, c_n = sum_r e^{-i n d_r} P^r_n with P^r_k = C - i S, P^r_{M-k} = -conj(P^r_k), P^r_{M/2} = -i S_{M/2} and
// P^r_{Mq+k} = (-1)^q P^r_k.
template <int M, int R>
__global__ void __launch_bounds__(128) out_kernel(const OutArgs a) {
  constexpr int RP = R / 2, QM = res_qm(R), MH = Res<M>::MH, TILE = Res<M>::TILE;
  __shared__ double2 tw[QM][2][RP];
  const int64_t nblk = (a.npts + blockDim.x - 1) / blockDim.x, pb = blockIdx.x / MH;
  const int inst = (int)(pb / nblk), k = blockIdx.x & (MH - 1), o = inst / a.nb, b = inst - o * a.nb;
  const int64_t p = (pb - inst * nblk) * blockDim.x + threadIdx.x;
  const bool valid = p < a.npts;
  const double *s = a.S + ((int64_t)inst * a.tiles + (p >> 3)) * TILE + Res<M>::row_of(k) * 8 + (p & 7);
  double *op = a.out[o] + (int64_t)(a.b0 + b) * a.bs[o] + p * a.ops;
  const int64_t ldm = a.ldm[o], rst = (int64_t)a.no * a.nb * a.tiles * TILE;
  double C[R], Sv[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    C[r] = valid ? s[r * rst] : 0.0;
    Sv[r] = valid ? s[r * rst + MH * 8] : 0.0;
  }
  load_twiddles<M, R>(tw, a.tw, a.m, k);
  __syncthreads();
  if (!valid) return;
#pragma unroll
  for (int q = 0; q < QM; ++q) {
    const double sg = (q & 1) ? -1.0 : 1.0;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int n = q * M + (side == 0 ? k : k == 0 ? MH : M - k);
      if (n >= a.m) continue;
      auto px = [&](int r) { return side == 0 ? C[r] : k == 0 ? 0.0 : -C[r]; };
      auto py = [&](int r) { return side == 0 && k == 0 ? 0.0 : -Sv[r]; };
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int r = 0; r < RP; ++r) {
        const double2 cs = tw[q][side][r];
        const double x0 = px(r), y0 = py(r), x1 = px(R - 1 - r), y1 = py(R - 1 - r);
        re += fma(cs.x, x0 + x1, cs.y * (y0 - y1));
        im += fma(cs.x, y0 + y1, -cs.y * (x0 - x1));
      }
      if (R & 1) {
        re += px(RP);
        im += py(RP);
      }
      const double wn = (n == 0 ? a.w0 : a.w) * sg;
      op[(int64_t)n * ldm] = wn * re;
      op[(int64_t)n * ldm + a.osin] = n == 0 ? 0.0 : -wn * im;
    }
  }
}

struct ProdArgs {
  const double *C;       // coefficients
  double *G;             // grid values of the shared fields, [residue][field][tile][angle tile][quadrant][e][32]
  double *S;             // sums
  const double *syn, *ana;
  int64_t tiles, ninst;  // instances of a residue in C
  int inst[kMaxIn];      // first instance of each field
  int nshared, nb;
};

// One tile of a residue: copies of the next fields, synthesis and folds of the current ones, analysis of products.
template <int M>
struct Tile {
  static constexpr int kNT = Res<M>::NT, kTile = Res<M>::TILE, kThreads = Res<M>::THREADS, KSE = Res<M>::KSE, MH = Res<M>::MH;
  double *xs, *xc, *ps;  // staged coefficients [3][KS][32], exchange, folded products [3][4][kNT][2][32]
  const double *syn, *ana;
  int lane, warp, tau, half;

  template <int NG>
  __device__ __forceinline__ void stage(const double *const (&src)[NG]) const {
#pragma unroll
    for (int f = 0; f < NG; ++f)
#pragma unroll
      for (int i = 0; i < kTile / 2 / kThreads; ++i) {
        const int e = 2 * ((int)threadIdx.x + i * kThreads);
        cp_async16(xs + f * kTile + e, src[f] + e);
      }
    cp_async_commit();
  }
  // The four quadrant values of NG staged fields at the lane's point and its angle 8 tau + 2 q + half; `next` starts
  // the following copies as soon as the staged rows are read.
  template <int NG, typename Next>
  __device__ __forceinline__ void transform(double (&v)[4][NG], Next next) const {
    cp_async_wait_0();
    __syncthreads();
    double acc_e[NG][2], acc_o[NG][2];
#pragma unroll
    for (int f = 0; f < NG; ++f) acc_e[f][0] = acc_e[f][1] = acc_o[f][0] = acc_o[f][1] = 0.0;
    const bool first = tau < kNT / 2;
    const int ke = 4 * KSE * half + (first ? 0 : KSE), ko = 4 * KSE * half + 2 * KSE;  // first k-steps: even part, odd class
    const double *xl = xs + a_frag_slot(lane & 3, lane >> 2);
    const double *be = syn + ((size_t)ke * kNT + (first ? tau : kNT - 1 - tau)) * 32 + lane;
    const double *bo = syn + ((size_t)ko * kNT + tau) * 32 + lane;
    double bn = __ldg(bo);
#pragma unroll
    for (int s = 0; s < 2 * KSE; ++s) {
      const double bv = bn;
      if (s + 1 < 2 * KSE) bn = __ldg(bo + (size_t)(s + 1) * kNT * 32);
#pragma unroll
      for (int f = 0; f < NG; ++f) dmma(acc_o[f], xl[f * kTile + (ko + s) * 32], bv);
      if (s < KSE) {
        const double b2 = __ldg(be + (size_t)s * kNT * 32);
#pragma unroll
        for (int f = 0; f < NG; ++f) dmma(acc_e[f], xl[f * kTile + (ke + s) * 32], b2);
      }
    }
    __syncthreads();
    next();
    fold_exchange<kNT, NG>(acc_e, acc_o, xc, tau, half, CtaSync{}, v);
  }
  // Analyses NO products gq[quadrant][o] of the lane's angle into out + o * stride (a tile block of 128 rows x 8
  // points each): a warp takes one output tile of an odd class and one of an even group.
  template <int NO>
  __device__ __forceinline__ void analyse(const double (&gq)[4][NO], double *out, int64_t stride) const {
    __syncthreads();  // the previous analysis has read ps
    prefold_store<kNT, NO>(gq, ps, 0, tau, half);
    __syncthreads();
    const int q = lane & 3, g = lane >> 2;
#pragma unroll
    for (int odd = 1; odd >= 0; --odd) {
      // groups: CO, SO (NUO output tiles of 8 modes each) or CE0, CE2, SE0, SE2 (NUE each)
      constexpr int NUE = MH / 32, NUO = MH / 16;
      const int ev = warp / NUE;
      const int gr = odd ? (warp < NUO ? 2 : 5) : ev + (ev >= 2 ? 1 : 0), u = odd ? warp % NUO : warp % NUE;
      const int c = odd ? (gr == 2 ? 1 : 3) : gr < 3 ? 0 : 2, TE = odd ? 2 * kNT : kNT;
      constexpr int AE = NUE * kNT, AO = 2 * NUO * kNT;  // analysis k-steps of an even group, of an odd class
      const int aof = gr == 0 ? 0 : gr == 1 ? AE : gr == 2 ? 2 * AE : gr == 3 ? 2 * AE + AO : gr == 4 ? 3 * AE + AO : 4 * AE + AO;
      const double sg = gr == 0 || gr == 4 ? 1.0 : -1.0;  // mirror sign: PE0 +, PE2 -, QE0 -, QE2 +
      const double *bt = ana + (size_t)(aof + u * TE) * 32 + lane;
      const double *pa = ps + (size_t)c * kNT * 64;
      double y[2][NO][2];
#pragma unroll
      for (int o = 0; o < NO; ++o) y[0][o][0] = y[0][o][1] = y[1][o][0] = y[1][o][1] = 0.0;
#pragma unroll
      for (int te = 0; te < (odd ? 2 * kNT : kNT); ++te) {
        const double bv = __ldg(bt + te * 32);
        const int t = te >> 1, e = te & 1;
#pragma unroll
        for (int o = 0; o < NO; ++o) {
          const double *po = pa + (size_t)o * 4 * kNT * 64;
          double av = po[(t * 2 + e) * 32 + lane];
          if (!odd) av += sg * po[((kNT - 1 - t) * 2 + 1 - e) * 32 + (lane ^ 3)];
          dmma(y[te & 1][o], av, bv);
        }
      }
      const int row0 = (gr % 3 == 0 ? 0 : gr % 3 == 1 ? MH / 4 : MH / 2) + (gr >= 3 ? MH : 0) + 8 * u + 2 * q;
#pragma unroll
      for (int o = 0; o < NO; ++o)
#pragma unroll
        for (int h = 0; h < 2; ++h) out[o * stride + (row0 + h) * 8 + g] = y[0][o][h] + y[1][o][h];
    }
  }
};

template <int M>
__device__ __forceinline__ Tile<M> make_tile(double *smem, const double *syn, const double *ana) {
  const int warp = threadIdx.x >> 5;
  double *xc = smem + 3 * Res<M>::TILE;
  return {smem, xc, xc + Res<M>::XC, syn, ana, (int)threadIdx.x & 31, warp, warp >> 1, warp & 1};
}

// Grid values of three shared fields (blockIdx.z) of a tile (blockIdx.x) on residue blockIdx.y.
template <int M>
__global__ void __launch_bounds__(Res<M>::THREADS, Res<M>::BLOCKS) base_kernel(const ProdArgs a) {
  constexpr int kTile = Res<M>::TILE, kNT = Res<M>::NT;
  extern __shared__ __align__(16) double smem[];
  const Tile<M> t = make_tile<M>(smem, a.syn, a.ana);
  const int f0 = 3 * blockIdx.z;
  const double *src[3];
#pragma unroll
  for (int f = 0; f < 3; ++f)
    src[f] = a.C + (((int64_t)blockIdx.y * a.ninst + a.inst[f0 + f]) * a.tiles + blockIdx.x) * kTile;
  t.stage(src);
  double v[4][3];
  t.transform(v, [] {});
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    double *g = a.G + ((((int64_t)blockIdx.y * a.nshared + f0 + f) * a.tiles + blockIdx.x) * kNT + t.tau) * 256 + t.half * 32 + t.lane;
#pragma unroll
    for (int r = 0; r < 4; ++r) g[r * 64] = v[r][f];
  }
}

// Program OP on one tile, batch entry and residue (blockIdx.x = tile * nb + entry, blockIdx.y = residue): the entry's
// fields are transformed three at a time, the first ones' quadrant values waiting in registers, and the outputs
// analysed three at a time.  The entries of a tile run next to each other, so that the base state's grid values come
// from L2 after the first.  At 80 registers 24 warps share an SM (three CTAs of 8 at M = 128, six of 4 at M = 64).
template <int OP, int M>
__global__ void __launch_bounds__(Res<M>::THREADS, Res<M>::BLOCKS) prod_kernel(const ProdArgs a) {
  constexpr int kTile = Res<M>::TILE, kNT = Res<M>::NT;
  extern __shared__ __align__(16) double smem[];
  const Tile<M> t = make_tile<M>(smem, a.syn, a.ana);
  const int64_t tile = blockIdx.x / a.nb;
  const int b = (int)(blockIdx.x - tile * a.nb), r = blockIdx.y;
  auto field = [&](int f) { return a.C + (((int64_t)r * a.ninst + a.inst[f] + b) * a.tiles + tile) * kTile; };
  constexpr int NO = op_nout(OP);
  double *S = a.S + (((int64_t)r * NO * a.nb + b) * a.tiles + tile) * kTile;  // output o: o * nb * tiles * kTile further
  const int64_t ost = (int64_t)a.nb * a.tiles * kTile;
  // shared field f at the lane's angle, quadrant rr
  auto base = [&](int f, int rr) {
    return __ldg(a.G + ((((int64_t)r * a.nshared + f) * a.tiles + tile) * kNT + t.tau) * 256 + rr * 64 + t.half * 32 + t.lane);
  };
  auto stage3 = [&](int f) {
    const double *src[3] = {field(f), field(f + 1), field(f + 2)};
    t.stage(src);
  };
  if constexpr (OP == OP_CROSS || OP == OP_DOT) {
    stage3(0);
    double u[4][3], v[4][3];
    t.transform(u, [&] { stage3(3); });
    t.transform(v, [] {});
    double gq[4][NO];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      if constexpr (OP == OP_CROSS)
        cross3(u[rr], v[rr], gq[rr]);
      else
        gq[rr][0] = u[rr][0] * v[rr][0] + u[rr][1] * v[rr][1] + u[rr][2] * v[rr][2];
    }
    t.analyse(gq, S, ost);
  } else if constexpr (OP == OP_SVECT) {
    stage3(0);
    double u[4][3], s[4][1];
    t.transform(u, [&] {
      const double *src[1] = {field(3)};
      t.stage(src);
    });
    t.transform(s, [] {});
    double gq[4][3];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
      for (int k = 0; k < 3; ++k) gq[rr][k] = s[rr][0] * u[rr][k];
    t.analyse(gq, S, ost);
  } else if constexpr (OP == OP_PROD) {
    const double *src[2] = {field(0), field(1)};
    t.stage(src);
    double v[4][2], gq[4][1];
    t.transform(v, [] {});
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) gq[rr][0] = v[rr][0] * v[rr][1];
    t.analyse(gq, S, ost);
  } else if constexpr (OP == OP_CROSS_JVP || OP == OP_MHD_JVP) {
    // [u, w(, b), du, dw(, db)]: du x w + u x dw (, du x b + u x db)
    constexpr int F0 = first_own(OP), NP = F0 / 3 - 1;
    stage3(F0);
    double du[4][3], d[4][3];
    t.transform(du, [&] { stage3(F0 + 3); });
#pragma unroll 1
    for (int k = 0; k < NP; ++k) {
      t.transform(d, [&] {
        if (k + 1 < NP) stage3(F0 + 6);
      });
      double gq[4][3];
#pragma unroll
      for (int rr = 0; rr < 4; ++rr) {
        double u[3], w[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          u[c] = base(c, rr);
          w[c] = base(3 * (k + 1) + c, rr);
        }
        cross3(du[rr], w, gq[rr]);
        cross3_acc(u, d[rr], gq[rr]);
      }
      t.analyse(gq, S + 3 * k * ost, ost);
    }
  } else {
    // [u, w(, b), c1(, c2)]: w x c1 (+ b x c2), c1 x u (, c2 x u)
    static_assert(OP == OP_CROSS_VJP || OP == OP_MHD_VJP, "program");
    constexpr int F0 = first_own(OP), NP = F0 / 3 - 1;
    stage3(F0);
    double sum[4][3];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) sum[rr][0] = sum[rr][1] = sum[rr][2] = 0.0;
#pragma unroll 1
    for (int k = 0; k < NP; ++k) {
      double c[4][3], gq[4][3];
      t.transform(c, [&] {
        if (k + 1 < NP) stage3(F0 + 3);
      });
#pragma unroll
      for (int rr = 0; rr < 4; ++rr) {
        double u[3], w[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          u[e] = base(e, rr);
          w[e] = base(3 * (k + 1) + e, rr);
        }
        cross3(c[rr], u, gq[rr]);
        cross3_acc(w, c[rr], sum[rr]);
      }
      t.analyse(gq, S + 3 * (k + 1) * ost, ost);
    }
    t.analyse(sum, S, ost);
  }
}

template <int OP, int M>
int launch_prod(const ProdArgs &pa, int R, cudaStream_t st) {
  static KernelSetup setup;
  if (int rc = setup.opt_in(reinterpret_cast<const void *>(prod_kernel<OP, M>), Res<M>::SMEM)) return rc;
  prod_kernel<OP, M><<<dim3((unsigned)(pa.tiles * pa.nb), (unsigned)R), Res<M>::THREADS, Res<M>::SMEM, st>>>(pa);
  return check_launch("residue grids: program");
}
template <int M>
int launch_base(const ProdArgs &pa, int R, cudaStream_t st) {
  static KernelSetup setup;
  if (int rc = setup.opt_in(reinterpret_cast<const void *>(base_kernel<M>), Res<M>::SMEM)) return rc;
  base_kernel<M><<<dim3((unsigned)pa.tiles, (unsigned)R, (unsigned)(pa.nshared / 3)), Res<M>::THREADS, Res<M>::SMEM, st>>>(pa);
  return check_launch("residue grids: base state");
}

template <int M, int R>
int launch_passes(const CoefArgs *ca, const OutArgs *oa, cudaStream_t st) {
  const int64_t nblk = ((ca ? ca->npts : oa->npts) + 127) / 128 * Res<M>::MH;
  if (ca)
    coef_kernel<M, R><<<(unsigned)(nblk * ca->inst[ca->nf]), 128, 0, st>>>(*ca);
  else
    out_kernel<M, R><<<(unsigned)(nblk * oa->no * oa->nb), 128, 0, st>>>(*oa);
  return check_launch("residue grids: coefficients and outputs");
}
template <int M>
int launch_passes(int R, const CoefArgs *ca, const OutArgs *oa, cudaStream_t st) {
  if constexpr (M == 64) switch (R) {  // 128 angles begin beyond 12 residues of 64
      case 4: return launch_passes<M, 4>(ca, oa, st);
      case 5: return launch_passes<M, 5>(ca, oa, st);
      case 6: return launch_passes<M, 6>(ca, oa, st);
    }
  switch (R) {
    case 7: return launch_passes<M, 7>(ca, oa, st);
    case 8: return launch_passes<M, 8>(ca, oa, st);
    case 9: return launch_passes<M, 9>(ca, oa, st);
    case 10: return launch_passes<M, 10>(ca, oa, st);
    case 11: return launch_passes<M, 11>(ca, oa, st);
    case 12: return launch_passes<M, 12>(ca, oa, st);
  }
  return set_error(SFNL_ERR_UNSUPPORTED, "residue grids: no such number of residues");
}

}  // namespace

// Residue grids of 64 angles while at most this many cover the grid (m <= 256), else of 128: the transforms of 64 angles
// have half the DMMAs per angle, and the passes' twiddles, twice as many, hide behind HBM.  Against 128 angles: cross
// product, 35,000 points, m = 128 0.558 -> 0.465 ms, m = 256 1.107 -> 1.012; MHD JVP, 7,000 points, 16 tangents, m = 128
// 3.47 -> 3.19 ms, m = 256 7.15 -> 7.07.
constexpr int kRes64Max = 12;

// From m = 65, where the fused kernels run on run-time loops: cross product, 30,000 points, m = 65 0.433 -> 0.274 ms, m =
// 100 0.769 -> 0.333; MHD VJP, 10,000 points, 4 cotangents, m = 65 1.91 -> 0.83 ms.  The cross product's JVP from m = 73:
// its two-pass fused program is the faster one before (m = 72 0.370 against 0.393 ms, m = 80 0.573 against 0.395).  Few
// points do not move the line, although three or four launches with small grids replace one (1,000 points, m = 65: cross
// product 18.7 against 18.7 us, dot product 16.6 against 17.4, MHD VJP 85.5 against 45.8; m = 85 cross product 22.8
// against 18.7), but by 1 us of 14 for the scalar product to m = 80.
bool res_supported(int op, int m) {
  if (m < (op == OP_CROSS_JVP ? 73 : 65) || m > 512) return false;
  return op == OP_CROSS || op == OP_DOT || op == OP_PROD || op == OP_SVECT || linear_op(op);
}

namespace {
constexpr size_t kResMinBytes = size_t(32) << 20;
// Points and batch entries go in chunks whose coefficients, base values and sums fit `cap` bytes of workspace.
template <int M>
int launch_res_m(const ProgArgs &a, size_t cap, cudaStream_t st) {
  constexpr int kTile = Res<M>::TILE;
  const int m = a.m, R = (3 * m - 2 + M - 1) / M, N = M * R;
  const int ni = op_nin(a.op), no = op_nout(a.op);
  const bool lin = linear_op(a.op);
  const int nsh = lin ? first_own(a.op) : 0, own = ni - nsh;
  ResTab T;
  if (int rc = get_residue_tables(m, N, R, &T)) return rc;
  // doubles per point: N for a field's coefficients, grid values or an output's sums
  const size_t shared_b = sizeof(double) * (size_t)N * 2 * nsh, entry_b = sizeof(double) * (size_t)N * (own + no);
  int64_t kb = 0, chunk = 0;
  size_t bytes = 0;
  auto plan = [&](size_t room) {
    kb = (int64_t)((room / 64 - shared_b) / entry_b);  // at least 64 points at a time where the room allows
    kb = room / 64 <= shared_b || kb < 1 ? 1 : kb > a.batch ? a.batch : kb;
    chunk = (int64_t)(room / (shared_b + kb * entry_b)) / 8 * 8;
    chunk = chunk < 8 ? 8 : chunk;
    const int64_t chunks = (a.np + chunk - 1) / chunk;  // of equal length
    chunk = ((a.np + chunks - 1) / chunks + 7) / 8 * 8;
    bytes = (size_t)chunk * (shared_b + kb * entry_b);
  };
  plan(cap);
  LargeWorkspace ws(st, 2);
  // Where the fused kernels fit, a call that needs more than the share of the free memory leaves it to them; beyond, the
  // points go in shorter chunks, down to kResMinBytes, while there is no memory for longer ones.
  const bool fused = fast_fused_fits(a.op, a.m);
  if (const size_t share = ws.share(bytes); share < bytes) {
    if (fused) return set_error(SFNL_ERR_ALLOC, "residue grids: little free memory");
    plan(share > kResMinBytes ? share : kResMinBytes);
  }
  double *W = nullptr;
  int rc = ws.get(bytes, &W);
  while (rc == SFNL_ERR_ALLOC && !fused && bytes > kResMinBytes) {
    plan(bytes / 2);
    rc = ws.get(bytes, &W);
  }
  if (rc) return rc;
  const bool adj_out = op_adjoint_out(a.op);
  for (int64_t c0 = 0; c0 < a.np; c0 += chunk)
    for (int b0 = 0; b0 < a.batch; b0 += (int)kb) {
      const int nb = a.batch - b0 < kb ? a.batch - b0 : (int)kb;
      CoefArgs ca{};
      ca.nf = ni;
      ca.m = m;
      ca.b0 = b0;
      ca.np = a.np;
      ca.npts = a.np - c0 < chunk ? a.np - c0 : chunk;
      ca.tiles = (ca.npts + 7) / 8;
      ca.tw = T.tw;
      ca.invN = 1.0 / N;
      for (int f = 0; f < ni; ++f) {
        ca.x[f] = a.in[f] + c0;
        ca.ldm[f] = a.in_ldm[f];
        ca.bs[f] = a.in_bs[f];
        ca.inst[f + 1] = ca.inst[f] + (f < nsh ? 1 : nb);
        if (op_adjoint_in(a.op, f)) ca.adj |= 1u << f;
      }
      const int64_t ninst = ca.inst[ni], tile_d = ca.tiles * kTile;
      ca.C = W;
      ProdArgs pa{};
      pa.C = W;
      pa.G = W + R * ninst * tile_d;
      pa.S = pa.G + (int64_t)R * nsh * tile_d;
      pa.syn = T.syn;
      pa.ana = T.ana;
      pa.tiles = ca.tiles;
      pa.ninst = ninst;
      for (int f = 0; f < ni; ++f) pa.inst[f] = ca.inst[f];
      pa.nshared = nsh;
      pa.nb = nb;
      if (rc = launch_passes<M>(R, &ca, nullptr, st)) return rc;
      if (lin)
        if (rc = launch_base<M>(pa, R, st)) return rc;
      switch (a.op) {
        case OP_CROSS: rc = launch_prod<OP_CROSS, M>(pa, R, st); break;
        case OP_DOT: rc = launch_prod<OP_DOT, M>(pa, R, st); break;
        case OP_PROD: rc = launch_prod<OP_PROD, M>(pa, R, st); break;
        case OP_SVECT: rc = launch_prod<OP_SVECT, M>(pa, R, st); break;
        case OP_CROSS_JVP: rc = launch_prod<OP_CROSS_JVP, M>(pa, R, st); break;
        case OP_CROSS_VJP: rc = launch_prod<OP_CROSS_VJP, M>(pa, R, st); break;
        case OP_MHD_JVP: rc = launch_prod<OP_MHD_JVP, M>(pa, R, st); break;
        case OP_MHD_VJP: rc = launch_prod<OP_MHD_VJP, M>(pa, R, st); break;
        default: rc = set_error(SFNL_ERR_ARG, "residue grids: unknown program");
      }
      if (rc) return rc;
      OutArgs oa{};
      oa.S = pa.S;
      oa.nb = nb;
      oa.no = no;
      oa.m = m;
      oa.b0 = b0;
      oa.npts = ca.npts;
      oa.tiles = ca.tiles;
      oa.osin = a.np * a.out_ps;
      oa.ops = a.out_ps;
      oa.w = adj_out ? 1.0 : 2.0 / N;
      oa.w0 = adj_out ? 1.0 : 1.0 / N;
      oa.tw = T.tw;
      for (int o = 0; o < no; ++o) {
        oa.out[o] = a.out[o] + c0 * a.out_ps;
        oa.ldm[o] = a.out_ldm[o];
        oa.bs[o] = a.out_bs[o];
      }
      if (rc = launch_passes<M>(R, nullptr, &oa, st)) return rc;
    }
  return SFNL_OK;
}
}  // namespace

int launch_res(const ProgArgs &a, size_t cap, cudaStream_t st) {
  if (3 * a.m - 2 <= 64 * kRes64Max) return launch_res_m<64>(a, cap, st);
  return launch_res_m<128>(a, cap, st);
}

}  // namespace sfnl
