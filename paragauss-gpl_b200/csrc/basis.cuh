// basis.cuh -- contracted real-solid-harmonic Gaussians and gradients on points.
//
// Restates, per point and per (atom, l) shell:
//   solid_harmonics_calculate  modules/solid_harmonics_module.f90:369-482
//     (Racah-normalised recursion, Y_00 = 1, Y_1 = (z, x, y)); the gradients
//     of :488-568 are obtained by differentiating the same recursion;
//   radial                     modules/orbital_module.f90:1742-1932
//     (norm*exp(-a r^2) only where a r^2 < 50, derivative factor -2a, the
//     first N_uncontracted primitives bare, then the contractions);
//   calculate_orbs_and_grads_v3 modules/orbital_module.f90:2421-2619
//     (phi = Y R, grad phi = (r - R_A) Y R' + grad(Y) R; function order
//     independent function -> radial function).
// All arithmetic is FP64 in both precision modes.
#pragma once

#include <type_traits>

#include "pgxc_common.cuh"

namespace pgxc {

// Y[l*l + m] and dY[c][l*l + m], c = x, y, z, for l <= L, in real type R.
template <int L, typename R>
__device__ __forceinline__ void solid_harmonics(R x, R y, R z, R* Y, R (*dY)[16]) {
  const R r2 = x * x + y * y + z * z;
  Y[0] = R(1);
  dY[0][0] = dY[1][0] = dY[2][0] = R(0);
  if (L == 0) return;
  Y[1] = z; Y[2] = x; Y[3] = y;
  dY[0][1] = 0; dY[1][1] = 0; dY[2][1] = 1;
  dY[0][2] = 1; dY[1][2] = 0; dY[2][2] = 0;
  dY[0][3] = 0; dY[1][3] = 1; dY[2][3] = 0;
#pragma unroll
  for (int l = 2; l <= L; ++l) {
    const int o = l * l, o1 = (l - 1) * (l - 1), o2 = (l - 2) * (l - 2);
    const R lr = R(l), l1r = R(l - 1), ll1r = R(2 * l - 1);
    const R dr2[3] = {R(2) * x, R(2) * y, R(2) * z};
    // m index 0
    {
      const R p1 = Y[o1], p2 = Y[o2];
      Y[o] = (ll1r * z * p1 - l1r * r2 * p2) / lr;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        dY[c][o] = (ll1r * ((c == 2 ? p1 : R(0)) + z * dY[c][o1]) - l1r * (dr2[c] * p2 + r2 * dY[c][o2])) / lr;
    }
#pragma unroll
    for (int im = 1; im <= l - 2; ++im) {
      const R sim = (R)(im * im);
      const R rlm = R(1) / sqrt(lr * lr - sim);
      const R rl1m = sqrt(l1r * l1r - sim);
      const R a = ll1r * z * rlm;
      const R b = rl1m * r2 * rlm;
#pragma unroll
      for (int mm = 2 * im - 1; mm <= 2 * im; ++mm) {
        const R p1 = Y[o1 + mm], p2 = Y[o2 + mm];
        Y[o + mm] = a * p1 - b * p2;
#pragma unroll
        for (int c = 0; c < 3; ++c)
          dY[c][o + mm] = (c == 2 ? ll1r * rlm * p1 : R(0)) + a * dY[c][o1 + mm] - rl1m * dr2[c] * rlm * p2 -
                          b * dY[c][o2 + mm];
      }
    }
    {
      const int im = l - 1;
      const R rlm = R(1) / sqrt(lr * lr - (R)(im * im));
      const R a = ll1r * z * rlm;
#pragma unroll
      for (int mm = 2 * im - 1; mm <= 2 * im; ++mm) {
        const R p1 = Y[o1 + mm];
        Y[o + mm] = a * p1;
#pragma unroll
        for (int c = 0; c < 3; ++c) dY[c][o + mm] = (c == 2 ? ll1r * rlm * p1 : R(0)) + a * dY[c][o1 + mm];
      }
    }
    {
      const R rll = sqrt(ll1r / (R(2) * lr));
      const R q2 = Y[o1 + 2 * l - 3], q1 = Y[o1 + 2 * l - 2];
      Y[o + 2 * l - 1] = (x * q2 - y * q1) * rll;
      Y[o + 2 * l] = (y * q2 + x * q1) * rll;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const R g2 = dY[c][o1 + 2 * l - 3], g1 = dY[c][o1 + 2 * l - 2];
        const R dx = R(c == 0), dy = R(c == 1);
        dY[c][o + 2 * l - 1] = (dx * q2 + x * g2 - dy * q1 - y * g1) * rll;
        dY[c][o + 2 * l] = (dy * q2 + y * g2 + dx * q1 + x * g1) * rll;
      }
    }
  }
}

// One normalised primitive norm*exp(-alpha r^2), zero where alpha r^2 >= 50
// (radial0/radial1, modules/orbital_module.f90:1823-1854).
__device__ __forceinline__ double prim_value(double alpha, double norm, double r2) {
  const double ar2 = alpha * r2;
  return ar2 < 50.0 ? norm * exp(-ar2) : 0.0;
}

// Evaluate the selected radial functions of one shell at one point.  The
// selected radial indices are the set bits of `mask` (nsel of them, in
// increasing order); selected function k of independent function i is stored
// at row base + i*nsel + k, column p of the [row][ld] arrays.  The dense
// layout is mask = all nrad bits, base = S.f0 (row = function index); the
// screened layout is the tile's significant radial functions and their slot.
// exps/norms/contr/rng may point to shared memory (plain loads); rng is the
// shell's [lo, hi) primitive range per contraction (used when S.seg).
template <int L, bool GRAD>
__device__ __forceinline__ void shell_at_point(const DevShell& S, const DevSA& sa, double x, double y, double z,
                                               const double* exps, const double* norms, const double* contr,
                                               const int2* rng, bool valid, uint64_t mask, int64_t base, int nsel,
                                               int64_t p,
                                               int64_t ld, double* __restrict__ phi, double* __restrict__ gx,
                                               double* __restrict__ gy, double* __restrict__ gz, double& vmax) {
  double Y[16];
  double dY[3][16];
  solid_harmonics<L, double>(x, y, z, Y, dY);
  const double r2 = x * x + y * y + z * z;
  // symmetry-adapted harmonics of this l
  double Ys[2 * L + 1], dYs[3][2 * L + 1];
#pragma unroll
  for (int i = 0; i < 2 * L + 1; ++i) {
    if (sa.identity) {
      Ys[i] = Y[L * L + i];
#pragma unroll
      for (int c = 0; c < 3; ++c) dYs[c][i] = dY[c][L * L + i];
    } else {
      double v = 0, g0 = 0, g1 = 0, g2 = 0;
#pragma unroll
      for (int m = 0; m < 2 * L + 1; ++m) {
        const double cf = sa.c[L][i][m];
        v += cf * Y[L * L + m];
        g0 += cf * dY[0][L * L + m];
        g1 += cf * dY[1][L * L + m];
        g2 += cf * dY[2][L * L + m];
      }
      Ys[i] = v; dYs[0][i] = g0; dYs[1][i] = g1; dYs[2][i] = g2;
    }
  }
  const double* ex = exps + S.exp_off;
  const double* nr = norms + S.exp_off;
  const double* cc = contr + S.con_off;
  if (S.seg) {
    // segmented contractions: each selected radial function sums only its own primitives
    uint64_t rem = mask;
    for (int k = 0; k < nsel; ++k) {
      const int rr = __ffsll((long long)rem) - 1;
      rem &= rem - 1;
      const int2 rg = rng[rr];
      double Rr = 0.0, dR = 0.0;
      if (valid) {
        for (int e = rg.x; e < rg.y; ++e) {
          const double alpha = ex[e];
          const double v = prim_value(alpha, nr[e], r2);
          const double cf = cc[e + (int64_t)S.nexp * rr];
          Rr += cf * v;
          dR += cf * ((-2.0 * alpha) * v);
        }
      }
#pragma unroll
      for (int i = 0; i < 2 * L + 1; ++i) {
        const int64_t f = base + (int64_t)i * nsel + k;
        phi[f * ld + p] = Ys[i] * Rr;
        vmax = fmax(vmax, fabs(Ys[i] * Rr));
        if (GRAD) {
          const double h = Ys[i] * dR;
          gx[f * ld + p] = x * h + dYs[0][i] * Rr;
          gy[f * ld + p] = y * h + dYs[1][i] * Rr;
          gz[f * ld + p] = z * h + dYs[2][i] * Rr;
        }
      }
    }
    return;
  }
  uint64_t rem = mask;
  for (int k0 = 0; k0 < nsel; k0 += kRadGroup) {
    int rr[kRadGroup];
#pragma unroll
    for (int r = 0; r < kRadGroup; ++r) {
      if (k0 + r < nsel) {
        rr[r] = __ffsll((long long)rem) - 1;
        rem &= rem - 1;
      } else {
        rr[r] = -1;
      }
    }
    double Rr[kRadGroup], dR[kRadGroup];
#pragma unroll
    for (int r = 0; r < kRadGroup; ++r) { Rr[r] = 0.0; dR[r] = 0.0; }
    if (valid) {
      for (int e = 0; e < S.nexp; ++e) {
        const double alpha = ex[e];
        const double v = prim_value(alpha, nr[e], r2);
        const double dv = (-2.0 * alpha) * v;
#pragma unroll
        for (int r = 0; r < kRadGroup; ++r) {
          if (rr[r] >= 0) {
            double cf;
            if (rr[r] < S.nunc) cf = (e == rr[r]) ? 1.0 : 0.0;
            else cf = cc[e + (int64_t)S.nexp * (rr[r] - S.nunc)];
            Rr[r] += cf * v;
            dR[r] += cf * dv;
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * L + 1; ++i) {
#pragma unroll
      for (int r = 0; r < kRadGroup; ++r) {
        if (rr[r] >= 0) {
          const int64_t f = base + (int64_t)i * nsel + k0 + r;
          phi[f * ld + p] = Ys[i] * Rr[r];
          vmax = fmax(vmax, fabs(Ys[i] * Rr[r]));
          if (GRAD) {
            const double h = Ys[i] * dR[r];
            gx[f * ld + p] = x * h + dYs[0][i] * Rr[r];
            gy[f * ld + p] = y * h + dYs[1][i] * Rr[r];
            gz[f * ld + p] = z * h + dYs[2][i] * Rr[r];
          }
        }
      }
    }
  }
}

// Stage one shell's exponents, norms and contraction matrix in shared memory
// (when they fit); returns the pointers to use.
constexpr int kStagePrim = 64;
constexpr int kStageCon = 512;
struct ShellStage {
  double e[kStagePrim], n[kStagePrim], c[kStageCon];
  int2 r[64];
};
// Stages the shell (when it fits) and its contraction ranges; returns the
// range pointer to use (shared memory).
__device__ __forceinline__ bool stage_shell(ShellStage& st, DevShell& S, const double* exps, const double* norms,
                                            const double* contr, const int2* rng) {
  const bool staged = S.nexp <= kStagePrim && S.nexp * S.ncontr <= kStageCon;
  if (staged) {
    const double *e_src = exps + S.exp_off, *n_src = norms + S.exp_off, *c_src = contr + S.con_off;
    for (int i = threadIdx.x; i < S.nexp; i += blockDim.x) {
      st.e[i] = e_src[i];
      st.n[i] = n_src[i];
    }
    for (int i = threadIdx.x; i < S.nexp * S.ncontr; i += blockDim.x) st.c[i] = c_src[i];
    S.exp_off = 0;
    S.con_off = 0;
  }
  if (S.seg)
    for (int i = threadIdx.x; i < S.nrad; i += blockDim.x) st.r[i] = rng[S.rad_off + i];
  __syncthreads();
  return staged;
}

__host__ __device__ constexpr uint64_t all_radial(int nrad) { return nrad >= 64 ? ~0ull : ((1ull << nrad) - 1); }

// ---------------------------------------------------------------------------
// K1 (dense): basis functions of the shells of one angular momentum L on a
// chunk of points.  grid = (chunk/128, shells of this L), block = 128 points.
// ---------------------------------------------------------------------------
template <int L, bool GRAD>
__global__ void __launch_bounds__(128) k_basis_l(const DevShell* __restrict__ shells, const int* __restrict__ ids,
                                                 const double* __restrict__ atoms, const double* __restrict__ exps,
                                                 const double* __restrict__ norms, const double* __restrict__ contr,
                                                 const int2* __restrict__ rng, DevSA sa, const double* __restrict__ px,
                                                 const double* __restrict__ py,
                                                 const double* __restrict__ pz, int64_t p0, int64_t nvalid, int64_t ld,
                                                 double* __restrict__ phi, double* __restrict__ gx,
                                                 double* __restrict__ gy, double* __restrict__ gz) {
  __shared__ ShellStage st;
  DevShell S = shells[ids[blockIdx.y]];
  const bool staged = stage_shell(st, S, exps, norms, contr, rng);
  const int64_t p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (p >= ld) return;
  const bool valid = p < nvalid;
  double x = 0, y = 0, z = 0;
  if (valid) {
    x = px[p0 + p] - atoms[3 * S.atom];
    y = py[p0 + p] - atoms[3 * S.atom + 1];
    z = pz[p0 + p] - atoms[3 * S.atom + 2];
  }
  double vmax = 0.0;
  shell_at_point<L, GRAD>(S, sa, x, y, z, staged ? st.e : exps, staged ? st.n : norms, staged ? st.c : contr, st.r,
                          valid, all_radial(S.nrad), S.f0, S.nrad, p, ld, phi, gx, gy, gz, vmax);
}

// ---------------------------------------------------------------------------
// K1 (screened): a work item is the significant radial functions of one shell
// on the 128 points of one tile.  Rows are slots of the chunk's compact
// [slot][128] arrays (slot - s0); with pmax, the largest |phi| of each point
// of the chunk (tile - t0) is max-reduced into it.
//
// An item carries every field its evaluation needs (atom position, primitive
// and contraction offsets), so that the loads of the next item do not depend
// on one another.  A block walks contiguous ranges of items (records as whole
// 16-byte words, the same for every lane); consecutive items of a tile reuse the
// point coordinates.
// ---------------------------------------------------------------------------
struct alignas(16) BasisItem {
  double ax, ay, az;        // words 0-5: atom position
  int64_t slot;             // 6-7: global slot of the shell's first significant function
  unsigned long long mask;  // 8-9: significant radial functions of the shell
  int tile;                 // 10: global tile index
  int nsig;                 // 11: popcount(mask)
  int exp_off;              // 12: into exponents / norms
  int con_off;              // 13: into contractions (nexp x ncontr column-major)
  int rad_off;              // 14: into the radial-range table (seg shells)
  int nexp;                 // 15
  int nunc;                 // 16
  int seg;                  // 17
  int pad_[2];
};
static_assert(sizeof(BasisItem) == 80 && alignof(BasisItem) == 16, "a record is copied as five 16-byte words");

// GT: the element type of the gradient planes (double; float in the INT8
// build, whose potential and density gradient tolerate 24-bit gradients).
// Blocks per SM that the registers are bounded for.
template <int L, bool GRAD>
constexpr int basis_blocks() {
  return GRAD ? (L == 0 ? 5 : L == 1 ? 4 : 4) : (L <= 1 ? 5 : 7);
}
// The tables and point arrays of a launch.
template <typename GT>
struct BasisIO {
  const double* exps;
  const double* norms;
  const double* contr;
  const int2* rng;
  const double2* prim;  // {exponent, norm x coefficient} of the primitives of segmented shells
  const double *qx, *qy, *qz;
  int64_t s0, t0;
  double* phi;
  GT *gx, *gy, *gz;
  unsigned long long* pmax;
};

// Points per thread: two consecutive ones for s and p functions (16-byte stores,
// and what an item and a primitive cost besides arithmetic is paid once for two
// points, whose chains run side by side), one for d and f functions, whose values
// would take 230 registers and more (60 atoms: basis phase 2.31 ms, 2.35 with two
// points for d too).
template <int L>
constexpr int kBasisPts = L <= 1 ? 2 : 1;

template <int N, typename T>
__device__ __forceinline__ void put_points(T* p, const double (&v)[N]) {
  if constexpr (N == 1) *p = (T)v[0];
  else if constexpr (sizeof(T) == 8) *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  else *reinterpret_cast<float2*>(p) = make_float2((float)v[0], (float)v[1]);
}
template <int N>
__device__ __forceinline__ void get_points(const double* p, double (&v)[N]) {
  if constexpr (N == 1) {
    v[0] = __ldg(p);
  } else {
    const double2 d = __ldg(reinterpret_cast<const double2*>(p));
    v[0] = d.x;
    v[1] = d.y;
  }
}

// Items [i0, i1) by 128 / kBasisPts threads (whole warps; p0: the thread's
// first point).  Bound by instruction issue (2.9 of 4 per cycle with one point
// per thread, lane-broadcast records and every primitive of a shell looked at
// for every function): so of a segmented shell only the primitives that reach
// some point of the warp are visited, a bit mask made once per item from the
// warp's smallest r^2; their exponent and coefficient (the norm folded in) come
// as one 16-byte load; and the largest |phi| takes one step per radial function
// (max_k fl(|Y_k| |R|) = fl(max_k |Y_k| |R|)).
// 60 atoms, threshold 0 (2.77 million listed functions x 128 points, 11.4 GB
// written): 3.20 -> 2.93 ms with these, 2.31 with two points per thread.
template <int L, bool GRAD, typename GT>
__device__ __forceinline__ void basis_items(const BasisItem* __restrict__ items, int64_t i0, int64_t i1, int p0,
                                            const BasisIO<GT>& io, const DevSA& sa) {
  if (i0 >= i1) return;
  constexpr int N = kBasisPts<L>, M = 2 * L + 1;
  const int lane = threadIdx.x & 31;
  double px[N], py[N], pz[N], tmax[N] = {};
  auto points = [&](int tile) {
    const int64_t q = (int64_t)tile * 128 + p0;
    get_points(io.qx + q, px);
    get_points(io.qy + q, py);
    get_points(io.qz + q, pz);
  };
  points(__ldg(&items[i0].tile));
  for (int64_t i = i0; i < i1; ++i) {
    const BasisItem it = items[i];
    // the next item's tile: also what brings its record into L1 a whole item ahead
    const int ntile = __ldg(&items[min(i + 1, i1 - 1)].tile);
    const int nsel = it.nsig, nexp = it.nexp;
    double x[N], y[N], z[N], r2[N], Ys[N][M], dYs[N][3][M], ymax[N], vmax[N] = {};
    float rmin = __int_as_float(0x7f800000);
#pragma unroll
    for (int u = 0; u < N; ++u) {
      x[u] = px[u] - it.ax;
      y[u] = py[u] - it.ay;
      z[u] = pz[u] - it.az;
      r2[u] = x[u] * x[u] + y[u] * y[u] + z[u] * z[u];
      rmin = fminf(rmin, __double2float_rd(r2[u]));
      double Y[16];
      double dY[3][16];
      solid_harmonics<L, double>(x[u], y[u], z[u], Y, dY);
      ymax[u] = 0.0;
#pragma unroll
      for (int k = 0; k < M; ++k) {
        if (sa.identity) {
          Ys[u][k] = Y[L * L + k];
#pragma unroll
          for (int c = 0; c < 3; ++c) dYs[u][c][k] = dY[c][L * L + k];
        } else {
          double v = 0, g0 = 0, g1 = 0, g2 = 0;
#pragma unroll
          for (int m = 0; m < M; ++m) {
            const double cf = sa.c[L][k][m];
            v += cf * Y[L * L + m];
            g0 += cf * dY[0][L * L + m];
            g1 += cf * dY[1][L * L + m];
            g2 += cf * dY[2][L * L + m];
          }
          Ys[u][k] = v; dYs[u][0][k] = g0; dYs[u][1][k] = g1; dYs[u][2][k] = g2;
        }
        ymax[u] = fmax(ymax[u], fabs(Ys[u][k]));
      }
    }
    // the primitives (of the first 32) with alpha r^2 < 50 somewhere in the warp
    unsigned live = 0;
    if (it.seg && nexp <= 32) {
      rmin = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(rmin)));
      const bool on = lane < nexp && __ldg(io.exps + it.exp_off + min(lane, nexp - 1)) * (double)rmin < 50.0;
      live = __ballot_sync(0xffffffffu, on);
    }
    const int64_t row0 = (it.slot - io.s0) * 128 + p0;
    // radial function k of the item: its 2 L + 1 functions
    auto store = [&](int k, const double (&R)[N], const double (&dR)[N]) {
#pragma unroll
      for (int u = 0; u < N; ++u) vmax[u] = fmax(vmax[u], fabs(R[u]));
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int64_t o = row0 + (m * nsel + k) * 128;
        double v[N];
#pragma unroll
        for (int u = 0; u < N; ++u) v[u] = Ys[u][m] * R[u];
        put_points(io.phi + o, v);
        if (GRAD) {
          double g[3][N];
#pragma unroll
          for (int u = 0; u < N; ++u) {
            const double h = Ys[u][m] * dR[u];
            g[0][u] = x[u] * h + dYs[u][0][m] * R[u];
            g[1][u] = y[u] * h + dYs[u][1][m] * R[u];
            g[2][u] = z[u] * h + dYs[u][2][m] * R[u];
          }
          put_points(io.gx + o, g[0]);
          put_points(io.gy + o, g[1]);
          put_points(io.gz + o, g[2]);
        }
      }
    };
    uint64_t rem = it.mask;
    if (it.seg) {
      // segmented contractions: each selected radial function sums only its own primitives
      const double2* pr = io.prim + it.exp_off;
      for (int k = 0; k < nsel; ++k) {
        const int rr = __ffsll((long long)rem) - 1;
        rem &= rem - 1;
        const int2 rg = __ldg(io.rng + it.rad_off + rr);
        double R[N] = {}, dR[N] = {};
        auto add = [&](int e) {
          const double2 p = __ldg(pr + e);
#pragma unroll
          for (int u = 0; u < N; ++u) {
            const double ar2 = p.x * r2[u];
            const double v = ar2 < 50.0 ? p.y * exp(-ar2) : 0.0;
            R[u] += v;
            dR[u] += (-2.0 * p.x) * v;
          }
        };
        if (nexp <= 32) {
          unsigned m = rg.y > rg.x ? live & (0xffffffffu >> (32 - (rg.y - rg.x))) << rg.x : 0u;
          for (; m; m &= m - 1) add(__ffs((int)m) - 1);
        } else {
          for (int e = rg.x; e < rg.y; ++e) add(e);
        }
        store(k, R, dR);
      }
    } else {
      // general contractions: each radial function over all primitives (bare ones: its own)
      for (int k = 0; k < nsel; ++k) {
        const int rr = __ffsll((long long)rem) - 1;
        rem &= rem - 1;
        const bool bare = rr < it.nunc;
        const double* cc = io.contr + it.con_off + (int64_t)nexp * (rr - it.nunc);
        double R[N] = {}, dR[N] = {};
        for (int e = bare ? rr : 0; e < (bare ? rr + 1 : nexp); ++e) {
          const double alpha = __ldg(io.exps + it.exp_off + e), nrm = __ldg(io.norms + it.exp_off + e);
          const double cf = bare ? 1.0 : __ldg(cc + e);
#pragma unroll
          for (int u = 0; u < N; ++u) {
            const double v = prim_value(alpha, nrm, r2[u]);
            R[u] += cf * v;
            dR[u] += cf * ((-2.0 * alpha) * v);
          }
        }
        store(k, R, dR);
      }
    }
    // largest |phi| of each point over the tile's functions, max-reduced once per run of
    // items of one tile (non-negative doubles order like their bits)
#pragma unroll
    for (int u = 0; u < N; ++u) tmax[u] = fmax(tmax[u], ymax[u] * vmax[u]);
    if (io.pmax && (ntile != it.tile || i + 1 == i1)) {
#pragma unroll
      for (int u = 0; u < N; ++u) {
        atomicMax(io.pmax + ((int64_t)it.tile - io.t0) * 128 + p0 + u,
                  (unsigned long long)__double_as_longlong(tmax[u]));
        tmax[u] = 0.0;
      }
    }
    if (ntile != it.tile) points(ntile);
  }
}

// One block of 128 threads: kBasisPts<L> item ranges side by side (range `v` of
// `ranges`, `per` items each).
template <int L, bool GRAD, typename GT>
__device__ __forceinline__ void basis_block(const BasisItem* __restrict__ items, int64_t nitems, int64_t per,
                                            unsigned block, const BasisIO<GT>& io, const DevSA& sa) {
  constexpr int N = kBasisPts<L>, T = 128 / N;  // threads of an item
  const int64_t i0 = ((int64_t)block * N + threadIdx.x / T) * per;
  basis_items<L, GRAD, GT>(items, i0, min(nitems, i0 + per), (int)(threadIdx.x % T) * N, io, sa);
}

template <int L, bool GRAD, typename GT>
__global__ void __launch_bounds__(128, (basis_blocks<L, GRAD>()))
    k_basis_items(const BasisItem* __restrict__ items, int64_t nitems, BasisIO<GT> io, DevSA sa) {
  constexpr int N = kBasisPts<L>;
  const int64_t ranges = (int64_t)gridDim.x * N;
  basis_block<L, GRAD, GT>(items, nitems, (nitems + ranges - 1) / ranges, blockIdx.x, io, sa);
}

// The same for every l in one launch, one item per range: grids of few tiles,
// where each launch is one short wave and the launches one after another are
// what takes the time.  n.v[l] blocks for the n.n[l] items of each l.
struct BasisCounts {
  const BasisItem* items[kMaxL + 1];
  unsigned n[kMaxL + 1], v[kMaxL + 1];
};
template <bool GRAD, typename GT>
__global__ void __launch_bounds__(128, 3) k_basis_small(BasisCounts n, BasisIO<GT> io, DevSA sa) {
  unsigned b = blockIdx.x;
  if (b < n.v[0]) return basis_block<0, GRAD, GT>(n.items[0], n.n[0], 1, b, io, sa);
  b -= n.v[0];
  if (b < n.v[1]) return basis_block<1, GRAD, GT>(n.items[1], n.n[1], 1, b, io, sa);
  b -= n.v[1];
  if (b < n.v[2]) return basis_block<2, GRAD, GT>(n.items[2], n.n[2], 1, b, io, sa);
  b -= n.v[2];
  basis_block<3, GRAD, GT>(n.items[3], n.n[3], 1, b, io, sa);
}

// Basis values of a chunk: items[l][0 .. n[l]).  One launch per l, blocks that
// each walk a range of items, or a single one while all items together are no
// more than the blocks of one such launch.  Returns launches.
template <bool GRAD, typename GT>
int launch_basis_items(const BasisItem* const (&items)[kMaxL + 1], const int64_t (&n)[kMaxL + 1], int nsm,
                       int blocks_per_sm, const BasisIO<GT>& io, const DevSA& sa, cudaStream_t st) {
  const int64_t most = (int64_t)nsm * blocks_per_sm, all = n[0] + n[1] + n[2] + n[3];
  if (all == 0) return 0;
  if (all <= most) {
    BasisCounts c;
    constexpr int pts[kMaxL + 1] = {kBasisPts<0>, kBasisPts<1>, kBasisPts<2>, kBasisPts<3>};
    unsigned blocks = 0;
    for (int l = 0; l <= kMaxL; ++l) {
      c.items[l] = items[l];
      c.n[l] = (unsigned)n[l];
      blocks += c.v[l] = (unsigned)((n[l] + pts[l] - 1) / pts[l]);
    }
    k_basis_small<GRAD, GT><<<blocks, 128, 0, st>>>(c, io, sa);
    return 1;
  }
  int launches = 0;
  auto one = [&](auto Lc) {
    constexpr int L = decltype(Lc)::value;
    if (n[L] == 0) return;
    const int64_t nb = (n[L] + kBasisPts<L> - 1) / kBasisPts<L>;
    k_basis_items<L, GRAD, GT><<<(unsigned)(nb < most ? nb : most), 128, 0, st>>>(items[L], n[L], io, sa);
    ++launches;
  };
  one(std::integral_constant<int, 0>());
  one(std::integral_constant<int, 1>());
  one(std::integral_constant<int, 2>());
  one(std::integral_constant<int, 3>());
  return launches;
}

}  // namespace pgxc
