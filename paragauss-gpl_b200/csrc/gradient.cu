// gradient.cu -- the post-SCF XC nuclear gradient (gradient.h).
//
// FP64 throughout, on the Morton-ordered 128-point tiles of a plan whose lists
// hold every function that is not identically zero on the tile (threshold 0,
// whatever the context's own screening): per chunk of tiles
//   k_hess_items   phi, grad phi and Hessians of the listed functions
//   grad_contract  X = phi P[S_t, S_t] with rho, grad rho (screened.cu, DMMA)
//   k_grad_coef    the functional and the coefficients of each point
//   k_grad_w       W = sum_j b_j d_j phi, then V = W P[S_t, S_t]
//   k_grad_orb     the orbital terms
// and over all tiles k_grad_weights, the Becke weight term (its points in the
// same order: a warp's points then share their live atoms).
#include <cmath>

#include "basis.cuh"
#include "dgemm.cuh"
#include "gradient.h"
#include "xc_functional.cuh"
#include "xc_mgga.cuh"
#include "screened_plan.h"

namespace pgxc {

namespace {

// Real solid harmonics, first and second derivatives, by the recursion of
// solid_harmonics (basis.cuh, modules/solid_harmonics_module.f90:369-482)
// differentiated twice.  H[k][.] holds xx, xy, xz, yy, yz, zz.
template <int L>
__device__ __forceinline__ void solid_harmonics_h(double x, double y, double z, double* Y, double (*dY)[16],
                                                  double (*H)[16]) {
  const double r2 = x * x + y * y + z * z;
  const double xv[3] = {x, y, z};
  constexpr int ci[6] = {0, 0, 0, 1, 1, 2}, di[6] = {0, 1, 2, 1, 2, 2};
  for (int i = 0; i < 16; ++i) {
    Y[i] = 0.0;
    for (int c = 0; c < 3; ++c) dY[c][i] = 0.0;
    for (int k = 0; k < 6; ++k) H[k][i] = 0.0;
  }
  Y[0] = 1.0;
  if (L == 0) return;
  Y[1] = z; Y[2] = x; Y[3] = y;
  dY[2][1] = 1.0; dY[0][2] = 1.0; dY[1][3] = 1.0;
#pragma unroll
  for (int l = 2; l <= L; ++l) {
    const int o = l * l, o1 = (l - 1) * (l - 1), o2 = (l - 2) * (l - 2);
    const double lr = l, l1r = l - 1, ll1r = 2 * l - 1;
    {
      const double p1 = Y[o1], p2 = Y[o2];
      Y[o] = (ll1r * z * p1 - l1r * r2 * p2) / lr;
      for (int c = 0; c < 3; ++c)
        dY[c][o] = (ll1r * ((c == 2 ? p1 : 0.0) + z * dY[c][o1]) - l1r * (2.0 * xv[c] * p2 + r2 * dY[c][o2])) / lr;
      for (int k = 0; k < 6; ++k) {
        const int c = ci[k], d = di[k];
        const double t1 = (c == 2 ? dY[d][o1] : 0.0) + (d == 2 ? dY[c][o1] : 0.0) + z * H[k][o1];
        const double t2 = (c == d ? 2.0 * p2 : 0.0) + 2.0 * xv[c] * dY[d][o2] + 2.0 * xv[d] * dY[c][o2] + r2 * H[k][o2];
        H[k][o] = (ll1r * t1 - l1r * t2) / lr;
      }
    }
    for (int im = 1; im <= l - 2; ++im) {
      const double sim = im * im;
      const double rlm = 1.0 / sqrt(lr * lr - sim);
      const double rl1m = sqrt(l1r * l1r - sim);
      const double a = ll1r * z * rlm;
      const double b = rl1m * r2 * rlm;
      for (int mm = 2 * im - 1; mm <= 2 * im; ++mm) {
        const double p1 = Y[o1 + mm], p2 = Y[o2 + mm];
        Y[o + mm] = a * p1 - b * p2;
        for (int c = 0; c < 3; ++c)
          dY[c][o + mm] = (c == 2 ? ll1r * rlm * p1 : 0.0) + a * dY[c][o1 + mm] - rl1m * 2.0 * xv[c] * rlm * p2 -
                          b * dY[c][o2 + mm];
        for (int k = 0; k < 6; ++k) {
          const int c = ci[k], d = di[k];
          H[k][o + mm] = (c == 2 ? ll1r * rlm * dY[d][o1 + mm] : 0.0) + (d == 2 ? ll1r * rlm * dY[c][o1 + mm] : 0.0) +
                         a * H[k][o1 + mm] -
                         rl1m * rlm * ((c == d ? 2.0 * p2 : 0.0) + 2.0 * xv[c] * dY[d][o2 + mm] + 2.0 * xv[d] * dY[c][o2 + mm]) -
                         b * H[k][o2 + mm];
        }
      }
    }
    {
      const int im = l - 1;
      const double rlm = 1.0 / sqrt(lr * lr - (double)(im * im));
      const double a = ll1r * z * rlm;
      for (int mm = 2 * im - 1; mm <= 2 * im; ++mm) {
        const double p1 = Y[o1 + mm];
        Y[o + mm] = a * p1;
        for (int c = 0; c < 3; ++c) dY[c][o + mm] = (c == 2 ? ll1r * rlm * p1 : 0.0) + a * dY[c][o1 + mm];
        for (int k = 0; k < 6; ++k) {
          const int c = ci[k], d = di[k];
          H[k][o + mm] = (c == 2 ? ll1r * rlm * dY[d][o1 + mm] : 0.0) + (d == 2 ? ll1r * rlm * dY[c][o1 + mm] : 0.0) +
                         a * H[k][o1 + mm];
        }
      }
    }
    {
      const double rll = sqrt(ll1r / (2.0 * lr));
      const int j2 = o1 + 2 * l - 3, j1 = o1 + 2 * l - 2;
      const double q2 = Y[j2], q1 = Y[j1];
      Y[o + 2 * l - 1] = (x * q2 - y * q1) * rll;
      Y[o + 2 * l] = (y * q2 + x * q1) * rll;
      for (int c = 0; c < 3; ++c) {
        const double dx = c == 0, dy = c == 1;
        dY[c][o + 2 * l - 1] = (dx * q2 + x * dY[c][j2] - dy * q1 - y * dY[c][j1]) * rll;
        dY[c][o + 2 * l] = (dy * q2 + y * dY[c][j2] + dx * q1 + x * dY[c][j1]) * rll;
      }
      for (int k = 0; k < 6; ++k) {
        const int c = ci[k], d = di[k];
        const double cx = c == 0, cy = c == 1, dx = d == 0, dy = d == 1;
        H[k][o + 2 * l - 1] = (cx * dY[d][j2] + dx * dY[c][j2] + x * H[k][j2] - cy * dY[d][j1] - dy * dY[c][j1] -
                               y * H[k][j1]) * rll;
        H[k][o + 2 * l] = (cy * dY[d][j2] + dy * dY[c][j2] + y * H[k][j2] + cx * dY[d][j1] + dx * dY[c][j1] +
                           x * H[k][j1]) * rll;
      }
    }
  }
}

// phi, grad phi and (hess) the Hessian of the items' functions on their tiles:
// plane c (phi; x, y, z; xx, xy, xz, yy, yz, zz) at out + c plane, rows of 128
// points per slot.  Block = the 128 points of a tile, a range of items.
template <int L>
__global__ void __launch_bounds__(128) k_hess_items(const BasisItem* __restrict__ items, int64_t nitems,
                                                    BasisIO<double> io, DevSA sa, bool hess, int64_t plane,
                                                    double* __restrict__ out) {
  const int64_t per = (nitems + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * per, i1 = min(nitems, i0 + per);
  constexpr int ci[6] = {0, 0, 0, 1, 1, 2}, di[6] = {0, 1, 2, 1, 2, 2};
  for (int64_t i = i0; i < i1; ++i) {
    const BasisItem it = items[i];
    const int64_t q = (int64_t)it.tile * 128 + threadIdx.x;
    const double x = __ldg(io.qx + q) - it.ax, y = __ldg(io.qy + q) - it.ay, z = __ldg(io.qz + q) - it.az;
    double Y[16], dY[3][16], H[6][16];
    solid_harmonics_h<L>(x, y, z, Y, dY, H);
    const double r2 = x * x + y * y + z * z;
    const double xv[3] = {x, y, z};
    // symmetry-adapted harmonics of this l
    double Ys[2 * L + 1], dYs[3][2 * L + 1], Hs[6][2 * L + 1];
#pragma unroll
    for (int m = 0; m < 2 * L + 1; ++m) {
      if (sa.identity) {
        Ys[m] = Y[L * L + m];
#pragma unroll
        for (int c = 0; c < 3; ++c) dYs[c][m] = dY[c][L * L + m];
#pragma unroll
        for (int k = 0; k < 6; ++k) Hs[k][m] = H[k][L * L + m];
      } else {
        double v = 0, g[3] = {0, 0, 0}, h[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int n = 0; n < 2 * L + 1; ++n) {
          const double cf = sa.c[L][m][n];
          v += cf * Y[L * L + n];
#pragma unroll
          for (int c = 0; c < 3; ++c) g[c] += cf * dY[c][L * L + n];
#pragma unroll
          for (int k = 0; k < 6; ++k) h[k] += cf * H[k][L * L + n];
        }
        Ys[m] = v;
#pragma unroll
        for (int c = 0; c < 3; ++c) dYs[c][m] = g[c];
#pragma unroll
        for (int k = 0; k < 6; ++k) Hs[k][m] = h[k];
      }
    }
    uint64_t rem = it.mask;
    for (int k = 0; k < it.nsig; ++k) {
      const int rr = __ffsll((long long)rem) - 1;
      rem &= rem - 1;
      // R, dR = sum c (-2 alpha) v and d2R = sum c (4 alpha^2) v of radial function rr:
      // d_c R = x_c dR, d_c d_d R = delta_cd dR + x_c x_d d2R
      double R = 0.0, dR = 0.0, d2R = 0.0;
      auto add = [&](double alpha, double c) {
        const double ar2 = alpha * r2;
        if (!__any_sync(0xffffffffu, ar2 < 50.0)) return;
        const double v = ar2 < 50.0 ? c * exp(-ar2) : 0.0;
        R += v;
        dR += (-2.0 * alpha) * v;
        d2R += (4.0 * alpha * alpha) * v;
      };
      if (it.seg) {
        const int2 rg = __ldg(io.rng + it.rad_off + rr);
        for (int e = rg.x; e < rg.y; ++e) {
          const double2 p = __ldg(io.prim + it.exp_off + e);
          add(p.x, p.y);
        }
      } else {
        const int e0 = rr < it.nunc ? rr : 0, e1 = rr < it.nunc ? rr + 1 : it.nexp;
        for (int e = e0; e < e1; ++e) {
          const double cf = rr < it.nunc ? 1.0 : __ldg(io.contr + it.con_off + e + (int64_t)it.nexp * (rr - it.nunc));
          add(__ldg(io.exps + it.exp_off + e), cf * __ldg(io.norms + it.exp_off + e));
        }
      }
#pragma unroll
      for (int m = 0; m < 2 * L + 1; ++m) {
        double* o = out + (it.slot - io.s0 + (int64_t)m * it.nsig + k) * 128 + threadIdx.x;
        o[0] = Ys[m] * R;
#pragma unroll
        for (int c = 0; c < 3; ++c) o[(1 + c) * plane] = dYs[c][m] * R + Ys[m] * xv[c] * dR;
        if (hess) {
#pragma unroll
          for (int h = 0; h < 6; ++h) {
            const int c = ci[h], d = di[h];
            o[(4 + h) * plane] = Hs[h][m] * R + (dYs[c][m] * xv[d] + dYs[d][m] * xv[c]) * dR +
                                 Ys[m] * ((c == d ? dR : 0.0) + xv[c] * xv[d] * d2R);
          }
        }
      }
    }
  }
}

// Zero the padding slots of each tile in the first np planes (grid = chunk tiles).
__global__ void __launch_bounds__(128) k_grad_pads(const int64_t* __restrict__ tso, const int* __restrict__ listed,
                                                   int64_t t0, int64_t s0, int np, int64_t plane,
                                                   double* __restrict__ out) {
  const int64_t t = t0 + blockIdx.x;
  for (int64_t r = tso[t] - s0 + listed[t]; r < tso[t + 1] - s0; ++r)
    for (int c = 0; c < np; ++c) out[c * plane + r * 128 + threadIdx.x] = 0.0;
}

// index of the Hessian component (c, d) in xx, xy, xz, yy, yz, zz
__device__ __forceinline__ int hidx(int c, int d) {
  const int a = c < d ? c : d, b = c < d ? d : c;
  return a == 0 ? b : (a == 1 ? 2 + b : 5);
}

// coef planes per spin: a, b_x, b_y, b_z, c (c = w df/dtau, meta-GGAs)
constexpr int kCoefPlanes = 5;

// Per point of the chunk: the functional at rho_s, grad rho_s (den[(7 s + c) ld
// + p], c = 0..3) and for meta-GGAs tau_s = 1/2 sum_j (2 tau_j) (c = 4..6), and
// the coefficients a_s, b_s, c_s (0 on padding points); ef = w_raw f, and
// sum w f is added into *exc.
__global__ void __launch_bounds__(128) k_grad_coef(XcConst K, int functional, bool gga, int ispin, int64_t ld,
                                                   const double* __restrict__ w, const double* __restrict__ wraw,
                                                   const double* __restrict__ den, double* __restrict__ coef,
                                                   double* __restrict__ ef, double* __restrict__ exc) {
  const int64_t p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const bool mgga = PGXC_XC_IS_MGGA(functional);
  const double wp = w[p], wr = wraw[p];
  double f = 0.0;
  if (wp == 0.0 && wr == 0.0) {
    for (int c = 0; c < kCoefPlanes * ispin; ++c) coef[c * ld + p] = 0.0;
  } else {
    double rho[2] = {0, 0}, gr[2][3] = {{0, 0, 0}, {0, 0, 0}}, tau[2] = {0, 0};
    for (int s = 0; s < ispin; ++s) {
      const double* d = den + (int64_t)(7 * s) * ld + p;
      rho[s] = d[0];
      if (gga)
        for (int c = 0; c < 3; ++c) gr[s][c] = d[(1 + c) * ld];
      if (mgga) tau[s] = 0.5 * (d[4 * ld] + d[5 * ld] + d[6 * ld]);
    }
    double fr[2] = {0, 0}, fg[3] = {0, 0, 0}, ft[2] = {0, 0};
    if (ispin == 1) {
      const double g = gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2];
      if (mgga) mgga::mgga_closed(functional, rho[0], g, tau[0], f, fr[0], fg[0], ft[0]);
      else if (gga) xc_gga(K, rho[0], g, f, fr[0], fg[0]);
      else xc_vwn(K, rho[0], f, fr[0]);
      coef[p] = wp * fr[0];
      for (int c = 0; c < 3; ++c) coef[(1 + c) * ld + p] = gga ? wp * 2.0 * fg[0] * gr[0][c] : 0.0;
      coef[4 * ld + p] = wp * ft[0];
    } else {
      const double r2[2] = {rho[0], rho[1]};
      const double g3[3] = {gr[0][0] * gr[0][0] + gr[0][1] * gr[0][1] + gr[0][2] * gr[0][2],
                            gr[1][0] * gr[1][0] + gr[1][1] * gr[1][1] + gr[1][2] * gr[1][2],
                            gr[0][0] * gr[1][0] + gr[0][1] * gr[1][1] + gr[0][2] * gr[1][2]};
      double fr2[2], fg3[3];
      if (mgga) mgga::mgga_open(functional, r2, g3, tau, f, fr2, fg3, ft);
      else if (gga) xc_open<true>(K, r2, g3, f, fr2, fg3);
      else xc_open<false>(K, r2, g3, f, fr2, fg3);
      for (int s = 0; s < 2; ++s) {
        coef[(kCoefPlanes * s) * ld + p] = wp * fr2[s];
        for (int c = 0; c < 3; ++c)
          coef[(kCoefPlanes * s + 1 + c) * ld + p] =
              gga ? wp * (2.0 * fg3[s] * gr[s][c] + fg3[2] * gr[1 - s][c]) : 0.0;
        coef[(kCoefPlanes * s + 4) * ld + p] = wp * ft[s];
      }
    }
  }
  ef[p] = wr * f;
  double e = wp * f;
  for (int off = 16; off > 0; off >>= 1) e += __shfl_down_sync(0xffffffffu, e, off);
  if ((threadIdx.x & 31) == 0 && e != 0.0) atomicAdd(exc, e);
}

// GGAs (not meta-GGAs): the Y_j enter the orbital terms only as
// sum_j b_j Y_j = W P with W = sum_j b_j d_j phi, one product instead of
// three.  Padding rows are zero (grid = chunk tiles).
__global__ void __launch_bounds__(128) k_grad_w(const int64_t* __restrict__ tso, const int* __restrict__ listed,
                                                int64_t t0, int64_t s0, const double* __restrict__ B, int64_t plane,
                                                const double* __restrict__ cb, int64_t ld, double* __restrict__ W) {
  const int64_t t = t0 + blockIdx.x, p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const double b0 = cb[p], b1 = cb[ld + p], b2 = cb[2 * ld + p];
  const int64_t o0 = (tso[t] - s0) * 128 + threadIdx.x;
  const int n = (int)(tso[t + 1] - tso[t]), nl = listed[t];
#pragma unroll 4
  for (int r = 0; r < nl; ++r) {
    const int64_t o = o0 + r * 128;
    W[o] = b0 * B[plane + o] + b1 * B[2 * plane + o] + b2 * B[3 * plane + o];
  }
  for (int r = nl; r < n; ++r) W[o0 + r * 128] = 0.0;
}

// The orbital terms in one pass: q^s_mu,k(p) is formed once per function and
// point.  Block = a tile, thread = point; a tile's slots come atom by atom, so
// -q is summed over an atom's functions in registers and reduced over the warp
// once per atom (a reduction per function took most of the instructions), +q
// goes to the point's host through the thread's running sum.  The functions of
// the point's own host are left out of both: -q + q = 0 on the same atom, and
// near a nucleus these terms are by far the largest, so that rounded once on
// each side they were most of the error (40 atoms: two runs differed by 4e-12
// of the gradient's norm and its sum over atoms was 2e-12, now 3e-15 and 1e-14).
__global__ void __launch_bounds__(128) k_grad_orb(bool gga, bool mgga, int ispin, int natm,
                                                  const int64_t* __restrict__ tso, const int* __restrict__ listed,
                                                  const int* __restrict__ slot_fn, int64_t t0, int64_t s0,
                                                  const int* __restrict__ fatom, const int* __restrict__ owner,
                                                  const double* __restrict__ B, int64_t plane,
                                                  const double* __restrict__ XY, int nxy,
                                                  const double* __restrict__ coef, int64_t ld,
                                                  double* __restrict__ grad) {
  extern __shared__ double gs[];  // [natm][3]
  for (int i = threadIdx.x; i < 3 * natm; i += 128) gs[i] = 0.0;
  __syncthreads();
  const int64_t t = t0 + blockIdx.x, p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const int lane = threadIdx.x & 31, nl = listed[t];
  const int* fn = slot_fn + (tso[t] - s0);
  double a[2] = {0, 0}, b[2][3] = {{0, 0, 0}, {0, 0, 0}}, ct[2] = {0, 0};
  for (int sp = 0; sp < ispin; ++sp) {
    a[sp] = coef[(kCoefPlanes * sp) * ld + p];
    if (gga)
      for (int j = 0; j < 3; ++j) b[sp][j] = coef[(kCoefPlanes * sp + 1 + j) * ld + p];
    if (mgga) ct[sp] = coef[(kCoefPlanes * sp + 4) * ld + p];
  }
  double tot[3] = {0, 0, 0}, qa[3] = {0, 0, 0};
  int atom = nl > 0 ? fatom[fn[0]] : 0;
  const int h = owner[t * 128 + threadIdx.x];
  auto flush = [&]() {
    for (int k = 0; k < 3; ++k) {
      double v = atom == h ? 0.0 : qa[k];
      tot[k] += v;
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) atomicAdd(&gs[3 * atom + k], -v);
      qa[k] = 0.0;
    }
  };
  const int64_t o0 = (tso[t] - s0) * 128 + threadIdx.x;
#pragma unroll 2
  for (int r = 0; r < nl; ++r) {
    const int at = fatom[fn[r]];
    if (at != atom) {
      flush();
      atom = at;
    }
    const int64_t o = o0 + r * 128;
    double d[3], H[6];
    for (int c = 0; c < 3; ++c) d[c] = B[(1 + c) * plane + o];
    if (gga)
      for (int k = 0; k < 6; ++k) H[k] = B[(4 + k) * plane + o];
    for (int sp = 0; sp < ispin; ++sp) {
      const double* xy = XY + (int64_t)(nxy * sp) * plane + o;
      const double X = xy[0];
      for (int k = 0; k < 3; ++k) qa[k] += 2.0 * a[sp] * d[k] * X;
      if (!gga) continue;
      if (!mgga) {  // sum_j b_j Y_j = (sum_j b_j d_j phi) P = V
        const double V = xy[plane];
        for (int k = 0; k < 3; ++k) {
          double u = d[k] * V;
          for (int j = 0; j < 3; ++j) u += b[sp][j] * H[hidx(k, j)] * X;
          qa[k] += 2.0 * u;
        }
        continue;
      }
      double Yj[3];
      for (int j = 0; j < 3; ++j) Yj[j] = xy[(1 + j) * plane];
      for (int k = 0; k < 3; ++k) {
        double u = 0.0;
        for (int j = 0; j < 3; ++j) u += b[sp][j] * (H[hidx(k, j)] * X + d[k] * Yj[j]);
        qa[k] += 2.0 * u;
        // meta-GGAs: tau moves with the functions through d_k d_j phi
        for (int j = 0; j < 3; ++j) qa[k] += ct[sp] * H[hidx(k, j)] * Yj[j];
      }
    }
  }
  flush();
  // host sums: one shared atomic per warp when its points share a host
  const int h0 = __shfl_sync(0xffffffffu, h, 0);
  if (__all_sync(0xffffffffu, h == h0)) {
    for (int k = 0; k < 3; ++k) {
      double v = tot[k];
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) atomicAdd(&gs[3 * h0 + k], v);
    }
  } else {
    for (int k = 0; k < 3; ++k) atomicAdd(&gs[3 * h + k], tot[k]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * natm; i += 128)
    if (gs[i] != 0.0) atomicAdd(grad + i, gs[i]);
}

// Thread per point.  Pass 1 stores, per atom b, the point's distance d_b,
// its reciprocal and the row of P_b = prod_{c != b} s(mu_bc): the product of
// its nonzero factors, their zero count and the index of a zero factor
// (scratch [atom][ld]).  Pass 2 gathers, per atom x, the terms of the pairs
// (x, y) and (y, x) in registers (no scatter):
//   dmu_xy/dR_x = -u_x/R - mu r_xy/R^2,  dmu_yx/dR_x = u_x/R + mu r_xy/R^2,
//   kappa_xy = c_x L_xy s'(mu_xy), c_b = ef (delta_bh - W_h) / Z,
// L_xy the product of row x without its factor y; the point moves with its
// host h, which collects kappa_xy (u_x - u_y)/R of every pair.  Each atom's sum
// is reduced over the warp and added to shared memory, then to grad.
//
// Rows whose leave-one-out products are all negligible ("dead" rows) take
// part only through their pairs with live rows.  Every factor is at most 1,
// so L_xy <= the product of row x's factors with the eight atoms nearest to the
// point, leaving out the smallest of them; where that bound is below 2^-60
// the row is dead (its P_x is below the same bound and is dropped from Z).
// Both loops of pass 2 run over all atoms in the same order on every lane of
// a warp; a pair is skipped when, for every lane, both its rows are dead.
// Where mu <= -0.994, s rounds to exactly 1 and leaves the row product
// unchanged.
//
// mu_bc = (d_b - d_c) RN(1/R_bc): pass 1 and pass 2 form it alike, and
// mu_cb = -mu_bc exactly, so s(mu_cb) = (1 + p3(mu_bc))/2 with the same
// bits as pass 1's factor (p3 is odd in floating point too): a factor that is
// exactly 0 in one pass is 0 in the other.
constexpr double kGradEdge = 0.9941;
constexpr double kGradTau = 0x1p-60;
constexpr int kGradNear = 8;  // atoms nearest to the point in the dead-row bound

// p3(mu) and ds/dmu (even in mu).  Each step RN(RN(q / 2) RN(3 - RN(q q)))
// is formed as RN(q RN(1.5 - RN(q q) / 2)) (one FMA inside): halving is exact
// and commutes with rounding for these normal operands, so the bits agree.
__device__ __forceinline__ void becke_p3(double mu, double& q3, double& ds) {
  const double q1 = __dmul_rn(mu, __fma_rn(-0.5, __dmul_rn(mu, mu), 1.5));
  const double q2 = __dmul_rn(q1, __fma_rn(-0.5, __dmul_rn(q1, q1), 1.5));
  q3 = __dmul_rn(q2, __fma_rn(-0.5, __dmul_rn(q2, q2), 1.5));
  ds = -0.5 * (1.5 * (1.0 - q2 * q2)) * (1.5 * (1.0 - q1 * q1)) * (1.5 * (1.0 - mu * mu));
}

template <bool MASK>
__global__ void __launch_bounds__(128) k_grad_weights(const double* __restrict__ atoms,
                                                      const double* __restrict__ dist,
                                                      const double* __restrict__ rdist, int natm,
                                                      const double* __restrict__ px, const double* __restrict__ py,
                                                      const double* __restrict__ pz, const int* __restrict__ owner,
                                                      int64_t p0, int64_t nvalid, int64_t ld,
                                                      const double* __restrict__ ef, double* __restrict__ sd,
                                                      double* __restrict__ sinv, double* __restrict__ spnz,
                                                      int* __restrict__ snz, double* __restrict__ grad) {
  extern __shared__ double G[];  // 3 natm sums of the block
  for (int i = threadIdx.x; i < 3 * natm; i += blockDim.x) G[i] = 0.0;
  __syncthreads();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = p < nvalid && ef[p] != 0.0;
  double rv[3] = {0, 0, 0}, e = 0.0, Z = 0.0, Wh = 0.0;
  int h = 0;
  uint64_t live_lo = 0, live_hi = 0;  // live rows of the point (atoms < 128; MASK)
  if (live) {
    rv[0] = px[p0 + p]; rv[1] = py[p0 + p]; rv[2] = pz[p0 + p];
    h = owner[p0 + p];
    e = ef[p];
    int nb[kGradNear];
    double nr[kGradNear];
#pragma unroll
    for (int c = 0; c < kGradNear; ++c) {
      nb[c] = -1;
      nr[c] = INFINITY;
    }
    for (int b = 0; b < natm; ++b) {
      const double t0 = rv[0] - atoms[3 * b], t1 = rv[1] - atoms[3 * b + 1], t2 = rv[2] - atoms[3 * b + 2];
      const double r = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
      sd[b * ld + p] = r;
      sinv[b * ld + p] = r > 0.0 ? 1.0 / r : 0.0;
      if (r < nr[kGradNear - 1]) {  // keep the kGradNear nearest sorted (ties in ascending atom order)
        int kk = b;
        double rr = r;
#pragma unroll
        for (int c = 0; c < kGradNear; ++c) {
          if (rr < nr[c]) {
            const double tr = nr[c];
            const int tk = nb[c];
            nr[c] = rr;
            nb[c] = kk;
            rr = tr;
            kk = tk;
          }
        }
      }
    }
    double Ph = 0.0;
    for (int b = 0; b < natm; ++b) {
      const double db = sd[b * ld + p];
      const double* Rb = dist + (int64_t)b * natm;
      const double* Yb = rdist + (int64_t)b * natm;
      // bound: the near factors' product with its smallest factor left out (with
      // no zero factor Q / smin; with one, Q, the others; with more, 0).  Taking
      // in a further factor never raises it, so the nearest atoms come first and
      // the loop stops once it is below tau.
      double Q = 1.0, smin = 1.0, bound = 1.0;
      int nzero = 0;
#pragma unroll
      for (int c = 0; c < kGradNear; ++c) {
        const int k = nb[c];
        if (k < 0 || k == b) continue;
        const double R = Rb[k], d = __dsub_rn(db, nr[c]);
        if (d <= -__dmul_rn(kGradEdge, R)) continue;
        double q3, ds;
        becke_p3(__dmul_rn(d, Yb[k]), q3, ds);
        const double sv = __dmul_rn(0.5, __dsub_rn(1.0, q3));
        if (sv == 0.0) ++nzero;
        else Q *= sv;
        smin = fmin(smin, sv);
        bound = nzero == 0 ? (smin > 0.0 ? Q / smin : 0.0) : (nzero == 1 ? Q : 0.0);
        if (bound < kGradTau) break;
      }
      if (bound < kGradTau) {
        spnz[b * ld + p] = 0.0;
        snz[b * ld + p] = -2;
        continue;
      }
      double pnz = 1.0, fmin_row = 1.0;
      int nz = 0, zc = -1;
      for (int c = 0; c < natm; ++c) {
        if (c == b) continue;
        const double R = Rb[c], d = __dsub_rn(db, sd[c * ld + p]);
        if (d <= -__dmul_rn(kGradEdge, R)) continue;  // s == 1 exactly
        double q3, ds;
        becke_p3(__dmul_rn(d, Yb[c]), q3, ds);
        const double sv = __dmul_rn(0.5, __dsub_rn(1.0, q3));
        if (sv == 0.0) { ++nz; zc = c; }
        else { pnz *= sv; fmin_row = fmin(fmin_row, sv); }
      }
      // the largest leave-one-out product of the whole row decides: below tau the row is dead
      const double lmax = nz == 0 ? pnz / fmin_row : (nz == 1 ? pnz : 0.0);
      if (lmax < kGradTau) {
        spnz[b * ld + p] = 0.0;
        snz[b * ld + p] = -2;
        continue;
      }
      spnz[b * ld + p] = pnz;
      snz[b * ld + p] = nz == 0 ? -1 : zc;  // -1: no zero; c: the one zero; -2: dead
      if (b < 64) live_lo |= 1ull << b;
      else if (b < 128) live_hi |= 1ull << (b - 64);
      const double P = nz ? 0.0 : pnz;
      Z += P;
      if (b == h) Ph = P;
    }
    if (Z > 0.0) Wh = Ph / Z;
  }
  const bool go = live && Z > 0.0;
  const double iZ = go ? 1.0 / Z : 0.0;
  double gh[3] = {0, 0, 0};
  const int lane = threadIdx.x & 31;
  // rows live on some lane of the warp (MASK)
  uint64_t ulo = 0, uhi = 0;
  if (MASK) {
    const uint64_t mlo = go ? live_lo : 0ull, mhi = go ? live_hi : 0ull;
    ulo = ((uint64_t)__reduce_or_sync(0xffffffffu, (unsigned)(mlo >> 32)) << 32) |
          __reduce_or_sync(0xffffffffu, (unsigned)mlo);
    uhi = ((uint64_t)__reduce_or_sync(0xffffffffu, (unsigned)(mhi >> 32)) << 32) |
          __reduce_or_sync(0xffffffffu, (unsigned)mhi);
  }
  for (int x = 0; x < natm; ++x) {
    double gx[3] = {0, 0, 0};
    int zx = -2;
    double dx = 0.0, cx = 0.0, pnx = 0.0, ux[3] = {0, 0, 0};
    if (go) {
      dx = sd[x * ld + p];
      cx = e * ((x == h ? 1.0 : 0.0) - Wh) * iZ;
      const double ix = sinv[x * ld + p];
      for (int k = 0; k < 3; ++k) ux[k] = (rv[k] - atoms[3 * x + k]) * ix;
      if (!MASK || ((x < 64 ? live_lo >> x : live_hi >> (x - 64)) & 1ull)) {
        zx = snz[x * ld + p];
        pnx = spnz[x * ld + p];
      }
    }
    const bool lx = zx != -2;
    const double* Yx = rdist + (int64_t)x * natm;
    // a row x dead on every lane pairs only with rows live on some lane: walk
    // those (the same y in the same order as the full loop takes them)
    const bool xall = MASK && !__any_sync(0xffffffffu, lx);
    uint64_t ylo = xall ? ulo : ~0ull, yhi = xall ? uhi : ~0ull;
    for (int y = 0; y < natm; ++y) {
      if (MASK && xall) {
        if (ylo) {
          y = __ffsll((long long)ylo) - 1;
          ylo &= ylo - 1;
        } else if (yhi) {
          y = 64 + __ffsll((long long)yhi) - 1;
          yhi &= yhi - 1;
        } else {
          break;
        }
        if (y >= natm) break;
      }
      if (y == x) continue;
      int zy = -2;
      bool ly;
      if (MASK) {
        ly = ((y < 64 ? live_lo >> y : live_hi >> (y - 64)) & 1ull) != 0;
      } else {
        zy = go ? snz[y * ld + p] : -2;
        ly = zy != -2;
      }
      const bool need = go && (lx || ly);
      if (!__any_sync(0xffffffffu, need)) continue;
      if (!need) continue;
      if (MASK && ly) zy = snz[y * ld + p];
      const double iR = Yx[y];
      const double dy = sd[y * ld + p];
      const double mu = __dmul_rn(__dsub_rn(dx, dy), iR);
      double q3, ds;
      becke_p3(mu, q3, ds);
      const double sxy = __dmul_rn(0.5, __dsub_rn(1.0, q3)), syx = __dmul_rn(0.5, __dadd_rn(1.0, q3));
      // leave-one-out products of rows x (without y) and y (without x)
      const double Lxy = zx == -1 ? (sxy != 0.0 ? pnx / sxy : 0.0) : (zx == y ? pnx : 0.0);
      const double pny = ly ? spnz[y * ld + p] : 0.0;
      const double Lyx = zy == -1 ? (syx != 0.0 ? pny / syx : 0.0) : (zy == x ? pny : 0.0);
      const double cy = e * ((y == h ? 1.0 : 0.0) - Wh) * iZ;
      const double kxy = cx * Lxy * ds, kyx = cy * Lyx * ds;
      if (kxy == 0.0 && kyx == 0.0) continue;
      const double iy = sinv[y * ld + p];
      const double mr = mu * iR * iR;
      for (int k = 0; k < 3; ++k) {
        const double rxy = atoms[3 * x + k] - atoms[3 * y + k];
        const double uy = (rv[k] - atoms[3 * y + k]) * iy;
        gx[k] += (kyx - kxy) * (ux[k] * iR + mr * rxy);
        gh[k] += kxy * (ux[k] - uy) * iR;
      }
    }
    for (int k = 0; k < 3; ++k)
      for (int off = 16; off > 0; off >>= 1) gx[k] += __shfl_down_sync(0xffffffffu, gx[k], off);
    if (lane == 0)
      for (int k = 0; k < 3; ++k)
        if (gx[k] != 0.0) atomicAdd(&G[3 * x + k], gx[k]);
  }
  if (go)
    for (int k = 0; k < 3; ++k) atomicAdd(&G[3 * h + k], gh[k]);
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * natm; i += blockDim.x)
    if (G[i] != 0.0) atomicAdd(grad + i, G[i]);
}

}  // namespace

int64_t grad_planes(bool gga, bool mgga, int ispin) {
  return mgga ? 10 + 4 * ispin : gga ? 11 + 2 * ispin : 4 + ispin;
}

void launch_grad_chunk(const GradChunk& g, const BuildArgs& a, ScreenPlan* sp, size_t c, cudaStream_t st) {
  const int64_t t0 = sp->chunk_t0[c], nt = sp->chunk_t0[c + 1] - t0, s0 = sp->h_tso[(size_t)t0], ld = g.ld;
  const int64_t plane = g.plane;
  const int* slot_fn = g.lists->slot_fn;
  grad_plan_lists(sp, a, c, *g.lists, st);
  double* B = g.rows;                                  // phi, grad phi and (GGAs) the Hessian
  double* XY = B + (g.gga ? 10 : 4) * plane;           // per spin X; X, V (GGA); X, Y_j (meta-GGA)
  const int nxy = g.mgga ? 4 : g.gga ? 2 : 1;
  double* W = XY + (int64_t)nxy * g.ispin * plane;
  const BasisIO<double> io{a.exps, a.norms, a.contr,  a.rng,   a.prim,  sp->qx,  sp->qy, sp->qz,
                           s0,     t0,      nullptr, nullptr, nullptr, nullptr, nullptr};
  auto hess = [&](auto Lc) {
    constexpr int L = decltype(Lc)::value;
    const BasisItem* it = g.lists->items[L];
    const int64_t n = sp->tile_item[L][(size_t)(t0 + nt)] - sp->tile_item[L][(size_t)t0];
    if (n > 0)
      k_hess_items<L><<<(unsigned)std::min<int64_t>(n, (int64_t)sp->nsm * 32), 128, 0, st>>>(it, n, io, a.sa, g.gga,
                                                                                             plane, B);
  };
  hess(std::integral_constant<int, 0>());
  hess(std::integral_constant<int, 1>());
  hess(std::integral_constant<int, 2>());
  hess(std::integral_constant<int, 3>());
  k_grad_pads<<<(unsigned)nt, 128, 0, st>>>(sp->tso, sp->listed, t0, s0, g.mgga ? 4 : 1, plane, B);
  const double *gx = B + plane, *gy = B + 2 * plane, *gz = B + 3 * plane;
  for (int s = 0; s < g.ispin; ++s) {
    double* d = g.den + (int64_t)(7 * s) * ld;
    double* X = XY + (int64_t)(nxy * s) * plane;
    grad_contract(sp, slot_fn, t0, nt, s0, B, g.gga ? gx : nullptr, gy, gz, g.P[s], a.ldc, X, d, d + ld, d + 2 * ld, d + 3 * ld,
                  g.orb[s], st);
    // the Y_j only for meta-GGAs (tau and its terms), GGAs take V = W P after the coefficients
    for (int j = 0; j < 3 && g.mgga; ++j)
      grad_contract(sp, slot_fn, t0, nt, s0, B + (1 + j) * plane, nullptr, nullptr, nullptr, g.P[s], a.ldc, X + (1 + j) * plane,
                    d + (4 + j) * ld, nullptr, nullptr, nullptr, g.orb[s], st);
  }
  k_grad_coef<<<(unsigned)nt, 128, 0, st>>>(a.xc, g.functional, g.gga, g.ispin, ld, sp->qw + t0 * 128,
                                            sp->qwraw + t0 * 128, g.den, g.coef, g.ef + t0 * 128, g.exc);
  for (int s = 0; s < g.ispin && g.gga && !g.mgga; ++s) {
    k_grad_w<<<(unsigned)nt, 128, 0, st>>>(sp->tso, sp->listed, t0, s0, B, plane,
                                           g.coef + (int64_t)(kCoefPlanes * s + 1) * ld, ld, W);
    grad_contract(sp, slot_fn, t0, nt, s0, W, nullptr, nullptr, nullptr, g.P[s], a.ldc, XY + (int64_t)(nxy * s + 1) * plane,
                  g.den, nullptr, nullptr, nullptr, g.orb[s], st);  // (rho is done with: its sum goes to scratch)
  }
  const int smem = (int)sizeof(double) * 3 * g.natm;
  if (smem > 48 * 1024) raise_smem_limit(k_grad_orb, smem);
  k_grad_orb<<<(unsigned)nt, 128, smem, st>>>(g.gga, g.mgga, g.ispin, g.natm, sp->tso, sp->listed, slot_fn, t0, s0,
                                              g.fatom, sp->qowner, B, plane, XY, nxy, g.coef, ld, g.grad);
}

void launch_grad_weights(const double* atoms, const double* dist, int natm, const double* px, const double* py,
                         const double* pz, const int* owner, int64_t p0, int64_t nvalid, int64_t ld, const double* ef,
                         double* scratch, double* grad, cudaStream_t st) {
  if (nvalid <= 0) return;
  const size_t smem = sizeof(double) * 3 * natm;
  if (smem > 48 * 1024) {
    cudaFuncSetAttribute(k_grad_weights<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_grad_weights<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }
  const double* rdist = dist + (size_t)natm * natm;
  double* sd = scratch;
  double* sinv = scratch + (size_t)natm * ld;
  double* spnz = scratch + (size_t)2 * natm * ld;
  int* snz = (int*)(scratch + (size_t)3 * natm * ld);
  const unsigned nb = (unsigned)((nvalid + 127) / 128);
  if (natm <= 128)
    k_grad_weights<true><<<nb, 128, smem, st>>>(atoms, dist, rdist, natm, px, py, pz, owner, p0, nvalid, ld, ef, sd,
                                                sinv, spnz, snz, grad);
  else
    k_grad_weights<false><<<nb, 128, smem, st>>>(atoms, dist, rdist, natm, px, py, pz, owner, p0, nvalid, ld, ef, sd,
                                                 sinv, spnz, snz, grad);
}

}  // namespace pgxc
