// screened.cu -- planning and FP64 kernels of the screened (tile-sparse) XC build.
//
// Per geometry (screen_create):
//   Morton order of the grid, tiles of 128 points (padded with weight-0 copies);
//   k_tile_atom_d2    smallest squared distance of each tile to each atom;
//   k_plan_count, k_plan_fill  per tile the listed functions (slots, padded to
//                     32) and the basis work items (tile, shell, radial mask);
//                     the host sums the counts and makes the chunks.
// Per build (screen_run), per chunk of tiles:
//   k_basis_items     phi, grad phi of listed functions only     [K1]
//   k_tile_init       (first) clears: the padding slots at the end of each tile's
//                     list, and what the INT8 stages max into
//   k_sdensity        X = phi_t P[S_t, S_t] on DMMA, P gathered by cp.async,
//                     fused rho, grad rho (or by the orbitals)     [K3]
//   k_functional      (kernels_fp64.cu)                            [K2]
//   k_svpot           H[S_t, S_t] += Z_t^T phi_t on DMMA with Z = A phi
//                     (+ B . grad phi) formed in shared memory, scatter-added
//                     into the full matrix with FP64 atomics       [K4]
// then k_spack packs V (LDA: H; GGA: H + H^T, the symmetrisation of
// modules/xc_hamiltonian.f90:1559-1566) into the tristore order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include <cuda_runtime.h>

#include "basis.cuh"
#include "dgemm.cuh"
#include "grid.h"
#include "kernels.h"
#include "screened.h"
#include "screened_mixed.h"
#include "screened_plan.h"

namespace pgxc {

namespace {

template <typename T>
cudaError_t sp_alloc(ScreenPlan* sp, T** p, size_t n) {
  void* q = nullptr;
  cudaError_t e = cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T));
  if (e == cudaSuccess) {
    sp->allocs.push_back(q);
    *p = (T*)q;
  }
  return e;
}

// ---------------------------------------------------------------------------
// planning kernels
// ---------------------------------------------------------------------------
// index of point q of the tiles among the n of the grid (order null: as they lie there), or -1: padding
__device__ __forceinline__ int64_t point_index(const int64_t* __restrict__ order, int64_t n, int64_t q) {
  return order ? order[q] : (q < n ? q : -1);
}

__global__ void k_gather_points(const int64_t* __restrict__ order, int64_t n, int64_t nq,
                                const double* __restrict__ px, const double* __restrict__ py,
                                const double* __restrict__ pz, const double* __restrict__ w, double* __restrict__ qx,
                                double* __restrict__ qy, double* __restrict__ qz, double* __restrict__ qw) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  int64_t i = point_index(order, n, q);
  double wt = 0.0;
  if (i >= 0) wt = w[i];
  else i = point_index(order, n, q & ~(int64_t)127);  // padding: a weight-0 copy of the tile's first point
  qx[q] = px[i];
  qy[q] = py[i];
  qz[q] = pz[i];
  qw[q] = wt;
}

// d2[t][a] = min over the tile's points of |r - R_a|^2, rounded down to float
__global__ void __launch_bounds__(128) k_tile_atom_d2(const int64_t* __restrict__ order, int64_t n,
                                                      const double* __restrict__ px, const double* __restrict__ py,
                                                      const double* __restrict__ pz, const double* __restrict__ atoms,
                                                      int natm, float* __restrict__ d2) {
  __shared__ float red[4];
  const int64_t t = blockIdx.x;
  int64_t i = point_index(order, n, t * 128 + threadIdx.x);
  if (i < 0) i = point_index(order, n, t * 128);
  const double x = px[i], y = py[i], z = pz[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int a = 0; a < natm; ++a) {
    const double dx = x - atoms[3 * a], dy = y - atoms[3 * a + 1], dz = z - atoms[3 * a + 2];
    float f = __double2float_rd(dx * dx + dy * dy + dz * dz);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f = fminf(f, __shfl_xor_sync(0xffffffffu, f, o));
    if (lane == 0) red[warp] = f;
    __syncthreads();
    if (threadIdx.x == 0) d2[t * natm + a] = fminf(fminf(red[0], red[1]), fminf(red[2], red[3]));
    __syncthreads();
  }
}

// The listing of a tile: shell s has the radial functions whose squared listing
// radius r2[s][rr] exceeds the tile's smallest squared distance to its atom.
__device__ __forceinline__ unsigned long long plan_mask(const DevShell& S, double dd, const double* __restrict__ r2) {
  unsigned long long m = 0;
  for (int rr = 0; rr < S.nrad; ++rr)
    if (dd < r2[rr]) m |= 1ull << rr;
  return m;
}

// cnt[t] = {listed functions, basis items of l = 0..3} of tile t (block per tile)
__global__ void __launch_bounds__(128) k_plan_count(const float* __restrict__ d2, int natm,
                                                    const DevShell* __restrict__ shells, int nsh,
                                                    const double* __restrict__ r2, const int* __restrict__ r2off,
                                                    int* __restrict__ cnt) {
  __shared__ int sum[1 + kMaxL + 1];
  const int64_t t = blockIdx.x;
  if (threadIdx.x < 2 + kMaxL) sum[threadIdx.x] = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < nsh; s += 128) {
    const DevShell S = shells[s];
    const int n = __popcll(plan_mask(S, d2[t * natm + S.atom], r2 + r2off[s]));
    if (!n) continue;
    atomicAdd(&sum[0], n * (2 * S.l + 1));
    atomicAdd(&sum[1 + S.l], 1);
  }
  __syncthreads();
  if (threadIdx.x < 2 + kMaxL) cnt[t * (2 + kMaxL) + threadIdx.x] = sum[threadIdx.x];
}

// The slot list (shell by shell: independent function -> radial function, then
// padding) and the basis items of tiles t0 + block, in shell order: 128 shells at a
// time, their places by a block scan.  start[t] = {first item of l = 0..3}.
__global__ void __launch_bounds__(128) k_plan_fill(const float* __restrict__ d2, int natm,
                                                   const double* __restrict__ atoms,
                                                   const DevShell* __restrict__ shells, int nsh,
                                                   const double* __restrict__ r2, const int* __restrict__ r2off,
                                                   const int64_t* __restrict__ tso, const int64_t* __restrict__ start,
                                                   int64_t t0, TileLists out) {
  __shared__ int scan_n[128];
  __shared__ unsigned scan_l[128];  // four 8-bit counts (at most 128 shells each)
  const int64_t t = t0 + blockIdx.x;
  const int tid = threadIdx.x;
  int64_t slot0 = tso[t], item0[kMaxL + 1];
  for (int l = 0; l <= kMaxL; ++l) item0[l] = start[t * (kMaxL + 1) + l] - out.i0[l];
  for (int s0 = 0; s0 < nsh; s0 += 128) {
    const int s = s0 + tid;
    DevShell S{};
    unsigned long long mask = 0;
    if (s < nsh) {
      S = shells[s];
      mask = plan_mask(S, d2[t * natm + S.atom], r2 + r2off[s]);
    }
    const int nsig = __popcll(mask), n = nsig * (2 * S.l + 1);
    const unsigned one = nsig ? 1u << (8 * S.l) : 0u;
    scan_n[tid] = n;
    scan_l[tid] = one;
    __syncthreads();
    for (int o = 1; o < 128; o <<= 1) {
      const int vn = tid >= o ? scan_n[tid - o] : 0;
      const unsigned vl = tid >= o ? scan_l[tid - o] : 0u;
      __syncthreads();
      scan_n[tid] += vn;
      scan_l[tid] += vl;
      __syncthreads();
    }
    if (nsig) {
      const int64_t slot = slot0 + scan_n[tid] - n;
      BasisItem it{};
      it.ax = atoms[3 * S.atom];
      it.ay = atoms[3 * S.atom + 1];
      it.az = atoms[3 * S.atom + 2];
      it.tile = (int)t;
      it.slot = slot;
      it.nsig = nsig;
      it.mask = mask;
      it.exp_off = S.exp_off;
      it.con_off = S.con_off;
      it.rad_off = S.rad_off;
      it.nexp = S.nexp;
      it.nunc = S.nunc;
      it.seg = S.seg;
      out.items[S.l][item0[S.l] + ((scan_l[tid] - one) >> (8 * S.l) & 255u)] = it;
      int64_t o = slot - out.s0;
      for (int i = 0; i < 2 * S.l + 1; ++i)
        for (unsigned long long m = mask; m; m &= m - 1) out.slot_fn[o++] = S.f0 + i * S.nrad + __ffsll((long long)m) - 1;
    }
    slot0 += scan_n[127];
    for (int l = 0; l <= kMaxL; ++l) item0[l] += scan_l[127] >> (8 * l) & 255u;
    __syncthreads();
  }
  for (int64_t o = slot0 + tid; o < tso[t + 1]; o += 128) out.slot_fn[o - out.s0] = -1;
}

// ---------------------------------------------------------------------------
// FP64 kernels
// ---------------------------------------------------------------------------
// Clears of one chunk before its basis values (grid = chunk tiles): the padding
// slots of each tile (after its listed functions: tso[t] + listed[t] ..
// tso[t+1]) and the points' largest |phi| (pmax not null).
template <bool GGA, typename GT = double>
__global__ void __launch_bounds__(128) k_tile_init(const int64_t* __restrict__ tso, const int* __restrict__ listed,
                                                  int64_t t0, int64_t s0, double* __restrict__ phi,
                                                  GT* __restrict__ gx, GT* __restrict__ gy,
                                                  GT* __restrict__ gz, unsigned long long* __restrict__ pmax) {
  if (pmax) pmax[(int64_t)blockIdx.x * 128 + threadIdx.x] = 0;
  const int64_t t = t0 + blockIdx.x;
  const int64_t r0 = tso[t] - s0 + listed[t], r1 = tso[t + 1] - s0;
  for (int64_t e = r0 * 128 + threadIdx.x; e < r1 * 128; e += 128) {
    phi[e] = 0.0;
    if (GGA) {
      gx[e] = (GT)0;
      gy[e] = (GT)0;
      gz[e] = (GT)0;
    }
  }
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = pred ? 8 : 0;  // 0: fill with zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}

// ---------------------------------------------------------------------------
// The two FP64 contractions of a tile run on DMMA (mma.sync m8n8k4) in CTAs of
// four warps, 16 K values per shared-memory stage.  Both are bound
// by the FP64 tensor pipe (35 TFLOP/s); what the layout is for is keeping it
// fed.  Each SM sub-partition has its own DMMA unit and a CTA holds one warp of
// each, so that three independent CTAs per SM fill one another's barriers and
// epilogues (with eight warps and two CTAs the pipe ran at 63%).  Whole 8-function
// fragments past the listed functions are left out, and the warps' places rotate
// with the tile so that the warps a ragged block leaves idle do not all fall on
// one sub-partition.
// ---------------------------------------------------------------------------
constexpr int kSThreads = 128;
constexpr int kSBlk = 64;   // functions (and points) of a block
constexpr int kRows = 32;   // functions i of a potential CTA, and functions j of a warp's block
constexpr int kSStages = 2;
constexpr int kDK = 16, kDStages = 3, kDLd = kSBlk + kPadMN;  // density stages
constexpr int kXLd = 66;    // row length of the X block: 2 kXLd = 4 mod 16 (conflict-free fragment stores)
constexpr int kZLd = 132;   // row length of the Z block: 128 points, 4 mod 16

template <int NI, int NJ>
struct SAcc {
  double v[NI][NJ][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) v[i][j][0] = v[i][j][1] = 0.0;
  }
};

// the fragments (0..most) of eight functions from `first` on that hold listed ones (warp-uniform)
__device__ __forceinline__ int live_frags(int first, int listed, int most) {
  return min(most, max(0, (listed - first + 7) >> 3));
}

// acc += A B over one K-deep stage, row fragments < mi and column fragments
// < nj.  a(i, k), b(j, k): shared-memory elements.  The fragments of the next
// four K values are read before the products of the current ones are issued.
template <int K, int NI, int NJ, typename FA, typename FB>
__device__ __forceinline__ void s_mma(SAcc<NI, NJ>& acc, FA a, FB b, int mi, int nj) {
  if (mi == 0 || nj == 0) return;
  double af[2][NI], bf[2][NJ];
  auto frags = [&](int u, int kk) {
#pragma unroll
    for (int i = 0; i < NI; ++i) af[u][i] = a(i, kk);
#pragma unroll
    for (int j = 0; j < NJ; ++j) bf[u][j] = b(j, kk);
  };
  frags(0, 0);
  if (mi == NI && nj == NJ) {
#pragma unroll
    for (int q = 0; q < K / 4; ++q) {
      if (q + 1 < K / 4) frags((q + 1) & 1, 4 * q + 4);
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma(acc.v[i][j], af[q & 1][i], bf[q & 1][j]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < K / 4; ++q) {
      if (q + 1 < K / 4) frags((q + 1) & 1, 4 * q + 4);
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        if (i >= mi) break;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (j < nj) dmma(acc.v[i][j], af[q & 1][i], bf[q & 1][j]);
      }
    }
  }
}

// up to three operand planes and their sums, chosen by grid z
struct SPlanes {
  const double *phi0, *phi1, *phi2;
  double *rho0, *rho1, *rho2;
  __device__ __forceinline__ const double* phi(int z) const { return z == 0 ? phi0 : (z == 1 ? phi1 : phi2); }
  __device__ __forceinline__ double* rho(int z) const { return z == 0 ? rho0 : (z == 1 ? rho1 : rho2); }
};
// psi's way through memory and the second launch (screen_orbital_form)
constexpr double kOrbitalMargin = 1.15;
// elements of psi held at once, 1 GB (60 atoms: 256 MB 6.7 ms, 1 GB 6.45: fewer half-empty last waves)
constexpr int64_t kPsiMost = int64_t(1) << 27;
// elements up to which psi's place is made with the context, 128 MB
constexpr int64_t kPsiReserved = int64_t(1) << 24;
// The tile's slot -> function list (slot_fn of the kernels below begins at the
// chunk's first slot s0) in shared memory, -1 from its slots to a
// whole block past them: every index the kernels form is inside it, guarded or
// not (a guarded shared-memory load may be executed all the same).
__host__ __device__ constexpr int sfn_len(int n) { return (n + kSBlk - 1) / kSBlk * kSBlk + kSBlk; }
__device__ __forceinline__ void load_sfn(int* sfn, const int* __restrict__ slot_fn, int n) {
  const int len = sfn_len(n);
  for (int i = threadIdx.x; i < len; i += kSThreads) sfn[i] = i < n ? slot_fn[i] : -1;
}

// K3 (screened): CTA = (tile, half of its 128 points).  X = phi_t P[S_t, S_t]
// in 64-wide column blocks, P gathered element-wise by 8-byte cp.async (thread
// = one column, every second row of a stage); each finished block of X passes
// through shared memory so that a thread then owns one point: the phi and grad phi
// it meets are read in whole rows and the sums take 4 registers.
// tri (GGA = false: only rho, a quadratic form): P is symmetric, so column
// block J takes the rows of the blocks before it doubled and its own block, half
// the products.  Grid z selects the operand plane and its sum (the three tau
// sums of a meta-GGA in one launch).  STORE: X itself is written too (the
// gradient's terms).
// Three CTAs per SM: 60 atoms, 304 of 690 functions per tile (226 GF, 6.4 ms at
// the pipe's rate) 10.8 -> 8.9 ms against one 128-thread CTA form that kept two
// CTAs at 254 registers; four CTAs at 128 registers 9.2, 32-deep stages 9.4.
// The sums' loop has eight slots' loads in flight: 8.9 -> 8.7 ms against four
// (20 atoms meta-GGA 1.04 -> 1.01).
// The orbital form of the same sums (FORM): kPsi, psi_o = sum_k phi_k C[k][o] of
// the tile's points (columns = the nop padded orbitals; P = C, ldc = nop), with
// rho = sum occ psi^2, written to X where grad rho follows; kFromPsi, X = sum_o
// psi_o occ_o C[.][o] (rows = psi; P = occ C by orbitals) with grad rho alone.
// kPsi with GGA: the planes are grad phi's (grid z), so that x = d_z psi: the tau
// sum, and grad rho_z = 2 sum occ psi d_z psi with psi from X (no kFromPsi).
// Taken while 2 nocc is below the tiles' mean length (screen_orbital_form).
enum { kFromP, kPsi, kFromPsi };
template <bool GGA, bool STORE = false, int FORM = kFromP>
__global__ void __launch_bounds__(kSThreads, 3)
    k_sdensity(SPlanes pl, const double* __restrict__ gx, const double* __restrict__ gy,
               const double* __restrict__ gz, const int64_t* __restrict__ tso, const int* __restrict__ listed,
               int64_t t0, int64_t s0, const int* __restrict__ slot_fn, const double* __restrict__ P, int64_t ldc,
               bool tri, double* __restrict__ grx, double* __restrict__ gry, double* __restrict__ grz,
               double* __restrict__ X = nullptr, int nop = 0, int nocc = 0, const double* __restrict__ occ = nullptr) {
  extern __shared__ double smem[];
  constexpr int E = kDK * kDLd;  // one operand of a stage
  static_assert(kSBlk * kXLd <= 2 * kDStages * E, "the X block lies in the stages");
  double* sA = smem;
  double* sB = smem + kDStages * E;
  double* sX = smem;
  int* sfn = reinterpret_cast<int*>(smem + 2 * kDStages * E);
  const double* __restrict__ phi = pl.phi(blockIdx.z);
  const int tid = threadIdx.x, lane = tid & 31, warp = ((tid >> 5) + blockIdx.x) & 3;
  const int64_t t = t0 + blockIdx.x;
  const int64_t sb = tso[t] - s0;
  const int nl = listed[t];
  const int m0 = blockIdx.y * kSBlk;
  load_sfn(sfn, slot_fn + sb, (int)(tso[t + 1] - tso[t]));
  const double* A = phi + (FORM == kFromPsi ? (int64_t)blockIdx.x * nop : sb) * 128 + m0;
  const int nk = FORM == kFromPsi ? nop : nl, nn = FORM == kPsi ? nop : nl;  // rows summed over, columns
  const int wm0 = (warp >> 1) * 32, wn0 = (warp & 1) * 32, fr = lane >> 2, fk = lane & 3;
  const int nslab = (nk + kDK - 1) / kDK;
  const int col = tid & 63, kq = tid >> 6;  // this thread's column of every gathered stage, rows kq + 2 i
  double r = 0.0, g[3] = {0.0, 0.0, 0.0};   // of point m0 + (tid & 63), columns tid >> 6 mod 2
  for (int n0 = 0; n0 < nn; n0 += kSBlk) {
    const int ns = tri ? min(nslab, n0 / kDK + kSBlk / kDK) : nslab;
    __syncthreads();  // sfn written; the X block before this one read
    const int fcol = FORM != kPsi ? sfn[n0 + col] : (n0 + col < nop ? n0 + col : -1);
    auto load = [&](int it) {
      double* a = sA + it % kDStages * E;
      double* b = sB + it % kDStages * E;
      const int k0 = it * kDK;
#pragma unroll
      for (int i = 0; i < kDK / 4; ++i) {
        const int c = tid + i * kSThreads, k = c >> 5, mn = (c & 31) * 2;
        cp_async16(a + k * kDLd + mn, A + (int64_t)(k0 + k) * 128 + mn);
      }
#pragma unroll
      for (int i = 0; i < kDK / 2; ++i) {
        const int k = kq + 2 * i, f = FORM == kFromPsi ? k0 + k : sfn[k0 + k];  // (nop: whole stages)
        const bool ok = f >= 0 && fcol >= 0;
        cp_async8(b + k * kDLd + col, ok ? P + (int64_t)f * ldc + fcol : P, ok);
      }
    };
#pragma unroll
    for (int s = 0; s < kDStages - 1; ++s) {
      if (s < ns) load(s);
      cp_async_commit();
    }
    const int nj = live_frags(n0 + wn0, nn, 4);
    SAcc<4, 4> acc;
    acc.zero();
    for (int it = 0; it < ns; ++it) {
      cp_async_wait<kDStages - 2>();
      __syncthreads();
      if (it + kDStages - 1 < ns) load(it + kDStages - 1);
      cp_async_commit();
      if (tri && it * kDK == n0) {  // the blocks before this one count twice
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc.v[i][j][0] *= 2.0;
            acc.v[i][j][1] *= 2.0;
          }
      }
      const double* a_s = sA + it % kDStages * E + wm0 + fr + fk * kDLd;
      const double* b_s = sB + it % kDStages * E + wn0 + fr + fk * kDLd;
      s_mma<kDK>(acc, [&](int i, int kk) { return a_s[i * 8 + kk * kDLd]; },
                 [&](int j, int kk) { return b_s[j * 8 + kk * kDLd]; }, 4, nj);
    }
    cp_async_wait<0>();
    __syncthreads();  // the stages are read: X takes their place
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          sX[(wn0 + j * 8 + 2 * fk + e) * kXLd + wm0 + i * 8 + fr] = acc.v[i][j][e];
    __syncthreads();
    const int cn = min(kSBlk, nn - n0);
    const int64_t o0 = ((FORM == kPsi ? (int64_t)blockIdx.x * nop : sb) + n0) * 128 + m0 + col;
#pragma unroll 8
    for (int c = kq; c < cn; c += 2) {
      const double x = sX[c * kXLd + col];
      const int64_t o = o0 + c * 128;
      if (STORE) X[o] = x;
      if (FORM == kPsi) {
        if (n0 + c < nocc) {
          const double y = occ[n0 + c] * x;
          r += y * x;
          if (GGA) g[0] += y * X[o];
        }
      } else if (FORM == kFromP) {
        r += x * phi[o];
      }
      if (GGA && FORM != kPsi) {
        g[0] += x * gx[o];
        g[1] += x * gy[o];
        g[2] += x * gz[o];
      }
    }
  }
  __syncthreads();
  double* red = smem;  // [4 quantities][2 column groups][64 points]
  red[tid] = r;
  if (GGA && FORM == kPsi) {
    red[kSThreads + tid] = g[0];
  } else if (GGA) {
#pragma unroll
    for (int q = 0; q < 3; ++q) red[(q + 1) * kSThreads + tid] = g[q];
  }
  __syncthreads();
  for (int q = kq; q < (GGA ? (FORM == kPsi ? 2 : 4) : 1); q += 2) {
    if (FORM == kFromPsi && q == 0) continue;
    const double v = red[q * kSThreads + col] + red[q * kSThreads + 64 + col];
    const int d = FORM == kPsi ? (int)blockIdx.z : q - 1;  // direction of grad rho
    double* out = q == 0 ? pl.rho(blockIdx.z) : (d == 0 ? grx : (d == 1 ? gry : grz));
    out[(int64_t)blockIdx.x * 128 + m0 + col] = q == 0 ? v : 2.0 * v;
  }
}
constexpr int sdensity_smem(int max_n) {
  return 2 * kDStages * kDK * kDLd * 8 + 4 * sfn_len(max_n);
}

// K4 (screened): H[fn_i][fn_j] += sum_p Z[i][p] phi[j][p] for the slots i, j of
// one tile, Z = A phi (+ B . grad phi).  CTA = (tile, 32 slots i): it forms its
// rows of Z in shared memory once (the whole K = 128 points) and streams the
// tile's phi against them, each warp its own blocks of 32 slots j through stages
// of its own: no barrier after Z.  A tile's CTAs follow one another in the grid,
// so that its phi comes from L2.  A separate pass that wrote Z
// for the contraction to read took 2.4 ms of the 60-atom build's 25.
// kFull: the whole square (GGA: V = H + H^T in k_spack).  kUpper: fn_i <= fn_j
// only (LDA: H is symmetric).  kTwice: the upper triangle with the off-diagonal
// elements doubled: the symmetric tau term of a meta-GGA, which k_spack's H + H^T
// then counts as the whole square does; grid z selects its plane.
// 60 atoms, 304 of 690 functions per tile: 11.1 -> 8.4 ms with the Z pass (8.7
// the contraction alone, a third of it on padding).
enum { kFull, kUpper, kTwice };
template <int MODE, bool GRAD>
__global__ void __launch_bounds__(kSThreads, 3)
    k_svpot(SPlanes pl, const double* __restrict__ gx, const double* __restrict__ gy, const double* __restrict__ gz,
            const double* __restrict__ A, const double* __restrict__ Bx, const double* __restrict__ By,
            const double* __restrict__ Bz, const int64_t* __restrict__ tso, const int* __restrict__ listed, int64_t t0,
            int64_t s0, const int* __restrict__ slot_fn, double* __restrict__ V, int64_t ldv, unsigned nI) {
  extern __shared__ double smem[];
  constexpr int E = OpTile<true, kRows>::kElems;
  const unsigned tile = blockIdx.x / nI;
  const int64_t t = t0 + tile;
  const int nl = listed[t], I0 = (int)(blockIdx.x - tile * nI) * kRows;
  if (I0 >= nl) return;
  double* sZ = smem;
  int* sfn = reinterpret_cast<int*>(smem + kRows * kZLd + 4 * kSStages * E);
  const double* __restrict__ phi = pl.phi(blockIdx.z);
  const int tid = threadIdx.x, lane = tid & 31, warp = ((tid >> 5) + tile) & 3;
  const int64_t sb = tso[t] - s0;
  const double* F = phi + sb * 128;
  // The warp's run: blocks of 32 slots j (every fourth of the tile's), 8 stages
  // of 16 points each, streamed through stages of its own.
  double* sF = smem + kRows * kZLd + warp * (kSStages * E);
  int lj = (MODE == kFull ? 0 : I0) + warp * kRows, lk = 0;  // the next stage to load
  auto load = [&]() {
    if (lj < nl) {
      const double* src = F + (int64_t)(lj + (lane >> 3)) * 128 + lk * kBK + (lane & 7) * 2;
      double* dst = sF + (lk & 1) * E + OpTile<true, kRows>::idx(lane >> 3, (lane & 7) * 2);
#pragma unroll
      for (int i = 0; i < 8; ++i) cp_async16(dst + 4 * i * (kBK + kPadK), src + 4 * i * 128);
    }
    cp_async_commit();
    if (++lk == 128 / kBK) {
      lk = 0;
      lj += 4 * kRows;
    }
  };
  load();
  load_sfn(sfn, slot_fn + sb, (int)(tso[t + 1] - tso[t]));
  {
    const int64_t pt = (int64_t)tile * 128 + tid;  // thread = point
    const double a = A[pt];
    double b[3] = {0.0, 0.0, 0.0};
    if (GRAD) {
      b[0] = Bx[pt];
      b[1] = By[pt];
      b[2] = Bz[pt];
    }
#pragma unroll(GRAD ? 8 : 16)  // (16 with gradients: 8.35 -> 8.6 ms; without, 20 atoms meta-GGA 1.03 -> 1.00)
    for (int i = 0; i < kRows; ++i) {  // rows past the listed functions are the tile's zero padding
      const int64_t o = (sb + I0 + i) * 128 + tid;
      double z = a * phi[o];
      if (GRAD) z += b[0] * gx[o] + b[1] * gy[o] + b[2] * gz[o];
      sZ[i * kZLd + tid] = z;
    }
  }
  __syncthreads();  // Z and sfn; the warps run on their own from here
  const int fr = lane >> 2, fk = lane & 3;
  const int nj = live_frags(I0, nl, 4);
  // rows of the fragments are slots j, so that a warp's atomics run along rows of V
  for (int j0 = (MODE == kFull ? 0 : I0) + warp * kRows; j0 < nl; j0 += 4 * kRows) {
    const int mi = live_frags(j0, nl, 4);
    SAcc<4, 4> acc;
    acc.zero();
#pragma unroll 2
    for (int it = 0; it < 128 / kBK; ++it) {
      cp_async_wait<0>();
      __syncwarp();
      load();  // into the stage read before this one
      const double* f_s = sF + (it & 1) * E + fr * (kBK + kPadK) + fk;
      const double* z_s = sZ + fr * kZLd + it * kBK + fk;
      s_mma<kBK>(acc, [&](int i, int kk) { return f_s[i * 8 * (kBK + kPadK) + kk]; },
            [&](int j, int kk) { return z_s[j * 8 * kZLd + kk]; }, mi, nj);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i >= mi) break;
      const int fj = sfn[j0 + i * 8 + fr];  // -1 past the listed functions
      if (fj < 0) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c >= nj) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int fi = sfn[I0 + c * 8 + 2 * fk + e];
          if (fi < 0) continue;
          double v = acc.v[i][c][e];
          if (MODE == kTwice && fj != fi) v *= 2.0;
          if (MODE == kFull || fj >= fi) atomicAdd(V + (int64_t)fi * ldv + fj, v);
        }
      }
    }
  }
}
constexpr int svpot_smem(int max_n) {
  return (kRows * kZLd + 4 * kSStages * OpTile<true, kRows>::kElems) * 8 + 4 * sfn_len(max_n);
}

}  // namespace

// ham[spin + ispin*(j(j+1)/2 + k)] = H(k, j), k <= j; GGA: H(k, j) + H(j, k)
// (exc_nel not null: and {E_xc, N_el} from acc).  failed not null and not 0: a
// wait of the build ran out, and the caller's outputs keep what they hold.
__global__ void k_spack(const double* __restrict__ V, int64_t nbas, bool sym2, int ispin, int spin,
                        double* __restrict__ ham, const double* __restrict__ acc, double* __restrict__ exc_nel,
                        const int* __restrict__ failed) {
  if (failed && *failed) return;
  const int64_t len = nbas * (nbas + 1) / 2;
  if (exc_nel && blockIdx.x == 0 && threadIdx.x < 2) exc_nel[threadIdx.x] = acc[2 * threadIdx.x];
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < len;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t j = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > idx) --j;
    while ((j + 1) * (j + 2) / 2 <= idx) ++j;
    const int64_t k = idx - j * (j + 1) / 2;
    double v = V[k * nbas + j];
    if (sym2) v += V[j * nbas + k];
    ham[spin + (int64_t)ispin * idx] = v;
  }
}

// ---------------------------------------------------------------------------
// host planning
// ---------------------------------------------------------------------------
namespace {

// Squared radius beyond which radial function rr of shell S is dropped.
double listing_r2(const DevShell& S, int rr, const double* exps, const double* norms, const double* contr,
                  double threshold, double sa_fac) {
  std::vector<double> cf((size_t)S.nexp, 0.0);
  if (rr < S.nunc) cf[(size_t)rr] = 1.0;
  else
    for (int e = 0; e < S.nexp; ++e) cf[(size_t)e] = contr[S.con_off + e + (int64_t)S.nexp * (rr - S.nunc)];
  double amin = 1e300;
  for (int e = 0; e < S.nexp; ++e)
    if (cf[(size_t)e] != 0.0) amin = std::min(amin, exps[S.exp_off + e]);
  if (amin == 1e300) return 0.0;  // identically zero function
  // every primitive vanishes where alpha_min r^2 >= 50; margin for rounding
  const double r2cut = 50.0 / amin * (1.0 + 1e-9);
  if (threshold <= 0.0) return r2cut;
  // bound on |phi| and |grad phi| at distance r:
  //   sum_e |c_e| N_e exp(-a_e r^2) (r^l + 2 a_e r^(l+1) + (2l+1) r^(l-1)) * sa_fac
  const int l = S.l;
  auto bound = [&](double r) {
    double b = 0.0;
    for (int e = 0; e < S.nexp; ++e) {
      if (cf[(size_t)e] == 0.0) continue;
      const double a = exps[S.exp_off + e];
      if (a * r * r >= 50.0) continue;
      const double g = std::fabs(cf[(size_t)e]) * norms[S.exp_off + e] * std::exp(-a * r * r);
      double poly = std::pow(r, l) + 2.0 * a * std::pow(r, l + 1);
      if (l > 0) poly += (2 * l + 1) * std::pow(r, l - 1);
      b += g * poly;
    }
    return b * sa_fac;
  };
  const double rcut = std::sqrt(r2cut);
  const int nstep = 4000;
  const double dr = rcut / nstep;
  // every term exp(-a r^2) r^k, k <= l + 1, falls for r >= sqrt((l + 1) / (2 a)): from the smallest
  // exponent's radius on the bound falls, and its last step at or above the threshold is found by halving
  int hi = std::min(nstep, (int)std::ceil(std::sqrt((l + 1) / (2.0 * amin)) / dr));
  if (bound(hi * dr) >= threshold) {
    int lo = hi;
    hi = nstep + 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      (bound(mid * dr) >= threshold ? lo : hi) = mid;
    }
    const double R = std::min(rcut, lo * dr + dr);
    return R * R;
  }
  for (int i = hi - 1; i >= 0; --i) {
    const double r = i * dr;
    if (bound(r) >= threshold) {
      const double R = std::min(rcut, r + dr);
      return R * R;
    }
  }
  return 0.0;
}

}  // namespace

void screen_listing_radii(const std::vector<DevShell>& shells, const double* exps, const double* norms,
                          const double* contr, double threshold, const DevSA& sa, std::vector<double>& R2,
                          std::vector<int>& r2off) {
  double sa_fac[kMaxL + 1];
  for (int l = 0; l <= kMaxL; ++l) {
    sa_fac[l] = 1.0;
    if (!sa.identity)
      for (int i = 0; i < 2 * l + 1; ++i) {
        double s = 0.0;
        for (int m = 0; m < 2 * l + 1; ++m) s += std::fabs(sa.c[l][i][m]);
        sa_fac[l] = std::max(sa_fac[l], s);
      }
  }
  for (const DevShell& S : shells) {
    r2off.push_back((int)R2.size());
    for (int rr = 0; rr < S.nrad; ++rr) R2.push_back(listing_r2(S, rr, exps, norms, contr, threshold, sa_fac[S.l]));
  }
}

constexpr int64_t kSortFrom = int64_t(1) << 17;  // points

// The tiles and the lengths of their lists: Morton-ordered points, per tile the
// number of listed functions (those whose listing radius exceeds the tile's
// distance to their atom) and of basis items, and so their places.  The tables that
// fill_lists reads stay in sp->tab.
// A build's plan (gradient false) keeps its points in Morton order.  A gradient's
// takes those of `from`, a plan of the same grid; without one its points go into
// the gradient's scratch (grad_plan_hosts), in Morton order from kSortFrom on: a
// grid of few points is that of few atoms, whose functions reach most of its
// points in any order, and the sort would be most of a first call (dense layout,
// 6 atoms: 1.0 ms before there was a plan, 2.1 with the sort, 0.95 without;
// 12 atoms 2.5, 3.4 and 1.7, a repeated call 1.09 with it and 1.18 without).
// A gradient's own arrays lie behind its tables (an allocation of 2 MB or more takes
// 0.35 ms whatever its size: the gradient of 6 atoms 1.03 ms before it had a plan, 1.6
// with eight allocations of the plan's, 0.92 now).  On the host the lists of a 41-atom
// grid (2,710 tiles, 170,000 items of 80 bytes, copied from pageable memory) were most
// of the 30 ms of a context's creation.
static int count_lists(ScreenPlan* sp, const BuildArgs& a, int natm, int64_t npts, const std::vector<DevShell>& shells,
                       const std::vector<double>& R2, const std::vector<int>& r2off, const ScreenPlan* from, bool gradient,
                       cudaStream_t st, std::string& err) {
#define BL_TRY(call, what)                                                       \
  do {                                                                           \
    cudaError_t e_ = (call);                                                     \
    if (e_ != cudaSuccess) {                                                     \
      err = std::string(what) + ": " + cudaGetErrorString(e_);                   \
      return e_ == cudaErrorMemoryAllocation ? PGXC_ENOMEM : PGXC_ECUDA;         \
    }                                                                            \
  } while (0)
  constexpr int kCnt = 2 + kMaxL;
  const int64_t ntiles = (npts + 127) / 128, nq = ntiles * 128;
  ListTables& T = sp->tab;
  sp->ntiles = ntiles;
  T.natm = natm;
  T.nsh = (int)shells.size();
  const double *px = a.px, *py = a.py, *pz = a.pz;
  int64_t n = npts;
  const int64_t* order = nullptr;
  if (from) {
    sp->order_of_points = from->order_of_points;
    px = sp->qx = from->qx;
    py = sp->qy = from->qy;
    pz = sp->qz = from->qz;
    sp->qw = from->qw;
    n = nq;
  } else if (!gradient || npts >= kSortFrom) {  // Morton order of the points, on the device (ties by point index)
    BL_TRY(sp_alloc(sp, &sp->order_of_points, (size_t)nq), "cudaMalloc");
    BL_TRY(morton_perm_device(a.px, a.py, a.pz, npts, nq, sp->order_of_points, st), "grid reordering");
    order = sp->order_of_points;
  }
  if (!gradient) {
    BL_TRY(sp_alloc(sp, &sp->qx, 4 * (size_t)nq), "grid reordering");
    sp->qy = sp->qx + nq;
    sp->qz = sp->qx + 2 * nq;
    sp->qw = sp->qx + 3 * nq;
    k_gather_points<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(order, npts, nq, a.px, a.py, a.pz, a.w, sp->qx, sp->qy,
                                                                 sp->qz, sp->qw);
    BL_TRY(cudaGetLastError(), "grid reordering");
  }
  // one allocation for the tables (and a gradient's tso and listed)
  const size_t nstart = (size_t)ntiles * (kMaxL + 1), n8 = nstart + (size_t)ntiles + 1 + std::max<size_t>(R2.size(), 1);
  const size_t n4 = (size_t)ntiles * natm + (size_t)ntiles * kCnt + shells.size() + (size_t)ntiles;
  BL_TRY(cudaMalloc(&T.base, 8 * n8 + 4 * n4), "tile lists");
  T.start = (int64_t*)T.base;
  sp->tso = T.start + nstart;
  T.r2 = (double*)(sp->tso + ntiles + 1);
  T.d2 = (float*)(T.start + n8);
  T.cnt = (int*)(T.d2 + (size_t)ntiles * natm);
  T.r2off = T.cnt + (size_t)ntiles * kCnt;
  sp->listed = T.r2off + shells.size();
  BL_TRY(cudaMemcpyAsync(T.r2, R2.data(), sizeof(double) * R2.size(), cudaMemcpyHostToDevice, st), "tile lists");
  BL_TRY(cudaMemcpyAsync(T.r2off, r2off.data(), sizeof(int) * r2off.size(), cudaMemcpyHostToDevice, st), "tile lists");
  k_tile_atom_d2<<<(unsigned)ntiles, 128, 0, st>>>(order, n, px, py, pz, a.atoms, natm, T.d2);
  k_plan_count<<<(unsigned)ntiles, 128, 0, st>>>(T.d2, natm, a.shells, T.nsh, T.r2, T.r2off, T.cnt);
  BL_TRY(cudaGetLastError(), "tile lists");
  std::vector<int> cnt((size_t)ntiles * kCnt), listed((size_t)ntiles);
  std::vector<int64_t> start((size_t)ntiles * (kMaxL + 1));
  BL_TRY(cudaMemcpyAsync(cnt.data(), T.cnt, sizeof(int) * cnt.size(), cudaMemcpyDeviceToHost, st), "tile lists");
  BL_TRY(cudaStreamSynchronize(st), "tile lists");
  std::vector<int64_t>& tso = sp->h_tso;
  tso.assign((size_t)ntiles + 1, 0);
  int64_t items[kMaxL + 1] = {};
  for (int l = 0; l <= kMaxL; ++l) sp->tile_item[l].assign((size_t)ntiles + 1, 0);
  for (int64_t t = 0; t < ntiles; ++t) {
    const int* c = &cnt[(size_t)t * kCnt];
    listed[(size_t)t] = c[0];
    const int nt = (c[0] + kSlotAlign - 1) / kSlotAlign * kSlotAlign;
    sp->nlisted += c[0];
    sp->sum_n2 += (double)c[0] * (double)c[0];
    sp->max_n = std::max(sp->max_n, nt);
    tso[(size_t)t + 1] = tso[(size_t)t] + nt;
    for (int l = 0; l <= kMaxL; ++l) {
      start[(size_t)t * (kMaxL + 1) + l] = items[l];
      items[l] += c[1 + l];
      sp->tile_item[l][(size_t)t + 1] = items[l];
    }
  }
  sp->nslots = tso[(size_t)ntiles];
  if (!gradient) {
    BL_TRY(sp_alloc(sp, &sp->tso, tso.size()), "tile lists");
    BL_TRY(sp_alloc(sp, &sp->listed, listed.size()), "tile lists");
  }
  BL_TRY(cudaMemcpyAsync(sp->tso, tso.data(), sizeof(int64_t) * tso.size(), cudaMemcpyHostToDevice, st), "tile lists");
  BL_TRY(cudaMemcpyAsync(sp->listed, listed.data(), sizeof(int) * listed.size(), cudaMemcpyHostToDevice, st),
         "tile lists");
  BL_TRY(cudaMemcpyAsync(T.start, start.data(), sizeof(int64_t) * start.size(), cudaMemcpyHostToDevice, st),
         "tile lists");
  return PGXC_OK;
#undef BL_TRY
}

// The lists of tiles [t0, t0 + nt) at the places counted for them.
static void fill_lists(const ScreenPlan* sp, const BuildArgs& a, int64_t t0, int64_t nt, const TileLists& out,
                       cudaStream_t st) {
  const ListTables& T = sp->tab;
  k_plan_fill<<<(unsigned)nt, 128, 0, st>>>(T.d2, T.natm, a.atoms, a.shells, T.nsh, T.r2, T.r2off, sp->tso, T.start, t0,
                                            out);
}

void screen_destroy(ScreenPlan* sp) {
  if (!sp) return;
  if (sp->mixed) screen_mixed_destroy(sp->mixed);
  for (void* p : sp->allocs) cudaFree(p);
  if (sp->tab.base) cudaFree(sp->tab.base);
  if (sp->psi_own) cudaFree(sp->psi_own);
  for (auto& c : sp->cev)
    for (auto& e : c)
      if (e) cudaEventDestroy(e);
  delete sp;
}

void screen_stats(const ScreenPlan* sp, int64_t* ntiles, int64_t* nslots, int64_t* nlisted, double* sum_n2,
                  int64_t* nchunks) {
  if (ntiles) *ntiles = sp->ntiles;
  if (nslots) *nslots = sp->nslots;
  if (nlisted) *nlisted = sp->nlisted;
  if (sum_n2) *sum_n2 = sp->sum_n2;
  if (nchunks) *nchunks = (int64_t)sp->chunk_t0.size() - 1;
}

#define SP_TRY(call, what)                                                       \
  do {                                                                           \
    cudaError_t e_ = (call);                                                     \
    if (e_ != cudaSuccess) {                                                     \
      err = std::string(what) + ": " + cudaGetErrorString(e_);                   \
      screen_destroy(sp);                                                        \
      return e_ == cudaErrorMemoryAllocation ? PGXC_ENOMEM : PGXC_ECUDA;         \
    }                                                                            \
  } while (0)

// Even tile lists of every chunk [t0[c], t0[c + 1]) (screen_mixed_order) on the device.
template <typename Alloc>
static cudaError_t make_order(const int64_t* tso, const std::vector<int64_t>& t0, int nsm, std::vector<char>& used,
                              Alloc alloc, int** order, int** start) {
  const size_t nch = t0.size() - 1;
  std::vector<int> ho((size_t)t0.back()), hs(nch * (size_t)(nsm + 1));
  used.assign(nch, 0);
  bool any = false;
  for (size_t c = 0; c < nch; ++c) {
    used[c] = screen_mixed_order(tso + t0[c], t0[c + 1] - t0[c], nsm, ho.data() + t0[c], hs.data() + c * (nsm + 1));
    any = any || used[c];
  }
  if (!any) return cudaSuccess;
  cudaError_t e = alloc(order, ho.size());
  if (e == cudaSuccess) e = alloc(start, hs.size());
  if (e == cudaSuccess) e = cudaMemcpy(*order, ho.data(), sizeof(int) * ho.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(*start, hs.data(), sizeof(int) * hs.size(), cudaMemcpyHostToDevice);
  return e;
}

int screen_create(ScreenPlan** out, const ScreenInput& in, const BuildArgs& a, cudaStream_t st, std::string& err) {
  *out = nullptr;
  ScreenPlan* sp = new ScreenPlan();
  sp->gga = in.gga;
  sp->mgga = in.mgga;
  sp->functional = in.functional;
  // The INT8 build keeps grad phi in FP32 (phi stays FP64): its density
  // gradient and potential then move 12 fewer bytes per basis value, within
  // the mixed-mode bars (measured on CH60-PBE: |dE_xc| 9.7e-8 Eh, max |dV_xc|
  // 3.1e-8 against the FP64 build; FP32 phi too would give 1.1e-6 Eh).  The
  // meta-GGA tau contractions run on the FP64 kernels and keep FP64 gradients.
  sp->gf32 = in.precision != PGXC_PREC_FP64 && in.gga && !in.mgga;
  sp->ispin = in.ispin;
  sp->nbas = in.nbas;
  sp->keep = in.keep_basis;
  const std::vector<DevShell>& shells = *in.shells;
  for (const DevShell& S : shells) {
    sp->n_exps = std::max<int64_t>(sp->n_exps, S.exp_off + S.nexp);
    sp->n_contr = std::max<int64_t>(sp->n_contr, S.con_off + (int64_t)S.nexp * S.ncontr);
    if (S.seg) sp->n_rng = std::max<int64_t>(sp->n_rng, S.rad_off + S.ncontr);
  }
  for (const DevShell& S : shells)
    if (S.nrad > 64) {
      err = "screened build: a shell has more than 64 radial functions";
      screen_destroy(sp);
      return PGXC_ENOTSUP;
    }
  {
    int dev = 0;
    SP_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    SP_TRY(cudaDeviceGetAttribute(&sp->nsm, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
  }
  // --- tiles and lists ----------------------------------------------------
  {
    std::vector<double> R2;
    std::vector<int> r2off;
    screen_listing_radii(shells, in.exps, in.norms, in.contr, in.threshold, a.sa, R2, r2off);
    if (const int st2 = count_lists(sp, a, in.natm, in.npts, shells, R2, r2off, nullptr, false, st, err)) {
      screen_destroy(sp);
      return st2;
    }
    TileLists L{};
    SP_TRY(sp_alloc(sp, &sp->slot_fn, (size_t)sp->nslots), "tile lists");
    L.slot_fn = sp->slot_fn;
    for (int l = 0; l <= kMaxL; ++l) {
      SP_TRY(sp_alloc(sp, &sp->items[l], (size_t)sp->tile_item[l].back()), "tile lists");
      L.items[l] = sp->items[l];
    }
    fill_lists(sp, a, 0, sp->ntiles, L, st);
    SP_TRY(cudaGetLastError(), "tile lists");
    SP_TRY(cudaStreamSynchronize(st), "tile lists");
    cudaFree(sp->tab.base);  // (a build's lists are filled once)
    sp->tab = ListTables{};
  }
  const std::vector<int64_t>& tso = sp->h_tso;
  const int64_t ntiles = sp->ntiles;
  // --- chunks -------------------------------------------------------------------
  const bool mixed = in.precision != PGXC_PREC_FP64;
  size_t freeb = 0, totb = 0;
  SP_TRY(cudaMemGetInfo(&freeb, &totb), "cudaMemGetInfo");
  if (sp->keep) {
    // resident basis values and point digits of every slot: phi (+ grad phi), INT8 digits
    const double gb = in.gga ? 3.0 * (sp->gf32 ? 4.0 : 8.0) : 0.0;
    const double need = (double)(sp->nslots + kSlack) * 128 * (8.0 + gb + (mixed ? 5.0 : 0.0));
    if (need > 0.6 * (double)freeb) {
      err = "screened build: the basis values of the whole grid (" + std::to_string((int64_t)(need / 1e9)) +
            " GB) do not fit beside the build's buffers; create the context without keep_orbitals";
      screen_destroy(sp);
      return PGXC_ENOMEM;
    }
    freeb -= (size_t)need;
  }
  const int64_t per_slot = 128 * (8 + (in.gga ? 3 * (sp->gf32 ? 4 : 8) : 0)) + (mixed ? screen_mixed_bytes_per_slot() : 0);
  const int64_t per_tile = 128 * 8 * 8 * in.ispin + (mixed ? screen_mixed_bytes_per_tile() : 0);
  int64_t budget_slots = (int64_t)(0.45 * (double)freeb) / per_slot;
  budget_slots = std::max<int64_t>(budget_slots, sp->max_n);
  int64_t budget_tiles = std::max<int64_t>(1, (int64_t)(0.05 * (double)freeb) / per_tile);
  if (in.max_chunk_points > 0) budget_tiles = std::min(budget_tiles, std::max<int64_t>(1, in.max_chunk_points / 128));
  budget_tiles = std::min<int64_t>(budget_tiles, 1 << 16);
  // INT8 path: the gathered density B operand, per tile
  std::vector<int64_t> boff((size_t)ntiles + 1, 0);
  if (mixed)
    for (int64_t t = 0; t < ntiles; ++t)
      boff[(size_t)t + 1] = boff[(size_t)t] + screen_mixed_bstages(tso[(size_t)t + 1] - tso[(size_t)t]);
  const int64_t budget_bstages =
      mixed ? std::max<int64_t>((int64_t)(0.25 * (double)freeb) / screen_mixed_bytes_per_bstage(),
                                screen_mixed_bstages(sp->max_n))
            : INT64_MAX;
  sp->chunk_t0.push_back(0);
  {
    int64_t t0 = 0;
    for (int64_t t = 0; t < ntiles; ++t) {
      const bool full_slots = tso[(size_t)t + 1] - tso[(size_t)t0] > budget_slots;
      const bool full_tiles = t - t0 + 1 > budget_tiles;
      const bool full_b = boff[(size_t)t + 1] - boff[(size_t)t0] > budget_bstages;
      if (t > t0 && (full_slots || full_tiles || full_b)) {
        sp->chunk_t0.push_back(t);
        t0 = t;
      }
    }
    sp->chunk_t0.push_back(ntiles);
  }
  int64_t chunk_bstages = 0;
  const size_t nch = sp->chunk_t0.size() - 1;
  for (size_t c = 0; c < nch; ++c) {
    const int64_t t0 = sp->chunk_t0[c], t1 = sp->chunk_t0[c + 1];
    sp->chunk_tiles = std::max(sp->chunk_tiles, t1 - t0);
    sp->chunk_slots = std::max(sp->chunk_slots, tso[(size_t)t1] - tso[(size_t)t0]);
    chunk_bstages = std::max(chunk_bstages, boff[(size_t)t1] - boff[(size_t)t0]);
  }
  for (int l = 0; l <= kMaxL; ++l)
    for (size_t c = 0; c <= nch; ++c) sp->item_off[l].push_back(sp->tile_item[l][(size_t)sp->chunk_t0[c]]);
  // --- buffers ------------------------------------------------------------------
  const size_t rows = (size_t)(sp->chunk_slots + kSlack) * 128;
  // basis arrays: one chunk's rows, or every slot of the grid when they stay resident
  const size_t brows = sp->keep ? (size_t)(sp->nslots + kSlack) * 128 : rows;
  // psi of the orbital form lies behind phi where it is small, for the longest that the form is taken for, so that
  // the first build does not allocate (12 atoms, first build 0.98 ms with an allocation of its own, 0.61 without).
  // A large one is made by the first build that takes the form (screen_orbital_form): the caller's P, symmetric
  // builds, energies and batches never do, and would hold up to 1 GB for nothing.
  int64_t psi = 0;
  if (in.gga && !mixed && sp->nlisted > 0) {
    const int64_t most = (int64_t)(sp->sum_n2 / (2.0 * kOrbitalMargin * (double)sp->nlisted));
    psi = sp->chunk_tiles * most * 128;
    if (psi > kPsiReserved || 8.0 * (double)psi > 0.1 * (double)freeb) psi = 0;
  }
  // one allocation for phi, psi and grad phi (an allocation takes 0.35 ms, whatever its size; 41 atoms, create,
  // weights, first build and destroy: 22.2 ms with four and psi behind phi, 22.0 with one and psi in the build)
  {
    const size_t gb = in.gga ? (sp->gf32 ? sizeof(float) : sizeof(double)) : 0;
    auto planes = [&] { return sp_alloc(sp, (char**)&sp->phi, sizeof(double) * (brows + (size_t)psi) + 3 * gb * brows); };
    cudaError_t e = planes();
    if (e != cudaSuccess && psi) {
      cudaGetLastError();
      psi = 0;
      e = planes();
    }
    SP_TRY(e, "cudaMalloc (phi, grad phi)");
    if (psi) {
      sp->psi = sp->phi + brows;
      sp->psi_cap = psi;
    }
    // (padding slots are zeroed by every evaluation; the rows after the last slot are read by whole-block copies)
    auto slack = [&](auto* p) { return cudaMemsetAsync(p + (brows - kSlack * 128), 0, sizeof(*p) * kSlack * 128, st); };
    auto place = [&](auto* g, auto** gx, auto** gy, auto** gz) -> cudaError_t {
      *gx = g;
      *gy = g + brows;
      *gz = g + 2 * brows;
      cudaError_t r = slack(*gx);
      if (r == cudaSuccess) r = slack(*gy);
      return r == cudaSuccess ? slack(*gz) : r;
    };
    double* g = sp->phi + brows + psi;
    SP_TRY(slack(sp->phi), "memset");
    if (in.gga && sp->gf32) SP_TRY(place((float*)g, &sp->fx, &sp->fy, &sp->fz), "memset");
    else if (in.gga) SP_TRY(place(g, &sp->gx, &sp->gy, &sp->gz), "memset");
  }
  const int64_t cp = sp->chunk_tiles * 128;
  SP_TRY(sp_alloc(sp, &sp->pt, 8 * (size_t)in.ispin * cp), "cudaMalloc");
  SP_TRY(cudaMemsetAsync(sp->pt, 0, sizeof(double) * 8 * in.ispin * cp, st), "memset");
  if (in.mgga) {
    SP_TRY(sp_alloc(sp, &sp->tq, 4 * (size_t)in.ispin * cp), "cudaMalloc");
    SP_TRY(cudaMemsetAsync(sp->tq, 0, sizeof(double) * 4 * in.ispin * cp, st), "memset");
  }
  const size_t npart = 2 * (size_t)((cp + 255) / 256);
  SP_TRY(sp_alloc(sp, &sp->partial, npart + 2), "cudaMalloc");
  SP_TRY(cudaMemsetAsync(sp->partial + npart, 0, sizeof(double) * 2, st), "memset");
  SP_TRY(sp_alloc(sp, &sp->V, (size_t)in.ispin * in.nbas * in.nbas), "cudaMalloc (V)");
  if (mixed) {
    ScreenMixedInput mi;
    mi.nbas = in.nbas;
    mi.ldc = a.ldc;
    mi.gga = in.gga;
    mi.nspin = in.ispin;
    mi.chunk_slots = sp->chunk_slots + kSlack;
    mi.chunk_tiles = sp->chunk_tiles;
    mi.max_n = sp->max_n;
    mi.chunk_bstages = chunk_bstages;
    if (sp->keep) {
      mi.resident_slots = sp->nslots + kSlack;
      mi.resident_tiles = sp->ntiles;
    }
    SP_TRY(sp_alloc(sp, &sp->pmax, (size_t)sp->chunk_tiles * 128), "cudaMalloc");
    SP_TRY(sp_alloc(sp, &sp->b_off, boff.size()), "cudaMalloc");
    SP_TRY(cudaMemcpy(sp->b_off, boff.data(), sizeof(int64_t) * boff.size(), cudaMemcpyHostToDevice), "copy");
    mi.b_off = sp->b_off;
    SP_TRY(make_order(tso.data(), sp->chunk_t0, sp->nsm, sp->ordered, [&](int** p, size_t k) { return sp_alloc(sp, p, k); },
                      &sp->order, &sp->order_start),
           "tile order");
    const int st2 = screen_mixed_create(&sp->mixed, mi, err);
    if (st2) {
      screen_destroy(sp);
      return st2;
    }
  }
  *out = sp;
  return PGXC_OK;
}

namespace {
// raw weight (0 for padding) and host atom of the plan's points
__global__ void k_gather_hosts(const int64_t* __restrict__ order, int64_t n, int64_t nq,
                               const double* __restrict__ wraw, const int* __restrict__ owner,
                               double* __restrict__ qwraw, int* __restrict__ qowner) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const int64_t i = point_index(order, n, q);
  qwraw[q] = i >= 0 ? wraw[i] : 0.0;
  qowner[q] = owner[i >= 0 ? i : point_index(order, n, q & ~(int64_t)127)];
}
}  // namespace

int grad_plan_create(ScreenPlan** out, const BuildArgs& a, int natm, int64_t npts, const std::vector<DevShell>& shells,
                     const std::vector<double>& R2, const std::vector<int>& r2off, const ScreenPlan* from,
                     int64_t max_rows, cudaStream_t st, std::string& err) {
  *out = nullptr;
  ScreenPlan* sp = new ScreenPlan();
  SP_TRY(cudaGetDevice(&sp->nsm), "cudaGetDevice");
  SP_TRY(cudaDeviceGetAttribute(&sp->nsm, cudaDevAttrMultiProcessorCount, sp->nsm), "cudaDeviceGetAttribute");
  if (const int st2 = count_lists(sp, a, natm, npts, shells, R2, r2off, from, true, st, err)) {
    screen_destroy(sp);
    return st2;
  }
  max_rows = std::max<int64_t>(max_rows, sp->max_n);
  sp->chunk_t0.push_back(0);
  for (int64_t t = 1; t <= sp->ntiles; ++t) {
    const int64_t t0 = sp->chunk_t0.back();
    if (t == sp->ntiles || sp->h_tso[(size_t)t + 1] - sp->h_tso[(size_t)t0] > max_rows) sp->chunk_t0.push_back(t);
  }
  for (size_t c = 0; c + 1 < sp->chunk_t0.size(); ++c) {
    const int64_t t0 = sp->chunk_t0[c], t1 = sp->chunk_t0[c + 1];
    sp->chunk_tiles = std::max(sp->chunk_tiles, t1 - t0);
    sp->chunk_slots = std::max(sp->chunk_slots, sp->h_tso[(size_t)t1] - sp->h_tso[(size_t)t0]);
    for (int l = 0; l <= kMaxL; ++l)
      sp->chunk_items[l] =
          std::max(sp->chunk_items[l], sp->tile_item[l][(size_t)t1] - sp->tile_item[l][(size_t)t0]);
  }
  *out = sp;
  return PGXC_OK;
}

void grad_plan_hosts(ScreenPlan* sp, const BuildArgs& a, int64_t npts, const double* wraw, const int* owner,
                     double* points, double* qwraw, int* qowner, cudaStream_t st) {
  sp->qwraw = qwraw;
  sp->qowner = qowner;
  const int64_t nq = sp->ntiles * 128;
  const unsigned nb = (unsigned)((nq + 255) / 256);
  if (points) {
    sp->qx = points;
    sp->qy = points + nq;
    sp->qz = points + 2 * nq;
    sp->qw = points + 3 * nq;
  }
  if (sp->filled >= 0) return;
  if (points)
    k_gather_points<<<nb, 256, 0, st>>>(sp->order_of_points, npts, nq, a.px, a.py, a.pz, a.w, sp->qx, sp->qy, sp->qz,
                                        sp->qw);
  k_gather_hosts<<<nb, 256, 0, st>>>(sp->order_of_points, npts, nq, wraw, owner, qwraw, qowner);
}

void grad_plan_lists(ScreenPlan* sp, const BuildArgs& a, size_t c, const TileLists& lists, cudaStream_t st) {
  if (sp->filled == (int64_t)c) return;
  const int64_t t0 = sp->chunk_t0[c];
  TileLists L = lists;
  L.s0 = sp->h_tso[(size_t)t0];
  for (int l = 0; l <= kMaxL; ++l) L.i0[l] = sp->tile_item[l][(size_t)t0];
  fill_lists(sp, a, t0, sp->chunk_t0[c + 1] - t0, L, st);
  sp->filled = (int64_t)c;
}

void grad_contract(const ScreenPlan* sp, const int* slot_fn, int64_t t0, int64_t nt, int64_t s0, const double* F, const double* gx,
                   const double* gy, const double* gz, const double* P, int64_t ldc, double* X, double* rho,
                   double* grx, double* gry, double* grz, const GradOrbitals* orb, cudaStream_t st) {
  const int smem = sdensity_smem(sp->max_n);
  if (orb) {
    raise_smem_limit(k_sdensity<false, true, kPsi>, smem);
    raise_smem_limit(k_sdensity<true, true, kFromPsi>, smem);
    raise_smem_limit(k_sdensity<false, true, kFromPsi>, smem);
    const int64_t parts = (nt + orb->psi_tiles - 1) / orb->psi_tiles, step = (nt + parts - 1) / parts;
    for (int64_t u = 0; u < nt; u += step) {
      const dim3 grid((unsigned)std::min(step, nt - u), 2);
      const int64_t p = u * 128;
      const SPlanes pu{F, F, F, rho + p, nullptr, nullptr}, px{orb->psi, nullptr, nullptr, nullptr, nullptr, nullptr};
      k_sdensity<false, true, kPsi><<<grid, kSThreads, smem, st>>>(
          pu, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0 + u, s0, slot_fn, orb->orb, orb->nop, false, nullptr,
          nullptr, nullptr, orb->psi, orb->nop, orb->nop, orb->occ);
      if (gx)
        k_sdensity<true, true, kFromPsi><<<grid, kSThreads, smem, st>>>(
            px, gx, gy, gz, sp->tso, sp->listed, t0 + u, s0, slot_fn, orb->scaled, ldc, false, grx + p, gry + p,
            grz + p, X, orb->nop, orb->nop, nullptr);
      else
        k_sdensity<false, true, kFromPsi><<<grid, kSThreads, smem, st>>>(
            px, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0 + u, s0, slot_fn, orb->scaled, ldc, false, nullptr,
            nullptr, nullptr, X, orb->nop, orb->nop, nullptr);
    }
    return;
  }
  const SPlanes pl{F, F, F, rho, rho, rho};
  const dim3 grid((unsigned)nt, 2);
  if (gx) {
    raise_smem_limit(k_sdensity<true, true>, smem);
    k_sdensity<true, true><<<grid, kSThreads, smem, st>>>(pl, gx, gy, gz, sp->tso, sp->listed, t0, s0, slot_fn, P,
                                                          ldc, false, grx, gry, grz, X);
  } else {
    raise_smem_limit(k_sdensity<false, true>, smem);
    k_sdensity<false, true><<<grid, kSThreads, smem, st>>>(pl, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0, s0,
                                                           slot_fn, P, ldc, false, nullptr, nullptr, nullptr, X);
  }
}

// The orbital form costs n (nop + nop) products per point where P costs n^2 (an
// LDA, and each tau plane: n nop against n^2 / 2), and forms no P.  60 atoms, 304
// functions per tile, 105 orbitals (2 nop / n = 0.74): contraction 8.7 -> 6.45 ms;
// 25 atoms open shell 0.955 -> 0.79, 20 atoms meta-GGA 1.007 -> 0.485, 12 atoms
// 0.155 -> 0.138.  Time over products is 1.04 of what P takes, so that with a
// margin of 1.15 the form chosen is the faster one; above it P stays (nocc near
// nbas, where the orbital form is up to twice the products).  INT8 keeps P, whose
// digits are what its products read.
bool orbital_form_pays(const ScreenPlan* sp, int64_t nop) {
  return kOrbitalMargin * 2.0 * (double)nop * (double)sp->nlisted < sp->sum_n2;
}
int64_t orbital_psi_tiles(const ScreenPlan* sp, int64_t nop) {
  const int64_t most = sp->psi_tiles_most > 0 ? std::min(sp->chunk_tiles, sp->psi_tiles_most) : sp->chunk_tiles;
  return std::min(most, std::max<int64_t>(1, kPsiMost / (nop * 128)));
}
bool screen_orbital_form(ScreenPlan* sp, int nop) {
  if (sp->mixed || !orbital_form_pays(sp, nop)) return false;
  if (!sp->gga) return true;
  const int64_t need = orbital_psi_tiles(sp, nop) * nop * 128;
  if (need <= sp->psi_cap) return true;
  // a buffer of its own (the builds before this one have ended); without room the builds take P, as long as they
  // would need as much
  if (need >= sp->psi_refused) return false;
  if (sp->psi_own) cudaFree(sp->psi_own);
  sp->psi_own = sp->psi = nullptr;
  sp->psi_cap = 0;
  if (cudaMalloc(&sp->psi_own, sizeof(double) * (size_t)need) != cudaSuccess) {
    cudaGetLastError();
    sp->psi_own = nullptr;
    sp->psi_refused = need;
    return false;
  }
  sp->psi = sp->psi_own;
  sp->psi_cap = need;
  return true;
}

// rho, grad rho and (tau not null) the tau sums of one spin by its orbitals
static int orbital_density(const ScreenPlan* sp, const BuildArgs& a, int s, int64_t t0, int64_t nt, int64_t s0,
                           const double* phi, const double* gx, const double* gy, const double* gz, const BuildArgs& b,
                           double* tau, int64_t cp, cudaStream_t st) {
  const int smem = sdensity_smem(sp->max_n), nop = a.nop, nocc = a.nocc;
  raise_smem_limit(k_sdensity<false, true, kPsi>, smem);
  raise_smem_limit(k_sdensity<false, false, kPsi>, smem);
  raise_smem_limit(k_sdensity<true, false, kPsi>, smem);
  raise_smem_limit(k_sdensity<true, false, kFromPsi>, smem);
  const SPlanes pl{phi, phi, phi, b.rho, b.rho, b.rho};
  int launches = 0;
  if (!gx) {
    k_sdensity<false, false, kPsi><<<dim3((unsigned)nt, 2), kSThreads, smem, st>>>(
        pl, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, a.orb[s], nop, false, nullptr, nullptr,
        nullptr, nullptr, nop, nocc, a.orb_occ[s]);
    return 1;
  }
  const int64_t most = orbital_psi_tiles(sp, nop), parts = (nt + most - 1) / most;
  const int64_t step = (nt + parts - 1) / parts;
  for (int64_t u = 0; u < nt; u += step) {
    const dim3 grid((unsigned)std::min(step, nt - u), 2);
    const int64_t p = u * 128;
    const SPlanes pu{phi, phi, phi, b.rho + p, nullptr, nullptr};
    k_sdensity<false, true, kPsi><<<grid, kSThreads, smem, st>>>(
        pu, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0 + u, s0, sp->slot_fn + s0, a.orb[s], nop, false, nullptr,
        nullptr, nullptr, sp->psi, nop, nocc, a.orb_occ[s]);
    launches += 2;
    if (tau) {
      const SPlanes pt{gx, gy, gz, tau + p, tau + cp + p, tau + 2 * cp + p};
      k_sdensity<true, false, kPsi><<<dim3(grid.x, 2, 3), kSThreads, smem, st>>>(
          pt, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0 + u, s0, sp->slot_fn + s0, a.orb[s], nop, false, b.grx + p,
          b.gry + p, b.grz + p, sp->psi, nop, nocc, a.orb_occ[s]);
      continue;
    }
    const SPlanes px{sp->psi, nullptr, nullptr, nullptr, nullptr, nullptr};
    k_sdensity<true, false, kFromPsi><<<grid, kSThreads, smem, st>>>(
        px, gx, gy, gz, sp->tso, sp->listed, t0 + u, s0, sp->slot_fn + s0, a.orb_scaled[s], a.ldc, false, b.grx + p,
        b.gry + p, b.grz + p, nullptr, nop, nocc, nullptr);
  }
  return launches;
}

int screen_run(ScreenPlan* sp, const BuildArgs& a, const double* Pb, cudaStream_t st, double* ham, ScreenTimes* tm,
               std::string& err, const ScreenExtra* extra) {
  const bool potential = !extra || extra->potential;
  const bool gga = sp->gga;
  const int ispin = sp->ispin;
  const double* P[2] = {a.P, Pb};
  const int64_t nb2 = sp->nbas * sp->nbas;
  const bool timed = tm != nullptr;  // untimed: no event records, synchronisation or host reads (capturable)
  // resident basis values filled by an earlier build: skip their evaluation (K1)
  const bool eval_basis = !(sp->keep && sp->basis_ready);
  ScreenTimes T;
#define SR_TRY(call)                                                          \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                  \
      err = std::string("screened build: ") + cudaGetErrorString(e_);         \
      return PGXC_ECUDA;                                                      \
    }                                                                         \
  } while (0)
  if (!a.cleared) SR_TRY(cudaMemsetAsync(sp->V, 0, sizeof(double) * ispin * nb2, st));
  if (sp->mixed) {
    for (int s = 0; s < ispin; ++s) T.launches += screen_mixed_prepare(sp->mixed, P[s], a.ldc, s, st);
    SR_TRY(cudaGetLastError());
  }
  if (timed)
    while (sp->cev.size() < sp->chunk_t0.size() - 1) {
      sp->cev.emplace_back();
      for (auto& e : sp->cev.back()) SR_TRY(cudaEventCreate(&e));
    }
  const int64_t cp = sp->chunk_tiles * 128;
  // per-chunk point arrays of spin s: 8 columns of cp (rho, grad rho, A, B) from pt + 8 s cp
  BuildArgs b[2];
  for (int s = 0; s < ispin; ++s) {
    double* q = sp->pt + 8 * s * cp;
    b[s] = a;
    b[s].ldp = cp;
    b[s].w = nullptr;
    b[s].rho = q;
    b[s].grx = q + cp;
    b[s].gry = q + 2 * cp;
    b[s].grz = q + 3 * cp;
    b[s].A = q + 4 * cp;
    b[s].Bx = q + 5 * cp;
    b[s].By = q + 6 * cp;
    b[s].Bz = q + 7 * cp;
    b[s].partial = sp->partial;
  }
  const size_t nch = sp->chunk_t0.size() - 1;
  for (size_t c = 0; c < nch; ++c) {
    cudaEvent_t* ev = timed ? sp->cev[c].data() : nullptr;
    const int64_t t0 = sp->chunk_t0[c], t1 = sp->chunk_t0[c + 1], nt = t1 - t0;
    const int64_t s0 = sp->h_tso[(size_t)t0], ns = sp->h_tso[(size_t)t1] - s0;
    const int64_t npt = nt * 128;
    // this chunk's rows of the basis arrays (resident: the chunk's place among all slots)
    const int64_t so = sp->keep ? s0 : 0, to = sp->keep ? t0 : 0;
    double* phi = sp->phi + so * 128;
    const bool gf = sp->gf32;
    double* gxc = gga && !gf ? sp->gx + so * 128 : nullptr;
    double* gyc = gga && !gf ? sp->gy + so * 128 : nullptr;
    double* gzc = gga && !gf ? sp->gz + so * 128 : nullptr;
    float* fxc = gga && gf ? sp->fx + so * 128 : nullptr;
    float* fyc = gga && gf ? sp->fy + so * 128 : nullptr;
    float* fzc = gga && gf ? sp->fz + so * 128 : nullptr;
    if (sp->mixed) {
      const bool use = sp->ordered[c];
      screen_mixed_set_order(sp->mixed, use ? sp->order + t0 : nullptr,
                             use ? sp->order_start + c * (size_t)(sp->nsm + 1) : nullptr);
    }
    if (timed) SR_TRY(cudaEventRecord(ev[0], st));
    // K1
    if (!eval_basis) {
      if (sp->mixed) T.launches += screen_mixed_gather(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, 0, st);
    } else {
      const unsigned g = (unsigned)nt;
      if (gga && gf) k_tile_init<true, float><<<g, 128, 0, st>>>(sp->tso, sp->listed, t0, s0, phi, fxc, fyc, fzc, sp->pmax);
      else if (gga) k_tile_init<true><<<g, 128, 0, st>>>(sp->tso, sp->listed, t0, s0, phi, gxc, gyc, gzc, sp->pmax);
      else k_tile_init<false><<<g, 128, 0, st>>>(sp->tso, sp->listed, t0, s0, phi, gxc, gyc, gzc, sp->pmax);
      ++T.launches;
      const BasisItem* items[kMaxL + 1];
      int64_t ni[kMaxL + 1];
      for (int l = 0; l <= kMaxL; ++l) {
        items[l] = sp->items[l] + sp->item_off[l][c];
        ni[l] = sp->item_off[l][c + 1] - sp->item_off[l][c];
      }
      auto io = [&](auto* gx, auto* gy, auto* gz) {
        using GT = std::remove_pointer_t<decltype(gx)>;
        return BasisIO<GT>{a.exps, a.norms, a.contr, a.rng, a.prim, sp->qx, sp->qy, sp->qz, s0, t0, phi, gx, gy, gz, sp->pmax};
      };
      if (gga && gf)
        T.launches += launch_basis_items<true, float>(items, ni, sp->nsm, kBasisBlocksPerSM, io(fxc, fyc, fzc), a.sa, st);
      else if (gga)
        T.launches += launch_basis_items<true, double>(items, ni, sp->nsm, kBasisBlocksPerSM, io(gxc, gyc, gzc), a.sa, st);
      else
        T.launches += launch_basis_items<false, double>(items, ni, sp->nsm, kBasisBlocksPerSM, io(gxc, gyc, gzc), a.sa, st);
      if (sp->mixed)
        T.launches += screen_mixed_basis(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, phi, sp->pmax, so, to, st);
    }
    if (timed) SR_TRY(cudaEventRecord(ev[1], st));
    // K3, per spin
    for (int s = 0; s < ispin; ++s) {
      if (sp->mixed) {
        if (s > 0) T.launches += screen_mixed_gather(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, s, st);
        if (gf)
          T.launches += screen_mixed_density(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, phi, fxc, fyc, fzc,
                                             b[s].rho, b[s].grx, b[s].gry, b[s].grz, so, to, st);
        else
          T.launches += screen_mixed_density(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, phi, gxc, gyc, gzc,
                                             b[s].rho, b[s].grx, b[s].gry, b[s].grz, so, to, st);
      } else if (a.nop) {
        T.launches += orbital_density(sp, a, s, t0, nt, s0, phi, gxc, gyc, gzc, b[s], sp->mgga ? sp->tq + 4 * s * cp : nullptr,
                                      cp, st);
        continue;
      } else {
        const int smem = sdensity_smem(sp->max_n);
        const SPlanes pl{phi, phi, phi, b[s].rho, b[s].rho, b[s].rho};
        if (gga) {
          raise_smem_limit(k_sdensity<true>, smem);
          k_sdensity<true><<<dim3((unsigned)nt, 2), kSThreads, smem, st>>>(
              pl, gxc, gyc, gzc, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, P[s], a.ldc, false, b[s].grx, b[s].gry,
              b[s].grz);
        } else {
          raise_smem_limit(k_sdensity<false>, smem);
          k_sdensity<false><<<dim3((unsigned)nt, 2), kSThreads, smem, st>>>(
              pl, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, P[s], a.ldc, a.p_symmetric,
              nullptr, nullptr, nullptr);
        }
        ++T.launches;
      }
      if (sp->mgga || (extra && extra->tau)) {
        // 2 tau_j = sum_nu (d_j phi P)_nu d_j phi_nu: the density contraction with d_j phi in the
        // place of phi (FP64 DMMA in every precision mode)
        const int smem = sdensity_smem(sp->max_n);
        raise_smem_limit(k_sdensity<false>, smem);
        double* tau = sp->tq + 4 * s * cp;
        const SPlanes pl{gxc, gyc, gzc, tau, tau + cp, tau + 2 * cp};
        k_sdensity<false><<<dim3((unsigned)nt, 2, 3), kSThreads, smem, st>>>(
            pl, nullptr, nullptr, nullptr, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, P[s], a.ldc, a.p_symmetric,
            nullptr, nullptr, nullptr);
        ++T.launches;
      }
    }
    if (timed) SR_TRY(cudaEventRecord(ev[2], st));
    // K2
    if (sp->mgga) {
      launch_functional_mgga(sp->functional, ispin, sp->qw, sp->pt, sp->tq, cp, t0 * 128, npt, sp->partial, a.acc,
                             st);
    } else if (ispin == 1) {
      BuildArgs bf = b[0];
      bf.w = sp->qw;
      launch_functional_f64(bf, t0 * 128, npt, gga, st);
    } else {
      launch_functional2_f64(a.xc, sp->qw, b[0].rho, b[1].rho, cp, t0 * 128, npt, gga, sp->partial, a.acc, st);
    }
    T.launches += sp->mgga ? 2 : 1;
    if (timed) SR_TRY(cudaEventRecord(ev[3], st));
    // K4, per spin: the contraction of spin s is bracketed by ev[4 + 2s], ev[5 + 2s]
    for (int s = 0; s < ispin && potential; ++s) {
      double* Vs = sp->V + s * nb2;
      cudaEvent_t k0 = timed ? ev[4 + 2 * s] : nullptr, k1 = timed ? ev[5 + 2 * s] : nullptr;
      if (sp->mixed) {
        if (gf)
          T.launches += screen_mixed_potential(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, phi,
                                               fxc, fyc, fzc, b[s].A, b[s].Bx, b[s].By, b[s].Bz, Vs, sp->nbas,
                                               st, k0, k1);
        else
          T.launches += screen_mixed_potential(sp->mixed, sp->tso, sp->slot_fn, t0, nt, s0, phi,
                                               gxc, gyc, gzc, b[s].A, b[s].Bx, b[s].By, b[s].Bz, Vs, sp->nbas,
                                               st, k0, k1);
      } else {
        const int smem = svpot_smem(sp->max_n);
        const unsigned nI = (unsigned)((sp->max_n + kRows - 1) / kRows);
        const dim3 grid((unsigned)nt * nI);
        const SPlanes pl{phi, phi, phi, nullptr, nullptr, nullptr};
        if (timed) SR_TRY(cudaEventRecord(k0, st));
        if (gga) {
          raise_smem_limit(k_svpot<kFull, true>, smem);
          k_svpot<kFull, true><<<grid, kSThreads, smem, st>>>(pl, gxc, gyc, gzc, b[s].A, b[s].Bx, b[s].By, b[s].Bz,
                                                              sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, Vs, sp->nbas, nI);
        } else {
          raise_smem_limit(k_svpot<kUpper, false>, smem);
          k_svpot<kUpper, false><<<grid, kSThreads, smem, st>>>(pl, nullptr, nullptr, nullptr, b[s].A, nullptr, nullptr,
                                                                nullptr, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, Vs,
                                                                sp->nbas, nI);
        }
        if (timed) SR_TRY(cudaEventRecord(k1, st));
        ++T.launches;
      }
      if (sp->mgga) {
        // tau term: per direction Z = C d_j phi and H += Z^T d_j phi over the upper triangle of
        // each tile (k_spack then forms H + H^T), FP64 DMMA in every precision mode
        const int smem = svpot_smem(sp->max_n);
        raise_smem_limit(k_svpot<kTwice, false>, smem);
        const SPlanes pl{gxc, gyc, gzc, nullptr, nullptr, nullptr};
        const unsigned nI = (unsigned)((sp->max_n + kRows - 1) / kRows);
        k_svpot<kTwice, false><<<dim3((unsigned)nt * nI, 1, 3), kSThreads, smem,
                                 st>>>(pl, nullptr, nullptr, nullptr, sp->tq + (4 * s + 3) * cp, nullptr, nullptr,
                                       nullptr, sp->tso, sp->listed, t0, s0, sp->slot_fn + s0, Vs, sp->nbas, nI);
        ++T.launches;
      }
    }
    // further functionals on the same density (after K4, whose A and B they overwrite)
    for (int i = 0; extra && i < extra->n; ++i) {
      if (extra->fid && PGXC_XC_IS_MGGA(extra->fid[i])) {
        launch_functional_mgga(extra->fid[i], ispin, sp->qw, sp->pt, sp->tq, cp, t0 * 128, npt, sp->partial,
                               extra->acc + 4 * i, st);
      } else if (ispin == 1) {
        BuildArgs bx = b[0];
        bx.w = sp->qw;
        bx.xc = extra->xc[i];
        bx.acc = extra->acc + 4 * i;
        launch_functional_f64(bx, t0 * 128, npt, extra->gga[i] != 0, st);
      } else {
        launch_functional2_f64(extra->xc[i], sp->qw, b[0].rho, b[1].rho, cp, t0 * 128, npt, extra->gga[i] != 0,
                               sp->partial, extra->acc + 4 * i, st);
      }
      T.launches += extra->fid && PGXC_XC_IS_MGGA(extra->fid[i]) ? 2 : 1;
    }
    SR_TRY(cudaGetLastError());
    // the packing counts with the last chunk's potential
    if (timed && c + 1 < nch) SR_TRY(cudaEventRecord(ev[8], st));
  }
  if (potential) {
    const int64_t len = sp->nbas * (sp->nbas + 1) / 2;
    const unsigned nbk = (unsigned)std::min<int64_t>((len + 255) / 256, 148 * 8);
    const int* failed = sp->mixed ? screen_mixed_error(sp->mixed) : nullptr;
    for (int s = 0; s < ispin; ++s) {
      k_spack<<<nbk, 256, 0, st>>>(sp->V + s * nb2, sp->nbas, gga, ispin, s, ham, a.acc, s == 0 ? a.exc_nel : nullptr,
                                   failed);
      ++T.launches;
    }
  }
  SR_TRY(cudaGetLastError());
  if (timed) {
    SR_TRY(cudaEventRecord(sp->cev[nch - 1][8], st));
    *tm = T;
  }
#undef SR_TRY
  return PGXC_OK;
}

int screen_finish(ScreenPlan* sp, cudaStream_t st, cudaEvent_t start, ScreenTimes* tm, std::string& err) {
  float ms;
  ScreenTimes& T = *tm;
#define SF_TRY(call)                                                          \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                  \
      err = std::string("screened build: ") + cudaGetErrorString(e_);         \
      return PGXC_ECUDA;                                                      \
    }                                                                         \
  } while (0)
  SF_TRY(cudaStreamSynchronize(st));
  const size_t nch = sp->chunk_t0.size() - 1;
  SF_TRY(cudaEventElapsedTime(&ms, start, sp->cev[0][0]));
  T.density += ms;  // the density matrix and its digits
  for (size_t c = 0; c < nch; ++c) {
    const auto& ev = sp->cev[c];
    SF_TRY(cudaEventElapsedTime(&ms, ev[0], ev[1])); T.basis += ms;
    SF_TRY(cudaEventElapsedTime(&ms, ev[1], ev[2])); T.density += ms; T.x += ms;
    SF_TRY(cudaEventElapsedTime(&ms, ev[2], ev[3])); T.functional += ms;
    SF_TRY(cudaEventElapsedTime(&ms, ev[3], ev[8])); T.potential += ms;
    for (int s = 0; s < sp->ispin; ++s) {
      SF_TRY(cudaEventElapsedTime(&ms, ev[4 + 2 * s], ev[5 + 2 * s]));
      T.v += ms;
    }
  }
#undef SF_TRY
  if (sp->mixed) {
    int flag = 0;
    if (screen_mixed_error_flag(sp->mixed, st, &flag) != PGXC_OK) {
      err = "screened build: error-flag read failed";
      return PGXC_ECUDA;
    }
    if (flag) {
      err = "screened build: a bounded tensor-core pipeline wait ran out";
      return PGXC_ETIMEOUT;
    }
  }
  if (sp->keep) sp->basis_ready = true;  // a completed build has filled the resident basis values
  return PGXC_OK;
}

double* screen_potential(ScreenPlan* sp, int64_t* n) {
  *n = sp->ispin * sp->nbas * sp->nbas;
  return sp->V;
}

int screen_enable_tau(ScreenPlan* sp, std::string& err) {
  if (sp->tq) return PGXC_OK;
  if (!sp->gga || sp->gf32) {
    err = "meta-GGA energies need the FP64 gradient planes of a GGA (or a meta-GGA) context";
    return PGXC_ENOTSUP;
  }
  const int64_t cp = sp->chunk_tiles * 128;
  if (sp_alloc(sp, &sp->tq, 4 * (size_t)sp->ispin * cp) != cudaSuccess ||
      cudaMemset(sp->tq, 0, sizeof(double) * 4 * sp->ispin * cp) != cudaSuccess) {
    err = "meta-GGA energies: the tau buffer";
    return PGXC_ENOMEM;
  }
  return PGXC_OK;
}

int screen_raise_error(ScreenPlan* sp, cudaStream_t st) {
  return sp->mixed ? screen_mixed_raise_error(sp->mixed, st) : PGXC_ENOTSUP;
}

int screen_error_flag(ScreenPlan* sp, cudaStream_t st, int* flag) {
  *flag = 0;
  if (!sp->mixed) return PGXC_OK;
  return screen_mixed_error_flag(sp->mixed, st, flag);
}


// ---------------------------------------------------------------------------
// Sets of contexts (screened.h): one launch per kernel over many contexts'
// tiles.
// ---------------------------------------------------------------------------
namespace {

// per context: where its E_xc / N_el accumulators, V and outputs live
struct SetOutDev {
  double* acc;        // {E, cE, N, cN}
  const double* V;    // [nbas][nbas]
  int64_t nbas;
  int gga;
  double* ham;        // packed out
  double* exc_nel;    // {E, N} out
};

// one segment of a chunk: tiles [t0, t0 + n) (chunk-relative) of context m
struct SetSeg {
  int64_t t0, n;
  int m;
  int pad_;
};

__global__ void k_set_adjust_items(BasisItem* __restrict__ it, int64_t n, int64_t dtile, int64_t dslot, int dexp,
                                   int dcon, int drng) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  it[i].tile += (int)dtile;
  it[i].slot += dslot;
  it[i].exp_off += dexp;
  it[i].con_off += dcon;
  it[i].rad_off += drng;
}

// Per segment (block): the fixed-order sum of its tiles' partials, Kahan-added
// into its context's acc.
__global__ void k_set_sum(const double* __restrict__ partial, const SetSeg* __restrict__ seg,
                          const SetOutDev* __restrict__ out) {
  const SetSeg g = seg[blockIdx.x];
  __shared__ double se[128], sq[128];
  double e = 0.0, q = 0.0;
  for (int64_t i = threadIdx.x; i < g.n; i += blockDim.x) {
    e += partial[2 * (g.t0 + i)];
    q += partial[2 * (g.t0 + i) + 1];
  }
  se[threadIdx.x] = e;
  sq[threadIdx.x] = q;
  __syncthreads();
  for (int s = 64; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      se[threadIdx.x] += se[threadIdx.x + s];
      sq[threadIdx.x] += sq[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double* acc = out[g.m].acc;
    const double vals[2] = {se[0], sq[0]};
    for (int k = 0; k < 2; ++k) {
      const double y = vals[k] - acc[2 * k + 1];
      const double t = acc[2 * k] + y;
      acc[2 * k + 1] = (t - acc[2 * k]) - y;
      acc[2 * k] = t;
    }
  }
}

// Block per context: the packed triangle (tristore order; GGA: H + H^T) and
// {E_xc, N_el}.
__global__ void k_set_pack(const SetOutDev* __restrict__ out) {
  const SetOutDev o = out[blockIdx.x];
  const int64_t len = o.nbas * (o.nbas + 1) / 2;
  for (int64_t idx = threadIdx.x; idx < len; idx += blockDim.x) {
    int64_t j = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > idx) --j;
    while ((j + 1) * (j + 2) / 2 <= idx) ++j;
    const int64_t k = idx - j * (j + 1) / 2;
    double v = o.V[k * o.nbas + j];
    if (o.gga) v += o.V[j * o.nbas + k];
    o.ham[idx] = v;
  }
  if (threadIdx.x == 0) {
    o.exc_nel[0] = o.acc[0];
    o.exc_nel[1] = o.acc[2];
  }
}

}  // namespace

struct ScreenSet {
  struct Group {
    XcConst xc;
    bool gga;
  };
  struct Chunk {
    int64_t t0, t1, s0;
    int64_t i0[kMaxL + 1], i1[kMaxL + 1];
    int group;
    int64_t seg0, nseg;
  };
  std::vector<SetMember> mem;
  std::vector<Group> groups;
  std::vector<Chunk> chunks;
  int64_t ntiles = 0, nslots = 0, chunk_slots = 0, chunk_tiles = 0;
  int max_n = 0;
  DevSA sa;
  // merged plan (device)
  double *qx = nullptr, *qy = nullptr, *qz = nullptr, *qw = nullptr;
  int64_t* tso = nullptr;
  int* slot_fn = nullptr;
  int* listed = nullptr;
  int* tile_mol = nullptr;
  BasisItem* items[kMaxL + 1] = {};
  double *exps = nullptr, *norms = nullptr, *contr = nullptr;
  int2* rng = nullptr;
  double2* prim = nullptr;
  SetMolDev* mols = nullptr;
  SetOutDev* outs = nullptr;
  SetSeg* segs = nullptr;
  int64_t* b_off = nullptr;
  // chunk buffers
  double* phi = nullptr;
  float *gx = nullptr, *gy = nullptr, *gz = nullptr;  // grad phi in 32 bits (the INT8 build's)
  double* pt = nullptr;
  double* partial = nullptr;
  unsigned long long* pmax = nullptr;
  ScreenMixed* mixed = nullptr;
  int nsm = 148;
  int64_t launches = 0;
  std::vector<void*> allocs;
};

void screen_set_destroy(ScreenSet* s) {
  if (!s) return;
  if (s->mixed) screen_mixed_destroy(s->mixed);
  for (void* p : s->allocs) cudaFree(p);
  delete s;
}

void screen_set_stats(const ScreenSet* s, int64_t* ntiles, int64_t* nchunks, int64_t* launches) {
  if (ntiles) *ntiles = s->ntiles;
  if (nchunks) *nchunks = (int64_t)s->chunks.size();
  if (launches) *launches = s->launches;
}

int screen_set_create(ScreenSet** out, const std::vector<SetMember>& members, int64_t max_chunk_points,
                      cudaStream_t st, std::string& err) {
  *out = nullptr;
  ScreenSet* S = new ScreenSet();
  auto fail = [&](int code, const std::string& m) {
    err = "set: " + m;
    screen_set_destroy(S);
    return code;
  };
#define SS_TRY(call, what)                                                                         \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess)                                                                         \
      return fail(e_ == cudaErrorMemoryAllocation ? PGXC_ENOMEM : PGXC_ECUDA,                       \
                  std::string(what) + ": " + cudaGetErrorString(e_));                              \
  } while (0)
  auto alloc = [&](auto** p, size_t n) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(**p));
    if (e == cudaSuccess) {
      S->allocs.push_back(q);
      *p = static_cast<std::remove_reference_t<decltype(*p)>>(q);
    }
    return e;
  };
  if (members.empty()) return fail(PGXC_EINVAL, "no contexts");
  // members grouped by functional (stable): a chunk holds one functional
  std::vector<int> order(members.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return members[(size_t)x].functional < members[(size_t)y].functional; });
  for (int i : order) S->mem.push_back(members[(size_t)i]);
  S->sa = S->mem[0].a->sa;
  for (const SetMember& m : S->mem) {
    const ScreenPlan* sp = m.sp;
    if (!sp->mixed || sp->ispin != 1 || sp->keep)
      return fail(PGXC_ENOTSUP, "every context must be a screened INT8 closed-shell one without keep_orbitals");
    if (!m.a->sa.identity) return fail(PGXC_ENOTSUP, "contexts with a symmetry adaptation table");
  }
  std::vector<int> mgroup(S->mem.size());
  for (size_t i = 0; i < S->mem.size(); ++i) {
    if (i == 0 || S->mem[i].functional != S->mem[i - 1].functional)
      S->groups.push_back({S->mem[i].a->xc, S->mem[i].sp->gga});
    mgroup[i] = (int)S->groups.size() - 1;
  }
  {
    int dev = 0;
    SS_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    SS_TRY(cudaDeviceGetAttribute(&S->nsm, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
  }
  // --- merged plan -----------------------------------------------------------
  const size_t nm = S->mem.size();
  std::vector<int64_t> toff(nm + 1, 0), soff(nm + 1, 0), eoff(nm + 1, 0), coff(nm + 1, 0), roff(nm + 1, 0);
  std::vector<int64_t> ioff[kMaxL + 1];
  for (int l = 0; l <= kMaxL; ++l) ioff[l].assign(nm + 1, 0);
  for (size_t i = 0; i < nm; ++i) {
    const ScreenPlan* sp = S->mem[i].sp;
    toff[i + 1] = toff[i] + sp->ntiles;
    soff[i + 1] = soff[i] + sp->nslots;
    eoff[i + 1] = eoff[i] + sp->n_exps;
    coff[i + 1] = coff[i] + sp->n_contr;
    roff[i + 1] = roff[i] + sp->n_rng;
    for (int l = 0; l <= kMaxL; ++l) ioff[l][i + 1] = ioff[l][i] + sp->item_off[l].back();
    S->max_n = std::max(S->max_n, sp->max_n);
  }
  S->ntiles = toff[nm];
  S->nslots = soff[nm];
  const int64_t T = S->ntiles;
  SS_TRY(alloc(&S->qx, 4 * (size_t)T * 128), "cudaMalloc");
  S->qy = S->qx + T * 128;
  S->qz = S->qx + 2 * T * 128;
  S->qw = S->qx + 3 * T * 128;
  SS_TRY(alloc(&S->tso, (size_t)T + 1), "cudaMalloc");
  SS_TRY(alloc(&S->slot_fn, (size_t)S->nslots), "cudaMalloc");
  SS_TRY(alloc(&S->listed, (size_t)T), "cudaMalloc");
  SS_TRY(alloc(&S->tile_mol, (size_t)T), "cudaMalloc");
  SS_TRY(alloc(&S->exps, (size_t)eoff[nm]), "cudaMalloc");
  SS_TRY(alloc(&S->norms, (size_t)eoff[nm]), "cudaMalloc");
  SS_TRY(alloc(&S->prim, (size_t)eoff[nm]), "cudaMalloc");
  SS_TRY(alloc(&S->contr, (size_t)coff[nm]), "cudaMalloc");
  SS_TRY(alloc(&S->rng, (size_t)roff[nm]), "cudaMalloc");
  for (int l = 0; l <= kMaxL; ++l) SS_TRY(alloc(&S->items[l], (size_t)ioff[l][nm]), "cudaMalloc");
  std::vector<int64_t> h_tso((size_t)T + 1, 0);
  std::vector<int> h_tile_mol((size_t)T);
  std::vector<SetMolDev> h_mols(nm);
  std::vector<SetOutDev> h_outs(nm);
  for (size_t i = 0; i < nm; ++i) {
    const ScreenPlan* sp = S->mem[i].sp;
    const BuildArgs* a = S->mem[i].a;
    const int64_t nt = sp->ntiles, t0 = toff[i];
    for (int c = 0; c < 4; ++c) {
      const double* src = c == 0 ? sp->qx : (c == 1 ? sp->qy : (c == 2 ? sp->qz : sp->qw));
      SS_TRY(cudaMemcpyAsync(S->qx + c * T * 128 + t0 * 128, src, sizeof(double) * nt * 128,
                             cudaMemcpyDeviceToDevice, st), "copy");
    }
    SS_TRY(cudaMemcpyAsync(S->slot_fn + soff[i], sp->slot_fn, sizeof(int) * sp->nslots, cudaMemcpyDeviceToDevice, st),
           "copy");
    SS_TRY(cudaMemcpyAsync(S->listed + t0, sp->listed, sizeof(int) * nt, cudaMemcpyDeviceToDevice, st), "copy");
    SS_TRY(cudaMemcpyAsync(S->exps + eoff[i], a->exps, sizeof(double) * sp->n_exps, cudaMemcpyDeviceToDevice, st),
           "copy");
    SS_TRY(cudaMemcpyAsync(S->norms + eoff[i], a->norms, sizeof(double) * sp->n_exps, cudaMemcpyDeviceToDevice, st),
           "copy");
    SS_TRY(cudaMemcpyAsync(S->prim + eoff[i], a->prim, sizeof(double2) * sp->n_exps, cudaMemcpyDeviceToDevice, st),
           "copy");
    if (sp->n_contr)
      SS_TRY(cudaMemcpyAsync(S->contr + coff[i], a->contr, sizeof(double) * sp->n_contr, cudaMemcpyDeviceToDevice,
                             st), "copy");
    if (sp->n_rng)
      SS_TRY(cudaMemcpyAsync(S->rng + roff[i], a->rng, sizeof(int2) * sp->n_rng, cudaMemcpyDeviceToDevice, st),
             "copy");
    for (int l = 0; l <= kMaxL; ++l) {
      const int64_t ni = ioff[l][i + 1] - ioff[l][i];
      if (!ni) continue;
      BasisItem* dst = S->items[l] + ioff[l][i];
      SS_TRY(cudaMemcpyAsync(dst, sp->items[l], sizeof(BasisItem) * ni, cudaMemcpyDeviceToDevice, st), "copy");
      k_set_adjust_items<<<(unsigned)((ni + 255) / 256), 256, 0, st>>>(dst, ni, t0, soff[i], (int)eoff[i],
                                                                      (int)coff[i], (int)roff[i]);
    }
    for (int64_t t = 0; t <= nt; ++t) h_tso[(size_t)(t0 + t)] = sp->h_tso[(size_t)t] + soff[i];
    for (int64_t t = 0; t < nt; ++t) h_tile_mol[(size_t)(t0 + t)] = (int)i;
    const unsigned long long* P8;
    const int* eP;
    screen_mixed_p8(sp->mixed, 0, &P8, &eP);
    h_mols[i] = {P8, eP, sp->nbas, sp->V, sp->nbas};
    h_outs[i] = {a->acc, sp->V, sp->nbas, sp->gga ? 1 : 0, S->mem[i].d_ham, S->mem[i].d_exc_nel};
  }
  SS_TRY(cudaGetLastError(), "item offsets");
  SS_TRY(cudaMemcpyAsync(S->tso, h_tso.data(), sizeof(int64_t) * h_tso.size(), cudaMemcpyHostToDevice, st), "copy");
  SS_TRY(cudaMemcpyAsync(S->tile_mol, h_tile_mol.data(), sizeof(int) * h_tile_mol.size(), cudaMemcpyHostToDevice, st),
         "copy");
  SS_TRY(alloc(&S->mols, nm), "cudaMalloc");
  SS_TRY(alloc(&S->outs, nm), "cudaMalloc");
  SS_TRY(cudaMemcpyAsync(S->mols, h_mols.data(), sizeof(SetMolDev) * nm, cudaMemcpyHostToDevice, st), "copy");
  SS_TRY(cudaMemcpyAsync(S->outs, h_outs.data(), sizeof(SetOutDev) * nm, cudaMemcpyHostToDevice, st), "copy");
  // --- chunks: runs of whole tiles of one functional group --------------------
  size_t freeb = 0, totb = 0;
  SS_TRY(cudaMemGetInfo(&freeb, &totb), "cudaMemGetInfo");
  const bool any_gga = std::any_of(S->groups.begin(), S->groups.end(), [](const ScreenSet::Group& g) { return g.gga; });
  const int64_t per_slot = 128 * (8 + (any_gga ? 12 : 0)) + screen_mixed_bytes_per_slot();
  const int64_t per_tile = 128 * 8 * 8 + screen_mixed_bytes_per_tile() + 128 * 8 + 16;
  int64_t budget_slots = std::max<int64_t>((int64_t)(0.40 * (double)freeb) / per_slot, S->max_n);
  int64_t budget_tiles = std::max<int64_t>(1, (int64_t)(0.05 * (double)freeb) / per_tile);
  if (max_chunk_points > 0) budget_tiles = std::min(budget_tiles, std::max<int64_t>(1, max_chunk_points / 128));
  budget_tiles = std::min<int64_t>(budget_tiles, 1 << 16);
  std::vector<int64_t> boff((size_t)T + 1, 0);
  for (int64_t t = 0; t < T; ++t)
    boff[(size_t)t + 1] = boff[(size_t)t] + screen_mixed_bstages(h_tso[(size_t)t + 1] - h_tso[(size_t)t]);
  const int64_t budget_b = std::max<int64_t>((int64_t)(0.20 * (double)freeb) / screen_mixed_bytes_per_bstage(),
                                             screen_mixed_bstages(S->max_n));
  std::vector<SetSeg> h_segs;
  int64_t chunk_b = 0;
  {
    int64_t t0 = 0;
    auto close_chunk = [&](int64_t t1) {
      ScreenSet::Chunk c{};
      c.t0 = t0;
      c.t1 = t1;
      c.s0 = h_tso[(size_t)t0];
      c.group = mgroup[(size_t)h_tile_mol[(size_t)t0]];
      // item ranges: items are ordered by tile within and across contexts
      for (int l = 0; l <= kMaxL; ++l) {
        auto first_item = [&](int64_t t) {
          if (t >= T) return ioff[l][nm];
          const int m = h_tile_mol[(size_t)t];
          // the context's items before its tile t - toff[m]
          return ioff[l][(size_t)m] + S->mem[(size_t)m].sp->tile_item[l][(size_t)(t - toff[(size_t)m])];
        };
        c.i0[l] = first_item(t0);
        c.i1[l] = first_item(t1);
      }
      c.seg0 = (int64_t)h_segs.size();
      for (int64_t t = t0; t < t1;) {
        const int m = h_tile_mol[(size_t)t];
        const int64_t te = std::min(t1, toff[(size_t)m + 1]);
        h_segs.push_back({t - t0, te - t, m, 0});
        t = te;
      }
      c.nseg = (int64_t)h_segs.size() - c.seg0;
      S->chunks.push_back(c);
      S->chunk_tiles = std::max(S->chunk_tiles, t1 - t0);
      S->chunk_slots = std::max(S->chunk_slots, h_tso[(size_t)t1] - h_tso[(size_t)t0]);
      chunk_b = std::max(chunk_b, boff[(size_t)t1] - boff[(size_t)t0]);
      t0 = t1;
    };
    for (int64_t t = 0; t < T; ++t) {
      if (t == t0) continue;
      const bool new_group = mgroup[(size_t)h_tile_mol[(size_t)t]] != mgroup[(size_t)h_tile_mol[(size_t)t0]];
      const bool full = h_tso[(size_t)t + 1] - h_tso[(size_t)t0] > budget_slots || t + 1 - t0 > budget_tiles ||
                        boff[(size_t)t + 1] - boff[(size_t)t0] > budget_b;
      if (new_group || full) close_chunk(t);
    }
    close_chunk(T);
  }
  SS_TRY(alloc(&S->segs, h_segs.size()), "cudaMalloc");
  SS_TRY(cudaMemcpyAsync(S->segs, h_segs.data(), sizeof(SetSeg) * h_segs.size(), cudaMemcpyHostToDevice, st), "copy");
  SS_TRY(alloc(&S->b_off, boff.size()), "cudaMalloc");
  SS_TRY(cudaMemcpyAsync(S->b_off, boff.data(), sizeof(int64_t) * boff.size(), cudaMemcpyHostToDevice, st), "copy");
  // --- chunk buffers -----------------------------------------------------------
  const size_t rows = (size_t)(S->chunk_slots + kSlack) * 128;
  SS_TRY(alloc(&S->phi, rows), "cudaMalloc (phi)");
  SS_TRY(cudaMemsetAsync(S->phi, 0, sizeof(double) * rows, st), "memset");
  if (any_gga) {
    SS_TRY(alloc(&S->gx, rows), "cudaMalloc (grad phi)");
    SS_TRY(alloc(&S->gy, rows), "cudaMalloc (grad phi)");
    SS_TRY(alloc(&S->gz, rows), "cudaMalloc (grad phi)");
    SS_TRY(cudaMemsetAsync(S->gx, 0, sizeof(float) * rows, st), "memset");
    SS_TRY(cudaMemsetAsync(S->gy, 0, sizeof(float) * rows, st), "memset");
    SS_TRY(cudaMemsetAsync(S->gz, 0, sizeof(float) * rows, st), "memset");
  }
  SS_TRY(alloc(&S->pt, 8 * (size_t)S->chunk_tiles * 128), "cudaMalloc");
  SS_TRY(alloc(&S->partial, 2 * (size_t)S->chunk_tiles), "cudaMalloc");
  SS_TRY(alloc(&S->pmax, (size_t)S->chunk_tiles * 128), "cudaMalloc");
  SS_TRY(cudaStreamSynchronize(st), "set-up");
  ScreenMixedInput mi;
  mi.nbas = 1;  // the members' own density-matrix digits are used
  mi.ldc = 1;
  mi.gga = any_gga;
  mi.nspin = 1;
  mi.chunk_slots = S->chunk_slots + kSlack;
  mi.chunk_tiles = S->chunk_tiles;
  mi.max_n = S->max_n;
  mi.chunk_bstages = chunk_b;
  mi.b_off = S->b_off;
  std::string e2;
  if (int st2 = screen_mixed_create(&S->mixed, mi, e2)) return fail(st2, e2);
#undef SS_TRY
  *out = S;
  return PGXC_OK;
}

int screen_set_run(ScreenSet* S, cudaStream_t st, std::string& err) {
  const int64_t cp = S->chunk_tiles * 128;
  int64_t launches = 0;
  for (const ScreenSet::Chunk& c : S->chunks) {
    const ScreenSet::Group& g = S->groups[(size_t)c.group];
    const bool gga = g.gga;
    const int64_t t0 = c.t0, nt = c.t1 - c.t0, s0 = c.s0;
    float* gxc = gga ? S->gx : nullptr;
    float* gyc = gga ? S->gy : nullptr;
    float* gzc = gga ? S->gz : nullptr;
    if (gga)
      k_tile_init<true, float><<<(unsigned)nt, 128, 0, st>>>(S->tso, S->listed, t0, s0, S->phi, gxc, gyc, gzc, S->pmax);
    else
      k_tile_init<false, float><<<(unsigned)nt, 128, 0, st>>>(S->tso, S->listed, t0, s0, S->phi, gxc, gyc, gzc, S->pmax);
    ++launches;
    const BasisItem* items[kMaxL + 1];
    int64_t ni[kMaxL + 1];
    for (int l = 0; l <= kMaxL; ++l) {
      items[l] = S->items[l] + c.i0[l];
      ni[l] = c.i1[l] - c.i0[l];
    }
    const BasisIO<float> io{S->exps, S->norms, S->contr, S->rng, S->prim, S->qx, S->qy, S->qz,
                            s0,      t0,       S->phi,   gxc,    gyc,     gzc,   S->pmax};
    launches += gga ? launch_basis_items<true, float>(items, ni, S->nsm, kBasisBlocksPerSM, io, S->sa, st)
                    : launch_basis_items<false, float>(items, ni, S->nsm, kBasisBlocksPerSM, io, S->sa, st);
    screen_mixed_set_gga(S->mixed, gga);
    launches += screen_mixed_basis(S->mixed, S->tso, S->slot_fn, t0, nt, s0, S->phi, S->pmax, 0, 0, st, S->tile_mol,
                                   S->mols);
    double* q = S->pt;
    BuildArgs b{};
    b.xc = g.xc;
    b.w = S->qw;
    b.rho = q;
    b.grx = q + cp;
    b.gry = q + 2 * cp;
    b.grz = q + 3 * cp;
    b.A = q + 4 * cp;
    b.Bx = q + 5 * cp;
    b.By = q + 6 * cp;
    b.Bz = q + 7 * cp;
    b.partial = S->partial;
    launches += screen_mixed_density(S->mixed, S->tso, S->slot_fn, t0, nt, s0, S->phi, gxc, gyc, gzc, b.rho, b.grx,
                                     b.gry, b.grz, 0, 0, st);
    launch_functional_tiles(b, t0 * 128, nt, gga, st);
    k_set_sum<<<(unsigned)c.nseg, 128, 0, st>>>(S->partial, S->segs + c.seg0, S->outs);
    launches += 2;
    launches += screen_mixed_potential(S->mixed, S->tso, S->slot_fn, t0, nt, s0, S->phi, gxc, gyc, gzc, b.A,
                                       b.Bx, b.By, b.Bz, nullptr, 0, st, nullptr, nullptr, S->tile_mol, S->mols);
  }
  k_set_pack<<<(unsigned)S->mem.size(), 256, 0, st>>>(S->outs);
  ++launches;
  S->launches = launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("set build: ") + cudaGetErrorString(e);
    return PGXC_ECUDA;
  }
  return PGXC_OK;
}

int screen_set_error_flag(ScreenSet* S, cudaStream_t st, int* flag) { return screen_mixed_error_flag(S->mixed, st, flag); }

int screen_set_prepare_member(ScreenPlan* sp, const double* P, int64_t ldc, cudaStream_t st) {
  screen_mixed_prepare(sp->mixed, P, ldc, 0, st);
  return cudaGetLastError() == cudaSuccess ? PGXC_OK : PGXC_ECUDA;
}

bool screen_set_eligible(const ScreenPlan* sp) { return sp->mixed && sp->ispin == 1 && !sp->keep && !sp->mgga; }

}  // namespace pgxc
