// screened_plan.h -- the screening plan of one context (internal to the
// screened builds: screened.cu and the multi-context set in set_build.cu).
#pragma once

#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "basis.cuh"
#include "screened.h"
#include "screened_mixed.h"
#include <array>

namespace pgxc {

constexpr int kSlotAlign = 32;   // slots per tile are padded to this (INT8 K step)
constexpr int64_t kSlack = 128;  // zero rows after the last slot of a chunk
constexpr int kBasisBlocksPerSM = 16;  // blocks of the basis kernels per SM (each walks a range of items)

// What the listing of tiles reads (device; one allocation): each tile's first
// item of each l, the listing radii, the tiles' smallest squared distances to the atoms.
struct ListTables {
  void* base = nullptr;
  int64_t* start = nullptr;  // [ntiles][kMaxL + 1]
  double* r2 = nullptr;
  float* d2 = nullptr;       // [ntiles][natm]
  int* cnt = nullptr;        // [ntiles] {listed functions, items of each l}
  int* r2off = nullptr;
  int natm = 0, nsh = 0;
};
// Where the lists of a run of tiles go: slot_fn from its first slot s0 on, items[l] from its first item i0[l] on.
struct TileLists {
  int* slot_fn;
  int64_t s0;
  BasisItem* items[kMaxL + 1];
  int64_t i0[kMaxL + 1];
};

struct ScreenPlan {
  int64_t ntiles = 0, nslots = 0, nlisted = 0;
  double sum_n2 = 0.0;
  int max_n = 0;
  bool gga = false;
  int ispin = 1;
  int64_t nbas = 0;
  int64_t n_exps = 0, n_contr = 0, n_rng = 0;  // lengths of the context's exponent, contraction and range tables
  bool keep = false;         // basis values (and INT8 point digits) of all slots stay resident
  bool basis_ready = false;  // ... and a completed build has filled them
  // device, whole grid
  double *qx = nullptr, *qy = nullptr, *qz = nullptr, *qw = nullptr;  // points in the tiles' order [ntiles*128]
  int64_t* order_of_points = nullptr;  // their indices in the caller's grid (null: as they lie there)
  int64_t* tso = nullptr;   // [ntiles+1] first slot of each tile
  int* slot_fn = nullptr;   // [nslots] function of each slot, -1 for padding
  int* listed = nullptr;    // [ntiles] listed (not padding) slots of each tile
  int64_t* b_off = nullptr;  // [ntiles+1] first density B stage of each tile (INT8 path)
  BasisItem* items[kMaxL + 1] = {};
  // host copies of the partition
  std::vector<int64_t> h_tso;
  std::vector<int64_t> chunk_t0;                   // chunk c covers tiles [chunk_t0[c], chunk_t0[c+1])
  std::vector<int64_t> item_off[kMaxL + 1];        // items of chunk c: [item_off[L][c], item_off[L][c+1])
  std::vector<int64_t> tile_item[kMaxL + 1];       // items before tile t, per L ([ntiles + 1])
  int64_t chunk_slots = 0, chunk_tiles = 0;        // buffer capacities
  // device, per chunk
  double *phi = nullptr, *gx = nullptr, *gy = nullptr, *gz = nullptr;
  // INT8 build (not a meta-GGA): grad phi in 32-bit planes instead of gx/gy/gz
  bool gf32 = false;
  float *fx = nullptr, *fy = nullptr, *fz = nullptr;
  double* pt = nullptr;      // 8 point arrays of chunk_tiles*128 per spin
  bool mgga = false;
  int functional = 0;        // PGXC_XC_* (the meta-GGA step selects its functional by id)
  double* tq = nullptr;      // meta-GGA: 4 point arrays per spin (2 tau_x, 2 tau_y, 2 tau_z, C)
  double* psi = nullptr;     // [tile][padded orbital][128] of the orbital form (FP64 GGA), psi_cap elements
  int64_t psi_cap = 0;
  double* psi_own = nullptr;  // psi's buffer where it does not lie behind phi
  int64_t psi_refused = INT64_MAX;  // elements that there was no room for
  int64_t psi_tiles_most = 0; // tiles whose psi is held at once, at most (0: as many as kPsiMost holds)
  double* partial = nullptr;
  double* V = nullptr;       // [ispin][nbas][nbas]
  unsigned long long* pmax = nullptr;  // [chunk_tiles*128] largest |phi| per point (INT8 path)
  ScreenMixed* mixed = nullptr;
  int *order = nullptr, *order_start = nullptr;  // INT8: even tile lists ([ntiles] chunk by chunk, [chunk][nsm + 1])
  std::vector<char> ordered;                     // chunks that use them
  std::vector<std::array<cudaEvent_t, 9>> cev;  // timing events of each chunk (made by the first timed build)
  int nsm = 148;
  std::vector<void*> allocs;
  ListTables tab;  // gradient plans (a build's are released with its creation)
  // gradient plans: raw weight and host atom of the Morton-ordered points and the lists lie in the gradient's scratch,
  // the lists one chunk's at a time (chunk_items: the most items of a chunk; filled: the chunk whose lists lie there,
  // or -1: nothing has been written there yet)
  double* qwraw = nullptr;
  int* qowner = nullptr;
  int64_t chunk_items[kMaxL + 1] = {};
  int64_t filled = -1;
};

// A plan of tiles and list lengths alone (no lists, no build buffers), in chunks of
// at most max_rows slot rows, for the nuclear gradient; R2 with threshold 0, so that
// unlisted functions and their derivatives are exactly zero on the tile.  from: the
// context's own plan of the same grid, whose points are taken, or null (grad_plan_hosts).  The lists
// themselves are made chunk by chunk (grad_plan_lists): of a whole grid they would grow
// with tiles x shells (200 atoms, 13,300 tiles: 0.4 GB) and stay until the context goes.
int grad_plan_create(ScreenPlan** out, const BuildArgs& a, int natm, int64_t npts, const std::vector<DevShell>& shells,
                     const std::vector<double>& R2, const std::vector<int>& r2off, const ScreenPlan* from,
                     int64_t max_rows, cudaStream_t st, std::string& err);
// Raw weights and host atoms in the plan's point order into qwraw, qowner ([ntiles * 128]), and (points not null:
// the plan has none) the points and weights (4 [ntiles * 128]), unless they lie there.
void grad_plan_hosts(ScreenPlan* sp, const BuildArgs& a, int64_t npts, const double* wraw, const int* owner,
                     double* points, double* qwraw, int* qowner, cudaStream_t st);
// Chunk c's lists into `lists` (s0 and i0 are set here), unless they are what it holds.
void grad_plan_lists(ScreenPlan* sp, const BuildArgs& a, size_t c, const TileLists& lists, cudaStream_t st);
// The orbitals in the place of P (orbital_form_pays): nop padded, C [function][nop], occ C
// [nop][ldc], occupations [nop], and psi for psi_tiles tiles at a time.
struct GradOrbitals {
  int nop;
  const double *orb, *scaled, *occ;
  double* psi;
  int64_t psi_tiles;
};
bool orbital_form_pays(const ScreenPlan* sp, int64_t nop);
// tiles whose psi is held at once: those of a chunk, as many as 1 GB holds
int64_t orbital_psi_tiles(const ScreenPlan* sp, int64_t nop);
// X = F_t P[S_t, S_t] (by the orbitals when orb is not null) of the chunk's tiles (slot_fn: the chunk's; [slot][128] rows, padding rows of F
// zero), with rho[p] = sum X F and (gx not null) gr[p] = 2 sum X grad phi.
void grad_contract(const ScreenPlan* sp, const int* slot_fn, int64_t t0, int64_t nt, int64_t s0, const double* F, const double* gx,
                   const double* gy, const double* gz, const double* P, int64_t ldc, double* X, double* rho,
                   double* grx, double* gry, double* grz, const GradOrbitals* orb, cudaStream_t st);


}  // namespace pgxc
