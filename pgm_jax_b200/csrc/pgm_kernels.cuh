// pgm_kernels.cuh -- the sm_100a kernels of the pGM step.
//
// Layout in HBM (all systems of a batch concatenated; a block never straddles two systems):
//   atoms      SoA per-atom parameters (T) and state; 3-vectors as 16/32-byte v4<T> for single loads
//   rows       [atom][chunk of 32 entries]: partner k (int32), x, y, z, G1, G2, G0, G3 (T), 32 of each (RowChunk);
//              molecule partners first (the rigid special table), then the in-cutoff neighbours
//   PME        per system a real grid K1 x K2 x K3 (k3 fastest) and a half-complex grid
//              K1 x K2 x (K3/2 + 1), both as flat offsets into batch-wide buffers
//   reductions per-system FP64 accumulators (CGSys, EnergyAcc), filled by block partials + atomics
//
// Reference correspondence (pgm_jax/md/...): row build forcefield.py:1140-1195, radial kernels
// kernels.py:76-118 + forcefield.py:1318-1338, direct field forcefield.py:1395-1433, PME
// pme.py:243-411, CG forcefield.py:1714-1821, start forcefield.py:1917-2008, energy and forces
// forcefield.py:2011-2045,2294-2430, strain derivative forcefield.py:608-662,2628-2695.
#pragma once
#include <type_traits>

#include "pgm_device.cuh"
#include "pgm_nn.cuh"

namespace pgm {

template <typename T>
struct Dev {
  int nsys, nt, nmol, mc, ncell, ncov;
  int order;
  int induce, perm, lj, lj_lrc;
  double beta, cutoff, c_self, tol, peek;
  double skin;            // Verlet skin of the candidate list
  int cc;                 // candidate capacity per atom
  int *nb_flag;           // candidate list must be rebuilt
  long long *nb_builds;   // rebuild counter
  int *cand, *ncand;      // candidates (N, cc) and counts
  double4 *pos_ref;       // positions at the last rebuild
  double4 *pos4;          // positions this step, .w = molecule
  float4 *pos4f;          // FP32 rows (mixed precision): the positions wrapped into the box, .w = molecule
  int max_iter;
  const SysInfo *sys;
  BoxInfo *box;
  CGSys *cg;
  EnergyAcc *eacc;
  unsigned *status;
  // block maps of 8, 32 and 256 atoms per block: (system, first atom, end of the system's atoms)
  const int4 *wb, *qb, *tb;
  int K0[3];  // the mesh of the first system (all there is, often: see where())
  // atoms
  const int *sysid, *molid, *molfirst, *molend, *mol_start;
  const T *q, *radius, *alpha, *ialpha, *rminh, *seps;
  const c2<T> *ljp;  // per atom (R*/2, sqrt(eps)): one load per LJ partner in the force pass
  const double *mass;
  const int *cov_start, *cov_j, *cov_i_flat, *cov_j_flat;
  const double *cov_c, *cov_c_flat;
  // per step
  const double *pos;
  int4 *base;
  v4<T> *frac;
  double4 *pperm, *off;
  int *cell_of, *slot_of, *cell_count, *cell_start, *cell_atoms;
  v4<T> *spos;  // positions in cell order (mixed: wrapped), .w = molecule
  const int *idx;
  int idx_width;
  // rows
  int *rn, *rnsp;
  unsigned char *rows;
  int *max_count;  // [0] largest electrostatic (or only) part, [1] largest van der Waals part
  // split rows: the electrostatic part of a row is [0, mce), the van der Waals part [mce, mc) with
  // its counts in rnv (null: one cutoff, mce == mc); rce2 = elec_cutoff^2
  int mce;
  int *rnv;
  double rce2;
  // the learned guess's graph (the row entries with float(r^2) < nn_rg2): per atom up to nn_emax
  // edges (x, y, z, partner bits) in row order and the full count, written by the row build when
  // nn_e4 is set (the consumers read the first nn_emax), with the pair kernels G1, G2 of each edge
  // in nn_g (same slots)
  float4 *nn_e4;
  float2 *nn_g;
  int *nn_ne;
  int nn_emax;
  float nn_rg2;
  // local preconditioner (local_niter > 0, forcefield.py:1766-1792): the row entries with
  // r^2 < lc2, entry-major (entry e of atom i at e nt + i, at most sh_max, sh_n per atom): partner
  // displacement, G1 and G2 written by the row build; the inner CG's vectors
  // rr (LRR), alpha rr (LZZ), its directions (LP0 / LP1, alternating), and r_new - r_old of the
  // outer update (DR)
  int *sh_n;
  int sh_max;
  double lc2;
  int *c_k;
  T *c_x, *c_y, *c_z, *c_g1, *c_g2;
  v4<T> *LRR, *LZZ, *LP0, *LP1, *DR;
  // iEL/0-SCF shadow energy: delta (Dl) and the reciprocal potential of delta alone (Phi2);
  // iel_keep = 1 - 1/omega for pairs inside a preconditioner block when iel_keep_on
  const v4<T> *Dl;
  const T *Phi2;
  double iel_keep;
  int iel_keep_on;
  // vectors
  v4<T> *X, *R, *Z, *P, *AP, *B, *D;
  v4<T> *F;  // row field of a sweep (computed concurrently with the PME chain)
  v4<T> *Fp; // the early-fork schedule: row field of the previous CG direction
  // grids
  T *Q, *Phi, *Ginf;
  c2<T> *C;
  const c2<T> *tw;
  const double *bmod;
  // outputs of the energy pass
  double *forces;
  double4 *dEdd;
};

// The system and atom of thread group `sub` of a block, and the end of the system's atoms.  With one system
// they follow from the block index and the kernel's arguments; the map and the system table would be two
// dependent loads at the head of every kernel of a latency-bound step (a load is 0.3 us from a cold L1).
struct Where {
  int s, i, end;
};
template <typename T>
__device__ __forceinline__ Where where(const Dev<T> &a, const int4 *map, int block, int per, int sub) {
  if (a.nsys == 1) return Where{0, block * per + sub, a.nt};
  const int4 m = map[block];
  return Where{m.x, m.y + sub, m.z};
}
template <typename T>
__device__ __forceinline__ int system_of(const Dev<T> &a, int i) { return a.nsys == 1 ? 0 : a.sysid[i]; }
// Whether a pass of the solve takes part in system s: act 0 always, 1 iterating, 2 plain start, 3 fallback.
template <typename T>
__device__ __forceinline__ bool solve_active(const Dev<T> &a, int s, int act) {
  return act == 0 || (act == 1 && a.cg[s].active) || (act == 2 && a.cg[s].sweep2) || (act == 3 && a.cg[s].fallback);
}
struct Mesh {
  int K1, K2, K3;
  long long r0;
};
template <typename T>
__device__ __forceinline__ Mesh mesh_of(const Dev<T> &a, int s) {
  if (a.nsys == 1) return Mesh{a.K0[0], a.K0[1], a.K0[2], 0};
  const SysInfo &S = a.sys[s];
  return Mesh{S.K[0], S.K[1], S.K[2], S.rgrid0};
}

// A chunk of 32 row entries: 32 each of k, x, y, z, G1, G2, G0, G3, so that a warp writes or reads
// every array of a chunk at constant offsets from one address (separate arrays took a 64-bit address each:
// a third of the row build's instructions) and the sweeps' six arrays are contiguous.
template <typename T>
struct RowChunk {
  static constexpr int SIZE = 32 * (4 + 7 * (int)sizeof(T));
  static constexpr int X = 128, Y = X + 32 * (int)sizeof(T), Z = Y + 32 * (int)sizeof(T), G1 = Z + 32 * (int)sizeof(T),
                       G2 = G1 + 32 * (int)sizeof(T), G0 = G2 + 32 * (int)sizeof(T), G3 = G0 + 32 * (int)sizeof(T);
};
template <typename T>
__device__ __forceinline__ unsigned char *row_of(const Dev<T> &a, int i) {
  return a.rows + (size_t)i * (a.mc >> 5) * RowChunk<T>::SIZE;
}
// Entry t of a row: its k (AT = 0) and the T values at RowChunk offset AT.
template <typename T>
__device__ __forceinline__ unsigned char *row_entry(unsigned char *row, int t) {
  return row + (size_t)(t >> 5) * RowChunk<T>::SIZE;
}
template <typename T>
__device__ __forceinline__ int &entry_k(unsigned char *chunk, int t) { return reinterpret_cast<int *>(chunk)[t & 31]; }
template <typename T, int AT>
__device__ __forceinline__ T &entry_v(unsigned char *chunk, int t) { return reinterpret_cast<T *>(chunk + AT)[t & 31]; }

// ------------------------------------------------------------------ box and per-atom set-up
// Box-dependent values of system s (every block of the system computes its own copy; the system's first
// block, `first`, publishes them and starts the step's status word).
template <typename T>
__device__ __forceinline__ void box_setup(Dev<T> &a, int s, const double *H, BoxInfo &B, bool first) {
  const SysInfo &S = a.sys[s];
  const double d = H[0] * (H[4] * H[8] - H[5] * H[7]) - H[1] * (H[3] * H[8] - H[5] * H[6]) + H[2] * (H[3] * H[7] - H[4] * H[6]);
  double *Hi = B.Hinv;  // cofactor inverse (box.py:195-234)
  Hi[0] = (H[4] * H[8] - H[5] * H[7]) / d; Hi[1] = (H[2] * H[7] - H[1] * H[8]) / d; Hi[2] = (H[1] * H[5] - H[2] * H[4]) / d;
  Hi[3] = (H[5] * H[6] - H[3] * H[8]) / d; Hi[4] = (H[0] * H[8] - H[2] * H[6]) / d; Hi[5] = (H[2] * H[3] - H[0] * H[5]) / d;
  Hi[6] = (H[3] * H[7] - H[4] * H[6]) / d; Hi[7] = (H[1] * H[6] - H[0] * H[7]) / d; Hi[8] = (H[0] * H[4] - H[1] * H[3]) / d;
  for (int k = 0; k < 9; ++k) B.H[k] = H[k];
  if (!first) return;
  B.vol = fabs(d);
  for (int c = 0; c < 3; ++c) B.idiag[c] = 1.0 / H[4 * c];
  for (int ax = 0; ax < 3; ++ax) {
    // plane height h_a = 1 / |column a of H^-1|
    double c0 = Hi[0 * 3 + ax], c1 = Hi[1 * 3 + ax], c2v = Hi[2 * 3 + ax];
    B.h[ax] = 1.0 / sqrt(c0 * c0 + c1 * c1 + c2v * c2v);
    const int nc = S.nc[ax];
    const double R = ceil((a.cutoff + a.skin) * nc / B.h[ax] - 1e-12);
    B.R[ax] = R >= 0.0 && 2.0 * R + 1.0 < nc ? (int)R : -1;  // -1: all cells (a degenerate box: R infinite or NaN)
  }
  int changed = 0;
  for (int k = 0; k < 9; ++k) changed |= (a.box[s].H[k] != H[k]);
  B.changed = changed;
  if (changed) atomicOr(a.nb_flag, 1);
  int bad = (fabs(H[1]) > 1e-12 * fabs(H[0])) || (fabs(H[2]) > 1e-12 * fabs(H[0])) || (fabs(H[5]) > 1e-12 * fabs(H[0])) ||
            !(H[0] > 0 && H[4] > 0 && H[8] > 0);
  double mc = 0.5 * fmin(H[0], fmin(H[4], H[8]));
  if (a.cutoff > mc) bad = 1;
  B.bad = bad;
  a.box[s] = B;
  a.status[s] = bad ? 0x8u : 0u;
  if (s == 0) { a.max_count[0] = 0; a.max_count[1] = 0; }  // the step's largest row counts start here
}

// The step's set-up in one launch (thread per atom): the box, fractional coordinates, spline base and offset
// (pme.py:269-304), permanent dipoles (forcefield.py:1032-1042), the list's displacement test, and, on the
// thread of a molecule's first atom, the offsets of its atoms from its centre of mass (the molecule made
// whole from its first atom), for the molecular virial.  A non-finite position is marked in base.w (the
// status word is being started by another block) and reported by the force pass.  Small kernels are bound by
// their launch: this and the merges of the start, finish and energy kernels took an MD step of 512 waters from 256 to
// 249 us, 24 boxes of 216 to 1,000 waters 2 % down.
template <typename T>
__global__ void k_prep(Dev<T> a, const double *boxes) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  __shared__ BoxInfo B;
  const Where w = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = w.s, i = w.i;
  const SysInfo &S = a.sys[s];
  if (threadIdx.x == 0) box_setup(a, s, boxes + 9 * (size_t)s, B, i == S.atom0);
  __syncthreads();
  if (i >= w.end) return;
  double px = a.pos[3 * i], py = a.pos[3 * i + 1], pz = a.pos[3 * i + 2];
  double uc[3];
  int4 b;
  v4<T> f;
  int bb[3];
  T ff[3];
  bool finite = true;
  for (int ax = 0; ax < 3; ++ax) {
    double u = px * B.Hinv[0 * 3 + ax] + py * B.Hinv[1 * 3 + ax] + pz * B.Hinv[2 * 3 + ax];
    double fr = u - floor(u);
    if (!(fr >= 0.0 && fr < 1.0)) { fr = 0.0; finite = false; }  // non-finite position: keep indices in range
    uc[ax] = fr;
    double w = fr * S.K[ax];
    double fl = floor(w);
    int bv = (int)fl;
    if (bv >= S.K[ax]) bv -= S.K[ax];  // w rounded up to K: grid point K is point 0
    if (bv < 0) bv = 0;
    bb[ax] = bv;
    ff[ax] = T(w - fl);
  }
  b.x = bb[0]; b.y = bb[1]; b.z = bb[2]; b.w = finite ? 0 : 1;
  f.x = ff[0]; f.y = ff[1]; f.z = ff[2]; f.w = T(0);
  a.base[i] = b;
  a.frac[i] = f;
  double4 p = make_double4(0, 0, 0, 0);
  if (a.perm) {
    for (int c = a.cov_start[i]; c < a.cov_start[i + 1]; ++c) {
      int j = a.cov_j[c];
      double vx = a.pos[3 * j] - px, vy = a.pos[3 * j + 1] - py, vz = a.pos[3 * j + 2] - pz;
      min_image(vx, vy, vz, B.H);
      double l = sqrt(vx * vx + vy * vy + vz * vz);
      double cc = a.cov_c[c] / l;
      p.x += cc * vx; p.y += cc * vy; p.z += cc * vz;
    }
  }
  a.pperm[i] = p;
  a.pos4[i] = make_double4(px, py, pz, (double)a.molid[i]);
  if (a.pos4f) {  // wrapped: |coordinates| below the box's, so FP32 keeps displacements to ~1e-6 nm
    double w[3];
    for (int c = 0; c < 3; ++c) w[c] = uc[0] * B.H[0 * 3 + c] + uc[1] * B.H[1 * 3 + c] + uc[2] * B.H[2 * 3 + c];
    a.pos4f[i] = make_float4(float(w[0]), float(w[1]), float(w[2]), float(a.molid[i]));
  }
  // Verlet list: rebuild when an atom moved more than skin / 2 since the last build
  double4 r0 = a.pos_ref[i];
  double dx = px - r0.x, dy = py - r0.y, dz = pz - r0.z;
  min_image(dx, dy, dz, B.H);
  double h2 = 0.25 * a.skin * a.skin;
  if (!(dx * dx + dy * dy + dz * dz <= h2)) atomicOr(a.nb_flag, 1);
  const int i0 = a.molfirst[i], i1 = a.molend[i];
  if (i != i0) return;
  double cx = 0, cy = 0, cz = 0, mt = 0;
  for (int j = i0; j < i1; ++j) {
    double vx = a.pos[3 * j] - px, vy = a.pos[3 * j + 1] - py, vz = a.pos[3 * j + 2] - pz;
    min_image(vx, vy, vz, B.H);
    a.off[j] = make_double4(vx, vy, vz, 0);
    cx += a.mass[j] * vx; cy += a.mass[j] * vy; cz += a.mass[j] * vz; mt += a.mass[j];
  }
  cx /= mt; cy /= mt; cz /= mt;
  for (int j = i0; j < i1; ++j) {
    double4 o = a.off[j];
    a.off[j] = make_double4(o.x - cx, o.y - cy, o.z - cz, 0);
  }
}

// Cell of every atom (only when the candidate list is rebuilt).
template <typename T>
__global__ void k_cell_assign(Dev<T> a) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  if (!*a.nb_flag) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  int s = system_of(a, i);
  const SysInfo &S = a.sys[s];
  const BoxInfo &B = a.box[s];
  double4 p = a.pos4[i];
  double uc[3];
  for (int ax = 0; ax < 3; ++ax) {
    double u = p.x * B.Hinv[0 * 3 + ax] + p.y * B.Hinv[1 * 3 + ax] + p.z * B.Hinv[2 * 3 + ax];
    double fr = u - floor(u);
    if (!(fr >= 0.0 && fr < 1.0)) fr = 0.0;
    uc[ax] = fr;
  }
  int c0 = max(0, min((int)(uc[0] * S.nc[0]), S.nc[0] - 1));
  int c1 = max(0, min((int)(uc[1] * S.nc[1]), S.nc[1] - 1));
  int c2v = max(0, min((int)(uc[2] * S.nc[2]), S.nc[2] - 1));
  int cell = S.cell0 + (c0 * S.nc[1] + c1) * S.nc[2] + c2v;
  a.cell_of[i] = cell;
  a.slot_of[i] = atomicAdd(&a.cell_count[cell], 1);
}

// Exclusive scan of the cell counts of all systems (one block), which are cleared for the next rebuild.
__global__ void k_scan_cells(int *count, int *start, int n, const int *flag) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  if (!*flag) return;
  __shared__ int part[1024];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    int i = base + threadIdx.x;
    int v = i < n ? count[i] : 0;
    if (v) count[i] = 0;
    part[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      int t = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
      __syncthreads();
      part[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < n) start[i] = carry + part[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += part[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) start[n] = carry;
}

template <typename T>
__global__ void k_scatter(Dev<T> a) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  if (!*a.nb_flag) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  int t = a.cell_start[a.cell_of[i]] + a.slot_of[i];
  a.cell_atoms[t] = i;
  if constexpr (sizeof(T) == 4) a.spos[t] = a.pos4f[i];
  else a.spos[t] = a.pos4[i];
}

// FP32 sequential minimum image (the mixed-precision candidate list and row build).  Rounding to the
// nearest integer by adding and subtracting 1.5 2^23 (wrapped positions: |argument| < 2): two
// additions, where rintf is a conversion at a quarter of their rate.
__device__ __forceinline__ float nearest_f(float x) { return __fadd_rn(__fadd_rn(x, 12582912.f), -12582912.f); }
__device__ __forceinline__ void min_image_scan(double &x, double &y, double &z, const double *H, const double *id) {
  min_image_fast(x, y, z, H, id);
}
__device__ __forceinline__ void min_image_scan(float &x, float &y, float &z, const float *H, const float *id) {
  float n = nearest_f(z * id[2]);
  x -= n * H[6]; y -= n * H[7]; z -= n * H[8];
  n = nearest_f(y * id[1]);
  x -= n * H[3]; y -= n * H[4];
  n = nearest_f(x * id[0]);
  x -= n * H[0];
}

// ------------------------------------------------------------------ Verlet candidate list
// One warp per atom when the list is rebuilt: every atom of another molecule within
// cutoff + skin, found through the cell list (cells within R along each axis), compacted by ballot;
// the positions of the build are kept for the displacement test (the reference's neighbour list,
// md/neighbors.py:169-304, rebuilt when an atom moved more than skin / 2).  The lanes look up the
// ranges of 32 cell columns at once (a column's range is a load that its atoms' loads wait for); mixed
// precision tests FP32 displacements against a radius wider by their error, which grows with the box.  A rectangular
// box trims the columns and their ranges to the sphere.  Latency of dependent loads bounds it: a rebuild took 1724 us
// at 98,304 atoms and 239 at 12,288 with a column at a time in FP64 over the cube of cells, 525 and 77 so.
template <typename T>
__global__ void __launch_bounds__(256) k_cand(Dev<T> a) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  if (!*a.nb_flag) return;
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Where at = where(a, a.wb, blockIdx.x, WARPS_PER_BLOCK, warp);
  const int s = at.s, i = at.i;
  if (i >= at.end) return;
  const SysInfo &S = a.sys[s];
  const BoxInfo &B = a.box[s];
  T H[9], id[3];
#pragma unroll
  for (int k = 0; k < 9; ++k) H[k] = T(B.H[k]);
  id[0] = T(B.idiag[0]); id[1] = T(B.idiag[1]); id[2] = T(B.idiag[2]);
  v4<T> pi;
  if constexpr (sizeof(T) == 4) pi = a.pos4f[i];
  else pi = a.pos4[i];
  // W: the largest coordinate of a wrapped position.  A displacement of two of them in FP32 is off by less than
  // 12 W 2^-24 a component (both positions, three lattice vectors and the subtractions), 1.3e-6 W in length; the
  // square's rounding is below 1e-6 of it.  At most a tenth of the radius: above 8e4 nm FP32 positions resolve less
  // than that, and the list must not outgrow its capacity for them.
  const double W = fmax(fabs(B.H[0]) + fabs(B.H[3]) + fabs(B.H[6]), fmax(fabs(B.H[4]) + fabs(B.H[7]), fabs(B.H[8])));
  const double r0 = a.cutoff + a.skin, rl = sizeof(T) == 4 ? r0 * (1.0 + 1e-6) + fmin(1.3e-6 * W, 0.1 * r0) : r0;
  const T rl2 = T(rl * rl);
  int *out = a.cand + (size_t)i * a.cc;
  int count = 0;
  int cell = a.cell_of[i] - S.cell0;
  int n0 = S.nc[0], n1 = S.nc[1], n2 = S.nc[2];
  int ci2 = cell % n2, ci1 = (cell / n2) % n1, ci0 = cell / (n1 * n2);
  int R0 = B.R[0], R1 = B.R[1], R2 = B.R[2];
  int lo0 = R0 < 0 ? 0 : -R0, hi0 = R0 < 0 ? n0 - 1 : R0;
  int lo1 = R1 < 0 ? 0 : -R1, hi1 = R1 < 0 ? n1 - 1 : R1;
  const int nd1 = hi1 - lo1 + 1, ncol = (hi0 - lo0 + 1) * nd1;
  // rectangular boxes: a column is as far as the nearest edge of its nearest image, and its range is what that
  // leaves of the radius (a quarter of the cube of cells that the index ranges span); cw: cell widths, fc: the
  // atom in its cell; reach: the radius with room for the rounding of these
  const bool rect = B.H[3] == 0.0 && B.H[6] == 0.0 && B.H[7] == 0.0;
  const T reach2 = T((rl + 1e-4 + 1e-6 * W) * (rl + 1e-4 + 1e-6 * W));  // a place along an axis: 2.4e-7 W in FP32
  auto in_cell = [](T u, int n, int ci) {
    const T f = (u - floor(u)) * T(n) - T(ci);
    return f < T(-0.5) ? f + T(n) : f > T(1.5) ? f - T(n) : f;
  };
  const T cw0 = T(B.H[0] / n0), cw1 = T(B.H[4] / n1), cw2 = T(B.H[8] / n2);
  const T fc0 = in_cell(pi.x * id[0], n0, ci0), fc1 = in_cell(pi.y * id[1], n1, ci1), fc2 = in_cell(pi.z * id[2], n2, ci2);
  auto gap = [](int d, int n, T f) {  // cells between the atom and a column d cells away, of its images the nearest
    d = d > n / 2 ? d - n : d < -(n / 2) ? d + n : d;
    const T up = d > 0 ? T(d) - f : T(d + n) - f, down = d < 0 ? f - T(d + 1) : f - T(d - n + 1);
    return d == 0 ? T(0) : min(up, down);
  };
  for (int cb = 0; cb < ncol; cb += 32) {
    // this lane's column: its one or two ranges along the third axis, in cell order
    int b0 = 0, l0 = 0, b1 = 0, l1 = 0;
    const int c = cb + lane;
    if (c < ncol) {
      const int d0 = lo0 + c / nd1, d1 = lo1 + c % nd1;
      const int c0 = R0 < 0 ? d0 : ((ci0 + d0) % n0 + n0) % n0, c1 = R1 < 0 ? d1 : ((ci1 + d1) % n1 + n1) % n1;
      const int *st = a.cell_start + S.cell0 + (c0 * n1 + c1) * n2;
      int lo = R2 < 0 ? 0 : ci2 - R2, hi = R2 < 0 ? n2 - 1 : ci2 + R2;
      bool reach = true;
      if (rect) {
        const T g0 = gap(c0 - ci0, n0, fc0) * cw0, g1 = gap(c1 - ci1, n1, fc1) * cw1;
        const T left = reach2 - g0 * g0 - g1 * g1;
        reach = left >= T(0);
        if (reach) cells_within(fc2, T(sqrt(left) / cw2), ci2, n2, lo, hi);
      }
      if (reach) {
        const CellRange z = wrapped_cells(lo, hi, n2);
        if (z.hi2 >= 0) { b1 = st[0]; l1 = st[z.hi2 + 1] - b1; }
        b0 = st[z.lo]; l0 = st[z.hi + 1] - b0;
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, l0 + l1 > 0); todo; todo &= todo - 1) {
      const int k = __ffs(todo) - 1;
      const int f0 = __shfl_sync(0xffffffffu, b0, k), m0 = __shfl_sync(0xffffffffu, l0, k);
      const int f1 = __shfl_sync(0xffffffffu, b1, k), tot = m0 + __shfl_sync(0xffffffffu, l1, k);
      for (int t0 = 0; t0 < tot; t0 += 32) {
        const int u = t0 + lane, t = u < m0 ? f0 + u : f1 + u - m0;
        bool keep = false;
        if (u < tot) {
          const v4<T> pj = a.spos[t];
          if (pj.w != pi.w) {
            T x = pi.x - pj.x, y = pi.y - pj.y, z = pi.z - pj.z;
            min_image_scan(x, y, z, H, id);
            keep = x * x + y * y + z * z < rl2;
          }
        }
        unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          int slot = count + __popc(bal & ((1u << lane) - 1u));
          if (slot < a.cc) out[slot] = a.cell_atoms[t];
        }
        count += __popc(bal);
      }
    }
  }
  if (lane == 0) {
    a.ncand[i] = count;
    a.pos_ref[i] = a.pos4[i];
    if (count > a.cc) atomicOr(&a.status[s], 0x10u);
  }
}

// ------------------------------------------------------------------ pair rows
// k_rows: one warp per atom finds the row -- the molecule partners (always kept inside the cutoff;
// the rigid special table of md/topology.py:161-178), then the candidates of the Verlet list (or
// the caller's rows), masked to r < rc (forcefield.py:1140-1195).  Kept entries go through a queue of
// the warp in shared memory; whenever 32 are waiting the warp evaluates their radial kernels
// (pair_kernels), every lane busy, and writes k, x, y, z, G0..G3 with them, contiguous over the lanes,
// and the local preconditioner's short entries and the learned guess's graph edges.
// Bound by issue (77 % of the slots at 12,288 atoms; DRAM 20 %, L1 52 %, a warp waits for a load 1.2 of its 9.0 cycles
// an instruction): the scan alone takes 137 of 232 us at 59,049 atoms (FP32; 305 with rows in eight arrays and a
// round that waited for its loads; 378 of 494 at 98,304, 57 of 78 at 12,288; FP64 127 of 147).  3 or 5 blocks per SM
// are slower (309, 296 against 272 at the time); four leave 64 registers, 64 bytes of spills.

// An atom's group of LPA lanes (32: the warp; 16, 8: a half, a quarter warp): its shuffle mask, and the sum over
// it (the warp's own reduction for a whole warp).
template <int LPA>
__device__ __forceinline__ unsigned group_mask() {
  if constexpr (LPA == 32) return 0xffffffffu;
  else return ((1u << LPA) - 1u) << ((threadIdx.x & 31) & ~(LPA - 1));
}
template <typename T, int LPA>
__device__ __forceinline__ T group_sum(T v, unsigned m) {
  if constexpr (LPA == 32) {
    return warp_sum<T>(v);
  } else {
#pragma unroll
    for (int o = LPA / 2; o > 0; o >>= 1) v += __shfl_xor_sync(m, v, o);
    return v;
  }
}

// The row scan of atom i by its warp: the molecule partners (special = true), then the
// candidates, two entries per lane and round; the indices two rounds ahead and the positions one round ahead
// are in flight while the current ones are tested (a round that waited for its indices and then for
// their positions took 1900 cycles on 32 resident warps).  visit(keep, j, x, y, z, special) runs on all
// lanes for every 32 entries (it may use the warp's collectives), then round() after every round; keep is
// r < rc for an entry of another atom, false on lanes without one; the displacement
// comes as T, as the rows store it.  Mixed precision: the candidates' FP32 displacements from the wrapped
// FP32 positions (16-byte gathers), the molecule partners' rounded from FP64.
template <typename T, typename Visit, typename Round>
__device__ __forceinline__ void row_scan(const Dev<T> &a, const SysInfo &S, const BoxInfo &B, int i, int lane, Visit &&visit,
                                         Round &&round) {
  double H[9], id[3];
#pragma unroll
  for (int k = 0; k < 9; ++k) H[k] = B.H[k];
  id[0] = B.idiag[0]; id[1] = B.idiag[1]; id[2] = B.idiag[2];
  // the caller's candidate rows (local indices, padding natom), or the engine's Verlet candidates (within
  // cutoff + skin at the last rebuild)
  const bool own = a.idx == nullptr;
  const int *row = own ? a.cand + (size_t)i * a.cc : a.idx + (size_t)i * a.idx_width;
  const int nc = own ? min(a.ncand[i], a.cc) : a.idx_width;
  const int first = own ? 0 : S.atom0, limit = own ? a.nt : S.natom;
  auto index = [&](int c) { return c < nc ? row[c] : -1; };  // as stored: nothing waits for the load here
  auto partner = [&](int jl) { return jl >= 0 && jl < limit ? jl + first : -1; };
  constexpr int U = 2;
  int jn[U], l2[U];
#pragma unroll
  for (int u = 0; u < U; ++u) { jn[u] = index(32 * u + lane); l2[u] = index(32 * (U + u) + lane); }
  const double4 pi = a.pos4[i];
  const double rc2 = a.cutoff * a.cutoff;
  const int mf = a.molfirst[i], me = a.molend[i];
  for (int j0 = mf; j0 < me; j0 += 32) {
    int j = j0 + lane;
    bool keep = false;
    double x = 0, y = 0, z = 0;
    if (j < me && j != i) {
      double4 pj = a.pos4[j];
      x = pi.x - pj.x; y = pi.y - pj.y; z = pi.z - pj.z;
      min_image_fast(x, y, z, H, id);
      keep = x * x + y * y + z * z < rc2;
    }
    visit(keep, j, T(x), T(y), T(z), true);
    round();
  }
  // positions in the scan's precision, .w the molecule
  const v4<T> *pos;
  T Ht[9], idt[3];
  if constexpr (sizeof(T) == 4) pos = a.pos4f;
  else pos = a.pos4;
#pragma unroll
  for (int k = 0; k < 9; ++k) Ht[k] = T(H[k]);
  idt[0] = T(id[0]); idt[1] = T(id[1]); idt[2] = T(id[2]);
  const v4<T> p0 = pos[i];
  const T rc2t = T(rc2);
  v4<T> pn[U];
#pragma unroll
  for (int u = 0; u < U; ++u) { jn[u] = partner(jn[u]); pn[u] = pos[jn[u] >= 0 ? jn[u] : i]; }
  for (int c0 = 0; c0 < nc; c0 += 32 * U) {
    int j[U];
    v4<T> pj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      j[u] = jn[u];
      pj[u] = pn[u];
      jn[u] = partner(l2[u]);
      l2[u] = index(c0 + 32 * (2 * U + u) + lane);
      pn[u] = pos[jn[u] >= 0 ? jn[u] : i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      T x = p0.x - pj[u].x, y = p0.y - pj[u].y, z = p0.z - pj[u].z;
      min_image_scan(x, y, z, Ht, idt);
      // a lane without a candidate holds atom i itself: its own molecule
      visit(j[u] >= 0 && pj[u].w != p0.w && x * x + y * y + z * z < rc2t, j[u], x, y, z, false);
    }
    round();
  }
}

// Kept entries waiting for their evaluation (ring; at most 95 at a time: 31 and a round's 64).
template <typename T>
struct RowQueue {
  int j[128];
  T x[128], y[128], z[128];
};

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) k_rows(Dev<T> a) {
  __shared__ RowQueue<T> queues[WARPS_PER_BLOCK];
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Where at = where(a, a.wb, blockIdx.x, WARPS_PER_BLOCK, warp);
  const int s = at.s, i = at.i;
  if (i >= at.end) return;
  const SysInfo &S = a.sys[s];
  RowQueue<T> &q = queues[warp];
  const unsigned lt = (1u << lane) - 1u;
  const T Ri2 = T(2) * a.radius[i] * a.radius[i], beta = T(a.beta);
  unsigned char *row = row_of(a, i);
  int head = 0, tail = 0, ecount = 0, vcount = 0, scount = 0, nsp = 0;  // head: evaluated, tail: found
  auto evaluate = [&](int n) {  // the next n <= 32 entries of the queue, to row slots head .. head + n - 1
    const int w = (head + lane) & 127, slot = head + lane;
    const bool in = lane < n && slot < a.mce;
    const int j = in ? q.j[w] : i;
    const T x = q.x[w], y = q.y[w], z = q.z[w];
    const T Rk = a.radius[j];
    const T r2 = x * x + y * y + z * z;
    bool sh = false, ed = false;
    int at_s = 0, at_e = 0;
    if (a.sh_n) {  // the local preconditioner's entries: partner, displacement, G1, G2, entry-major
      sh = in && r2 < T(a.lc2);
      const unsigned sb = __ballot_sync(0xffffffffu, sh);
      at_s = scount + __popc(sb & lt);
      scount += __popc(sb);
      sh = sh && at_s < a.sh_max;
    }
    if (a.nn_e4) {  // the learned guess's graph edges: the entries closer than rg, with G1, G2
      ed = in && float(r2) < a.nn_rg2;
      const unsigned eb = __ballot_sync(0xffffffffu, ed);
      at_e = ecount + __popc(eb & lt);
      ecount += __popc(eb);
      ed = ed && at_e < a.nn_emax;
    }
    if (in) {
      using C = RowChunk<T>;
      unsigned char *chunk = row_entry<T>(row, head);  // head is a multiple of 32
      entry_k<T>(chunk, lane) = j;
      entry_v<T, C::X>(chunk, lane) = x; entry_v<T, C::Y>(chunk, lane) = y; entry_v<T, C::Z>(chunk, lane) = z;
      T g[4];
      pair_kernels<T>(Ri2 + T(2) * Rk * Rk, beta, r2, g);
      entry_v<T, C::G1>(chunk, lane) = g[1]; entry_v<T, C::G2>(chunk, lane) = g[2];
      entry_v<T, C::G0>(chunk, lane) = g[0]; entry_v<T, C::G3>(chunk, lane) = g[3];
      if (sh) {
        const size_t c = (size_t)at_s * a.nt + i;
        a.c_k[c] = j;
        a.c_x[c] = x; a.c_y[c] = y; a.c_z[c] = z;
        a.c_g1[c] = g[1]; a.c_g2[c] = g[2];
      }
      if (ed) {
        const size_t e = (size_t)i * a.nn_emax + at_e;
        a.nn_e4[e] = make_float4(float(x), float(y), float(z), __int_as_float(j));
        a.nn_g[e] = make_float2(float(g[1]), float(g[2]));
      }
    }
    head += n;
  };
  row_scan<T>(a, S, a.box[s], i, lane, [&](bool keep, int j, T x, T y, T z, bool special) {
    if (a.rnv) {  // split rows: beyond elec_cutoff only pairs with an LJ term stay, in the row's second part
      bool kv = false;
      if (keep && !(x * x + y * y + z * z < T(a.rce2))) {
        kv = !special && j >= 0 && a.seps[i] * a.seps[j] != T(0);  // molecule partners have LJ weight 0
        keep = false;
      }
      const unsigned bv = __ballot_sync(0xffffffffu, kv);
      const int sv = vcount + __popc(bv & lt);
      if (kv && sv < a.mc - a.mce) {
        using C = RowChunk<T>;
        const int t = a.mce + sv;
        unsigned char *chunk = row_entry<T>(row, t);
        entry_k<T>(chunk, t) = j;
        entry_v<T, C::X>(chunk, t) = x; entry_v<T, C::Y>(chunk, t) = y; entry_v<T, C::Z>(chunk, t) = z;
      }
      vcount += __popc(bv);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int w = (tail + __popc(bal & lt)) & 127;
      q.j[w] = j;
      q.x[w] = x; q.y[w] = y; q.z[w] = z;
    }
    tail += __popc(bal);
    if (special) nsp = tail;
  }, [&] {
    if (tail - head < 32) return;
    __syncwarp();  // the queue's entries, stored by other lanes
    do evaluate(32); while (tail - head >= 32);
    __syncwarp();  // read before their slots are filled again
  });
  __syncwarp();
  if (tail > head) evaluate(tail - head);
  if (lane == 0) {
    a.rn[i] = tail;
    a.rnsp[i] = nsp;
    if (a.nn_e4) a.nn_ne[i] = ecount;
    if (a.sh_n) {
      a.sh_n[i] = min(scount, a.sh_max);
      if (scount > a.sh_max) atomicOr(&a.status[s], 0x20u);  // the preconditioner kept the first sh_max
    }
    if (tail > a.mce) atomicOr(&a.status[s], 0x1u);
    if (tail > __ldca(a.max_count)) atomicMax(a.max_count, tail);  // a stale count only costs an atomic
    if (a.rnv) {
      a.rnv[i] = vcount;
      if (vcount > a.mc - a.mce) atomicOr(&a.status[s], 0x1u);
      if (vcount > __ldca(a.max_count + 1)) atomicMax(a.max_count + 1, vcount);
    }
  }
}

// ------------------------------------------------------------------ PME influence function
// G(m) = exp(-pi^2 |m*|^2 / beta^2) / (2 pi V |m*|^2) / (b1 b2 b3), 0 at m = 0 (pme.py:243-267),
// on the half spectrum, computed in FP64, stored in T; recomputed only when the box changed.
// Two closing jobs of the row build ride in the launch: a rebuild of the candidate list is counted and its flag
// lowered, and in mixed precision the molecule partners' kernels are evaluated again in FP64 and rounded once.  Their
// pairs carry most of the energy at distances that a rigid molecule never changes, so a rounding error of theirs is a
// bias: the energy of a water box at zero induced dipoles was 7.2 to 8.2e-8 off with all kernels in FP32, 4.9e-8 with
// this (3.1e-8 now, without the rounded charge products of the force pass; 2.6e-8 is the rounding of the parameters
// to FP32).  Cost: 4 us at 12,288 atoms of water, none seen at 59,049; in the row build, where a warp would run it
// for a few lanes, 12 us of 57 and 58 us of 230.
// An atom's partners go to two threads up to FEW of them (a water has two), to 32 threads above: an evaluation is
// 0.5 us of dependent FP64 arithmetic.  A call at given dipoles on 1,536 atoms in molecules of 256: 221 us with two
// threads for every atom, 155 so; one molecule of 201 atoms in 98,304 atoms of water: 924 with two, 980 with 32 for
// every atom, 910 so.  big: the nbig atoms of molecules large enough for more than FEW.
constexpr int FEW = 8;
template <typename T>
__global__ void k_influence(Dev<T> a, long long total, const int *big, int nbig) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  if (blockIdx.x == 0 && threadIdx.x == 0 && !a.idx && *a.nb_flag) { *a.nb_flag = 0; *a.nb_builds += 1; }
  if constexpr (sizeof(T) == 4) {
    using C = RowChunk<T>;
    const long long many = 32ll * nbig;
    for (long long u = blockIdx.x * blockDim.x + threadIdx.x; u < many + 2ll * a.nt; u += gridDim.x * blockDim.x) {
      const bool wide = u < many;
      const int i = wide ? big[u >> 5] : (int)((u - many) >> 1), step = wide ? 32 : 2;
      const int n = min(a.rnsp[i], a.mce);
      if ((n > FEW) != wide) continue;  // the other part's
      unsigned char *row = row_of(a, i);
      const T Ri = a.radius[i];
      for (int t = (int)(wide ? u : u - many) & (step - 1); t < n; t += step) {
        unsigned char *c = row_entry<T>(row, t);
        const T Rk = a.radius[entry_k<T>(c, t)], x = entry_v<T, C::X>(c, t), y = entry_v<T, C::Y>(c, t), z = entry_v<T, C::Z>(c, t);
        double g[4];
        pair_kernels<double>(2.0 * (double(Ri) * double(Ri) + double(Rk) * double(Rk)), a.beta,
                             double(x) * double(x) + double(y) * double(y) + double(z) * double(z), g);
        entry_v<T, C::G0>(c, t) = T(g[0]); entry_v<T, C::G1>(c, t) = T(g[1]);
        entry_v<T, C::G2>(c, t) = T(g[2]); entry_v<T, C::G3>(c, t) = T(g[3]);
      }
    }
  }
  int any = 0;
  for (int s = threadIdx.x; s < a.nsys; s += blockDim.x) any |= a.box[s].changed;
  if (!__syncthreads_or(any)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x) {
    int s = 0;
    while (s + 1 < a.nsys && a.sys[s + 1].cgrid0 <= g) ++s;
    const SysInfo &S = a.sys[s];
    const BoxInfo &B = a.box[s];
    if (!B.changed) continue;
    long long l = g - S.cgrid0;
    if (l >= (long long)S.K[0] * S.K[1] * S.K3h) continue;  // alignment gap between systems
    int m3 = (int)(l % S.K3h);
    long long t = l / S.K3h;
    int k2 = (int)(t % S.K[1]), k1 = (int)(t / S.K[1]);
    int m1 = k1 <= (S.K[0] - 1) / 2 ? k1 : k1 - S.K[0];
    int m2 = k2 <= (S.K[1] - 1) / 2 ? k2 : k2 - S.K[1];
    if (S.K[0] % 2 == 0 && k1 == S.K[0] / 2) m1 = -S.K[0] / 2;
    if (S.K[1] % 2 == 0 && k2 == S.K[1] / 2) m2 = -S.K[1] / 2;
    double mv[3];
    for (int c = 0; c < 3; ++c) mv[c] = m1 * B.Hinv[c * 3 + 0] + m2 * B.Hinv[c * 3 + 1] + m3 * B.Hinv[c * 3 + 2];
    double msq = mv[0] * mv[0] + mv[1] * mv[1] + mv[2] * mv[2];
    double G = 0.0;
    if (msq > 0) {
      G = exp(-PI * PI * msq / (a.beta * a.beta)) / (2.0 * PI * B.vol * msq);
      G /= a.bmod[S.mod0[0] + k1] * a.bmod[S.mod0[1] + k2] * a.bmod[S.mod0[2] + m3];
    }
    a.Ginf[g] = T(G);
  }
}

// ------------------------------------------------------------------ spline stencils
// The PME kernels give an atom QL = 8 lanes (four atoms per warp, 32 per block).  The P x P stencil rows along
// k3 are taken SLOTS at a time, a row's points as GPL aligned vectors of VW (16 bytes where K3 allows it, else
// two points), one lane each: the vectors of a row sit side by side, so a warp's request touches 16 rows in whole
// sectors, and a lane's k3 weights stay in registers for all rows.  What bounds them is load latency (8 of a gather's 14
// cycles an instruction, 6 of a spread's 14, at 30 % of the warps) and then L1 (44 and 55 %): with one point or vector
// per lane and the k3 weights read from shared memory for every point, a row cost three times the instructions.
// At 98,304 atoms, 192^3: gather 59.5 -> 37.0 us, spread 43.2 -> 38.9; at 59,049 atoms 31.0 -> 22.6 and 25.5 -> 24.7
// (the spread keeps its vector atomics; L2 takes them in 20 % of its cycles).
constexpr int QL = 8, ATOMS_PER_BLOCK = 32;
template <typename T, int VW> struct VecOf;
template <> struct VecOf<float, 4> { using type = float4; };
template <> struct VecOf<float, 2> { using type = float2; };
template <> struct VecOf<double, 2> { using type = double2; };

template <int P, int VW>
struct Stencil {
  static constexpr int GPL = VW == 4 ? 2 : 4, SLOTS = QL / GPL, ROUNDS = P * P / SLOTS;
  static constexpr int NG = (VW + P - 2) / VW + 1;    // most vectors of a row
  static constexpr int NQ = (NG + GPL - 1) / GPL;     // per lane
  static_assert(P * P % SLOTS == 0 && SLOTS <= P, "rows in whole rounds");
};

// A lane's vectors of a row: their k3 weights (0 outside the stencil), places along k3 and whether they are needed.
template <typename T, int P, int VW, int NW>
struct RowVectors {
  static constexpr int NQ = Stencil<P, VW>::NQ;
  T w[NW][NQ][VW];
  int at[NQ];
  bool on[NQ];
  // wk[n] (P values each): the weights along k3 and their derivatives, in shared memory
  __device__ __forceinline__ void set(int lane, int bz, int K3, const T *(&wk)[NW], int stride) {
    const int o = bz % VW, g0 = bz / VW, ng = (o + P - 1) / VW + 1, KV = K3 / VW;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int g = lane % Stencil<P, VW>::GPL + q * Stencil<P, VW>::GPL;
      on[q] = g < ng;
      at[q] = g0 + g < KV ? g0 + g : g0 + g - KV;
#pragma unroll
      for (int e = 0; e < VW; ++e) {
        const int j = VW * g + e - o;
#pragma unroll
        for (int n = 0; n < NW; ++n) w[n][q][e] = j >= 0 && j < P ? wk[n][j * stride] : T(0);
      }
    }
  }
};

// f(j1, j2, row) for the rows of a lane's slot; row = index of the row's first vector.
template <int P, int VW, int UNROLL, typename F>
__device__ __forceinline__ void for_rows(int lane, int4 b, int K1, int K2, int K3, F &&f) {
  using S = Stencil<P, VW>;
  int j1 = 0, j2 = lane / S::GPL;
  const int KV = K3 / VW;
#pragma unroll(UNROLL)
  for (int r = 0; r < S::ROUNDS; ++r) {
    int i1 = b.x + j1; if (i1 >= K1) i1 -= K1;
    int i2 = b.y + j2; if (i2 >= K2) i2 -= K2;
    f(j1, j2, (size_t)(i1 * K2 + i2) * KV);
    j2 += S::SLOTS;
    if (j2 >= P) { j2 -= P; ++j1; }
  }
}

__device__ __forceinline__ void add_vec(float *p, const float (&v)[4]) {
  atomicAdd(reinterpret_cast<float4 *>(p), make_float4(v[0], v[1], v[2], v[3]));
}
__device__ __forceinline__ void add_vec(float *p, const float (&v)[2]) {
  atomicAdd(reinterpret_cast<float2 *>(p), make_float2(v[0], v[1]));
}
__device__ __forceinline__ void add_vec(double *p, const double (&v)[2]) {
  if (v[0] != 0.0) atomicAdd(p, v[0]);
  if (v[1] != 0.0) atomicAdd(p + 1, v[1]);
}
template <typename T, int VW>
__device__ __forceinline__ void load_vec(const T *p, T (&v)[VW]) {
  const auto u = *reinterpret_cast<const typename VecOf<T, VW>::type *>(p);
  v[0] = u.x; v[1] = u.y;
  if constexpr (VW == 4) { v[2] = u.z; v[3] = u.w; }
}
// f(integral_constant VW) with the widest vector that the mesh allows (K3 is even; grids start 256-byte aligned)
template <typename T, typename F>
__device__ __forceinline__ void with_vec(int K3, F &&f) {
  if constexpr (sizeof(T) == 4) {
    if ((K3 & 3) == 0) { f(std::integral_constant<int, 4>{}); return; }
  }
  f(std::integral_constant<int, 2>{});
}

// ------------------------------------------------------------------ spread (pme.py:306-337)
// Vector atomic adds into the system's grid: the weight of a point is A(j1, j2) t3 + B(j1, j2) u3 with
// A = (q t1 + e1 u1) t2 + e2 t1 u2, B = e3 t1 t2.  With UPDATE_P the CG direction is first advanced,
// p = z + beta p (forcefield.py:1812), and spread.
template <typename T, int P, bool WITH_Q, bool UPDATE_P, int ACT>
__global__ void __launch_bounds__(ATOMS_PER_BLOCK * QL) k_spread(Dev<T> a, const v4<T> *__restrict__ vin) {
  pdl_enter();
  __shared__ c2<T> sh[ATOMS_PER_BLOCK][3][P];  // per atom of the block: weight and derivative
  const int sub = threadIdx.x / QL, lane = threadIdx.x % QL;  // the atom's group of lanes
  const unsigned gm = group_mask<QL>();
  const Where wh = where(a, a.qb, blockIdx.x, ATOMS_PER_BLOCK, sub);
  const int s = wh.s, i = wh.i;
  if (i >= wh.end) return;
  // the loads go out before the test of the system's flag
  const int4 b = a.base[i];
  const v4<T> f = a.frac[i];
  const v4<T> z = UPDATE_P ? a.Z[i] : vin[i], p = UPDATE_P ? a.P[i] : z;
  const Mesh M = mesh_of(a, s);
  if (!solve_active(a, s, ACT)) return;
  v4<T> d;
  if (UPDATE_P) {
    T bt = T(a.cg[s].beta);
    d.x = z.x + bt * p.x; d.y = z.y + bt * p.y; d.z = z.z + bt * p.z; d.w = T(0);
    __syncwarp(gm);
    if (lane == 0) a.P[i] = d;
  } else {
    d = z;
  }
  const BoxInfo &B = a.box[s];
  const int K1 = M.K1, K2 = M.K2, K3 = M.K3;
  T e = 0;
  if (lane < 3) {
    T th[P], dth[P];
    bspline<T, P, false>(lane == 0 ? f.x : (lane == 1 ? f.y : f.z), th, dth, nullptr);
#pragma unroll
    for (int k = 0; k < P; ++k) { sh[sub][lane][k].x = th[k]; sh[sub][lane][k].y = dth[k]; }
    e = T((double(d.x) * B.Hinv[lane] + double(d.y) * B.Hinv[3 + lane] + double(d.z) * B.Hinv[6 + lane]) * (lane == 0 ? K1 : lane == 1 ? K2 : K3));
  }
  const int l0 = (threadIdx.x & 31) & ~(QL - 1);
  const T e0 = __shfl_sync(gm, e, l0), e1 = __shfl_sync(gm, e, l0 + 1), e2 = __shfl_sync(gm, e, l0 + 2);
  __syncwarp(gm);
  const T qi = WITH_Q ? a.q[i] : T(0);
  T *grid = a.Q + M.r0;
  with_vec<T>(K3, [&](auto vw) {
    constexpr int VW = decltype(vw)::value;
    RowVectors<T, P, VW, 2> rv;
    const T *wk[2] = {&sh[sub][2][0].x, &sh[sub][2][0].y};
    rv.set(lane, b.z, K3, wk, 2);
    for_rows<P, VW, Stencil<P, VW>::ROUNDS <= 9 ? Stencil<P, VW>::ROUNDS : 4>(lane, b, K1, K2, K3, [&](int j1, int j2, size_t row) {
      const c2<T> w1 = sh[sub][0][j1], w2 = sh[sub][1][j2];
      const T A = (qi * w1.x + e0 * w1.y) * w2.x + e1 * w1.x * w2.y, Bw = e2 * w1.x * w2.x;
#pragma unroll
      for (int q = 0; q < rv.NQ; ++q) {
        if (!rv.on[q]) continue;
        T v[VW];
#pragma unroll
        for (int k = 0; k < VW; ++k) v[k] = A * rv.w[0][q][k] + Bw * rv.w[1][q][k];
        add_vec(grid + (row + rv.at[q]) * VW, v);
      }
    });
  });
}

// ------------------------------------------------------------------ row field + PME gather
// s_i = sum_k de_ik/dd_i (forcefield.py:1395-1402) + dU_rec/dd_i (pme.py:378-388), then by MODE:
//   0 FIELD  out = -(s - c_self d)                       (forcefield.py:1428-1433)
//   1 OPER   out = d / alpha + s - c_self d, and p.Ap    (forcefield.py:1694-1712, 1806-1807)
// The row part alone: F_i = sum_k de_ik/dd_i (runs beside the PME chain).  LPR lanes per row
// (32: a warp per atom; 16 or 8: two or four atoms per warp, each row split over fewer lanes, more
// rows in flight per warp), 8 atoms per block of 8 LPR threads either way -- the autotuner's choice
// (Engine::autotune).  The lane partial sums are combined by a butterfly within each LPR group,
// so the variants differ only in the order of the row's additions.  Bound by HBM: 24 bytes a pair, 111.8 us
// at 30.2 M pairs = 0.99 of the measured copy bandwidth (116.8 with the arrays apart); cached instead of evict-first
// loads lose 4 to 10 % of a step (they push the grids out of L2).
template <typename T, bool WITH_Q, int ACT, int LPR = 32>
__global__ void __launch_bounds__(8 * LPR) k_rowfield(Dev<T> a, const v4<T> *__restrict__ D, v4<T> *__restrict__ F, int nvb) {
  static_assert(LPR == 32 || LPR == 16 || LPR == 8, "lanes per row");
  pdl_enter();
  const int sub = threadIdx.x / LPR, lane = threadIdx.x % LPR;
  // blocks of 8 rows (nvb of them); a grid smaller than nvb walks them at its stride (the row field
  // beside the FFT chain on a limited number of SMs)
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
  const Where wh = where(a, a.wb, vb, WARPS_PER_BLOCK, sub);
  const int s = wh.s, i = wh.i;
  const bool valid = i < wh.end;
  int n = valid ? min(a.rn[i], a.mce) : 0;
  if (!solve_active(a, s, ACT)) continue;  // uniform over the block
  if (LPR == 32 && !valid) continue;  // uniform over the warp
  unsigned char *row = row_of(a, valid ? i : 0);
  using C = RowChunk<T>;
  T f0 = 0, f1 = 0, f2 = 0;
  auto pair = [&](int k, T x, T y, T z, T g1, T g2) {
    v4<T> dk = D[k];
    T dkx = dk.x * x + dk.y * y + dk.z * z;
    T c = -g2 * dkx;
    if (WITH_Q) c -= dk.w * g1;  // the charge rides with the dipole (k_start1, k_load_vec)
    f0 += c * x + g1 * dk.x;
    f1 += c * y + g1 * dk.y;
    f2 += c * z + g1 * dk.z;
  };
  if constexpr (sizeof(T) == 4) {
    // streaming loads (evict first): the 90+ MB of rows pass through L2 once per sweep and must
    // not push out the PME grids that the FFT passes read next.  The next group of four entries
    // is loaded before the current one is used (two groups of row data in flight per lane).
    // Eight lanes cover a chunk, so a lane steps by whole chunks from one address.
    const unsigned char *at = row + (lane >> 3) * C::SIZE + (lane & 7) * 16;
    constexpr int STEP = LPR / 8 * C::SIZE;
    auto v4at = [](const unsigned char *p) { return __ldcs(reinterpret_cast<const float4 *>(p)); };
    int4 kk = make_int4(0, 0, 0, 0);
    float4 xx = make_float4(0, 0, 0, 0), yy = xx, zz = xx, g1 = xx, g2 = xx;
    if (4 * lane < n) {
      kk = __ldcs(reinterpret_cast<const int4 *>(at));
      xx = v4at(at + C::X); yy = v4at(at + C::Y); zz = v4at(at + C::Z); g1 = v4at(at + C::G1); g2 = v4at(at + C::G2);
    }
    for (int t4 = lane; 4 * t4 < n; t4 += LPR) {
      const int t4n = t4 + LPR;
      at += STEP;
      int4 kn = make_int4(0, 0, 0, 0);
      float4 xn = make_float4(0, 0, 0, 0), yn = xn, zn = xn, g1n = xn, g2n = xn;
      if (4 * t4n < n) {
        kn = __ldcs(reinterpret_cast<const int4 *>(at));
        xn = v4at(at + C::X); yn = v4at(at + C::Y); zn = v4at(at + C::Z); g1n = v4at(at + C::G1); g2n = v4at(at + C::G2);
      }
      int t = 4 * t4;
      pair(kk.x, xx.x, yy.x, zz.x, g1.x, g2.x);
      if (t + 1 < n) pair(kk.y, xx.y, yy.y, zz.y, g1.y, g2.y);
      if (t + 2 < n) pair(kk.z, xx.z, yy.z, zz.z, g1.z, g2.z);
      if (t + 3 < n) pair(kk.w, xx.w, yy.w, zz.w, g1.w, g2.w);
      kk = kn; xx = xn; yy = yn; zz = zn; g1 = g1n; g2 = g2n;
    }
  } else {
    for (int t = lane; t < n; t += LPR) {
      unsigned char *c = row_entry<T>(row, t);
      pair(entry_k<T>(c, t), entry_v<T, C::X>(c, t), entry_v<T, C::Y>(c, t), entry_v<T, C::Z>(c, t), entry_v<T, C::G1>(c, t),
           entry_v<T, C::G2>(c, t));
    }
  }
  // every lane of the warp takes part in the butterfly (a row past the system's end adds zeros)
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) {
    f0 += __shfl_xor_sync(0xffffffffu, f0, o);
    f1 += __shfl_xor_sync(0xffffffffu, f1, o);
    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
  }
  if (valid && lane == 0) {
    v4<T> o;
    o.x = f0; o.y = f1; o.z = f2; o.w = T(0);
    F[i] = o;
  }
  }
}

// The PME gather of the system's potential at every atom, with the row field a.F: assembles the field (MODE 0) or
// the operator and p.Ap (MODE 1).  COMBINE (the CG direction's sweep with the row field started before the
// spread): a.F holds the rows of z, and the rows of p = z + beta p_prev are a.F + beta a.Fp (a.Fp: those
// of p_prev, rewritten).
template <typename T, int P, int MODE, int ACT, bool COMBINE = false>
__global__ void __launch_bounds__(ATOMS_PER_BLOCK * QL) k_gather(Dev<T> a, const v4<T> *__restrict__ D, v4<T> *__restrict__ out) {
  pdl_enter();
  __shared__ c2<T> sh[ATOMS_PER_BLOCK][3][P];  // per atom of the block: weight and derivative
  __shared__ double red[ATOMS_PER_BLOCK];
  const int sub = threadIdx.x / QL, lane = threadIdx.x % QL;  // the atom's group of lanes
  const unsigned gm = group_mask<QL>();
  const Where wh = where(a, a.qb, blockIdx.x, ATOMS_PER_BLOCK, sub);
  const int s = wh.s, i = wh.i;
  const bool valid = i < wh.end;
  // the loads go out before the test of the system's flag, and the assembly's are in flight during the stencil
  const int il = valid ? i : wh.end - 1;
  const int4 b = a.base[il];
  const v4<T> fr = a.frac[il];
  const v4<T> rowf = a.F[il], di = D[il];
  const T ia = MODE == 1 ? a.ialpha[il] : T(0);
  const Mesh M = mesh_of(a, s);
  if (!solve_active(a, s, ACT)) return;   // uniform over the block
  double dotv = 0.0;
  if (valid) {
    const BoxInfo &B = a.box[s];
    if (lane < 3) {
      T th[P], dth[P];
      bspline<T, P, false>(lane == 0 ? fr.x : (lane == 1 ? fr.y : fr.z), th, dth, nullptr);
#pragma unroll
      for (int k = 0; k < P; ++k) { sh[sub][lane][k].x = th[k]; sh[sub][lane][k].y = dth[k]; }
    }
    __syncwarp(gm);
    const T *phi = a.Phi + M.r0;
    const int K1 = M.K1, K2 = M.K2, K3 = M.K3;
    T g0 = 0, g1 = 0, g2 = 0;
    with_vec<T>(K3, [&](auto vw) {
      constexpr int VW = decltype(vw)::value;
      RowVectors<T, P, VW, 2> rv;
      const T *wk[2] = {&sh[sub][2][0].x, &sh[sub][2][0].y};
      rv.set(lane, b.z, K3, wk, 2);
      for_rows<P, VW, Stencil<P, VW>::ROUNDS <= 9 ? Stencil<P, VW>::ROUNDS : 4>(lane, b, K1, K2, K3, [&](int j1, int j2, size_t row) {
        T st = 0, su = 0;  // the row's sums with the k3 weights and their derivatives
#pragma unroll
        for (int q = 0; q < rv.NQ; ++q) {
          if (!rv.on[q]) continue;
          T v[VW];
          load_vec<T, VW>(phi + (row + rv.at[q]) * VW, v);
#pragma unroll
          for (int k = 0; k < VW; ++k) { st += v[k] * rv.w[0][q][k]; su += v[k] * rv.w[1][q][k]; }
        }
        const c2<T> w1 = sh[sub][0][j1], w2 = sh[sub][1][j2];
        g0 += w1.y * w2.x * st;
        g1 += w1.x * w2.y * st;
        g2 += w1.x * w2.x * su;
      });
    });
    g0 = group_sum<T, QL>(g0, gm); g1 = group_sum<T, QL>(g1, gm); g2 = group_sum<T, QL>(g2, gm);
    if (lane == 0) {
      T f0 = rowf.x, f1 = rowf.y, f2 = rowf.z;
      if (COMBINE) {
        const double beta = a.cg[s].beta;
        if (beta != 0.0) {
          const v4<T> fp = a.Fp[i];
          f0 += T(beta) * fp.x; f1 += T(beta) * fp.y; f2 += T(beta) * fp.z;
        }
        a.Fp[i] = v4<T>{f0, f1, f2, T(0)};
      }
      // dU/dd_b = sum_a g_a Hinv[b][a] K_a
      T es[9];
#pragma unroll
      for (int bb = 0; bb < 3; ++bb)
#pragma unroll
        for (int aa = 0; aa < 3; ++aa) es[bb * 3 + aa] = T(B.Hinv[bb * 3 + aa] * (aa == 0 ? K1 : aa == 1 ? K2 : K3));
      T r0 = g0 * es[0] + g1 * es[1] + g2 * es[2];
      T r1 = g0 * es[3] + g1 * es[4] + g2 * es[5];
      T r2 = g0 * es[6] + g1 * es[7] + g2 * es[8];
      T cs = T(a.c_self);
      v4<T> o;
      if (MODE == 0) {
        o.x = -(f0 + r0 - cs * di.x); o.y = -(f1 + r1 - cs * di.y); o.z = -(f2 + r2 - cs * di.z);
      } else {
        o.x = di.x * ia + f0 + r0 - cs * di.x;
        o.y = di.y * ia + f1 + r1 - cs * di.y;
        o.z = di.z * ia + f2 + r2 - cs * di.z;
        dotv = double(di.x * o.x) + double(di.y * o.y) + double(di.z * o.z);
      }
      o.w = T(0);
      out[i] = o;
    }
  }
  if (MODE == 1) {
    if (lane == 0) red[sub] = dotv;
    __syncthreads();
    if (threadIdx.x < 32) {
      const double v = warp_sum<double>(red[threadIdx.x]);
      if (threadIdx.x == 0) atomicAdd(&a.cg[s].acc_pap, v);
    }
  }
}

// ------------------------------------------------------------------ learned guess: features
// The model predicts the correction delta = mu* - x4 to the mu4 extrapolation x4 = 4 mu1 - 6 mu2 +
// 4 mu3 - mu4 (mu_j the converged dipoles j steps back), so the untrained model (zero output) is the
// reference's mu4 predictor, and the solver keeps its fused one-sweep start: everything the model
// sees is known before the step's first field sweep.
//
// Step 1, one warp per atom over its pair row, edges r < rg (the short-range graph): the permanent
// field of the graph, b_i = -sum_k [(-q_k G1 - G2 (p_k . x)) x + G1 p_k] (the real-space row field
// of charges and permanent dipoles, restricted to the graph), and three per-atom channel vectors
// (e nm): c0 = alpha_i (b_i - b_prev,i) (zero when there is no previous b), c1 = mu1 - mu2,
// c2 = x4 - mu1.  b overwrites b_prev (the same thread reads it first), for the next step.
// NN_CHAN floats per atom: c0, c1, c2 (3 each) and mu1 (3).
constexpr int NN_CHAN = 12;
// The graph edges of atom i from the list the row build wrote, one edge per lane and round (edges past
// nn_emax are not read, as in the message-passing model).
template <int LPA = 32, typename T, typename F>
__device__ __forceinline__ void for_graph_edges(const Dev<T> &a, int i, F &&edge) {
  const int lane = threadIdx.x % LPA;
  const int ne = min(a.nn_ne[i], a.nn_emax);
  const float4 *list = a.nn_e4 + (size_t)i * a.nn_emax;
  for (int e = lane; e < ne; e += LPA) {
    const float4 v = list[e];
    edge(__float_as_int(v.w), v.x, v.y, v.z, e);
  }
}

// Step 1, one warp per atom over the graph edges of its pair row (r < rg): the permanent field of
// the graph, b_i = -sum_k [(-q_k G1 - G2 (p_k . x)) x + G1 p_k] (the real-space row field of
// charges and permanent dipoles, restricted to the graph), and three per-atom channel vectors
// (e nm): c0 = alpha_i (b_i - b_prev,i) (zero when there is no previous b), c1 = mu1 - mu2,
// c2 = x4 - mu1.  b overwrites b_prev (the same thread reads it first), for the next step.
// NN_CHAN floats per atom: c0, c1, c2 (3 each) and mu1 (3).
template <typename T, int LPA = 32>
__global__ void __launch_bounds__(8 * LPA, 8 * 32 / LPA) k_nn_chan(Dev<T> a, const double *hist, const float4 *bl_prev,
                                                                  const int *valid, float rg, float4 *bl_out, float *chan) {
  static_assert(LPA == 32 || LPA == 16 || LPA == 8, "lanes per atom");
  const int warp = threadIdx.x / LPA, lane = threadIdx.x % LPA;  // the atom's group of LPA lanes
  const unsigned gm = group_mask<LPA>();
  const Where at = where(a, a.wb, blockIdx.x, WARPS_PER_BLOCK, warp);
  const int i = at.i;
  if (i >= at.end) return;
  (void)rg;  // the graph radius is a.nn_rg2 here
  float f0 = 0.f, f1 = 0.f, f2 = 0.f;
  const float2 *G = a.nn_g + (size_t)i * a.nn_emax;
  for_graph_edges<LPA>(a, i, [&](int k, float x, float y, float z, int e) {
    const float2 g = G[e];  // the edge's pair kernels G1, G2, as the row build evaluated them
    const float g1 = g.x, g2 = g.y;
    double4 pk = a.pperm[k];
    float px = float(pk.x), py = float(pk.y), pz = float(pk.z);
    float c = -float(a.q[k]) * g1 - g2 * (px * x + py * y + pz * z);
    f0 += c * x + g1 * px;
    f1 += c * y + g1 * py;
    f2 += c * z + g1 * pz;
  });
  f0 = -group_sum<float, LPA>(f0, gm); f1 = -group_sum<float, LPA>(f1, gm); f2 = -group_sum<float, LPA>(f2, gm);
  if (lane >= 3) return;
  // lanes 0..2 write one component each
  const float fb = lane == 0 ? f0 : (lane == 1 ? f1 : f2);
  const float *bp = bl_prev ? reinterpret_cast<const float *>(bl_prev + i) : nullptr;
  const bool have_prev = bp && (!valid || *valid);
  const float db = have_prev ? fb - bp[lane] : 0.f;
  const size_t st = (size_t)a.nt * 3;
  double m1 = hist[3 * (size_t)i + lane], m2 = hist[st + 3 * (size_t)i + lane], m3 = hist[2 * st + 3 * (size_t)i + lane],
         m4 = hist[3 * st + 3 * (size_t)i + lane];
  double x4 = 4.0 * m1 - 6.0 * m2 + 4.0 * m3 - m4;
  reinterpret_cast<float *>(bl_out + i)[lane] = fb;
  if (lane == 0) reinterpret_cast<float *>(bl_out + i)[3] = 0.f;
  float *C = chan + (size_t)i * NN_CHAN;
  C[lane] = float(a.alpha[i]) * db;
  C[3 + lane] = float(m1 - m2);
  C[6 + lane] = float(x4 - m1);
  C[9 + lane] = float(m1);
}

// Step 2, one warp per atom over the same edges: vector channels (NN_CH = 15) v0..v2 = the atom's own
// c0..c2 and, for each c and 2 radial bases phi_k(r) = exp(-((r - (0.15 + 0.2 k) nm) / 0.15 nm)^2)
// (cos(pi r / rg) + 1) / 2, the aggregates A_ck = sum_j phi_k c_j and D_ck = sum_j phi_k (c_j . u) u
// (u = x / r), 36 sums in one pass over the edges with a transposing warp reduction; 16 rotation
// invariants (asinh of magnitudes and dot products over the change scale sigma, |mu1| over
// 0.02 e nm, alpha, radius).  The model mixes the 15 channels, so the predicted correction turns
// with the system.  Sets *valid (the next step has a previous b).
// One halving step of a transposing warp reduction: lanes with bit (N/2) set keep the upper half of
// their N values and receive the partner's upper half, the others the lower halves.
template <int N>
__device__ __forceinline__ void transpose_step(float (&v)[32], int lane) {
  const bool up = lane & (N / 2);
#pragma unroll
  for (int j = 0; j < N / 2; ++j) {
    float send = up ? v[j] : v[j + N / 2];
    float keep = up ? v[j + N / 2] : v[j];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, N / 2);
  }
}
// Warp sums of 32 values per lane in 31 shuffles: lane l returns the total of v[l].
__device__ __forceinline__ float warp_transpose_sum(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
  transpose_step<32>(v, lane);
  transpose_step<16>(v, lane);
  transpose_step<8>(v, lane);
  transpose_step<4>(v, lane);
  transpose_step<2>(v, lane);
  return v[0];
}

// The 36 sums over the graph edges in one pass, value o = ((q * 3 + c) * 2 + k) * 3 + x for the
// plain (q = 0: A) and projected (q = 1: D) sums of channel c with radial basis k; returns on lane l
// the total of value l (l < 32) and in tail[0..3] the totals of values 32..35.
template <typename T>
__device__ __forceinline__ float nn_aggregate(const Dev<T> &a, int i, const float *chan, float rg, float (&tail)[4]) {
  float acc[36];
#pragma unroll
  for (int o = 0; o < 36; ++o) acc[o] = 0.f;
  const float irg = 1.f / rg;
  for_graph_edges(a, i, [&](int j, float x, float y, float z, int) {
    float r = sqrtf(x * x + y * y + z * z);
    float ir = 1.f / r, u[3] = {x * ir, y * ir, z * ir};
    float fc = 0.5f * (cospif(r * irg) + 1.f);
    float phi[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float d = (r - (0.15f + 0.2f * k)) * (1.f / 0.15f);
      phi[k] = expf(-d * d) * fc;
    }
    const float4 *cj = reinterpret_cast<const float4 *>(chan + (size_t)j * NN_CHAN);
    float4 c01 = cj[0], c12 = cj[1], c2m = cj[2];
    float v[3][3] = {{c01.x, c01.y, c01.z}, {c01.w, c12.x, c12.y}, {c12.z, c12.w, c2m.x}};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float pr = v[c][0] * u[0] + v[c][1] * u[1] + v[c][2] * u[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int xx = 0; xx < 3; ++xx) {
          acc[(c * 2 + k) * 3 + xx] += phi[k] * v[c][xx];
          acc[18 + (c * 2 + k) * 3 + xx] += phi[k] * pr * u[xx];
        }
    }
  });
#pragma unroll
  for (int o = 0; o < 4; ++o) tail[o] = warp_sum<float>(acc[32 + o]);
  float (&head)[32] = *reinterpret_cast<float (*)[32]>(acc);
  return warp_transpose_sum(head);
}

template <typename T>
__global__ void __launch_bounds__(256, 4) k_nn_features(Dev<T> a, const float *chan, float sigma, float rg, float *inv, float *vec,
                                                     int *valid) {
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (valid && blockIdx.x == 0 && threadIdx.x == 0) *valid = 1;  // read by the previous kernel only
  const Where at = where(a, a.wb, blockIdx.x, WARPS_PER_BLOCK, warp);
  const int i = at.i;
  if (i >= at.end) return;
  float *V = vec + (size_t)i * pgmnn::NN_CH * 3;
  float *F = inv + (size_t)i * pgmnn::NN_IN;
  const float is = 1.f / sigma, is2 = is * is;
  float tail[4];
  // lane l holds value l; the norms of the first eight (c, k) groups of three for the invariants
  float mine = nn_aggregate(a, i, chan, rg, tail);
  V[9 + lane] = mine;
  if (lane < 4) V[9 + 32 + lane] = tail[lane];
  float sq = mine * mine;
  float n2 = sq + __shfl_down_sync(0xffffffffu, sq, 1) + __shfl_down_sync(0xffffffffu, sq, 2);
  // the 16 invariants on 16 lanes at once: F[8 + l / 3] on lanes l = 0, 3, .., 21 (the group norms),
  // F[l - 24] on lanes 24..31 (the atom's own channels, |mu1|, alpha, radius); V[0..8] the own channels
  const float *ci = chan + (size_t)i * NN_CHAN;
  if (lane < 9) V[lane] = ci[lane];
  float arg = 0.f;
  bool ash = true;
  int slot = -1;
  if (lane < 24) {
    if (lane % 3 == 0) { arg = sqrtf(n2) * is; slot = 8 + lane / 3; }
  } else {
    const float s0[3] = {ci[0], ci[1], ci[2]}, s1[3] = {ci[3], ci[4], ci[5]}, s2[3] = {ci[6], ci[7], ci[8]};
    const float m1[3] = {ci[9], ci[10], ci[11]};
    auto dot = [](const float *p, const float *q) { return p[0] * q[0] + p[1] * q[1] + p[2] * q[2]; };
    auto norm3 = [](const float *p) { return sqrtf(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]); };
    slot = lane - 24;
    switch (slot) {
      case 0: arg = float(a.alpha[i]) * 1e3f; ash = false; break;
      case 1: arg = float(a.radius[i]) / 0.06f; ash = false; break;
      case 2: arg = norm3(s0) * is; break;
      case 3: arg = norm3(m1) * 50.f; ash = false; break;
      case 4: arg = norm3(s1) * is; break;
      case 5: arg = norm3(s2) * is; break;
      case 6: arg = dot(s0, s1) * is2; break;
      default: arg = dot(s0, s2) * is2; break;
    }
  }
  if (slot >= 0) F[slot] = ash ? asinhf(arg) : arg;
}

// ------------------------------------------------------------------ CG
// Which start a solve takes (forcefield.py:1951-1966): `have` the history predictor applies, `fused`
// its one-sweep start.  mode 1: the guess is the state's mu, plain start (energy, forcefield.py:2606-2612).
struct StartRule {
  int K, fused, refresh, mode, use_nn;
  const int32_t *count;
  const double *norm;
  __device__ __forceinline__ bool have(int s) const { return mode == 1 || (K > 0 && count[s] >= K); }
  __device__ __forceinline__ bool is_fused(int s) const { return mode == 0 && fused && have(s) && count[s] % refresh != 0; }
};
// The system's solver state before the start, and the condition of the plain start's node.
__device__ __forceinline__ void cg_setup(CGSys &G, int s, const StartRule &r, cudaGraphConditionalHandle plain, int use_cond) {
  G.have = r.have(s);
  G.nn = r.use_nn && G.have;  // k_start1 adds the model's correction to the extrapolation
  G.fallback = 0;
  G.iel_ext = 0; G.iel_first = 0; G.maxit_s = -1; G.tol_s = -1.0;
  G.fused = r.is_fused(s);
  G.sweep2 = !G.fused;
  if (use_cond && G.sweep2) cudaGraphSetConditional(plain, 1u);  // the plain start's sweep runs (default 0)
  G.active = 0;
  G.norm = G.fused ? r.norm[s] : 1.0;
  G.acc_abs = 0; G.acc_rz = 0; G.acc_max = 0; G.acc_pap = 0; G.acc_num = 0;
}

// Start, step 1 (thread per atom): the predictor guess x0h = sum c_j hist_j (forcefield.py:605,
// 1956-1958) and the dipoles of the first field sweep: p + x0h (fused start) or p (plain); the thread of a
// system's first atom sets up its solver state.
template <typename T>
__global__ void k_start1(Dev<T> a, StartRule rule, const double *hist, double c0, double c1, double c2, double c3, const float *xnn,
                         cudaGraphConditionalHandle plain, int use_cond) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  int s = system_of(a, i);
  const bool have = rule.have(s), fused = rule.is_fused(s);
  if (i == a.sys[s].atom0) cg_setup(a.cg[s], s, rule, plain, use_cond);
  double x0[3] = {0, 0, 0};
  if (have) {
    const double cc[4] = {c0, c1, c2, c3};
    for (int j = 0; j < rule.K; ++j)
      for (int c = 0; c < 3; ++c) x0[c] += cc[j] * hist[((size_t)j * a.nt + i) * 3 + c];
    if (xnn)  // the learned correction to the extrapolation
      for (int c = 0; c < 3; ++c) x0[c] += double(xnn[3 * (size_t)i + c]);
  }
  double4 p = a.pperm[i];
  v4<T> d, x;
  if (fused) { d.x = T(p.x + x0[0]); d.y = T(p.y + x0[1]); d.z = T(p.z + x0[2]); }
  else { d.x = T(p.x); d.y = T(p.y); d.z = T(p.z); }
  d.w = a.q[i];  // read with the dipole by the field sweep
  x.x = T(x0[0]); x.y = T(x0[1]); x.z = T(x0[2]); x.w = T(0);
  a.D[i] = d;
  a.X[i] = x;
}

// What a solve's begin needs beside the systems' state (cg_begin).
struct BeginArgs {
  CGSys *cg;
  int nsys;
  double tol;
  int max_iter;
  int *any;
  double fb_factor;
  cudaGraphConditionalHandle fbcond;
  int use_fbcond;
  int *fb_any;
  unsigned *done;
};

// Per-system scalars after the start (one block): norm, r.z, err, active; *any = some system iterates.
// which 0: the systems with the fused start (*any and *fb_any start here); 1: those with the plain start;
// 2: all; 3: the learned guess's fallbacks, re-evaluated after their sweep.
// The learned guess's check (fb_factor > 0): a system that started from x4 + the model's
// correction falls back to x4 when its start residual err exceeds fb_factor times the running
// mean of the extrapolation's (raising the fallback node's condition, *fb_any); a system that
// started from the extrapolation itself adds its err to that mean, and so does a fallback (which is counted).
__device__ __forceinline__ void cg_begin(const BeginArgs &b, int which) {
  __shared__ int act, fb;
  if (threadIdx.x == 0) { act = 0; fb = 0; }
  __syncthreads();
  constexpr double W = 0.1;  // weight of a new sample in the running mean
  for (int s = threadIdx.x; s < b.nsys; s += blockDim.x) {
    CGSys &G = b.cg[s];
    const bool mine = which == 2 || (which == 0 && G.fused) || (which == 1 && !G.fused) || (which == 3 && G.fallback);
    if (mine) {
      if (!G.fused && which != 3) G.norm = G.acc_abs / G.n3 + 1e-300;  // a fallback keeps the norm of its solve's b
      G.rz = G.acc_rz;
      G.err = __longlong_as_double((long long)G.acc_max) / G.norm;
      G.beta = 0.0;
      G.it = 0;
      G.active = (G.err > (G.tol_s >= 0.0 ? G.tol_s : b.tol)) && ((G.maxit_s >= 0 ? G.maxit_s : b.max_iter) > 0);
      G.acc_abs = 0; G.acc_rz = 0; G.acc_max = 0; G.acc_pap = 0; G.acc_num = 0;
      const bool record = which == 3 || (b.fb_factor > 0.0 && G.have && !G.nn);
      if (which != 3 && b.fb_factor > 0.0 && G.nn && G.ref_n > 0 && G.err > b.fb_factor * G.ref_err) {
        G.fallback = 1;
        atomicOr(&fb, 1);
      } else if (record) {
        G.ref_err = G.ref_n == 0 ? G.err : (1.0 - W) * G.ref_err + W * G.err;
        G.ref_n += 1;
        if (which == 3) G.fallbacks += 1;
      }
    }
    if (G.active) atomicOr(&act, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *b.any = act;
    if (which != 3 && b.fb_any) *b.fb_any = which == 1 ? (*b.fb_any | fb) : fb;
    if (which != 3 && b.use_fbcond && fb) cudaGraphSetConditional(b.fbcond, 1u);  // the fallback node runs (default 0)
  }
}
// The block that finishes last (a counter after a memory fence) takes the caller's closing step.
__device__ __forceinline__ bool last_block(unsigned *done) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partial sums are visible before it is counted
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    __threadfence();
    if (threadIdx.x == 0) *done = 0u;
  }
  return last;
}

// A block's sums of rz and max m of the start, added to its system's accumulators.
__device__ __forceinline__ void start_sums(CGSys &G, double rz, double m) {
  __shared__ double red[THREADS_PER_BLOCK / 32];
  __shared__ unsigned long long mx[THREADS_PER_BLOCK / 32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  rz = warp_sum<double>(rz);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) { red[warp] = rz; mx[warp] = (unsigned long long)__double_as_longlong(m); }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0;
    unsigned long long mm = 0;
    for (int w = 0; w < THREADS_PER_BLOCK / 32; ++w) { v += red[w]; mm = max(mm, mx[w]); }
    atomicAdd(&G.acc_rz, v);
    atomicMax(&G.acc_max, mm);
  }
}

// Start, step 2: fused: r0 = field(q, p + x0) - x0 / alpha, and the CG's initial z = alpha r, p = z, r.z and
// max|alpha r| (forcefield.py:1796-1819); plain: b = field(q, p), the norm mean|alpha b| and, without history,
// x0 = alpha b (forcefield.py:1960-1997).  The last block evaluates the fused systems' scalars (cg_begin).
// LOCAL (the local preconditioner): only max|alpha r|; z, p, r.z and the scalars come with its kernels.
template <typename T, bool LOCAL>
__global__ void k_start2(Dev<T> a, BeginArgs begin) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  __shared__ double red[THREADS_PER_BLOCK / 32];
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  const int i = wh.i;
  CGSys &G = a.cg[s];
  const bool fused = G.fused;  // uniform over the block
  double sab = 0.0, rz = 0.0, m = 0.0;
  if (i < wh.end) {
    v4<T> b = a.B[i];
    v4<T> x = a.X[i];
    T al = a.alpha[i];
    if (fused) {
      T ia = a.ialpha[i];
      v4<T> r, z;
      r.x = b.x - x.x * ia; r.y = b.y - x.y * ia; r.z = b.z - x.z * ia; r.w = T(0);
      a.R[i] = r;
      z.x = al * r.x; z.y = al * r.y; z.z = al * r.z; z.w = T(0);
      if (!LOCAL) {
        a.Z[i] = z;
        a.P[i] = z;
        rz = double(r.x * z.x) + double(r.y * z.y) + double(r.z * z.z);
      }
      m = fmax(fabs(double(z.x)), fmax(fabs(double(z.y)), fabs(double(z.z))));
    } else {
      double ax = double(al) * double(b.x), ay = double(al) * double(b.y), az = double(al) * double(b.z);
      sab = fabs(ax) + fabs(ay) + fabs(az);
      if (!G.have) { x.x = T(ax); x.y = T(ay); x.z = T(az); x.w = T(0); a.X[i] = x; }
    }
  }
  if (fused) {
    start_sums(G, rz, m);
  } else {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    sab = warp_sum<double>(sab);
    if (lane == 0) red[warp] = sab;
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = 0;
      for (int w = 0; w < THREADS_PER_BLOCK / 32; ++w) v += red[w];
      atomicAdd(&G.acc_abs, v);
    }
  }
  if (!LOCAL && last_block(begin.done)) cg_begin(begin, 0);
}

// Start, step 3 (plain start only): r0 = b - A x0.
template <typename T>
__global__ void k_start3(Dev<T> a) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  int s = system_of(a, i);
  if (a.cg[s].fused) return;
  v4<T> b = a.B[i], ap = a.AP[i], r;
  r.x = b.x - ap.x; r.y = b.y - ap.y; r.z = b.z - ap.z; r.w = T(0);
  a.R[i] = r;
}

// CG initialisation of the plain start's systems: z = alpha r, p = z, r.z and max|alpha r|, and, in the last
// block, their scalars (cg_begin).
// FB (the learned guess's fallback, systems with the flag only): first back to the extrapolation,
// x = x4 = x - delta and r0 = b - A x4 = r0 + A delta (A delta in AP).
// LOCAL (the local preconditioner): only max|alpha r|; z, p, r.z and the scalars come with its kernels.
template <typename T, bool FB, bool LOCAL>
__global__ void k_cg_init(Dev<T> a, const float *delta, BeginArgs begin) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  if (FB ? a.cg[s].fallback : !a.cg[s].fused) {  // uniform over the block
    const int i = wh.i;
    double rz = 0, m = 0;
    if (i < wh.end) {
      v4<T> r = a.R[i];
      if (FB) {
        v4<T> ad = a.AP[i], x = a.X[i];
        r.x += ad.x; r.y += ad.y; r.z += ad.z;
        x.x -= T(delta[3 * (size_t)i]); x.y -= T(delta[3 * (size_t)i + 1]); x.z -= T(delta[3 * (size_t)i + 2]);
        a.R[i] = r;
        a.X[i] = x;
      }
      T al = a.alpha[i];
      v4<T> z;
      z.x = al * r.x; z.y = al * r.y; z.z = al * r.z; z.w = T(0);
      if (!LOCAL) {
        a.Z[i] = z;
        a.P[i] = z;
        rz = double(r.x * z.x) + double(r.y * z.y) + double(r.z * z.z);
      }
      m = fmax(fabs(double(z.x)), fmax(fabs(double(z.y)), fabs(double(z.z))));
    }
    start_sums(a.cg[s], rz, m);
  }
  if (!LOCAL && last_block(begin.done)) cg_begin(begin, FB ? 3 : 1);
}

// Fallback, step 1: the model's correction delta of every fallback system's atoms as the dipoles
// of one operator sweep (A delta).
template <typename T>
__global__ void k_fb_prep(Dev<T> a, const float *delta) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt || !a.cg[system_of(a, i)].fallback) return;
  v4<T> d;
  d.x = T(delta[3 * (size_t)i]); d.y = T(delta[3 * (size_t)i + 1]); d.z = T(delta[3 * (size_t)i + 2]); d.w = T(0);
  a.D[i] = d;
}

// One CG update (thread per atom): x += a p, r' = r - a Ap, z' = alpha r', and the sums of
// z'.(r' - r), r'.z', max|z'| (forcefield.py:1802-1814).
// One CG update (thread per atom): x += st p, r -= st Ap, z = alpha r (Jacobi), with the block
// partials of z.(r_new - r), r.z and max|z| added to the system's accumulators.
template <typename T>
__device__ __forceinline__ void cg_update_body(Dev<T> &a) {
  __shared__ double red[2][THREADS_PER_BLOCK / 32];
  __shared__ unsigned long long mx[THREADS_PER_BLOCK / 32];
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  CGSys &G = a.cg[s];
  const int i = wh.i, il = min(i, wh.end - 1);
  v4<T> x = a.X[il], r = a.R[il], p = a.P[il], ap = a.AP[il];  // out before the test of the system's flag
  const T al = a.alpha[il];
  if (!G.active) return;  // the block's system has converged
  double num = 0, rzn = 0, m = 0;
  if (i < wh.end) {
    T st = T(G.rz / fmax(G.acc_pap, 1e-300));
    x.x += st * p.x; x.y += st * p.y; x.z += st * p.z;
    v4<T> rn, z;
    rn.x = r.x - st * ap.x; rn.y = r.y - st * ap.y; rn.z = r.z - st * ap.z; rn.w = T(0);
    z.x = al * rn.x; z.y = al * rn.y; z.z = al * rn.z; z.w = T(0);
    num = double(z.x * (rn.x - r.x)) + double(z.y * (rn.y - r.y)) + double(z.z * (rn.z - r.z));
    rzn = double(rn.x * z.x) + double(rn.y * z.y) + double(rn.z * z.z);
    m = fmax(fabs(double(z.x)), fmax(fabs(double(z.y)), fabs(double(z.z))));
    a.X[i] = x;
    a.R[i] = rn;
    a.Z[i] = z;
  }
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  num = warp_sum<double>(num);
  rzn = warp_sum<double>(rzn);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) { red[0][warp] = num; red[1][warp] = rzn; mx[warp] = (unsigned long long)__double_as_longlong(m); }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v0 = 0, v1 = 0;
    unsigned long long mm = 0;
    for (int w = 0; w < THREADS_PER_BLOCK / 32; ++w) { v0 += red[0][w]; v1 += red[1][w]; mm = max(mm, mx[w]); }
    atomicAdd(&G.acc_num, v0);
    atomicAdd(&G.acc_rz, v1);
    atomicMax(&G.acc_max, mm);
  }
}

// The per-system scalars after an update (run by the last block of k_cg_update_check).
__device__ __forceinline__ void cg_check_body(CGSys *cg, int nsys, double tol, int max_iter, int *any,
                                              cudaGraphConditionalHandle cond, int use_cond) {
  __shared__ int act;
  if (threadIdx.x == 0) act = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < nsys; s += blockDim.x) {
    CGSys &G = cg[s];
    if (G.active) {
      G.beta = G.acc_num / fmax(G.rz, 1e-300);
      G.rz = G.acc_rz;
      G.err = __longlong_as_double((long long)G.acc_max) / G.norm;
      G.it += 1;
      G.active = (G.err > (G.tol_s >= 0.0 ? G.tol_s : tol)) && (G.it < (G.maxit_s >= 0 ? G.maxit_s : max_iter));
    }
    G.acc_num = 0; G.acc_rz = 0; G.acc_max = 0; G.acc_pap = 0;
    if (G.active) atomicOr(&act, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *any = act;
    if (use_cond) cudaGraphSetConditional(cond, act ? 1u : 0u);  // the captured while loop of the solve
  }
}

// The CG update and the per-system check in one launch: every block adds its partial sums, and the block that
// finishes last (a counter after a memory fence) evaluates the per-system scalars and the loop
// condition, then resets the counter for the next iteration.
template <typename T>
__global__ void k_cg_update_check(Dev<T> a, int nsys, double tol, int max_iter, int *any, cudaGraphConditionalHandle cond,
                                  int use_cond, unsigned *done) {
  pdl_enter();
  cg_update_body(a);
  if (last_block(done)) cg_check_body(a.cg, nsys, tol, max_iter, any, cond, use_cond);
}

// ------------------------------------------------------------------ local preconditioner
// z = M^-1 r with local_niter > 0 inner CG iterations on A_loc v = v / alpha + sum over the row
// entries closer than local_cut of T v_k, T v = -G2 (v . x) x + G1 v (the row field's pair term),
// started from z = alpha r (forcefield.py:1766-1792; the outer CG is then flexible, with the
// Polak-Ribiere beta it already uses).  Thread per atom; the short entries compacted entry-major.

// sum over atom i's short entries of T v_k (get(k) = v_k)
template <typename T, typename Get>
__device__ __forceinline__ void short_sum(const Dev<T> &a, int i, Get &&get, T &f0, T &f1, T &f2) {
  const int n = a.sh_n[i];
#pragma unroll 4
  for (int e = 0; e < n; ++e) {
    const size_t c = (size_t)e * a.nt + i;
    const T x = a.c_x[c], y = a.c_y[c], z = a.c_z[c], g1 = a.c_g1[c], g2 = a.c_g2[c];
    const v4<T> v = get(a.c_k[c]);
    const T cc = -g2 * (v.x * x + v.y * y + v.z * z);
    f0 += cc * x + g1 * v.x;
    f1 += cc * y + g1 * v.y;
    f2 += cc * z + g1 * v.z;
  }
}

// the block's sum of v added to *dst (one atomic per block)
__device__ __forceinline__ void block_add(double v, double *dst) {
  __shared__ double red[THREADS_PER_BLOCK / 32];
  v = warp_sum<double>(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < THREADS_PER_BLOCK / 32; ++w) t += red[w];
    atomicAdd(dst, t);
  }
}

// Which systems a chain kernel serves: 0 all, 1 the iterating ones, 3 those falling back.
__device__ __forceinline__ bool lp_skip(int act, const CGSys &G) {
  return (act == 1 && !G.active) || (act == 3 && !G.fallback);
}

// Inner start: z = alpha r, rr = r - A_loc(alpha r) = -sum T (alpha r)_k, zz = alpha rr (the first
// inner direction), partial rr . zz.
template <typename T, int ACT>
__global__ void k_lp_start(Dev<T> a) {
  pdl_enter();
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  CGSys &G = a.cg[s];
  if (lp_skip(ACT, G)) return;  // uniform over the block
  const int i = wh.i;
  double rz = 0.0;
  if (i < wh.end) {
    T f0 = 0, f1 = 0, f2 = 0;
    short_sum(a, i, [&](int k) {
      const v4<T> r = a.R[k];
      const T al = a.alpha[k];
      v4<T> w;
      w.x = al * r.x; w.y = al * r.y; w.z = al * r.z; w.w = T(0);
      return w;
    }, f0, f1, f2);
    const v4<T> r = a.R[i];
    const T al = a.alpha[i];
    v4<T> z, rr, zz;
    z.x = al * r.x; z.y = al * r.y; z.z = al * r.z; z.w = T(0);
    rr.x = -f0; rr.y = -f1; rr.z = -f2; rr.w = T(0);
    zz.x = al * rr.x; zz.y = al * rr.y; zz.z = al * rr.z; zz.w = T(0);
    a.Z[i] = z;
    a.LRR[i] = rr;
    a.LZZ[i] = zz;
    a.LP0[i] = zz;  // the first inner direction (kept: the next direction adds to it)
    rz = double(rr.x * zz.x) + double(rr.y * zz.y) + double(rr.z * zz.z);
  }
  block_add(rz, &G.acc_lrz);
}

// Inner direction and its product: p = zz (FIRST) or zz + lb p_prev (written to Pout), Ap =
// A_loc(p) into AP (the neighbours' p formed the same way), partial p . Ap.
template <typename T, int ACT, bool FIRST>
__global__ void k_lp_ap(Dev<T> a, const v4<T> *__restrict__ Pin, v4<T> *__restrict__ Pout) {
  pdl_enter();
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  CGSys &G = a.cg[s];
  if (lp_skip(ACT, G)) return;
  const int i = wh.i;
  const T b = T(G.lb);
  auto pget = [&](int k) {
    v4<T> p = a.LZZ[k];
    if (!FIRST) {
      const v4<T> q = Pin[k];
      p.x += b * q.x; p.y += b * q.y; p.z += b * q.z;
    }
    return p;
  };
  double pap = 0.0;
  if (i < wh.end) {
    T f0 = 0, f1 = 0, f2 = 0;
    short_sum(a, i, pget, f0, f1, f2);
    const v4<T> p = pget(i);
    const T ia = a.ialpha[i];
    v4<T> ap;
    ap.x = p.x * ia + f0; ap.y = p.y * ia + f1; ap.z = p.z * ia + f2; ap.w = T(0);
    if (!FIRST) Pout[i] = p;
    a.AP[i] = ap;
    pap = double(p.x * ap.x) + double(p.y * ap.y) + double(p.z * ap.z);
  }
  block_add(pap, &G.acc_lpap);
}

// Inner update: z += al p (al = rr.zz / p.Ap); not LAST: rr -= al Ap, zz = alpha rr, partial rr.zz
// for the next inner iteration.  LAST: the outer quantities -- MODE 0 (start, fallback): p = z,
// r.z and the start's scalars (cg_begin); MODE 1 (iteration): z.(r_new - r_old) and r_new.z.  The block that finishes last
// evaluates the inner scalars (lb, the next rr.zz) and, in MODE 1, the outer CG's per-system check
// and loop condition (cg_check_body).
template <typename T, int ACT, bool LAST, int MODE>
__global__ void k_lp_step(Dev<T> a, const v4<T> *__restrict__ Pcur, BeginArgs b, cudaGraphConditionalHandle cond, int use_cond) {
  pdl_enter();
  {
    const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
    const int s = wh.s;
    CGSys &G = a.cg[s];
    if (!lp_skip(ACT, G)) {
      const int i = wh.i;
      const T al = T(G.acc_lrz / fmax(G.acc_lpap, 1e-300));
      double v0 = 0.0, v1 = 0.0;
      if (i < wh.end) {
        const v4<T> p = Pcur[i];
        v4<T> z = a.Z[i];
        z.x += al * p.x; z.y += al * p.y; z.z += al * p.z;
        a.Z[i] = z;
        if (!LAST) {
          const v4<T> ap = a.AP[i];
          v4<T> rr = a.LRR[i], zz;
          const T alpha = a.alpha[i];
          rr.x -= al * ap.x; rr.y -= al * ap.y; rr.z -= al * ap.z;
          zz.x = alpha * rr.x; zz.y = alpha * rr.y; zz.z = alpha * rr.z; zz.w = T(0);
          a.LRR[i] = rr;
          a.LZZ[i] = zz;
          v0 = double(rr.x * zz.x) + double(rr.y * zz.y) + double(rr.z * zz.z);
        } else if (MODE == 0) {
          const v4<T> r = a.R[i];
          a.P[i] = z;
          v0 = double(r.x * z.x) + double(r.y * z.y) + double(r.z * z.z);
        } else {
          const v4<T> r = a.R[i], dr = a.DR[i];
          v0 = double(z.x * dr.x) + double(z.y * dr.y) + double(z.z * dr.z);
          v1 = double(r.x * z.x) + double(r.y * z.y) + double(r.z * z.z);
        }
      }
      if (!LAST) {
        block_add(v0, &G.acc_lrz2);
      } else if (MODE == 0) {
        block_add(v0, &G.acc_rz);
      } else {
        block_add(v0, &G.acc_num);
        __syncthreads();
        block_add(v1, &G.acc_rz);
      }
    }
  }
  if (!last_block(b.done)) return;
  for (int s = threadIdx.x; s < b.nsys; s += blockDim.x) {
    CGSys &G = a.cg[s];
    if (!LAST) {
      G.lb = G.acc_lrz2 / fmax(G.acc_lrz, 1e-300);
      G.acc_lrz = G.acc_lrz2;
    } else {
      G.acc_lrz = 0.0;
    }
    G.acc_lrz2 = 0.0;
    G.acc_lpap = 0.0;
  }
  if (LAST) {
    __syncthreads();
    if (MODE == 1) cg_check_body(a.cg, b.nsys, b.tol, b.max_iter, b.any, cond, use_cond);
    else cg_begin(b, ACT == 3 ? 3 : 2);  // the start's scalars
  }
}

// The outer CG update with the local preconditioner (thread per atom): x += st p, r_new = r - st
// Ap, DR = r_new - r, and max|alpha r_new| (the convergence test stays pmemd-pgm's); z, r.z and
// the check follow in the preconditioner's kernels.
template <typename T>
__global__ void k_cg_update_r(Dev<T> a) {
  pdl_enter();
  __shared__ unsigned long long mx[THREADS_PER_BLOCK / 32];
  const Where wh = where(a, a.tb, blockIdx.x, THREADS_PER_BLOCK, threadIdx.x);
  const int s = wh.s;
  CGSys &G = a.cg[s];
  if (!G.active) return;  // uniform over the block
  const int i = wh.i;
  double m = 0.0;
  if (i < wh.end) {
    const T st = T(G.rz / fmax(G.acc_pap, 1e-300));
    v4<T> x = a.X[i], r = a.R[i];
    const v4<T> p = a.P[i], ap = a.AP[i];
    const T al = a.alpha[i];
    x.x += st * p.x; x.y += st * p.y; x.z += st * p.z;
    v4<T> rn, dr;
    rn.x = r.x - st * ap.x; rn.y = r.y - st * ap.y; rn.z = r.z - st * ap.z; rn.w = T(0);
    dr.x = rn.x - r.x; dr.y = rn.y - r.y; dr.z = rn.z - r.z; dr.w = T(0);
    a.X[i] = x;
    a.R[i] = rn;
    a.DR[i] = dr;
    m = fmax(fabs(double(al * rn.x)), fmax(fabs(double(al * rn.y)), fabs(double(al * rn.z))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) mx[threadIdx.x >> 5] = (unsigned long long)__double_as_longlong(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long mm = 0;
    for (int w = 0; w < THREADS_PER_BLOCK / 32; ++w) mm = max(mm, mx[w]);
    atomicMax(&G.acc_max, mm);
  }
}

// After the loop: the peek step mu = x + peek alpha r (forcefield.py:1819-1820), the dipoles
// in FP64, the history push (forcefield.py:2005-2007), mu + p and zero accumulators for the energy pass, and the
// systems' solver state.
struct StateOut {
  int32_t *count;
  double *norm;
  int32_t *iters;
  double *resid;
  unsigned *status;
  int push;
  double tol;
};
__device__ __forceinline__ void cg_state_out(const CGSys *cg, int s, const StateOut &o) {
  const CGSys &G = cg[s];
  if (o.push) { o.count[s] += 1; o.norm[s] = G.norm; }
  if (o.iters) o.iters[s] = G.it;
  if (o.resid) o.resid[s] = G.err;
  if (G.err > o.tol && !G.iel_ext) atomicOr(&o.status[s], 0x2u);  // an extended iEL step stops short of tol by design
}
template <typename T>
__device__ __forceinline__ void energy_start(Dev<T> &a, int i, const double *m) {  // all threads of the launch
  constexpr int NACC = sizeof(EnergyAcc) / sizeof(double);
  for (int t = i; t < NACC * a.nsys; t += gridDim.x * blockDim.x) reinterpret_cast<double *>(a.eacc)[t] = 0.0;
  if (i >= a.nt) return;
  const double4 p = a.pperm[i];
  v4<T> d;
  d.x = T(p.x + m[0]); d.y = T(p.y + m[1]); d.z = T(p.z + m[2]); d.w = a.q[i];
  a.D[i] = d;
}
template <typename T>
__global__ void k_cg_finish(Dev<T> a, double *mu, double *hist, int push, StateOut out) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (int s = i; s < a.nsys; s += gridDim.x * blockDim.x) cg_state_out(a.cg, s, out);
  double m[3] = {0, 0, 0};
  if (i < a.nt) {
    v4<T> x = a.X[i], r = a.R[i];
    T al = a.alpha[i];
    T pk = T(a.peek);
    if (a.peek != 0.0) { x.x += pk * r.x * al; x.y += pk * r.y * al; x.z += pk * r.z * al; }
    m[0] = double(x.x); m[1] = double(x.y); m[2] = double(x.z);
    for (int c = 0; c < 3; ++c) mu[3 * i + c] = m[c];
    if (push) {
      size_t st = (size_t)a.nt * 3;
      for (int c = 0; c < 3; ++c) {
        size_t o = (size_t)3 * i + c;
        hist[3 * st + o] = hist[2 * st + o];
        hist[2 * st + o] = hist[st + o];
        hist[st + o] = hist[o];
        hist[o] = m[c];
      }
    }
  }
  energy_start(a, i, m);
}

__global__ void k_cg_state_out(const CGSys *cg, int nsys, StateOut out) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < nsys) cg_state_out(cg, s, out);
}

// Energy-only start: x0 = the state's mu, first sweep at d = p.
template <typename T>
__global__ void k_energy_start(Dev<T> a, StartRule rule, const double *mu, cudaGraphConditionalHandle plain, int use_cond) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  const int s = system_of(a, i);
  if (i == a.sys[s].atom0) cg_setup(a.cg[s], s, rule, plain, use_cond);
  double4 p = a.pperm[i];
  v4<T> d, x;
  d.x = T(p.x); d.y = T(p.y); d.z = T(p.z); d.w = a.q[i];
  x.x = T(mu[3 * i]); x.y = T(mu[3 * i + 1]); x.z = T(mu[3 * i + 2]); x.w = T(0);
  a.D[i] = d;
  a.X[i] = x;
}

// ------------------------------------------------------------------ extended-Lagrangian dipoles
// iEL (forcefield.py:1452-1650, Niklasson's dissipative extended-Lagrangian Verlet): the
// auxiliary dipoles xl (K1, N, 3) FP64, newest first; warm-up steps (count < warmup) solve to tol,
// extended steps take x = xl[0]: 0-SCF mu = x + omega delta (no CG), SCF iel_iter CG iterations
// (to tol with 0) from x.

// Per system: first / warm-up / extended, the start the shared solver machinery takes (plain with
// its second sweep in the warm-up, fused from x otherwise), whether the first step starts from a
// given mu (any nonzero dipole of the system: one block per system), and the overrides of tol and
// max_iter (SCF with a set number of iterations: tol 0).
__global__ void k_iel_setup(CGSys *cg, const SysInfo *sys, int nsys, const int32_t *count, const double *norm, const double *mu,
                            int warmup, int scheme, int iel_iter, cudaGraphConditionalHandle plain, int use_cond) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int s = blockIdx.x;
  if (s >= nsys) return;
  const SysInfo &S = sys[s];
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  const int c = count[s];
  if (c == 0)
    for (int t = threadIdx.x; t < 3 * S.natom; t += blockDim.x)
      if (mu[3 * (size_t)S.atom0 + t] != 0.0) any = 1;
  __syncthreads();
  if (threadIdx.x) return;
  CGSys &G = cg[s];
  const int warm = c < warmup;
  G.iel_first = c == 0;
  G.iel_ext = !warm;
  G.have = c == 0 ? any : 1;
  G.nn = 0;
  G.fallback = 0;
  G.fused = !warm;
  G.sweep2 = warm;
  if (use_cond && warm) cudaGraphSetConditional(plain, 1u);  // the plain start's sweep runs (default 0)
  G.active = 0;
  G.norm = warm ? 1.0 : norm[s];
  G.tol_s = -1.0;
  G.maxit_s = -1;
  if (!warm && scheme == 2 && iel_iter > 0) { G.tol_s = 0.0; G.maxit_s = iel_iter; }
  G.acc_abs = 0; G.acc_rz = 0; G.acc_max = 0; G.acc_pap = 0; G.acc_num = 0;
}

// The start's first sweep: x0 = xl[0] (the first step: the given mu, or 0 and then alpha b), the
// dipoles p + x0 of the fused start or p of the plain one.
template <typename T>
__global__ void k_iel_start1(Dev<T> a, const double *xl, const double *mu) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  const CGSys &G = a.cg[system_of(a, i)];
  double x0[3] = {0, 0, 0};
  for (int c = 0; c < 3; ++c) x0[c] = G.iel_first ? (G.have ? mu[3 * (size_t)i + c] : 0.0) : xl[3 * (size_t)i + c];
  double4 p = a.pperm[i];
  v4<T> d, x;
  if (G.fused) { d.x = T(p.x + x0[0]); d.y = T(p.y + x0[1]); d.z = T(p.z + x0[2]); }
  else { d.x = T(p.x); d.y = T(p.y); d.z = T(p.z); }
  d.w = a.q[i];  // read with the dipole by the field sweep
  x.x = T(x0[0]); x.y = T(x0[1]); x.z = T(x0[2]); x.w = T(0);
  a.D[i] = d;
  a.X[i] = x;
}

// Solve M d = r for one molecule's block in FP64 (Gaussian elimination, partial pivoting), M =
// diag(1/alpha) + the same-molecule row tensors G1 I - G2 x x^T (forcefield.py:1530-1556).
template <typename T>
__device__ void iel_block_solve(const Dev<T> &a, int i0, int nb, double (*M)[25], double *d) {
  const int N = 3 * nb;
  for (int u = 0; u < N; ++u)
    for (int v = 0; v <= N; ++v) M[u][v] = 0.0;
  for (int li = 0; li < nb; ++li) {
    const int i = i0 + li;
    const v4<T> r = a.R[i];
    const double ia = 1.0 / double(a.alpha[i]);
    const double rr[3] = {double(r.x), double(r.y), double(r.z)};
    for (int c = 0; c < 3; ++c) { M[3 * li + c][3 * li + c] += ia; M[3 * li + c][N] = rr[c]; }
    const int nsp = a.rnsp[i];  // molecule partners first in every row
    using C = RowChunk<T>;
    unsigned char *row = row_of(a, i);
    for (int t = 0; t < nsp; ++t) {
      unsigned char *c = row_entry<T>(row, t);
      const int k = entry_k<T>(c, t);
      const int lk = k - i0;
      if (lk < 0 || lk >= nb) continue;
      const double x[3] = {double(entry_v<T, C::X>(c, t)), double(entry_v<T, C::Y>(c, t)), double(entry_v<T, C::Z>(c, t))};
      const double g1 = double(entry_v<T, C::G1>(c, t)), g2 = double(entry_v<T, C::G2>(c, t));
      for (int u = 0; u < 3; ++u)
        for (int v = 0; v < 3; ++v) M[3 * li + u][3 * lk + v] += (u == v ? g1 : 0.0) - g2 * x[u] * x[v];
    }
  }
  for (int c = 0; c < N; ++c) {
    int pr = c;
    for (int u = c + 1; u < N; ++u)
      if (fabs(M[u][c]) > fabs(M[pr][c])) pr = u;
    if (pr != c)
      for (int v = 0; v <= N; ++v) { double t = M[c][v]; M[c][v] = M[pr][v]; M[pr][v] = t; }
    for (int u = c + 1; u < N; ++u) {
      const double f = M[u][c] / M[c][c];
      for (int v = c; v <= N; ++v) M[u][v] -= f * M[c][v];
    }
  }
  for (int c = N - 1; c >= 0; --c) {
    double acc = M[c][N];
    for (int v = c + 1; v < N; ++v) acc -= M[c][v] * d[v];
    d[c] = acc / M[c][c];
  }
}

// 0-SCF, one thread per molecule: for the extended systems delta = omega alpha r (Jacobi, and for
// molecules outside 2..8 atoms) or omega M^-1 r (block), mu = x + delta in FP64 (x = xl[0]), delta
// in Dl for the shadow energy, and max|delta| for the residual; zero delta elsewhere.
template <typename T>
__global__ void k_iel_delta(Dev<T> a, const double *xl, double omega, int block, double *mu, v4<T> *Dl) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.nmol) return;
  const int i0 = a.mol_start[m], nb = a.mol_start[m + 1] - i0;
  CGSys &G = a.cg[system_of(a, i0)];
  if (!G.iel_ext) {
    for (int i = i0; i < i0 + nb; ++i) Dl[i] = v4<T>{T(0), T(0), T(0), T(0)};
    return;
  }
  double d[24];
  double M[24][25];
  if (block && nb >= 2 && nb <= 8) {
    iel_block_solve(a, i0, nb, M, d);
  } else {
    for (int li = 0; li < nb && li < 8; ++li) {
      const v4<T> r = a.R[i0 + li];
      const double al = double(a.alpha[i0 + li]);
      d[3 * li] = al * double(r.x); d[3 * li + 1] = al * double(r.y); d[3 * li + 2] = al * double(r.z);
    }
  }
  double mx = 0.0;
  for (int li = 0; li < nb; ++li) {
    const int i = i0 + li;
    double dl[3];
    if (li < 8) {
      for (int c = 0; c < 3; ++c) dl[c] = omega * d[3 * li + c];
    } else {  // molecules above 8 atoms: Jacobi, atom by atom
      const v4<T> r = a.R[i];
      const double al = double(a.alpha[i]);
      dl[0] = omega * al * double(r.x); dl[1] = omega * al * double(r.y); dl[2] = omega * al * double(r.z);
    }
    for (int c = 0; c < 3; ++c) {
      mu[3 * (size_t)i + c] = xl[3 * (size_t)i + c] + dl[c];
      mx = fmax(mx, fabs(dl[c]));
    }
    Dl[i] = v4<T>{T(dl[0]), T(dl[1]), T(dl[2]), T(0)};
  }
  atomicMax(&G.acc_max, (unsigned long long)__double_as_longlong(mx));
}

// After the start (zscf: and the 0-SCF update): the extended 0-SCF systems' residual max|delta| /
// norm and no CG; *any over the systems that still iterate (warm-up solves, SCF from x), which
// with use_cond is also the captured loop's condition.
__global__ void k_iel_begin(CGSys *cg, int nsys, int *any, int zscf, cudaGraphConditionalHandle cond, int use_cond) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  __shared__ int act;
  if (threadIdx.x == 0) act = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < nsys; s += blockDim.x) {
    CGSys &G = cg[s];
    if (zscf && G.iel_ext) {
      G.err = __longlong_as_double((long long)G.acc_max) / G.norm;
      G.active = 0;
      G.acc_max = 0;
    }
    if (G.active) atomicOr(&act, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *any = act;
    if (use_cond) cudaGraphSetConditional(cond, act ? 1u : 0u);
  }
}

// After the solve: mu (the CG result with the peek step; 0-SCF extended systems: already written),
// the history push, and the auxiliary dipoles' step x_{n+1} = 2 Xh[0] - Xh[1] + kappa dx + a sum_k
// c_k Xh[k] with Xh = (mu, mu, ...) on the first step, xl with Xh[0] = mu in the warm-up, xl after,
// dx = mu - x on extended steps (0 in the warm-up); xl becomes (x_{n+1}, Xh[0], ..., Xh[K1 - 2]).
struct IelCoef {
  double kappa, a, c[10];
  int nc, K1, zscf;
};
template <typename T>
__global__ void k_iel_finish(Dev<T> a, double *mu, double *hist, double *xl, IelCoef co) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  const CGSys &G = a.cg[system_of(a, i)];
  const size_t st = (size_t)a.nt * 3;
  double m[3];
  if (G.iel_ext && co.zscf) {
    for (int c = 0; c < 3; ++c) m[c] = mu[3 * (size_t)i + c];
  } else {
    v4<T> x = a.X[i], r = a.R[i];
    const T al = a.alpha[i], pk = T(a.peek);
    if (a.peek != 0.0) { x.x += pk * r.x * al; x.y += pk * r.y * al; x.z += pk * r.z * al; }
    m[0] = double(x.x); m[1] = double(x.y); m[2] = double(x.z);
    for (int c = 0; c < 3; ++c) mu[3 * (size_t)i + c] = m[c];
  }
  for (int c = 0; c < 3; ++c) {
    const size_t o = (size_t)3 * i + c;
    hist[3 * st + o] = hist[2 * st + o];
    hist[2 * st + o] = hist[st + o];
    hist[st + o] = hist[o];
    hist[o] = m[c];
    double X[12];
    for (int j = 0; j < co.K1; ++j) X[j] = G.iel_first ? m[c] : ((j == 0 && !G.iel_ext) ? m[c] : xl[j * st + o]);
    double v = 2.0 * X[0] - X[1] + (G.iel_ext ? co.kappa * (m[c] - X[0]) : 0.0);
    if (co.a != 0.0)
      for (int k = 0; k < co.nc; ++k) v += co.a * co.c[k] * X[k];
    xl[o] = v;
    for (int j = 1; j < co.K1; ++j) xl[j * st + o] = X[j - 1];
  }
}

// ------------------------------------------------------------------ energy, forces, virial
// One group of QL lanes per atom over its row: pair energies and their row gradients with the analytic
// kernels G0..G3 (forcefield.py:2294-2360), LJ rows, the row field at (q, d) (dE/dd), the pair
// virial sum g (x) x - gx (x) off; then the PME gradients of the atom: dU/dd and dU/dr through the
// spline derivatives (the autodiff of pme.py:390-411 written out).
// SHADOW (iEL/0-SCF, forcefield.py:2011-2045, 2294-2360): the energy is the shadow potential's,
// minus the pair and reciprocal energies of the dipoles Dl = delta alone (inside a molecule of 2..8
// atoms with the block preconditioner, the i-side delta scaled by a.iel_keep = 1 - 1/omega); their
// position gradients at fixed delta go to the forces, not to the virial (the fixed-mu strain
// derivative); the sums of |delta|^2 and |delta|^2 / (2 alpha) go to the energy accumulators.
// Bound by the latency of the row stream (40 bytes a pair) and of the partners' gathers (7 of 12 cycles an instruction;
// DRAM 31 %, L1 52 %, issue 42 %, at 12,288 atoms and four blocks per SM).  The stencil comes first and its sums wait in
// shared memory, so that registers serve one part at a time: 303 -> 257 us at 98,304 atoms, 198 -> 169 at 59,049.
template <typename T, int P, int MINB = 3, bool SHADOW = false>
__global__ void __launch_bounds__(ATOMS_PER_BLOCK * QL, MINB) k_forces(Dev<T> a, const double *mu) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  __shared__ T sh[ATOMS_PER_BLOCK][3][3][P];  // per atom of the block: weights, first and second derivatives
  __shared__ T rec[ATOMS_PER_BLOCK][6];        // dU/dd and dU/dr along the mesh axes
  __shared__ double red[ATOMS_PER_BLOCK][16];
  const int sub = threadIdx.x / QL, lane = threadIdx.x % QL;  // the atom's group of lanes
  const unsigned gm = group_mask<QL>();
  const Where wh = where(a, a.qb, blockIdx.x, ATOMS_PER_BLOCK, sub);
  const int s = wh.s, i = wh.i;
  const bool valid = i < wh.end;
  const Mesh M = mesh_of(a, s);
  double vals[16];
  for (int k = 0; k < 16; ++k) vals[k] = 0.0;
  if (valid) {
    const BoxInfo &B = a.box[s];
    v4<T> di = a.D[i];
    T qi = a.q[i], rhi = a.rminh[i], sei = a.seps[i];
    int n = min(a.rn[i], a.mce), nsp = a.rnsp[i];
    unsigned char *row = row_of(a, i);
    using C = RowChunk<T>;
    T gx0 = 0, gx1 = 0, gx2 = 0, gl0 = 0, gl1 = 0, gl2 = 0, fd0 = 0, fd1 = 0, fd2 = 0;
    T ee = 0, el = 0;
    T w[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    T gs0 = 0, gs1 = 0, gs2 = 0;  // SHADOW: gradient of the delta-delta pair terms (forces only)
    v4<T> Dli = v4<T>{T(0), T(0), T(0), T(0)};
    bool blk_i = false;
    if constexpr (SHADOW) {
      Dli = a.Dl[i];
      const int msz = a.molend[i] - a.molfirst[i];
      blk_i = a.iel_keep_on && msz >= 2 && msz <= 8;
    }
    // reciprocal gradients of the atom first; their sums wait in shared memory, not in registers, for
    // the pair loop
    int4 b = a.base[i];
    v4<T> fr = a.frac[i];
    if (b.w && lane == 0) atomicOr(&a.status[s], 0x4u);  // a non-finite position
    if (lane < 3) {
      T th[P], dth[P], d2[P];
      bspline<T, P, true>(lane == 0 ? fr.x : (lane == 1 ? fr.y : fr.z), th, dth, d2);
#pragma unroll
      for (int k = 0; k < P; ++k) { sh[sub][0][lane][k] = th[k]; sh[sub][1][lane][k] = dth[k]; sh[sub][2][lane][k] = d2[k]; }
    }
    __syncwarp(gm);
    auto scaled = [&](int bb, int aa) { return T(B.Hinv[bb * 3 + aa] * (aa == 0 ? M.K1 : aa == 1 ? M.K2 : M.K3)); };  // dU/dr_b = sum_a g_a scaled(b, a)
    {
    T es[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) es[k] = scaled(k / 3, k % 3);
    const int K1 = M.K1, K2 = M.K2, K3 = M.K3;
    // The stencil rows of a potential: f(j1, A, B, C, D, E, F) with the row's sums along k3 (weights, first, second
    // derivatives: st, su, sv) times the k2 weights t2, u2, v2: A = t2 st, B = u2 st, C = t2 su, D = v2 st,
    // E = u2 su, F = t2 sv.
    auto stencil = [&](const T *phi, auto &&f) {
      with_vec<T>(K3, [&](auto vw) {
        constexpr int VW = decltype(vw)::value;
        RowVectors<T, P, VW, 3> rv;
        const T *wk[3] = {sh[sub][0][2], sh[sub][1][2], sh[sub][2][2]};
        rv.set(lane, b.z, K3, wk, 1);
        for_rows<P, VW, 3>(lane, b, K1, K2, K3, [&](int j1, int j2, size_t row) {
          T st = 0, su = 0, sv = 0;
#pragma unroll
          for (int q = 0; q < rv.NQ; ++q) {
            if (!rv.on[q]) continue;
            T v[VW];
            load_vec<T, VW>(phi + (row + rv.at[q]) * VW, v);
#pragma unroll
            for (int k = 0; k < VW; ++k) { st += v[k] * rv.w[0][q][k]; su += v[k] * rv.w[1][q][k]; sv += v[k] * rv.w[2][q][k]; }
          }
          const T t2 = sh[sub][0][1][j2], u2 = sh[sub][1][1][j2], v2 = sh[sub][2][1][j2];
          f(j1, t2 * st, u2 * st, t2 * su, v2 * st, u2 * su, t2 * sv);
        });
      });
    };
    T ge0 = 0, ge1 = 0, ge2 = 0, gw0 = 0, gw1 = 0, gw2 = 0;
    if constexpr (SHADOW) {  // d/dr of the reciprocal energy of delta alone (its potential in Phi2)
      const T f0 = Dli.x * es[0] + Dli.y * es[3] + Dli.z * es[6];
      const T f1 = Dli.x * es[1] + Dli.y * es[4] + Dli.z * es[7];
      const T f2 = Dli.x * es[2] + Dli.y * es[5] + Dli.z * es[8];
      T h0 = 0, h1 = 0, h2 = 0;
      stencil(a.Phi2 + M.r0, [&](int j1, T A, T Bv, T C, T Dv, T E, T F) {
        const T t1 = sh[sub][0][0][j1], u1 = sh[sub][1][0][j1], v1 = sh[sub][2][0][j1];
        h0 += f0 * v1 * A + f1 * u1 * Bv + f2 * u1 * C;
        h1 += f0 * u1 * Bv + f1 * t1 * Dv + f2 * t1 * E;
        h2 += f0 * u1 * C + f1 * t1 * E + f2 * t1 * F;
      });
      // the pair part is KE (gx + gs); the reciprocal part of -U_rec(0, delta) enters with a minus sign
      gs0 = -h0 * es[0] - h1 * es[1] - h2 * es[2];
      gs1 = -h0 * es[3] - h1 * es[4] - h2 * es[5];
      gs2 = -h0 * es[6] - h1 * es[7] - h2 * es[8];
    }
    const T e0 = di.x * es[0] + di.y * es[3] + di.z * es[6];
    const T e1 = di.x * es[1] + di.y * es[4] + di.z * es[7];
    const T e2 = di.x * es[2] + di.y * es[5] + di.z * es[8];
    stencil(a.Phi + M.r0, [&](int j1, T A, T Bv, T C, T Dv, T E, T F) {
      const T t1 = sh[sub][0][0][j1], u1 = sh[sub][1][0][j1], v1 = sh[sub][2][0][j1];
      const T qt = qi * t1 + e0 * u1, qu = qi * u1 + e0 * v1;
      ge0 += u1 * A;
      ge1 += t1 * Bv;
      ge2 += t1 * C;
      gw0 += qu * A + e1 * u1 * Bv + e2 * u1 * C;
      gw1 += qt * Bv + e1 * t1 * Dv + e2 * t1 * E;
      gw2 += qt * C + e1 * t1 * E + e2 * t1 * F;
    });
    ge0 = group_sum<T, QL>(ge0, gm); ge1 = group_sum<T, QL>(ge1, gm); ge2 = group_sum<T, QL>(ge2, gm);
    gw0 = group_sum<T, QL>(gw0, gm); gw1 = group_sum<T, QL>(gw1, gm); gw2 = group_sum<T, QL>(gw2, gm);
    if (lane == 0) {
      T *o = rec[sub];
      o[0] = ge0; o[1] = ge1; o[2] = ge2; o[3] = gw0; o[4] = gw1; o[5] = gw2;
    }
    }
    auto pair = [&](int k, T x, T y, T z, T G0, T G1, T G2, T G3, int t) {
      v4<T> dk = a.D[k];
      if constexpr (SHADOW) {
        const v4<T> Dk = a.Dl[k];
        const T wb = (blk_i && t < nsp) ? T(a.iel_keep) : T(1);  // molecule partners come first in a row
        const T Dix = wb * (Dli.x * x + Dli.y * y + Dli.z * z), Dkx = Dk.x * x + Dk.y * y + Dk.z * z;
        const T DiDk = wb * (Dli.x * Dk.x + Dli.y * Dk.y + Dli.z * Dk.z);
        ee += G2 * Dix * Dkx - G1 * DiDk;
        const T rad2 = -G3 * Dix * Dkx + G2 * DiDk;
        gs0 += rad2 * x + G2 * (wb * Dli.x * Dkx + Dk.x * Dix);
        gs1 += rad2 * y + G2 * (wb * Dli.y * Dkx + Dk.y * Dix);
        gs2 += rad2 * z + G2 * (wb * Dli.z * Dkx + Dk.z * Dix);
      }
      const T qk = dk.w;
      T dix = di.x * x + di.y * y + di.z * z;
      T dkx = dk.x * x + dk.y * y + dk.z * z;
      T didk = di.x * dk.x + di.y * dk.y + di.z * dk.z;
      const T qq = qi * qk, pp = dix * dkx;
      const T tt = qi * dkx - qk * dix;
      // not qq G0: the rounding of a charge product is the same for every pair of its kind, a bias (2.2e-8 of a water
      // box's energy in FP32)
      ee += qi * (qk * G0) + tt * G1 - G2 * pp + G1 * didk;
      const T radial = -qq * G1 - tt * G2 + G3 * pp - G2 * didk;
      // the gradient is radial x + u1 dk - u2 di, the field of (q_k, d_k) G1 dk - u2 x
      const T u1 = qi * G1 - G2 * dix, u2 = qk * G1 + G2 * dkx;
      T gxv = radial * x + u1 * dk.x - u2 * di.x;
      T gyv = radial * y + u1 * dk.y - u2 * di.y;
      T gzv = radial * z + u1 * dk.z - u2 * di.z;
      fd0 += G1 * dk.x - u2 * x; fd1 += G1 * dk.y - u2 * y; fd2 += G1 * dk.z - u2 * z;
      T kx = T(KE) * gxv, ky = T(KE) * gyv, kz = T(KE) * gzv;
      c2<T> lj;
      lj.x = T(0); lj.y = T(0);
      if (a.lj && sei != T(0)) lj = a.ljp[k];  // only the rows of atoms with an LJ term ask for it
      T ep = sei * lj.y;
      if (t >= nsp && ep != T(0)) {  // LJ: not for molecule partners, nor pairs without an LJ term
        T rm = rhi + lj.x;
        T r2 = x * x + y * y + z * z;
        const T ir2 = T(1) / r2;
        T s2 = rm * rm * ir2, s6 = s2 * s2 * s2;
        el += ep * (s6 * s6 - T(2) * s6);
        T dl = ep * T(12) * (s6 - s6 * s6) * ir2;
        gl0 += dl * x; gl1 += dl * y; gl2 += dl * z;
        kx += dl * x; ky += dl * y; kz += dl * z;
      }
      gx0 += gxv; gx1 += gyv; gx2 += gzv;
      w[0] += kx * x; w[1] += kx * y; w[2] += kx * z;
      w[3] += ky * x; w[4] += ky * y; w[5] += ky * z;
      w[6] += kz * x; w[7] += kz * y; w[8] += kz * z;
    };
    if constexpr (sizeof(T) == 4) {
      // 16-byte loads of four consecutive entries of every row array: a chunk per round
      static_assert(QL == 8, "eight lanes cover a chunk");
      const unsigned char *at = row + lane * 16;
      auto v4at = [](const unsigned char *p) { return __ldcs(reinterpret_cast<const float4 *>(p)); };
      for (int t = 4 * lane; t < n; t += 32, at += C::SIZE) {
        const int4 kk = __ldcs(reinterpret_cast<const int4 *>(at));
        const float4 xx = v4at(at + C::X), yy = v4at(at + C::Y), zz = v4at(at + C::Z);
        const float4 a1 = v4at(at + C::G1), a2 = v4at(at + C::G2), a0 = v4at(at + C::G0), a3 = v4at(at + C::G3);
        pair(kk.x, xx.x, yy.x, zz.x, a0.x, a1.x, a2.x, a3.x, t);
        if (t + 1 < n) pair(kk.y, xx.y, yy.y, zz.y, a0.y, a1.y, a2.y, a3.y, t + 1);
        if (t + 2 < n) pair(kk.z, xx.z, yy.z, zz.z, a0.z, a1.z, a2.z, a3.z, t + 2);
        if (t + 3 < n) pair(kk.w, xx.w, yy.w, zz.w, a0.w, a1.w, a2.w, a3.w, t + 3);
      }
    } else {
      for (int t = lane; t < n; t += QL) {
        unsigned char *c = row_entry<T>(row, t);
        pair(entry_k<T>(c, t), entry_v<T, C::X>(c, t), entry_v<T, C::Y>(c, t), entry_v<T, C::Z>(c, t), entry_v<T, C::G0>(c, t),
             entry_v<T, C::G1>(c, t), entry_v<T, C::G2>(c, t), entry_v<T, C::G3>(c, t), t);
      }
    }
    if (a.rnv) {  // split rows: the LJ pairs between elec_cutoff and cutoff
      const int nv = min(a.rnv[i], a.mc - a.mce);
      for (int t = lane; t < nv; t += QL) {
        const int e = a.mce + t;
        unsigned char *c = row_entry<T>(row, e);
        const int k = entry_k<T>(c, e);
        const T x = entry_v<T, C::X>(c, e), y = entry_v<T, C::Y>(c, e), z = entry_v<T, C::Z>(c, e);
        T rm = rhi + a.rminh[k], ep = sei * a.seps[k];
        T r2 = x * x + y * y + z * z;
        const T ir2 = T(1) / r2;
        T s2 = rm * rm * ir2, s6 = s2 * s2 * s2;
        el += ep * (s6 * s6 - T(2) * s6);
        T dl = ep * T(12) * (s6 - s6 * s6) * ir2;
        gl0 += dl * x; gl1 += dl * y; gl2 += dl * z;
        T kx = dl * x, ky = dl * y, kz = dl * z;
        w[0] += kx * x; w[1] += kx * y; w[2] += kx * z;
        w[3] += ky * x; w[4] += ky * y; w[5] += ky * z;
        w[6] += kz * x; w[7] += kz * y; w[8] += kz * z;
      }
    }
    T red_in[20] = {gx0, gx1, gx2, gl0, gl1, gl2, fd0, fd1, fd2, ee, el, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8]};
#pragma unroll
    for (int k = 0; k < 20; ++k) red_in[k] = group_sum<T, QL>(red_in[k], gm);
    if constexpr (SHADOW) { gs0 = group_sum<T, QL>(gs0, gm); gs1 = group_sum<T, QL>(gs1, gm); gs2 = group_sum<T, QL>(gs2, gm); }
    if (lane == 0) {
      double gd[3], gr[3];
      for (int bb = 0; bb < 3; ++bb) {
        const double s0 = double(scaled(bb, 0)), s1 = double(scaled(bb, 1)), s2 = double(scaled(bb, 2));
        gd[bb] = double(rec[sub][0]) * s0 + double(rec[sub][1]) * s1 + double(rec[sub][2]) * s2;
        gr[bb] = double(rec[sub][3]) * s0 + double(rec[sub][4]) * s1 + double(rec[sub][5]) * s2;
      }
      double d3[3] = {double(di.x), double(di.y), double(di.z)};
      double gx[3] = {double(red_in[0]), double(red_in[1]), double(red_in[2])};
      double gl[3] = {double(red_in[3]), double(red_in[4]), double(red_in[5])};
      double fd[3] = {double(red_in[6]), double(red_in[7]), double(red_in[8])};
      double4 of = a.off[i];
      double ofs[3] = {of.x, of.y, of.z};
      double cs = a.c_self;
      double dE[3];
      const double gsh[3] = {double(gs0), double(gs1), double(gs2)};
      for (int c = 0; c < 3; ++c) {
        a.forces[3 * i + c] = -(KE * gx[c] + gl[c] + KE * gr[c] + (SHADOW ? KE * gsh[c] : 0.0));
        dE[c] = KE * (fd[c] + gd[c] - cs * d3[c]);
      }
      if constexpr (SHADOW) {
        const double dl2 = double(Dli.x) * double(Dli.x) + double(Dli.y) * double(Dli.y) + double(Dli.z) * double(Dli.z);
        vals[13] = dl2;
        vals[14] = dl2 / (2.0 * double(a.alpha[i]));
      }
      a.dEdd[i] = make_double4(dE[0], dE[1], dE[2], 0);
      vals[0] = double(red_in[9]);
      vals[1] = double(red_in[10]);
      vals[2] = d3[0] * d3[0] + d3[1] * d3[1] + d3[2] * d3[2];
      if (a.induce && mu) {
        double m0 = mu[3 * i], m1 = mu[3 * i + 1], m2 = mu[3 * i + 2];
        vals[3] = (m0 * m0 + m1 * m1 + m2 * m2) / (2.0 * double(a.alpha[i]));
      }
      // virial: 1/2 sum_rows g (x) x - (KE gx + gl) (x) off - KE (dU/dr (x) off + dU/dd (x) d)
      for (int aa = 0; aa < 3; ++aa)
        for (int bb = 0; bb < 3; ++bb)
          vals[4 + aa * 3 + bb] = 0.5 * double(red_in[11 + aa * 3 + bb]) - (KE * gx[aa] + gl[aa]) * ofs[bb] - KE * (gr[aa] * ofs[bb] + gd[aa] * d3[bb]);
    }
  }
  constexpr int NV = SHADOW ? 15 : 13;
  if (lane == 0)
    for (int k = 0; k < NV; ++k) red[sub][k] = vals[k];
  __syncthreads();
  if (threadIdx.x < NV) {
    double v = 0;
    for (int w2 = 0; w2 < ATOMS_PER_BLOCK; ++w2) v += red[w2][threadIdx.x];
    EnergyAcc &E = a.eacc[s];
    double *dst = threadIdx.x == 0 ? &E.e_pair : threadIdx.x == 1 ? &E.e_lj : threadIdx.x == 2 ? &E.d2
                  : threadIdx.x == 3 ? &E.upol : threadIdx.x == 13 ? &E.dd2 : threadIdx.x == 14 ? &E.dda
                  : &E.vir[threadIdx.x - 4];
    atomicAdd(dst, v);
  }
}

// Energies and virial of every system (forcefield.py:2011-2045, 2420-2430, lj.py:87-114):
// E_elec = KE [rows/2 + U_rec + U_self + U_bg + U_pol], E_vdw = rows/2 + tail.
template <typename T>
__device__ __forceinline__ void energy_finish(const Dev<T> &a, int s, double *energy, double *virial, const EnergyAcc *E2, double omega) {
  const double beta = a.beta, c_self = a.c_self, cutoff = a.cutoff;
  const int lj = a.lj, lj_lrc = a.lj_lrc, induce = a.induce;
  unsigned *status = a.status;
  const EnergyAcc &e = a.eacc[s];
  const SysInfo &S = a.sys[s];
  double vol = a.box[s].vol;
  double uself = -(beta / SQRT_PI) * S.sum_q2 - 0.5 * c_self * e.d2;
  double urec_delta = 0.0;
  if (E2) {  // iEL/0-SCF shadow energy (forcefield.py:2037-2042)
    uself += 0.5 * c_self * e.dd2 - (1.0 - 1.0 / omega) * e.dda;
    urec_delta = E2[s].vinf[0];
  }
  double ubg = -PI * S.sum_q * S.sum_q / (2.0 * vol * beta * beta);
  double upol = induce ? e.upol : 0.0;
  double elec = 0.5 * KE * e.e_pair + KE * (e.vinf[0] - urec_delta + uself + ubg + upol);
  double tail = (lj && lj_lrc) ? -2.0 * PI * S.tail_sb / (3.0 * vol * cutoff * cutoff * cutoff) : 0.0;
  double vdw = 0.5 * e.e_lj + tail;
  if (energy) {
    energy[3 * s] = elec;
    energy[3 * s + 1] = vdw;
    energy[3 * s + 2] = elec + vdw;
  }
  if (!isfinite(elec + vdw)) atomicOr(&status[s], 0x4u);
  if (virial) {
    double W[9];
    for (int k = 0; k < 9; ++k) W[k] = e.vir[k];
    W[0] += KE * e.vinf[1]; W[4] += KE * e.vinf[2]; W[8] += KE * e.vinf[3];
    W[1] += KE * e.vinf[4]; W[3] += KE * e.vinf[4];
    W[2] += KE * e.vinf[5]; W[6] += KE * e.vinf[5];
    W[5] += KE * e.vinf[6]; W[7] += KE * e.vinf[6];
    for (int c = 0; c < 3; ++c) W[4 * c] += -KE * ubg - 2.0 * tail;
    for (int k = 0; k < 9; ++k) virial[9 * s + k] = W[k];
  }
}

// Covalent-dipole frames: p_i = sum c unit(r_j - r_i); the pull-back of dE/dd_i onto r_i and r_j
// (the vector-Jacobian product of forcefield.py:2412).  One thread per covalent dipole; the first threads
// finish the systems' energies.
template <typename T>
__global__ void k_finish(Dev<T> a, double *energy, double *virial, const EnergyAcc *E2, double omega) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  for (int s = m; s < a.nsys; s += gridDim.x * blockDim.x) energy_finish(a, s, energy, virial, E2, omega);
  if (m >= a.ncov || !a.perm) return;
  int i = a.cov_i_flat[m], j = a.cov_j_flat[m];
  const BoxInfo &B = a.box[system_of(a, i)];
  double vx = a.pos[3 * j] - a.pos[3 * i], vy = a.pos[3 * j + 1] - a.pos[3 * i + 1], vz = a.pos[3 * j + 2] - a.pos[3 * i + 2];
  min_image(vx, vy, vz, B.H);
  double l = sqrt(vx * vx + vy * vy + vz * vz);
  double ux = vx / l, uy = vy / l, uz = vz / l;
  double4 g = a.dEdd[i];
  double ug = ux * g.x + uy * g.y + uz * g.z;
  double c = a.cov_c_flat[m] / l;
  double gx = c * (g.x - ux * ug), gy = c * (g.y - uy * ug), gz = c * (g.z - uz * ug);
  atomicAdd(&a.forces[3 * j], -gx); atomicAdd(&a.forces[3 * j + 1], -gy); atomicAdd(&a.forces[3 * j + 2], -gz);
  atomicAdd(&a.forces[3 * i], gx); atomicAdd(&a.forces[3 * i + 1], gy); atomicAdd(&a.forces[3 * i + 2], gz);
}

// d = p + mu (energy pass), in T; the energy accumulators of the pass start at zero.
template <typename T>
__global__ void k_total_dipoles(Dev<T> a, const double *mu) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double m[3] = {0, 0, 0};
  if (mu && i < a.nt)
    for (int c = 0; c < 3; ++c) m[c] = mu[3 * (size_t)i + c];
  energy_start(a, i, m);
}

// Copy of a (N, 3) FP64 array into v4<T> (pgm_field input).
template <typename T>
__global__ void k_load_vec(Dev<T> a, const double *v, v4<T> *out) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  v4<T> d;
  d.x = T(v[3 * i]); d.y = T(v[3 * i + 1]); d.z = T(v[3 * i + 2]); d.w = a.q[i];
  out[i] = d;
}

template <typename T>
__global__ void k_store_vec(Dev<T> a, const v4<T> *in, double *v) {
  pdl_enter();  // launched as a programmatic dependent of the previous kernel
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  v4<T> d = in[i];
  v[3 * i] = double(d.x); v[3 * i + 1] = double(d.y); v[3 * i + 2] = double(d.z);
}

}  // namespace pgm
