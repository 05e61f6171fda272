// pgm_fft.cuh -- the 3D FFTs of the PME convolution: per mesh length N a compiled two-step transform.
//
// N = N1 N2 (N1 the smallest divisor >= sqrt(N)): n = n2 + N2 n1, k = k1 + N1 k2,
//   X[k1 + N1 k2] = sum_n2 w_N2^(n2 k2) [ w_N^(n2 k1) sum_n1 w_N1^(n1 k1) x[n2 + N2 n1] ],
// w_M = exp(-2 pi i / M).  A thread holds the N1 points of one n2 (step 1), then the N2 points of one
// k1 (step 2), both in registers; the line crosses shared memory once in between, and the data
// come from and go to global memory straight from registers.  Step 2 leaves a thread with the points
// k1 + N1 k2, which is what the inverse transform starts from, so the convolution pass runs both
// directions with two exchanges.  The inverse transform is the forward one on swapped real and
// imaginary parts.
//
// What bounds a pass: the meshes sit in L2 and a pass reads and writes them once.  By the counters: the plane passes
// (96^3) by their barriers and by having 96 CTAs for 148 SMs, issue 30 % of the slots; at 192^3 the k3 passes by L1
// throughput (71 to 75 %), the k2 and k1 passes by load latency and barriers (issue 42 to 50 %).  A staged
// shared-memory Stockham plan
// (radix 8, 4, 2, 3, 5; one barrier and one shared round trip per radix) had 4 to 6 barriers a line.
// Chains of a convolution, FP32, that plan -> this: 192^3 122 -> 73 us, 96^3 20.3 -> 15.6; a length that the plan
// had at run time only, 108^3: 68 -> 20.
#pragma once
#include "pgm_device.cuh"

namespace pgmfft {

using pgm::BoxInfo;
using pgm::c2;
using pgm::CGSys;
using pgm::EnergyAcc;

// What the passes read and write (the buffers of all systems).
template <typename T>
struct Args {
  T *Q, *Phi;
  const T *Ginf;
  c2<T> *C;
  const c2<T> *tw;
  const CGSys *cg;
  const BoxInfo *box;
  EnergyAcc *eacc;
  double beta;
};

// One CTA of a pass: system s, its first line, pair or column c0 (planes: k1) of n, the mesh, its twiddle
// table, grid offsets, and (k2 pass) the share [q0, q1) of the real grid it clears.
struct Tile {
  int s, c0, n, K3h;
  int K2, K3, tw, pad;
  long long rg, cg, q0, q1;
};

// The tiles of a launch: a table, or, with one system, `base` and what follows from the block index --
// c0 = b c_step, rg + b r_step, cg + b g_step, pairs left of `lines`, the share of b -- so that a pass does not
// begin with a load that its other loads wait for.
struct Tiles {
  const Tile *table;
  int one, c_step, lines, pad;
  long long r_step, g_step, share, total;
  Tile base;
};

// Passes of a convolution.
enum Pass { X_FWD, X_INV, Y_PASS, Z_CONV, Z_ENERGY, PLANE_FWD, PLANE_INV };

// Columns (k2, k1 passes) or line pairs (k3 passes) per CTA: 128 bytes of consecutive columns.
template <typename T>
constexpr int tile_width() { return sizeof(T) == 4 ? 16 : 8; }

// Mesh lengths with k3 + k2 plane passes, and the shared memory of one.
constexpr int PLANE_MAX = 128;
size_t plane_smem(int N, size_t real_size);

template <typename T>
bool supported(int N);
template <typename T>
cudaError_t prepare(Pass p, int N);
// One launch of pass p over `ntiles` tiles; sign is the k2 pass's direction (-1 forward).
template <typename T>
cudaError_t launch(Pass p, int N, const Args<T> &a, const Tiles &tiles, int ntiles, int act, int sign, cudaStream_t st, bool dependent);

}  // namespace pgmfft
