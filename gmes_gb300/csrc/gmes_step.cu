// One FDTD time step on the GPU: ghost-plane copies, the fused E and H
// half-step kernels over all material classes, and the point sources.
//
// Reference path replaced (GMES): FDTD.step (gmes/fdtd.py:1099-1122) with
// talk_with_*_neighbors (gmes/fdtd.py:811-1097), update_e?/h?
// (gmes/fdtd.py:673-809) and the per-point updaters of src/pw_*.hh.
//
// Index geometry.  With N = whole_field_size, every E component is updated
// on the N0 x N1 x N2 "cells" (i, j, k) (the last plane along each non-own
// axis is a ghost, src/pw_dummy.hh semantics via gmes/fdtd.py:365-470), and
// every H component on the same cells shifted by +1 along its two non-own
// axes (its first planes are the ghosts).  One thread owns one cell and
// updates the three components of its half-step there, so each kernel reads
// every neighbouring field value through L1/L2 and writes each updated value
// once.  For component c with own axis a and curl axes a1 = a+1, a2 = a+2
// (mod 3):
//   E_c at x:  D1 = H_{a2}[x + e_a + e_a1] - H_{a2}[x + e_a]
//              D2 = H_{a1}[x + e_a + e_a2] - H_{a1}[x + e_a]
//   H_c at x + e_a1 + e_a2:
//              D1 = E_{a2}[x + e_a1] - E_{a2}[x],  D2 = E_{a1}[x + e_a2] - E_{a1}[x]
// which is exactly the (in1, in2, d1, d2) binding of gmes/fdtd.py:673-809
// and the stencils of src/pw_dielectric.hh:118-371.
#include <cstring>

#include "gmes_cell.cuh"

namespace gmes {
namespace {

// Threads per block of the cell kernels, single-grid and multi-grid:
// kCellThreads (16 cells along k by 8 rows).  Measured on GB300, Gcell/s at
// 128 / 256 / 512 threads (the same registers and resident warps per SM):
//   256^3 cube        FP64 17.34 / 16.70 / 14.97   FP32 33.66 / 33.42   df64 21.80 / 20.98
//   192^3 dispersive  FP64  9.81 /  9.36 /  8.70   FP32 20.26 / 19.85   df64 14.76 / 13.75
// GMES_CELL_THREADS overrides it (tuning builds).
//
// Resident blocks per SM the cell kernels' register budget targets (blocks
// of 128 threads).  Measured on GB300 with the warp-uniform plain path
// (256^3 cube, Gcell/s):
//   FP64  7 blocks (72 registers) 17.29   8 (64) 18.48   9 (56) 18.90
//   FP32  10 blocks (48) 34.31           11 (46) 39.40  12 (40) 39.42
//   df64  7 blocks 20.44                 8 (64) 22.33   9 (56) 22.60  10 (48) 24.19
//   (FP64 at 10 blocks 18.71; FP32 at 14 or 16 blocks, spilling, 35.7)
// FP32 is bound by the loads in flight, so extra resident warps pay most
// there; FP64 is bound by its pipe.  GMES_CELL_BLOCKS_F64 / _F32 / _DF
// override them (tuning builds).
#ifndef GMES_CELL_BLOCKS_F64
#define GMES_CELL_BLOCKS_F64 9
#endif
#ifndef GMES_CELL_BLOCKS_F32
#define GMES_CELL_BLOCKS_F32 12
#endif
#ifndef GMES_CELL_BLOCKS_DF
#define GMES_CELL_BLOCKS_DF 10
#endif
// The H half (GMES_CELL_BLOCKS_F64_H / _F32_H / _DF_H) and the E half of
// dispersive grids (the kernel with the Drude / Lorentz / DCP updates, _D)
// take their own budgets.  Measured on GB300, ms per half-step:
//   df64 H, 256^3 cube, 10 / 9 / 8 blocks: 0.3275 / 0.3403 / 0.3223 (8: 64
//     registers, no spills; at 10 the hot path spilled)
//   dispersive E, 192^3, blocks 12 or 10 (the E budget) / 9 / 8 / 7 / 6:
//     FP32 0.1937 / 0.1701 / 0.1812 / -      / -      (9: no spills)
//     df64 0.2733 / 0.2581 / 0.2693 / 0.2574 / 0.2751
//     FP64 0.4052 (9) / -   / 0.4041 / 0.4035 / 0.4107
//   (FP32 H at 10 blocks and FP64 H at 8 ran 1-2 % slower than their E
//   budgets.  Re-measured with these: 256^3 cube df64 E at 8 blocks 0.329
//   vs 0.316; FP32 E / H at 9 or 8 blocks 0.230 / 0.254 vs 0.203 / 0.205,
//   H alone at 9 0.254; FP64 E at 8 0.4485 vs 0.4435, H at 7 0.4638 vs
//   0.4428.)
#ifndef GMES_CELL_BLOCKS_F64_H
#define GMES_CELL_BLOCKS_F64_H GMES_CELL_BLOCKS_F64
#endif
#ifndef GMES_CELL_BLOCKS_F32_H
#define GMES_CELL_BLOCKS_F32_H GMES_CELL_BLOCKS_F32
#endif
#ifndef GMES_CELL_BLOCKS_DF_H
#define GMES_CELL_BLOCKS_DF_H 8
#endif
#ifndef GMES_CELL_BLOCKS_F64_D
#define GMES_CELL_BLOCKS_F64_D 7
#endif
#ifndef GMES_CELL_BLOCKS_F32_D
#define GMES_CELL_BLOCKS_F32_D 9
#endif
#ifndef GMES_CELL_BLOCKS_DF_D
#define GMES_CELL_BLOCKS_DF_D 9
#endif
constexpr int cell_blocks(int e, int h, int d, int side, bool disp) {
  return (side == 1 ? h : (disp ? d : e)) * 128 / kCellThreads;
}
template <class P, int SIDE, bool DISP>
struct CellMinBlocks {
  static constexpr int value = cell_blocks(GMES_CELL_BLOCKS_F64, GMES_CELL_BLOCKS_F64_H,
                                           GMES_CELL_BLOCKS_F64_D, SIDE, DISP);
};
template <int SIDE, bool DISP>
struct CellMinBlocks<PolF32, SIDE, DISP> {
  static constexpr int value = cell_blocks(GMES_CELL_BLOCKS_F32, GMES_CELL_BLOCKS_F32_H,
                                           GMES_CELL_BLOCKS_F32_D, SIDE, DISP);
};
template <int SIDE, bool DISP>
struct CellMinBlocks<PolDF, SIDE, DISP> {
  static constexpr int value = cell_blocks(GMES_CELL_BLOCKS_DF, GMES_CELL_BLOCKS_DF_H,
                                           GMES_CELL_BLOCKS_DF_D, SIDE, DISP);
};
// The multi-grid cell kernels carry a tile loop and a grid look-up on top of
// the cell body (GMES_MULTI_BLOCKS_F64 / _F32 / _DF override the budgets).
// Measured on GB300 (one 160^3 cube in a batch, descriptors as launch
// arguments, ms per step): FP32 at 8 / 10 / 12 blocks 0.203 / 0.174 / 0.187;
// FP64 at 7 / 8 / 9 blocks 0.304 / 0.302 / 0.292.  Re-measured with chunks
// replayed as CUDA graphs and the tile range from the host: FP32 at 10 / 12
// blocks 0.158 / 0.164; df64 at 9 / 10 / 12 blocks 0.224 / 0.236 / 0.246.
#ifndef GMES_MULTI_BLOCKS_F64
#define GMES_MULTI_BLOCKS_F64 9
#endif
#ifndef GMES_MULTI_BLOCKS_F32
#define GMES_MULTI_BLOCKS_F32 10
#endif
#ifndef GMES_MULTI_BLOCKS_DF
#define GMES_MULTI_BLOCKS_DF 9
#endif
// The H half (_H) and the E half of dispersive grids (_D) may take their
// own budgets; by default the precision's.  (FP64, 34 grids of the serving
// mix below 2^20 cells, 25 of them dispersive, ms per 64-step chunk: 141.5
// at 9 blocks; H at 8 / 7 blocks 143.6 / 146.5, dispersive E at 7 145.1.)
#ifndef GMES_MULTI_BLOCKS_F64_H
#define GMES_MULTI_BLOCKS_F64_H GMES_MULTI_BLOCKS_F64
#endif
#ifndef GMES_MULTI_BLOCKS_F32_H
#define GMES_MULTI_BLOCKS_F32_H GMES_MULTI_BLOCKS_F32
#endif
#ifndef GMES_MULTI_BLOCKS_DF_H
#define GMES_MULTI_BLOCKS_DF_H GMES_MULTI_BLOCKS_DF
#endif
#ifndef GMES_MULTI_BLOCKS_F64_D
#define GMES_MULTI_BLOCKS_F64_D GMES_MULTI_BLOCKS_F64
#endif
#ifndef GMES_MULTI_BLOCKS_F32_D
#define GMES_MULTI_BLOCKS_F32_D GMES_MULTI_BLOCKS_F32
#endif
#ifndef GMES_MULTI_BLOCKS_DF_D
#define GMES_MULTI_BLOCKS_DF_D GMES_MULTI_BLOCKS_DF
#endif
template <class P, int SIDE, bool DISP>
struct MultiMinBlocks {
  static constexpr int value = cell_blocks(GMES_MULTI_BLOCKS_F64, GMES_MULTI_BLOCKS_F64_H,
                                           GMES_MULTI_BLOCKS_F64_D, SIDE, DISP);
};
template <int SIDE, bool DISP>
struct MultiMinBlocks<PolF32, SIDE, DISP> {
  static constexpr int value = cell_blocks(GMES_MULTI_BLOCKS_F32, GMES_MULTI_BLOCKS_F32_H,
                                           GMES_MULTI_BLOCKS_F32_D, SIDE, DISP);
};
template <int SIDE, bool DISP>
struct MultiMinBlocks<PolDF, SIDE, DISP> {
  static constexpr int value = cell_blocks(GMES_MULTI_BLOCKS_DF, GMES_MULTI_BLOCKS_DF_H,
                                           GMES_MULTI_BLOCKS_DF_D, SIDE, DISP);
};
// Whether a batch of at most kParamJobs grids takes its descriptors from
// the argument bank (k_multi_cell_arg) or copies them to shared memory per
// block (k_multi_cell); GMES_MULTI_ARG_F64 / _F32 / _DF override it.
// Measured on GB300 (one 160^3 cube in a batch, ms per step, argument bank
// / shared memory, single-grid kernel): FP32 0.173 / 0.194 (0.148), df64
// 0.266 / 0.290 (0.220), FP64 0.289 / 0.279 (0.265).
#ifndef GMES_MULTI_ARG_F64
#define GMES_MULTI_ARG_F64 0
#endif
#ifndef GMES_MULTI_ARG_F32
#define GMES_MULTI_ARG_F32 1
#endif
#ifndef GMES_MULTI_ARG_DF
#define GMES_MULTI_ARG_DF 1
#endif
template <class P>
struct ArgDescs {
  static constexpr bool value = GMES_MULTI_ARG_F64 != 0;
};
template <>
struct ArgDescs<PolF32> {
  static constexpr bool value = GMES_MULTI_ARG_F32 != 0;
};
template <>
struct ArgDescs<PolDF> {
  static constexpr bool value = GMES_MULTI_ARG_DF != 0;
};

template <class P, int SIDE, bool STRICT, bool DISP, class I>
__global__ void __launch_bounds__(kCellThreads, CellMinBlocks<P, SIDE, DISP>::value)
    k_cell(const GridDev g, int bx_log2, int i0) {
  after_launch();
  const int bx = 1 << bx_log2;
  const int tx = threadIdx.x & (bx - 1);
  const int ty = threadIdx.x >> bx_log2;
  const int k = blockIdx.x * bx + tx;
  const int j = blockIdx.y * (kCellThreads >> bx_log2) + ty;
  const int i = i0 + (int)blockIdx.z;
  if (k >= g.n[2] || j >= g.n[1] || i >= g.n[0]) return;
  if constexpr (STRICT)
    cell_body<P, SIDE, STRICT, DISP, I>(g, i, j, k);
  else
    cell_body_fast<P, SIDE, DISP, I>(g, i, j, k);
}

// Cells per block row along k (log2): a warp covers 16 cells of two rows
// (128 bytes per row in FP64 and df64, 64 in FP32).  (Measured with blocks
// of 256 threads.)  Against 32 cells of
// one row, a warp straddles a material or CPML edge along k in half as many
// places, so fewer warps run two kinds' code or a psi block for a few
// lanes.  Measured on GB300, Gcell/s, rows of 32 / 16 / 8 cells:
//   256^3 cube (dielectric + CPML)   FP64 16.17 / 16.81 / 15.99
//                                    FP32 32.99 / 33.74 / 29.36
//                                    df64 19.72 / 21.12 / 20.12
//   192^3 dispersive + UPML          FP64  8.06 /  9.42 /  9.69
//                                    FP32 19.34 / 20.08 / 18.47
//                                    df64 12.73 / 13.86 / 13.80
// (FP64 E half of the cube: 14.4 -> 13.7 FP64 warp-instructions per cell,
// what a warp-level count of the slabs predicts for both shapes.)  The row
// length is kRowLog2 (cell_tiling).

template <class P, bool STRICT, class I>
void launch_cell(const GridDev& d, int side, bool disp, dim3 grid, int bx_log2, int i0,
                 cudaStream_t s) {
  auto go = [&](auto kernel) { launch_after(true, kernel, grid, kCellThreads, 0, s, d, bx_log2, i0); };
  if (side == 0) {
    if (disp)
      go(k_cell<P, 0, STRICT, true, I>);
    else
      go(k_cell<P, 0, STRICT, false, I>);
  } else {
    go(k_cell<P, 1, STRICT, false, I>);
  }
}

// Ghost planes of one half's components (gmes/fdtd.py:811-1097 with the
// single-domain cyclic communicator): E ghosts are the last planes along the
// non-own axes and receive plane 0; H ghosts are the first planes and
// receive the last plane.  A ghost point's source is found by mapping every
// ghost coordinate at once, so corners get the value the reference's two
// successive plane copies give them and no source is itself a ghost.
template <class T>
__device__ __forceinline__ void ghost_point(const GridDev& g, int side, int item, int64_t t) {
  const int c = side * 3 + item / 2;
  if (!(g.active & (1 << c))) return;
  const int own = c % 3;
  const int ga = (item & 1) ? (own + 2) % 3 : (own + 1) % 3;
  const int pa = (ga + 1) % 3, qa = (ga + 2) % 3;
  const int p_ = pa < qa ? pa : qa, q_ = pa < qa ? qa : pa;  // q_ is the faster axis
  const int64_t np = g.sh[c][p_] * g.sh[c][q_];
  if (t >= np) return;
  int64_t x[3];
  x[p_] = t / g.sh[c][q_];
  x[q_] = t - x[p_] * g.sh[c][q_];
  x[ga] = side == 0 ? g.sh[c][ga] - 1 : 0;
  int64_t s[3] = {x[0], x[1], x[2]};
  const int a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  for (int h = 0; h < 2; ++h) {
    const int ax = h == 0 ? a1 : a2;
    if (side == 0) {
      if (x[ax] == g.sh[c][ax] - 1) s[ax] = 0;
    } else {
      if (x[ax] == 0) s[ax] = g.sh[c][ax] - 1;
    }
  }
  T* f = static_cast<T*>(g.f[c]);
  const int64_t dst = x[0] * g.st[c][0] + x[1] * g.st[c][1] + x[2];
  const int64_t src = s[0] * g.st[c][0] + s[1] * g.st[c][1] + s[2];
  f[dst] = f[src];
}

template <class T>
__global__ void k_ghost(const GridDev g, int side, int64_t maxplane) {
  after_launch();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= maxplane) return;
  ghost_point<T>(g, side, blockIdx.y, t);
}

// The same for grids whose components hold fewer than 2^31 points: 32-bit
// index arithmetic (one unsigned division per point instead of a 64-bit
// one).  Same points, same copies.
template <class T>
__global__ void k_ghost32(const GridDev g, int side, unsigned maxplane) {
  after_launch();
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= maxplane) return;
  const int item = blockIdx.y;
  const int c = side * 3 + item / 2;
  if (!(g.active & (1 << c))) return;
  const int own = c % 3;
  const int ga = (item & 1) ? (own + 2) % 3 : (own + 1) % 3;
  const int pa = (ga + 1) % 3, qa = (ga + 2) % 3;
  const int p_ = pa < qa ? pa : qa, q_ = pa < qa ? qa : pa;  // q_ is the faster axis
  const unsigned sh[3] = {(unsigned)g.sh[c][0], (unsigned)g.sh[c][1], (unsigned)g.sh[c][2]};
  if (t >= sh[p_] * sh[q_]) return;
  unsigned x[3];
  x[p_] = t / sh[q_];
  x[q_] = t - x[p_] * sh[q_];
  x[ga] = side == 0 ? sh[ga] - 1 : 0;
  unsigned s[3] = {x[0], x[1], x[2]};
  const int a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  if (side == 0) {
    if (x[a1] == sh[a1] - 1) s[a1] = 0;
    if (x[a2] == sh[a2] - 1) s[a2] = 0;
  } else {
    if (x[a1] == 0) s[a1] = sh[a1] - 1;
    if (x[a2] == 0) s[a2] = sh[a2] - 1;
  }
  const unsigned st0 = (unsigned)g.st[c][0], st1 = (unsigned)g.st[c][1];
  T* f = static_cast<T*>(g.f[c]);
  f[x[0] * st0 + x[1] * st1 + x[2]] = f[s[0] * st0 + s[1] * st1 + s[2]];
}

// Ghost planes of a complex grid (Bloch boundary, gmes/fdtd.py:811-1097):
// as ghost_point, but the value is multiplied by the phase factor of each
// ghost axis in the reference's copy order (own+1, then own+2).  The
// imaginary plane follows the real plane of every component.  Strict: the
// product in the fused form numpy's SIMD complex multiply uses,
// re = fma(pr, vr, -(pi vi)), im = fma(pr, vi, pi vr).
template <bool STRICT>
__device__ __forceinline__ void ghost_point_c(const GridDev& g, int side, int item, int64_t t) {
  const int c = side * 3 + item / 2;
  if (!(g.active & (1 << c))) return;
  const int own = c % 3;
  const int ga = (item & 1) ? (own + 2) % 3 : (own + 1) % 3;
  const int pa = (ga + 1) % 3, qa = (ga + 2) % 3;
  const int p_ = pa < qa ? pa : qa, q_ = pa < qa ? qa : pa;
  const int64_t np = g.sh[c][p_] * g.sh[c][q_];
  if (t >= np) return;
  int64_t x[3];
  x[p_] = t / g.sh[c][q_];
  x[q_] = t - x[p_] * g.sh[c][q_];
  x[ga] = side == 0 ? g.sh[c][ga] - 1 : 0;
  int64_t s[3] = {x[0], x[1], x[2]};
  bool ghost[2];
  const int axes[2] = {(own + 1) % 3, (own + 2) % 3};
  for (int h = 0; h < 2; ++h) {
    const int ax = axes[h];
    ghost[h] = side == 0 ? x[ax] == g.sh[c][ax] - 1 : x[ax] == 0;
    if (ghost[h]) s[ax] = side == 0 ? 0 : g.sh[c][ax] - 1;
  }
  double* fr = static_cast<double*>(g.f[c]);
  double* fi = fr + g.npts[c];
  const int64_t dst = x[0] * g.st[c][0] + x[1] * g.st[c][1] + x[2];
  const int64_t src = s[0] * g.st[c][0] + s[1] * g.st[c][1] + s[2];
  double vr = fr[src], vi = fi[src];
  for (int h = 0; h < 2; ++h) {
    if (!ghost[h]) continue;
    const double pr = g.phase[c][h][0], pi = g.phase[c][h][1];
    double nr, ni;
    if (STRICT) {
      nr = __fma_rn(pr, vr, -__dmul_rn(pi, vi));
      ni = __fma_rn(pr, vi, __dmul_rn(pi, vr));
    } else {
      nr = pr * vr - pi * vi;
      ni = pr * vi + pi * vr;
    }
    vr = nr;
    vi = ni;
  }
  fr[dst] = vr;
  fi[dst] = vi;
}

template <bool STRICT>
__global__ void k_ghost_c(const GridDev g, int side, int64_t maxplane) {
  after_launch();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= maxplane) return;
  ghost_point_c<STRICT>(g, side, blockIdx.y, t);
}

// Point sources of one half-step (gmes/pw_source.py:74-131), applied after
// that half's material update.  The values were computed on the host in FP64.
template <class P, bool STRICT>
__global__ void k_sources(const GridDev g, int side, int64_t slot) {
  after_launch();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.nsrc) return;
  source_point<P, STRICT>(g, side, slot, q);
}

// TFSF consistency corrections of one half (gmes/pw_source.py:134-486):
// after the material update and the point sources, every face of a
// transparent point adds coef * (r0 A[s] + r1 A[s+1]) in face order, A the
// incident-field grid's Hy (E side) or Ex (H side).  Strict: the
// reference's operation order (coef is the signed dt/(eps d) * amp).
template <class P, bool STRICT>
__global__ void k_transparent(const GridDev g, int side) {
  after_launch();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.ntfsf) return;
  const gmes_transparent& t = g.tfsf[q];
  const int c = __ldg(&t.comp);
  if (c < 0 || c > 5 || !(g.active & (1 << c)) || (c < 3) != (side == 0)) return;
  const int64_t off = __ldg(&t.offset);
  if (off < 0 || off >= g.npts[c]) return;
  const int nf = __ldg(&t.nface);
  using T = typename P::T;
  using R = typename P::R;
  const T* A = static_cast<const T*>(g.tf_field[side]);
  const int64_t na = g.tf_npts[side];
  T* f = static_cast<T*>(g.f[c]) + off;
  if constexpr (STRICT) {
    double v = *reinterpret_cast<double*>(f);
    const double* a = reinterpret_cast<const double*>(A);
    for (int k = 0; k < nf && k < GMES_TFSF_MAX_FACES; ++k) {
      const int64_t sp = __ldg(&t.sample[k]);
      if (sp < 0 || sp + 1 >= na) continue;
      const double inc = __dadd_rn(__dmul_rn(__ldg(&t.r0[k]), a[sp]),
                                   __dmul_rn(__ldg(&t.r1[k]), a[sp + 1]));
      v = __dadd_rn(v, __dmul_rn(__ldg(&t.coef[k]), inc));
    }
    *reinterpret_cast<double*>(f) = v;
  } else {
    R v = P::ldw(f);
    for (int k = 0; k < nf && k < GMES_TFSF_MAX_FACES; ++k) {
      const int64_t sp = __ldg(&t.sample[k]);
      if (sp < 0 || sp + 1 >= na) continue;
      const R inc = P::from_double(__ldg(&t.r0[k])) * P::ldw(A + sp) +
                    P::from_double(__ldg(&t.r1[k])) * P::ldw(A + sp + 1);
      v = v + P::from_double(__ldg(&t.coef[k])) * inc;
    }
    P::st(f, v);
  }
}

// Probe recording of one half: the value of every probe of this half's
// components after its updates, sources and TFSF corrections.
template <class P>
__global__ void k_probes(const GridDev g, int side, int64_t slot) {
  after_launch();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.nprobe) return;
  const gmes_probe pr = g.probe[q];
  if (pr.comp < 0 || pr.comp > 5 || (pr.comp < 3) != (side == 0)) return;
  double v = 0.0;
  if ((g.active & (1 << pr.comp)) && pr.offset >= 0 && pr.offset < g.npts[pr.comp])
    v = to_double(P::ldw(static_cast<const typename P::T*>(g.f[pr.comp]) + pr.offset));
  g.probe_val[slot * g.nprobe + q] = v;
}

// ---------------------------------------------------------------------------
// Multi-grid ("batch") form: one launch per half-step advances every grid of
// a batch.  The per-grid views live in a caller-allocated workspace with
// prefix sums of each grid's blocks, ghost-plane points and sources; a block
// (or thread) finds its grid by binary search in the prefix array and runs
// exactly the per-grid code, so a grid's result does not depend on what else
// is in the batch.  Grids with steps[g] <= s sit out step s of the chunk.
// ---------------------------------------------------------------------------
template <class I>
__device__ __forceinline__ int find_job(const I* prefix, int njobs, I v) {
  int lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(prefix + mid) <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

static_assert(sizeof(GridDev) % 16 == 0, "GridDev is copied as 16-byte words");

// The tile's grid descriptor is copied to shared memory when the block's
// job changes and read from there: read from global memory, its fields
// (pointers, strides, tables of six components) cost the batched FP32
// half-step ~70 extra global loads per cell and ran it 1.7x slower than
// the single-grid kernel, whose descriptor is a kernel parameter; from
// shared memory it runs 1.3x slower (measured on GB300, 160^3 cube).
template <class P, int SIDE, bool STRICT, bool DISP>
__global__ void __launch_bounds__(kBatchThreads, MultiMinBlocks<P, SIDE, DISP>::value)
    k_multi_cell(const BatchView v, int s, int64_t per) {
  after_launch();
  __shared__ __align__(16) unsigned char desc[sizeof(GridDev)];
  const GridDev& g = *reinterpret_cast<const GridDev*>(desc);
  int cached = -1;
  // a persistent grid (fewer blocks than tiles) gives each block a
  // contiguous range of per tiles (ceil(tiles / blocks), from the host: a
  // 64-bit division here cost every thread tens of instructions), so that a
  // block mostly stays on one grid and copies its descriptor once
  const int64_t b0 = (int64_t)blockIdx.x * per;
  const int64_t b1 = b0 + per < v.tiles ? b0 + per : v.tiles;
  for (int64_t b = b0; b < b1; ++b) {
    const int job = find_job<int64_t>(v.tile_prefix, v.njobs, b);  // block-uniform
    if (s >= __ldg(v.steps + job)) continue;
    if (job != cached) {
      __syncthreads();  // the previous descriptor is no longer read
      const uint4* src = reinterpret_cast<const uint4*>(v.jobs + job);
      uint4* dst = reinterpret_cast<uint4*>(desc);
      for (int w = threadIdx.x; w < (int)(sizeof(GridDev) / 16); w += blockDim.x)
        dst[w] = __ldg(src + w);
      __syncthreads();
      cached = job;
    }
    const TileDiv& td = v.td[job];
    const int bxl = __ldg(&td.bxl);
    const int bx = 1 << bxl, by = kBatchThreads >> bxl;
    // a grid has fewer than 2^31 tiles: quotients by multiply and shift
    const unsigned local = (unsigned)(b - __ldg(v.tile_prefix + job));
    const unsigned plane = __ldg(&td.plane), nkb = __ldg(&td.nkb);
    const int i = (int)tile_quot(local, __ldg(&td.m_plane), __ldg(&td.s_plane));
    const unsigned rem = local - (unsigned)i * plane;
    const unsigned jq = tile_quot(rem, __ldg(&td.m_nkb), __ldg(&td.s_nkb));
    const int jb = (int)jq, kb = (int)(rem - jq * nkb);
    const int k = kb * bx + (threadIdx.x & (bx - 1));
    const int j = jb * by + (threadIdx.x >> bxl);
    // batched grids hold fewer than 2^31 points per component (checked when
    // the batch is prepared)
    if (k < g.n[2] && j < g.n[1]) {
      if constexpr (STRICT)
        cell_body<P, SIDE, STRICT, DISP, int32_t>(g, i, j, k);
      else
        cell_body_fast<P, SIDE, DISP, int32_t>(g, i, j, k);
    }
  }
}

// The same with the descriptors in the kernel's argument bank (batches of
// at most kParamJobs grids): no shared-memory copy and no barrier per tile.
template <class P, int SIDE, bool STRICT, bool DISP>
__global__ void __launch_bounds__(kBatchThreads, MultiMinBlocks<P, SIDE, DISP>::value)
    k_multi_cell_arg(const BatchView v, int s, int64_t per, const __grid_constant__ BatchDescs d) {
  after_launch();
  const int64_t b0 = (int64_t)blockIdx.x * per;
  const int64_t b1 = b0 + per < v.tiles ? b0 + per : v.tiles;
  for (int64_t b = b0; b < b1; ++b) {
    const int job = find_job<int64_t>(v.tile_prefix, v.njobs, b);  // block-uniform
    if (s >= __ldg(v.steps + job)) continue;
    const GridDev& g = d.jobs[job];
    const TileDiv& td = v.td[job];
    const int bxl = __ldg(&td.bxl);
    const int bx = 1 << bxl, by = kBatchThreads >> bxl;
    // a grid has fewer than 2^31 tiles: quotients by multiply and shift
    const unsigned local = (unsigned)(b - __ldg(v.tile_prefix + job));
    const unsigned plane = __ldg(&td.plane), nkb = __ldg(&td.nkb);
    const int i = (int)tile_quot(local, __ldg(&td.m_plane), __ldg(&td.s_plane));
    const unsigned rem = local - (unsigned)i * plane;
    const unsigned jq = tile_quot(rem, __ldg(&td.m_nkb), __ldg(&td.s_nkb));
    const int jb = (int)jq, kb = (int)(rem - jq * nkb);
    const int k = kb * bx + (threadIdx.x & (bx - 1));
    const int j = jb * by + (threadIdx.x >> bxl);
    if (k < g.n[2] && j < g.n[1]) {
      if constexpr (STRICT)
        cell_body<P, SIDE, STRICT, DISP, int32_t>(g, i, j, k);
      else
        cell_body_fast<P, SIDE, DISP, int32_t>(g, i, j, k);
    }
  }
}

template <class T>
__global__ void k_multi_ghost(const BatchView v, int side, int s) {
  after_launch();
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < v.ghosts;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int job = find_job<int64_t>(v.ghost_prefix, v.njobs, t);
    if (s >= __ldg(v.steps + job)) continue;
    const GridDev& g = v.jobs[job];
    const int64_t local = t - __ldg(v.ghost_prefix + job);
    const int64_t per = (__ldg(v.ghost_prefix + job + 1) - __ldg(v.ghost_prefix + job)) / 6;
    ghost_point<T>(g, side, (int)(local / per), local % per);
  }
}

template <class P, bool STRICT>
__global__ void k_multi_sources(const BatchView v, int side, int s) {
  after_launch();
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < v.srcs; t += gridDim.x * blockDim.x) {
    const int job = find_job<int>(v.src_prefix, v.njobs, t);
    if (s >= __ldg(v.steps + job)) continue;
    source_point<P, STRICT>(v.jobs[job], side, 2 * (int64_t)s + side, t - __ldg(v.src_prefix + job));
  }
}

template <class P, bool STRICT>
[[nodiscard]] cudaError_t run_steps(const Plan& p, int nsteps, int side_mask, int st0,
                                    cudaStream_t s);

// One half-step: ghost copy of the other half's components, the fused
// update of this half's components, this half's point sources, TFSF
// corrections and probes; after the E half, one full step of the TFSF
// incident-field grid (FDTD.step's _step_aux_fdtd, gmes/fdtd.py:1113).
// A complex grid runs every per-plane kernel on its real and imaginary
// planes; only the ghost copy couples them.
template <class P, bool STRICT>
[[nodiscard]] cudaError_t run_half(const Plan& p, int side, int st, bool early, bool last, cudaStream_t s) {
  using T = typename P::T;
  const GridDev& d = p.re;
  int64_t maxplane = 1;
  for (int c = 0; c < 6; ++c)
    for (int a = 0; a < 3; ++a)
      for (int b = a + 1; b < 3; ++b) {
        const int64_t v = d.sh[c][a] * d.sh[c][b];
        maxplane = v > maxplane ? v : maxplane;
      }
  const dim3 ggrid((unsigned)((maxplane + 255) / 256), 6);
  constexpr int kMaxY = 65535;
  if (p.cplx)
    launch_after(early, k_ghost_c<STRICT>, ggrid, 256, 0, s, d, 1 - side, maxplane);
  else if (offsets_fit_i32(d))
    launch_after(early, k_ghost32<T>, ggrid, 256, 0, s, d, 1 - side, (unsigned)maxplane);
  else
    launch_after(early, k_ghost<T>, ggrid, 256, 0, s, d, 1 - side, maxplane);
  const CellTiling tl = cell_tiling(d.n);
  const int bx_log2 = tl.bx_log2, bx = tl.bx, by = tl.by;
  const int nplanes = p.cplx ? 2 : 1;
  for (int part = 0; part < nplanes; ++part) {
    const GridDev& v = part == 0 ? p.re : p.im;
    for (int i0 = 0; i0 < d.n[0]; i0 += kMaxY) {
      const dim3 grid((unsigned)((d.n[2] + bx - 1) / bx), (unsigned)((d.n[1] + by - 1) / by),
                      (unsigned)min(kMaxY, d.n[0] - i0));
      // Measured on GB300 (256^3 cube): 32-bit offsets run the FP64 step 7%
      // and the df64 step 6% faster than 64-bit ones (fewer registers and
      // spills), so every grid whose components hold fewer than 2^31 points
      // takes them; a compile-time active mask (all six components) ran ~35%
      // slower, so the mask stays a runtime value.
      if (offsets_fit_i32(d))
        launch_cell<P, STRICT, int32_t>(v, side, p.disp, grid, bx_log2, i0, s);
      else
        launch_cell<P, STRICT, int64_t>(v, side, p.disp, grid, bx_log2, i0, s);
    }
  }
  for (int part = 0; part < nplanes; ++part) {
    const GridDev& v = part == 0 ? p.re : p.im;
    if (v.nsrc > 0)
      launch_after(true, k_sources<P, STRICT>, dim3((v.nsrc + 127) / 128), 128, 0, s, v, side,
                   2 * (int64_t)st + side);
    if (v.ntfsf > 0)
      launch_after(true, k_transparent<P, STRICT>, dim3((v.ntfsf + 127) / 128), 128, 0, s, v, side);
    if (v.nprobe > 0)
      launch_after(true, k_probes<P>, dim3((v.nprobe + 127) / 128), 128, 0, s, v, side, (int64_t)st);
  }
  if (side == 0 && p.incident != nullptr) {
    Meeting meet = p.incident->meet;
    if (!last) meet.done = nullptr;  // the call's last launch answers for all
    if (meet.at != nullptr && persist_takes(*p.incident, 1)) {
      const cudaError_t e = launch_persist(*p.incident, meet, 1, st, s);
      if (!no_room(e)) return e;
      (void)cudaGetLastError();
    }
    return run_steps<P, STRICT>(*p.incident, 1, 3, st, s);
  }
  return cudaSuccess;
}

template <class P, bool STRICT>
cudaError_t run_steps(const Plan& p, int nsteps, int side_mask, int st0, cudaStream_t s) {
  for (int st = 0; st < nsteps; ++st) {
    const bool last = st + 1 == nsteps;
    for (int side = 0; side < 2; ++side) {
      if (!((side_mask >> side) & 1)) continue;
      const bool early = side == 0 ? st > 0 : (st > 0 || (side_mask & 1)) && p.incident == nullptr;
      const cudaError_t e = run_half<P, STRICT>(p, side, st0 + st, early, last, s);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaGetLastError();
}

cudaError_t dispatch_precision(const gmes_grid_desc& g, const Plan& p, int nsteps,
                               int side_mask, int st0, cudaStream_t s) {
  switch (g.precision) {
    case GMES_FP64:
      return run_steps<PolF64, false>(p, nsteps, side_mask, st0, s);
    case GMES_FP64_STRICT:
      return run_steps<PolF64, true>(p, nsteps, side_mask, st0, s);
    case GMES_FP32:
      return run_steps<PolF32, false>(p, nsteps, side_mask, st0, s);
    case GMES_DF64:
      return run_steps<PolDF, false>(p, nsteps, side_mask, st0, s);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace

template <class P, bool STRICT>
cudaError_t run_batch(const BatchView& v, const GridDev* host_jobs, bool disp, int nsteps,
                      int blocks, cudaStream_t st) {
  using T = typename P::T;
  const int cells = blocks > 0 ? blocks : (int)(v.tiles < (1 << 30) ? v.tiles : (1 << 30));
  const int64_t per = cells > 0 ? (v.tiles + cells - 1) / cells : 0;  // tiles per block
  const int gblocks = (int)((v.ghosts + 255) / 256 < 65535 * 16 ? (v.ghosts + 255) / 256 : 65535 * 16);
  const int sblocks = (v.srcs + 127) / 128;
  const bool arg = ArgDescs<P>::value && host_jobs != nullptr && v.njobs <= kParamJobs;
  static thread_local BatchDescs descs;
  if (arg) {
    std::memset(&descs, 0, sizeof(descs));
    for (int q = 0; q < v.njobs; ++q) descs.jobs[q] = host_jobs[q];
  }
  bool early = false;  // the first launch is a plain one
  auto go = [&](auto kernel, int blocks_, int threads, auto... args) {
    if (blocks_ <= 0) return;
    launch_after(early, kernel, dim3((unsigned)blocks_), threads, 0, st, v, args...);
    early = true;
  };
  auto cell = [&](int s, auto by_arg, auto by_copy) {
    if (arg)
      go(by_arg, cells, kBatchThreads, s, per, descs);
    else
      go(by_copy, cells, kBatchThreads, s, per);
  };
  for (int s = 0; s < nsteps; ++s) {
    for (int side = 0; side < 2; ++side) {
      go(k_multi_ghost<T>, gblocks, 256, 1 - side, s);
      if (side == 1)
        cell(s, k_multi_cell_arg<P, 1, STRICT, false>, k_multi_cell<P, 1, STRICT, false>);
      else if (disp)
        cell(s, k_multi_cell_arg<P, 0, STRICT, true>, k_multi_cell<P, 0, STRICT, true>);
      else
        cell(s, k_multi_cell_arg<P, 0, STRICT, false>, k_multi_cell<P, 0, STRICT, false>);
      go(k_multi_sources<P, STRICT>, sblocks, 128, side, s);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_batch(const BatchView& v, const GridDev* host_jobs, int precision, bool disp,
                         int nsteps, int blocks, cudaStream_t s) {
  switch (precision) {
    case GMES_FP64:
      return run_batch<PolF64, false>(v, host_jobs, disp, nsteps, blocks, s);
    case GMES_FP64_STRICT:
      return run_batch<PolF64, true>(v, host_jobs, disp, nsteps, blocks, s);
    case GMES_FP32:
      return run_batch<PolF32, false>(v, host_jobs, disp, nsteps, blocks, s);
    case GMES_DF64:
      return run_batch<PolDF, false>(v, host_jobs, disp, nsteps, blocks, s);
    default:
      return cudaErrorInvalidValue;
  }
}

// Non-finite guard (gmes_nonfinite): an infinity or NaN has an all-ones
// exponent; the test is on the bits, so no floating-point pipe is used.
__device__ __forceinline__ bool nonfinite(double v) {
  return ((__double_as_longlong(v) >> 52) & 0x7ff) == 0x7ff;
}
__device__ __forceinline__ bool nonfinite(float v) {
  return ((__float_as_uint(v) >> 23) & 0xff) == 0xff;
}
__device__ __forceinline__ bool nonfinite(float2 v) { return nonfinite(v.x); }  // hi word

template <class T>
__global__ void k_nonfinite(const GridDev g, int planes, int32_t* flag) {
  bool bad = false;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int c = 0; c < 6; ++c) {
    if (!((g.active >> c) & 1)) continue;
    const T* f = static_cast<const T*>(g.f[c]);
    const int64_t n = g.npts[c] * planes;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride)
      bad = bad || nonfinite(f[t]);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *flag = 1;
}

cudaError_t launch_nonfinite(const gmes_grid_desc& g, const GridDev& d, int32_t* flag,
                             cudaStream_t s) {
  const int planes = (g.flags & GMES_FLAG_COMPLEX) ? 2 : 1;
  int64_t most = 1;
  for (int c = 0; c < 6; ++c) most = d.npts[c] * planes > most ? d.npts[c] * planes : most;
  const int blocks = (int)((most + 255) / 256 < 152 * 8 ? (most + 255) / 256 : 152 * 8);
  switch (g.precision) {
    case GMES_FP64:
    case GMES_FP64_STRICT:
      k_nonfinite<double><<<blocks, 256, 0, s>>>(d, planes, flag);
      break;
    case GMES_FP32:
      k_nonfinite<float><<<blocks, 256, 0, s>>>(d, planes, flag);
      break;
    case GMES_DF64:
      k_nonfinite<float2><<<blocks, 256, 0, s>>>(d, planes, flag);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_step(const gmes_grid_desc& g, const Plan& p, int nsteps, cudaStream_t s) {
  if (p.meet.at != nullptr && persist_takes(p, nsteps)) {
    const cudaError_t e = launch_persist(p, p.meet, nsteps, 0, s);
    if (!no_room(e)) return e;
    (void)cudaGetLastError();
  }
  return dispatch_precision(g, p, nsteps, 3, 0, s);
}

cudaError_t launch_half(const gmes_grid_desc& g, const Plan& p, int side, int step,
                        cudaStream_t s) {
  return dispatch_precision(g, p, 1, side == 0 ? 1 : 2, step, s);
}

}  // namespace gmes
