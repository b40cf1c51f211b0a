// Differentiation: gradient of a monitor objective with respect to the
// permittivity of a design region, for a batch of TMz designs that share
// geometry, PML and sources and differ only in the design pixels.
//
// The reference has no adjoint; the forward map differentiated here is its
// TMz time step (gmes/fdtd.py:1099-1122) with the Dielectric and CPML
// updaters of src/pw_dielectric.hh:281-371 (Hx, Hy), src/pw_dielectric.hh:186-199
// (Ez), src/pw_cpml.hh:211-237, 319-397 and the point sources of
// gmes/pw_source.py:74-131.
//
// Lattice.  With N = (nx, ny, 1), the TMz fields live on one periodic
// nx x ny lattice per design:
//   E(i, j) = Ez[i, j, 0],  X(i, j) = Hx[i, j+1, 1],  Y(i, j) = Hy[i+1, j, 1]
// The reference's ghost planes (Ez[nx, :], Ez[:, ny], Hx[:, 0, :], Hy[0])
// only ever hold copies of these points (talk_with_*_neighbors,
// gmes/fdtd.py:811-1097), so the kernels read the periodic image directly
// (index nx-1 for -1, 0 for nx) and never store a ghost.  Then
//   E(i,j) += c1 (Y(i,j) - Y(i-1,j)) - c2 (X(i,j) - X(i,j-1))   (or its CPML form)
//   X(i,j) -= c1x (E(i,j+1) - E(i,j))
//   Y(i,j) += c2y (E(i+1,j) - E(i,j))
//
// Adjoint.  The objective is J_b = dt * sum_{n=1..N} sum_{m in monitor} E_n(m)^2.
// Reverse-mode through one step applies, in reverse order, the transposes
// of: H sources, H update, E sources, E update.  Every update is
// F' = F + (linear in the two curl differences and the psi state), so its
// transpose keeps lambda_F, adds the "curl weight" lambda_D = dF'/dD *
// lambda_F' to the neighbours the differences read, and runs the psi
// recursion backwards:  L = phi + (dF'/dpsi') lambda_F',
// lambda_D = (dpsi'/dD) L + (dF'/dD)|direct lambda_F',  phi <- b L.
// The psi adjoints are double-buffered so a thread can evaluate its
// neighbours' curl weights from the previous buffer while the owner writes
// the next one: one kernel per half, gather form, no atomics.
// The design enters only through c1, c2 of the design pixels:
//   dJ/deps_p = sum_n lambda_E'(p) * dE'/deps_p = -1/eps_p sum_n lambda_E'(p) inc_p(n)
// with inc_p(n) = c1 D1 - c2 D2 of forward step n, recorded when the step
// is recomputed from a checkpoint.
//
// Resolved map.  Every lattice point's update is resolved once per design
// set (k_tmz_map): most points (dielectric, design pixels, CPML outside
// both profiles) update as F + c1 D1 + c2 D2 with two coefficients that
// the kernels read from a small per-point map shared by the batch (L2
// resident) instead of following class map -> class table -> profile
// look-ups every step; CPML points inside a profile go through the
// per-point functions below.
//
// Three kernel forms.  The one-step kernels advance every lattice point by one
// half-step per launch; up to some millions of points the steps of a call are
// one cooperative launch of the same bodies (k_tmz_chunk_fwd, k_tmz_chunk_adj).
// The temporally blocked kernels (FP32) advance a tile of one design by up to
// kTbHalo steps per launch from a region in registers (see k_tmz_tb_fwd), or in
// shared memory for tiles of mixed points.  All use the same map and arithmetic
// functions, and this file is compiled without implicit multiply-add
// contraction (every fused operation is an explicit fmadd), so the
// forms give bit-identical fields, adjoints and gradients.
#include "gmes_barrier.cuh"

namespace gmes {
namespace {

constexpr int kBX = 32, kBY = 8;

// a + b * c: one rounding in FP32 and FP64, the float-float operators for
// the df type.
template <class R>
__device__ __forceinline__ R fmadd(R a, R b, R c) {
  return a + b * c;
}
template <>
__device__ __forceinline__ float fmadd<float>(float a, float b, float c) {
  return __fmaf_rn(b, c, a);
}
template <>
__device__ __forceinline__ double fmadd<double>(double a, double b, double c) {
  return __fma_rn(b, c, a);
}

struct Lat {
  int i, j, b;
  int64_t base, lin;
};

__device__ __forceinline__ bool lattice_point(const TmzDev& t, Lat& p) {
  p.j = blockIdx.x * kBX + threadIdx.x;
  p.i = blockIdx.y * kBY + threadIdx.y;
  p.b = blockIdx.z;
  if (p.i >= t.nx || p.j >= t.ny) return false;
  p.base = (int64_t)p.b * t.plane;
  p.lin = (int64_t)p.i * t.ny + p.j;
  return true;
}

// Point `at` of all designs' lattices (persistent kernels).
struct LatDiv {
  uint32_t m_plane, m_row;
  int s_plane, s_row;
};
__device__ __forceinline__ Lat lattice_at(const TmzDev& t, const LatDiv& d, unsigned at) {
  Lat p;
  p.b = (int)tile_quot(at, d.m_plane, d.s_plane);
  const unsigned r = at - (unsigned)p.b * (unsigned)t.plane;
  p.i = (int)tile_quot(r, d.m_row, d.s_row);
  p.j = (int)(r - (unsigned)p.i * (unsigned)t.ny);
  p.base = (int64_t)p.b * t.plane;
  p.lin = r;
  return p;
}

__device__ __forceinline__ int64_t design_index(const TmzDev& t, int i, int j) {
  const int di = i - t.d0[0], dj = j - t.d0[1];
  if (di < 0 || di >= t.dn[0] || dj < 0 || dj >= t.dn[1]) return -1;
  return (int64_t)di * t.dn[1] + dj;
}

__device__ __forceinline__ int64_t monitor_index(const TmzDev& t, int i, int j) {
  const int di = i - t.m0[0], dj = j - t.m0[1];
  if (di < 0 || di >= t.mn[0] || dj < 0 || dj >= t.mn[1]) return -1;
  return (int64_t)di * t.mn[1] + dj;
}

// Class entries of the three lattice components (template grid maps).
__device__ __forceinline__ const ClassCoef& class_e(const GridDev& g, int i, int j) {
  return g.tab[2][__ldg(g.cls[2] + (int64_t)i * g.st[2][0] + (int64_t)j * g.st[2][1])];
}
__device__ __forceinline__ const ClassCoef& class_x(const GridDev& g, int i, int j) {
  return g.tab[3][__ldg(g.cls[3] + (int64_t)i * g.st[3][0] + (int64_t)(j + 1) * g.st[3][1] + 1)];
}
__device__ __forceinline__ const ClassCoef& class_y(const GridDev& g, int i, int j) {
  return g.tab[4][__ldg(g.cls[4] + (int64_t)(i + 1) * g.st[4][0] + (int64_t)j * g.st[4][1] + 1)];
}

// CPML profile rows of one lattice point: q1 along the component's first
// curl axis, q2 along its second (Ez: x, y; Hx: y, z; Hy: z, x).
struct Prof {
  const Coef* q1;
  const Coef* q2;
};
__device__ __forceinline__ Prof prof_e(const GridDev& g, int pm, int i, int j) {
  return {g.prof[pm][2][0] + (int64_t)i * kProfStride, g.prof[pm][2][1] + (int64_t)j * kProfStride};
}
__device__ __forceinline__ Prof prof_x(const GridDev& g, int pm, int i, int j) {
  (void)i;
  return {g.prof[pm][3][1] + (int64_t)(j + 1) * kProfStride, g.prof[pm][3][2] + kProfStride};
}
__device__ __forceinline__ Prof prof_y(const GridDev& g, int pm, int i, int j) {
  (void)j;
  return {g.prof[pm][4][2] + kProfStride, g.prof[pm][4][0] + (int64_t)(i + 1) * kProfStride};
}

// ---------------------------------------------------------------------------
// CPML points inside a profile.
// ---------------------------------------------------------------------------
// Their updates are those of the reference's CPML updaters
// (src/pw_cpml.hh:211-237, 319-397) with psi:
//   Ez: psi1' = b1 psi1 + c1 D1 (where profile 1 is on), likewise psi2;
//       Ez' = Ez + cdt ((psi1' - psi2') + k1 D1 - k2 D2)
//   Hx: psi' = b psi + c D1 (on);  Hx' = Hx - cdt (psi' + k D1)
//   Hy: psi' = b psi + c D2 (on);  Hy' = Hy - cdt (-psi' - k D2)
// with b, c, k the profile row (entries 0, 3, 4) at the point's index along
// the profile's axis.  The map (k_tmz_map) holds the class's cdt in the
// point's coefficient slot, the profile set in the flags' pml fields and
// which profiles are on, so no class look-up is needed here.
template <class P>
__device__ __forceinline__ typename P::R e_cpml(const GridDev& g, unsigned fl, typename P::R cdt,
                                                int i, int j, typename P::R e, typename P::R D1,
                                                typename P::R D2, typename P::T* s1,
                                                typename P::T* s2) {
  using R = typename P::R;
  const int pm = (fl >> kTmzPmlE) & 3;
  const Coef* q1 = g.prof[pm][2][0] + (int64_t)i * kProfStride;
  const Coef* q2 = g.prof[pm][2][1] + (int64_t)j * kProfStride;
  R psi1 = P::ldw(s1), psi2 = P::ldw(s2);
  if (fl & kTmzOnE1) {
    psi1 = fmadd(P::cfg(q1) * psi1, P::cfg(q1 + 3), D1);
    P::st(s1, psi1);
  }
  if (fl & kTmzOnE2) {
    psi2 = fmadd(P::cfg(q2) * psi2, P::cfg(q2 + 3), D2);
    P::st(s2, psi2);
  }
  const R xv = fmadd(fmadd(psi1 - psi2, P::cfg(q1 + 4), D1), -P::cfg(q2 + 4), D2);
  return fmadd(e, cdt, xv);
}

template <class P>
__device__ __forceinline__ typename P::R x_cpml(const GridDev& g, unsigned fl, typename P::R cdt,
                                                int j, typename P::R x, typename P::R dx,
                                                typename P::T* s) {
  using R = typename P::R;
  const Coef* q = g.prof[(fl >> kTmzPmlX) & 3][3][1] + (int64_t)(j + 1) * kProfStride;
  R psi = P::ldw(s);
  if (fl & kTmzOnX) {
    psi = fmadd(P::cfg(q) * psi, P::cfg(q + 3), dx);
    P::st(s, psi);
  }
  return fmadd(x, -cdt, fmadd(psi, P::cfg(q + 4), dx));
}

template <class P>
__device__ __forceinline__ typename P::R y_cpml(const GridDev& g, unsigned fl, typename P::R cdt,
                                                int i, typename P::R y, typename P::R dy,
                                                typename P::T* s) {
  using R = typename P::R;
  const Coef* q = g.prof[(fl >> kTmzPmlY) & 3][4][0] + (int64_t)(i + 1) * kProfStride;
  R psi = P::ldw(s);
  if (fl & kTmzOnY) {
    psi = fmadd(P::cfg(q) * psi, P::cfg(q + 3), dy);
    P::st(s, psi);
  }
  return fmadd(y, -cdt, fmadd(-psi, -P::cfg(q + 4), dy));
}

// Their transposes.  Curl weight of an Hx point: lambda_D1 = dX'/dD1
// applied to its adjoint lx; phr: its psi adjoint before this step, OWN:
// the advanced one is written to *phw.
template <class P, bool OWN>
__device__ __forceinline__ typename P::R adjx_cpml(const GridDev& g, unsigned fl,
                                                   typename P::R cdt, int j, typename P::R lx,
                                                   const typename P::T* phr,
                                                   typename P::T* phw) {
  using R = typename P::R;
  const Coef* q = g.prof[(fl >> kTmzPmlX) & 3][3][1] + (int64_t)(j + 1) * kProfStride;
  const R direct = -(cdt * (P::cfg(q + 4) * lx));
  if (!(fl & kTmzOnX)) return direct;
  const R L = fmadd(P::ldw(phr), -cdt, lx);
  if (OWN) P::st(phw, P::cfg(q) * L);
  return fmadd(direct, P::cfg(q + 3), L);
}

// Curl weight of an Hy point: lambda_D2, D2 = E(i+1, j) - E(i, j).
template <class P, bool OWN>
__device__ __forceinline__ typename P::R adjy_cpml(const GridDev& g, unsigned fl,
                                                   typename P::R cdt, int i, typename P::R ly,
                                                   const typename P::T* phr,
                                                   typename P::T* phw) {
  using R = typename P::R;
  const Coef* q = g.prof[(fl >> kTmzPmlY) & 3][4][0] + (int64_t)(i + 1) * kProfStride;
  const R direct = cdt * (P::cfg(q + 4) * ly);
  if (!(fl & kTmzOnY)) return direct;
  const R L = fmadd(P::ldw(phr), cdt, ly);
  if (OWN) P::st(phw, P::cfg(q) * L);
  return fmadd(direct, P::cfg(q + 3), L);
}

// Curl weights (lambda_D1, lambda_D2) of an Ez point from its adjoint le;
// NEED1/NEED2: which weights the caller uses (both when OWN).
template <class P, bool OWN, bool NEED1, bool NEED2>
__device__ __forceinline__ void adje_cpml(const GridDev& g, unsigned fl, typename P::R cdt, int i,
                                          int j, typename P::R le, const typename P::T* phr0,
                                          typename P::T* phw0, const typename P::T* phr1,
                                          typename P::T* phw1, typename P::R& w1,
                                          typename P::R& w2) {
  using R = typename P::R;
  const int pm = (fl >> kTmzPmlE) & 3;
  w1 = P::zero();
  w2 = P::zero();
  if (NEED1 || OWN) {
    const Coef* q1 = g.prof[pm][2][0] + (int64_t)i * kProfStride;
    const R direct = cdt * (P::cfg(q1 + 4) * le);
    if (fl & kTmzOnE1) {
      const R L = fmadd(P::ldw(phr0), cdt, le);
      if (OWN) P::st(phw0, P::cfg(q1) * L);
      w1 = fmadd(direct, P::cfg(q1 + 3), L);
    } else {
      w1 = direct;
    }
  }
  if (NEED2 || OWN) {
    const Coef* q2 = g.prof[pm][2][1] + (int64_t)j * kProfStride;
    const R direct = -(cdt * (P::cfg(q2 + 4) * le));
    if (fl & kTmzOnE2) {
      const R L = fmadd(P::ldw(phr1), -cdt, le);
      if (OWN) P::st(phw1, P::cfg(q2) * L);
      w2 = fmadd(direct, P::cfg(q2 + 3), L);
    } else {
      w2 = direct;
    }
  }
}

// dJ/dE_n of a monitor value e of a design of weight w.
__device__ __forceinline__ double seed_value(const GridDev& g, double w, double e) {
  return 2.0 * g.dt * w * e;
}

// Objective seed of lattice point (i, j) of design b at reverse step n:
// dJ/dE_n = 2 dt w_b E_n on monitor points (*has), nothing elsewhere.
__device__ __forceinline__ double seed_of(const GridDev& g, const TmzDev& t, int b, int i, int j,
                                          int n, bool* has) {
  const int64_t m = monitor_index(t, i, j);
  *has = m >= 0;
  if (m < 0) return 0.0;
  const int64_t nm = (int64_t)t.mn[0] * t.mn[1];
  const double w = t.weight != nullptr ? t.weight[b] : 1.0;
  const double e = t.mon[((int64_t)b * t.total_steps + (n - 1)) * nm + m];
  return seed_value(g, w, e);
}

// ---------------------------------------------------------------------------
// The resolved lattice map.
// ---------------------------------------------------------------------------
// Whether a CPML point's profile is on along either curl axis.
__device__ __forceinline__ bool profile_on(const Prof& q) {
  return coef_nonzero(q.q1 + 1) || coef_nonzero(q.q2 + 1);
}

template <class P>
__device__ __forceinline__ const typename P::T* map_coef(const TmzDev& t, int k) {
  return static_cast<const typename P::T*>(t.pcoef[k]);
}

// Flags and plain-form coefficients of every lattice point, built once per
// design set from the class maps, class table and CPML profiles.  The
// coefficients are c1, c2 of a Dielectric class, or of a CPML class outside
// both profiles (whose update reduces to the dielectric form).  Design
// pixels take theirs from the per-design table.  CPML points inside a
// profile keep their class's cdt in the coefficient slot, and the flags
// name the profile set and which of the point's profiles are on.
template <class P>
__global__ void k_tmz_map(const GridDev g, const TmzDev t) {
  using R = typename P::R;
  using T = typename P::T;
  const int64_t ll = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ll >= t.plane) return;
  const int i = (int)(ll / t.ny), j = (int)(ll - (int64_t)i * t.ny);
  unsigned f = 0;
  R c1 = P::zero(), c2n = P::zero(), cxn = P::zero(), cy = P::zero();
  if (design_index(t, i, j) >= 0) {
    f |= kTmzPlainE | kTmzDesign;
  } else {
    const ClassCoef& cc = class_e(g, i, j);
    const int kind = __ldg(&cc.kind);
    const int pm = __ldg(&cc.pml);
    if (kind == GMES_KIND_CPML && profile_on(prof_e(g, pm, i, j))) {
      const Prof q = prof_e(g, pm, i, j);
      f |= kTmzPsiE | ((unsigned)pm << kTmzPmlE);
      if (coef_nonzero(q.q1 + 1)) f |= kTmzOnE1;
      if (coef_nonzero(q.q2 + 1)) f |= kTmzOnE2;
      c1 = P::cfg(&cc.cdt);
    } else if (kind == GMES_KIND_DIELECTRIC || kind == GMES_KIND_CPML) {
      f |= kTmzPlainE;
      c1 = P::cfg(&cc.c1);
      c2n = -P::cfg(&cc.c2);
    }
  }
  {
    const ClassCoef& cc = class_x(g, i, j);
    const int kind = __ldg(&cc.kind);
    const int pm = __ldg(&cc.pml);
    if (kind == GMES_KIND_CPML && profile_on(prof_x(g, pm, i, j))) {
      f |= kTmzPsiX | ((unsigned)pm << kTmzPmlX);
      if (coef_nonzero(prof_x(g, pm, i, j).q1 + 1)) f |= kTmzOnX;
      cxn = P::cfg(&cc.cdt);
    } else if (kind == GMES_KIND_DIELECTRIC || kind == GMES_KIND_CPML) {
      f |= kTmzPlainX;
      cxn = -P::cfg(&cc.c1);
    }
  }
  {
    const ClassCoef& cc = class_y(g, i, j);
    const int kind = __ldg(&cc.kind);
    const int pm = __ldg(&cc.pml);
    if (kind == GMES_KIND_CPML && profile_on(prof_y(g, pm, i, j))) {
      f |= kTmzPsiY | ((unsigned)pm << kTmzPmlY);
      if (coef_nonzero(prof_y(g, pm, i, j).q2 + 1)) f |= kTmzOnY;
      cy = P::cfg(&cc.cdt);
    } else if (kind == GMES_KIND_DIELECTRIC || kind == GMES_KIND_CPML) {
      f |= kTmzPlainY;
      cy = P::cfg(&cc.c2);
    }
  }
  if (monitor_index(t, i, j) >= 0) f |= kTmzMonitor;
  const_cast<uint32_t*>(t.pflags)[ll] = f;
  P::st(const_cast<T*>(map_coef<P>(t, 0)) + ll, c1);
  P::st(const_cast<T*>(map_coef<P>(t, 1)) + ll, c2n);
  P::st(const_cast<T*>(map_coef<P>(t, 2)) + ll, cxn);
  P::st(const_cast<T*>(map_coef<P>(t, 3)) + ll, cy);
}

// Marks the points that carry a point source of either half, with a place in
// the list to look for it from (after k_tmz_map, which clears both).
__global__ void k_tmz_map_sources(const TmzDev t) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= t.nsrc) return;
  const gmes_point_source s = t.src[k];
  if (s.comp < 2 || s.comp > 4 || s.offset < 0 || s.offset >= t.plane) return;
  uint32_t* p = const_cast<uint32_t*>(t.pflags) + s.offset;
  const uint32_t place = (uint32_t)(k + 1 < kTmzPlaces ? k + 1 : kTmzPlaces) << kTmzPlace;
  constexpr uint32_t low = (1u << kTmzPlace) - 1;
  uint32_t was = *p, seen;
  do {
    seen = was;
    const uint32_t high = (seen & ~low) > place ? seen & ~low : place;
    was = atomicCAS(p, seen, (seen & low) | high | (s.comp == 2 ? kTmzSrcE : kTmzSrcH));
  } while (was != seen);
}

// The point source of lattice point ll in the array of Ez, Hx or Hy (k = 0, 1,
// 2), -1: none; fl: the point's flags.  The last of several in the list.
__device__ __forceinline__ int source_at(const TmzDev& t, unsigned fl, int k, int64_t ll) {
  const int place = (int)(fl >> kTmzPlace) & kTmzPlaces;
  int q = (place < kTmzPlaces && place < t.nsrc ? place : t.nsrc) - 1;
  while (q >= 0 && (t.src[q].offset != ll || t.src[q].comp != k + 2)) --q;
  return q;
}

// Point sources (gmes/pw_source.py:74-131) of that point: a field value after
// the source of step n, and whether a hard source sits there (the value it
// writes does not depend on the field before it, so its adjoint is zero;
// current sources leave it as it is).
template <class P>
__device__ __forceinline__ typename P::R with_source(const TmzDev& t, unsigned fl, int k,
                                                     int64_t ll, int n, typename P::R f) {
  const int q = source_at(t, fl, k, ll);
  if (q < 0) return f;
  const typename P::R v = P::from_double(
      __ldg(t.src_val + ((int64_t)(n - 1) * 2 + (k == 0 ? 0 : 1)) * t.nsrc + q));
  return t.src[q].mode == 0 ? v : f - v;
}
__device__ __forceinline__ bool hard_source(const TmzDev& t, unsigned fl, int k, int64_t ll) {
  if (!(fl & (k == 0 ? kTmzSrcE : kTmzSrcH))) return false;
  const int q = source_at(t, fl, k, ll);
  return q >= 0 && t.src[q].mode == 0;
}

// Plain-form Ez coefficients (c1, -c2) of lattice point (i, j) = ll of
// design b.
template <class P>
__device__ __forceinline__ void e_coef(const TmzDev& t, int b, int i, int j, int64_t ll,
                                       unsigned fl, typename P::R& c1, typename P::R& c2n) {
  c1 = P::ldc(map_coef<P>(t, 0) + ll);
  c2n = P::ldc(map_coef<P>(t, 1) + ll);
  if (fl & kTmzDesign) {
    const DesignCoef* dc = t.dc + (int64_t)b * t.dn[0] * t.dn[1] + design_index(t, i, j);
    c1 = P::cfg(&dc->c1);
    c2n = -P::cfg(&dc->c2);
  }
}

// Adjoint curl weights through the map: the plain form, the CPML form on
// points inside a profile, zero on points that are not updated.  ll:
// lattice offset; base: the design's offset.
template <class P, bool OWN>
__device__ __forceinline__ typename P::R weight_x(const GridDev& g, const TmzDev& t, int i, int j,
                                                  int64_t ll, int64_t base, int rb, int wb) {
  using T = typename P::T;
  const T* lx = static_cast<const T*>(t.l[1]) + base + ll;
  const typename P::R c = P::ldc(map_coef<P>(t, 2) + ll);  // issued with the flags
  const unsigned fl = __ldg(t.pflags + ll);
  const typename P::R l = hard_source(t, fl, 1, ll) ? P::zero() : P::ldw(lx);
  if (fl & kTmzPlainX) return c * l;
  if (!(fl & kTmzPsiX)) return P::zero();
  return adjx_cpml<P, OWN>(g, fl, c, j, l,
                           static_cast<const T*>(t.phi[rb][2]) + base + ll,
                           OWN ? static_cast<T*>(t.phi[wb][2]) + base + ll : nullptr);
}

template <class P, bool OWN>
__device__ __forceinline__ typename P::R weight_y(const GridDev& g, const TmzDev& t, int i, int j,
                                                  int64_t ll, int64_t base, int rb, int wb) {
  using T = typename P::T;
  const T* ly = static_cast<const T*>(t.l[2]) + base + ll;
  const typename P::R c = P::ldc(map_coef<P>(t, 3) + ll);  // issued with the flags
  const unsigned fl = __ldg(t.pflags + ll);
  const typename P::R l = hard_source(t, fl, 2, ll) ? P::zero() : P::ldw(ly);
  if (fl & kTmzPlainY) return c * l;
  if (!(fl & kTmzPsiY)) return P::zero();
  return adjy_cpml<P, OWN>(g, fl, c, i, l,
                           static_cast<const T*>(t.phi[rb][3]) + base + ll,
                           OWN ? static_cast<T*>(t.phi[wb][3]) + base + ll : nullptr);
}

template <class P, bool OWN, bool NEED1, bool NEED2>
__device__ __forceinline__ void weight_e(const GridDev& g, const TmzDev& t, int b, int i, int j,
                                         int64_t ll, int64_t base, int rb, int wb,
                                         typename P::R& w1, typename P::R& w2) {
  using R = typename P::R;
  using T = typename P::T;
  const T* le = static_cast<const T*>(t.l[0]) + base + ll;
  const unsigned fl = __ldg(t.pflags + ll);
  R c1, c2n;
  e_coef<P>(t, b, i, j, ll, fl, c1, c2n);
  if (fl & kTmzPlainE) {
    const R v = P::ldw(le);
    w1 = c1 * v;
    w2 = c2n * v;
    return;
  }
  if (!(fl & kTmzPsiE)) {
    w1 = w2 = P::zero();
    return;
  }
  adje_cpml<P, OWN, NEED1, NEED2>(g, fl, c1, i, j, P::ldw(le),
                                  static_cast<const T*>(t.phi[rb][0]) + base + ll,
                                  OWN ? static_cast<T*>(t.phi[wb][0]) + base + ll : nullptr,
                                  static_cast<const T*>(t.phi[rb][1]) + base + ll,
                                  OWN ? static_cast<T*>(t.phi[wb][1]) + base + ll : nullptr, w1,
                                  w2);
}

// ---------------------------------------------------------------------------
// One step of one lattice point, forward (step n; slot: where its design
// increment is recorded, row: its monitor row, -1 not).
// ---------------------------------------------------------------------------
template <class P>
__device__ __forceinline__ void point_fe(const GridDev& g, const TmzDev& t, const Lat& p, int n,
                                         int slot) {
  using R = typename P::R;
  using T = typename P::T;
  const int im = p.i == 0 ? t.nx - 1 : p.i - 1, jm = p.j == 0 ? t.ny - 1 : p.j - 1;
  T* E = static_cast<T*>(t.f[0]) + p.base;
  const T* X = static_cast<const T*>(t.f[1]) + p.base;
  const T* Y = static_cast<const T*>(t.f[2]) + p.base;
  const unsigned fl = __ldg(t.pflags + p.lin);
  const R D1 = P::ldw(Y + p.lin) - P::ldw(Y + (int64_t)im * t.ny + p.j);
  const R D2 = P::ldw(X + p.lin) - P::ldw(X + (int64_t)p.i * t.ny + jm);
  const R e = P::ldw(E + p.lin);
  R r = e;
  if (fl & kTmzPlainE) {
    R c1, c2n;
    e_coef<P>(t, p.b, p.i, p.j, p.lin, fl, c1, c2n);
    r = fmadd(fmadd(e, c1, D1), c2n, D2);
    if ((fl & kTmzDesign) && slot >= 0) {
      const int64_t nd = (int64_t)t.dn[0] * t.dn[1];
      P::st(static_cast<T*>(t.hist) + ((int64_t)slot * t.nb + p.b) * nd +
                design_index(t, p.i, p.j),
            fmadd(c2n * D2, c1, D1));
    }
  } else if (fl & kTmzPsiE) {
    r = e_cpml<P>(g, fl, P::ldc(map_coef<P>(t, 0) + p.lin), p.i, p.j, e, D1, D2,
                  static_cast<T*>(t.f[3]) + p.base + p.lin,
                  static_cast<T*>(t.f[4]) + p.base + p.lin);
  }
  if (fl & kTmzSrcE) r = with_source<P>(t, fl, 0, p.lin, n, r);
  P::st(E + p.lin, r);
}

template <class P>
__device__ __forceinline__ void point_fh(const GridDev& g, const TmzDev& t, const Lat& p, int n,
                                         int row) {
  using R = typename P::R;
  using T = typename P::T;
  const int ip = p.i + 1 == t.nx ? 0 : p.i + 1, jp = p.j + 1 == t.ny ? 0 : p.j + 1;
  const T* E = static_cast<const T*>(t.f[0]) + p.base;
  T* X = static_cast<T*>(t.f[1]) + p.base;
  T* Y = static_cast<T*>(t.f[2]) + p.base;
  const unsigned fl = __ldg(t.pflags + p.lin);
  const R cxn = P::ldc(map_coef<P>(t, 2) + p.lin), cy = P::ldc(map_coef<P>(t, 3) + p.lin);
  const R e0 = P::ldw(E + p.lin);
  const R dx = P::ldw(E + (int64_t)p.i * t.ny + jp) - e0;  // D1 of Hx
  const R dy = P::ldw(E + (int64_t)ip * t.ny + p.j) - e0;  // D2 of Hy
  const R x0 = P::ldw(X + p.lin), y0 = P::ldw(Y + p.lin);
  R x = x0, y = y0;
  if (fl & kTmzPlainX)
    x = fmadd(x0, cxn, dx);
  else if (fl & kTmzPsiX)
    x = x_cpml<P>(g, fl, cxn, p.j, x0, dx, static_cast<T*>(t.f[5]) + p.base + p.lin);
  if (fl & kTmzPlainY)
    y = fmadd(y0, cy, dy);
  else if (fl & kTmzPsiY)
    y = y_cpml<P>(g, fl, cy, p.i, y0, dy, static_cast<T*>(t.f[6]) + p.base + p.lin);
  if (fl & kTmzSrcH) {
    x = with_source<P>(t, fl, 1, p.lin, n, x);
    y = with_source<P>(t, fl, 2, p.lin, n, y);
  }
  P::st(X + p.lin, x);
  P::st(Y + p.lin, y);
  if (row >= 0 && (fl & kTmzMonitor)) {
    const int64_t nm = (int64_t)t.mn[0] * t.mn[1];
    t.mon[((int64_t)p.b * t.total_steps + row) * nm + monitor_index(t, p.i, p.j)] = to_double(e0);
  }
}

// ---------------------------------------------------------------------------
// One step of one lattice point, adjoint.
// ---------------------------------------------------------------------------
// Transpose of the H half of step n, plus the objective's seed for the
// state after step n: lambda_E gathers the curl weights of its four H
// neighbours; the owner advances the Hx/Hy psi adjoints.
template <class P>
__device__ __forceinline__ void point_ah(const GridDev& g, const TmzDev& t, const Lat& p, int n,
                                         int rb, int wb) {
  using R = typename P::R;
  using T = typename P::T;
  const int im = p.i == 0 ? t.nx - 1 : p.i - 1, jm = p.j == 0 ? t.ny - 1 : p.j - 1;
  T* LE = static_cast<T*>(t.l[0]) + p.base + p.lin;
  R le = P::ldw(LE);
  const unsigned fl = __ldg(t.pflags + p.lin);
  if (fl & kTmzMonitor) {
    bool has;
    le = le + P::from_double(seed_of(g, t, p.b, p.i, p.j, n, &has));
  }
  const int64_t ljm = (int64_t)p.i * t.ny + jm, lim = (int64_t)im * t.ny + p.j;
  const R a = weight_x<P, false>(g, t, p.i, jm, ljm, p.base, rb, wb);
  const R bx = weight_x<P, true>(g, t, p.i, p.j, p.lin, p.base, rb, wb);
  const R c = weight_y<P, false>(g, t, im, p.j, lim, p.base, rb, wb);
  const R d = weight_y<P, true>(g, t, p.i, p.j, p.lin, p.base, rb, wb);
  le = le + ((a - bx) + (c - d));
  P::st(LE, hard_source(t, fl, 0, p.lin) ? P::zero() : le);
}

// Transpose of the E half of step n: lambda_X, lambda_Y gather the curl
// weights of their two Ez neighbours; the owner advances the Ez psi
// adjoints and, in the design region, accumulates the gradient.
template <class P>
__device__ __forceinline__ void point_ae(const GridDev& g, const TmzDev& t, const Lat& p,
                                         int slot, int rb, int wb) {
  using R = typename P::R;
  using T = typename P::T;
  const int ip = p.i + 1 == t.nx ? 0 : p.i + 1, jp = p.j + 1 == t.ny ? 0 : p.j + 1;
  const int64_t ljp = (int64_t)p.i * t.ny + jp, lip = (int64_t)ip * t.ny + p.j;
  R w1, w2, u1, u2, v1, v2;
  weight_e<P, true, true, true>(g, t, p.b, p.i, p.j, p.lin, p.base, rb, wb, w1, w2);
  weight_e<P, false, false, true>(g, t, p.b, p.i, jp, ljp, p.base, rb, wb, u1, u2);
  weight_e<P, false, true, false>(g, t, p.b, ip, p.j, lip, p.base, rb, wb, v1, v2);
  T* LX = static_cast<T*>(t.l[1]) + p.base + p.lin;
  T* LY = static_cast<T*>(t.l[2]) + p.base + p.lin;
  const unsigned fl = __ldg(t.pflags + p.lin);
  const R lx = hard_source(t, fl, 1, p.lin) ? P::zero() : P::ldw(LX);
  const R ly = hard_source(t, fl, 2, p.lin) ? P::zero() : P::ldw(LY);
  P::st(LX, lx + (w2 - u2));
  P::st(LY, ly + (w1 - v1));
  if (fl & kTmzDesign) {
    const int64_t nd = (int64_t)t.dn[0] * t.dn[1];
    const int64_t dp = design_index(t, p.i, p.j);
    const int64_t k = (int64_t)p.b * nd + dp;
    const double le = to_double(P::ldw(static_cast<const T*>(t.l[0]) + p.base + p.lin));
    const double inc =
        to_double(P::ldw(static_cast<const T*>(t.hist) + ((int64_t)slot * t.nb + p.b) * nd + dp));
    t.grad[k] += le * inc * t.dc[k].neg_reps;
  }
}

// ---------------------------------------------------------------------------
// One-step kernels: a half-step of every lattice point per launch, or a whole
// call's steps in one cooperative launch with a grid-wide barrier after each
// half (gmes_barrier.cuh).  The point's sources act in the body (with_source,
// hard_source), so a step is two launches, not four: FP64 300x243 x 6 designs,
// 200 steps with checkpoints, forward / backward 5.95 / 14.2 ms -> 4.39 / 11.4.
// What is left at that size is the launches themselves, 7-11 us per half-step
// of 0.44 M points; one cooperative launch of 512-thread blocks, two to an SM
// (62 registers), pays a 1.4 us barrier instead: 3.33 / 8.65 ms.  tmz_chunked
// says up to what size.
// ---------------------------------------------------------------------------
template <class P>
__global__ void __launch_bounds__(kBX* kBY)
    k_tmz_fe(const GridDev g, const TmzDev t, int n, int slot) {
  after_launch();
  Lat p;
  if (lattice_point(t, p)) point_fe<P>(g, t, p, n, slot);
}
template <class P>
__global__ void __launch_bounds__(kBX* kBY)
    k_tmz_fh(const GridDev g, const TmzDev t, int n, int row) {
  after_launch();
  Lat p;
  if (lattice_point(t, p)) point_fh<P>(g, t, p, n, row);
}
template <class P>
__global__ void __launch_bounds__(kBX* kBY)
    k_tmz_ah(const GridDev g, const TmzDev t, int n, int rb, int wb) {
  after_launch();
  Lat p;
  if (lattice_point(t, p)) point_ah<P>(g, t, p, n, rb, wb);
}
template <class P>
__global__ void __launch_bounds__(kBX* kBY)
    k_tmz_ae(const GridDev g, const TmzDev t, int slot, int rb, int wb) {
  after_launch();
  Lat p;
  if (lattice_point(t, p)) point_ae<P>(g, t, p, slot, rb, wb);
}

// Lattice points of all designs up to which a call's steps run as one
// cooperative launch.  Measured on GB300, 60 steps forward / adjoint ms, two
// launches per step -> one launch (with the sources in kernels of their own,
// four launches per step, in brackets):
//   FP64  128x123 x 1    (1.28 / 1.24)   0.74 / 0.75  -> 0.53 / 0.51
//         256x251 x 4    (1.82 / 2.19)   1.33 / 1.74  -> 0.87 / 1.21
//         400x395 x 24   (6.39 / 12.0)   5.80 / 11.6  -> 5.47 / 10.5
//         512x507 x 64   (20.3 / 40.8)   19.4 / 40.5  -> 23.2 / 46.8
//   df64  128x123 x 8    (1.39 / 1.27)   0.96 / 0.86  -> 0.63 / 0.60
//         256x251 x 16   (2.20 / 2.61)   1.70 / 2.12  -> 1.53 / 2.25
//         512x507 x 64   (19.7 / 29.6)   16.8 / 27.9  -> 22.0 / 43.3
// A small lattice's half-step is bound by its launch; a large one by the FP64
// pipe or L2, for which the one-launch kernel has fewer warps (62 registers).
constexpr int64_t kChunkPoints = 1 << 22, kChunkPointsDf = 1 << 20;

constexpr int kChunkThreads = 512;

// A long list of point sources, walked entry by entry (per design): the kernels
// that take it have t.nsrc = 0, so that their bodies look nothing up.
struct SourceList {
  const gmes_point_source* src;
  const double* src_val;
  int n;
};
// An entry of the list at point `at` of all designs' lattices.
struct ListSource {
  int comp, mode;  // comp -1: names no lattice point
  int64_t at;
};
__device__ __forceinline__ ListSource list_source(const TmzDev& t, const SourceList& l, int b,
                                                  int k) {
  const gmes_point_source s = l.src[k];
  const bool on = s.comp >= 2 && s.comp <= 4 && s.offset >= 0 && s.offset < t.plane;
  return {on ? s.comp : -1, s.mode, (int64_t)b * t.plane + s.offset};
}
// Its action (entry k) in half `side` of step n of the forward, and in the
// adjoint, where a hard source zeroes the adjoint of the value it overwrites.
template <class P>
__device__ __forceinline__ void source_fwd(const TmzDev& t, const SourceList& l, int side, int n,
                                           const ListSource& s, int k) {
  if (s.comp < 0 || (s.comp == 2) != (side == 0)) return;
  typename P::T* f = static_cast<typename P::T*>(t.f[s.comp - 2]) + s.at;
  const typename P::R was = P::ldw(f);  // issued with the value
  const typename P::R v =
      P::from_double(__ldg(l.src_val + ((int64_t)(n - 1) * 2 + side) * l.n + k));
  P::st(f, s.mode == 0 ? v : was - v);
}
template <class P>
__device__ __forceinline__ void source_adj(const TmzDev& t, int side, const ListSource& s) {
  if (s.comp < 0 || s.mode != 0 || (s.comp == 2) != (side == 0)) return;
  P::st(static_cast<typename P::T*>(t.l[s.comp - 2]) + s.at, P::zero());
}
template <class P>
__global__ void k_tmz_src(const TmzDev t, const SourceList l, int side, int n) {
  after_launch();
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)l.n * t.nb) return;
  const int b = (int)(q / l.n), k = (int)(q - (int64_t)b * l.n);
  source_fwd<P>(t, l, side, n, list_source(t, l, b, k), k);
}
template <class P>
__global__ void k_tmz_adj_src(const TmzDev t, const SourceList l, int side) {
  after_launch();
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)l.n * t.nb) return;
  const int b = (int)(q / l.n), k = (int)(q - (int64_t)b * l.n);
  source_adj<P>(t, side, list_source(t, l, b, k));
}

// The entries of a list that sit on this block's points (for_points), one-launch
// kernels: found once per launch (the adjoint's: hard ones alone); a block with
// more of them than fit walks the whole list.
constexpr int kOwnSources = 1024;
struct OwnSources {
  int count;
  unsigned at[kOwnSources];  // point | (comp - 2) << 24 | hard << 26
  int entry[kOwnSources];
};
static_assert(kChunkPoints <= 1 << 24, "a point's place in 24 bits");
// f(entry, number) for this block's share of the list.
template <bool HARD, class F>
__device__ __forceinline__ void walk_list(const TmzDev& t, const SourceList& l, F f) {
  const unsigned all = (unsigned)l.n * (unsigned)t.nb;
  for (unsigned q = threadIdx.x; q < all; q += kChunkThreads) {
    const unsigned b = q / (unsigned)l.n, k = q - b * (unsigned)l.n;
    const ListSource s = list_source(t, l, (int)b, (int)k);
    if (s.comp >= 0 && !(HARD && s.mode != 0) &&
        ((unsigned)s.at >> 5) % gridDim.x == blockIdx.x)
      f(s, (int)k);
  }
}
template <bool HARD>
__device__ __forceinline__ void find_sources(const TmzDev& t, const SourceList& l, OwnSources& own) {
  if (l.n == 0) return;
  if (threadIdx.x == 0) own.count = 0;
  __syncthreads();
  walk_list<HARD>(t, l, [&](const ListSource& s, int k) {
    const int q = atomicAdd(&own.count, 1);
    if (q >= kOwnSources) return;
    own.at[q] = (unsigned)s.at | (unsigned)(s.comp - 2) << 24 | (s.mode == 0 ? 1u << 26 : 0u);
    own.entry[q] = k;
  });
  __syncthreads();
}
// f for each of them, after the block's points.
template <bool HARD, class F>
__device__ __forceinline__ void for_sources(const TmzDev& t, const SourceList& l,
                                            const OwnSources& own, F f) {
  if (l.n == 0 || own.count == 0) return;
  __syncthreads();
  if (own.count > kOwnSources) {
    walk_list<HARD>(t, l, f);
    return;
  }
  for (int q = threadIdx.x; q < own.count; q += kChunkThreads) {
    const unsigned a = own.at[q];
    f(ListSource{(int)(a >> 24 & 3) + 2, (int)(~a >> 26 & 1), (int64_t)(a & 0xffffffu)},
      own.entry[q]);
  }
}

// Groups of 32 points go round the blocks in turn, so that every SM gets its
// share of the absorbing layer, the design and the sources.
template <class F>
__device__ __forceinline__ void for_points(const TmzDev& t, const LatDiv& d, F f) {
  const unsigned total = (unsigned)(t.plane * t.nb), groups = (total + 31) / 32;
  for (unsigned q = blockIdx.x + (threadIdx.x >> 5) * gridDim.x; q < groups;
       q += kChunkThreads / 32 * gridDim.x) {
    const unsigned at = q * 32 + (threadIdx.x & 31);
    if (at < total) f(lattice_at(t, d, at));
  }
}

// Forward steps step0 + 1 .. step0 + nsteps (flags: GMES_TMZ_RECORD_*).
template <class P>
__global__ void __launch_bounds__(kChunkThreads, 2)
    k_tmz_chunk_fwd(const __grid_constant__ GridDev g, const __grid_constant__ TmzDev t,
                    const LatDiv d, const SourceList l, const __grid_constant__ Meeting meet,
                    int step0, int nsteps, int flags, int* error) {
  __shared__ OwnSources own;
  find_sources<false>(t, l, own);
  auto met = [&] {
    if (grid_barrier(meet, error)) return true;
    const int64_t es = sizeof(typename P::T), nd = (int64_t)t.dn[0] * t.dn[1];
    for (int q = 0; q < 3; ++q) spoil(t.f[q], t.nb * t.plane * es);
    if (flags & GMES_TMZ_RECORD_HIST) spoil(t.hist, (int64_t)t.hist_steps * t.nb * nd * es);
    if (flags & GMES_TMZ_RECORD_MONITOR)
      spoil(t.mon, (int64_t)t.nb * t.total_steps * t.mn[0] * t.mn[1] * 8);
    return false;
  };
  for (int k = 0; k < nsteps; ++k) {
    const int n = step0 + k + 1;
    for_points(t, d, [&](const Lat& p) {
      point_fe<P>(g, t, p, n, (flags & GMES_TMZ_RECORD_HIST) ? k : -1);
    });
    for_sources<false>(t, l, own, [&](const ListSource& s, int q) {
      source_fwd<P>(t, l, 0, n, s, q);
    });
    if (!met()) return;
    if (k + 1 == nsteps) leave_barrier(meet);
    for_points(t, d, [&](const Lat& p) {
      point_fh<P>(g, t, p, n, (flags & GMES_TMZ_RECORD_MONITOR) ? n - 1 : -1);
    });
    for_sources<false>(t, l, own, [&](const ListSource& s, int q) {
      source_fwd<P>(t, l, 1, n, s, q);
    });
    if (k + 1 < nsteps && !met()) return;
  }
}

// Adjoint steps step0 + nsteps down to step0 + 1.
template <class P>
__global__ void __launch_bounds__(kChunkThreads, 2)
    k_tmz_chunk_adj(const __grid_constant__ GridDev g, const __grid_constant__ TmzDev t,
                    const LatDiv d, const SourceList l, const __grid_constant__ Meeting meet,
                    int step0, int nsteps, int* error) {
  __shared__ OwnSources own;
  find_sources<true>(t, l, own);
  auto met = [&] {
    if (grid_barrier(meet, error)) return true;
    spoil(t.grad, (int64_t)t.nb * t.dn[0] * t.dn[1] * 8);
    return false;
  };
  if (l.n > 0) {  // the H sources of the first step
    for_sources<true>(t, l, own, [&](const ListSource& s, int) { source_adj<P>(t, 1, s); });
    if (!met()) return;
  }
  for (int k = nsteps - 1; k >= 0; --k) {
    const int n = step0 + k + 1, rb = n & 1, wb = rb ^ 1;
    for_points(t, d, [&](const Lat& p) { point_ah<P>(g, t, p, n, rb, wb); });
    for_sources<true>(t, l, own, [&](const ListSource& s, int) { source_adj<P>(t, 0, s); });
    if (!met()) return;
    if (k == 0) leave_barrier(meet);
    for_points(t, d, [&](const Lat& p) { point_ae<P>(g, t, p, k, rb, wb); });
    if (k > 0)
      for_sources<true>(t, l, own, [&](const ListSource& s, int) { source_adj<P>(t, 1, s); });
    if (k > 0 && !met()) return;
  }
}

// ---------------------------------------------------------------------------
// Temporally blocked kernels (FP32).
// ---------------------------------------------------------------------------
// A block owns a TI x TJ tile of one design's lattice and advances the region
// of RI x RJ = (TI + 2 H) x (TJ + 2 H) points around it (region point (a, c) is
// lattice point (ri0 + a, rj0 + c) taken periodically, so tiles at the lattice
// edge see its periodic images) by up to H steps per launch.  An E update reads
// its low-side neighbours (i-1, j-1) and an H update its high-side ones
// (i+1, j+1), so each half-step leaves the values exact on the region shrunk by
// one more row and column on one side; after s <= H steps they are exact on
// [s, RI-1-s] (H fields) and [s, RI-s] (E), which contain the tile.  What the
// region's edge points hold meanwhile is never stored.  DRAM traffic per step
// falls from a read and write of every field per half-step to one read of the
// region and one write of the tile per H steps.
//
// The region lives in registers: a warp holds Q whole rows, a lane columns 2 l
// and 2 l + 1 of each.  The neighbour along j is in the lane or one shuffle
// away (one per two points), the neighbour along i in the lane, or, for the
// warp's first or last row, in the row that the next warp left in shared
// memory (two rows per warp and half-step, one barrier).  Measured on GB300
// (512^2, 64 designs, 200 steps, ms forward / adjoint), against the form with
// every field in shared memory (13 accesses per point-step forward, 21
// adjoint; 113 instructions), which general tiles still take: 27.6 / 31.7 ->
// 12.4 / 16.1.  The plain tiles alone (121 of 220) take 4.3 / 5.0 of it, near
// the time of reading their regions and writing their tiles (5 TB/s); the
// absorbing ones are bound by instruction issue at 32 warps per SM.
//
// What a tile's points are is settled once per design set (k_tmz_tiles), so
// that the loops carry no per-point look-ups: plain tiles, most of them with
// one set of coefficients; tiles with absorbing rows or absorbing columns,
// whose psi stay in registers; and general tiles (TbTile), which take a
// per-point loop over fields in shared memory.
constexpr int kTbHalo = GMES_TMZ_MAX_BLOCK_STEPS;  // most steps per launch
constexpr int kTbRJ = 64;                          // region columns (j)
constexpr int kTbTJ = kTbRJ - 2 * kTbHalo;
constexpr int kTbWarps = 16;
constexpr int kTbThreads = 32 * kTbWarps;
static_assert(kTbHalo % 2 == 0, "a lane's two columns lie in the tile together");

__device__ __forceinline__ int wrap_index(int v, int n) {
  if (v < 0) v += n;
  if (v >= n) v -= n;
  if (v >= 0 && v < n) return v;
  v %= n;  // regions wider than twice the lattice
  return v < 0 ? v + n : v;
}

// Q: rows per warp.
template <class P, int Q>
struct TbGeom {
  using R = typename P::R;
  static constexpr int RI = Q * kTbWarps, TI = RI - 2 * kTbHalo, NP = RI * kTbRJ;
  // shared memory (values): the exchanged rows (one slot more per direction
  // for the region's edge) and the layer's row and column entries, then, over the same
  // bytes, a special tile's gradient state (2 FP64 per point, adjoint) and
  // source map, or a general tile's 7 (forward) or 11 (adjoint) arrays
  static constexpr int kRows = 2 * (kTbWarps + 1) * kTbRJ;
  static constexpr int kHead = kRows + 6 * RI + 6 * kTbRJ;
  static constexpr size_t special = (size_t)NP * (2 * sizeof(double) + sizeof(uint16_t));
  static constexpr size_t fwd_bytes =
      (size_t)kHead * sizeof(R) + (7 * NP * sizeof(R) > special ? 7 * NP * sizeof(R) : special);
  static constexpr size_t adj_bytes =
      (size_t)kHead * sizeof(R) + (11 * NP * sizeof(R) > special ? 11 * NP * sizeof(R) : special);
  static_assert((kHead * sizeof(R)) % 16 == 0, "FP64 state is aligned");
};

// A point in the region's source maps: entry + 1, and whether it is hard.
constexpr unsigned kTbHard = 0x8000u;

// The block's tile and design: the designs of one tile are neighbours, so
// that the blocks of an SM mostly run the same form and share the map.
struct TbBlock {
  int b, tile, row, col;
  __device__ __forceinline__ TbBlock(const TmzDev& t) {
    const unsigned n = (unsigned)t.nb, cols = (unsigned)(t.ny + kTbTJ - 1) / kTbTJ;
    tile = (int)(blockIdx.x / n);
    b = (int)(blockIdx.x - (unsigned)tile * n);
    row = (int)((unsigned)tile / cols);
    col = (int)((unsigned)tile - (unsigned)row * cols);
  }
};

// What every thread of a block knows of its place.
template <class P, int Q>
struct TbPlace {
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  int lane, warp, b, ri0, rj0, j0, j1;
  int64_t base;
  bool pair, jt0, jt1;  // columns adjacent in memory; columns in the tile
  int li[Q];
  __device__ __forceinline__ TbPlace(const TmzDev& t) {
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    const TbBlock k(t);
    b = k.b;
    ri0 = k.row * G::TI - kTbHalo;
    rj0 = k.col * kTbTJ - kTbHalo;
    const int c = 2 * lane;
    j0 = wrap_index(rj0 + c, t.ny);
    j1 = wrap_index(rj0 + c + 1, t.ny);
    pair = (t.ny & 1) == 0;
    const bool in = c >= kTbHalo && c < kTbHalo + kTbTJ;
    jt0 = in && rj0 + c < t.ny;
    jt1 = in && rj0 + c + 1 < t.ny;
    base = (int64_t)b * t.plane;
#pragma unroll
    for (int q = 0; q < Q; ++q) li[q] = wrap_index(ri0 + warp * Q + q, t.nx);
  }
  __device__ __forceinline__ bool row_in_tile(const TmzDev& t, int q) const {
    const int a = warp * Q + q;
    return a >= kTbHalo && a < kTbHalo + G::TI && ri0 + a < t.nx;
  }
  // the lane's two values of row q of an array of the design
  __device__ __forceinline__ void load(const TmzDev& t, const void* p, int q, R v[2]) const {
    const R* row = static_cast<const R*>(p) + base + (int64_t)li[q] * t.ny;
    if (pair) {
      struct alignas(2 * sizeof(R)) Two {
        R a, b;
      };
      const Two w = *reinterpret_cast<const Two*>(row + j0);
      v[0] = w.a;
      v[1] = w.b;
    } else {
      v[0] = row[j0];
      v[1] = row[j1];
    }
  }
  __device__ __forceinline__ void store(const TmzDev& t, void* p, int q, const R v[2]) const {
    R* row = static_cast<R*>(p) + base + (int64_t)li[q] * t.ny;
    if (pair && jt0 && jt1) {
      struct alignas(2 * sizeof(R)) Two {
        R a, b;
      };
      *reinterpret_cast<Two*>(row + j0) = Two{v[0], v[1]};
    } else {
      if (jt0) row[j0] = v[0];
      if (jt1) row[j1] = v[1];
    }
  }
};

// Two neighbouring values of a shared-memory row.
template <class R>
struct alignas(2 * sizeof(R)) Row2 {
  R a, b;
};

// Entry m (b, c / d, 1 / (kappa d)) of layer pm's profiles: Ez and Hy along x,
// Ez and Hx along y, at a lattice index.
__device__ __forceinline__ int tb_entry(int m) { return m == 0 ? 0 : m + 2; }
template <class P>
__device__ __forceinline__ typename P::R prof_ex(const GridDev& g, int pm, int m, int i) {
  return P::cfg(g.prof[pm][2][0] + (int64_t)i * kProfStride + tb_entry(m));
}
template <class P>
__device__ __forceinline__ typename P::R prof_yx(const GridDev& g, int pm, int m, int i) {
  return P::cfg(g.prof[pm][4][0] + (int64_t)(i + 1) * kProfStride + tb_entry(m));
}
template <class P>
__device__ __forceinline__ typename P::R prof_ey(const GridDev& g, int pm, int m, int j) {
  return P::cfg(g.prof[pm][2][1] + (int64_t)j * kProfStride + tb_entry(m));
}
template <class P>
__device__ __forceinline__ typename P::R prof_xy(const GridDev& g, int pm, int m, int j) {
  return P::cfg(g.prof[pm][3][1] + (int64_t)(j + 1) * kProfStride + tb_entry(m));
}

// A tile's absorbing rows (KIND kTbRows: on along x, Ez and Hy), columns
// (kTbCols: on along y, Ez and Hx) or both (kTbBoth), with their psi (or psi adjoints) in
// registers.  The updates are those of e_cpml and its siblings, term for term,
// with the psi that is off left out (it is zero).  A row's state is
// warp-uniform and branches; a column's selects.
template <class P, int Q, int KIND>
struct TbLayer {};

template <class P, int Q>
struct TbLayer<P, Q, kTbRows> {
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  bool re[Q], ry[Q];  // row on for Ez / Hy
  R se[Q][2], sy[Q][2], k2[2];  // k2: the lane's columns' 1 / (kappa d) along y
  __device__ __forceinline__ void load(const TmzDev& t, const TbPlace<P, Q>& p,
                                       void* const* src) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned f = __ldg(t.pflags + (int64_t)p.li[q] * t.ny + p.j0);
      re[q] = __any_sync(0xffffffffu, f & kTmzOnE1);
      ry[q] = __any_sync(0xffffffffu, f & kTmzOnY);
      p.load(t, src[0], q, se[q]);
      p.load(t, src[3], q, sy[q]);
    }
  }
  // the region rows' entries: Ez's b, c / d, 1 / (kappa d), then Hy's
  __device__ __forceinline__ void fill(const GridDev& g, const TmzDev& t, const TbPlace<P, Q>& p,
                                       const TbTile<R>& tile, R* sR) const {
    for (int k = threadIdx.x; k < G::RI; k += kTbThreads) {
      const int i = wrap_index(p.ri0 + k, t.nx);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        sR[m * G::RI + k] = prof_ex<P>(g, tile.pm, m, i);
        sR[(3 + m) * G::RI + k] = prof_yx<P>(g, tile.pm, m, i);
      }
    }
    for (int c = threadIdx.x; c < kTbRJ; c += kTbThreads)
      sR[6 * G::RI + c] = prof_ey<P>(g, tile.pm, 2, wrap_index(p.rj0 + c, t.ny));
  }
  __device__ __forceinline__ void columns(const R* sR, int lane) {
    k2[0] = sR[6 * G::RI + 2 * lane];
    k2[1] = sR[6 * G::RI + 2 * lane + 1];
  }
  __device__ __forceinline__ void store(const TmzDev& t, const TbPlace<P, Q>& p,
                                        void* const* dst) const {
    const R none[2] = {P::zero(), P::zero()};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!p.row_in_tile(t, q)) continue;
      if (re[q]) {  // both psi of every absorbing Ez point
        p.store(t, dst[0], q, se[q]);
        p.store(t, dst[1], q, none);
      }
      if (ry[q]) p.store(t, dst[3], q, sy[q]);
    }
  }
  __device__ __forceinline__ R e_fwd(const R* sR, int a, int q, int h, R e, R c1, R c2n, R cdt,
                                     R D1, R D2) {
    if (!re[q]) return fmadd(fmadd(e, c1, D1), c2n, D2);
    se[q][h] = fmadd(sR[a] * se[q][h], sR[G::RI + a], D1);
    return fmadd(e, cdt, fmadd(fmadd(se[q][h] - P::zero(), sR[2 * G::RI + a], D1), -k2[h], D2));
  }
  __device__ __forceinline__ R x_fwd(int, int, R x, R cxn, R, R D1) { return fmadd(x, cxn, D1); }
  __device__ __forceinline__ R y_fwd(const R* sR, int a, int q, int h, R y, R cy, R cdt, R D2) {
    if (!ry[q]) return fmadd(y, cy, D2);
    sy[q][h] = fmadd(sR[3 * G::RI + a] * sy[q][h], sR[4 * G::RI + a], D2);
    return fmadd(y, -cdt, fmadd(-sy[q][h], -sR[5 * G::RI + a], D2));
  }
  // curl weights; the psi adjoint of an absorbing point advances
  __device__ __forceinline__ R y_adj(const R* sR, int a, int q, int h, R l, R cy, R cdt) {
    if (!ry[q]) return cy * l;
    const R direct = cdt * (sR[5 * G::RI + a] * l);
    const R t = fmadd(sy[q][h], cdt, l);
    sy[q][h] = sR[3 * G::RI + a] * t;
    return fmadd(direct, sR[4 * G::RI + a], t);
  }
  __device__ __forceinline__ R x_adj(int, int, R l, R cxn, R) { return cxn * l; }
  __device__ __forceinline__ void e_adj(const R* sR, int a, int q, int h, R l, R c1, R c2n, R cdt,
                                        R& v1, R& v2) {
    if (!re[q]) {
      v1 = c1 * l;
      v2 = c2n * l;
      return;
    }
    const R t = fmadd(se[q][h], cdt, l);
    v1 = fmadd(cdt * (sR[2 * G::RI + a] * l), sR[G::RI + a], t);
    v2 = -(cdt * (k2[h] * l));
    se[q][h] = sR[a] * t;
  }
};

template <class P, int Q>
struct TbLayer<P, Q, kTbCols> {
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  bool ce[2], cx[2];  // column on for Ez / Hx
  R ey[3][2], xy[3][2];
  R se[Q][2], sx[Q][2];
  __device__ __forceinline__ void load(const TmzDev& t, const TbPlace<P, Q>& p,
                                       void* const* src) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned f = __ldg(t.pflags + (int64_t)p.li[0] * t.ny + (h ? p.j1 : p.j0));
      ce[h] = f & kTmzOnE2;
      cx[h] = f & kTmzOnX;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      p.load(t, src[1], q, se[q]);
      p.load(t, src[2], q, sx[q]);
    }
  }
  // the region columns' entries (Ez's, then Hx's) and the rows' 1 / (kappa d)
  __device__ __forceinline__ void fill(const GridDev& g, const TmzDev& t, const TbPlace<P, Q>& p,
                                       const TbTile<R>& tile, R* sR) const {
    for (int k = threadIdx.x; k < G::RI; k += kTbThreads)
      sR[2 * G::RI + k] = prof_ex<P>(g, tile.pm, 2, wrap_index(p.ri0 + k, t.nx));
    for (int c = threadIdx.x; c < kTbRJ; c += kTbThreads) {
      const int j = wrap_index(p.rj0 + c, t.ny);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        sR[6 * G::RI + m * kTbRJ + c] = prof_ey<P>(g, tile.pm, m, j);
        sR[6 * G::RI + (3 + m) * kTbRJ + c] = prof_xy<P>(g, tile.pm, m, j);
      }
    }
  }
  // the lane's columns' entries (after a barrier); off its slab a column's psi
  // stays zero: b = c = 0, whatever the buffer holds there
  __device__ __forceinline__ void columns(const R* sR, int lane) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        ey[m][h] = sR[6 * G::RI + m * kTbRJ + 2 * lane + h];
        xy[m][h] = sR[6 * G::RI + (3 + m) * kTbRJ + 2 * lane + h];
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (!ce[h]) se[q][h] = P::zero();
        if (!cx[h]) sx[q][h] = P::zero();
      }
    }
  }
  __device__ __forceinline__ void store(const TmzDev& t, const TbPlace<P, Q>& p,
                                        void* const* dst) const {
    const R none[2] = {P::zero(), P::zero()};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!p.row_in_tile(t, q)) continue;
      if (__any_sync(0xffffffffu, ce[0] || ce[1])) {
        p.store(t, dst[0], q, none);
        p.store(t, dst[1], q, se[q]);
      }
      p.store(t, dst[2], q, sx[q]);
    }
  }
  __device__ __forceinline__ R e_fwd(const R* sR, int a, int q, int h, R e, R c1, R c2n, R cdt,
                                     R D1, R D2) {
    const R n = fmadd(ey[0][h] * se[q][h], ey[1][h], D2);
    const R on = fmadd(e, cdt, fmadd(fmadd(P::zero() - n, sR[2 * G::RI + a], D1), -ey[2][h], D2));
    const R off = fmadd(fmadd(e, c1, D1), c2n, D2);
    se[q][h] = ce[h] ? n : se[q][h];
    return ce[h] ? on : off;
  }
  __device__ __forceinline__ R x_fwd(int q, int h, R x, R cxn, R cdt, R D1) {
    const R n = fmadd(xy[0][h] * sx[q][h], xy[1][h], D1);
    const R on = fmadd(x, -cdt, fmadd(n, xy[2][h], D1));
    const R off = fmadd(x, cxn, D1);
    sx[q][h] = cx[h] ? n : sx[q][h];
    return cx[h] ? on : off;
  }
  __device__ __forceinline__ R y_fwd(const R*, int, int, int, R y, R cy, R, R D2) {
    return fmadd(y, cy, D2);
  }
  __device__ __forceinline__ R y_adj(const R*, int, int, int, R l, R cy, R) { return cy * l; }
  __device__ __forceinline__ R x_adj(int q, int h, R l, R cxn, R cdt) {
    const R direct = -(cdt * (xy[2][h] * l));
    const R t = fmadd(sx[q][h], -cdt, l);
    const R on = fmadd(direct, xy[1][h], t);
    sx[q][h] = cx[h] ? xy[0][h] * t : sx[q][h];
    return cx[h] ? on : cxn * l;
  }
  __device__ __forceinline__ void e_adj(const R* sR, int a, int q, int h, R l, R c1, R c2n, R cdt,
                                        R& v1, R& v2) {
    const R t = fmadd(se[q][h], -cdt, l);
    const R n2 = fmadd(-(cdt * (ey[2][h] * l)), ey[1][h], t);
    v1 = ce[h] ? cdt * (sR[2 * G::RI + a] * l) : c1 * l;
    v2 = ce[h] ? n2 : c2n * l;
    se[q][h] = ce[h] ? ey[0][h] * t : se[q][h];
  }
};

template <class P, int Q>
struct TbLayer<P, Q, kTbBoth> {
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  bool re[Q], ry[Q], ce[2], cx[2];
  R ey[3][2], xy[3][2];
  R s1[Q][2], s2[Q][2], sx[Q][2], sy[Q][2];
  __device__ __forceinline__ void load(const TmzDev& t, const TbPlace<P, Q>& p,
                                       void* const* src) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned f = __ldg(t.pflags + (int64_t)p.li[0] * t.ny + (h ? p.j1 : p.j0));
      ce[h] = f & kTmzOnE2;
      cx[h] = f & kTmzOnX;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned f = __ldg(t.pflags + (int64_t)p.li[q] * t.ny + p.j0);
      re[q] = __any_sync(0xffffffffu, f & kTmzOnE1);
      ry[q] = __any_sync(0xffffffffu, f & kTmzOnY);
      p.load(t, src[0], q, s1[q]);
      p.load(t, src[1], q, s2[q]);
      p.load(t, src[2], q, sx[q]);
      p.load(t, src[3], q, sy[q]);
    }
  }
  __device__ __forceinline__ void fill(const GridDev& g, const TmzDev& t, const TbPlace<P, Q>& p,
                                       const TbTile<R>& tile, R* sR) const {
    for (int k = threadIdx.x; k < G::RI; k += kTbThreads) {
      const int i = wrap_index(p.ri0 + k, t.nx);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        sR[m * G::RI + k] = prof_ex<P>(g, tile.pm, m, i);
        sR[(3 + m) * G::RI + k] = prof_yx<P>(g, tile.pm, m, i);
      }
    }
    for (int c = threadIdx.x; c < kTbRJ; c += kTbThreads) {
      const int j = wrap_index(p.rj0 + c, t.ny);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        sR[6 * G::RI + m * kTbRJ + c] = prof_ey<P>(g, tile.pm, m, j);
        sR[6 * G::RI + (3 + m) * kTbRJ + c] = prof_xy<P>(g, tile.pm, m, j);
      }
    }
  }
  __device__ __forceinline__ void columns(const R* sR, int lane) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        ey[m][h] = sR[6 * G::RI + m * kTbRJ + 2 * lane + h];
        xy[m][h] = sR[6 * G::RI + (3 + m) * kTbRJ + 2 * lane + h];
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (!re[q]) s1[q][h] = P::zero();
        if (!ry[q]) sy[q][h] = P::zero();
        if (!ce[h]) s2[q][h] = P::zero();
        if (!cx[h]) sx[q][h] = P::zero();
      }
    }
  }
  __device__ __forceinline__ void store(const TmzDev& t, const TbPlace<P, Q>& p,
                                        void* const* dst) const {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!p.row_in_tile(t, q)) continue;
      p.store(t, dst[0], q, s1[q]);
      p.store(t, dst[1], q, s2[q]);
      p.store(t, dst[2], q, sx[q]);
      p.store(t, dst[3], q, sy[q]);
    }
  }
  __device__ __forceinline__ R e_fwd(const R* sR, int a, int q, int h, R e, R c1, R c2n, R cdt,
                                     R D1, R D2) {
    if (re[q]) s1[q][h] = fmadd(sR[a] * s1[q][h], sR[G::RI + a], D1);
    const R n2 = fmadd(ey[0][h] * s2[q][h], ey[1][h], D2);
    s2[q][h] = ce[h] ? n2 : s2[q][h];
    const R on =
        fmadd(e, cdt, fmadd(fmadd(s1[q][h] - s2[q][h], sR[2 * G::RI + a], D1), -ey[2][h], D2));
    if (re[q]) return on;
    const R off = fmadd(fmadd(e, c1, D1), c2n, D2);
    return ce[h] ? on : off;
  }
  __device__ __forceinline__ R x_fwd(int q, int h, R x, R cxn, R cdt, R D1) {
    const R n = fmadd(xy[0][h] * sx[q][h], xy[1][h], D1);
    const R on = fmadd(x, -cdt, fmadd(n, xy[2][h], D1));
    const R off = fmadd(x, cxn, D1);
    sx[q][h] = cx[h] ? n : sx[q][h];
    return cx[h] ? on : off;
  }
  __device__ __forceinline__ R y_fwd(const R* sR, int a, int q, int h, R y, R cy, R cdt, R D2) {
    if (!ry[q]) return fmadd(y, cy, D2);
    sy[q][h] = fmadd(sR[3 * G::RI + a] * sy[q][h], sR[4 * G::RI + a], D2);
    return fmadd(y, -cdt, fmadd(-sy[q][h], -sR[5 * G::RI + a], D2));
  }
  __device__ __forceinline__ R y_adj(const R* sR, int a, int q, int h, R l, R cy, R cdt) {
    if (!ry[q]) return cy * l;
    const R direct = cdt * (sR[5 * G::RI + a] * l);
    const R t = fmadd(sy[q][h], cdt, l);
    sy[q][h] = sR[3 * G::RI + a] * t;
    return fmadd(direct, sR[4 * G::RI + a], t);
  }
  __device__ __forceinline__ R x_adj(int q, int h, R l, R cxn, R cdt) {
    const R direct = -(cdt * (xy[2][h] * l));
    const R t = fmadd(sx[q][h], -cdt, l);
    const R on = fmadd(direct, xy[1][h], t);
    sx[q][h] = cx[h] ? xy[0][h] * t : sx[q][h];
    return cx[h] ? on : cxn * l;
  }
  __device__ __forceinline__ void e_adj(const R* sR, int a, int q, int h, R l, R c1, R c2n, R cdt,
                                        R& v1, R& v2) {
    const R d1 = cdt * (sR[2 * G::RI + a] * l), d2 = -(cdt * (ey[2][h] * l));
    const R t2 = fmadd(s2[q][h], -cdt, l);
    const R n2 = fmadd(d2, ey[1][h], t2);
    s2[q][h] = ce[h] ? ey[0][h] * t2 : s2[q][h];
    if (re[q]) {
      const R t1 = fmadd(s1[q][h], cdt, l);
      s1[q][h] = sR[a] * t1;
      v1 = fmadd(d1, sR[G::RI + a], t1);
      v2 = ce[h] ? n2 : d2;
    } else {
      v1 = ce[h] ? d1 : c1 * l;
      v2 = ce[h] ? n2 : c2n * l;
    }
  }
};

// The region's map of Ez sources: every copy of every source's point.
template <class P, int Q>
__device__ __forceinline__ void tb_source_map(const TmzDev& t, int ri0, int rj0, uint16_t* map) {
  using G = TbGeom<P, Q>;
  static_assert(G::NP % 8 == 0, "cleared as 16-byte words");
  for (int k = threadIdx.x; k < G::NP / 8; k += kTbThreads)
    reinterpret_cast<uint4*>(map)[k] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int k = threadIdx.x; k < t.nsrc; k += kTbThreads) {
    const gmes_point_source s = t.src[k];
    if (s.comp != 2 || s.offset < 0 || s.offset >= t.plane) continue;
    int li, lj;
    if (t.plane < (int64_t(1) << 31)) {
      li = (int)((unsigned)s.offset / (unsigned)t.ny);
      lj = (int)((unsigned)s.offset - (unsigned)li * (unsigned)t.ny);
    } else {
      li = (int)(s.offset / t.ny);
      lj = (int)(s.offset - (int64_t)li * t.ny);
    }
    const uint16_t v = (uint16_t)((k + 1) | (s.mode == 0 ? kTbHard : 0u));
    for (int a = wrap_index(li - ri0, t.nx); a < G::RI; a += t.nx)
      for (int c = wrap_index(lj - rj0, t.ny); c < kTbRJ; c += t.ny) map[a * kTbRJ + c] = v;
  }
  __syncthreads();
}

// The value of the E half's source of step n at map entry v (0: none), and a
// field value after that source.
template <class P>
__device__ __forceinline__ typename P::R tb_value(const TmzDev& t, unsigned v, int n) {
  if (v == 0) return P::zero();
  const int k = (int)(v & (kTbHard - 1)) - 1;
  return P::from_double(__ldg(t.src_val + (int64_t)(n - 1) * 2 * t.nsrc + k));
}
template <class R>
__device__ __forceinline__ R tb_source(unsigned v, R f, R s) {
  return v == 0 ? f : ((v & kTbHard) ? s : f - s);
}

// A special tile: the flags that each of the lane's rows holds (warp-uniform),
// so that a row without any takes the bare update, and per point what its
// source, monitor and design pixel need.
template <class P, int Q>
struct TbSpecial {
  using R = typename P::R;
  using T = typename P::T;
  using G = TbGeom<P, Q>;
  unsigned row[Q];
  unsigned mine;   // the lane's points, bit 2 q + h: on the monitor; 8 above: its own pixels
  uint16_t* map;   // Ez sources
  double* acc;     // gradient of the launch, then -1 / eps, per region point
  R v[Q][2];       // source values (forward) or design increments (adjoint)
  R seeds[Q][2];   // adjoint
  __device__ __forceinline__ void init(unsigned char* smem) {
    acc = reinterpret_cast<double*>(smem + G::kHead * sizeof(R));
    map = reinterpret_cast<uint16_t*>(acc + 2 * G::NP);
#pragma unroll
    for (int q = 0; q < Q; ++q) row[q] = 0;
  }
  __device__ __forceinline__ unsigned flags(const TmzDev& t, const TbPlace<P, Q>& p, int q,
                                            int h) const {
    return __ldg(t.pflags + (int64_t)p.li[q] * t.ny + (h ? p.j1 : p.j0));
  }
  __device__ __forceinline__ bool owned(const TmzDev& t, const TbPlace<P, Q>& p, int q,
                                        int h) const {
    return p.row_in_tile(t, q) && (h ? p.jt1 : p.jt0);
  }
  __device__ __forceinline__ int64_t pixel(const TmzDev& t, const TbPlace<P, Q>& p, int q,
                                           int h) const {
    return design_index(t, p.li[q], h ? p.j1 : p.j0);
  }
  __device__ __forceinline__ int at(const TbPlace<P, Q>& p, int q, int h) const {
    return (p.warp * Q + q) * kTbRJ + 2 * p.lane + h;
  }
  __device__ __forceinline__ void load(const TmzDev& t, const TbPlace<P, Q>& p,
                                       const TbTile<R>& tile) {
    mine = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned f[2] = {flags(t, p, q, 0), flags(t, p, q, 1)};
      row[q] = __reduce_or_sync(0xffffffffu, f[0] | f[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (f[h] & kTmzMonitor) mine |= 1u << (2 * q + h);
        if ((f[h] & kTmzDesign) && owned(t, p, q, h)) mine |= 256u << (2 * q + h);
      }
    }
    if (tile.any & kTmzSrcE) tb_source_map<P, Q>(t, p.ri0, p.rj0, map);
  }
  // forward: the sources' values of step n, fetched a step ahead
  __device__ __forceinline__ void fetch(const TmzDev& t, const TbPlace<P, Q>& p, int n) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (row[q] & kTmzSrcE) {
        v[q][0] = tb_value<P>(t, map[at(p, q, 0)], n);
        v[q][1] = tb_value<P>(t, map[at(p, q, 1)], n);
      }
  }
  __device__ __forceinline__ void source(const TbPlace<P, Q>& p, int q, R e[2]) const {
    if (!(row[q] & kTmzSrcE)) return;
    e[0] = tb_source((unsigned)map[at(p, q, 0)], e[0], v[q][0]);
    e[1] = tb_source((unsigned)map[at(p, q, 1)], e[1], v[q][1]);
  }
  // forward: the design increment of a point of step slot
  __device__ __forceinline__ void record(const TmzDev& t, const TbPlace<P, Q>& p, int q, int h,
                                         int slot, R c1, R c2n, R D1, R D2) const {
    if ((flags(t, p, q, h) & kTmzDesign) && owned(t, p, q, h))
      static_cast<T*>(t.hist)[((int64_t)slot * t.nb + p.b) * t.dn[0] * t.dn[1] +
                              pixel(t, p, q, h)] = fmadd(c2n * D2, c1, D1);
  }
  __device__ __forceinline__ void monitor(const TmzDev& t, const TbPlace<P, Q>& p, int q, int n,
                                          const R e[2]) const {
    if (!(row[q] & kTmzMonitor)) return;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if ((flags(t, p, q, h) & kTmzMonitor) && owned(t, p, q, h))
        t.mon[((int64_t)p.b * t.total_steps + (n - 1)) * t.mn[0] * t.mn[1] +
              monitor_index(t, p.li[q], h ? p.j1 : p.j0)] = to_double(e[h]);
  }
  // adjoint: the objective's seeds of step n and the design increments of slot,
  // fetched together and a step ahead (one after another in the rows, with the
  // flags read again, the tiles of a 200x200 design took 16.5 us per launch, the
  // slowest 31; now 14 and 24); hard sources; and the design gradient, which
  // accumulates in shared memory over the launch
  __device__ __forceinline__ void seed_fetch(const GridDev& g, const TmzDev& t,
                                             const TbPlace<P, Q>& p, int n) {
    if ((mine & 255u) == 0) return;
    const double w = t.weight != nullptr ? t.weight[p.b] : 1.0;
    const double* at =
        t.mon + ((int64_t)p.b * t.total_steps + (n - 1)) * t.mn[0] * t.mn[1];
    double m[Q][2];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        m[q][h] = (mine >> (2 * q + h)) & 1
                      ? at[monitor_index(t, p.li[q], h ? p.j1 : p.j0)] : 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) seeds[q][h] = P::from_double(seed_value(g, w, m[q][h]));
  }
  __device__ __forceinline__ void seed(int q, R e[2]) const {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if ((mine >> (2 * q + h)) & 1) e[h] = e[h] + seeds[q][h];
  }
  __device__ __forceinline__ void zero(const TbPlace<P, Q>& p, int q, R e[2]) const {
    if (!(row[q] & kTmzSrcE)) return;
    if (map[at(p, q, 0)] & kTbHard) e[0] = P::zero();
    if (map[at(p, q, 1)] & kTbHard) e[1] = P::zero();
  }
  template <class F>
  __device__ __forceinline__ void pixels(const TmzDev& t, const TbPlace<P, Q>& p, F f) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (row[q] & kTmzDesign) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if ((mine >> (8 + 2 * q + h)) & 1) f(q, h, pixel(t, p, q, h));
      }
  }
  __device__ __forceinline__ void grad_load(const TmzDev& t, const TbPlace<P, Q>& p) {
    const int64_t b = (int64_t)p.b * t.dn[0] * t.dn[1];
    pixels(t, p, [&](int q, int h, int64_t dp) {
      acc[at(p, q, h)] = t.grad[b + dp];
      acc[G::NP + at(p, q, h)] = t.dc[b + dp].neg_reps;
    });
  }
  __device__ __forceinline__ void grad_fetch(const TmzDev& t, const TbPlace<P, Q>& p, int slot) {
    const int64_t b = ((int64_t)slot * t.nb + p.b) * t.dn[0] * t.dn[1];
    pixels(t, p, [&](int q, int h, int64_t dp) {
      v[q][h] = P::ldw(static_cast<const T*>(t.hist) + b + dp);
    });
  }
  __device__ __forceinline__ void grad_add(const TbPlace<P, Q>& p, int q, const R e[2]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if ((mine >> (8 + 2 * q + h)) & 1) {
        const int k = at(p, q, h);
        acc[k] += to_double(e[h]) * to_double(v[q][h]) * acc[G::NP + k];
      }
  }
  __device__ __forceinline__ void grad_store(const TmzDev& t, const TbPlace<P, Q>& p) {
    const int64_t b = (int64_t)p.b * t.dn[0] * t.dn[1];
    pixels(t, p, [&](int q, int h, int64_t dp) { t.grad[b + dp] = acc[at(p, q, h)]; });
  }
};

// Ez's coefficients of the lane's two points of row q: the tile's, or, where
// they vary, those that load() took (c1 and c2n; an absorbing point's cdt is
// its c1).
template <class P, int Q, bool VARY>
struct TbCoef {
  using R = typename P::R;
  R c1[Q][2], c2n[Q][2];
  __device__ __forceinline__ void load(const TmzDev& t, const TbPlace<P, Q>& p) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = h ? p.j1 : p.j0;
        const int64_t ll = (int64_t)p.li[q] * t.ny + j;
        e_coef<P>(t, p.b, p.li[q], j, ll, __ldg(t.pflags + ll), c1[q][h], c2n[q][h]);
      }
  }
  __device__ __forceinline__ void get(const TbTile<R>&, int q, int h, R& a, R& b) const {
    a = c1[q][h];
    b = c2n[q][h];
  }
};
template <class P, int Q>
struct TbCoef<P, Q, false> {
  using R = typename P::R;
  __device__ __forceinline__ void load(const TmzDev&, const TbPlace<P, Q>&) {}
  __device__ __forceinline__ void get(const TbTile<R>& tile, int, int, R& a, R& b) const {
    a = tile.c[0];
    b = tile.c[1];
  }
};

template <bool B>
struct BoolTag {
  static constexpr bool value = B;
};

// Plain-form coefficients of one region point.
template <class R>
struct TbPoint {
  R c1, c2n;  // Ez: c1, -c2
  R cxn, cy;  // Hx: -c1, Hy: c2
};

// Flags and plain-form coefficients of lattice point (i, j) of design b,
// from the resolved map.
template <class P>
__device__ __forceinline__ unsigned tb_point(const TmzDev& t, int b, int i, int j,
                                             TbPoint<typename P::R>& p) {
  const int64_t ll = (int64_t)i * t.ny + j;
  const unsigned f = __ldg(t.pflags + ll);
  e_coef<P>(t, b, i, j, ll, f, p.c1, p.c2n);
  p.cxn = P::ldc(map_coef<P>(t, 2) + ll);
  p.cy = P::ldc(map_coef<P>(t, 3) + ll);
  return f;
}

// Apply this half's sources of step n to every copy of their point in the
// region: the forward (ADJ false: hard sources set the value, current
// sources subtract theirs) or the adjoint (ADJ true: hard sources zero it).
template <class P, bool ADJ>
__device__ __forceinline__ void tb_sources(const TmzDev& t, int side, int n, int ri0, int rj0,
                                           int RI, int RJ, typename P::R* fE,
                                           typename P::R* fX, typename P::R* fY) {
  using R = typename P::R;
  const int tid = threadIdx.x;
  for (int k = tid; k < t.nsrc; k += kTbThreads) {
    const gmes_point_source s = t.src[k];
    if (s.comp < 2 || s.comp > 4 || (s.comp == 2) != (side == 0)) continue;
    if (s.offset < 0 || s.offset >= t.plane) continue;
    if (ADJ && s.mode != 0) continue;
    const int li = (int)(s.offset / t.ny), lj = (int)(s.offset - (int64_t)li * t.ny);
    R* f = s.comp == 2 ? fE : (s.comp == 3 ? fX : fY);
    const R v =
        ADJ ? P::zero()
            : P::from_double(t.src_val[((int64_t)(n - 1) * 2 + side) * t.nsrc + k]);
    for (int a = wrap_index(li - ri0, t.nx); a < RI; a += t.nx)
      for (int c = wrap_index(lj - rj0, t.ny); c < RJ; c += t.ny) {
        R* q = f + a * RJ + c;
        *q = (ADJ || s.mode == 0) ? v : *q - v;
      }
  }
}

// The forward steps of a general tile: every field in shared memory, a thread
// the points of one column a few rows apart, per-point updates (e_cpml and its
// siblings) where the flags ask for them.
template <class P, int QW>
__device__ void tb_general_fwd(const GridDev& g, const TmzDev& t, int n0, int nsub, int slot0,
                               int rec_mon, unsigned char* smem) {
  using R = typename P::R;
  using T = typename P::T;
  using G = TbGeom<P, QW>;
  constexpr int H = kTbHalo, RJ = kTbRJ, RI = G::RI, TI = G::TI, TJ = kTbTJ, NP = G::NP;
  constexpr int kRowsAtOnce = kTbThreads / RJ, Q = RI / kRowsAtOnce;
  R* sE = reinterpret_cast<R*>(smem) + G::kHead;
  R* sX = sE + NP;
  R* sY = sX + NP;
  R* sS = sY + NP;  // psi of Ez (x, y), Hx, Hy: sS + k * NP
  const TbBlock blk(t);
  const int c = threadIdx.x % RJ, ty = threadIdx.x / RJ, b = blk.b;
  const int ri0 = blk.row * TI - H, rj0 = blk.col * TJ - H;
  const int j = wrap_index(rj0 + c, t.ny);
  const bool jtile = c >= H && c < H + TJ && rj0 + c < t.ny;
  const int64_t base = (int64_t)b * t.plane;
  int li[Q];
  TbPoint<R> pt[Q];
  unsigned fl[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int a = ty + kRowsAtOnce * q, k = a * RJ + c;
    li[q] = wrap_index(ri0 + a, t.nx);
    fl[q] = tb_point<P>(t, b, li[q], j, pt[q]);
    if (jtile && a >= H && a < H + TI && ri0 + a < t.nx) fl[q] |= 1u << 31;  // tile point
    const int64_t lin = base + (int64_t)li[q] * t.ny + j;
    sE[k] = static_cast<const T*>(t.f[0])[lin];
    sX[k] = static_cast<const T*>(t.f[1])[lin];
    sY[k] = static_cast<const T*>(t.f[2])[lin];
    if (fl[q] & kTmzPsiE) {
      sS[k] = static_cast<const T*>(t.f[3])[lin];
      sS[NP + k] = static_cast<const T*>(t.f[4])[lin];
    }
    if (fl[q] & kTmzPsiX) sS[2 * NP + k] = static_cast<const T*>(t.f[5])[lin];
    if (fl[q] & kTmzPsiY) sS[3 * NP + k] = static_cast<const T*>(t.f[6])[lin];
  }
  unsigned any = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) any |= fl[q];
  const bool src_e = __syncthreads_or(any & kTmzSrcE) != 0;  // also orders the loads
  const bool src_h = __syncthreads_or(any & kTmzSrcH) != 0;
  const int64_t nd = (int64_t)t.dn[0] * t.dn[1];
  const int64_t nm = (int64_t)t.mn[0] * t.mn[1];
  // Regions without CPML points inside a profile (most tiles) run a copy of
  // the sub-step loop without that code path: the choice is block-uniform,
  // and the arithmetic of every point is the same in both copies.
  const bool psi_any = __syncthreads_or(any & (kTmzPsiE | kTmzPsiX | kTmzPsiY)) != 0;
  auto steps = [&](auto tag) {
    constexpr bool PSI = decltype(tag)::value;
    for (int s = 0; s < nsub; ++s) {
      const int n = n0 + s + 1;
  #pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int a = ty + kRowsAtOnce * q, k = a * RJ + c;
        if (a >= 1 && c >= 1) {
          const R D1 = sY[k] - sY[k - RJ], D2 = sX[k] - sX[k - 1];
          if (fl[q] & kTmzPlainE) {
            sE[k] = fmadd(fmadd(sE[k], pt[q].c1, D1), pt[q].c2n, D2);
            if ((fl[q] & kTmzDesign) && (fl[q] >> 31) && slot0 >= 0)
              static_cast<T*>(t.hist)[((int64_t)(slot0 + s) * t.nb + b) * nd +
                                          design_index(t, li[q], j)] =
                  fmadd(pt[q].c2n * D2, pt[q].c1, D1);
          } else if (PSI && (fl[q] & kTmzPsiE)) {
            sE[k] = e_cpml<P>(g, fl[q], pt[q].c1, li[q], j, sE[k], D1, D2, sS + k, sS + NP + k);
          }
        }
      }
      __syncthreads();
      if (src_e) {
        tb_sources<P, false>(t, 0, n, ri0, rj0, RI, RJ, sE, sX, sY);
        __syncthreads();
      }
  #pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int a = ty + kRowsAtOnce * q, k = a * RJ + c;
        if (a < RI - 1 && c < RJ - 1) {
          const R e0 = sE[k];
          const R dx = sE[k + 1] - e0, dy = sE[k + RJ] - e0;
          if (fl[q] & kTmzPlainX)
            sX[k] = fmadd(sX[k], pt[q].cxn, dx);
          else if (PSI && (fl[q] & kTmzPsiX))
            sX[k] = x_cpml<P>(g, fl[q], pt[q].cxn, j, sX[k], dx, sS + 2 * NP + k);
          if (fl[q] & kTmzPlainY)
            sY[k] = fmadd(sY[k], pt[q].cy, dy);
          else if (PSI && (fl[q] & kTmzPsiY))
            sY[k] = y_cpml<P>(g, fl[q], pt[q].cy, li[q], sY[k], dy, sS + 3 * NP + k);
          if (rec_mon && (fl[q] & kTmzMonitor) && (fl[q] >> 31))
            t.mon[((int64_t)b * t.total_steps + (n - 1)) * nm + monitor_index(t, li[q], j)] =
                to_double(e0);
        }
      }
      __syncthreads();
      if (src_h) {
        tb_sources<P, false>(t, 1, n, ri0, rj0, RI, RJ, sE, sX, sY);
        __syncthreads();
      }
    }
  };
  if (psi_any)
    steps(BoolTag<true>{});
  else
    steps(BoolTag<false>{});
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!(fl[q] >> 31)) continue;
    const int k = (ty + kRowsAtOnce * q) * RJ + c;
    const int64_t lin = base + (int64_t)li[q] * t.ny + j;
    static_cast<T*>(t.tmp[0])[lin] = sE[k];
    static_cast<T*>(t.tmp[1])[lin] = sX[k];
    static_cast<T*>(t.tmp[2])[lin] = sY[k];
    if (fl[q] & kTmzPsiE) {
      static_cast<T*>(t.tmp[3])[lin] = sS[k];
      static_cast<T*>(t.tmp[4])[lin] = sS[NP + k];
    }
    if (fl[q] & kTmzPsiX) static_cast<T*>(t.tmp[5])[lin] = sS[2 * NP + k];
    if (fl[q] & kTmzPsiY) static_cast<T*>(t.tmp[6])[lin] = sS[3 * NP + k];
  }
}

// The adjoint steps of a general tile, as tb_general_fwd.
template <class P, int QW>
__device__ void tb_general_adj(const GridDev& g, const TmzDev& t, int n0, int nsub, int step0,
                               int rb, unsigned char* smem) {
  using R = typename P::R;
  using T = typename P::T;
  using G = TbGeom<P, QW>;
  constexpr int H = kTbHalo, RJ = kTbRJ, RI = G::RI, TI = G::TI, TJ = kTbTJ, NP = G::NP;
  constexpr int kRowsAtOnce = kTbThreads / RJ, Q = RI / kRowsAtOnce;
  R* sLE = reinterpret_cast<R*>(smem) + G::kHead;
  R* sLX = sLE + NP;
  R* sLY = sLX + NP;
  R* sP = sLY + NP;      // psi adjoints of Ez (x, y), Hx, Hy: sP + k * NP
  R* sW1 = sP + 4 * NP;  // curl weights of the H half: Hx
  R* sW2 = sW1 + NP;     //   and Hy
  R* sV1 = sW2 + NP;     // curl weights of the E half: Ez's first
  R* sV2 = sV1 + NP;     //   and its second
  const TbBlock blk(t);
  const int c = threadIdx.x % RJ, ty = threadIdx.x / RJ, b = blk.b;
  const int ri0 = blk.row * TI - H, rj0 = blk.col * TJ - H;
  const int j = wrap_index(rj0 + c, t.ny);
  const bool jtile = c >= H && c < H + TJ && rj0 + c < t.ny;
  const int64_t base = (int64_t)b * t.plane;
  const int wb = rb ^ 1;
  int li[Q];
  TbPoint<R> pt[Q];
  unsigned fl[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int a = ty + kRowsAtOnce * q;
    li[q] = wrap_index(ri0 + a, t.nx);
    fl[q] = tb_point<P>(t, b, li[q], j, pt[q]);
    if (jtile && a >= H && a < H + TI && ri0 + a < t.nx) fl[q] |= 1u << 31;  // tile point
  }
  after_previous();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int k = (ty + kRowsAtOnce * q) * RJ + c;
    const int64_t lin = base + (int64_t)li[q] * t.ny + j;
    sLE[k] = static_cast<const T*>(t.l[0])[lin];
    sLX[k] = static_cast<const T*>(t.l[1])[lin];
    sLY[k] = static_cast<const T*>(t.l[2])[lin];
    if (fl[q] & kTmzPsiE) {
      sP[k] = static_cast<const T*>(t.phi[rb][0])[lin];
      sP[NP + k] = static_cast<const T*>(t.phi[rb][1])[lin];
    }
    if (fl[q] & kTmzPsiX) sP[2 * NP + k] = static_cast<const T*>(t.phi[rb][2])[lin];
    if (fl[q] & kTmzPsiY) sP[3 * NP + k] = static_cast<const T*>(t.phi[rb][3])[lin];
  }
  unsigned any = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) any |= fl[q];
  const bool src_e = __syncthreads_or(any & kTmzSrcE) != 0;  // also orders the loads
  const bool src_h = __syncthreads_or(any & kTmzSrcH) != 0;
  const int64_t nd = (int64_t)t.dn[0] * t.dn[1];
  // as in k_tmz_tb_fwd: a copy of the loop without the CPML path for
  // regions that have no CPML point inside a profile
  const bool psi_any = __syncthreads_or(any & (kTmzPsiE | kTmzPsiX | kTmzPsiY)) != 0;
  // Per step (n = n0 + s + 1, s from nsub - 1 down to 0), the transposes of
  // the one-step kernels in their order: H-side sources, the curl weights
  // of every Hx / Hy point (hw), lambda_E gathering them (eu), E-side
  // sources, the curl weights of every Ez point and the gradient (ew),
  // lambda_X / lambda_Y gathering those (xu).  A point's weights depend
  // only on its own adjoints, so ew runs in the same pass as eu and the
  // next step's hw in the same pass as xu (into other arrays than the
  // neighbours read): two barriers per step.  A block holding a source
  // point applies it between the two, with barriers around it.
  auto steps = [&](auto tag) {
    constexpr bool PSI = decltype(tag)::value;
    auto hw = [&](int q) {
      const int k = (ty + kRowsAtOnce * q) * RJ + c;
      sW1[k] = (fl[q] & kTmzPlainX) ? pt[q].cxn * sLX[k]
               : (PSI && (fl[q] & kTmzPsiX))
                   ? adjx_cpml<P, true>(g, fl[q], pt[q].cxn, j, sLX[k], sP + 2 * NP + k,
                                        sP + 2 * NP + k)
                   : P::zero();
      sW2[k] = (fl[q] & kTmzPlainY) ? pt[q].cy * sLY[k]
               : (PSI && (fl[q] & kTmzPsiY))
                   ? adjy_cpml<P, true>(g, fl[q], pt[q].cy, li[q], sLY[k], sP + 3 * NP + k,
                                        sP + 3 * NP + k)
                   : P::zero();
    };
    auto eu = [&](int q, int n) {
      const int a = ty + kRowsAtOnce * q, k = a * RJ + c;
      if (a >= 1 && c >= 1) {
        R le = sLE[k];
        if (fl[q] & kTmzMonitor) {
          bool has;
          le = le + P::from_double(seed_of(g, t, b, li[q], j, n, &has));
        }
        sLE[k] = le + ((sW1[k - 1] - sW1[k]) + (sW2[k - RJ] - sW2[k]));
      }
    };
    auto ew = [&](int q, int n) {
      const int k = (ty + kRowsAtOnce * q) * RJ + c;
      R w1, w2;
      if (fl[q] & kTmzPlainE) {
        const R le = sLE[k];
        w1 = pt[q].c1 * le;
        w2 = pt[q].c2n * le;
      } else {
        w1 = w2 = P::zero();
        if (PSI && (fl[q] & kTmzPsiE))
          adje_cpml<P, true, true, true>(g, fl[q], pt[q].c1, li[q], j, sLE[k], sP + k, sP + k,
                                         sP + NP + k, sP + NP + k, w1, w2);
      }
      sV1[k] = w1;
      sV2[k] = w2;
      if ((fl[q] & kTmzDesign) && (fl[q] >> 31)) {
        const int64_t kk = (int64_t)b * nd + design_index(t, li[q], j);
        const double le = to_double(sLE[k]);
        const double inc = to_double(static_cast<const T*>(
            t.hist)[((int64_t)(n - step0 - 1) * t.nb + b) * nd + (kk - (int64_t)b * nd)]);
        t.grad[kk] += le * inc * t.dc[kk].neg_reps;
      }
    };
    auto xu = [&](int q) {
      const int a = ty + kRowsAtOnce * q, k = a * RJ + c;
      if (a < RI - 1 && c < RJ - 1) {
        sLX[k] = sLX[k] + (sV2[k] - sV2[k + 1]);
        sLY[k] = sLY[k] + (sV1[k] - sV1[k + RJ]);
      }
    };
    if (src_h) {
      tb_sources<P, true>(t, 1, n0 + nsub, ri0, rj0, RI, RJ, sLE, sLX, sLY);
      __syncthreads();
    }
  #pragma unroll
    for (int q = 0; q < Q; ++q) hw(q);
    __syncthreads();
    for (int s = nsub - 1; s >= 0; --s) {
      const int n = n0 + s + 1;
  #pragma unroll
      for (int q = 0; q < Q; ++q) eu(q, n);
      if (src_e) {
        __syncthreads();
        tb_sources<P, true>(t, 0, n, ri0, rj0, RI, RJ, sLE, sLX, sLY);
        __syncthreads();
      }
  #pragma unroll
      for (int q = 0; q < Q; ++q) ew(q, n);
      __syncthreads();
  #pragma unroll
      for (int q = 0; q < Q; ++q) xu(q);
      if (s > 0) {
        if (src_h) {
          __syncthreads();
          tb_sources<P, true>(t, 1, n - 1, ri0, rj0, RI, RJ, sLE, sLX, sLY);
          __syncthreads();
        }
  #pragma unroll
        for (int q = 0; q < Q; ++q) hw(q);
      }
      __syncthreads();
    }
  };
  if (psi_any)
    steps(BoolTag<true>{});
  else
    steps(BoolTag<false>{});
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!(fl[q] >> 31)) continue;
    const int k = (ty + kRowsAtOnce * q) * RJ + c;
    const int64_t lin = base + (int64_t)li[q] * t.ny + j;
    static_cast<T*>(t.tmp[0])[lin] = sLE[k];
    static_cast<T*>(t.tmp[1])[lin] = sLX[k];
    static_cast<T*>(t.tmp[2])[lin] = sLY[k];
    if (fl[q] & kTmzPsiE) {
      static_cast<T*>(t.phi[wb][0])[lin] = sP[k];
      static_cast<T*>(t.phi[wb][1])[lin] = sP[NP + k];
    }
    if (fl[q] & kTmzPsiX) static_cast<T*>(t.phi[wb][2])[lin] = sP[2 * NP + k];
    if (fl[q] & kTmzPsiY) static_cast<T*>(t.phi[wb][3])[lin] = sP[3 * NP + k];
  }
}

// Calls steps with the tile's form.
template <int KIND, bool FANCY>
struct TbForm {
  static constexpr int kind = KIND;
  static constexpr bool fancy = FANCY;
};
template <bool ADJ, class R, class F>
__device__ __forceinline__ void tb_dispatch(const TbTile<R>& tile, F& steps) {
  if (tile.kind == kTbRows)
    steps(TbForm<kTbRows, false>{});
  else if (tile.kind == kTbCols)
    steps(TbForm<kTbCols, false>{});
  else if (tile.kind == kTbBoth && (ADJ || !tile.fancy))
    steps(TbForm<kTbBoth, false>{});
  else if (tile.kind == kTbBoth)
    steps(TbForm<kTbBoth, !ADJ>{});
  else if (tile.fancy)
    steps(TbForm<kTbPlain, true>{});
  else
    steps(TbForm<kTbPlain, false>{});
}

// Forward steps n0+1 .. n0+nsub (nsub <= kTbHalo) of one tile, from the
// state in t.f to the state in t.tmp (the launch's other blocks still read
// t.f for their halos, so the result must not overwrite it).  slot0 >= 0:
// record the design increments of step n0+1+s at hist slot slot0+s;
// rec_mon: record monitor row n-1 of every step n.
template <class P, int Q>
__global__ void __launch_bounds__(kTbThreads, 2)
    k_tmz_tb_fwd(const GridDev g, const TmzDev t, int n0, int nsub, int slot0, int rec_mon) {
  after_launch();
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  using Two = Row2<R>;
  extern __shared__ __align__(16) unsigned char tb_smem[];
  const TbTile<R> tile =
      static_cast<const TbTile<R>*>(t.tiles)[TbBlock(t).tile];
  if (tile.kind == kTbGeneral) {
    tb_general_fwd<P, Q>(g, t, n0, nsub, slot0, rec_mon, tb_smem);
    return;
  }
  // rows left by the warps: sU slot w + 1 the last row of Hy of warp w, sD
  // slot w the first row of Ez of warp w; slots 0 / kTbWarps: beyond the region
  Two* const sU = reinterpret_cast<Two*>(tb_smem);
  Two* const sD = sU + (kTbWarps + 1) * kTbRJ / 2;
  R* const sR = reinterpret_cast<R*>(tb_smem) + G::kRows;  // layer rows' entries: Ez, Hy
  const TbPlace<P, Q> p(t);
  const int lane = p.lane, w = p.warp;
  R e[Q][2], x[Q][2], y[Q][2];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    p.load(t, t.f[0], q, e[q]);
    p.load(t, t.f[1], q, x[q]);
    p.load(t, t.f[2], q, y[q]);
  }
  if (w == 0) sU[lane] = Two{P::zero(), P::zero()};
  if (w == kTbWarps - 1) sD[kTbWarps * 32 + lane] = Two{P::zero(), P::zero()};
  sU[(w + 1) * 32 + lane] = Two{y[Q - 1][0], y[Q - 1][1]};
  constexpr unsigned kAll = 0xffffffffu;
  const R cxn = tile.c[2], cy = tile.c[3], de = tile.d[0], dx = tile.d[1], dy = tile.d[2];
  const bool design = slot0 >= 0 && (tile.any & kTmzDesign);
  const bool src = tile.any & kTmzSrcE, mon = rec_mon && (tile.any & kTmzMonitor);
  auto steps = [&](auto form) {
    constexpr int KIND = decltype(form)::kind;
    constexpr bool LAYER = KIND != kTbPlain, SP = decltype(form)::fancy;
    TbCoef<P, Q, SP> cf;
    TbLayer<P, Q, KIND> L;
    TbSpecial<P, Q> sp;
    cf.load(t, p);
    if constexpr (SP) {
      sp.init(tb_smem);
      sp.load(t, p, tile);
      if (src) sp.fetch(t, p, n0 + 1);
    }
    if constexpr (LAYER) {
      L.load(t, p, t.f + 3);
      L.fill(g, t, p, tile, sR);
    }
    __syncthreads();
    if constexpr (LAYER) L.columns(sR, lane);
    for (int s = 0; s < nsub; ++s) {
      const int n = n0 + s + 1;
      const Two up = sU[w * 32 + lane];
      R u[2] = {up.a, up.b};
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const R xl = __shfl_up_sync(kAll, x[q][1], 1);
        const R D2[2] = {x[q][0] - xl, x[q][1] - x[q][0]};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const R D1 = y[q][h] - u[h];
          u[h] = y[q][h];
          R c1, c2n;
          cf.get(tile, q, h, c1, c2n);
          if constexpr (SP)
            if (design && (sp.row[q] & kTmzDesign))
              sp.record(t, p, q, h, slot0 + s, c1, c2n, D1, D2[h]);
          if constexpr (LAYER)
            e[q][h] = L.e_fwd(sR, w * Q + q, q, h, e[q][h], c1, c2n, SP ? c1 : de, D1, D2[h]);
          else
            e[q][h] = fmadd(fmadd(e[q][h], c1, D1), c2n, D2[h]);
        }
        if constexpr (SP)
          if (src) sp.source(p, q, e[q]);
      }
      if constexpr (SP)
        if (src && s + 1 < nsub) sp.fetch(t, p, n + 1);
      sD[w * 32 + lane] = Two{e[0][0], e[0][1]};
      __syncthreads();
      const Two dn = sD[(w + 1) * 32 + lane];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const R er = __shfl_down_sync(kAll, e[q][0], 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const R below = q + 1 < Q ? e[q + 1 < Q ? q + 1 : q][h] : (h ? dn.b : dn.a);
          const R D1 = (h ? er : e[q][1]) - e[q][h], D2 = below - e[q][h];
          if constexpr (LAYER) {
            x[q][h] = L.x_fwd(q, h, x[q][h], cxn, dx, D1);
            y[q][h] = L.y_fwd(sR, w * Q + q, q, h, y[q][h], cy, dy, D2);
          } else {
            x[q][h] = fmadd(x[q][h], cxn, D1);
            y[q][h] = fmadd(y[q][h], cy, D2);
          }
        }
        if constexpr (SP)
          if (mon) sp.monitor(t, p, q, n, e[q]);
      }
      sU[(w + 1) * 32 + lane] = Two{y[Q - 1][0], y[Q - 1][1]};
      __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!p.row_in_tile(t, q)) continue;
      p.store(t, t.tmp[0], q, e[q]);
      p.store(t, t.tmp[1], q, x[q]);
      p.store(t, t.tmp[2], q, y[q]);
    }
    if constexpr (LAYER) L.store(t, p, t.tmp + 3);
  };
  tb_dispatch<false>(tile, steps);
}

// Adjoint steps n0 + nsub down to n0 + 1 of one tile (the transposes of
// k_tmz_ah / k_tmz_ae, same order), the field adjoints from t.l to
// t.tmp[0..2]; the gradient of step n uses hist slot n - step0 - 1.  The
// psi adjoints are read from buffer rb and written to the other one, so no
// block overwrites what another still reads (adjoint_blocked chooses rb so
// that a call leaves them where the one-step kernels' step-parity
// convention expects them).
//
// Per step: H-side sources, the curl weights w1, w2 of every Hx / Hy point,
// lambda_E gathering them, E-side sources, the curl weights v1, v2 of every Ez
// point and the gradient, lambda_X / lambda_Y gathering those.  The weights of
// the neighbour along j come by a shuffle, those along i from the lane or the
// next warp's row (w2 of its last row, v1 of its first).
//
// What no kernel of the chain writes is read before the wait for the launch
// before: the tile's record and, in special and general tiles, the map and the
// first step's seeds and increments.  Adjoint of 200x200 x 3, 100 steps, ms: all
// after the wait 0.59, so 0.52.
template <class P, int Q>
__global__ void __launch_bounds__(kTbThreads, 2)
    k_tmz_tb_adj(const GridDev g, const TmzDev t, int n0, int nsub, int step0, int rb) {
  release_next();
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  using Two = Row2<R>;
  extern __shared__ __align__(16) unsigned char tb_smem[];
  const TbTile<R> tile =
      static_cast<const TbTile<R>*>(t.tiles)[TbBlock(t).tile];
  // (an absorbing tile with sources, monitor or design pixels takes the
  // general form here: 22 us per launch of a 128 x 123 lattice against 36 in
  // registers, which spill)
  if (tile.kind == kTbGeneral || (tile.kind == kTbBoth && tile.fancy)) {
    tb_general_adj<P, Q>(g, t, n0, nsub, step0, rb, tb_smem);
    return;
  }
  Two* const sU = reinterpret_cast<Two*>(tb_smem);        // w2 of the last rows
  Two* const sD = sU + (kTbWarps + 1) * kTbRJ / 2;        // v1 of the first rows
  R* const sR = reinterpret_cast<R*>(tb_smem) + G::kRows;
  const TbPlace<P, Q> p(t);
  const int lane = p.lane, w = p.warp;
  R e[Q][2], x[Q][2], y[Q][2];
  auto load = [&] {
    after_previous();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      p.load(t, t.l[0], q, e[q]);
      p.load(t, t.l[1], q, x[q]);
      p.load(t, t.l[2], q, y[q]);
    }
  };
  if (!tile.fancy) load();  // a special tile has more to do first
  if (w == 0) sU[lane] = Two{P::zero(), P::zero()};
  if (w == kTbWarps - 1) sD[kTbWarps * 32 + lane] = Two{P::zero(), P::zero()};
  constexpr unsigned kAll = 0xffffffffu;
  const R cxn = tile.c[2], cy = tile.c[3], de = tile.d[0], dx = tile.d[1], dy = tile.d[2];
  const bool design = tile.any & kTmzDesign, mon = tile.any & kTmzMonitor;
  const bool src = tile.any & kTmzSrcE;
  auto steps = [&](auto form) {
    constexpr int KIND = decltype(form)::kind;
    constexpr bool LAYER = KIND != kTbPlain, SP = decltype(form)::fancy;
    TbCoef<P, Q, SP> cf;
    TbLayer<P, Q, KIND> L;
    TbSpecial<P, Q> sp;
    cf.load(t, p);
    if constexpr (SP) {
      sp.init(tb_smem);
      sp.load(t, p, tile);
    }
    // the seeds and increments of step n, fetched a step ahead
    auto fetch = [&](int n) {
      if constexpr (SP) {
        if (design) sp.grad_fetch(t, p, n - step0 - 1);
        if (mon) sp.seed_fetch(g, t, p, n);
      }
    };
    fetch(n0 + nsub);
    if constexpr (SP) {
      load();
      if (design) sp.grad_load(t, p);
    }
    if constexpr (LAYER) {
      L.load(t, p, t.phi[rb]);
      L.fill(g, t, p, tile, sR);
      __syncthreads();
      L.columns(sR, lane);
    }
    // w2 of every point (a layer row's advance its psi adjoint)
    R ya[Q][2];
    auto hside = [&]() {
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if constexpr (LAYER)
            ya[q][h] = L.y_adj(sR, w * Q + q, q, h, y[q][h], cy, dy);
          else
            ya[q][h] = cy * y[q][h];
        }
      sU[(w + 1) * 32 + lane] = Two{ya[Q - 1][0], ya[Q - 1][1]};
    };
    hside();
    __syncthreads();
    for (int s = nsub - 1; s >= 0; --s) {
      const int n = n0 + s + 1;
      const Two up = sU[w * 32 + lane];
      R u[2] = {up.a, up.b};
      R v1[Q][2], v2[Q][2];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        R wx[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if constexpr (LAYER)
            wx[h] = L.x_adj(q, h, x[q][h], cxn, dx);
          else
            wx[h] = cxn * x[q][h];
        }
        const R wl = __shfl_up_sync(kAll, wx[1], 1);
        if constexpr (SP)
          if (mon) sp.seed(q, e[q]);
        e[q][0] = e[q][0] + ((wl - wx[0]) + (u[0] - ya[q][0]));
        e[q][1] = e[q][1] + ((wx[0] - wx[1]) + (u[1] - ya[q][1]));
        u[0] = ya[q][0];
        u[1] = ya[q][1];
        if constexpr (SP)
          if (src) sp.zero(p, q, e[q]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          R c1, c2n;
          cf.get(tile, q, h, c1, c2n);
          if constexpr (LAYER) {
            L.e_adj(sR, w * Q + q, q, h, e[q][h], c1, c2n, SP ? c1 : de, v1[q][h], v2[q][h]);
          } else {
            v1[q][h] = c1 * e[q][h];
            v2[q][h] = c2n * e[q][h];
          }
        }
        if constexpr (SP)
          if (design) sp.grad_add(p, q, e[q]);
      }
      if (s > 0) fetch(n - 1);
      sD[w * 32 + lane] = Two{v1[0][0], v1[0][1]};
      __syncthreads();
      const Two dn = sD[(w + 1) * 32 + lane];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const R vr = __shfl_down_sync(kAll, v2[q][0], 1);
        const R d0 = q + 1 < Q ? v1[q + 1 < Q ? q + 1 : q][0] : dn.a;
        const R d1 = q + 1 < Q ? v1[q + 1 < Q ? q + 1 : q][1] : dn.b;
        x[q][0] = x[q][0] + (v2[q][0] - v2[q][1]);
        x[q][1] = x[q][1] + (v2[q][1] - vr);
        y[q][0] = y[q][0] + (v1[q][0] - d0);
        y[q][1] = y[q][1] + (v1[q][1] - d1);
      }
      if (s > 0) hside();
      __syncthreads();
    }
    if constexpr (SP)
      if (design) sp.grad_store(t, p);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!p.row_in_tile(t, q)) continue;
      p.store(t, t.tmp[0], q, e[q]);
      p.store(t, t.tmp[1], q, x[q]);
      p.store(t, t.tmp[2], q, y[q]);
    }
    if constexpr (LAYER) L.store(t, p, t.phi[rb ^ 1]);
  };
  tb_dispatch<true>(tile, steps);
}

// What each tile is (TbTile), one block per tile; after k_tmz_map.
template <class P, int Q>
__global__ void __launch_bounds__(kTbThreads) k_tmz_tiles(const TmzDev t) {
  using R = typename P::R;
  using G = TbGeom<P, Q>;
  constexpr unsigned plain = kTmzPlainE | kTmzPlainX | kTmzPlainY;
  constexpr unsigned rowbits = kTmzOnE1 | kTmzOnY, colbits = kTmzOnE2 | kTmzOnX;
  constexpr unsigned layer = rowbits | colbits | kTmzPsiE | kTmzPsiX | kTmzPsiY;
  constexpr unsigned pmbits = 3u << kTmzPmlE | 3u << kTmzPmlX | 3u << kTmzPmlY;
  __shared__ unsigned any_s;
  __shared__ int same_s, vary_s, first_s[7], pm_s;
  if (threadIdx.x == 0) {
    any_s = 0;
    same_s = 1;
    vary_s = 0;
    pm_s = -1;
    for (int k = 0; k < 7; ++k) first_s[k] = -1;
  }
  __syncthreads();
  const int cols = (t.ny + kTbTJ - 1) / kTbTJ;
  const int ri0 = (int)blockIdx.x / cols * G::TI - kTbHalo;
  const int rj0 = (int)blockIdx.x % cols * kTbTJ - kTbHalo;
  auto at = [&](int a, int c) {
    return (int64_t)wrap_index(ri0 + a, t.nx) * t.ny + wrap_index(rj0 + c, t.ny);
  };
  // coefficient k of a point, one of: plain c1, c2n, cx, cy; absorbing cdt of
  // Ez, Hx, Hy
  auto holds = [&](unsigned f, int k) {
    constexpr unsigned bit[7] = {kTmzPlainE, kTmzPlainE, kTmzPlainX, kTmzPlainY,
                                 kTmzPsiE,   kTmzPsiX,   kTmzPsiY};
    return (f & bit[k]) != 0;
  };
  auto coef = [&](int64_t ll, int k) {
    return P::ldc(map_coef<P>(t, k < 4 ? k : (k == 4 ? 0 : k - 3)) + ll);
  };
  unsigned any = 0;
  int first[7] = {-1, -1, -1, -1, -1, -1, -1}, pm_any = -1;
  for (int q = threadIdx.x; q < G::NP; q += kTbThreads) {
    const unsigned f = __ldg(t.pflags + at(q / kTbRJ, q % kTbRJ));
    any |= f;
    for (int k = 0; k < 7; ++k)
      if (holds(f, k)) first[k] = q;  // any point that has one will do
    if (f & kTmzPsiE) pm_any = f >> kTmzPmlE & 3;
    if (f & kTmzPsiX) pm_any = f >> kTmzPmlX & 3;
    if (f & kTmzPsiY) pm_any = f >> kTmzPmlY & 3;
  }
  any = __reduce_or_sync(0xffffffffu, any);
  pm_any = __reduce_max_sync(0xffffffffu, pm_any);
  for (int k = 0; k < 7; ++k) first[k] = __reduce_max_sync(0xffffffffu, first[k]);
  if ((threadIdx.x & 31) == 0) {
    atomicOr(&any_s, any);
    atomicMax(&pm_s, pm_any);
    for (int k = 0; k < 7; ++k) atomicMax(&first_s[k], first[k]);
  }
  __syncthreads();
  R c[7];
  for (int k = 0; k < 7; ++k)
    c[k] = first_s[k] < 0 ? P::zero() : coef(at(first_s[k] / kTbRJ, first_s[k] % kTbRJ), k);
  const unsigned pm = pm_s < 0 ? 0u : (unsigned)pm_s;
  constexpr unsigned specials =
      kTmzSrcE | kTmzMonitor | kTmzDesign | ~((1u << kTmzPlace) - 1);
  bool same = (any_s & ~(plain | layer | pmbits | specials)) == 0, even = true;
  for (int q = threadIdx.x; q < G::NP && same; q += kTbThreads) {
    const int a = q / kTbRJ, cc = q % kTbRJ;
    const int64_t ll = at(a, cc);
    const unsigned f = __ldg(t.pflags + ll) & ~specials;
    const unsigned row = __ldg(t.pflags + at(a, 0)), col = __ldg(t.pflags + at(0, cc));
    // absorbing exactly where the row or the column is on, plain elsewhere
    const unsigned on = (row & rowbits) | (col & colbits);
    unsigned want = on;
    want |= (on & (kTmzOnE1 | kTmzOnE2)) ? kTmzPsiE | pm << kTmzPmlE : kTmzPlainE;
    want |= (on & kTmzOnX) ? kTmzPsiX | pm << kTmzPmlX : kTmzPlainX;
    want |= (on & kTmzOnY) ? kTmzPsiY | pm << kTmzPmlY : kTmzPlainY;
    same = f == want;
    for (int k = 0; k < 7; ++k)
      if (holds(f, k) && coef(ll, k) != c[k]) {
        if (k < 2 || k == 4)
          even = false;  // Ez
        else
          same = false;
      }
  }
  if (!same) same_s = 0;
  if (!even || (any_s & kTmzDesign)) vary_s = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    TbTile<R> o;
    o.any = any_s;
    const bool rows = any_s & rowbits, cols = any_s & colbits;
    o.fancy = vary_s || (any_s & specials);
    o.kind = rows ? (cols ? kTbBoth : kTbRows) : (cols ? kTbCols : kTbPlain);
    if (o.kind != kTbPlain && o.fancy) o.kind = kTbBoth;  // one form for these
    if (!same_s) o.kind = kTbGeneral;
    o.pm = (int)pm;
    for (int k = 0; k < 4; ++k) o.c[k] = c[k];
    for (int k = 0; k < 3; ++k) o.d[k] = c[4 + k];
    static_cast<TbTile<R>*>(t.tiles)[blockIdx.x] = o;
  }
}

template <class P, int Q>
unsigned tb_tiles(const TmzDev& t) {
  using G = TbGeom<P, Q>;
  return (unsigned)((t.ny + kTbTJ - 1) / kTbTJ) * (unsigned)((t.nx + G::TI - 1) / G::TI);
}

// ---------------------------------------------------------------------------
// Setup and objective.
// ---------------------------------------------------------------------------
// Design coefficients in FP64, formed exactly as a dielectric class's
// (dt / eps, then / dx and / dy).
__global__ void k_tmz_design(const GridDev g, const TmzDev t, const double* eps) {
  const int64_t nd = (int64_t)t.dn[0] * t.dn[1];
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nd * t.nb) return;
  const double e = eps[k];
  const double cdt = g.dt / e;
  DesignCoef d;
  d.c1 = make_coef(cdt / g.dr[0]);
  d.c2 = make_coef(cdt / g.dr[1]);
  d.neg_reps = -1.0 / e;
  d.eps = e;
  const_cast<DesignCoef*>(t.dc)[k] = d;
}

// J[b] = dt * sum over the first nsteps monitor rows of E^2, one block per
// design, fixed summation order (deterministic).
__global__ void k_tmz_objective(const GridDev g, const TmzDev t, int nsteps, double* J) {
  __shared__ double part[256];
  const int b = blockIdx.x;
  const int64_t nm = (int64_t)t.mn[0] * t.mn[1];
  const int64_t count = (int64_t)nsteps * nm;
  const double* mon = t.mon + (int64_t)b * t.total_steps * nm;
  double s = 0.0;
  for (int64_t k = threadIdx.x; k < count; k += blockDim.x) s += mon[k] * mon[k];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) J[b] = g.dt * part[0];
}

dim3 lattice_grid(const TmzDev& t) {
  return dim3((unsigned)((t.ny + kBX - 1) / kBX), (unsigned)((t.nx + kBY - 1) / kBY),
              (unsigned)t.nb);
}

// Blocks of a chunk kernel and its index quotients.
template <class K>
cudaError_t chunk_shape(K* kernel, const TmzDev& t, LatDiv& d, int& blocks) {
  int per_sm = 0;
  const cudaError_t e =
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kChunkThreads, 0);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int64_t groups = (t.plane * t.nb + 31) / 32, sms = sm_count();
  // one block per SM while its warps take at most one group each
  const int64_t most = groups <= sms * (kChunkThreads / 32) ? sms : sms * per_sm;
  blocks = (int)(groups < most ? groups : most);
  tile_div_of((uint32_t)t.plane, d.m_plane, d.s_plane);
  tile_div_of((uint32_t)t.ny, d.m_row, d.s_row);
  return cudaSuccess;
}

// A call's sources: looked up in the bodies (u.nsrc > 0; their points are named
// as they are now: a caller may have set others since the design), or a list.
SourceList one_step_sources(TmzDev& u, cudaStream_t s) {
  SourceList l = {u.src, u.src_val, 0};
  if (u.nsrc > kTmzLookUp) {
    l.n = u.nsrc;
    u.nsrc = 0;
  } else if (u.nsrc > 0) {
    k_tmz_map_sources<<<(u.nsrc + 127) / 128, 128, 0, s>>>(u);
  }
  return l;
}

template <class K, class... A>
cudaError_t launch_chunk(K* kernel, const GridDev& g, const TmzDev& t, const SourceList& l,
                         const Meeting& meet, cudaStream_t s, A... steps) {
  LatDiv d;
  int blocks = 0;
  const cudaError_t e = chunk_shape(kernel, t, d, blocks);
  if (e != cudaSuccess) return e;
  int* error = wait_error_word();
  void* args[] = {(void*)&g, (void*)&t, &d, (void*)&l, (void*)&meet, &steps..., &error};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)blocks),
                                     dim3(kChunkThreads), args, 0, s);
}

template <class P>
cudaError_t forward(const GridDev& g, const TmzDev& t, const Meeting& meet, int step0, int nsteps,
                    int flags, cudaStream_t s) {
  if (nsteps <= 0) return cudaSuccess;
  TmzDev u = t;
  const SourceList l = one_step_sources(u, s);
  if (meet.at != nullptr) {
    const cudaError_t e = launch_chunk(k_tmz_chunk_fwd<P>, g, u, l, meet, s, step0, nsteps, flags);
    if (!no_room(e)) return e;
    (void)cudaGetLastError();
  }
  const dim3 grid = lattice_grid(t), block(kBX, kBY);
  const dim3 entries((unsigned)(((int64_t)l.n * t.nb + 127) / 128));
  for (int k = 0; k < nsteps; ++k) {
    const int n = step0 + k + 1;
    launch_after(k > 0, k_tmz_fe<P>, grid, block, 0, s, g, u, n,
                 (flags & GMES_TMZ_RECORD_HIST) ? k : -1);
    if (l.n > 0) launch_after(true, k_tmz_src<P>, entries, 128, 0, s, u, l, 0, n);
    launch_after(true, k_tmz_fh<P>, grid, block, 0, s, g, u, n,
                 (flags & GMES_TMZ_RECORD_MONITOR) ? n - 1 : -1);
    if (l.n > 0) launch_after(true, k_tmz_src<P>, entries, 128, 0, s, u, l, 1, n);
  }
  return cudaGetLastError();
}

template <class P>
cudaError_t adjoint(const GridDev& g, const TmzDev& t, const Meeting& meet, int step0, int nsteps,
                    cudaStream_t s) {
  if (nsteps <= 0) return cudaSuccess;
  TmzDev u = t;
  const SourceList l = one_step_sources(u, s);
  if (meet.at != nullptr) {
    const cudaError_t e = launch_chunk(k_tmz_chunk_adj<P>, g, u, l, meet, s, step0, nsteps);
    if (!no_room(e)) return e;
    (void)cudaGetLastError();
  }
  const dim3 grid = lattice_grid(t), block(kBX, kBY);
  const dim3 entries((unsigned)(((int64_t)l.n * t.nb + 127) / 128));
  bool early = false;
  for (int k = nsteps - 1; k >= 0; --k) {
    const int n = step0 + k + 1;
    const int rb = n & 1, wb = rb ^ 1;
    if (l.n > 0) launch_after(early, k_tmz_adj_src<P>, entries, 128, 0, s, u, l, 1);
    launch_after(early || l.n > 0, k_tmz_ah<P>, grid, block, 0, s, g, u, n, rb, wb);
    if (l.n > 0) launch_after(true, k_tmz_adj_src<P>, entries, 128, 0, s, u, l, 0);
    launch_after(true, k_tmz_ae<P>, grid, block, 0, s, g, u, k, rb, wb);
    early = true;
  }
  return cudaGetLastError();
}

// The blocked kernels read one copy of the state and write the other, so
// the launches alternate between the state and its scratch copy; with an
// odd number of launches the state is first copied to the scratch, so that
// the last launch writes the state.
void swap_fields(TmzDev& u) {  // forward: state <-> scratch
  for (int k = 0; k < kTmzState; ++k) {
    void* f = u.f[k];
    u.f[k] = u.tmp[k];
    u.tmp[k] = f;
  }
}

void swap_adjoints(TmzDev& u) {  // adjoint: field adjoints <-> scratch
  for (int k = 0; k < 3; ++k) {
    void* l = u.l[k];
    u.l[k] = u.tmp[k];
    u.tmp[k] = l;
  }
}

cudaError_t copy_state(void* const* dst, void* const* src, int n, int64_t bytes, cudaStream_t s) {
  for (int k = 0; k < n; ++k) {
    const cudaError_t e = cudaMemcpyAsync(dst[k], src[k], (size_t)bytes, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Rows per warp of the blocked kernels: regions of 32 x 64 points.  Measured on
// GB300 (512^2 x 64 designs, 200 steps, forward / adjoint ms, 512 threads at 64
// registers): 2 rows 12.8 / 16.2, 3 rows 12.1 / 21.8 (the adjoint spills); 256
// threads at 128 registers, 4 rows 15.9 / 18.0, 6 rows 17.2 / 30.0.
constexpr int kTbQ = 2;

// Shared memory of a launch of `blocks` blocks that need `bytes` each, at most
// kTbSmemMost.  A launch that one block per SM holds asks for more than half an
// SM: with the next launch's blocks coming up beside it, the SMs left over would
// otherwise take two of its blocks, and the slowest tile sets its time.  Measured
// on GB300, 100 steps forward / adjoint ms (plain launches of the kernels before |
// overlapped | overlapped, one block per SM):
//   100x100 x 12   0.724 / 0.541   0.739 / 0.595   0.636 / 0.447
//   128x123 x 8    0.732 / 0.513   0.653 / 0.568   0.580 / 0.433
//   200x200 x 3    0.675 / 0.566   0.578 / 0.517   0.563 / 0.462
constexpr size_t kTbSmemMost = 116 * 1024;
size_t launch_smem(size_t bytes, unsigned blocks) {
  return blocks <= (unsigned)sm_count() ? kTbSmemMost : bytes;
}

template <class P, int Q>
cudaError_t forward_blocked(const GridDev& g, const TmzDev& t, int step0, int nsteps, int flags,
                            int per_launch, cudaStream_t s) {
  const unsigned grid = tb_tiles<P, Q>(t) * (unsigned)t.nb;
  static_assert(TbGeom<P, Q>::fwd_bytes <= kTbSmemMost, "the attribute below");
  const size_t smem = launch_smem(TbGeom<P, Q>::fwd_bytes, grid);
  cudaError_t e = cudaFuncSetAttribute(k_tmz_tb_fwd<P, Q>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTbSmemMost);
  if (e != cudaSuccess) return e;
  if (t.tmp[0] == nullptr) return cudaErrorInvalidValue;
  const int launches = (nsteps + per_launch - 1) / per_launch;
  TmzDev u = t;
  if (launches % 2 == 1) {
    e = copy_state(t.tmp, t.f, kTmzState, (int64_t)t.nb * t.plane * (int64_t)sizeof(typename P::T), s);
    if (e != cudaSuccess) return e;
    swap_fields(u);
  }
  for (int k = 0; k < nsteps; k += per_launch) {
    const int m = nsteps - k < per_launch ? nsteps - k : per_launch;
    launch_after(k > 0, k_tmz_tb_fwd<P, Q>, dim3(grid), kTbThreads, smem, s, g, u, step0 + k, m,
                 (flags & GMES_TMZ_RECORD_HIST) ? k : -1,
                 (flags & GMES_TMZ_RECORD_MONITOR) ? 1 : 0);
    swap_fields(u);
  }
  return cudaGetLastError();
}

// Launches of the blocked adjoint for nsteps steps of at most per_launch
// each.  Each launch reads the psi adjoints from one buffer and writes the
// other; a call starts from the buffer the one-step kernels' step n0 + nsteps
// reads ((n0 + nsteps) & 1) and must end in the one step n0 + 1 writes
// (n0 & 1), so the number of launches has the parity of nsteps: the fewest
// launches of that parity, their step counts as even as possible.  (Odd
// step counts per launch, the earlier rule, capped launches at 3 steps
// against the forward's 4.)
int adj_launches(int nsteps, int per_launch) {
  int k = (nsteps + per_launch - 1) / per_launch;
  if ((k & 1) != (nsteps & 1)) ++k;
  return k < nsteps ? k : nsteps;
}

template <class P, int Q>
cudaError_t adjoint_blocked(const GridDev& g, const TmzDev& t, int step0, int nsteps,
                            int per_launch, cudaStream_t s) {
  const unsigned grid = tb_tiles<P, Q>(t) * (unsigned)t.nb;
  static_assert(TbGeom<P, Q>::adj_bytes <= kTbSmemMost, "the attribute below");
  const size_t smem = launch_smem(TbGeom<P, Q>::adj_bytes, grid);
  cudaError_t e = cudaFuncSetAttribute(k_tmz_tb_adj<P, Q>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTbSmemMost);
  if (e != cudaSuccess) return e;
  if (t.tmp[0] == nullptr) return cudaErrorInvalidValue;
  if (nsteps <= 0) return cudaSuccess;
  const int launches = adj_launches(nsteps, per_launch);
  TmzDev u = t;
  if (launches % 2 == 1) {
    e = copy_state(t.tmp, t.l, 3, (int64_t)t.nb * t.plane * (int64_t)sizeof(typename P::T), s);
    if (e != cudaSuccess) return e;
    swap_adjoints(u);
  }
  int rb = (step0 + nsteps) & 1;
  int hi = nsteps;
  for (int q = 0; q < launches; ++q) {
    // launch q takes an even share of the steps left
    const int m = (hi + (launches - q) - 1) / (launches - q);
    launch_after(q > 0, k_tmz_tb_adj<P, Q>, dim3(grid), kTbThreads, smem, s, g, u,
                 step0 + hi - m, m, step0, rb);
    swap_adjoints(u);
    rb ^= 1;
    hi -= m;
  }
  return cudaGetLastError();
}

// Steps per launch for a precision and the caller's request (0: default).
// (The blocked kernels' source maps hold 15-bit source numbers.)
int steps_per_launch(int precision, const TmzDev& t, int requested) {
  if (precision != GMES_FP32 || t.nsrc >= (int)kTbHard - 1) return 1;
  if (requested <= 0) return kTbHalo;
  return requested < kTbHalo ? requested : kTbHalo;
}

}  // namespace

cudaError_t launch_tmz_design(int precision, const GridDev& g, const TmzDev& t,
                              const double* eps, cudaStream_t s) {
  const int64_t n = (int64_t)t.dn[0] * t.dn[1] * t.nb;
  if (n > 0) k_tmz_design<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, t, eps);
  const unsigned mblocks = (unsigned)((t.plane + 255) / 256);
  switch (precision) {
    case GMES_FP64:
      k_tmz_map<PolF64><<<mblocks, 256, 0, s>>>(g, t);
      break;
    case GMES_FP32:
      k_tmz_map<PolF32><<<mblocks, 256, 0, s>>>(g, t);
      break;
    case GMES_DF64:
      k_tmz_map<PolDF><<<mblocks, 256, 0, s>>>(g, t);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  if (t.nsrc > 0) k_tmz_map_sources<<<(t.nsrc + 127) / 128, 128, 0, s>>>(t);
  if (precision == GMES_FP32)
    k_tmz_tiles<PolF32, kTbQ><<<tb_tiles<PolF32, kTbQ>(t), kTbThreads, 0, s>>>(t);
  return cudaGetLastError();
}

bool tmz_chunked(int precision, const TmzDev& t, int block_steps) {
  return steps_per_launch(precision, t, block_steps) == 1 && wait_error_word() != nullptr &&
         (int64_t)t.nsrc * t.nb < (int64_t(1) << 31) &&
         t.plane * t.nb <= (precision == GMES_DF64 ? kChunkPointsDf : kChunkPoints);
}

int64_t tmz_launches(int precision, const TmzDev& t, int block_steps, int nsteps, bool adj) {
  const int per = steps_per_launch(precision, t, block_steps);
  if (nsteps <= 0) return 0;
  if (per > 1) return adj ? adj_launches(nsteps, per) : (nsteps + per - 1) / per;
  const bool list = t.nsrc > kTmzLookUp, named = t.nsrc > 0 && !list;
  if (tmz_chunked(precision, t, block_steps)) return named + 1;
  return named + (list ? 4 : 2) * (int64_t)nsteps;
}

cudaError_t launch_tmz_forward(int precision, const GridDev& g, const TmzDev& t,
                               const Meeting& meet, int step0, int nsteps, int flags,
                               int block_steps, cudaStream_t s) {
  const int per = steps_per_launch(precision, t, block_steps);
  switch (precision) {
    case GMES_FP64:
      return forward<PolF64>(g, t, meet, step0, nsteps, flags, s);
    case GMES_FP32:
      if (per > 1)
        return forward_blocked<PolF32, kTbQ>(g, t, step0, nsteps, flags, per, s);
      return forward<PolF32>(g, t, meet, step0, nsteps, flags, s);
    case GMES_DF64:
      return forward<PolDF>(g, t, meet, step0, nsteps, flags, s);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_tmz_adjoint(int precision, const GridDev& g, const TmzDev& t,
                               const Meeting& meet, int step0, int nsteps, int block_steps,
                               cudaStream_t s) {
  const int per = steps_per_launch(precision, t, block_steps);
  switch (precision) {
    case GMES_FP64:
      return adjoint<PolF64>(g, t, meet, step0, nsteps, s);
    case GMES_FP32:
      if (per > 1)
        return adjoint_blocked<PolF32, kTbQ>(g, t, step0, nsteps, per, s);
      return adjoint<PolF32>(g, t, meet, step0, nsteps, s);
    case GMES_DF64:
      return adjoint<PolDF>(g, t, meet, step0, nsteps, s);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_tmz_objective(const GridDev& g, const TmzDev& t, int nsteps, double* J,
                                 cudaStream_t s) {
  k_tmz_objective<<<(unsigned)t.nb, 256, 0, s>>>(g, t, nsteps, J);
  return cudaGetLastError();
}

}  // namespace gmes
