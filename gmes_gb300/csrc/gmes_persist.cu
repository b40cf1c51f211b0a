// A chunk of time steps of one small grid in one launch.
//
// A small grid's step is bound by its launches: six dependent kernels (ghost
// copy, cell update and sources of each half) of 2-3 us each, whatever they
// compute.  Here the whole chunk is one cooperative launch that walks the steps
// with one grid-wide barrier after each half; the thread that updates a point
// also writes its ghost images, and its block applies its point sources, so a
// half needs no further phase.  What then bounds a half-step, measured on GB300
// (200^2 TMz, FP64, us per step): two barriers 2.8 (1.4 each: the stores reach
// L2, one atomic, one poll), and in between the longest chain of dependent
// loads and the FP64 pipe of the SM with most work:
//   six launches per step                                  15.4
//   one launch, k_cell's cell body, blocks of contiguous
//   cells                                                   8.4
//   tables in shared memory for class ids, coefficients
//   and profiles                                            7.8
//   the same number of cells on every SM                    7.1
//   cells dealt to the blocks in groups of 32 (absorbing
//   layer and media spread over the SMs)                    6.9
//   one component per warp and group instead of three       6.1
// (48x40x44 cells in 3-D: 22.9, 22.1, 24.0, 20.6, 18.9, 13.0.)  Blocks of 256
// threads (4 per SM) ran 6.6 / 15.0, 1024 threads (1 per SM) 6.5 / 13.5, three
// blocks of 512 (40 registers) 6.6 / 13.4.
//
// The ghost planes are left as FDTD.step leaves them (gmes/fdtd.py:1099-1122):
// E's hold the present values, H's those from before the last E half.  A point
// source on a ghost point only shows until the next ghost copy, so it is
// applied only where that copy does not follow: an H source in the last step.
#include <cstring>

#include "gmes_barrier.cuh"
#include "gmes_cell.cuh"

namespace gmes {
namespace {

#ifndef GMES_PERSIST_THREADS
#define GMES_PERSIST_THREADS 512
#endif
constexpr int kPersistThreads = GMES_PERSIST_THREADS;
constexpr int kPersistSources = 64;  // point sources a grid may have here

// Tables that a block keeps in shared memory for the whole chunk, so that a
// cell's update waits for one round trip to L2 (its field and psi values)
// instead of a chain of them (class id, class, profile, psi): the class ids of
// its cells, the plain-form coefficients of the first kTabClasses classes of
// each component and the CPML profiles of the first PML layer.  Cells of other
// kinds, classes or layers take the general path.
constexpr int kTabClasses = 32;
template <class R>
struct alignas(16) TabClass {
  R c1, c2, cdt;
  int kind;  // -1: not in the tables' reach
};
// Byte offsets: class table; per component its ids and, for its two transverse
// axes, the profile's b, c/d, 1/(kappa d) as rows of prof_n values, then flags.
struct TabLayout {
  int cls[6], ids[6], prof[6][2], prof_n[6][2];
  int bytes;
};
enum : int { kProfOn = 1, kProfKappa = 2 };

struct PersistCfg {
  int cells;
  uint32_t m_row, m_plane; // quotients of a cell index (tile_quot)
  int s_row, s_plane;
  int nsteps, st0;
  Meeting meet;
  TabLayout tab;
};

// One axis' profile entry of a point.
template <class P>
struct TabProf {
  using R = typename P::R;
  const unsigned char* base;
  int n, at;
  __device__ __forceinline__ R cf(int m) const {  // 0: b, 1: c / d, 2: 1 / (kappa d)
    return reinterpret_cast<const R*>(base)[m * n + at];
  }
  __device__ __forceinline__ int flags() const { return base[3 * n * sizeof(R) + at]; }
};

// The CPML part of a point of component C: which slabs are on and its psi
// values there (psi stays zero elsewhere).
template <class P, int C>
struct TabPsi {
  using R = typename P::R;
  using T = typename P::T;
  static constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  static constexpr bool E = C < 3;
  TabProf<P> q1, q2;
  int f1, f2;
  R s1, s2;
  __device__ __forceinline__ void load(const GridDev& g, const unsigned char* sm,
                                       const TabLayout& L, bool cpml, const int x[3], int lin) {
    q1 = {sm + L.prof[C][0], L.prof_n[C][0], x[a1]};
    q2 = {sm + L.prof[C][1], L.prof_n[C][1], x[a2]};
    f1 = cpml ? q1.flags() : 0;
    f2 = cpml ? q2.flags() : 0;
    const T* aux = static_cast<const T*>(g.aux[C]);
    s1 = s2 = P::zero();
    if (f1 & kProfOn) s1 = P::ldw(aux + lin);
    if (f2 & kProfOn) s2 = P::ldw(aux + (int)g.npts[C] + lin);
  }
  // update_fast's and cpml_separate's arithmetic, term for term
  template <int MASK>
  __device__ __forceinline__ void update(const GridDev& g, const TabClass<R>& q, int lin, R F,
                                         R p1, R p2, bool valid) {
    const bool on1 = f1 & kProfOn, on2 = f2 & kProfOn;
    R t = plain_upd<E>(F, q.c1, q.c2, p1, p2);
    if (__any_sync(0xffffffffu, on1 || on2)) {
      T* aux = static_cast<T*>(g.aux[C]);
      bool scaled = true;
      if constexpr (SharedCpml<P>::value) scaled = f1 == kProfOn || f2 == kProfOn;
      R n1 = s1, n2 = s2;
      if (on1) {
        n1 = step(scaled, q1.cf(0), s1, q1.cf(1), p1);
        if (valid) P::st(aux + lin, n1);
      }
      if (on2) {
        n2 = step(scaled, q2.cf(0), s2, q2.cf(1), p2);
        if (valid) P::st(aux + (int)g.npts[C] + lin, n2);
      }
      if (scaled && (on1 || on2)) {
        const R X = madd(-q2.cf(2), p2, madd(q1.cf(2), p1, n1 - n2));
        t = E ? madd(q.cdt, X, F) : madd(-q.cdt, X, F);
      } else if constexpr (SharedCpml<P>::value) {
        if (on1) t = E ? t + q.cdt * n1 : t - q.cdt * n1;
        if (on2) t = E ? t - q.cdt * n2 : t + q.cdt * n2;
      }
    }
    if (valid) P::st(static_cast<T*>(g.f[C]) + lin, t);
  }
  static __device__ __forceinline__ R step(bool scaled, R b, R s, R c, R d) {
    if constexpr (SharedCpml<P>::value)
      if (!scaled) return b * s + c * d;
    return madd(c, d, b * s);
  }
};

// Own point l of component C at cell (i, j, k), and its curl differences.
template <class P, int C, int MASK>
struct Point {
  using R = typename P::R;
  static constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  static constexpr bool E = C < 3;
  int x[3], l;
  __device__ __forceinline__ Point(const GridDev& g, int i, int j, int k)
      : x{i + (!E && own != 0), j + (!E && own != 1), k + (!E && own != 2)},
        l(x[0] * (int)g.fst[own][0] + x[1] * (int)g.fst[own][1] + x[2]) {}
  // component B of the other half at this point's index moved by (si, sj, sk)
  template <int B>
  __device__ __forceinline__ R at(const GridDev& g, int si, int sj, int sk) const {
    const int f0 = (int)g.fst[B % 3][0], f1 = (int)g.fst[B % 3][1];
    return ldf<P, MASK, B>(g, (x[0] + si) * f0 + (x[1] + sj) * f1 + x[2] + sk);
  }
  __device__ __forceinline__ void diffs(const GridDev& g, R& p1, R& p2) const {
    constexpr int B1 = (E ? 3 : 0) + a2, B2 = (E ? 3 : 0) + a1;  // read by D1, D2
    if constexpr (E) {
      // D1 = H_a2[x + own + a1] - H_a2[x + own], D2 = H_a1[x + own + a2] - H_a1[x + own]
      p1 = curl_diff(at<B1>(g, (own == 0) + (a1 == 0), (own == 1) + (a1 == 1), (own == 2) + (a1 == 2)),
                     at<B1>(g, own == 0, own == 1, own == 2));
      p2 = curl_diff(at<B2>(g, (own == 0) + (a2 == 0), (own == 1) + (a2 == 1), (own == 2) + (a2 == 2)),
                     at<B2>(g, own == 0, own == 1, own == 2));
    } else {
      // from x - a1 - a2: D1 = E_a2[. + a1] - E_a2[.], D2 = E_a1[. + a2] - E_a1[.]
      constexpr int o0 = -(own != 0), o1 = -(own != 1), o2 = -(own != 2);
      p1 = curl_diff(at<B1>(g, o0 + (a1 == 0), o1 + (a1 == 1), o2 + (a1 == 2)), at<B1>(g, o0, o1, o2));
      p2 = curl_diff(at<B2>(g, o0 + (a2 == 0), o1 + (a2 == 1), o2 + (a2 == 2)), at<B2>(g, o0, o1, o2));
    }
  }
};

// The update of one point of component C; u: its cell's number in the block's
// tables.  valid: lanes past the grid's last cell repeat it without storing.
template <class P, int C, bool DISP, int MASK>
__device__ __forceinline__ void table_point(const GridDev& g, const unsigned char* sm,
                                            const TabLayout& L, int i, int j, int k, int u,
                                            bool valid) {
  using R = typename P::R;
  using T = typename P::T;
  const Point<P, C, MASK> pt(g, i, j, k);
  const R F = ldf<P, MASK, C>(g, pt.l);
  R p1, p2;
  pt.diffs(g, p1, p2);
  int id, kind = -1;
  const TabClass<R>* cls = reinterpret_cast<const TabClass<R>*>(sm + L.cls[C]);
  if (L.bytes > 0) {
    id = sm[L.ids[C] + u];
    if (id < kTabClasses) kind = cls[id].kind;
  } else {
    id = __ldg(g.cls[C] + pt.l);
  }
  constexpr unsigned kAll = 0xffffffffu;
  if (__all_sync(kAll, kind == GMES_KIND_DIELECTRIC) && !g.pointwise) {
    const R r = plain_mask<MASK, C>(F, cls[id].c1, cls[id].c2, p1, p2);
    if (valid) P::st(static_cast<T*>(g.f[C]) + pt.l, r);
  } else if (__all_sync(kAll, kind == GMES_KIND_DIELECTRIC || kind == GMES_KIND_CPML) &&
             !g.pointwise) {
    TabPsi<P, C> psi;
    psi.load(g, sm, L, kind == GMES_KIND_CPML, pt.x, pt.l);
    psi.template update<MASK>(g, cls[id], pt.l, F, p1, p2, valid);
  } else if (valid) {
    const Pre<P> pre = prefetch_state<P, C>(g, pt.l, pt.x, (uint8_t)id);
    update_fast<P, C, DISP>(g, pt.l, pt.x, p1, p2, F, (uint8_t)id, pre);
  }
}

// table_point and the ghost images of component C of both planes.
template <class P, int C, bool DISP, int MASK, bool CX>
__device__ __forceinline__ void step_point(const GridDev& g, const GridDev& gi,
                                           const unsigned char* sm, const TabLayout& L, int i,
                                           int j, int k, int u, bool valid, bool images,
                                           bool all) {
  table_point<P, C, DISP && C < 3, MASK>(g, sm, L, i, j, k, u, valid);
  if constexpr (CX) table_point<P, C, DISP && C < 3, MASK>(gi, sm, L, i, j, k, u, valid);
  if (images && valid) {
    const Point<P, C, MASK> pt(g, i, j, k);
    const int x[3] = {i, j, k};
    ghost_images<P, C, CX>(g, gi, x, pt.l, all);
  }
}

// A point source owned by this block: its entry and its cell.
struct OwnSource {
  int q, comp, i, j, k;
};

#ifndef GMES_PERSIST_BLOCKS
#define GMES_PERSIST_BLOCKS 2
#endif
template <class P, bool DISP, int MASK, bool CX>
__global__ void __launch_bounds__(kPersistThreads, GMES_PERSIST_BLOCKS)
    k_persist(const __grid_constant__ GridDev g, const __grid_constant__ GridDev gi,
              const __grid_constant__ PersistCfg c, int* error) {
  __shared__ OwnSource own[kPersistSources];
  __shared__ int nown;
  extern __shared__ __align__(16) unsigned char tab[];
  using R = typename P::R;
  const TabLayout& L = c.tab;
  // Groups of 32 cells go round the blocks in turn, so that every SM gets its
  // share of the cells that cost most (absorbing layer, dispersive media): the
  // barrier waits for the slowest SM.  Group v of the block is group
  // blockIdx.x + v gridDim.x of the grid; warp w takes v = w, w + 16, ...
  constexpr int kWarps = kPersistThreads / 32;
  auto meet = [&] {
    if (grid_barrier(c.meet, error)) return true;
    for (int comp = 0; comp < 6; ++comp)
      if ((g.active >> comp) & 1)
        spoil(g.f[comp], g.npts[comp] * (CX ? 2 : 1) * (int64_t)sizeof(typename P::T));
    return false;
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (c.cells + 31) / 32;
  const int mine = (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  auto cell_at = [&](int v) { return (((int)blockIdx.x + v * (int)gridDim.x) << 5) + lane; };
  const int n1 = g.n[1], n2 = g.n[2];
  auto cell_of = [&](int t, int& i, int& j, int& k) {
    i = (int)tile_quot((unsigned)t, c.m_plane, c.s_plane);
    const int r = t - i * n1 * n2;
    j = (int)tile_quot((unsigned)r, c.m_row, c.s_row);
    k = r - j * n2;
  };
  if (threadIdx.x == 0) nown = 0;
  if (L.bytes > 0) {
    for (int q = threadIdx.x; q < 6 * kTabClasses; q += kPersistThreads) {
      const int comp = q / kTabClasses, id = q % kTabClasses;
      if (!((g.active >> comp) & 1)) continue;
      const ClassCoef& cc = g.tab[comp][id];
      TabClass<R> t;
      t.c1 = P::cfg(&cc.c1);
      t.c2 = P::cfg(&cc.c2);
      t.cdt = P::cfg(&cc.cdt);
      t.kind = __ldg(&cc.kind);
      if (t.kind == GMES_KIND_CPML && __ldg(&cc.pml) != 0) t.kind = -1;
      reinterpret_cast<TabClass<R>*>(tab + L.cls[comp])[id] = t;
    }
    for (int comp = 0; comp < 6; ++comp) {
      if (!((g.active >> comp) & 1)) continue;
      for (int h = 0; h < 2 && g.npml > 0; ++h) {
        const int ax = (comp % 3 + 1 + h) % 3, n = L.prof_n[comp][h];
        R* row = reinterpret_cast<R*>(tab + L.prof[comp][h]);
        unsigned char* flags = reinterpret_cast<unsigned char*>(row + 3 * n);
        for (int q = threadIdx.x; q < n; q += kPersistThreads) {
          const Coef* e = g.prof[0][comp][ax] + (int64_t)q * kProfStride;
          row[q] = P::cfg(e);
          row[n + q] = P::cfg(e + 3);
          row[2 * n + q] = P::cfg(e + 4);
          flags[q] = (coef_nonzero(e + 1) ? kProfOn : 0) | (kappa_one(e) ? kProfKappa : 0);
        }
      }
      const int half = comp / 3;
      const int ai = comp % 3;
      for (int v = warp; v < mine; v += kWarps) {
        const int t = cell_at(v);
        if (t >= c.cells) continue;
        int i, j, k;
        cell_of(t, i, j, k);
        if (half) i += ai != 0, j += ai != 1, k += ai != 2;
        tab[L.ids[comp] + v * 32 + lane] =
            __ldg(g.cls[comp] + i * (int)g.st[comp][0] + j * (int)g.st[comp][1] + k);
      }
    }
  }
  __syncthreads();
  // the sources on this block's points; block 0 also takes those on H ghost
  // points (cell -1 along i), which it applies in the last step
  for (int q = threadIdx.x; q < g.nsrc; q += kPersistThreads) {
    const gmes_point_source ps = g.src[q];
    if (ps.comp < 0 || ps.comp > 5 || !((g.active >> ps.comp) & 1)) continue;
    if (ps.offset < 0 || ps.offset >= g.npts[ps.comp]) continue;
    const int side = ps.comp < 3 ? 0 : 1, ax = ps.comp % 3;
    const int s0 = (int)g.st[ps.comp][0], s1 = (int)g.st[ps.comp][1];
    const int off = (int)ps.offset, x = off / s0, y = (off - x * s0) / s1, z = off - x * s0 - y * s1;
    OwnSource o{q, ps.comp, x - (side && ax != 0), y - (side && ax != 1), z - (side && ax != 2)};
    const bool ghost = o.i < 0 || o.j < 0 || o.k < 0 || o.i >= g.n[0] || o.j >= n1 || o.k >= n2;
    if (ghost) o.i = -1;
    const int t = (o.i * n1 + o.j) * n2 + o.k;
    if (ghost ? (side == 1 && blockIdx.x == 0) : (t >> 5) % (int)gridDim.x == (int)blockIdx.x)
      own[atomicAdd(&nown, 1)] = o;
  }
  __syncthreads();
  // the H ghosts of the present fields, which the first E half reads
  for (int v = warp; v < mine; v += kWarps) {
    const int t = cell_at(v);
    if (t >= c.cells) continue;
    int i, j, k;
    cell_of(t, i, j, k);
    ghost_cell<P, 1, MASK, CX>(g, gi, i, j, k, c.nsteps == 1);
  }
  if (!meet()) return;
  for (int st = 0; st < c.nsteps; ++st) {
    const bool last = st + 1 == c.nsteps;
    auto half = [&](auto tag) {
      constexpr int SIDE = decltype(tag)::value;
      // E ghosts always follow; H ghosts of the last step stay as they are
      const bool images = SIDE == 0 || !last;
      const bool all = SIDE == 0 ? last : st + 2 == c.nsteps;
      // items of a warp: one active component of one group of cells
      constexpr int C0 = 3 * SIDE;
      const int act = (MASK ? MASK : g.active) >> C0 & 7, per = __popc(act);
      for (int q = warp; q < mine * per; q += kWarps) {
        const int v = q / per, r = q - v * per;
        const int rest = act & (act - 1);  // without the lowest component
        const int comp = __ffs(r == 0 ? act : (r == 1 ? rest : rest & (rest - 1))) - 1;
        const int tx = cell_at(v);
        const bool valid = tx < c.cells;
        const int t = valid ? tx : c.cells - 1;
        const int u = v * 32 + (valid ? lane : (c.cells - 1) & 31);
        int i, j, k;
        cell_of(t, i, j, k);
        if (is_active<MASK, C0>(g) && comp == 0)
          step_point<P, C0, DISP, MASK, CX>(g, gi, tab, L, i, j, k, u, valid, images, all);
        else if (is_active<MASK, C0 + 1>(g) && comp == 1)
          step_point<P, C0 + 1, DISP, MASK, CX>(g, gi, tab, L, i, j, k, u, valid, images, all);
        else if (is_active<MASK, C0 + 2>(g))
          step_point<P, C0 + 2, DISP, MASK, CX>(g, gi, tab, L, i, j, k, u, valid, images, all);
      }
      if (nown > 0) {
        __syncthreads();
        const OwnSource o = own[threadIdx.x < (unsigned)nown ? threadIdx.x : 0];
        const bool on = (int)threadIdx.x < nown && (o.comp < 3) == (SIDE == 0);
        if (on && (o.i >= 0 || last)) {
          const int64_t slot = 2 * (int64_t)(c.st0 + st) + SIDE;
          source_point<P, false>(g, SIDE, slot, o.q);
          if constexpr (CX) source_point<P, false>(gi, SIDE, slot, o.q);
        }
        __syncthreads();  // sources may share a point
        if (images && on && o.i >= 0) {
          const int x[3] = {o.i, o.j, o.k};
          ghost_own<P, CX>(g, gi, o.comp, x, (int)g.src[o.q].offset);
        }
      }
    };
    half(std::integral_constant<int, 0>{});
    if (!meet()) return;
    if (last) leave_barrier(c.meet);
    half(std::integral_constant<int, 1>{});
    if (!last && !meet()) return;
  }
}

// Shared memory of the tables: at most kTabMost, so that two blocks stay
// resident on an SM; a grid that needs more does without them, and so does a call
// too short to earn what building them takes.  Measured on GB300, us per step of
// calls of 1 / 2 / 4 / 20 steps, six launches per step | tables | none:
//   64^2   FP64  18.9 16.4 15.9 15.2 | 16.7 10.9  8.3  6.1 | 14.5 10.6  8.8  7.2
//   600^2  FP32  29.0 27.2 26.3 25.8 | 27.0 17.7 13.9 10.7 | 22.5 16.6 14.4 12.6
//   900^2  FP64  76.2 73.9 72.8 72.5 | 49.8 36.0 28.3 22.3 | 37.3 28.9 26.5 24.6
//   24^3   df64  20.8 19.6 18.5 17.8 | 22.1 14.5 10.8  7.7 | 16.8 12.4 10.1  8.4
//   32^3   FP32  20.7 18.8 18.1 17.6 | 20.9 13.5  9.9  7.2 | 15.3 11.5  9.3  7.6
// Beyond the tables' reach (every component's axes and cells in kTabMost), calls
// of 20 steps, six launches | none: 1024^2 FP64 88.9 | 43.0, 4096^2 FP64 1266 | 749,
// FP32 766 | 609, df64 950 | 862, 6000x6500 FP32 1761 | 968.
constexpr int kTabMost = 100 * 1024;
constexpr int kTabSteps = 4;

TabLayout table_layout(const GridDev& d, int per, int es, int nsteps) {
  TabLayout L;
  std::memset(&L, 0, sizeof(L));
  if (nsteps < kTabSteps) return L;
  int64_t off = 0;
  for (int c = 0; c < 6; ++c) {
    if (!((d.active >> c) & 1)) continue;
    L.cls[c] = (int)off;
    off += kTabClasses * (es == 8 ? 32 : 16);
    for (int h = 0; h < 2; ++h) {
      const int64_t n = d.sh[c][(c % 3 + 1 + h) % 3];
      L.prof[c][h] = (int)off;
      L.prof_n[c][h] = (int)n;
      off += (3 * n * es + n + 15) / 16 * 16;
    }
    L.ids[c] = (int)off;
    off += (per + 15) / 16 * 16;
    if (off > kTabMost) break;
  }
  L.bytes = off <= kTabMost ? (int)off : 0;
  return L;
}

template <class P, bool DISP, int MASK, bool CX>
cudaError_t launch_one(const Plan& p, const Meeting& meet, int nsteps, int st0, cudaStream_t s) {
  const GridDev& d = p.re;
  auto* kernel = k_persist<P, DISP, MASK, CX>;
  int per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTabMost);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPersistThreads,
                                                    kTabMost);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  PersistCfg c;
  c.cells = d.n[0] * d.n[1] * d.n[2];
  // the same number of cells on every SM: the FP64 pipe of the SM with most
  // cells sets the pace
  const int sms = sm_count();
  const int want = (int64_t)c.cells * 3 <= (int64_t)sms * kPersistThreads ? sms : sms * per_sm;
  const int groups = (c.cells + 31) / 32;
  const int blocks = groups < want ? groups : want;
  const int per = (groups + blocks - 1) / blocks * 32;
  tile_div_of((uint32_t)d.n[2], c.m_row, c.s_row);
  tile_div_of((uint32_t)(d.n[1] * d.n[2]), c.m_plane, c.s_plane);
  c.nsteps = nsteps;
  c.meet = meet;
  c.st0 = st0;
  c.tab = table_layout(d, per, (int)sizeof(typename P::T), nsteps);
  GridDev re = p.re, im = p.im;
  int* error = wait_error_word();
  void* args[] = {&re, &im, &c, &error};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)blocks),
                                     dim3(kPersistThreads), args, (size_t)c.tab.bytes, s);
}

template <class P, bool DISP, bool CX>
cudaError_t launch_mask(const Plan& p, const Meeting& meet, int nsteps, int st0, cudaStream_t s) {
  constexpr int kTMz = 1 << GMES_EZ | 1 << GMES_HX | 1 << GMES_HY;
  constexpr int kTEz = 1 << GMES_EX | 1 << GMES_EY | 1 << GMES_HZ;
  switch (p.re.active) {
    case kTMz:
      return launch_one<P, DISP, kTMz, CX>(p, meet, nsteps, st0, s);
    case kTEz:
      return launch_one<P, DISP, kTEz, CX>(p, meet, nsteps, st0, s);
    case 63:
      return launch_one<P, DISP, 63, CX>(p, meet, nsteps, st0, s);
    default:
      return launch_one<P, DISP, 0, CX>(p, meet, nsteps, st0, s);
  }
}

template <class P, bool CX = false>
cudaError_t launch_disp(const Plan& p, const Meeting& meet, int nsteps, int st0, cudaStream_t s) {
  return p.disp ? launch_mask<P, true, CX>(p, meet, nsteps, st0, s)
                : launch_mask<P, false, CX>(p, meet, nsteps, st0, s);
}

}  // namespace

// Grids that step this way.  Measured on GB300, us per step, six launches per
// step -> one launch per chunk:
//   TMz / TEz   200^2 FP64 15.4 -> 6.1, 301x277 FP64 19.9 -> 8.4 FP32 16.9 -> 7.6,
//               1000x777 FP64 73.6 -> 26.4, 1400^2 FP64 159 -> 56 FP32 95 -> 32
//               df64 132 -> 67, 2000^2 FP64 313 -> 127 FP32 189 -> 91
// Grids of at most three components gain at every size (only their active
// components' points are visited, with the inactive curl terms left out), from
// the first step on (64^2 FP64 18.9 -> 14.5, 300^2 21.0 -> 16.5).  3-D grids
// gain while their launches weigh more than the one-plane kernel's shared
// neighbour loads; with the launches overlapped, a call of 1 / 2 / 4 / 20 steps
// (in brackets: with the tables that short calls no longer build):
//   48x40x44 FP64   26.9 -> (30.9)   23.7 -> 17.6   23.2 -> 19.1   22.3 -> 16.0
//            FP32   21.2 -> (25.1)   19.6 -> 14.6   18.5 -> 13.4   17.8 -> 10.4
//            df64   22.5 -> (26.9)   20.6 -> 16.5   19.2 -> 15.0   18.9 -> 12.1
//   24^3     FP64   24.9 -> 16.7     22.7 -> 12.5   22.5 -> 10.4   21.5 ->  7.6
//   32^3     FP32   20.7 -> 15.4     18.8 -> 11.5   18.1 -> 10.3   17.6 ->  7.3
//   64^3     FP64   38.7 -> (54.0)   36.3 -> (45.6)   34.7 -> 41.0   33.8 -> 37.0
//            FP32   25.0 -> (36.0)   22.1 -> (26.9)   20.0 -> 22.3   18.9 -> 18.6
//   63x45x37 Drude / Lorentz / DCP + UPML
//            FP64   42.8 -> (37.5)   40.5 -> (30.9)   38.6 -> 27.1   37.7 -> 24.0
//   complex 32x31x30  27.0 -> 20.6   25.8 -> 15.5   25.2 -> 11.8   24.5 ->  9.6
//   complex 64x64x48  41.5 -> (41.5)   39.8 -> (35.0)   38.5 -> 32.3   37.5 -> 29.4
constexpr int64_t kPersistCells = 1 << 17, kPersistCellsComplex = 1 << 18;
constexpr int64_t kPersistCellsOneStep = 1 << 15;

bool persist_takes(const Plan& p, int nsteps) {
  const GridDev& d = p.re;
  if (p.precision == GMES_FP64_STRICT || wait_error_word() == nullptr) return false;
  if (d.nsrc > kPersistSources || d.ntfsf > 0 || d.nprobe > 0 || !offsets_fit_i32(d)) return false;
  if (__builtin_popcount((unsigned)d.active) <= 3) return true;
  const int64_t most =
      nsteps == 1 ? kPersistCellsOneStep : (p.cplx ? kPersistCellsComplex : kPersistCells);
  return (int64_t)d.n[0] * d.n[1] * d.n[2] <= most;
}

__device__ Slot barrier_slots[kStreamSlots + kGraphSlots];

cudaError_t slots_address(Slot** at) {
  return cudaGetSymbolAddress(reinterpret_cast<void**>(at), barrier_slots);
}

__global__ void k_clear_slots() {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < kStreamSlots + kGraphSlots) barrier_slots[k] = Slot{0, 0, 0};
}

cudaError_t clear_slots() {
  k_clear_slots<<<(kStreamSlots + kGraphSlots + 255) / 256, 256>>>();
  return cudaGetLastError();
}

__global__ void k_wait_check(const Meeting m, int absent, void* out, int64_t bytes, int* error) {
  if ((int)blockIdx.x == absent) return;
  if (!grid_barrier(m, error)) {
    spoil(out, bytes);
    return;
  }
  leave_barrier(m);
}

cudaError_t launch_wait_check(const Meeting& meet, int blocks, int absent, void* out,
                              int64_t bytes, cudaStream_t s) {
  Meeting m = meet;
  int* error = wait_error_word();
  void* args[] = {&m, &absent, &out, &bytes, &error};
  return cudaLaunchCooperativeKernel((const void*)k_wait_check, dim3((unsigned)blocks), dim3(32),
                                     args, 0, s);
}

cudaError_t launch_persist(const Plan& p, const Meeting& meet, int nsteps, int st0, cudaStream_t s) {
  if (p.cplx) return launch_disp<PolF64, true>(p, meet, nsteps, st0, s);
  switch (p.precision) {
    case GMES_FP64:
      return launch_disp<PolF64>(p, meet, nsteps, st0, s);
    case GMES_FP32:
      return launch_disp<PolF32>(p, meet, nsteps, st0, s);
    case GMES_DF64:
      return launch_disp<PolDF>(p, meet, nsteps, st0, s);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace gmes
