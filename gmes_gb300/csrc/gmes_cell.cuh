// The update of one cell in a half-step, shared by the one-plane, multi-grid
// and persistent kernels: per-point updates of every material class, the
// fast-precision and strict cell bodies, and the point sources.  See
// gmes_step.cu for the index geometry.
#pragma once

#include <type_traits>

#include "gmes_internal.cuh"

namespace gmes {
namespace {

// ---------------------------------------------------------------------------
// Per-point update, fast form: precomputed reciprocals, FMA contraction
// allowed (FP64, FP32) or float-float arithmetic (DF64).
//   side 0 (E): F += c1 D1 - c2 D2            (Dielectric E)
//   side 1 (H): F += c2 D2 - c1 D1            (Dielectric H)
// ---------------------------------------------------------------------------
// State values of a CPML (psi1, psi2) or UPML (d) point, loaded for all
// three components of a cell before any of them is computed.
template <class P>
struct Pre {
  typename P::R a, b;
};

template <class P, int C>
__device__ __forceinline__ Pre<P> prefetch_state(const GridDev& g, int64_t lin, const int x[3],
                                                 uint8_t id) {
  (void)x;
  Pre<P> r{P::zero(), P::zero()};
  const int kind = __ldg(&g.tab[C][id].kind);
  const typename P::T* aux = static_cast<const typename P::T*>(g.aux[C]);
  if (kind == GMES_KIND_CPML) {
    // loaded unconditionally: testing the profile first (to skip the loads
    // outside the slabs) adds a dependent lookup and measured slower
    r.a = P::ldw(aux + lin);
    r.b = P::ldw(aux + g.npts[C] + lin);
  } else if (kind == GMES_KIND_UPML) {
    r.a = P::ldw(aux + lin);
  }
  return r;
}

// Whether the CPML psi updates run behind a warp-wide vote.  Measured on
// GB300 (256^3 cube): FP64 13.58 -> 14.18 Gcell/s (19.0 -> 17.6 FP64
// instructions per cell) and FP32 31.2 -> 32.7; the float-float type runs
// slower with it (19.6 -> 18.3; with a __syncwarp opening each voted block
// and 16-cell rows, 21.05 -> 20.67).  Votes in front of the other kinds'
// blocks were slower in every precision.
// (The float-float type keeps plain branches in its own CPML block in
// update_fast.)
template <class P>
struct PsiVote {
  static constexpr bool value = true;
};

// Whether a profile entry has kappa == 1 (the default CPML grading,
// kappa_max = 1, and every point outside the slab).
__device__ __forceinline__ bool kappa_one(const Coef* q) {
  return __ldg(reinterpret_cast<const unsigned long long*>(&q[2].d)) == 0x3FF0000000000000ull;
}

// CPML point with kappa == 1 on its live axes, written as the dielectric
// update plus the psi terms:
//   E: F + cdt ((psi1 - psi2) + D1/d1 - D2/d2) = ((F + c1 D1) - c2 D2) + cdt psi1 - cdt psi2
// (c1 = cdt/d1, c2 = cdt/d2), so the dielectric and CPML points of a warp
// share the first two FMAs, and a psi block runs only in warps where some
// lane is inside that axis' slab.  The separate CPML form ran both forms in
// every warp that straddles a slab edge along the contiguous axis.  Points
// with kappa != 1 take the separate form.  A __syncwarp at the top of each
// voted psi block keeps it a branch: without it the compiler predicated
// the blocks and every warp with a CPML lane issued both.  Measured on
// GB300 (256^3 cube, 10-cell CPML), FP64 warp-instructions per cell and
// half-step (E side) and Gcell/s:
//   separate form, psi votes                 17.6   14.23
//   shared form, votes                       16.8   14.93
//   shared form, votes + __syncwarp          14.4   16.17
// 14.4 is what a warp-level count of the slabs predicts when each psi block
// issues only in warps that need it.  FP32 (32.7 -> 30.7 Gcell/s) and the
// float-float type (19.6 -> 18.5) run slower with the shared form, and
// slower with __syncwarp in their own psi votes, so both keep the
// separate form.
template <class P>
struct SharedCpml {
  static constexpr bool value = false;
};
template <>
struct SharedCpml<PolF64> {
  static constexpr bool value = true;
};

// The plain update of a point (a dielectric class, or a CPML point outside
// both of its slabs): E: (F + c1 D1) - c2 D2, H: (F + c2 D2) - c1 D1, with
// both multiply-adds fused explicitly, so that the per-point path, the
// uniform-tile path and the multi-grid kernels round identically.
__device__ __forceinline__ double plain_e(double F, double c1, double c2, double p1, double p2) {
  return __fma_rn(-c2, p2, __fma_rn(c1, p1, F));
}
__device__ __forceinline__ float plain_e(float F, float c1, float c2, float p1, float p2) {
  return __fmaf_rn(-c2, p2, __fmaf_rn(c1, p1, F));
}
__device__ __forceinline__ df plain_e(df F, df c1, df c2, df p1, df p2) {
  return df_fma(-c2, p2, df_fma(c1, p1, F));
}
// A curl difference a - b of neighbouring field values.  Float-float: the
// high words' difference exactly (two-sum), the low words' difference
// added once (11 FP32 operations against 20 for the fully compensated
// difference); its error is about 2^-48 of the operands, the precision the
// float-float values are stored to.
__device__ __forceinline__ double curl_diff(double a, double b) { return a - b; }
__device__ __forceinline__ float curl_diff(float a, float b) { return a - b; }
__device__ __forceinline__ df curl_diff(df a, df b) {
  df s = df_two_sum(a.hi, -b.hi);
  s.lo = __fadd_rn(s.lo, __fsub_rn(a.lo, b.lo));
  return df_fast_two_sum(s.hi, s.lo);
}

template <bool E, class R>
__device__ __forceinline__ R plain_upd(R F, R c1, R c2, R p1, R p2) {
  return E ? plain_e(F, c1, c2, p1, p2) : plain_e(F, c2, c1, p2, p1);
}

// a b + c, fused explicitly, so that the CPML update rounds the same wherever
// it is inlined.
__device__ __forceinline__ double madd(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ df madd(df a, df b, df c) { return df_fma(a, b, c); }

// Whether component C's curl term t (1 or 2) reads an active component, for a
// compile-time mask (E: D1 of H_(own+2), D2 of H_(own+1); H likewise of E);
// true when the mask is read from the grid.
template <int MASK, int C, int t>
__device__ __forceinline__ constexpr bool curl_term() {
  constexpr int other = (C < 3 ? 3 : 0) + (C % 3 + (t == 1 ? 2 : 1)) % 3;
  return MASK == 0 || ((MASK >> other) & 1);
}
// plain_upd without the terms whose component is inactive in a compile-time
// mask (their difference is zero, so the value is the same): a 2-D grid's
// half-steps then take 4 + 4 FP64 instructions per cell instead of 10 + 8.
template <int MASK, int C, class R>
__device__ __forceinline__ R plain_mask(R F, R c1, R c2, R p1, R p2) {
  constexpr bool E = C < 3, t1 = curl_term<MASK, C, 1>(), t2 = curl_term<MASK, C, 2>();
  if constexpr (t1 && t2) return plain_upd<E>(F, c1, c2, p1, p2);
  if constexpr (t1) return madd(E ? c1 : -c1, p1, F);
  if constexpr (t2) return madd(E ? -c2 : c2, p2, F);
  return F;
}

// Update of a CPML point in the separate form (src/pw_cpml.hh:115-132 E,
// 327-344 H): psi1 = b1 psi1 + (c1/d1) D1 and psi2 likewise where the point
// is inside that axis' slab (c != 0; elsewhere psi stays exactly 0), then
// F +/- cdt ((psi1 - psi2) + D1/(kappa1 d1) - D2/(kappa2 d2)); a point
// outside both slabs takes the dielectric form.  Per point in update_fast,
// and for warps of one class per component in cell_body_fast.
template <class P, int C>
__device__ __forceinline__ void cpml_separate(const GridDev& g, int64_t lin, const int x[3],
                                              typename P::R p1, typename P::R p2,
                                              typename P::R F, const ClassCoef& cc,
                                              Pre<P> pre) {
  using R = typename P::R;
  using T = typename P::T;
  constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  constexpr bool E = C < 3;
  T* fp = static_cast<T*>(g.f[C]) + lin;
  T* aux = static_cast<T*>(g.aux[C]);
  const int64_t np = g.npts[C];
  const int pm = __ldg(&cc.pml);
  const Coef* q1 = g.prof[pm][C][a1] + (int64_t)x[a1] * kProfStride;
  const Coef* q2 = g.prof[pm][C][a2] + (int64_t)x[a2] * kProfStride;
  const bool on1 = coef_nonzero(q1 + 1), on2 = coef_nonzero(q2 + 1);
  if (!on1 && !on2) {
    // outside both slabs kappa = 1 and psi = 0: the dielectric update
    const R c1 = P::cfg(&cc.c1), c2 = P::cfg(&cc.c2);
    P::st(fp, plain_upd<E>(F, c1, c2, p1, p2));
    return;
  }
  R psi1 = pre.a, psi2 = pre.b;
  if constexpr (PsiVote<P>::value) {
    // A warp-wide vote before each psi update: the compiler otherwise
    // predicates the short update blocks, and every warp of the shell then
    // issues their instructions whether or not a lane is in that slab.
    // Each lane still keeps its own value (psi changes only where on).
    const unsigned am = __activemask();
    if (__any_sync(am, on1)) {
      const R n1 = madd(P::cfg(q1 + 3), p1, P::cfg(q1) * psi1);
      if (on1) {
        psi1 = n1;
        P::st(aux + lin, psi1);
      }
    }
    if (__any_sync(am, on2)) {
      const R n2 = madd(P::cfg(q2 + 3), p2, P::cfg(q2) * psi2);
      if (on2) {
        psi2 = n2;
        P::st(aux + np + lin, psi2);
      }
    }
  } else {
    if (on1) {
      psi1 = madd(P::cfg(q1 + 3), p1, P::cfg(q1) * psi1);
      P::st(aux + lin, psi1);
    }
    if (on2) {
      psi2 = madd(P::cfg(q2 + 3), p2, P::cfg(q2) * psi2);
      P::st(aux + np + lin, psi2);
    }
  }
  const R X = madd(-P::cfg(q2 + 4), p2, madd(P::cfg(q1 + 4), p1, psi1 - psi2));
  const R cdt = P::cfg(&cc.cdt);
  P::st(fp, E ? madd(cdt, X, F) : madd(-cdt, X, F));
}

template <class P, int C, bool DISP>
__device__ __forceinline__ void update_fast(const GridDev& g, int64_t lin, const int x[3],
                                            typename P::R p1, typename P::R p2,
                                            typename P::R F, uint8_t id, Pre<P> pre) {
  using R = typename P::R;
  using T = typename P::T;
  constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  constexpr bool E = C < 3;
  const ClassCoef& cc = g.tab[C][id];
  const int kind = __ldg(&cc.kind);
  if (kind == GMES_KIND_DUMMY) return;
  T* fp = static_cast<T*>(g.f[C]) + lin;
  if constexpr (SharedCpml<P>::value) {
    if (kind == GMES_KIND_DIELECTRIC || kind == GMES_KIND_CPML) {
      const bool cp = kind == GMES_KIND_CPML;
      // dielectric lanes point their profile entries at valid memory (the
      // class's own coefficients) so that a warp-wide psi block may load
      // them; their results are never used
      const Coef* q1 = &cc.eps;
      const Coef* q2 = &cc.eps;
      bool on1 = false, on2 = false, scaled = false;
      if (cp) {
        const int pm = __ldg(&cc.pml);
        q1 = g.prof[pm][C][a1] + (int64_t)x[a1] * kProfStride;
        q2 = g.prof[pm][C][a2] + (int64_t)x[a2] * kProfStride;
        on1 = coef_nonzero(q1 + 1);
        on2 = coef_nonzero(q2 + 1);
        scaled = (on1 && !kappa_one(q1)) || (on2 && !kappa_one(q2));
      }
      if (!scaled) {
        const R c1 = P::cfg(&(cc.c1)), c2 = P::cfg(&(cc.c2));
        R t = plain_upd<E>(F, c1, c2, p1, p2);
        const unsigned am = __activemask();
        if (__any_sync(am, on1 || on2)) {
          T* aux = static_cast<T*>(g.aux[C]);
          const R cdt = P::cfg(&cc.cdt);
          if (__any_sync(am, on1)) {
            __syncwarp(am);  // keeps the block a branch
            const R n1 = P::cfg(q1) * pre.a + P::cfg(q1 + 3) * p1;
            if (on1) {
              P::st(aux + lin, n1);
              t = E ? t + cdt * n1 : t - cdt * n1;
            }
          }
          if (__any_sync(am, on2)) {
            __syncwarp(am);  // keeps the block a branch
            const R n2 = P::cfg(q2) * pre.b + P::cfg(q2 + 3) * p2;
            if (on2) {
              P::st(aux + g.npts[C] + lin, n2);
              t = E ? t - cdt * n2 : t + cdt * n2;
            }
          }
        }
        P::st(fp, t);
        return;
      }
    }
  }
  if (kind == GMES_KIND_DIELECTRIC) {
    const R c1 = P::cfg(&(cc.c1)), c2 = P::cfg(&(cc.c2));
    P::st(fp, plain_upd<E>(F, c1, c2, p1, p2));
    return;
  }
  T* aux = static_cast<T*>(g.aux[C]);
  const int64_t np = g.npts[C];
  if (kind == GMES_KIND_CPML) {
    if constexpr (!std::is_same<P, PolDF>::value) {
      cpml_separate<P, C>(g, lin, x, p1, p2, F, cc, pre);
    } else {
      // the float-float type keeps this block inline: in cpml_separate it
      // spilled more and ran 1.5 % slower (256^3 cube, 24.21 -> 23.84
      // Gcell/s); the arithmetic is cpml_separate's, term for term (its
      // warp-uniform CPML path takes cpml_separate)
      const Coef* q1 = g.prof[__ldg(&cc.pml)][C][a1] + (int64_t)x[a1] * kProfStride;
      const Coef* q2 = g.prof[__ldg(&cc.pml)][C][a2] + (int64_t)x[a2] * kProfStride;
      const bool on1 = coef_nonzero(q1 + 1), on2 = coef_nonzero(q2 + 1);
      if (!on1 && !on2) {
        P::st(fp, plain_upd<E>(F, P::cfg(&cc.c1), P::cfg(&cc.c2), p1, p2));
        return;
      }
      R psi1 = pre.a, psi2 = pre.b;
      if (on1) {
        psi1 = madd(P::cfg(q1 + 3), p1, P::cfg(q1) * psi1);
        P::st(aux + lin, psi1);
      }
      if (on2) {
        psi2 = madd(P::cfg(q2 + 3), p2, P::cfg(q2) * psi2);
        P::st(aux + np + lin, psi2);
      }
      const R X = madd(-P::cfg(q2 + 4), p2, madd(P::cfg(q1 + 4), p1, psi1 - psi2));
      const R cdt = P::cfg(&cc.cdt);
      P::st(fp, E ? madd(cdt, X, F) : madd(-cdt, X, F));
    }
    return;
  }
  const R r1 = P::cf(g.rdr[a1]);
  const R r2 = P::cf(g.rdr[a2]);
  if (kind == GMES_KIND_UPML) {
    const Coef* q1 = g.prof[cc.pml][C][a1] + (int64_t)x[a1] * kProfStride;
    const Coef* q2 = g.prof[cc.pml][C][a2] + (int64_t)x[a2] * kProfStride;
    const Coef* q3 = g.prof[cc.pml][C][own] + (int64_t)x[own] * kProfStride;
    T* sp = aux + lin;
    const R d_old = pre.a;
    const R curl = p1 * r1 - p2 * r2;
    const R d_new = E ? P::cfg(&(q1[0])) * d_old + P::cfg(&(q1[1])) * curl
                      : P::cfg(&(q1[0])) * d_old - P::cfg(&(q1[1])) * curl;
    P::st(sp, d_new);
    P::st(fp, P::cfg(&(q2[0])) * F +
                  P::cfg(&(q2[2])) * (P::cfg(&(q3[3])) * d_new - P::cfg(&(q3[4])) * d_old) *
                      P::cfg(&(cc.reps)));
    return;
  }
  if (kind == GMES_KIND_CONST) {
    P::st(fp, P::cfg(g.part ? &(cc.value_im) : &(cc.value)));
    return;
  }
  if constexpr (DISP && E) {
    const Coef* pool = g.pool[C] + (int64_t)id * kPoolStride;
    const R curl = p1 * r1 - p2 * r2;
    const R e_now = F;
    if (kind == GMES_KIND_DRUDE || kind == GMES_KIND_LORENTZ) {
      // src/pw_drude.hh:89-151, src/pw_lorentz.hh:96-157
      R sum = P::zero();
      for (int q = 0; q < cc.npole; ++q) {
        T* qn = aux + (int64_t)(2 * q) * np + lin;      // q_now
        T* qw = aux + (int64_t)(2 * q + 1) * np + lin;  // q_new
        const R q_old = P::ldw(qn);
        const R q_now = P::ldw(qw);
        const R q_new = P::cfg(&(pool[kPoolA + 3 * q])) * q_old +
                        P::cfg(&(pool[kPoolA + 3 * q + 1])) * q_now +
                        P::cfg(&(pool[kPoolA + 3 * q + 2])) * e_now;
        P::st(qn, q_now);
        P::st(qw, q_new);
        sum = sum + (q_new - q_now);
      }
      P::st(fp, P::cfg(&(pool[kPoolC])) * curl + P::cfg(&(pool[kPoolC + 1])) * sum +
                    P::cfg(&(pool[kPoolC + 2])) * e_now);
      return;
    }
    if (kind == GMES_KIND_DCP) {
      // src/pw_dcp.hh:105-225
      T* eo = aux + lin;
      const R e_old = P::ldw(eo);
      R sd = P::zero(), sc = P::zero();
      for (int q = 0; q < cc.npole; ++q) {
        const R qo = P::ldw(aux + (int64_t)(1 + 2 * q) * np + lin);
        const R qn = P::ldw(aux + (int64_t)(2 + 2 * q) * np + lin);
        const R a0 = P::cfg(&(pool[kPoolA + 3 * q])), a1c = P::cfg(&(pool[kPoolA + 3 * q + 1]));
        sd = sd + ((P::from_double(1.0) - a1c) * qn - a0 * qo);
      }
      const int cb = 1 + 2 * cc.npole;
      for (int q = 0; q < cc.ncp; ++q) {
        const R po = P::ldw(aux + (int64_t)(cb + 2 * q) * np + lin);
        const R pn = P::ldw(aux + (int64_t)(cb + 2 * q + 1) * np + lin);
        const R b0 = P::cfg(&(pool[kPoolB + 5 * q])), b1 = P::cfg(&(pool[kPoolB + 5 * q + 1]));
        sc = sc + ((P::from_double(1.0) - b1) * pn - b0 * po);
      }
      const R e_new = P::cfg(&(pool[kPoolC])) * curl + P::cfg(&(pool[kPoolC + 1])) * (sd + sc) +
                      P::cfg(&(pool[kPoolC + 2])) * e_old + P::cfg(&(pool[kPoolC + 3])) * e_now;
      const R esum = (e_old + P::from_double(2.0) * e_now) + e_new;
      for (int q = 0; q < cc.npole; ++q) {
        T* qop = aux + (int64_t)(1 + 2 * q) * np + lin;
        T* qnp = aux + (int64_t)(2 + 2 * q) * np + lin;
        const R qo = P::ldw(qop), qn = P::ldw(qnp);
        const R q_new = P::cfg(&(pool[kPoolA + 3 * q])) * qo + P::cfg(&(pool[kPoolA + 3 * q + 1])) * qn +
                        P::cfg(&(pool[kPoolA + 3 * q + 2])) * esum;
        P::st(qop, qn);
        P::st(qnp, q_new);
      }
      for (int q = 0; q < cc.ncp; ++q) {
        T* pop = aux + (int64_t)(cb + 2 * q) * np + lin;
        T* pnp = aux + (int64_t)(cb + 2 * q + 1) * np + lin;
        const R po = P::ldw(pop), pn = P::ldw(pnp);
        const Coef* b = pool + kPoolB + 5 * q;
        const R p_new = P::cfg(&(b[0])) * po + P::cfg(&(b[1])) * pn + P::cfg(&(b[2])) * e_old +
                        P::cfg(&(b[3])) * e_now + P::cfg(&(b[4])) * e_new;
        P::st(pop, pn);
        P::st(pnp, p_new);
      }
      P::st(eo, e_now);
      P::st(fp, e_new);
      return;
    }
    if (kind == GMES_KIND_DCP_PLRC) {
      // src/pw_dcp.hh:466-583: psi_dp[npole] real, psi_cp[ncp] complex (re, im)
      const int cb = cc.npole;
      R psum = P::zero(), csum = P::zero();
      for (int q = 0; q < cc.npole; ++q) psum = psum + P::ldw(aux + (int64_t)q * np + lin);
      for (int q = 0; q < cc.ncp; ++q)
        csum = csum + P::ldw(aux + (int64_t)(cb + 2 * q) * np + lin);
      const R e_new = (P::cfg(&(pool[kPoolC])) * curl + P::cfg(&(pool[kPoolC + 1])) * e_now) +
                      P::cfg(&(pool[kPoolC + 2])) * (psum + csum);
      for (int q = 0; q < cc.npole; ++q) {
        T* sp = aux + (int64_t)q * np + lin;
        const Coef* a = pool + kPoolA + 3 * q;
        P::st(sp, (P::cfg(a) * e_new + P::cfg(a + 1) * e_now) + P::cfg(a + 2) * P::ldw(sp));
      }
      for (int q = 0; q < cc.ncp; ++q) {
        T* pr_ = aux + (int64_t)(cb + 2 * q) * np + lin;
        T* pi_ = aux + (int64_t)(cb + 2 * q + 1) * np + lin;
        const R pr = P::ldw(pr_), pi = P::ldw(pi_);
        const Coef* b = pool + kPoolB + 6 * q;
        P::st(pr_, (P::cfg(b) * e_new + P::cfg(b + 2) * e_now) +
                       (P::cfg(b + 4) * pr - P::cfg(b + 5) * pi));
        P::st(pi_, (P::cfg(b + 1) * e_new + P::cfg(b + 3) * e_now) +
                       (P::cfg(b + 4) * pi + P::cfg(b + 5) * pr));
      }
      P::st(fp, e_new);
      return;
    }
  }
}

// ---------------------------------------------------------------------------
// Per-point update in the reference's exact operation order (FP64, no FMA,
// IEEE division): bit-for-bit the arithmetic of src/pw_*.hh.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double ADD(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double SUB(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double MUL(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double DIV(double a, double b) { return __ddiv_rn(a, b); }

template <int C, bool DISP>
__device__ __forceinline__ void update_strict(const GridDev& g, int64_t lin, const int x[3],
                                              double D1, double D2, double F, uint8_t id) {
  constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  constexpr bool E = C < 3;
  const ClassCoef& cc = g.tab[C][id];
  const int kind = cc.kind;
  if (kind == GMES_KIND_DUMMY) return;
  double* fp = static_cast<double*>(g.f[C]) + lin;
  const double dt = g.dt, d1 = g.dr[a1], d2 = g.dr[a2], eps = cc.eps.d;
  if (kind == GMES_KIND_DIELECTRIC) {
    // E: e += dt/eps * (D1/d1 - D2/d2); H: h += dt/mu * (D2/d2 - D1/d1)
    const double X = E ? SUB(DIV(D1, d1), DIV(D2, d2)) : SUB(DIV(D2, d2), DIV(D1, d1));
    *fp = ADD(F, MUL(DIV(dt, eps), X));
    return;
  }
  double* aux = static_cast<double*>(g.aux[C]);
  const int64_t np = g.npts[C];
  if (kind == GMES_KIND_CPML) {
    // src/pw_cpml.hh:115-132 (E), 327-344 (H)
    const Coef* q1 = g.prof[cc.pml][C][a1] + (int64_t)x[a1] * kProfStride;
    const Coef* q2 = g.prof[cc.pml][C][a2] + (int64_t)x[a2] * kProfStride;
    double* s1 = aux + lin;
    double* s2 = aux + np + lin;
    const double psi1 = ADD(MUL(q1[0].d, *s1), DIV(MUL(q1[1].d, D1), d1));
    const double psi2 = ADD(MUL(q2[0].d, *s2), DIV(MUL(q2[1].d, D2), d2));
    *s1 = psi1;
    *s2 = psi2;
    const double X =
        SUB(ADD(SUB(DIV(DIV(D1, d1), q1[2].d), DIV(DIV(D2, d2), q2[2].d)), psi1), psi2);
    const double inc = MUL(DIV(dt, eps), X);
    *fp = E ? ADD(F, inc) : SUB(F, inc);
    return;
  }
  const double curl = SUB(DIV(D1, d1), DIV(D2, d2));
  if (kind == GMES_KIND_UPML) {
    // src/pw_upml.hh:113-128 (E), 317-332 (H)
    const Coef* q1 = g.prof[cc.pml][C][a1] + (int64_t)x[a1] * kProfStride;
    const Coef* q2 = g.prof[cc.pml][C][a2] + (int64_t)x[a2] * kProfStride;
    const Coef* q3 = g.prof[cc.pml][C][own] + (int64_t)x[own] * kProfStride;
    double* sp = aux + lin;
    const double dstore = *sp;
    const double dn = E ? ADD(MUL(q1[0].d, dstore), MUL(q1[1].d, curl))
                        : SUB(MUL(q1[0].d, dstore), MUL(q1[1].d, curl));
    *sp = dn;
    *fp = ADD(MUL(q2[0].d, F),
              DIV(MUL(q2[2].d, SUB(MUL(q3[3].d, dn), MUL(q3[4].d, dstore))), eps));
    return;
  }
  if (kind == GMES_KIND_CONST) {
    *fp = g.part ? cc.value_im.d : cc.value.d;
    return;
  }
  if constexpr (DISP && E) {
    const Coef* pool = g.pool[C] + (int64_t)id * kPoolStride;
    const double e_now = F;
    if (kind == GMES_KIND_DRUDE || kind == GMES_KIND_LORENTZ) {
      double sum = 0.0;
      for (int q = 0; q < cc.npole; ++q) {
        double* qn = aux + (int64_t)(2 * q) * np + lin;
        double* qw = aux + (int64_t)(2 * q + 1) * np + lin;
        const double q_old = *qn, q_now = *qw;
        const double q_new = ADD(ADD(MUL(pool[kPoolA + 3 * q].d, q_old),
                                     MUL(pool[kPoolA + 3 * q + 1].d, q_now)),
                                 MUL(pool[kPoolA + 3 * q + 2].d, e_now));
        *qn = q_now;
        *qw = q_new;
        sum = ADD(sum, SUB(q_new, q_now));
      }
      *fp = ADD(ADD(MUL(pool[kPoolC].d, curl), MUL(pool[kPoolC + 1].d, sum)),
                MUL(pool[kPoolC + 2].d, e_now));
      return;
    }
    if (kind == GMES_KIND_DCP) {
      double* eo = aux + lin;
      const double e_old = *eo;
      double sd = 0.0, sc = 0.0;
      for (int q = 0; q < cc.npole; ++q) {
        const double qo = aux[(int64_t)(1 + 2 * q) * np + lin];
        const double qn = aux[(int64_t)(2 + 2 * q) * np + lin];
        sd = ADD(sd, SUB(MUL(SUB(1.0, pool[kPoolA + 3 * q + 1].d), qn),
                         MUL(pool[kPoolA + 3 * q].d, qo)));
      }
      const int cb = 1 + 2 * cc.npole;
      for (int q = 0; q < cc.ncp; ++q) {
        const double po = aux[(int64_t)(cb + 2 * q) * np + lin];
        const double pn = aux[(int64_t)(cb + 2 * q + 1) * np + lin];
        sc = ADD(sc, SUB(MUL(SUB(1.0, pool[kPoolB + 5 * q + 1].d), pn),
                         MUL(pool[kPoolB + 5 * q].d, po)));
      }
      const double e_new =
          ADD(ADD(ADD(MUL(pool[kPoolC].d, curl), MUL(pool[kPoolC + 1].d, ADD(sd, sc))),
                  MUL(pool[kPoolC + 2].d, e_old)),
              MUL(pool[kPoolC + 3].d, e_now));
      const double esum = ADD(ADD(e_old, MUL(2.0, e_now)), e_new);
      for (int q = 0; q < cc.npole; ++q) {
        double* qop = aux + (int64_t)(1 + 2 * q) * np + lin;
        double* qnp = aux + (int64_t)(2 + 2 * q) * np + lin;
        const double qo = *qop, qn = *qnp;
        const double q_new = ADD(ADD(MUL(pool[kPoolA + 3 * q].d, qo),
                                     MUL(pool[kPoolA + 3 * q + 1].d, qn)),
                                 MUL(pool[kPoolA + 3 * q + 2].d, esum));
        *qop = qn;
        *qnp = q_new;
      }
      for (int q = 0; q < cc.ncp; ++q) {
        double* pop = aux + (int64_t)(cb + 2 * q) * np + lin;
        double* pnp = aux + (int64_t)(cb + 2 * q + 1) * np + lin;
        const double po = *pop, pn = *pnp;
        const Coef* b = pool + kPoolB + 5 * q;
        const double p_new =
            ADD(ADD(ADD(ADD(MUL(b[0].d, po), MUL(b[1].d, pn)), MUL(b[2].d, e_old)),
                    MUL(b[3].d, e_now)),
                MUL(b[4].d, e_new));
        *pop = pn;
        *pnp = p_new;
      }
      *eo = e_now;
      *fp = e_new;
      return;
    }
    if (kind == GMES_KIND_DCP_PLRC) {
      // src/pw_dcp.hh:466-583 in its operation order; psi_cp complex
      // products as (ac - bd, ad + bc)
      const int cb = cc.npole;
      double psum = 0.0, csum = 0.0;
      for (int q = 0; q < cc.npole; ++q) psum = ADD(psum, aux[(int64_t)q * np + lin]);
      for (int q = 0; q < cc.ncp; ++q) csum = ADD(csum, aux[(int64_t)(cb + 2 * q) * np + lin]);
      const double e_new = ADD(ADD(MUL(pool[kPoolC].d, curl), MUL(pool[kPoolC + 1].d, e_now)),
                               MUL(pool[kPoolC + 2].d, ADD(psum, csum)));
      for (int q = 0; q < cc.npole; ++q) {
        double* sp = aux + (int64_t)q * np + lin;
        const Coef* a = pool + kPoolA + 3 * q;
        *sp = ADD(ADD(MUL(a[0].d, e_new), MUL(a[1].d, e_now)), MUL(a[2].d, *sp));
      }
      for (int q = 0; q < cc.ncp; ++q) {
        double* pr_ = aux + (int64_t)(cb + 2 * q) * np + lin;
        double* pi_ = aux + (int64_t)(cb + 2 * q + 1) * np + lin;
        const double pr = *pr_, pi = *pi_;
        const Coef* b = pool + kPoolB + 6 * q;
        *pr_ = ADD(ADD(MUL(b[0].d, e_new), MUL(b[2].d, e_now)),
                   SUB(MUL(b[4].d, pr), MUL(b[5].d, pi)));
        *pi_ = ADD(ADD(MUL(b[1].d, e_new), MUL(b[3].d, e_now)),
                   ADD(MUL(b[4].d, pi), MUL(b[5].d, pr)));
      }
      *fp = e_new;
      return;
    }
  }
}

// ---------------------------------------------------------------------------
// The half-step kernel.  One thread per cell (i, j, k) of the N0 x N1 x N2
// update domain; the thread updates the three components of its half there.
// Every value the cell needs from DRAM -- the class ids, the component's own
// values and the nine neighbour values of the curls -- is loaded up front,
// before any store, so a thread waits for one memory latency instead of a
// chain of them; only state slots (PML, ADE) are loaded after the class is
// known.  Block = bx x by threads over (k, j) with bx = min(32, n2 rounded up
// to a power of two), so thin (2-D) grids still fill whole warps along j;
// grid.z walks i.
// ---------------------------------------------------------------------------
template <int MASK, int C>
__device__ __forceinline__ bool is_active(const GridDev& g) {
  if constexpr (MASK != 0)
    return (MASK >> C) & 1;
  else
    return (g.active >> C) & 1;
}

// Fields are read with plain loads: the kernels that call this come up while the
// kernel before them still writes (after_launch), or step several times in one
// launch, and a read-only load is for data that nobody writes meanwhile.
template <class P, int MASK, int C, class I>
__device__ __forceinline__ typename P::R ldf(const GridDev& g, I off) {
  if (!is_active<MASK, C>(g)) return P::zero();
  return P::ldw(static_cast<const typename P::T*>(g.f[C]) + off);
}

template <int MASK, int C, class I>
__device__ __forceinline__ uint8_t ldc(const GridDev& g, I off) {
  if (!is_active<MASK, C>(g)) return 0;
  return __ldg(g.cls[C] + off);
}

template <class P, int C, bool STRICT, bool DISP>
__device__ __forceinline__ void upd(const GridDev& g, int64_t lin, const int x[3],
                                    typename P::R p1, typename P::R p2, typename P::R F,
                                    uint8_t id, Pre<P> pre) {
  if (!is_active<0, C>(g)) return;
  if constexpr (STRICT)
    update_strict<C, DISP>(g, lin, x, p1, p2, F, id);
  else
    update_fast<P, C, DISP>(g, lin, x, p1, p2, F, id, pre);
}

template <class P, int C, bool STRICT>
__device__ __forceinline__ Pre<P> pre_of(const GridDev& g, int64_t lin, const int x[3],
                                         uint8_t id) {
  if constexpr (STRICT) {
    return Pre<P>{P::zero(), P::zero()};
  } else {
    if (!is_active<0, C>(g)) return Pre<P>{P::zero(), P::zero()};
    return prefetch_state<P, C>(g, lin, x, id);
  }
}

// I: offset type (int32_t for grids whose components hold
// fewer than 2^31 points, int64_t otherwise).
template <class P, int SIDE, bool STRICT, bool DISP, class I>
__device__ __forceinline__ void cell_body(const GridDev& g, int i, int j, int k) {
  using R = typename P::R;
  const I s00 = (I)g.st[0][0], s01 = (I)g.st[0][1], s10 = (I)g.st[1][0], s11 = (I)g.st[1][1];
  const I s20 = (I)g.st[2][0], s21 = (I)g.st[2][1], s30 = (I)g.st[3][0], s31 = (I)g.st[3][1];
  const I s40 = (I)g.st[4][0], s41 = (I)g.st[4][1], s50 = (I)g.st[5][0], s51 = (I)g.st[5][1];
  const I ii = (I)i, jj = (I)j, kk = (I)k;
  const int xc[3] = {i, j, k};
  if constexpr (SIDE == 0) {
    // own points: Ex, Ey, Ez at (i, j, k)
    const I lx = ii * s00 + jj * s01 + kk;
    const I ly = ii * s10 + jj * s11 + kk;
    const I lz = ii * s20 + jj * s21 + kk;
    const uint8_t idx = ldc<0, 0>(g, lx), idy = ldc<0, 1>(g, ly), idz = ldc<0, 2>(g, lz);
    const R ex = ldf<P, 0, 0>(g, lx), ey = ldf<P, 0, 1>(g, ly), ez = ldf<P, 0, 2>(g, lz);
    // neighbour H values
    const I hx = ii * s30 + jj * s31 + kk;         // Hx[i, j, k]
    const I hy = (ii + 1) * s40 + jj * s41 + kk;   // Hy[i+1, j, k]
    const I hz = (ii + 1) * s50 + jj * s51 + kk;   // Hz[i+1, j, k]
    const R hz_a = ldf<P, 0, 5>(g, hz + s51);          // Hz[i+1, j+1, k]
    const R hz_b = ldf<P, 0, 5>(g, hz);                // Hz[i+1, j,   k]
    const R hz_c = ldf<P, 0, 5>(g, hz + s51 - s50);    // Hz[i,   j+1, k]
    const R hy_a = ldf<P, 0, 4>(g, hy + 1);            // Hy[i+1, j, k+1]
    const R hy_b = ldf<P, 0, 4>(g, hy);                // Hy[i+1, j, k]
    const R hy_c = ldf<P, 0, 4>(g, hy + 1 - s40);      // Hy[i,   j, k+1]
    const R hx_a = ldf<P, 0, 3>(g, hx + s31 + 1);      // Hx[i, j+1, k+1]
    const R hx_b = ldf<P, 0, 3>(g, hx + s31);          // Hx[i, j+1, k]
    const R hx_c = ldf<P, 0, 3>(g, hx + 1);            // Hx[i, j,   k+1]
    const Pre<P> px = pre_of<P, 0, STRICT>(g, lx, xc, idx);
    const Pre<P> py = pre_of<P, 1, STRICT>(g, ly, xc, idy);
    const Pre<P> pz = pre_of<P, 2, STRICT>(g, lz, xc, idz);
    upd<P, 0, STRICT, DISP>(g, lx, xc, hz_a - hz_b, hy_a - hy_b, ex, idx, px);
    upd<P, 1, STRICT, DISP>(g, ly, xc, hx_a - hx_b, hz_a - hz_c, ey, idy, py);
    upd<P, 2, STRICT, DISP>(g, lz, xc, hy_a - hy_c, hx_a - hx_c, ez, idz, pz);
  } else {
    // own points: Hx[i, j+1, k+1], Hy[i+1, j, k+1], Hz[i+1, j+1, k]
    const I lx = ii * s30 + (jj + 1) * s31 + kk + 1;
    const I ly = (ii + 1) * s40 + jj * s41 + kk + 1;
    const I lz = (ii + 1) * s50 + (jj + 1) * s51 + kk;
    const uint8_t idx = ldc<0, 3>(g, lx), idy = ldc<0, 4>(g, ly), idz = ldc<0, 5>(g, lz);
    const R hx = ldf<P, 0, 3>(g, lx), hy = ldf<P, 0, 4>(g, ly), hz = ldf<P, 0, 5>(g, lz);
    const I ex = ii * s00 + jj * s01 + kk;
    const I ey = ii * s10 + jj * s11 + kk;
    const I ez = ii * s20 + jj * s21 + kk;
    const R ez_0 = ldf<P, 0, 2>(g, ez);           // Ez[i, j, k]
    const R ez_j = ldf<P, 0, 2>(g, ez + s21);     // Ez[i, j+1, k]
    const R ez_i = ldf<P, 0, 2>(g, ez + s20);     // Ez[i+1, j, k]
    const R ey_0 = ldf<P, 0, 1>(g, ey);           // Ey[i, j, k]
    const R ey_k = ldf<P, 0, 1>(g, ey + 1);       // Ey[i, j, k+1]
    const R ey_i = ldf<P, 0, 1>(g, ey + s10);     // Ey[i+1, j, k]
    const R ex_0 = ldf<P, 0, 0>(g, ex);           // Ex[i, j, k]
    const R ex_k = ldf<P, 0, 0>(g, ex + 1);       // Ex[i, j, k+1]
    const R ex_j = ldf<P, 0, 0>(g, ex + s01);     // Ex[i, j+1, k]
    const int x3[3] = {i, j + 1, k + 1}, x4[3] = {i + 1, j, k + 1}, x5[3] = {i + 1, j + 1, k};
    const Pre<P> px = pre_of<P, 3, STRICT>(g, lx, x3, idx);
    const Pre<P> py = pre_of<P, 4, STRICT>(g, ly, x4, idy);
    const Pre<P> pz = pre_of<P, 5, STRICT>(g, lz, x5, idz);
    upd<P, 3, STRICT, DISP>(g, lx, x3, ez_j - ez_0, ey_k - ey_0, hx, idx, px);
    upd<P, 4, STRICT, DISP>(g, ly, x4, ex_k - ex_0, ez_i - ez_0, hy, idy, py);
    upd<P, 5, STRICT, DISP>(g, lz, x5, ey_i - ey_0, ex_j - ex_0, hz, idz, pz);
  }
}

// Whether a warp whose class triple is uniform, with DIELECTRIC or CPML
// classes (the CPML shell), takes those kinds' updates directly instead of
// the per-point kind dispatch.  Measured on GB300 (256^3 cube, Gcell/s, one
// box): FP32 39.78 -> 40.64; with it df64 ran 24.21 -> 23.01 and FP64 18.90
// -> 18.91, so only FP32 takes it (GMES_UNIFORM_CPML = 1 gives it every
// precision, 0 none).  Re-measured per half with the per-half register
// budgets (ms): df64 E 0.3185 -> 0.403, H 0.3245 -> 0.3200; FP64 E 0.4435
// -> 0.4697, H 0.4428 -> 0.4497; so the float-float type takes it on its H
// half too.  The CPML update it shares with the per-point path
// (cpml_separate) fuses every multiply-add explicitly: inlined in two places
// with implicit contraction, the two copies rounded differently and a grid
// batched with another warp layout lost bit-identity with its solo run.
template <class P, int SIDE>
struct UniformCpml {
#if defined(GMES_UNIFORM_CPML)
  static constexpr bool value = GMES_UNIFORM_CPML != 0;
#else
  static constexpr bool value = false;
#endif
};
template <int SIDE>
struct UniformCpml<PolF32, SIDE> {
#if defined(GMES_UNIFORM_CPML)
  static constexpr bool value = GMES_UNIFORM_CPML != 0;
#else
  static constexpr bool value = true;
#endif
};
template <int SIDE>
struct UniformCpml<PolDF, SIDE> {
#if defined(GMES_UNIFORM_CPML)
  static constexpr bool value = GMES_UNIFORM_CPML != 0;
#else
  static constexpr bool value = SIDE == 1;
#endif
};

// The psi pair (psi1, psi2) of a CPML point of component c.
template <class P>
__device__ __forceinline__ Pre<P> psi_pair(const GridDev& g, int c, int64_t lin) {
  const typename P::T* aux = static_cast<const typename P::T*>(g.aux[c]);
  return {P::ldw(aux + lin), P::ldw(aux + g.npts[c] + lin)};
}

// Whether a warp on the warp-uniform CPML path reads its classes'
// plain-form coefficients together with their kinds (one round trip to the
// class table instead of two).  Measured on GB300 (256^3 cube, ms per E / H
// half): df64 0.3143 / 0.3192 -> 0.3145 / 0.3135; FP32 0.2044 / 0.2070 ->
// 0.2269 / 0.2098 (three more live values at 40 registers), so the
// float-float type only (GMES_EARLY_COEF = 0 / 1 sets it for both).
template <class P>
struct EarlyCoef {
#if defined(GMES_EARLY_COEF)
  static constexpr bool value = GMES_EARLY_COEF != 0;
#else
  static constexpr bool value = std::is_same<P, PolDF>::value;
#endif
};

// The half-step update of one cell in the fast precisions.  Every field
// value and class id the cell reads is loaded first, so that no load waits
// for another.  Then a warp whose cells all carry the same class triple, each
// class of kind DIELECTRIC (one vote, __match_all_sync, and three
// warp-uniform kind look-ups), updates its three points with those classes'
// coefficients and nothing else (FP32 and the float-float H half also take
// warps of one DIELECTRIC or CPML class per component directly:
// UniformCpml); every other warp goes through the per-point path
// (update_fast), whose dielectric and CPML branches are the same
// arithmetic, so the paths agree bit for bit.  The offsets come from
// the three array-shape families (fst): an active component's strides are
// its family's.  Measured on GB300 (256^3 cube / 192^3 dispersive scene,
// Gcell/s, per-point path only -> with the warp-uniform path):
//   cube FP64 17.42 -> 18.60, FP32 34.17 -> 34.91, df64 21.89 -> 23.63;
//   dispersive FP64 9.85 -> 10.09, FP32 20.48 -> 22.36, df64 14.85 -> 15.04.
// A per-warp table of plain warps built at set-up (read with the field
// values, class maps read only by the other warps) ran slower: cube FP64
// 18.20, FP32 31.90, df64 22.95.  So did two cells per thread, (i, j, k) and
// (i + 1, j, k), with the loads of both issued before either update (twice
// the bytes in flight per warp, four shared neighbour loads): cube FP32
// 42.54 -> 30.1 / 29.7 / 34.3 / 31.1 Gcell/s at 6 / 7 / 8 / 10 blocks per SM
// (64 registers at 8), dispersive FP32 25.42 -> 22.35; df64 (5, 6 blocks)
// 26.74 -> 17.5 / 20.7, FP64 (6 blocks) 19.25 -> 16.99.
template <class P, int SIDE, bool DISP, class I>
__device__ __forceinline__ void cell_body_fast(const GridDev& g, int i, int j, int k) {
  using R = typename P::R;
  using T = typename P::T;
  constexpr int c0 = 3 * SIDE;
  const I X0 = (I)g.fst[0][0], X1 = (I)g.fst[0][1];
  const I Y0 = (I)g.fst[1][0], Y1 = (I)g.fst[1][1];
  const I Z0 = (I)g.fst[2][0], Z1 = (I)g.fst[2][1];
  const I ii = (I)i, jj = (I)j, kk = (I)k;
  const I oX = ii * X0 + jj * X1 + kk;
  const I oY = ii * Y0 + jj * Y1 + kk;
  const I oZ = ii * Z0 + jj * Z1 + kk;
  // own points: E (i, j, k); Hx[i, j+1, k+1], Hy[i+1, j, k+1], Hz[i+1, j+1, k]
  const I l0 = SIDE == 0 ? oX : oX + X1 + 1;
  const I l1 = SIDE == 0 ? oY : oY + Y0 + 1;
  const I l2 = SIDE == 0 ? oZ : oZ + Z0 + Z1;
  const R f0 = ldf<P, 0, c0>(g, l0), f1 = ldf<P, 0, c0 + 1>(g, l1),
          f2 = ldf<P, 0, c0 + 2>(g, l2);
  R d01, d02, d11, d12, d21, d22;  // (D1, D2) of each component
  if constexpr (SIDE == 0) {
    const R hz_a = ldf<P, 0, 5>(g, oZ + Z0 + Z1);  // Hz[i+1, j+1, k]
    const R hz_b = ldf<P, 0, 5>(g, oZ + Z0);       // Hz[i+1, j,   k]
    const R hz_c = ldf<P, 0, 5>(g, oZ + Z1);       // Hz[i,   j+1, k]
    const R hy_a = ldf<P, 0, 4>(g, oY + Y0 + 1);   // Hy[i+1, j, k+1]
    const R hy_b = ldf<P, 0, 4>(g, oY + Y0);       // Hy[i+1, j, k]
    const R hy_c = ldf<P, 0, 4>(g, oY + 1);        // Hy[i,   j, k+1]
    const R hx_a = ldf<P, 0, 3>(g, oX + X1 + 1);   // Hx[i, j+1, k+1]
    const R hx_b = ldf<P, 0, 3>(g, oX + X1);       // Hx[i, j+1, k]
    const R hx_c = ldf<P, 0, 3>(g, oX + 1);        // Hx[i, j,   k+1]
    d01 = curl_diff(hz_a, hz_b); d02 = curl_diff(hy_a, hy_b);
    d11 = curl_diff(hx_a, hx_b); d12 = curl_diff(hz_a, hz_c);
    d21 = curl_diff(hy_a, hy_c); d22 = curl_diff(hx_a, hx_c);
  } else {
    const R ez_0 = ldf<P, 0, 2>(g, oZ);       // Ez[i, j, k]
    const R ez_j = ldf<P, 0, 2>(g, oZ + Z1);  // Ez[i, j+1, k]
    const R ez_i = ldf<P, 0, 2>(g, oZ + Z0);  // Ez[i+1, j, k]
    const R ey_0 = ldf<P, 0, 1>(g, oY);       // Ey[i, j, k]
    const R ey_k = ldf<P, 0, 1>(g, oY + 1);   // Ey[i, j, k+1]
    const R ey_i = ldf<P, 0, 1>(g, oY + Y0);  // Ey[i+1, j, k]
    const R ex_0 = ldf<P, 0, 0>(g, oX);       // Ex[i, j, k]
    const R ex_k = ldf<P, 0, 0>(g, oX + 1);   // Ex[i, j, k+1]
    const R ex_j = ldf<P, 0, 0>(g, oX + X1);  // Ex[i, j+1, k]
    d01 = curl_diff(ez_j, ez_0); d02 = curl_diff(ey_k, ey_0);
    d11 = curl_diff(ex_k, ex_0); d12 = curl_diff(ez_i, ez_0);
    d21 = curl_diff(ey_i, ey_0); d22 = curl_diff(ex_j, ex_0);
  }
  const uint8_t id0 = ldc<0, c0>(g, l0), id1 = ldc<0, c0 + 1>(g, l1),
                id2 = ldc<0, c0 + 2>(g, l2);
  const uint32_t t = (uint32_t)id0 | (uint32_t)id1 << 8 | (uint32_t)id2 << 16;
  int same = 0;
  __match_all_sync(__activemask(), t, &same);
  const bool uniform = same && !g.pointwise;
  // the warp's kinds when its class triple is uniform (inactive components
  // count as dielectric: they are skipped)
  int ka = GMES_KIND_DIELECTRIC, kb = GMES_KIND_DIELECTRIC, kc = GMES_KIND_DIELECTRIC;
  bool fast;
  // plain-form coefficients of the warp's three classes, read with the kinds
  // (one round trip to the class table instead of two)
  R ca1 = P::zero(), ca2 = P::zero(), cb1 = P::zero(), cb2 = P::zero(), cc1 = P::zero(),
    cc2 = P::zero();
  if constexpr (UniformCpml<P, SIDE>::value) {
    if (uniform) {
      if (is_active<0, c0>(g)) {
        const ClassCoef& q = g.tab[c0][id0];
        ka = q.kind;
        if (EarlyCoef<P>::value) ca1 = P::cfg(&q.c1), ca2 = P::cfg(&q.c2);
      }
      if (is_active<0, c0 + 1>(g)) {
        const ClassCoef& q = g.tab[c0 + 1][id1];
        kb = q.kind;
        if (EarlyCoef<P>::value) cb1 = P::cfg(&q.c1), cb2 = P::cfg(&q.c2);
      }
      if (is_active<0, c0 + 2>(g)) {
        const ClassCoef& q = g.tab[c0 + 2][id2];
        kc = q.kind;
        if (EarlyCoef<P>::value) cc1 = P::cfg(&q.c1), cc2 = P::cfg(&q.c2);
      }
    }
    fast = uniform && ka == GMES_KIND_DIELECTRIC && kb == GMES_KIND_DIELECTRIC &&
           kc == GMES_KIND_DIELECTRIC;
  } else {
    fast = uniform &&
           (!is_active<0, c0>(g) || g.tab[c0][id0].kind == GMES_KIND_DIELECTRIC) &&
           (!is_active<0, c0 + 1>(g) || g.tab[c0 + 1][id1].kind == GMES_KIND_DIELECTRIC) &&
           (!is_active<0, c0 + 2>(g) || g.tab[c0 + 2][id2].kind == GMES_KIND_DIELECTRIC);
  }
  constexpr bool E = SIDE == 0;
  if (fast) {  // warp-uniform
    const ClassCoef& qa = g.tab[c0][id0];
    const ClassCoef& qb = g.tab[c0 + 1][id1];
    const ClassCoef& qc = g.tab[c0 + 2][id2];
    if (UniformCpml<P, SIDE>::value && EarlyCoef<P>::value) {
      if (is_active<0, c0>(g))
        P::st(static_cast<T*>(g.f[c0]) + l0, plain_upd<E>(f0, ca1, ca2, d01, d02));
      if (is_active<0, c0 + 1>(g))
        P::st(static_cast<T*>(g.f[c0 + 1]) + l1, plain_upd<E>(f1, cb1, cb2, d11, d12));
      if (is_active<0, c0 + 2>(g))
        P::st(static_cast<T*>(g.f[c0 + 2]) + l2, plain_upd<E>(f2, cc1, cc2, d21, d22));
      return;
    }
    if (is_active<0, c0>(g))
      P::st(static_cast<T*>(g.f[c0]) + l0,
            plain_upd<E>(f0, P::cfg(&qa.c1), P::cfg(&qa.c2), d01, d02));
    if (is_active<0, c0 + 1>(g))
      P::st(static_cast<T*>(g.f[c0 + 1]) + l1,
            plain_upd<E>(f1, P::cfg(&qb.c1), P::cfg(&qb.c2), d11, d12));
    if (is_active<0, c0 + 2>(g))
      P::st(static_cast<T*>(g.f[c0 + 2]) + l2,
            plain_upd<E>(f2, P::cfg(&qc.c1), P::cfg(&qc.c2), d21, d22));
    return;
  }
  if constexpr (UniformCpml<P, SIDE>::value) {
    const auto dc = [](int kd) {
      return kd == GMES_KIND_DIELECTRIC || kd == GMES_KIND_CPML;
    };
    if (uniform && dc(ka) && dc(kb) && dc(kc)) {
      // one class per component across the warp, each DIELECTRIC or CPML
      // (the CPML shell): those kinds' updates with the kinds known for the
      // whole warp, the psi values of the CPML components loaded first
      const int xa[3] = {i, SIDE == 0 ? j : j + 1, SIDE == 0 ? k : k + 1};
      const int xb[3] = {SIDE == 0 ? i : i + 1, j, SIDE == 0 ? k : k + 1};
      const int xq[3] = {SIDE == 0 ? i : i + 1, SIDE == 0 ? j : j + 1, k};
      Pre<P> pa{P::zero(), P::zero()}, pb = pa, pc = pa;
      if (ka == GMES_KIND_CPML) pa = psi_pair<P>(g, c0, l0);
      if (kb == GMES_KIND_CPML) pb = psi_pair<P>(g, c0 + 1, l1);
      if (kc == GMES_KIND_CPML) pc = psi_pair<P>(g, c0 + 2, l2);
      const ClassCoef& qa = g.tab[c0][id0];
      const ClassCoef& qb = g.tab[c0 + 1][id1];
      const ClassCoef& qc = g.tab[c0 + 2][id2];
      if (ka == GMES_KIND_CPML)
        cpml_separate<P, c0>(g, l0, xa, d01, d02, f0, qa, pa);
      else if (is_active<0, c0>(g))
        P::st(static_cast<T*>(g.f[c0]) + l0,
              plain_upd<E>(f0, P::cfg(&qa.c1), P::cfg(&qa.c2), d01, d02));
      if (kb == GMES_KIND_CPML)
        cpml_separate<P, c0 + 1>(g, l1, xb, d11, d12, f1, qb, pb);
      else if (is_active<0, c0 + 1>(g))
        P::st(static_cast<T*>(g.f[c0 + 1]) + l1,
              plain_upd<E>(f1, P::cfg(&qb.c1), P::cfg(&qb.c2), d11, d12));
      if (kc == GMES_KIND_CPML)
        cpml_separate<P, c0 + 2>(g, l2, xq, d21, d22, f2, qc, pc);
      else if (is_active<0, c0 + 2>(g))
        P::st(static_cast<T*>(g.f[c0 + 2]) + l2,
              plain_upd<E>(f2, P::cfg(&qc.c1), P::cfg(&qc.c2), d21, d22));
      return;
    }
  }
  if constexpr (SIDE == 0) {
    const int xc[3] = {i, j, k};
    const Pre<P> pa = pre_of<P, 0, false>(g, l0, xc, id0);
    const Pre<P> pb = pre_of<P, 1, false>(g, l1, xc, id1);
    const Pre<P> pc = pre_of<P, 2, false>(g, l2, xc, id2);
    upd<P, 0, false, DISP>(g, l0, xc, d01, d02, f0, id0, pa);
    upd<P, 1, false, DISP>(g, l1, xc, d11, d12, f1, id1, pb);
    upd<P, 2, false, DISP>(g, l2, xc, d21, d22, f2, id2, pc);
  } else {
    const int x3[3] = {i, j + 1, k + 1}, x4[3] = {i + 1, j, k + 1}, x5[3] = {i + 1, j + 1, k};
    const Pre<P> pa = pre_of<P, 3, false>(g, l0, x3, id0);
    const Pre<P> pb = pre_of<P, 4, false>(g, l1, x4, id1);
    const Pre<P> pc = pre_of<P, 5, false>(g, l2, x5, id2);
    upd<P, 3, false, false>(g, l0, x3, d01, d02, f0, id0, pa);
    upd<P, 4, false, false>(g, l1, x4, d11, d12, f1, id1, pb);
    upd<P, 5, false, false>(g, l2, x5, d21, d22, f2, id2, pc);
  }
}

// The ghost images of own point l of component C, cell x (gmes/fdtd.py:
// 811-1097): an E point at index 0 along a transverse axis is copied to that
// axis' last plane, an H point at the last index to plane 0, points on two
// such planes also to the corner; complex grids (CX: the real plane, gi the
// imaginary one) multiply by the phase of each axis in the order own+1, own+2.
// all: also the planes that no active component's curl reads.
template <class P, int C, bool CX>
__device__ __forceinline__ void ghost_images(const GridDev& g, const GridDev& gi, const int x[3],
                                             int l, bool all) {
  using T = typename P::T;
  constexpr int own = C % 3, a1 = (own + 1) % 3, a2 = (own + 2) % 3;
  constexpr bool E = C < 3;
  bool b1 = E ? x[a1] == 0 : x[a1] == g.n[a1] - 1;
  bool b2 = E ? x[a2] == 0 : x[a2] == g.n[a2] - 1;
  // the ghost plane along a1 is read by the other half's component along a2
  b1 = b1 && (all || ((g.active >> ((E ? 3 : 0) + a2)) & 1));
  b2 = b2 && (all || ((g.active >> ((E ? 3 : 0) + a1)) & 1));
  if (!b1 && !b2) return;
  const int s1 = a1 == 2 ? 1 : (int)g.fst[own][a1], s2 = a2 == 2 ? 1 : (int)g.fst[own][a2];
  const int d1 = E ? g.n[a1] * s1 : -g.n[a1] * s1, d2 = E ? g.n[a2] * s2 : -g.n[a2] * s2;
  T* f = static_cast<T*>(g.f[C]) + l;
  if constexpr (!CX) {
    const T v = *f;
    if (b1) f[d1] = v;
    if (b2) f[d2] = v;
    if (b1 && b2) f[d1 + d2] = v;
  } else {
    T* fi = static_cast<T*>(gi.f[C]) + l;
    const double vr = *f, vi = *fi;
    double r1 = vr, i1 = vi;
    if (b1) {
      const double pr = g.phase[C][0][0], pi = g.phase[C][0][1];
      r1 = pr * vr - pi * vi;
      i1 = pr * vi + pi * vr;
      f[d1] = r1;
      fi[d1] = i1;
    }
    if (b2) {
      const double pr = g.phase[C][1][0], pi = g.phase[C][1][1];
      f[d2] = pr * vr - pi * vi;
      fi[d2] = pr * vi + pi * vr;
      if (b1) {
        f[d1 + d2] = pr * r1 - pi * i1;
        fi[d1 + d2] = pr * i1 + pi * r1;
      }
    }
  }
}

// ghost_images of the three own points of one half at cell (i, j, k).
template <class P, int SIDE, int MASK, bool CX>
__device__ __forceinline__ void ghost_cell(const GridDev& g, const GridDev& gi, int i, int j,
                                           int k, bool all) {
  const bool edge = SIDE == 0 ? (i == 0 || j == 0 || k == 0)
                              : (i == g.n[0] - 1 || j == g.n[1] - 1 || k == g.n[2] - 1);
  if (!edge) return;
  const int X0 = (int)g.fst[0][0], X1 = (int)g.fst[0][1], Y0 = (int)g.fst[1][0];
  const int Z0 = (int)g.fst[2][0], Z1 = (int)g.fst[2][1];
  constexpr int c0 = 3 * SIDE;
  const int l0 = i * X0 + (j + SIDE) * X1 + k + SIDE;
  const int l1 = (i + SIDE) * Y0 + j * X1 + k + SIDE;
  const int l2 = (i + SIDE) * Z0 + (j + SIDE) * Z1 + k;
  const int x[3] = {i, j, k};
  if (is_active<MASK, c0>(g)) ghost_images<P, c0, CX>(g, gi, x, l0, all);
  if (is_active<MASK, c0 + 1>(g)) ghost_images<P, c0 + 1, CX>(g, gi, x, l1, all);
  if (is_active<MASK, c0 + 2>(g)) ghost_images<P, c0 + 2, CX>(g, gi, x, l2, all);
}

// ghost_images of component c's own point alone.
template <class P, bool CX>
__device__ __forceinline__ void ghost_own(const GridDev& g, const GridDev& gi, int c,
                                          const int x[3], int l) {
  switch (c) {
    case 0: ghost_images<P, 0, CX>(g, gi, x, l, true); break;
    case 1: ghost_images<P, 1, CX>(g, gi, x, l, true); break;
    case 2: ghost_images<P, 2, CX>(g, gi, x, l, true); break;
    case 3: ghost_images<P, 3, CX>(g, gi, x, l, true); break;
    case 4: ghost_images<P, 4, CX>(g, gi, x, l, true); break;
    case 5: ghost_images<P, 5, CX>(g, gi, x, l, true); break;
  }
}

// Point sources of one half-step (gmes/pw_source.py:74-131), applied after
// that half's material update.  `v` has been computed on the host in FP64.
template <class P, bool STRICT>
__device__ __forceinline__ void source_point(const GridDev& g, int side, int64_t slot, int q) {
  const gmes_point_source ps = g.src[q];
  // the table is caller-provided device memory: skip entries that do not
  // name a point of an active component
  if (ps.comp < 0 || ps.comp > 5 || !(g.active & (1 << ps.comp))) return;
  if (ps.offset < 0 || ps.offset >= g.npts[ps.comp]) return;
  if ((ps.comp < 3) != (side == 0)) return;
  const double v = g.src_val[slot * g.nsrc + q];
  using T = typename P::T;
  T* f = static_cast<T*>(g.f[ps.comp]) + ps.offset;
  if (ps.mode == 0) {
    P::st(f, P::from_double(v));
  } else if constexpr (STRICT) {
    *reinterpret_cast<double*>(f) = __dsub_rn(*reinterpret_cast<double*>(f), v);
  } else {
    P::st(f, P::ldw(f) - P::from_double(v));
  }
}

}  // namespace
}  // namespace gmes
