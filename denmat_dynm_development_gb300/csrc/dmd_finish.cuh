// The finish of one state (nb = 2 or 4, the window the whole density matrix) with one thread per element of
// rho_k, and the preparation of the next RK4 stage in the same kernel.
//
// Why. k_finish gives a k-point one thread, whose chain of some 150 to 400 FP64 operations runs at one result per
// 19 clocks and SM (the FP64 pipe) however few k-points there are: 9 us for 500 k-points, 17 us with a
// coherent term, 45 us for nb = 4. Here nb^2 lanes share a k-point and exchange operands by shuffles, blocks are one
// warp (with the next stage's phases two) so that small systems spread over the SMs, and H(t)'s phases are the prep's. Element by element the
// operations and their order are k_finish's. With the next stage's input in registers the same lanes write its
// coordinates (k_prep_herm's values), reset the sums they have just read and form the phases of the next time,
// which saves the prep launch of every stage.
#pragma once
#include "dmd_kernels.cuh"
#include "dmd_pairs_cb.cuh"

namespace dmd {

// the next evaluation's coordinates, as k_prep_herm's arguments of the same names
struct NextPrep {
  void* rs;              // relem: Hermitian part [nk][2][NB2], then the anti-Hermitian part
  double2* acc;
  const double2* acc0;
  double2* ph;           // phases, replaced by the next time's
  const double* fref;    // deviation and linearized forms
  unsigned int* hflag;   // the next evaluation's flag (FinishArgs::hflag: this one's)
  int phase, lin;
  int same_time;         // the next time is this evaluation's: its phases stay
  TimeArg ta;
};

// A stage of the RKF45 step: its slope goes to slot FinishArgs::stage of K and the next stage's input (the last stage:
// the new y, in place, and the error ratio) is formed from the slopes so far
struct RkfStage {
  RkComb next, err;
  int last;
  double eps_abs, eps_rel;
  unsigned long long* rmax;
};

template <int NB>
__device__ __forceinline__ double2 group_get(double2 v, int lane) {
  return mk2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// A: coordinate type of the next evaluation (PREP); RKF: stages of the RKF45 step instead of RK4's
template <int NB, typename A, bool PREP, bool RKF = false>
__global__ void __launch_bounds__(PREP ? 64 : 32) k_finish_el(FinishArgs a, NextPrep p, RkfStage r) {
  constexpr int NB2 = NB * NB;
  __shared__ double2 next_d[PREP ? 32 : 1];
  const int lane = threadIdx.x & 31, e = lane % NB2, i = e / NB, j = e % NB, g0 = lane - e;  // group's first lane
  const int ji = j * NB + i, tl = g0 + ji;                                             // the transposed element's lane
  const int kl = (blockIdx.x * 32 + lane) / NB2;
  const bool live = kl < a.nk;  // dead groups still take part in the shuffles
  const int k = live ? kl : a.nk - 1;
  const size_t el = (size_t)k * NB2 + e;
  const bool new_ph = PREP && p.phase && !p.same_time;
  if (PREP && threadIdx.x >= 32) {  // second warp: the next phases
    if (!new_ph) return;
    double2 dk = mk2(1.0, 0.0);
    if (i < j) dk = ccis((a.ew[(size_t)k * NB + i] - a.ew[(size_t)k * NB + j]) * eval_time(p.ta));
    next_d[lane] = dk;
    __syncthreads();  // (and the first warp has read this evaluation's)
    if (live && i <= j) p.ph[el] = dk;
    if (live && i < j) p.ph[(size_t)k * NB2 + ji] = cconj(dk);
    return;
  }
  if (a.hflag && blockIdx.x == 0 && lane == 0) *a.hflag = 0u;  // every pair launch of this evaluation has completed
  const double t = eval_time(a.ta);
  const double2 y = a.y[el];
  const double2 d = (a.want_eph && a.ph && i != j) ? a.ph[el] : mk2(1.0, 0.0);  // D_k(i, j)
  double2 f = mk2(0.0, 0.0);
  // herm_up of the matrix spread over the group: this lane's element, read through the upper triangle
  auto upper = [&](double2 v) {
    const double2 o = group_get<NB>(v, tl);
    return i == j ? mk2(v.x, 0.0) : (i < j ? v : cconj(o));
  };

  // coherent term: -i [H(t), rho] (DenMat.cpp:29-55)
  if (a.want_coh) {
    const double* ek = a.edm + (size_t)k * NB;
    if (a.H) {
      double2 Ht = a.H[el];
      if (a.picture == 0 && i != j) Ht = cmul_rn(Ht, (a.want_eph && a.ph) ? d : ccis((ek[i] - ek[j]) * t));
      const double2 hu = upper(Ht);
      double2 s1 = mk2(0.0, 0.0), s2 = mk2(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < NB; ++l) {
        const double2 yil = group_get<NB>(y, g0 + i * NB + l), hlj = group_get<NB>(hu, g0 + l * NB + j);
        s1 = cadd_rn(s1, cmul_rn(yil, hlj));
      }
#pragma unroll
      for (int l = 0; l < NB; ++l) {
        const double2 hil = group_get<NB>(hu, g0 + i * NB + l), ylj = group_get<NB>(y, g0 + l * NB + j);
        s2 = cadd_rn(s2, cmul_rn(hil, ylj));
      }
      const double2 c1 = cmul_rn(mk2(1.0, 0.0), s1);
      const double2 o = cadd_rn(cmul_rn(mk2(1.0, 0.0), s2), cmul_rn(mk2(-1.0, 0.0), c1));
      f = cadd_rn(mk2(0.0, 0.0), cmul_rn(o, mk2(0.0, -1.0)));
    } else if (a.picture == 1) {  // commutator_mat_diag(C, e, dm, nb, -i)
      const double2 c = mk2(-__dmul_rn(y.x, ek[j]), -__dmul_rn(y.y, ek[j]));
      f = cadd_rn(mk2(0.0, 0.0), cmul_rn(cadd_rn(c, cmul_rn(mk2(ek[i], 0.0), y)), mk2(0.0, -1.0)));
    }
  }

  // scattering finish (evolve_eph.cpp:140-162, evolve_driver :21-32)
  const size_t ax = (size_t)(a.pos ? a.pos[k] : k) * 2 * NB2 + e;
  if (a.want_eph) {
    double2 X = a.acc[ax], Y = a.acc[ax + NB2];
    if (a.herm) {  // X = (M^H)^-1 X': X_ij = (X'_ij + i X'_ji) / 2, X_ji = (X'_ij - i X'_ji) / 2 for i < j
      const double2 xo = group_get<NB>(X, tl), yo = group_get<NB>(Y, tl);
      if (i < j) {
        X = mk2(0.5 * (X.x - xo.y), 0.5 * (X.y + xo.x));
        Y = mk2(0.5 * (Y.x - yo.y), 0.5 * (Y.y + yo.x));
      } else if (i > j) {
        X = mk2(0.5 * (xo.x + X.y), 0.5 * (xo.y - X.x));
        Y = mk2(0.5 * (yo.x + Y.y), 0.5 * (yo.y - Y.x));
      }
    }
    double2 Pdm = X, dmP = Y;
    if (a.phase && i != j) {
      Pdm = cmul_rn(d, X);
      dmP = cmul_rn(d, Y);
    }
    double2 c;
    if (a.lin) {
      c = Pdm;
    } else {
      // c = (1 - dm) Pdm - dm1P dm (zhemm Left alpha 1 beta 0, then zhemm Right alpha -1 beta 1)
      const double2 su = upper((i == j) ? mk2(1.0 - y.x, 0.0 - y.y) : mk2(-y.x, -y.y)), ru = upper(y);
      c = mk2(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < NB; ++l)
        c = cfma(group_get<NB>(su, g0 + i * NB + l), group_get<NB>(Pdm, g0 + l * NB + j), c);
#pragma unroll
      for (int l = 0; l < NB; ++l) {
        const double2 m = group_get<NB>(dmP, g0 + i * NB + l);
        c = cfma(mk2(-m.x, -m.y), group_get<NB>(ru, g0 + l * NB + j), c);
      }
    }
    // (prefac/2)(c + c^dagger); the (j, i) element is the exact conjugate of the (i, j) one
    const double pf = a.prefac * 0.5;
    const double2 co = group_get<NB>(c, tl);
    double2 u = i <= j ? cscale_rn(pf, cadd_rn(c, cconj(co))) : cconj(cscale_rn(pf, cadd_rn(co, cconj(c))));
    if (a.eq) {
      const double2 q = a.eq[el];
      if (i == j || a.picture == 1) u = csub_rn(u, q);
      else u = csub_rn(u, cmul_rn(q, a.ph ? d : ccis((a.ew[(size_t)k * NB + i] - a.ew[(size_t)k * NB + j]) * t)));
    }
    f = cadd_rn(f, u);
  }

  if (a.mode == 0) {
    if (live) a.out[el] = f;
    return;
  }
  const size_t n = (size_t)a.nk * NB2;
  const double h = RKF ? 0.0 : a.tref[1];
  double2 yn = y;
  if (RKF) {
    auto slope = [&](int s) { return s == a.stage ? f : a.K[(size_t)s * n + el]; };
    const double2 yb = a.ybase[el];
    yn = mk2(__dadd_rn(yb.x, r.next([&](int s) { return slope(s).x; })),
             __dadd_rn(yb.y, r.next([&](int s) { return slope(s).y; })));
    if (live) {
      a.K[(size_t)a.stage * n + el] = f;
      (r.last ? a.ybase : a.ytmp)[el] = yn;
    }
    if (r.last) {
      const double ex = rk_ratio(r.err([&](int s) { return slope(s).x; }), yn.x, r.eps_abs, r.eps_rel);
      const double ey = rk_ratio(r.err([&](int s) { return slope(s).y; }), yn.y, r.eps_abs, r.eps_rel);
      rk_max(live ? fmax(ex, ey) : 0.0, r.rmax);
    }
  } else if (a.mode == 2) {  // update_dm_euler: dm += 0.5*dt*(ddmdt + ddmdt^dagger)
    const double2 fo = group_get<NB>(f, tl);
    yn = cadd_rn(a.ybase[el], cscale_rn(0.5 * h, cadd_rn(f, cconj(fo))));
    if (live) a.ybase[el] = yn;
    return;
  } else if (a.stage < 3) {
    const double2 yb = a.ybase[el];
    yn = cadd_rn(yb, cscale_rn(a.stage == 2 ? h : 0.5 * h, f));
    if (live) {
      a.K[(size_t)a.stage * n + el] = f;
      a.ytmp[el] = yn;
    }
  } else {
    const double h6 = h / 6.0;
    const double2 yb = a.ybase[el];
    const double2 k1 = a.K[el], k2 = a.K[n + el], k3 = a.K[2 * n + el];
    // y + h/6 * (k1 + 2 k2 + 2 k3 + k4), evaluated left to right
    const double sx = __dadd_rn(__dadd_rn(__dadd_rn(k1.x, __dmul_rn(2.0, k2.x)), __dmul_rn(2.0, k3.x)), f.x);
    const double sy = __dadd_rn(__dadd_rn(__dadd_rn(k1.y, __dmul_rn(2.0, k2.y)), __dmul_rn(2.0, k3.y)), f.y);
    yn = mk2(__dadd_rn(yb.x, __dmul_rn(h6, sx)), __dadd_rn(yb.y, __dmul_rn(h6, sy)));
    if (live) {
      a.K[3 * n + el] = f;
      a.ybase[el] = yn;
    }
  }
  if constexpr (PREP) {
    const double2 vo = group_get<NB>(yn, tl);  // the transposed element
    if (new_ph) __syncthreads();
    if (!live) return;
    typedef typename A::relem V;
    p.acc[ax] = p.acc0 ? p.acc0[ax] : mk2(0.0, 0.0);
    p.acc[ax + NB2] = p.acc0 ? p.acc0[ax + NB2] : mk2(0.0, 0.0);
    V* const rh = (V*)p.rs + (ax - e);
    V* const ra = rh + (size_t)a.nk * 2 * NB2;
    constexpr bool F64C = std::is_same<V, double>::value;
    if (i == j) {
      // H_ii = Re rho_ii, A_ii = Im rho_ii; 1 - rho: (1 - Re rho_ii, -Im rho_ii) (set_oneminusdm)
      if (p.fref) {
        const double dv = __dsub_rn(yn.x, p.fref[(size_t)k * NB + i]);
        rh[e] = A::from_double(dv);
        rh[NB2 + e] = A::from_double(p.lin ? 0.0 : -dv);
      } else {
        rh[e] = A::from_double(yn.x);
        rh[NB2 + e] = A::from_double(1.0 - yn.x);
      }
      ra[e] = A::from_double(yn.y);
      ra[NB2 + e] = A::from_double(p.lin ? 0.0 : 0.0 - yn.y);
      if (yn.y != 0.0) atomicOr(p.hflag, DMD_HFLAG_NONHERM);
      if (F64C && !(isfinite(yn.x) && isfinite(yn.y))) atomicOr(p.hflag, DMD_HFLAG_NONFINITE);
    } else if (i < j) {
      const double2 dn = new_ph ? cconj(next_d[lane]) : p.phase ? cconj(d) : mk2(1.0, 0.0);
      // H_ij = (rho_ij + conj(rho_ji)) / 2, A_ij = (rho_ij - conj(rho_ji)) / (2i); exact for Hermitian rho
      const double2 hij = mk2(__dmul_rn(__dadd_rn(yn.x, vo.x), 0.5), __dmul_rn(__dsub_rn(yn.y, vo.y), 0.5));
      const double2 dif = mk2(__dsub_rn(yn.x, vo.x), __dadd_rn(yn.y, vo.y));
      const double2 r1 = cmul_rn(dn, hij);
      rh[e] = A::from_double(r1.x);
      rh[ji] = A::from_double(r1.y);
      rh[NB2 + e] = A::from_double(p.lin ? 0.0 : -r1.x);
      rh[NB2 + ji] = A::from_double(p.lin ? 0.0 : -r1.y);
      if (F64C && !(isfinite(r1.x) && isfinite(r1.y))) atomicOr(p.hflag, DMD_HFLAG_NONFINITE);
      double2 r2 = mk2(0.0, 0.0);
      if (dif.x != 0.0 || dif.y != 0.0) {  // the anti-Hermitian part is read only when hflag is raised
        atomicOr(p.hflag, DMD_HFLAG_NONHERM);
        r2 = cmul_rn(dn, mk2(__dmul_rn(dif.y, 0.5), __dmul_rn(-dif.x, 0.5)));
      }
      ra[e] = A::from_double(r2.x);
      ra[ji] = A::from_double(r2.y);
      ra[NB2 + e] = A::from_double(p.lin ? 0.0 : -r2.x);
      ra[NB2 + ji] = A::from_double(p.lin ? 0.0 : -r2.y);
    }
  }
}

}  // namespace dmd
