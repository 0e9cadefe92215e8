// Device physics of the Stokes synthesis path (sm_100a).
//
//  * FP64, one warp per column, lanes over the 92 elements: partition
//    functions, Saha ionisation equilibrium and the damped electron-density
//    fixed point GET_RHO (src/chemical_equilibrium.f90:165-278, :1601-1701),
//    continuum opacity (src/cont_opacity.f90:48-357), line opacity
//    (src/line_opacity.f90:34-108) and damping (src/damping.f90:842-1012).
//  * FP32, one wavelength: Hui-Armstrong-Wray Voigt/Faraday
//    (src/voigt.f:17-98) and the Landi Degl'Innocenti evolution operator
//    (src/rtesolver.f90:269-473) written on per-layer optical depths
//    (fz_layer2.cuh has the forms of two wavelengths a thread).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define FZ_TABLE_QUAL static __device__ const
#include "fz_tables.h"
#include "fz_pftable.h"

namespace fzd {

// ------------------------------------------------------------------ constants
struct Consts {
  double csaha1, csaha2, rbohr, deno_sa, deno_sam;
  double ab10[FZ_NELEM];   // 10**(ABUND-12)
  // element handled by lane l in slot j of the warp chemistry: lane_elem[32*j+l]
  // (-1 = idle).  Slot 0 holds every element whose partition function has an
  // exponential piece, so slots 1 and 2 never evaluate one; hydrogen is first
  // (lane 0, slot 0 for every L).
  int lane_elem[96];
  double exp2_32[32];   // 2^(j/32), exp_tab's table
};

constexpr double DPI = 3.141592653589793238462643;
constexpr double LIGHT = 2.99792458e+10;
constexpr double KBOL = 1.38056503e-16;
constexpr double MELE = 9.10938215e-28;
constexpr double QELE = 4.80320425e-10;
constexpr double EVOLT = 1.60217656e-12;
constexpr double MAMU = 1.66053892e-24;
constexpr double HPLA = 6.62606957e-27;
constexpr double GRAV = 2.7414e4;
constexpr double KC5THRESHOLD = 2.0e10;   // src/forward.f90:884


// ------------------------------------------------------- partition functions
__device__ __forceinline__ double horner_exact(const double* c, int n, double x) {
  double r = c[n - 1];
  for (int i = n - 2; i >= 0; --i) r = __dadd_rn(c[i], __dmul_rn(x, r));
  return r;
}

__device__ __forceinline__ bool pf_cond(int cond, double th, double T, double u) {
  return cond == 0 || (cond == 1 && T > th) || (cond == 2 && T < th) || (cond == 3 && T <= th) ||
         (cond == 4 && T >= th) || (cond == 5 && u != th);
}

// Horner with fused multiply-adds (the FP64 chemistry kernels evaluate the
// pieces millions of times; the unfused form of horner_exact is kept for the
// per-line opacities, which follow the reference's rounding step by step).
__device__ __forceinline__ double horner6(const double* c, double x) {
  double r = c[5];
  r = fma(x, r, c[4]);
  r = fma(x, r, c[3]);
  r = fma(x, r, c[2]);
  r = fma(x, r, c[1]);
  r = fma(x, r, c[0]);
  return r;
}

// U_I, U_II, U_III of element zn (1-based), src/atom_database.f90:121-1035
// (generated piece table; branchy, used outside the warp chemistry).
__device__ __forceinline__ double pf_vpiece(const fz_pf_vpiece& p, const double var[3]) {
  const double h = horner_exact(p.c, p.nc, var[p.var]);
  if (p.form == 1) return p.base + exp(h);
  if (p.form == 2) return fmax(p.clamp, h);
  return h;
}

__device__ __forceinline__ void partition_u(int zn, double T, const double var[3], double U[3]) {
  const int e = zn - 1;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int nv = fz_tab_pf_nv[e][s];
    int act = -1;
    for (int i = 0; i < nv; ++i)
      if (pf_cond(fz_tab_pf_v[e][s][i].cond, fz_tab_pf_v[e][s][i].th, T, 0.0)) act = i;
    U[s] = act >= 0 ? pf_vpiece(fz_tab_pf_v[e][s][act], var) : 0.0;
  }
}

// 1/y to ~1 ulp: the hardware approximation (relative error below 1e-6)
// corrected by one third-order (Halley) step, whose own error is its cube:
// three FMAs, one fewer in number and in the dependent chain than two Newton
// steps (measured over 2^20 values of 400 binades: at most 2.3e-16).
__device__ __forceinline__ double rcp_d(double y) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(y));
  const double e = fma(-y, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// exp_tab's constants, read as operands from the constant bank: 1.5 * 2^52
// (the sum's low word is the rounded integer), 32 / ln 2, ln 2 / 32 in two
// parts (the first with its low 20 bits zero, so n times it is exact), 1/6!,
// 1/5!, 1/4!, 1/3!.
__constant__ double EXP_C[8] = {6755399441055744.0, 46.16624130844683, -0.021660849390173098, -2.325192846878874e-12,
                                1.0 / 720.0, 1.0 / 120.0, 1.0 / 24.0, 1.0 / 6.0};

// exp(x) to ~1 ulp by the table method (Tang, ACM TOMS 15, 1989): x =
// n ln2/32 + r, exp(x) = 2^(n/32) (1 + r + ... + r^6/720), the 32 fractional
// powers of two from a table (in shared memory).  11 FP64 operations, for
// |x| <= 700 (NaN gives NaN); with CUT, larger |x| ends at 2^+-1020.
template <bool CUT>
__device__ __forceinline__ double exp_tab(double x, const double* __restrict__ tab) {
  const double t = fma(x, EXP_C[1], EXP_C[0]);
  const int n = __double2loint(t);
  const double nd = t - EXP_C[0];
  const double r = fma(nd, EXP_C[3], fma(nd, EXP_C[2], x));
  double q = fma(r, EXP_C[4], EXP_C[5]);
  q = fma(r, q, EXP_C[6]);
  q = fma(r, q, EXP_C[7]);
  q = fma(r, q, 0.5);
  q = fma(__dmul_rn(r, r), q, r);
  const double s = tab[n & 31];
  const double v = fma(s, q, s);
  const int m = CUT ? min(max(n >> 5, -1020), 1020) : n >> 5;
  return __hiloint2double(__double2hiint(v) + (m << 20), __double2loint(v));
}

// exp(x) of any x: the table method, replaced by exp() outside its range (the
// high word orders the magnitudes; infinities and NaN take exp()).  The rare
// branch comes last, so that the code around can be scheduled into the rest.
__device__ __forceinline__ double exp_any(double x, const double* __restrict__ tab) {
  double v = exp_tab<true>(x, tab);
  if ((__double2hiint(x) & 0x7fffffff) >= 0x4085e000) v = exp(x);
  return v;
}

// --------------------------------------------------------- warp chemistry
// One column's chemistry on a group of L lanes (L = 32: a warp; L = 16: a
// half-warp, two columns per warp), lanes over the elements: the element of
// lane l in slot j is lane_elem[L*j + l], NS = 96 / L slots per lane.  The
// exponential-form elements come first in lane_elem (after hydrogen), so
// only the first 32 / L slots of a lane (the first 32 of the 96) evaluate an
// exponential.
//
// An element's Saha factors enter GET_RHO as alpha_II and the product
// alpha_I alpha_II (a2 and c): see get_rho_warp.
template <int L>
struct WarpSahaT {
  static constexpr int NS = 96 / L;
  double T, kt, idkt;   // T, k T, 1 / (DENO_SA k T)
  double a2[NS], c[NS];
};
using WarpSaha = WarpSahaT<32>;

__device__ __forceinline__ double clamp650(double e) {
  if (e > 0.0) e = fmin(e, 650.0);
  if (e < 0.0) e = fmax(e, -650.0);
  return e;
}

// The same limits by the magnitude's high word (no FP64 compare).
__device__ __forceinline__ double cut650(double e) {
  return (__double2hiint(e) & 0x7fffffff) < 0x40845000 ? e : copysign(650.0, e);
}

// The temperature terms the Saha factors of every element share: 1/T,
// T^(-3/2) x CSAHA1 / 2 and the partition functions' variables (T, T/1000,
// log(5040/T)).
struct SahaT {
  double it, hl, var[3];
};

__device__ __forceinline__ SahaT saha_t(double T, const Consts& K) {
  SahaT t;
  t.it = rcp_d(T);
  t.hl = __dmul_rn(0.5 * K.csaha1, __dmul_rn(t.it, sqrt(t.it)));
  t.var[0] = T;
  t.var[1] = 1.0e-3 * T;
  t.var[2] = log(5040.0 / T);
  return t;
}

// The condition of a value piece on T: the generated table holds none
// (piece 0), T > th (1) and T < th (2) only (checked when a context is made).
__device__ __forceinline__ bool piece_on(int cond, double th, double T) { return cond == 1 ? T > th : T < th; }

// (alpha_II, alpha_I alpha_II) of one element from its partition functions
// and the two Boltzmann factors (SHORT_PRE_ION_CALC_TEMPRHO,
// src/chemical_equilibrium.f90:1601-1652: alpha_I = U_I / (2 U_II) lambda e1,
// alpha_II = U_II / (2 U_III) lambda e2; U_II cancels in the product, so one
// reciprocal serves both).  Products only, rounded one by one, so that every
// kernel that forms them gets the same bits.
__device__ __forceinline__ double2 saha_factors(double u0, double u1, double u2, double e1, double e2, double hl) {
  const double w = __dmul_rn(__dmul_rn(hl, rcp_d(u2)), e2);
  return make_double2(__dmul_rn(u1, w), __dmul_rn(__dmul_rn(__dmul_rn(u0, hl), e1), w));
}

// The bound of a value piece's second form: the base of base + exp(h), the
// lower limit of max(clamp, h), and a limit that never holds for h alone.
__device__ __forceinline__ double piece_bc(int form, double base, double clamp) {
  return form == 1 ? base : (form == 2 ? clamp : -1.0e300);
}

// U of a value piece at its variable x (Horner, then the piece's form).
template <bool EXPF>
__device__ __forceinline__ double piece_value(const double c[6], double x, bool expo, double bc,
                                              const double* __restrict__ tab) {
  const double h = horner6(c, x);
  if (EXPF && expo) return bc + exp_tab<true>(h, tab);
  return h < bc ? bc : h;
}

// The Saha factors of element el at one temperature (an idle slot, -1, gets
// hydrogen's: its abundance is 0).  EXPF: the element's pieces may hold an exponential.
template <bool EXPF>
__device__ __forceinline__ double2 saha_elem(int el, const SahaT& t, const Consts& K, const PFTable* __restrict__ tb) {
  const int e = el < 0 ? 0 : el;
  const double T = t.var[0];
  double u[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int nv = tb->nv[e][s];
    int act = 0;
#pragma unroll
    for (int i = 1; i < FZ_PF_MAXV; ++i)
      if (i < nv && piece_on(__ldg(&tb->p[e][s][i].cond), __ldg(&tb->p[e][s][i].th), T)) act = i;
    const PFPiece* p = &tb->p[e][s][act];
    double c[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) c[i] = __ldg(&p->c[i]);
    const int form = __ldg(&p->form), v = __ldg(&p->var);
    u[s] = piece_value<EXPF>(c, v == 0 ? t.var[0] : (v == 1 ? t.var[1] : t.var[2]), form == 1,
                             piece_bc(form, __ldg(&p->base), __ldg(&p->clamp)), K.exp2_32);
  }
  const double e1 = exp_tab<false>(cut650(__dmul_rn(K.csaha2 * fz_tab_xi[e], t.it)), K.exp2_32);
  const double e2 = exp_tab<false>(cut650(__dmul_rn(K.csaha2 * fz_tab_xii[e], t.it)), K.exp2_32);
  return saha_factors(u[0], u[1], u[2], e1, e2, t.hl);
}

// The scalars of GET_RHO that depend on the temperature alone.
template <int L>
__device__ __forceinline__ void saha_scalars(WarpSahaT<L>& w, double T, const Consts& K) {
  w.T = T;
  w.kt = __dmul_rn(KBOL, T);
  w.idkt = rcp_d(__dmul_rn(K.deno_sa, w.kt));
}

// Per-lane Saha factors of the lane's elements at temperature T.
template <int L>
__device__ __forceinline__ void saha_prepare(WarpSahaT<L>& w, double T, const Consts& K,
                                             const PFTable* __restrict__ tb, int lane) {
  constexpr int NS = WarpSahaT<L>::NS;
  constexpr int NEXP = 32 / L;   // the lane's slots among the first 32
  saha_scalars(w, T, K);
  const SahaT t = saha_t(T, K);
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int el = K.lane_elem[L * j + lane];
    const double2 f = j < NEXP ? saha_elem<true>(el, t, K, tb) : saha_elem<false>(el, t, K, tb);
    w.a2[j] = f.x;
    w.c[j] = f.y;
  }
}

// One FP64 tensor-core product D = A B (8x4 by 4x8): a lane holds A(lane/4,
// lane%4) and B(lane%4, lane/4) and gets D(lane/4, 2 (lane%4) + {0, 1}).
__device__ __forceinline__ void dmma(double a, double b, double& d0, double& d1) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
      : "=d"(d0), "=d"(d1)
      : "d"(a), "d"(b), "d"(0.0));
}

// Sum over the L lanes of a group, the same bits in each of them.  L = 32:
// two tensor-core products with ones (the 8 sums of 4 lanes, two of them to
// each lane; their pair's sum; the sum of the 4 pairs), 69 cycles of latency
// against 195 for five shuffle levels -- this form serves the small batches,
// which wait for their chains.  L = 16 serves full batches, where a product's
// 16 FP64 pipe cycles would cost more than the shuffles.
template <int L>
__device__ __forceinline__ double group_sum(double v, unsigned mask) {
  if (L == 32) {
    double d0, d1;
    dmma(1.0, v, d0, d1);
    dmma(d0 + d1, 1.0, d0, d1);
    return d0;
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// The lanes of this thread's group of L.
template <int L>
__device__ __forceinline__ unsigned group_mask() {
  return L == 32 ? 0xffffffffu : (((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1)));
}

struct RhoOut {
  double nhyd, pelec, dens;
  int status;
};

// MOLECW of a GET_RHO result at gas pressure PG (ipg = 1/PG).
__device__ __forceinline__ double rho_molecw(const RhoOut& r, double kt, double ipg) {
  return ((r.dens * kt) * (1.0 / MAMU)) * ipg;
}

// GET_RHO, src/chemical_equilibrium.f90:165-278.  All lanes of the group
// call it with the same arguments; nelec (the warm-start chain) is updated in
// every lane identically.  The electron sum of SHORT_ION_CALC_TEMPRHO
// (:1659-1701), NELEC_EST = N_H+ - N_H- + sum_{Z>1} (N_II + N_III), is
// evaluated per element as ab*(1+y)/(1+y+xy) (hydrogen: ab*(1-xy)/(1+y+xy))
// with x = ne*alpha_I, y = ne*alpha_II: algebraically the reference's three
// quotients.  With a2 = alpha_II and c = alpha_I alpha_II that is two FMAs
// for numerator and denominator, one reciprocal (three FMAs), a product and
// the accumulating FMA: 7 FP64 operations an element and iteration (12 with
// x, y and two Newton steps).  ab[j] = 10**(ABUND-12) of the lane's elements
// (0 past element 92); hydrogen is lane 0's slot 0.
//
// pgf() gives PG.  EARLY: the sum at the starting NELEC, which does not depend on
// it, is formed first, so that Pg's exponential and what leads up to it run
// beside the sum instead of ahead of it -- for hydrostatic chains of a warp a
// column, where latency counts (one column of 128 heights 0.439 -> 0.405 ms; with
// 16 lanes the second copy of the sum costs 3 %).  Same bits either way.
template <bool EARLY, int L, class F>
__device__ __forceinline__ RhoOut get_rho_warp(const WarpSahaT<L>& w, const double ab[WarpSahaT<L>::NS], F pgf,
                                               double& nelec, const Consts& K, int lane) {
  constexpr int NS = WarpSahaT<L>::NS;
  const unsigned mask = group_mask<L>();
  RhoOut r;
  const double T = w.T;
  auto sum = [&](double ne) {
    const double ne2 = ne * ne;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      double num = fma(ne, w.a2[j], 1.0);
      const double den = fma(ne2, w.c[j], num);
      if (j == 0 && lane == 0) num = fma(-ne2, w.c[j], 1.0);   // hydrogen: N_H+ - N_H-
      if (j & 1)
        s1 = fma(ab[j] * num, rcp_d(den), s1);
      else
        s0 = fma(ab[j] * num, rcp_d(den), s0);
    }
    return group_sum<L>(s0 + s1, mask);
  };
  double s = EARLY ? sum(nelec) : 0.0, nhyd = 0.0;
  const double PG = pgf();
  bool again = !EARLY;
  if (!(nelec >= 1.0)) {   // NaN counts as 0
    nelec = PG / (101.0 * KBOL * T);
    again = true;
  }
  const double pelec = nelec * KBOL * T;
  if (pelec > PG) {
    nelec = (PG * 0.5) / (KBOL * T);
    again = true;
  }
  int iter = 1;
  double nnew = nelec;
  const double kt = w.kt, idkt = w.idkt;
  while (true) {
    if (again) s = sum(nnew);
    again = true;
    const double nold = nnew;
    nhyd = fma(-nnew, kt, PG) * idkt;
    // (max(EST, 0) + NOLD) / 2 with EST = nhyd s (a NaN estimate counts as 0)
    const double half = 0.5 * nold, v = fma(0.5 * nhyd, s, half);
    nnew = v > half ? v : half;
    iter = iter + 1;
    // ERROR = |(NEW-OLD)/NEW| > 1e-4, ITER <= 100, NHYD >= 0
    if (!(fabs(nnew - nold) > 1.0e-4 * fabs(nnew) && iter <= 100 && nhyd >= 0.0)) break;
  }
  r.status = 0;
  if (iter >= 100 || nhyd < 0.0) r.status = 1;
  nelec = nnew;
  nhyd = fma(-nelec, kt, PG) * idkt;
  r.dens = fma(nhyd, K.deno_sam, nelec * MELE);
  if (nhyd != nhyd || nnew != nnew) r.status = 2;
  if (nelec < 0.0 || nhyd <= 0.0) r.status = 1;
  r.nhyd = nhyd;
  r.pelec = pelec;   // pressure of the initial guess, as the reference returns it
  return r;
}

// ----------------------------------------------------- continuum opacity
// OPAC_CONTINUUM, src/cont_opacity.f90:305-357, with every factor that
// depends only on the wavelength precomputed on the host (ContP):
//   H- free-free  (:48-120):  1e-29 k ne T sum_i c_i theta^(1+i/2)
//   H- bound-free (:124-181): T^-2.5 e^(a1/T) (1 - e^(-a2/T)) sigma ne k T
//   Thomson (:187-217), Rayleigh (:221-239), neutral H bf/ff (:243-301).
struct ContP {
  int nff, n0, pad0, pad1;
  double ffc[6];
  double sbf, bfa1, bfa2;        // sigma_bf (0 if lambda >= 1.6419 um), ALPHA/LAMBDAP, ALPHA/lambda_um
  double hpre, c3l, c4, ray;     // C2 lambda^3, C3/lambda, C4, Rayleigh
  double ct;                     // Thomson constant
};

__device__ __forceinline__ double opac_continuum(double T, double ne, double nh, const ContP& c) {
  const double th = 5040.0 / T;
  const double sq = sqrt(th);
  const double th2 = th * th;
  double part1 = c.ffc[0] * th + c.ffc[1] * th * sq + c.ffc[2] * th2 + c.ffc[3] * th2 * sq;
  if (c.nff == 6) part1 += c.ffc[4] * th2 * th + c.ffc[5] * th2 * th * sq;
  const double hmff = 1e-29 * part1 * KBOL * ne * T;
  double hmbf = 0.0;
  if (c.sbf != 0.0) {
    const double part = (1.0 / (T * T * sqrt(T))) * exp(c.bfa1 / T) * (1.0 - exp(-c.bfa2 / T));
    hmbf = part * c.sbf * ne * KBOL * T;
  }
  const double thom = c.ct * (ne / nh);
  double sum;
  if (c.n0 <= 8) {
    sum = 0.0;
    for (int i = c.n0; i <= 8; ++i) {
      const double di = (double)i;
      sum += exp(c.c4 / (T * di * di)) / (di * di * di);
    }
    sum += (0.117 + exp(c.c4 / (T * 81.0))) * (T / (2.0 * c.c4));
  } else {
    const double dn = (double)c.n0;
    sum = (0.117 + exp(c.c4 / (T * dn * dn))) * (T / (2.0 * c.c4));
  }
  const double hyd = c.hpre * sum * (1.0 - exp(-c.c3l / T)) * exp(-c.c4 / T);
  return nh * (hmff + hmbf + thom + c.ray + hyd);
}

// ------------------------------------------------------ line opacity, damping
// Per-line constants precomputed on the host.
struct LineP {
  double l0, wdif;
  double term1;      // TERM1 of OPAC_LINE, src/line_opacity.f90:95
  double m2k;        // matom m_u / (2 k): TERM2 = sqrt(m2k / T)
  double chik;       // EPLOW e / k:        TERM4 = exp(-chik / T)
  double hclk;       // h c / (lambda k):   TERM5 = 1 - exp(-hclk / T)
  double nab;        // 10**(ABUND-12)
  double xi_k, xii_k;    // CSAHA2 * XI, XII of the element
  double vdk;        // 2 k / (m_u matom): v_D = sqrt(vdk T)
  double grad;       // radiative damping 0.2223 / lambda^2
  double gc, ge;     // collisional: gamma_col = gc nH T^ge
  double dfac;       // lambda / (4 pi)
  int zn, ion;
};

// OPAC_LINE (LTE) with ION_CALC_TEMPX, src/line_opacity.f90:34-108,
// src/chemical_equilibrium.f90:1511-1597.
__device__ __forceinline__ double opac_line(const LineP& L, double T, double ne, double nh, const Consts& K) {
  const double var[3] = {T, 1.0e-3 * T, log(5040.0 / T)};
  double U[3];
  partition_u(L.zn, T, var, U);
  const double lamelec = K.csaha1 / (T * sqrt(T));
  const double al1 = (U[0] / (2.0 * U[1])) * lamelec * exp(clamp650(L.xi_k / T));
  const double al2 = (U[1] / (2.0 * U[2])) * lamelec * exp(clamp650(L.xii_k / T));
  const double deno = ne * ne * al1 * al2 + ne * al2 + 1.0;
  const double nume = L.ion == 1 ? ne * ne * al1 * al2 : (L.ion == 2 ? ne * al2 : 1.0);
  const double npi = nh * L.nab * nume / deno;
  const double t2 = sqrt(L.m2k / T);
  const double t4 = exp(-L.chik / T);
  const double t5 = 1.0 - exp(-L.hclk / T);
  return L.term1 * t2 * (npi / U[L.ion - 1]) * t4 * t5;
}

// GET_DAMPING, src/damping.f90:842-1012: a = (gamma_rad + gamma_col) lambda / (4 pi v_D)
__device__ __forceinline__ double get_damping(const LineP& L, double nh, double T) {
  const double gcol = L.gc * nh * pow(T, L.ge);
  return (L.grad + gcol) * L.dfac / sqrt(L.vdk * T);
}

// ------------------------------------------------------------ FP32 Voigt
// Hui, Armstrong & Wray (1978) 7-pole rational approximation of the complex
// probability function, as src/voigt.f:17-98: H = Re w, F = sign(v) Im w
// with w = P(z)/Q(z) at z = a - i|v|.  P (degree 6) and Q (monic, degree 7)
// have real coefficients, so each is reduced modulo the real quadratic
// (z^2 - 2 Re z z + |z|^2) that z solves (Knuth, TAOCP vol. 2, 4.6.4):
// 2 FMA per degree instead of a complex multiply-add.  Real coefficients also
// make w(conj z) = conj w(z), so z = a - i v gives F with its sign and no
// absolute value.  With P = p1 z + p0, Q = q1 z + q0:
//   H = ((p1 a + p0)(q1 a + q0) + p1 q1 v^2) / |Q|^2,  F = v (p0 q1 - p1 q0) / |Q|^2
// (the quotient by the approximate reciprocal, a few ulp in all, far inside
// the approximation's own error).  Every coefficient carries a factor 2^-62:
// |Q|^2 then stays in range up to |z| = 2e5 and no scaling is computed.
// 38 FMA-pipe operations and one reciprocal a component with its two sums;
// the form with a scaled denominator and Smith's signs took some 50.
__device__ __forceinline__ float rcp_a(float y) {   // 1/y, approximate (1 ulp)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
struct VoigtW {
  float h, f, id;   // H = h id, F = f id
};
__device__ __forceinline__ VoigtW voigt_w(float a, float u) {
  const float K = 2.168404344971009e-19f;   // 2^-62
  const float A0 = 122.607931777104326f * K, A1 = 214.382388694706425f * K, A2 = 181.928533092181549f * K,
              A3 = 93.155580458138441f * K, A4 = 30.180142196210589f * K, A5 = 5.912626209773153f * K,
              A6 = .564189583562615f * K, B0 = 122.60793177387535f * K, B1 = 352.730625110963558f * K,
              B2 = 457.334478783897737f * K, B3 = 348.703917719495792f * K, B4 = 170.354001821091472f * K,
              B5 = 53.992906912940207f * K, B6 = 10.479857114260399f * K;
  const float uu = u * u, r = a + a, s = fmaf(a, a, uu);
  float p1 = A6, p0 = A5, t;
#define FZ_KSTEP(C, hi, lo) \
  t = hi;                   \
  hi = fmaf(r, t, lo);      \
  lo = fmaf(-s, t, (C));
  FZ_KSTEP(A4, p1, p0) FZ_KSTEP(A3, p1, p0) FZ_KSTEP(A2, p1, p0) FZ_KSTEP(A1, p1, p0) FZ_KSTEP(A0, p1, p0)
  float q1 = K, q0 = B6;
  FZ_KSTEP(B5, q1, q0) FZ_KSTEP(B4, q1, q0) FZ_KSTEP(B3, q1, q0) FZ_KSTEP(B2, q1, q0) FZ_KSTEP(B1, q1, q0)
  FZ_KSTEP(B0, q1, q0)
#undef FZ_KSTEP
  const float nr = fmaf(p1, a, p0), dr = fmaf(q1, a, q0), y = q1 * uu;
  VoigtW w;
  w.id = rcp_a(fmaf(q1, y, dr * dr));
  w.h = fmaf(p1, y, nr * dr);
  w.f = u * fmaf(p0, q1, -(p1 * q0));
  return w;
}
__device__ __forceinline__ void voigt_f32(float a, float u, float& H, float& F) {
  const VoigtW w = voigt_w(a, u);
  H = w.h * w.id;
  F = w.f * w.id;
}

// ------------------------------------- FP32 formal solution of one layer
// Weighted least-maximum fits: (e^r - 1 - r) / r^2 on |r| <= ln2/2, (sin r - r) /
// r^3 and (cos r - 1) / r^2 on |r| <= pi/2 (relative error of e^r - 1 below
// 1.7e-8, of the others 1e-8); pi in three parts of few bits.
constexpr float EXP_Q0 = 0.49999997f, EXP_Q1 = 0.166665435f, EXP_Q2 = 0.0416672006f, EXP_Q3 = 0.00836653821f, EXP_Q4 = 0.00138825155f;
constexpr float SIN_Q0 = -0.166666597f, SIN_Q1 = 0.00833306648f, SIN_Q2 = -0.00019809595f, SIN_Q3 = 2.60576121e-06f;
constexpr float COS_Q0 = -0.5f, COS_Q1 = 0.0416666418f, COS_Q2 = -0.00138884038f, COS_Q3 = 2.47618755e-05f, COS_Q4 = -2.60769184e-07f;
constexpr float PI_F_HI = 3.140625f, PI_F_MID = 0.000967502594f, PI_F_LO = 1.50995803e-07f;

// The smaller of two values; NaN if either is.
__device__ __forceinline__ float min_nan(float x, float y) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}

// 1/sqrt(y), approximate.
__device__ __forceinline__ float rsqrt_a(float y) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}

// Evolution operator O of one layer from its optical-depth increments
// t = eta*dz (src/rtesolver.f90:269-473), and om0 = 1 - O(1,1).  The reference's clamp of cosh and
// sinh at 2^53 (-> 1e15, :464-465) is reproduced; below it the operator is
// evaluated with cancellation-free forms (cosh x -+ cos y via sinh^2(x/2),
// sin^2(y/2); lambda_1,2 from the larger root).
// The layer's scalars of the operator: |eta|^2, |rho|^2, eta.rho, their
// difference d, R = theta / 2, the roots x = lambda_1 dz and y = lambda_2
// dz, sign(eta.rho), 1/theta, e^-tI and the hyperbolic / trigonometric
// factors (P = cosh-like, Qm = sinh^2(x/2) + sin^2(y/2), sh = sinh x,
// s2v = sin y, c2v = cos y, ch = cosh x, amb = P - 1).
struct EvolCore {
  float eta2, rho2, er, d, R, x, y, sg, it, E, P, Qm, sh, s2v, c2v, ch, amb;
  bool clamp;
};

__device__ __forceinline__ void evol_core(float tI, float tQ, float tU, float tV, float rQ, float rU, float rV,
                                          EvolCore& c) {
  c.eta2 = tQ * tQ + tU * tU + tV * tV;
  c.rho2 = rQ * rQ + rU * rU + rV * rV;
  c.er = tQ * rQ + tU * rU + tV * rV;
  c.d = c.eta2 - c.rho2;
  c.R = sqrtf(0.25f * c.d * c.d + c.er * c.er);
  if (c.d >= 0.0f) {
    c.x = sqrtf(c.R + 0.5f * c.d);
    c.y = c.x > 0.0f ? fabsf(c.er) / c.x : 0.0f;
  } else {
    c.y = sqrtf(c.R - 0.5f * c.d);
    c.x = c.y > 0.0f ? fabsf(c.er) / c.y : 0.0f;
  }
  c.sg = c.er > 0.0f ? 1.0f : (c.er < 0.0f ? -1.0f : 0.0f);
  const float theta = 2.0f * c.R;
  c.it = theta > 0.0f ? 1.0f / theta : 0.0f;
  c.E = expf(-tI);
  const float XCLAMP = 37.42994775f;   // cosh, sinh >= 2^53 in float64
  c.amb = 0.0f;
  c.s2v = sinf(c.y);
  c.clamp = c.x >= XCLAMP;
  if (c.clamp) {
    const float c2 = cosf(c.y);
    c.P = 0.5f * (1e15f + c2);
    c.Qm = 0.5f * (1e15f - c2);
    c.sh = 1e15f;
    c.ch = 1e15f;
    c.c2v = c2;
  } else {
    const float shx = sinhf(0.5f * c.x), siy = sinf(0.5f * c.y);
    const float a = shx * shx, b = siy * siy;
    c.amb = a - b;
    c.P = 1.0f + c.amb;
    c.Qm = a + b;
    c.sh = sinhf(c.x);
    c.ch = 1.0f + 2.0f * a;
    c.c2v = 1.0f - 2.0f * b;
  }
}

// O and om0 = 1 - O(1,1) from the layer's scalars.
__device__ __forceinline__ void evol_matrix(const EvolCore& c, float tI, float tQ, float tU, float tV, float rQ,
                                            float rU, float rV, float O[16], float& om0) {
  const float x = c.x, y = c.y, sg = c.sg, it = c.it;
  // M2, M3, M4 (Fortran (row,col) -> O[4*(row-1)+(col-1)])
  const float m2_21 = (y * tQ - sg * x * rQ) * it, m2_31 = (y * tU - sg * x * rU) * it,
              m2_41 = (y * tV - sg * x * rV) * it;
  const float m2_32 = (sg * x * tV + y * rV) * it, m2_42 = (-sg * x * tU - y * rU) * it,
              m2_43 = (sg * x * tQ + y * rQ) * it;
  const float m3_21 = (x * tQ + sg * y * rQ) * it, m3_31 = (x * tU + sg * y * rU) * it,
              m3_41 = (x * tV + sg * y * rV) * it;
  const float m3_32 = (-sg * y * tV + x * rV) * it, m3_42 = (sg * y * tU - x * rU) * it,
              m3_43 = (-sg * y * tQ + x * rQ) * it;
  const float m4_11 = (c.eta2 + c.rho2) * it;   // 2*((eta2+rho2)/2)/theta
  const float m4_21 = 2.0f * (tV * rU - tU * rV) * it, m4_31 = 2.0f * (tQ * rV - tV * rQ) * it,
              m4_41 = 2.0f * (tU * rQ - tQ * rU) * it;
  const float m4_22 = 2.0f * (tQ * tQ + rQ * rQ) * it - m4_11, m4_33 = 2.0f * (tU * tU + rU * rU) * it - m4_11,
              m4_44 = 2.0f * (tV * tV + rV * rV) * it - m4_11;
  const float m4_32 = 2.0f * (tQ * tU + rQ * rU) * it, m4_42 = 2.0f * (tV * tQ + rV * rQ) * it,
              m4_43 = 2.0f * (tU * tV + rU * rV) * it;
  const float E = c.E;
  const float eP = E * c.P, eQ = E * c.Qm, eS = E * c.s2v, eH = E * c.sh;
  O[0] = eP + eQ * m4_11;
  // 1 - O(1,1) without cancellation in optically thin layers:
  // (1 - e^-tI) - e^-tI (P - 1 + Qm M4(1,1))
  om0 = c.clamp ? 1.0f - O[0] : -expm1f(-tI) - E * (c.amb + c.Qm * m4_11);
  O[5] = eP + eQ * m4_22;
  O[10] = eP + eQ * m4_33;
  O[15] = eP + eQ * m4_44;
  // (2,1),(1,2): M2,M3 symmetric; M4 antisymmetric
  O[4] = -eS * m2_21 - eH * m3_21 + eQ * m4_21;
  O[1] = -eS * m2_21 - eH * m3_21 - eQ * m4_21;
  O[8] = -eS * m2_31 - eH * m3_31 + eQ * m4_31;
  O[2] = -eS * m2_31 - eH * m3_31 - eQ * m4_31;
  O[12] = -eS * m2_41 - eH * m3_41 + eQ * m4_41;
  O[3] = -eS * m2_41 - eH * m3_41 - eQ * m4_41;
  // (3,2),(2,3): M2,M3 antisymmetric; M4 symmetric
  O[9] = -eS * m2_32 - eH * m3_32 + eQ * m4_32;
  O[6] = eS * m2_32 + eH * m3_32 + eQ * m4_32;
  O[13] = -eS * m2_42 - eH * m3_42 + eQ * m4_42;
  O[7] = eS * m2_42 + eH * m3_42 + eQ * m4_42;
  O[14] = -eS * m2_43 - eH * m3_43 + eQ * m4_43;
  O[11] = eS * m2_43 + eH * m3_43 + eQ * m4_43;
}

}  // namespace fzd
