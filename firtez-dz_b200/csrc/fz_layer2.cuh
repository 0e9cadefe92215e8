// The formal solution of two wavelengths at once in FP32 (sm_100a): a thread's
// two wavelengths sit in the halves of 64-bit registers, and FFMA2 (fma.rn.f32x2)
// runs both in one issue slot at the FP32 pipe's full rate.  Measured on
// dependent chains: 16 FMAs take 17.2 cycles of an SM sub-partition as 8
// FFMA2, 19.3 as 16 FFMA, and with 16 integer operations beside them 19.5
// against 28.6 -- the scalar form's other instructions cost issue slots that
// the packed form has free.  Each half is rounded as the scalar operation is.
#pragma once
#include "fz_physics.cuh"

namespace fzd {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void f2_get(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 operator-(F2 x) {
  float a, b;
  f2_get(x, a, b);
  return f2(-a, -b);
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return a + (-b); }
__device__ __forceinline__ F2 rcp2(F2 x) {
  float a, b;
  f2_get(x, a, b);
  return f2(rcp_a(a), rcp_a(b));
}
__device__ __forceinline__ F2 rsqrt2(F2 x) {
  float a, b;
  f2_get(x, a, b);
  return f2(rsqrt_a(a), rsqrt_a(b));
}

// The terms of voigt_w that a line's components at one height share.
struct VoigtA {
  F2 a, r, aa;   // a, 2 a, a^2
};
__device__ __forceinline__ VoigtA voigt_a(float a) { return VoigtA{f2(a), f2(a + a), f2(a * a)}; }

// voigt_w (fz_physics.cuh) at two arguments u.
__device__ __forceinline__ void voigt_w2(const VoigtA& A, F2 u, F2& h, F2& f, F2& id) {
  const float K = 2.168404344971009e-19f;   // 2^-62
  const float A0 = 122.607931777104326f * K, A1 = 214.382388694706425f * K, A2 = 181.928533092181549f * K,
              A3 = 93.155580458138441f * K, A4 = 30.180142196210589f * K, A5 = 5.912626209773153f * K,
              A6 = .564189583562615f * K, B0 = 122.60793177387535f * K, B1 = 352.730625110963558f * K,
              B2 = 457.334478783897737f * K, B3 = 348.703917719495792f * K, B4 = 170.354001821091472f * K,
              B5 = 53.992906912940207f * K, B6 = 10.479857114260399f * K;
  const F2 uu = u * u, ns = -(uu + A.aa);
  F2 p1 = f2(A6), p0 = f2(A5), t;
#define FZ_KSTEP2(C, hi, lo) \
  t = hi;                    \
  hi = fma2(A.r, t, lo);     \
  lo = fma2(ns, t, f2(C));
  FZ_KSTEP2(A4, p1, p0) FZ_KSTEP2(A3, p1, p0) FZ_KSTEP2(A2, p1, p0) FZ_KSTEP2(A1, p1, p0) FZ_KSTEP2(A0, p1, p0)
  F2 q1 = f2(K), q0 = f2(B6);
  FZ_KSTEP2(B5, q1, q0) FZ_KSTEP2(B4, q1, q0) FZ_KSTEP2(B3, q1, q0) FZ_KSTEP2(B2, q1, q0) FZ_KSTEP2(B1, q1, q0)
  FZ_KSTEP2(B0, q1, q0)
#undef FZ_KSTEP2
  const F2 nr = fma2(p1, A.a, p0), dr = fma2(q1, A.a, q0), y = q1 * uu;
  id = rcp2(fma2(q1, y, dr * dr));
  h = fma2(p1, y, nr * dr);
  f = u * fma2(p0, q1, -(p1 * q0));
}

// e^x = S (1 + p) with S a power of two: the reduction by ln 2 in two parts
// (Cody & Waite, Software Manual for the Elementary Functions, 1980, ch. 6)
// and p = e^r - 1 on |r| <= ln2/2 (weighted least-maximum fit of degree 6,
// relative error 1.7e-8), so that e^x and e^x - 1 both come without
// cancellation; NaN gives NaN.  S is 0 below 2^-126 and 2^127 at most, which
// serves arguments up to 2^22 ln 2 above; further down r leaves its interval
// and p its range, so depths from DEPTH_RARE on are cut to 104 first.
constexpr float DEPTH_RARE = 1.0e12f;
struct ExpF2 {
  F2 S, p;
  __device__ __forceinline__ F2 exp() const { return fma2(S, p, S); }
  __device__ __forceinline__ F2 expm1() const { return fma2(S, p, S + f2(-1.0f)); }
};
// 2^n from t = n + 1.5 * 2^23, cut on the bits of t itself: any float may come
// here, and the difference of its bits to that constant's may leave an int.
__device__ __forceinline__ float exp_scale(float t) {
  const int i = min(max(__float_as_int(t), 0x4b400000 - 127), 0x4b400000 + 127);
  return __int_as_float((i - 0x4b400000 + 127) << 23);
}
// An optical depth, or 104 above it, where e^-x is 0.
__device__ __forceinline__ F2 depth_cut2(F2 x) {
  float a, b;
  f2_get(x, a, b);
  return f2(min_nan(a, 104.0f), min_nan(b, 104.0f));
}
__device__ __forceinline__ ExpF2 exp_parts2(F2 x) {
  const float MAGIC = 12582912.0f;
  const F2 t = fma2(x, f2(1.4426950408889634f), f2(MAGIC)), n = t + f2(-MAGIC);
  const F2 r = fma2(n, f2(-1.428606765330187e-06f), fma2(n, f2(-0.693145751953125f), x));
  F2 q = fma2(r, f2(EXP_Q4), f2(EXP_Q3));
  q = fma2(r, q, f2(EXP_Q2));
  q = fma2(r, q, f2(EXP_Q1));
  q = fma2(r, q, f2(EXP_Q0));
  ExpF2 e;
  e.p = fma2(r * r, q, r);
  float t0, t1;
  f2_get(t, t0, t1);
  e.S = f2(exp_scale(t0), exp_scale(t1));
  return e;
}

// c2 / T at two wavelengths, the quotient corrected by its remainder (rt
// approximately 1/T; T of a slab row, so at least SLAB_TMIN or below 0).
__device__ __forceinline__ F2 planck_q2(F2 c2, float T, float rt) {
  const F2 q0 = c2 * f2(rt);
  return fma2(fma2(-q0, f2(T), c2), f2(rt), q0);
}
// c1 / em1 with em1 = e^(c2/T) - 1 and rm approximately its reciprocal.
__device__ __forceinline__ F2 planck_s2(F2 c1, F2 em1, F2 rm) {
  const F2 s0 = c1 * rm;
  return fma2(fma2(-s0, em1, c1), rm, s0);
}

// The evolution operator of one layer (src/rtesolver.f90:269-473) from its
// optical-depth increments t = eta dz, written on three scalar functions of
// d = |eta|^2 - |rho|^2 and e = eta.rho (x = lambda_1 dz, y = lambda_2 dz with
// sign(x y) = sign(e), x^2 - y^2 = d, x y = e, theta = x^2 + y^2):
//   O = e^-tI { (1 + am) 1 - al X - be Y + ga M }
//   am = (cosh x + cos y) / 2 - 1,  al = (x sinh x + y sin y) / theta,
//   be = (x sin y - y sinh x) / theta,  ga = (cosh x - cos y) / theta,
// where X has the elements of (eta, rho), Y those of (-rho, eta) and M is the
// reference's M4 before its factor 2/theta.  The functions are entire in d
// and e^2: where both are below 1/4 (a layer of optical depth up to about 1/2:
// most of an atmosphere) their series have no quotient by theta and no root;
// above, from the roots, with the reference's clamp of cosh and sinh at 2^53
// (-> 1e15, :464-465).  A half far below the limit beside one above takes the
// series too: the quotients lose its digits as theta goes to 0 (a derivative
// some 1e-7 / theta, at 0 everything); one little below it takes the roots,
// whose code is running.

// From the roots, with what the derivatives need: x, y, 1/theta, sinh x, cosh
// x, sin y, cos y.
struct Roots2 {
  F2 am, al, be, ga, x, y, it, sh, ch, sy, cy;
};
__device__ __forceinline__ Roots2 roots2(F2 d, F2 e) {
  // R = theta / 2 and 1/R, then the larger root and its reciprocal (one Newton
  // step each: about 1 ulp)
  float d0, d1;
  f2_get(d, d0, d1);
  Roots2 o;
  const F2 HALF = f2(0.5f);
  const F2 z = fma2(f2(0.25f) * d, d, e * e);
  F2 g = rsqrt2(z);
  g = fma2(HALF * g, fma2(-z * g, g, f2(1.0f)), g);
  const F2 ad = f2(fabsf(d0), fabsf(d1));
  const F2 w = fma2(z, g, HALF * ad);
  F2 k = rsqrt2(w);
  k = fma2(HALF * k, fma2(-w * k, k, f2(1.0f)), k);
  const F2 big = w * k, small = e * k;
  float b0, b1, s0, s1;
  f2_get(big, b0, b1);
  f2_get(small, s0, s1);
  const bool p0 = d0 >= 0.0f, p1 = d1 >= 0.0f;
  const float x0 = p0 ? b0 : s0, x1 = p1 ? b1 : s1, y0 = p0 ? s0 : b0, y1 = p1 ? s1 : b1;
  const F2 x = f2(x0, x1), y = f2(y0, y1);
  const ExpF2 ex = exp_parts2(HALF * x);
  const F2 t = ex.expm1(), v = ex.exp();
  F2 ri = rcp2(v);
  ri = fma2(ri, fma2(-v, ri, f2(1.0f)), ri);
  const F2 tr = t * ri, sh2 = t + tr;
  const F2 a = f2(0.25f) * (sh2 * sh2);
  F2 sh = sh2 * fma2(HALF * t, tr, f2(1.0f));
  const F2 hy = HALF * y;
  F2 sn, cs;
  if (fmaxf(fabsf(y0), fabsf(y1)) < 6.0e4f) {
    float h0, h1;
    f2_get(hy * f2(0.3183098861837907f), h0, h1);
    const F2 n = f2(rintf(h0), rintf(h1));
    const F2 r = fma2(n, f2(-PI_F_LO), fma2(n, f2(-PI_F_MID), fma2(n, f2(-PI_F_HI), hy)));
    const F2 ss = r * r;
    sn = fma2(r * ss, fma2(ss, fma2(ss, fma2(ss, f2(SIN_Q3), f2(SIN_Q2)), f2(SIN_Q1)), f2(SIN_Q0)), r);
    cs = fma2(ss, fma2(ss, fma2(ss, fma2(ss, fma2(ss, f2(COS_Q4), f2(COS_Q3)), f2(COS_Q2)), f2(COS_Q1)), f2(COS_Q0)),
              f2(1.0f));
  } else {
    sn = f2(sinf(0.5f * y0), sinf(0.5f * y1));
    cs = f2(cosf(0.5f * y0), cosf(0.5f * y1));
  }
  const F2 b = sn * sn, sy = f2(2.0f) * (sn * cs);
  F2 q = a + b;
  o.am = a - b;
  o.ch = fma2(f2(2.0f), a, f2(1.0f));
  o.cy = fma2(f2(-2.0f), b, f2(1.0f));
  if (fmaxf(fabsf(x0), fabsf(x1)) >= 37.42994775f) {   // the reference's clamp, half by half
    float am[2], qq[2], sv[2], cv[2], bb[2];
    const float xx[2] = {x0, x1};
    f2_get(o.am, am[0], am[1]);
    f2_get(q, qq[0], qq[1]);
    f2_get(sh, sv[0], sv[1]);
    f2_get(o.ch, cv[0], cv[1]);
    f2_get(b, bb[0], bb[1]);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (fabsf(xx[i]) >= 37.42994775f) {
        const float c2 = fmaf(-2.0f, bb[i], 1.0f);
        sv[i] = copysignf(1e15f, xx[i]);
        cv[i] = 1e15f;
        am[i] = 0.5f * (1e15f + c2) - 1.0f;
        qq[i] = 0.5f * (1e15f - c2);
      }
    sh = f2(sv[0], sv[1]);
    o.ch = f2(cv[0], cv[1]);
    o.am = f2(am[0], am[1]);
    q = f2(qq[0], qq[1]);
  }
  o.x = x;
  o.y = y;
  o.sh = sh;
  o.sy = sy;
  o.it = HALF * g;
  o.al = fma2(x, sh, y * sy) * o.it;
  o.be = fma2(x, sy, -(y * sh)) * o.it;
  o.ga = q * g;
  return o;
}

// Whether both halves are below the series' limit, and which of them is far
// enough below it to take the series beside one above.
constexpr float EVOL_TINY = 1.0f / 64.0f;
__device__ __forceinline__ bool evol_low(F2 d, F2 e) {
  float d0, d1, e0, e1;
  f2_get(d, d0, d1);
  f2_get(e, e0, e1);
  return fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(e0), fabsf(e1))) <= 0.25f;
}
struct Low2 {
  bool a, b;
};
__device__ __forceinline__ Low2 evol_low2(F2 d, F2 e) {
  float d0, d1, e0, e1;
  f2_get(d, d0, d1);
  f2_get(e, e0, e1);
  return Low2{fmaxf(fabsf(d0), fabsf(e0)) <= EVOL_TINY, fmaxf(fabsf(d1), fabsf(e1)) <= EVOL_TINY};
}
__device__ __forceinline__ void low_put(const Low2& w, F2& x, F2 y) {   // y in the halves w
  float x0, x1, y0, y1;
  f2_get(x, x0, x1);
  f2_get(y, y0, y1);
  x = f2(w.a ? y0 : x0, w.b ? y1 : x1);
}

// The four functions at two arguments.
struct EvolABG2 {
  F2 am, al, be, ga;
};
__device__ __forceinline__ EvolABG2 evol_series2(F2 d, F2 e) {
  EvolABG2 o;
  const F2 ee = e * e, dd = d * d;
  const F2 g1 = dd + ee, g2 = fma2(f2(2.0f), ee, dd), g3 = d * g2;
  const F2 g4 = d * fma2(f2(3.0f), ee, dd), g5 = fma2(g2, g2, f2(-2.0f) * (ee * ee));
  o.al = fma2(g3, f2(1.0f / 5040.0f), fma2(g1, f2(1.0f / 120.0f), fma2(d, f2(1.0f / 6.0f), f2(1.0f))));
  o.be = -e * fma2(g3, f2(1.0f / 362880.0f), fma2(g1, f2(1.0f / 5040.0f), fma2(d, f2(1.0f / 120.0f), f2(1.0f / 6.0f))));
  o.ga = fma2(g3, f2(1.0f / 40320.0f), fma2(g1, f2(1.0f / 720.0f), fma2(d, f2(1.0f / 24.0f), f2(0.5f))));
  o.am = fma2(g5, f2(1.0f / 80640.0f), fma2(g4, f2(1.0f / 1440.0f), fma2(g2, f2(1.0f / 48.0f), f2(0.25f) * d)));
  return o;
}
__device__ __forceinline__ EvolABG2 evol_abg2(F2 d, F2 e) {
  if (evol_low(d, e)) return evol_series2(d, e);
  const Low2 w = evol_low2(d, e);
  const Roots2 R = roots2(d, e);
  EvolABG2 o{R.am, R.al, R.be, R.ga};
  if (__builtin_expect(w.a || w.b, 0)) {
    const EvolABG2 q = evol_series2(d, e);
    low_put(w, o.am, q.am);
    low_put(w, o.al, q.al);
    low_put(w, o.be, q.be);
    low_put(w, o.ga, q.ga);
  }
  return o;
}

// What the formal solution needs of one layer at two wavelengths: one height of
// OLD_ANALYTICAL_SOLVER (src/rtesolver.f90:163-187), I <- (1 - O) S e0 + O I,
// applied as I + O (I - S e0) + S e0 row by row without forming O.  The
// operator's vectors are u = al eta - be rho and v = al rho + be eta, and 1 - O(1,1)
// = om0 comes without cancellation from e^-tI - 1: I <- I - om0 w0 - E um.I, ...
// with w0 = I0 - S.
struct Layer2 {
  F2 S, om0, E, dg, ga, t[3], r[3], um[3], up[3], v[3];
};
constexpr int LAYER2_F2 = sizeof(Layer2) / sizeof(F2);

// The layer from its optical depths (t: eta_Q, U, V; r: rho_Q, U, V); a half
// with a non-finite matrix becomes the identity.  Returns whether one did.
__device__ __forceinline__ bool layer_set(Layer2& L, F2 tI) {
  const F2 eta2 = fma2(L.t[2], L.t[2], fma2(L.t[1], L.t[1], L.t[0] * L.t[0]));
  const F2 rho2 = fma2(L.r[2], L.r[2], fma2(L.r[1], L.r[1], L.r[0] * L.r[0]));
  const F2 er = fma2(L.t[2], L.r[2], fma2(L.t[1], L.r[1], L.t[0] * L.r[0]));
  const F2 sum = eta2 + rho2;
  float c0, c1;
  f2_get(tI + sum, c0, c1);
  const bool rare = !(fabsf(c0) < DEPTH_RARE) || !(fabsf(c1) < DEPTH_RARE);
  if (__builtin_expect(rare, 0)) tI = depth_cut2(tI);
  const EvolABG2 f = evol_abg2(eta2 - rho2, er);
  const ExpF2 ex = exp_parts2(-tI);
  const F2 gh = f.ga * (f2(0.5f) * sum);
  L.ga = f.ga;
  L.E = ex.exp();
  L.om0 = -fma2(L.E, f.am + gh, ex.expm1());
  L.dg = (f2(1.0f) - gh) + f.am;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    const F2 u = fma2(f.al, L.t[i], -(f.be * L.r[i]));
    const F2 c = f.ga * fma2(L.t[j], L.r[k], -(L.t[k] * L.r[j]));
    L.um[i] = u - c;
    L.up[i] = u + c;
    L.v[i] = fma2(f.al, L.r[i], f.be * L.t[i]);
  }
  const bool b0 = !(fabsf(c0) < 3.0e38f), b1 = !(fabsf(c1) < 3.0e38f);
  if (__builtin_expect(rare && (b0 || b1), 0)) {
    auto put = [&](F2& x, float v) {
      float a, b;
      f2_get(x, a, b);
      x = f2(b0 ? v : a, b1 ? v : b);
    };
    put(L.om0, 0.0f);
    put(L.E, 1.0f);
    put(L.dg, 1.0f);
    put(L.ga, 0.0f);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      put(L.t[i], 0.0f);
      put(L.r[i], 0.0f);
      put(L.um[i], 0.0f);
      put(L.up[i], 0.0f);
      put(L.v[i], 0.0f);
    }
    return true;
  }
  return false;
}

__device__ __forceinline__ void layer_apply(const Layer2& L, F2 I[4]) {
  const F2 w0 = I[0] - L.S;
  const F2 ge = L.ga * fma2(L.t[2], I[3], fma2(L.t[1], I[2], L.t[0] * I[1]));
  const F2 gr = L.ga * fma2(L.r[2], I[3], fma2(L.r[1], I[2], L.r[0] * I[1]));
  const F2 n0 = fma2(L.um[2], I[3], fma2(L.um[1], I[2], L.um[0] * I[1]));
  F2 n[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    n[i] = fma2(L.r[i], gr,
                fma2(L.t[i], ge, fma2(L.v[k], I[1 + j], fma2(-L.v[j], I[1 + k], fma2(L.dg, I[1 + i], -(L.up[i] * w0))))));
  }
  I[0] = fma2(-L.E, n0, fma2(-L.om0, w0, I[0]));
#pragma unroll
  for (int i = 0; i < 3; ++i) I[1 + i] = L.E * n[i];
}

// ------------------------------------------------ response functions
// evol_abg2's functions and their derivatives with respect to d and e (those
// of am are al / 4 and -be / 2).
struct EvolD2 {
  F2 am, al, be, ga, al_d, al_e, be_d, be_e, ga_d, ga_e;
};
__device__ __forceinline__ EvolD2 evol_series_d2(F2 d, F2 e) {
  EvolD2 o;
  const F2 ee = e * e, dd = d * d;
  const F2 s1 = dd + ee, s2 = fma2(f2(2.0f), ee, dd), s3 = d * s2;
  const F2 s4 = d * fma2(f2(3.0f), ee, dd), s5 = fma2(s2, s2, f2(-2.0f) * (ee * ee));
  const F2 u2 = fma2(f2(3.0f), dd, f2(2.0f) * ee);                        // d s3 / d d
  const F2 u3 = d * fma2(f2(4.0f), dd, f2(6.0f) * ee);                    // d (d^4 + 3 d^2 e^2 + e^4) / d d
  const F2 u4 = fma2(f2(6.0f), dd, f2(4.0f) * ee);                        // ... / d e, over e
  o.al = fma2(s3, f2(1.0f / 5040.0f), fma2(s1, f2(1.0f / 120.0f), fma2(d, f2(1.0f / 6.0f), f2(1.0f))));
  o.al_d = fma2(u3, f2(1.0f / 362880.0f), fma2(u2, f2(1.0f / 5040.0f), fma2(d, f2(1.0f / 60.0f), f2(1.0f / 6.0f))));
  o.al_e = e * fma2(u4, f2(1.0f / 362880.0f), fma2(d, f2(1.0f / 1260.0f), f2(1.0f / 60.0f)));
  o.be = -e * fma2(s3, f2(1.0f / 362880.0f), fma2(s1, f2(1.0f / 5040.0f), fma2(d, f2(1.0f / 120.0f), f2(1.0f / 6.0f))));
  o.be_d = -e * fma2(u2, f2(1.0f / 362880.0f), fma2(d, f2(1.0f / 2520.0f), f2(1.0f / 120.0f)));
  o.be_e = -fma2(d * fma2(f2(6.0f), ee, dd), f2(1.0f / 362880.0f),
                 fma2(fma2(f2(3.0f), ee, dd), f2(1.0f / 5040.0f), fma2(d, f2(1.0f / 120.0f), f2(1.0f / 6.0f))));
  o.ga = fma2(s3, f2(1.0f / 40320.0f), fma2(s1, f2(1.0f / 720.0f), fma2(d, f2(1.0f / 24.0f), f2(0.5f))));
  o.ga_d = fma2(u3, f2(1.0f / 3628800.0f), fma2(u2, f2(1.0f / 40320.0f), fma2(d, f2(1.0f / 360.0f), f2(1.0f / 24.0f))));
  o.ga_e = e * fma2(u4, f2(1.0f / 3628800.0f), fma2(d, f2(1.0f / 10080.0f), f2(1.0f / 360.0f)));
  o.am = fma2(s5, f2(1.0f / 80640.0f), fma2(s4, f2(1.0f / 1440.0f), fma2(s2, f2(1.0f / 48.0f), f2(0.25f) * d)));
  return o;
}
__device__ __forceinline__ EvolD2 evol_roots_d2(F2 d, F2 e) {
  EvolD2 o;
  const Roots2 R = roots2(d, e);
  o.am = R.am;
  o.al = R.al;
  o.be = R.be;
  o.ga = R.ga;
  // the quotient rule on (x sinh x + y sin y) / theta and its kin, with dx =
  // (x dd / 2 + y de) / theta, dy = (x de - y dd / 2) / theta
  const F2 x = R.x, y = R.y, it = R.it, HALF = f2(0.5f);
  const F2 xs = x * R.sh, ys = y * R.sy, xy = fma2(x, R.sy, y * R.sh);   // x sinh x, y sin y, x sin y + y sinh x
  const F2 xc = (x * x) * R.ch, yc = (y * y) * R.cy, ec = e * (R.ch + R.cy);
  const F2 dit = d * it, e4 = f2(4.0f) * (e * it);
  const F2 hit = HALF * it;
  o.al_d = it * fma2(hit, (xs - ys) + (xc - yc), -(o.al * dit));
  o.al_e = it * fma2(it, xy + ec, -(o.al * e4));
  o.be_d = it * fma2(hit, xy - ec, -(o.be * dit));
  o.be_e = it * fma2(it, (ys - xs) + (fma2(x * x, R.cy, -((y * y) * R.ch))), -(o.be * e4));
  o.ga_d = it * fma2(hit, xs - ys, -(o.ga * dit));
  o.ga_e = it * fma2(it, xy, -(o.ga * e4));
  return o;
}
__device__ __forceinline__ EvolD2 evol_d2(F2 d, F2 e) {
  if (evol_low(d, e)) return evol_series_d2(d, e);
  const Low2 w = evol_low2(d, e);
  EvolD2 o = evol_roots_d2(d, e);
  if (__builtin_expect(w.a || w.b, 0)) {
    const EvolD2 q = evol_series_d2(d, e);
    low_put(w, o.am, q.am);
    low_put(w, o.al, q.al);
    low_put(w, o.be, q.be);
    low_put(w, o.ga, q.ga);
    low_put(w, o.al_d, q.al_d);
    low_put(w, o.al_e, q.al_e);
    low_put(w, o.be_d, q.be_d);
    low_put(w, o.be_e, q.be_e);
    low_put(w, o.ga_d, q.ga_d);
    low_put(w, o.ga_e, q.ga_e);
  }
  return o;
}

// A layer of the response-function kernel: its operator O and what the
// derivatives need.
struct LayerD2 {
  F2 t[3], r[3], c[3], h, E, om0;   // c = eta x rho, h = (|eta|^2 + |rho|^2) / 2
  EvolD2 f;
  F2 O[16];
  unsigned long long on;   // all bits, but none of a half whose matrix is not finite: the identity, without response
};

__device__ __forceinline__ bool layer_d2(LayerD2& L, F2 tI) {
  F2 eta2 = fma2(L.t[2], L.t[2], fma2(L.t[1], L.t[1], L.t[0] * L.t[0]));
  F2 rho2 = fma2(L.r[2], L.r[2], fma2(L.r[1], L.r[1], L.r[0] * L.r[0]));
  F2 er = fma2(L.t[2], L.r[2], fma2(L.t[1], L.r[1], L.t[0] * L.r[0]));
  float c0, c1;
  f2_get(tI + (eta2 + rho2), c0, c1);
  bool gap = false;
  L.on = ~0ull;
  if (__builtin_expect(!(fabsf(c0) < DEPTH_RARE) || !(fabsf(c1) < DEPTH_RARE), 0)) {
    const bool b0 = !(fabsf(c0) < 3.0e38f), b1 = !(fabsf(c1) < 3.0e38f);
    gap = b0 || b1;
    L.on = (b0 ? 0ull : 0xffffffffull) | (b1 ? 0ull : 0xffffffff00000000ull);
    tI = depth_cut2(tI);
    auto zero = [&](F2& x) {
      float a, b;
      f2_get(x, a, b);
      x = f2(b0 ? 0.0f : a, b1 ? 0.0f : b);
    };
    zero(tI);
    zero(eta2);
    zero(rho2);
    zero(er);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      zero(L.t[i]);
      zero(L.r[i]);
    }
  }
  L.f = evol_d2(eta2 - rho2, er);
  const EvolD2& f = L.f;
  const ExpF2 ex = exp_parts2(-tI);
  L.E = ex.exp();
  L.h = f2(0.5f) * (eta2 + rho2);
  const F2 gh = f.ga * L.h;
  const F2 ag = f.am + gh;
  L.om0 = -fma2(L.E, ag, ex.expm1());
  const F2 dg = L.E * ((f2(1.0f) - gh) + f.am), ga = L.E * f.ga;
  {
    // O(1,1) = E (1 + am + gh): as 1 - om0 where that holds more digits, in thin layers
    float m0, m1, a0, a1, e0, e1;
    f2_get(L.om0, m0, m1);
    f2_get(f2(1.0f) - L.om0, a0, a1);
    f2_get(fma2(L.E, ag, L.E), e0, e1);
    L.O[0] = f2(m0 < 0.5f ? a0 : e0, m1 < 0.5f ? a1 : e1);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    L.c[i] = fma2(L.t[j], L.r[k], -(L.t[k] * L.r[j]));
    const F2 u = L.E * fma2(f.al, L.t[i], -(f.be * L.r[i])), c = ga * L.c[i];
    L.O[1 + i] = c - u;
    L.O[4 * (1 + i)] = -(u + c);
    L.O[5 * (1 + i)] = fma2(ga, fma2(L.t[i], L.t[i], L.r[i] * L.r[i]), dg);
    // the pair (j, k): the symmetric part of M and the vector al rho + be eta
    const F2 v = L.E * fma2(f.al, L.r[i], f.be * L.t[i]);
    const F2 s = ga * fma2(L.t[j], L.t[k], L.r[j] * L.r[k]);
    L.O[4 * (1 + j) + 1 + k] = s + v;
    L.O[4 * (1 + k) + 1 + j] = s - v;
  }
  return gap;
}

__device__ __forceinline__ F2 dot3(const F2 a[3], const F2 b[3]) { return fma2(a[2], b[2], fma2(a[1], b[1], a[0] * b[0])); }
__device__ __forceinline__ void mat4(const F2 O[16], const F2 w[4], F2 y[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) y[i] = fma2(O[4 * i], w[0], fma2(O[4 * i + 1], w[1], fma2(O[4 * i + 2], w[2], O[4 * i + 3] * w[3])));
}

// The derivative of O w for any direction of the seven optical depths, from
// the layer and w: with dd, de the changes of d and e,
//   dO w = Ad dd + Ae de + (r.deta - q.drho, g deta + g' drho + deta x q + drho x r) - dtI O w.
struct Resp2 {
  F2 Ad[4], Ae[4], q[3], r[3], g, gp, Ow[4];
};
__device__ __forceinline__ void resp_w(const LayerD2& L, const F2 w[4], Resp2& R) {
  const EvolD2& f = L.f;
  const F2 wv[3] = {w[1], w[2], w[3]};
  const F2 ew = dot3(L.t, wv), rw = dot3(L.r, wv);
  F2 X[4], Y[4], M[4];   // X w, Y w and M w
  X[0] = ew;
  Y[0] = -rw;
  M[0] = fma2(L.h, w[0], dot3(L.c, wv));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    X[1 + i] = fma2(L.t[i], w[0], fma2(L.r[j], wv[k], -(L.r[k] * wv[j])));
    Y[1 + i] = fma2(-L.r[i], w[0], fma2(L.t[j], wv[k], -(L.t[k] * wv[j])));
    M[1 + i] = fma2(L.t[i], ew, fma2(L.r[i], rw, -fma2(L.c[i], w[0], L.h * wv[i])));
  }
  mat4(L.O, w, R.Ow);
  const F2 E = L.E;
  const F2 md = E * (f2(0.25f) * f.al), me = E * (f2(-0.5f) * f.be);
  const F2 ad = E * f.al_d, ae = E * f.al_e, bd = E * f.be_d, be = E * f.be_e, gd = E * f.ga_d, ge = E * f.ga_e;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    R.Ad[i] = fma2(gd, M[i], fma2(-bd, Y[i], fma2(-ad, X[i], md * w[i])));
    R.Ae[i] = fma2(ge, M[i], fma2(-be, Y[i], fma2(-ae, X[i], me * w[i])));
  }
  const F2 al = E * f.al, bt = E * f.be, ga = E * f.ga;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    R.q[i] = fma2(ga, Y[1 + i], -(bt * wv[i]));
    R.r[i] = fma2(ga, X[1 + i], -(al * wv[i]));
  }
  R.g = fma2(ga, ew, -(al * w[0]));
  R.gp = fma2(ga, rw, bt * w[0]);
}

__device__ __forceinline__ void resp_dir(const LayerD2& L, const Resp2& R, F2 dI, const F2 dt[3], const F2 dr[3], F2 o[4]) {
  const F2 dd = f2(2.0f) * (dot3(L.t, dt) - dot3(L.r, dr)), de = dot3(L.r, dt) + dot3(L.t, dr);
  o[0] = fma2(R.Ad[0], dd, fma2(R.Ae[0], de, fma2(-dI, R.Ow[0], dot3(R.r, dt) - dot3(R.q, dr))));
  o[0].v &= L.on;   // where the matrix is not finite neither are the changes of its depths
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    F2 v = fma2(R.g, dt[i], R.gp * dr[i]);
    v = fma2(dt[j], R.q[k], fma2(-dt[k], R.q[j], v));
    v = fma2(dr[j], R.r[k], fma2(-dr[k], R.r[j], v));
    o[1 + i] = fma2(R.Ad[1 + i], dd, fma2(R.Ae[1 + i], de, fma2(-dI, R.Ow[1 + i], v)));
    o[1 + i].v &= L.on;
  }
}

}  // namespace fzd
