// jk_zmath.cuh -- device complex 2x2 HSVD of the J-Kogbetliantz step
// (src/Z/ztransf.F90), operation for operation; complex values are double2.
#pragma once

#include "jk_math.cuh"

namespace jk {

__device__ __forceinline__ void zswap(double2 &a, double2 &b) { const double2 t = a; a = b; b = t; }

// C1A, src/Z/ztransf.F90:231-241
__device__ __forceinline__ void zc1a(const double B[4], double2 &a1, double2 &a2)
{
  const double2 c1 = zddiv(zdfma(B[M12], a2, a1), B[M11]);
  const double2 c2 = zddiv(zdfma(B[M21], a1, a2), B[M22]);
  a1 = c1; a2 = c2;
}

// C2A, src/Z/ztransf.F90:245-258
__device__ __forceinline__ void zc2a(const double B[4], double2 A[4])
{
  double2 C[4];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    C[2 * j + 0] = zddiv(zdfma(B[M12], A[2 * j + 1], A[2 * j + 0]), B[M11]);
    C[2 * j + 1] = zddiv(zdfma(B[M21], A[2 * j + 0], A[2 * j + 1]), B[M22]);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) A[k] = C[k];
}

// A2C, src/Z/ztransf.F90:262-275
__device__ __forceinline__ void za2c(double2 A[4], const double B[4])
{
  double2 C[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    C[i + 0] = zddiv(zdfma(B[M21], A[i + 2], A[i + 0]), B[M11]);
    C[i + 2] = zddiv(zdfma(B[M12], A[i + 0], A[i + 2]), B[M22]);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) A[k] = C[k];
}

// ZPOLAR, src/Z/ztransf.F90:112-126
__device__ __forceinline__ void zpolar(double2 z, double &a, double2 &e)
{
  a = hypot2(z.x, z.y);
  const double c = copysign(fmin(__ddiv_rn(fabs(z.x), a), 1.0), z.x);
  const double s = __ddiv_rn(z.y, fmax(a, JK_MINF));
  e = zc(c, s);
}

// ZHSVD2T, src/Z/ztransf.F90:641-835
__device__ __forceinline__ void zhsvd2t(double2 A[4], const int J0, const int J1, double2 U[4], double2 Z[4], int &info)
{
  double c, t, w;
  double2 r, s;
  bool p, d = true;
  if (zeq0(A[M21])) c = zabs(A[M11]);
  else if (zeq0(A[M11])) { c = zabs(A[M21]); d = false; }
  else { c = hypot2(zabs(A[M11]), zabs(A[M21])); d = false; }
  if (zeq0(A[M12])) t = zabs(A[M22]);
  else if (zeq0(A[M22])) { t = zabs(A[M12]); d = false; }
  else { t = hypot2(zabs(A[M12]), zabs(A[M22])); d = false; }

  if (c < t) {
    zswap(A[M11], A[M12]); zswap(A[M21], A[M22]);
    if (J0 == J1) { zswap(Z[M11], Z[M12]); zswap(Z[M21], Z[M22]); }
    p = true;
    w = t;
  }
  else { p = false; w = c; }

  zpolar(A[M11], c, r);
  if (zne1(r)) {
    s = conj(r);
    U[M11] = zzmul(U[M11], s); U[M12] = zzmul(U[M12], s);
    A[M11] = zzmul(A[M11], s); A[M12] = zzmul(A[M12], s);
  }
  zpolar(A[M21], t, s);
  if (zne1(s)) {
    r = conj(s);
    U[M21] = zzmul(U[M21], r); U[M22] = zzmul(U[M22], r);
    A[M21] = zzmul(A[M21], r); A[M22] = zzmul(A[M22], r);
  }

  if (A[M11].x < A[M21].x) {
    zswap(U[M11], U[M21]); zswap(U[M12], U[M22]);
    zswap(A[M11], A[M21]); zswap(A[M12], A[M22]);
  }

  if (!d) {
    t = __ddiv_rn(A[M21].x, A[M11].x);
    c = sqrt(fma(t, t, 1.0));
    const double Q[4] = { c, -t, t, c };
    zc2a(Q, U);
    zc1a(Q, A[M12], A[M22]);
  }
  A[M11] = zc(w, 0.0);
  A[M21] = zc(0.0, 0.0);

  if ((J0 != J1) && p) {
    zswap(A[M11], A[M12]); zswap(A[M21], A[M22]);
    zswap(U[M11], U[M21]); zswap(U[M12], U[M22]);
    zswap(A[M11], A[M21]); zswap(A[M12], A[M22]);
    zpolar(A[M21], t, s);
    if (zne1(s)) {
      r = conj(s);
      Z[M11] = zzmul(Z[M11], r); Z[M21] = zzmul(Z[M21], r);
      A[M11] = zzmul(A[M11], r); A[M21] = zzmul(A[M21], r);
    }
    zpolar(A[M11], c, r);
    if (zne1(r)) {
      s = conj(r);
      U[M11] = zzmul(U[M11], s); U[M12] = zzmul(U[M12], s);
      A[M11] = zzmul(A[M11], s);
    }
  }
  else {
    zpolar(A[M12], c, r);
    if (zne1(r)) {
      s = conj(r);
      Z[M12] = zzmul(Z[M12], s); Z[M22] = zzmul(Z[M22], s);
      A[M12] = zzmul(A[M12], s); A[M22] = zzmul(A[M22], s);
    }
    zpolar(A[M22], t, s);
    if (zne1(s)) {
      r = conj(s);
      U[M21] = zzmul(U[M21], r); U[M22] = zzmul(U[M22], r);
      A[M22] = zzmul(A[M22], r);
    }
  }
  info = d ? 0 : 1;
}

// ZHSVD2S, src/Z/ztransf.F90:839-880
__device__ __forceinline__ void zhsvd2s(double2 A[4], const int J0, const int J1, double2 U[4], double2 Z[4], int &info)
{
  const int t = J0 + J1;
  if (((t == 2) && (A[M11].x < A[M22].x)) || ((t == -2) && (A[M22].x < A[M11].x))) {
    A[M21] = U[M11]; A[M12] = U[M12];
    U[M11] = U[M21]; U[M12] = U[M22];
    U[M21] = A[M21]; U[M22] = A[M12];
    A[M21] = A[M11]; A[M11] = A[M22]; A[M22] = A[M21];
    A[M21] = Z[M11]; A[M12] = Z[M21];
    Z[M11] = Z[M12]; Z[M21] = Z[M22];
    Z[M12] = A[M21]; Z[M22] = A[M12];
  }
  if (!(info & 8)) { A[M21] = zc(0.0, 0.0); A[M12] = zc(0.0, 0.0); }
  if (zne1(U[M11]) || !zeq0(U[M21]) || !zeq0(U[M12]) || zne1(U[M22])) info += 2;
  if (zne1(Z[M11]) || !zeq0(Z[M21]) || !zeq0(Z[M12]) || zne1(Z[M22])) info += 4;
}

// ZSCALEA, src/Z/ztransf.F90:884-921
__device__ __forceinline__ void zscalea(double2 A[4], int &s)
{
  s = 0x7FFFFFFF;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      double aa = fabs(A[2 * j + i].x);
      if (!(aa <= JK_HUGE)) { s = -((j + 1) * 2 + (i + 1)); return; }
      s = imin(s, JK_EH - exponent(fmax(aa, JK_MINF)) - 2);
      aa = fabs(A[2 * j + i].y);
      if (!(aa <= JK_HUGE)) { s = -((j + 1) * 2 + (i + 1)); return; }
      s = imin(s, JK_EH - exponent(fmax(aa, JK_MINF)) - 2);
    }
  if (s != 0)
#pragma unroll
    for (int k = 0; k < 4; ++k) A[k] = zc(scale(A[k].x, s), scale(A[k].y, s));
}

// ZHSVD2 (argument-checking form), src/Z/ztransf.F90:925-1009, for every input; out of line, it
// serves what zhsvd2_near does not take
static __device__ __noinline__ void zhsvd2_any(double2 A[4], const int J0, const int J1, double2 U[4], double2 Z[4], double th1, int &info)
{
  double G[2] = { 0.0, 0.0 }, W[4] = { 0.0, 0.0, 0.0, 0.0 }, B[4] = { 0.0, 0.0, 0.0, 0.0 }, C[4] = { 0.0, 0.0, 0.0, 0.0 };
  int s;
  if (abs(J0) != 1) info = -1;
  else if (abs(J1) != 1) info = -2;
  else info = 0;
  if (info) return;
  zscalea(A, s);
  if (s <= -3) { info = s; return; }
  U[M11] = zc(1.0, 0.0); U[M21] = zc(0.0, 0.0); U[M12] = zc(0.0, 0.0); U[M22] = zc(1.0, 0.0);
  Z[M11] = zc(1.0, 0.0); Z[M21] = zc(0.0, 0.0); Z[M12] = zc(0.0, 0.0); Z[M22] = zc(1.0, 0.0);
  zhsvd2t(A, J0, J1, U, Z, info);
  if (info > 0) {
    W[M11] = A[M11].x; W[M21] = A[M21].x; W[M12] = A[M12].x; W[M22] = A[M22].x;
    khsvd2(W, J0, J1, G, B, C, s, th1, info);
  }
  else if (info == 0) {
    if (s == 0) { W[M11] = A[M11].x; W[M22] = A[M22].x; }
    else { W[M11] = scale(A[M11].x, -s); W[M22] = scale(A[M22].x, -s); }
  }
  if (info < 0) return;
  bool th1fix = false;
  if (info > 0) {
    zc2a(B, U);
    za2c(Z, C);
    if (!(info & 8)) { W[M11] = G[0]; W[M22] = G[1]; }
    else {
      if (s != 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) A[k] = zc(scale(A[k].x, -s), scale(A[k].y, -s));
      zc2a(B, A);
      za2c(A, C);
      th1fix = true;
    }
  }
  if (!th1fix) { A[M11] = zc(W[M11], 0.0); A[M22] = zc(W[M22], 0.0); }
  zhsvd2s(A, J0, J1, U, Z, info);
}

// ------------------------------------------------------------------------
// the straight-line forms for complex blocks far from the ends of the exponent range (see
// quot, root in jk_math.cuh)
// ------------------------------------------------------------------------

// zero, or at least 2^-300 in magnitude
__device__ __forceinline__ bool near_ratio(double x) { return x == 0.0 || fabs(x) >= 4.909093465297727e-91; }
__device__ __forceinline__ bool near_parts(double2 z) { return near_ratio(z.x) && near_ratio(z.y); }

// hypot2 for two operands below 2^300 of which the larger is zero or at least 2^-1000
__device__ __forceinline__ double hypot2_near0(double x, double y)
{
  return (x == 0.0 && y == 0.0) ? 0.0 : hypot2_near(x, y);
}
__device__ __forceinline__ double zabs_near(double2 a) { return hypot2_near0(a.x, a.y); }
__device__ __forceinline__ double2 zdown600(double2 a) { return zc(down600(a.x), down600(a.y)); }

// a division of both parts by the same number, y = recip(b)
__device__ __forceinline__ double2 zquot(double2 a, double b, double y) { return zc(quot(a.x, b, y), quot(a.y, b, y)); }
__device__ __forceinline__ bool zquot_num(double2 a) { return quot_num(a.x) && quot_num(a.y); }

// e of ZPOLAR (see zpolar) for a scaled entry
__device__ __forceinline__ void zpolar_scaled(double2 z, double2 &e, bool &ok)
{
  const double2 x = zdown600(z);
  const double a = zabs_near(x), y = recip(a);
  const int ea = bexp(a), ex = bexp(x.x), ey = bexp(x.y);
  const bool zero = zeq0(z);
  ok = ok && (zero || (ea >= 123 && (z.x == 0.0 || (ex >= 123 && ex - ea >= -1000)) && (z.y == 0.0 || (ey >= 123 && ey - ea >= -1000))));
  const double c = zero ? 1.0 : fmin(quot(fabs(x.x), a, y), 1.0);
  e = zc(copysign(c, z.x), zero ? z.y : quot(x.y, a, y));
}

template <int N>
__device__ __forceinline__ void zquots(double2 *a, double b, double y, bool &ok)
{
  bool num = true;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    num = num && zquot_num(a[k]);
    a[k] = zquot(a[k], b, y);
  }
  ok = ok && (num || b == 1.0);
}

// C2A and A2C (src/Z/ztransf.F90:245-275) with the rotations of c2a_near, a2c_near
__device__ __forceinline__ void zc2a_near(double t, double c, double y, double2 A[4], bool &ok)
{
  double2 v[4] = { zdfma(t, A[M21], A[M11]), zdfma(-t, A[M11], A[M21]), zdfma(t, A[M22], A[M12]), zdfma(-t, A[M12], A[M22]) };
  zquots<4>(v, c, y, ok);
#pragma unroll
  for (int k = 0; k < 4; ++k) A[k] = v[k];
}
__device__ __forceinline__ void za2c_near(double2 A[4], double t21, double t12, double c, double y, bool &ok)
{
  double2 v[4] = { zdfma(t21, A[M12], A[M11]), zdfma(t21, A[M22], A[M21]), zdfma(t12, A[M11], A[M12]), zdfma(t12, A[M21], A[M22]) };
  zquots<4>(v, c, y, ok);
#pragma unroll
  for (int k = 0; k < 4; ++k) A[k] = v[k];
}

__device__ __forceinline__ double2 zsel(bool c, double2 a, double2 b) { return zc(c ? a.x : b.x, c ? a.y : b.y); }
__device__ __forceinline__ void zcswap(bool c, double2 &a, double2 &b) { cswap(c, a.x, b.x); cswap(c, a.y, b.y); }
// a v where c, else a
__device__ __forceinline__ double2 zcmul(bool c, double2 a, double2 v) { return zsel(c, zzmul(a, v), a); }

// ZHSVD2 for a block without a zero column whose largest part lies in 2^(+-300): the operations
// of zhsvd2_any in the same order, as dhsvd2_near.  Returns false, with nothing written, when the
// block does not allow it.  Without FULL, U and the new diagonal are left out.
template <bool FULL>
__device__ __forceinline__ bool zhsvd2_near(double2 Ain[4], const int J0, const int J1, double2 Uo[4], double2 Zo[4], double th1, int &info_o)
{
  int hi = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) hi = max(hi, max(bexp(Ain[k].x), bexp(Ain[k].y)));
  if (hi < 723 || hi > 1323 || (zeq0(Ain[M11]) && zeq0(Ain[M21])) || (zeq0(Ain[M12]) && zeq0(Ain[M22])) || abs(J0) != 1 ||
      abs(J1) != 1) return false;
  bool ok = true;
  const bool tg = (J0 == J1);
  const int sc = 2044 - hi;  // ZSCALEA's
  const double fs = pow2(sc - 600);
  const double2 one = zc(1.0, 0.0), zero = zc(0.0, 0.0);
  double2 A[4], U[4] = { one, zero, zero, one }, Z[4] = { one, zero, zero, one };
#pragma unroll
  for (int k = 0; k < 4; ++k) A[k] = zc(up600(__dmul_rn(Ain[k].x, fs)), up600(__dmul_rn(Ain[k].y, fs)));
  // ZHSVD2T, src/Z/ztransf.F90:641-835
  const bool d = zeq0(A[M21]) && zeq0(A[M12]);
  const double c = up600(hypot2_near(zabs_near(zdown600(A[M11])), zabs_near(zdown600(A[M21]))));
  const double t0 = up600(hypot2_near(zabs_near(zdown600(A[M12])), zabs_near(zdown600(A[M22]))));
  const bool p = (c < t0);
  const double w = p ? t0 : c;
  zcswap(p, A[M11], A[M12]); zcswap(p, A[M21], A[M22]);
  zcswap(p && tg, Z[M11], Z[M12]); zcswap(p && tg, Z[M21], Z[M22]);
  double2 r, s;
  zpolar_scaled(A[M11], r, ok);
  zpolar_scaled(A[M21], s, ok);
  {
    const bool nr = zne1(r), ns = zne1(s);
    const double2 vr = conj(r), vs = conj(s);
    U[M11] = zcmul(nr, U[M11], vr); U[M12] = zcmul(nr, U[M12], vr);
    A[M11] = zcmul(nr, A[M11], vr); A[M12] = zcmul(nr, A[M12], vr);
    U[M21] = zcmul(ns, U[M21], vs); U[M22] = zcmul(ns, U[M22], vs);
    A[M21] = zcmul(ns, A[M21], vs); A[M22] = zcmul(ns, A[M22], vs);
  }
  const bool sw = (A[M11].x < A[M21].x);
  zcswap(sw, U[M11], U[M21]); zcswap(sw, U[M12], U[M22]);
  zcswap(sw, A[M11], A[M21]); zcswap(sw, A[M12], A[M22]);
  {
    ok = ok && (d || A[M11].x > 0.0);
    const double t = quot_scaled(A[M21].x, A[M11].x, recip(down600(A[M11].x)), ok);
    const double q = root(fma(t, t, 1.0)), y = recip(q);
    if constexpr (FULL) {
      double2 V[4] = { U[0], U[1], U[2], U[3] };
      zc2a_near(t, q, y, V, ok);
#pragma unroll
      for (int k = 0; k < 4; ++k) U[k] = zsel(d, U[k], V[k]);
    }
    double2 v[2] = { zdfma(t, A[M22], A[M12]), zdfma(-t, A[M12], A[M22]) };  // C1A
    zquots<2>(v, q, y, ok);
    A[M12] = zsel(d, A[M12], v[0]);
    A[M22] = zsel(d, A[M22], v[1]);
  }
  A[M11] = zc(w, 0.0);
  A[M21] = zero;
  // unequal signs and swapped columns: rows and columns swapped back, a lower triangle
  const bool lo = !tg && p;
  zcswap(lo, A[M11], A[M12]); zcswap(lo, A[M21], A[M22]);
  zcswap(lo, U[M11], U[M21]); zcswap(lo, U[M12], U[M22]);
  zcswap(lo, A[M11], A[M21]); zcswap(lo, A[M12], A[M22]);
  {
    zpolar_scaled(zsel(lo, A[M21], A[M12]), s, ok);
    const bool ns = zne1(s);
    const double2 vs = conj(s);
    Z[M11] = zcmul(ns && lo, Z[M11], vs); Z[M21] = zcmul(ns && lo, Z[M21], vs);
    Z[M12] = zcmul(ns && !lo, Z[M12], vs); Z[M22] = zcmul(ns && !lo, Z[M22], vs);
    A[M11] = zcmul(ns && lo, A[M11], vs); A[M21] = zcmul(ns && lo, A[M21], vs);
    A[M12] = zcmul(ns && !lo, A[M12], vs); A[M22] = zcmul(ns && !lo, A[M22], vs);
    zpolar_scaled(zsel(lo, A[M11], A[M22]), r, ok);
    const bool nr = zne1(r);
    const double2 vr = conj(r);
    U[M11] = zcmul(nr && lo, U[M11], vr); U[M12] = zcmul(nr && lo, U[M12], vr); A[M11] = zcmul(nr && lo, A[M11], vr);
    U[M21] = zcmul(nr && !lo, U[M21], vr); U[M22] = zcmul(nr && !lo, U[M22], vr); A[M22] = zcmul(nr && !lo, A[M22], vr);
  }
  int info = d ? 0 : 1;
  double w11, w22;
  if (d) {
    w11 = scale(A[M11].x, -sc);
    w22 = scale(A[M22].x, -sc);
  }
  else {
    const double W[4] = { A[M11].x, A[M21].x, A[M12].x, A[M22].x };
    NearK k;
    khsvd2_near<FULL>(W, tg, sc, th1, info, k, ok);
    if constexpr (FULL) zc2a_near(k.tu, k.cu, k.yu, U, ok);
    za2c_near(Z, k.tz, k.c12, k.cz, k.yz, ok);
    w11 = FULL ? k.g0 : 0.0;
    w22 = FULL ? k.g1 : 0.0;
    if (info & 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) A[i] = zc(scale(A[i].x, -sc), scale(A[i].y, -sc));
      zc2a_near(k.tu, k.cu, k.yu, A, ok);
      za2c_near(A, k.tz, k.c12, k.cz, k.yz, ok);
    }
  }
  if (!ok) return false;
  if (!(info & 8)) { A[M11] = zc(w11, 0.0); A[M22] = zc(w22, 0.0); }
  zhsvd2s(A, J0, J1, U, Z, info);
#pragma unroll
  for (int i = 0; i < 4; ++i) { Ain[i] = A[i]; Uo[i] = U[i]; Zo[i] = Z[i]; }
  info_o = info;
  return true;
}

// ZHSVD2, src/Z/ztransf.F90:925-1009; without FULL what zhsvd2_near leaves out is undefined
template <bool FULL = true>
__device__ __forceinline__ void zhsvd2(double2 A[4], const int J0, const int J1, double2 U[4], double2 Z[4], double th1, int &info)
{
  if (!zhsvd2_near<FULL>(A, J0, J1, U, Z, th1, info)) {
    double2 a[4] = { A[0], A[1], A[2], A[3] }, u[4] = {}, z[4] = {};
    int inf = 0;
    zhsvd2_any(a, J0, J1, u, z, th1, inf);
#pragma unroll
    for (int k = 0; k < 4; ++k) { A[k] = a[k]; U[k] = u[k]; Z[k] = z[k]; }
    info = inf;
  }
}

// complex rotation coefficients: BA (src/Z/ztransf.F90:298-364) and AB / ABODNZF2 (:385-447, :478-636)
struct ZRot {
  double2 r1, r2, m1, m2;
  int c1, c2;
};

// n/d as zratio, straight-line, for nonzero near d
__device__ __forceinline__ double2 zratio_near(double2 n, double2 d)
{
  const bool real = (d.y == 0.0);
  const double f = hypot2_near(d.x, d.y), y = recip(f);
  const double2 m = zzmul(conj(zquot(d, f, y)), n);
  const double g = real ? d.x : f;
  return zquot(real ? n : m, g, recip(g));
}

// the coefficients of a rotation: per side the ratio of the smaller to the larger of two entries
// (a1, b1), (a2, b2) of B and the larger one (ties: the first)
__device__ __forceinline__ ZRot zrot_of(double2 a1, double2 b1, double2 a2, double2 b2)
{
  ZRot t;
  const double big = 2.037035976334486e+90;  // 2^300
  const bool ok = near_parts(a1) && near_parts(b1) && near_parts(a2) && near_parts(b2) &&
                  fmax(fmax(fabs(a1.x), fabs(a1.y)), fmax(fabs(b1.x), fabs(b1.y))) <= big &&
                  fmax(fmax(fabs(a2.x), fabs(a2.y)), fmax(fabs(b2.x), fabs(b2.y))) <= big &&
                  !(zeq0(a1) && zeq0(b1)) && !(zeq0(a2) && zeq0(b2));
  if (ok) {
    t.c1 = (zabs_near(a1) >= zabs_near(b1));
    t.c2 = (zabs_near(a2) >= zabs_near(b2));
    t.m1 = t.c1 ? a1 : b1;
    t.m2 = t.c2 ? a2 : b2;
    t.r1 = zratio_near(t.c1 ? b1 : a1, t.m1);
    t.r2 = zratio_near(t.c2 ? b2 : a2, t.m2);
  }
  else {
    t.c1 = (zabs(a1) >= zabs(b1));
    t.c2 = (zabs(a2) >= zabs(b2));
    t.m1 = t.c1 ? a1 : b1;
    t.m2 = t.c2 ? a2 : b2;
    t.r1 = zratio_call(t.c1 ? b1 : a1, t.m1);
    t.r2 = zratio_call(t.c2 ? b2 : a2, t.m2);
  }
  return t;
}

__device__ __forceinline__ ZRot zrot_ba(const double2 B[4], int quirk)
{
  ZRot t = zrot_of(B[M11], B[M12], B[M22], B[M21]);
  // src/Z/ztransf.F90:325 uses R1 in the (c1, !c2) branch where src/D/dtransf.F90:155 uses R2
  if (quirk && t.c1 && !t.c2) t.r2 = t.r1;
  return t;
}

// BA applies ZZFMA(R, data, data) then ZZMUL(XX, B)
__device__ __forceinline__ void zrot_apply_ba(const ZRot &t, double2 &x, double2 &y)
{
  const double2 xx = t.c1 ? zzfma(t.r1, y, x) : zzfma(t.r1, x, y);
  const double2 yy = t.c2 ? zzfma(t.r2, x, y) : zzfma(t.r2, y, x);
  x = zzmul(xx, t.m1);
  y = zzmul(yy, t.m2);
}

__device__ __forceinline__ ZRot zrot_ab(const double2 B[4]) { return zrot_of(B[M11], B[M21], B[M22], B[M12]); }

// AB and ABODNZF2 apply ZZFMA(data, R, data) then ZZMUL(XX, B)
__device__ __forceinline__ void zrot_apply_ab(const ZRot &t, double2 &x, double2 &y)
{
  const double2 xx = t.c1 ? zzfma(y, t.r1, x) : zzfma(x, t.r1, y);
  const double2 yy = t.c2 ? zzfma(x, t.r2, y) : zzfma(y, t.r2, x);
  x = zzmul(xx, t.m1);
  y = zzmul(yy, t.m2);
}

}  // namespace jk
