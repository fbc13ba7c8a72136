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

// both parts zero or at least 2^-300 in magnitude
__device__ __forceinline__ bool near_parts(double2 z)
{
  return near_ratio(fabs(z.x)) && near_ratio(fabs(z.y));
}

// hypot2 for two operands below 2^300 of which the larger is zero or at least 2^-1000
__device__ __forceinline__ double hypot2_near0(double x, double y)
{
  return (x == 0.0 && y == 0.0) ? 0.0 : hypot2_near(x, y);
}
__device__ __forceinline__ double zabs_near(double2 a) { return hypot2_near0(a.x, a.y); }

// a division of both parts by the same number, y = recip(b)
__device__ __forceinline__ double2 zquot(double2 a, double b, double y) { return zc(quot(a.x, b, y), quot(a.y, b, y)); }

// ZPOLAR (see zpolar) for parts that are zero or near
__device__ __forceinline__ void zpolar_near(double2 z, double2 &e)
{
  const double a = zabs_near(z), y = recip(a);
  const bool zero = (a == 0.0);
  const double c = copysign(zero ? 1.0 : fmin(quot(fabs(z.x), a, y), 1.0), z.x);
  e = zc(c, zero ? z.y : quot(z.y, a, y));
}

// the exponents of a block's nonzero parts all within 2^-150 of the largest, which lies in
// 2^(+-100), and no zero column
__device__ __forceinline__ bool znear_block(const double2 A[4])
{
  int hi = 0, lo = 0x7FF;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = (__double2hiint(A[k].x) >> 20) & 0x7FF, f = (__double2hiint(A[k].y) >> 20) & 0x7FF;
    hi = max(hi, max(e, f));
    lo = imin(lo, imin((A[k].x == 0.0) ? 0x7FF : e, (A[k].y == 0.0) ? 0x7FF : f));
  }
  return hi >= 923 && hi <= 1123 && lo >= hi - 150 && !(zeq0(A[M11]) && zeq0(A[M21])) && !(zeq0(A[M12]) && zeq0(A[M22]));
}

// ZHSVD2 for the blocks that znear_block takes: the operations of zhsvd2_any in the same order on
// the unscaled block, as dhsvd2_near.  Every quantity that is divided is tested (near_parts,
// near_ratio), so that no product of two of them leaves the normal numbers.  Returns false, with
// nothing written, when the block does not allow it.
__device__ __forceinline__ bool zhsvd2_near(double2 Ain[4], const int J0, const int J1, double2 Uo[4], double2 Zo[4], double th1, int &info_o)
{
  if (!znear_block(Ain) || abs(J0) != 1 || abs(J1) != 1) return false;
  const double2 one = zc(1.0, 0.0), zero = zc(0.0, 0.0);
  double2 A[4] = { Ain[0], Ain[1], Ain[2], Ain[3] }, U[4] = { one, zero, zero, one }, Z[4] = { one, zero, zero, one };
  // ZHSVD2T, src/Z/ztransf.F90:641-835
  const bool d = zeq0(A[M21]) && zeq0(A[M12]);
  const double c = hypot2_near(zabs_near(A[M11]), zabs_near(A[M21]));
  const double t0 = hypot2_near(zabs_near(A[M12]), zabs_near(A[M22]));
  const bool p = (c < t0);
  const double w = p ? t0 : c;
  if (p) {
    zswap(A[M11], A[M12]); zswap(A[M21], A[M22]);
    if (J0 == J1) { zswap(Z[M11], Z[M12]); zswap(Z[M21], Z[M22]); }
  }
  double2 r, s;
  zpolar_near(A[M11], r);
  zpolar_near(A[M21], s);
  if (zne1(r)) {
    const double2 v = conj(r);
    U[M11] = zzmul(U[M11], v); U[M12] = zzmul(U[M12], v);
    A[M11] = zzmul(A[M11], v); A[M12] = zzmul(A[M12], v);
  }
  if (zne1(s)) {
    const double2 v = conj(s);
    U[M21] = zzmul(U[M21], v); U[M22] = zzmul(U[M22], v);
    A[M21] = zzmul(A[M21], v); A[M22] = zzmul(A[M22], v);
  }
  if (A[M11].x < A[M21].x) {
    zswap(U[M11], U[M21]); zswap(U[M12], U[M22]);
    zswap(A[M11], A[M21]); zswap(A[M12], A[M22]);
  }
  if (!d) {
    if (!(A[M11].x > 0.0)) return false;
    const double t = quot(A[M21].x, A[M11].x, recip(A[M11].x));
    const double q = root(fma(t, t, 1.0)), y = recip(q);
    const double2 u11 = zdfma(t, U[M21], U[M11]), u21 = zdfma(-t, U[M11], U[M21]);
    const double2 u12 = zdfma(t, U[M22], U[M12]), u22 = zdfma(-t, U[M12], U[M22]);
    const double2 a1 = zdfma(t, A[M22], A[M12]), a2 = zdfma(-t, A[M12], A[M22]);
    U[M11] = zquot(u11, q, y); U[M21] = zquot(u21, q, y); U[M12] = zquot(u12, q, y); U[M22] = zquot(u22, q, y);
    A[M12] = zquot(a1, q, y); A[M22] = zquot(a2, q, y);
  }
  A[M11] = zc(w, 0.0);
  A[M21] = zero;
  if (!near_parts(A[M12]) || !near_parts(A[M22])) return false;
  if ((J0 != J1) && p) {
    zswap(A[M11], A[M12]); zswap(A[M21], A[M22]);
    zswap(U[M11], U[M21]); zswap(U[M12], U[M22]);
    zswap(A[M11], A[M21]); zswap(A[M12], A[M22]);
    zpolar_near(A[M21], s);
    if (zne1(s)) {
      const double2 v = conj(s);
      Z[M11] = zzmul(Z[M11], v); Z[M21] = zzmul(Z[M21], v);
      A[M11] = zzmul(A[M11], v); A[M21] = zzmul(A[M21], v);
    }
    if (!near_parts(A[M11])) return false;
    zpolar_near(A[M11], r);
    if (zne1(r)) {
      const double2 v = conj(r);
      U[M11] = zzmul(U[M11], v); U[M12] = zzmul(U[M12], v);
      A[M11] = zzmul(A[M11], v);
    }
  }
  else {
    zpolar_near(A[M12], r);
    if (zne1(r)) {
      const double2 v = conj(r);
      Z[M12] = zzmul(Z[M12], v); Z[M22] = zzmul(Z[M22], v);
      A[M12] = zzmul(A[M12], v); A[M22] = zzmul(A[M22], v);
    }
    if (!near_parts(A[M22])) return false;
    zpolar_near(A[M22], s);
    if (zne1(s)) {
      const double2 v = conj(s);
      U[M21] = zzmul(U[M21], v); U[M22] = zzmul(U[M22], v);
      A[M22] = zzmul(A[M22], v);
    }
  }
  int info = d ? 0 : 1;
  double w11 = A[M11].x, w22 = A[M22].x;
  if (info) {
    double W[4] = { A[M11].x, A[M21].x, A[M12].x, A[M22].x };
    NearK k;
    if (!khsvd2_near(W, J0, J1, th1, info, k)) return false;
    if (!near_ratio(fabs(k.tu)) || !near_ratio(fabs(k.tz))) return false;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (!near_parts(U[i]) || !near_parts(Z[i])) return false;
    const double2 u11 = zdfma(k.tu, U[M21], U[M11]), u21 = zdfma(-k.tu, U[M11], U[M21]);
    const double2 u12 = zdfma(k.tu, U[M22], U[M12]), u22 = zdfma(-k.tu, U[M12], U[M22]);
    U[M11] = zquot(u11, k.cu, k.yu); U[M21] = zquot(u21, k.cu, k.yu);
    U[M12] = zquot(u12, k.cu, k.yu); U[M22] = zquot(u22, k.cu, k.yu);
    const double2 z11 = zdfma(k.tz, Z[M12], Z[M11]), z12 = zdfma(k.c12, Z[M11], Z[M12]);
    const double2 z21 = zdfma(k.tz, Z[M22], Z[M21]), z22 = zdfma(k.c12, Z[M21], Z[M22]);
    Z[M11] = zquot(z11, k.cz, k.yz); Z[M12] = zquot(z12, k.cz, k.yz);
    Z[M21] = zquot(z21, k.cz, k.yz); Z[M22] = zquot(z22, k.cz, k.yz);
    if (!(info & 8)) { w11 = k.g0; w22 = k.g1; }
    else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!near_parts(A[i])) return false;
      const double2 a11 = zdfma(k.tu, A[M21], A[M11]), a21 = zdfma(-k.tu, A[M11], A[M21]);
      const double2 a12 = zdfma(k.tu, A[M22], A[M12]), a22 = zdfma(-k.tu, A[M12], A[M22]);
      A[M11] = zquot(a11, k.cu, k.yu); A[M21] = zquot(a21, k.cu, k.yu);
      A[M12] = zquot(a12, k.cu, k.yu); A[M22] = zquot(a22, k.cu, k.yu);
      const double2 b11 = zdfma(k.tz, A[M12], A[M11]), b12 = zdfma(k.c12, A[M11], A[M12]);
      const double2 b21 = zdfma(k.tz, A[M22], A[M21]), b22 = zdfma(k.c12, A[M21], A[M22]);
      A[M11] = zquot(b11, k.cz, k.yz); A[M12] = zquot(b12, k.cz, k.yz);
      A[M21] = zquot(b21, k.cz, k.yz); A[M22] = zquot(b22, k.cz, k.yz);
    }
  }
  if (!(info & 8)) { A[M11] = zc(w11, 0.0); A[M22] = zc(w22, 0.0); }
  zhsvd2s(A, J0, J1, U, Z, info);
#pragma unroll
  for (int i = 0; i < 4; ++i) { Ain[i] = A[i]; Uo[i] = U[i]; Zo[i] = Z[i]; }
  info_o = info;
  return true;
}

// ZHSVD2, src/Z/ztransf.F90:925-1009
__device__ __forceinline__ void zhsvd2(double2 A[4], const int J0, const int J1, double2 U[4], double2 Z[4], double th1, int &info)
{
  if (!zhsvd2_near(A, J0, J1, U, Z, th1, info)) {
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
