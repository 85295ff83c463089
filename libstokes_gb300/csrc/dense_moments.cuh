// dense_moments.cuh -- pair moments of the dense builders: the sums of scalar x
// e..e over the images and reciprocal vectors of a pair that its 3 x 3, 6 x 6
// or 11 x 11 block is linear in (src/ewald.c:1092-1677, src/ft.c:61-75,
// src/fts.c:72-104).
#pragma once

#include "ewald_device.cuh"

namespace lsg {

template <int V> struct Moments;
template <> struct Moments<0> { static constexpr int N = 7; };
template <> struct Moments<1> { static constexpr int N = 17; };
template <> struct Moments<2> { static constexpr int N = 68; };
// layout: A0 | A2[6] | B1[3] | C0 | C2[6] | G1[3] | G2[3] | G3[10] | H2[6] |
//         M4[15] | M2[6] | M3 | M4b[6] | M5
enum {
  MO_A0 = 0, MO_A2 = 1, MO_B1 = 7, MO_C0 = 10, MO_C2 = 11,
  MO_G1 = 17, MO_G2 = 20, MO_G3 = 23, MO_H2 = 33, MO_M4 = 39, MO_M2 = 54,
  MO_M3 = 60, MO_M4B = 61, MO_M5 = 67
};

// symmetric index tables: 2nd order (xx xy xz yy yz zz), 3rd, 4th
__host__ __device__ __forceinline__ int sym2 (int a, int b)
{
  if (a > b) { int t = a; a = b; b = t; }
  return a == 0 ? b : (a == 1 ? 2 + b : 5);
}
__host__ __device__ __forceinline__ int sym3 (int a, int b, int c)
{
  // sort a <= b <= c
  if (a > b) { int t = a; a = b; b = t; }
  if (b > c) { int t = b; b = c; c = t; }
  if (a > b) { int t = a; a = b; b = t; }
  // xxx xxy xxz xyy xyz xzz yyy yyz yzz zzz
  const int nx = (a == 0) + (b == 0) + (c == 0);
  const int ny = (a == 1) + (b == 1) + (c == 1);
  // enumerate by (nx, ny)
  if (nx == 3) return 0;
  if (nx == 2) return ny == 1 ? 1 : 2;
  if (nx == 1) return ny == 2 ? 3 : (ny == 1 ? 4 : 5);
  return ny == 3 ? 6 : (ny == 2 ? 7 : (ny == 1 ? 8 : 9));
}
__host__ __device__ __forceinline__ int sym4 (int a, int b, int c, int d)
{
  // xxxx xxxy xxxz xxyy xxyz xxzz xyyy xyyz xyzz xzzz yyyy yyyz yyzz yzzz zzzz
  const int nx = (a == 0) + (b == 0) + (c == 0) + (d == 0);
  const int ny = (a == 1) + (b == 1) + (c == 1) + (d == 1);
  switch (nx)
    {
    case 4: return 0;
    case 3: return ny == 1 ? 1 : 2;
    case 2: return ny == 2 ? 3 : (ny == 1 ? 4 : 5);
    case 1: return ny == 3 ? 6 : (ny == 2 ? 7 : (ny == 1 ? 8 : 9));
    default: return ny == 4 ? 10 : (ny == 3 ? 11 : (ny == 2 ? 12 : (ny == 1 ? 13 : 14)));
    }
}

template <int V, typename R = double>
__host__ __device__ __forceinline__ void
moments_add (const R e[3], const PairScalars<R> &s, R *mo)
{
  const R e2[6] = {e[0] * e[0], e[0] * e[1], e[0] * e[2], e[1] * e[1], e[1] * e[2], e[2] * e[2]};
  const R a2 = s.xa - s.ya;
  mo[MO_A0] += s.ya;
#pragma unroll
  for (int q = 0; q < 6; q++) mo[MO_A2 + q] += a2 * e2[q];
  if (V == V_F) return;
  const R c2 = s.xc - s.yc;
#pragma unroll
  for (int q = 0; q < 3; q++) mo[MO_B1 + q] += s.yb * e[q];
  mo[MO_C0] += s.yc;
#pragma unroll
  for (int q = 0; q < 6; q++) mo[MO_C2 + q] += c2 * e2[q];
  if (V == V_FT) return;
  const R g1 = -s.xg / R (3.0), g2 = s.yg, g3 = s.xg - R (2.0) * s.yg;
  const R m1 = R (1.5) * s.xm - R (2.0) * s.ym + R (0.5) * s.zm;
  const R m2 = -R (0.5) * s.xm + R (0.5) * s.zm;
  const R m3 = s.xm / R (6.0) - R (0.5) * s.zm;
  const R m4 = R (0.5) * s.ym - R (0.5) * s.zm;
  const R m5 = R (0.5) * s.zm;
#pragma unroll
  for (int q = 0; q < 3; q++)
    {
      mo[MO_G1 + q] += g1 * e[q];
      mo[MO_G2 + q] += g2 * e[q];
    }
  // e3: xxx xxy xxz xyy xyz xzz yyy yyz yzz zzz
  const R e3[10] = {e2[0] * e[0], e2[0] * e[1], e2[0] * e[2], e2[1] * e[1], e2[1] * e[2],
                         e2[2] * e[2], e2[3] * e[1], e2[3] * e[2], e2[4] * e[2], e2[5] * e[2]};
#pragma unroll
  for (int q = 0; q < 10; q++) mo[MO_G3 + q] += g3 * e3[q];
#pragma unroll
  for (int q = 0; q < 6; q++)
    {
      mo[MO_H2 + q] += s.yh * e2[q];
      mo[MO_M2 + q] += m2 * e2[q];
      mo[MO_M4B + q] += m4 * e2[q];
    }
  // e4: xxxx xxxy xxxz xxyy xxyz xxzz xyyy xyyz xyzz xzzz yyyy yyyz yyzz yzzz zzzz
  const R e4[15] = {e2[0] * e2[0], e2[0] * e2[1], e2[0] * e2[2], e2[0] * e2[3], e2[0] * e2[4],
                         e2[0] * e2[5], e2[1] * e2[3], e2[1] * e2[4], e2[1] * e2[5], e2[2] * e2[5],
                         e2[3] * e2[3], e2[3] * e2[4], e2[3] * e2[5], e2[4] * e2[5], e2[5] * e2[5]};
#pragma unroll
  for (int q = 0; q < 15; q++) mo[MO_M4 + q] += m1 * e4[q];
  mo[MO_M3] += m3;
  mo[MO_M5] += m5;
}

template <typename R = double>
__host__ __device__ __forceinline__ R
levi (int a, int b, int c)
{
  if (a == b || b == c || a == c) return R (0);
  return ((a == 0 && b == 1) || (a == 1 && b == 2) || (a == 2 && b == 0)) ? R (1) : R (-1);
}

// stresslet slots (xx, xy, xz, yz, yy) -> tensor indices
__host__ __device__ __forceinline__ void
slot_ab (int q, int &a, int &b)
{
  const int A[5] = {0, 0, 0, 1, 1}, B[5] = {0, 1, 2, 2, 1};
  a = A[q];
  b = B[q];
}

template <typename R = double>
__host__ __device__ __forceinline__ R kd (int a, int b) { return a == b ? R (1) : R (0); }

// G_(ab)c from moments
template <typename R>
__host__ __device__ __forceinline__ R
g_tensor (const R *mo, int a, int b, int c)
{
  return mo[MO_G1 + c] * kd<R> (a, b) + mo[MO_G2 + a] * kd<R> (b, c) + mo[MO_G2 + b] * kd<R> (a, c)
    + mo[MO_G3 + sym3 (a, b, c)];
}
// H_(ab)c = sum_n eps_bcn H2[an] + eps_acn H2[bn]
template <typename R>
__host__ __device__ __forceinline__ R
h_tensor (const R *mo, int a, int b, int c)
{
  R v = R (0);
  for (int n = 0; n < 3; n++)
    v += levi<R> (b, c, n) * mo[MO_H2 + sym2 (a, n)] + levi<R> (a, c, n) * mo[MO_H2 + sym2 (b, n)];
  return v;
}
// M_(ab)(cd)
template <typename R>
__host__ __device__ __forceinline__ R
m_tensor (const R *mo, int a, int b, int c, int d)
{
  return mo[MO_M4 + sym4 (a, b, c, d)]
    + mo[MO_M2 + sym2 (c, d)] * kd<R> (a, b) + mo[MO_M2 + sym2 (a, b)] * kd<R> (c, d)
    + mo[MO_M3] * kd<R> (a, b) * kd<R> (c, d)
    + mo[MO_M4B + sym2 (a, d)] * kd<R> (b, c) + mo[MO_M4B + sym2 (a, c)] * kd<R> (b, d)
    + mo[MO_M4B + sym2 (b, d)] * kd<R> (a, c) + mo[MO_M4B + sym2 (b, c)] * kd<R> (a, d)
    + mo[MO_M5] * (kd<R> (a, c) * kd<R> (b, d) + kd<R> (b, c) * kd<R> (a, d));
}

// one block entry (extracted form) from the moments; same = (i == j)
template <int V, typename R = double>
__host__ __device__ __forceinline__ R
block_entry (const R *mo, int row, int col, bool same)
{
  const R sgn = same ? R (-1) : R (1);   // src/ft.c:61-75, src/fts.c:72-104
  if (row < 3)
    {
      const int a = row;
      if (col < 3)
        return mo[MO_A0] * kd<R> (a, col) + mo[MO_A2 + sym2 (a, col)];
      if (col < 6)
        {
          const int b = col - 3;
          R v = R (0);
          for (int n = 0; n < 3; n++) v += levi<R> (a, b, n) * mo[MO_B1 + n];
          return sgn * v;
        }
      int p, q;
      slot_ab (col - 6, p, q);
      return -sgn * g_tensor (mo, p, q, a);
    }
  if (row < 6)
    {
      const int a = row - 3;
      if (col < 3)
        {
          R v = R (0);
          for (int n = 0; n < 3; n++) v += levi<R> (a, col, n) * mo[MO_B1 + n];
          return v;
        }
      if (col < 6)
        return mo[MO_C0] * kd<R> (a, col - 3) + mo[MO_C2 + sym2 (a, col - 3)];
      int p, q;
      slot_ab (col - 6, p, q);
      return h_tensor (mo, p, q, a);
    }
  int a, b;
  slot_ab (row - 6, a, b);
  if (col < 3) return g_tensor (mo, a, b, col);
  if (col < 6) return h_tensor (mo, a, b, col - 3);
  int c, d;
  slot_ab (col - 6, c, d);
  return m_tensor (mo, a, b, c, d);
}

}  // namespace lsg
