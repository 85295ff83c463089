// radial.cuh -- the independent radial functions of a real-space pair term of
// equal spheres, and their table (real_tab.cu, where both are explained).
#pragma once

#include "ewald_device.cuh"

namespace lsg {

constexpr int RT_LOG = 6;                     // log2 of the bins per octave
constexpr int RT_DEG = 8;                     // coefficients per function

template <int V> struct NFun;
template <> struct NFun<0> { static constexpr int value = 2; };
template <> struct NFun<1> { static constexpr int value = 5; };
template <> struct NFun<2> { static constexpr int value = 10; };

// the independent coefficients at distance r, s = r^2
template <int V>
__device__ __forceinline__ void
radial (double xi, double xisp, double r, double s, double *f)
{
  PairScalars<double> c;
  real_scalars_mono<V, double> (xi, xisp, r, c);
  f[0] = c.ya;
  f[1] = (c.xa - c.ya) / s;
  if (V == V_F) return;
  f[2] = c.yb / r;
  f[3] = c.yc;
  f[4] = (c.xc - c.yc) / s;
  if (V == V_FT) return;
  f[5] = c.yg / r;                                            // g2
  f[6] = (c.xg - 2.0 * c.yg) / (r * s);                       // g3
  f[7] = (1.5 * c.xm - 2.0 * c.ym + 0.5 * c.zm) / (s * s);    // m1
  f[8] = (c.ym - c.zm) / s;                                   // m4
  f[9] = c.zm;
}

__device__ __forceinline__ double
bin_mid (int bin)
{
  return __hiloint2double ((bin << (20 - RT_LOG)) | (1 << (19 - RT_LOG)), 0);
}

// bin of s, less the first one of the table
__device__ __forceinline__ int
radial_bin (double s, int bin0)
{
  return (__double2hiint (s) >> (20 - RT_LOG)) - bin0;
}

// the functions at s in bin >= 0
template <int NF>
__device__ __forceinline__ void
table_radial (const double *tab, double s, int bin, int bin0, int nbin, double *f)
{
  const double z = s - bin_mid (bin + bin0);
  const double2 *c = reinterpret_cast<const double2 *> (tab) + (size_t) min (bin, nbin - 1) * (NF * RT_DEG / 2);
#pragma unroll
  for (int q = 0; q < NF; q++)
    {
      const double2 c3 = __ldg (c + 4 * q + 3), c2 = __ldg (c + 4 * q + 2),
                    c1 = __ldg (c + 4 * q + 1), c0 = __ldg (c + 4 * q);
      f[q] = fma (fma (fma (fma (fma (fma (fma (c3.y, z, c3.x), z, c2.y), z, c2.x), z, c1.y),
                            z, c1.x), z, c0.y), z, c0.x);
    }
}

// y += M x_j of one pair at displacement d, s = d.d, coefficients f
template <int V, typename R>
__device__ __forceinline__ void
apply_radial (const R d[3], R s, const R *f, const R *__restrict__ x, R *y)
{
  const R F0 = x[0], F1 = x[1], F2 = x[2];
  const R dF = d[0] * F0 + d[1] * F1 + d[2] * F2;
  R along = f[1] * dF;
  if (V == V_F)
    {
      y[0] += fma (f[0], F0, along * d[0]);
      y[1] += fma (f[0], F1, along * d[1]);
      y[2] += fma (f[0], F2, along * d[2]);
      return;
    }
  const R T0 = x[3], T1 = x[4], T2 = x[5];
  const R t0 = T1 * d[2] - T2 * d[1], t1 = T2 * d[0] - T0 * d[2], t2 = T0 * d[1] - T1 * d[0];
  const R f0 = F1 * d[2] - F2 * d[1], f1 = F2 * d[0] - F0 * d[2], f2 = F0 * d[1] - F1 * d[0];
  const R w = f[4] * (d[0] * T0 + d[1] * T1 + d[2] * T2);
  y[3] = fma (w, d[0], fma (f[3], T0, fma (f[2], f0, y[3])));
  y[4] = fma (w, d[1], fma (f[3], T1, fma (f[2], f1, y[4])));
  y[5] = fma (w, d[2], fma (f[3], T2, fma (f[2], f2, y[5])));
  if (V == V_FT)
    {
      y[0] = fma (along, d[0], fma (f[0], F0, fma (f[2], t0, y[0])));
      y[1] = fma (along, d[1], fma (f[0], F1, fma (f[2], t1, y[1])));
      y[2] = fma (along, d[2], fma (f[0], F2, fma (f[2], t2, y[2])));
      return;
    }
  const R sxx = x[6], sxy = x[7], sxz = x[8], syz = x[9], syy = x[10];
  const R Sxx = fma (R (2), sxx, syy), Syy = fma (R (2), syy, sxx);
  const R s0 = Sxx * d[0] + sxy * d[1] + sxz * d[2];
  const R s1 = sxy * d[0] + Syy * d[1] + syz * d[2];
  const R s2 = sxz * d[0] + syz * d[1];
  const R ss = d[0] * s0 + d[1] * s1 + d[2] * s2, tr = Sxx + Syy;
  const R third = R (-1.0 / 3.0), g2 = f[5], g3 = f[6], m1 = f[7], m4 = f[8], zm = f[9];
  const R g1 = fma (g3, s, R (2) * g2) * third;
  const R m2 = fma (m1, s, R (2) * m4) * third;
  const R m3 = fma (m2, s, zm) * third;
  along = fma (-g1, tr, fma (-g3, ss, along));
  const R n2 = R (-2) * g2, nc = -f[4];
  y[0] = fma (along, d[0], fma (f[0], F0, fma (f[2], t0, fma (n2, s0, y[0]))));
  y[1] = fma (along, d[1], fma (f[0], F1, fma (f[2], t1, fma (n2, s1, y[1]))));
  y[2] = fma (along, d[2], fma (f[0], F2, fma (f[2], t2, fma (n2, s2, y[2]))));
  const R h2 = R (2) * nc;
  y[3] = fma (h2, d[1] * s2 - d[2] * s1, y[3]);
  y[4] = fma (h2, d[2] * s0 - d[0] * s2, y[4]);
  y[5] = fma (h2, d[0] * s1 - d[1] * s0, y[5]);
  const R v0 = fma (g2, F0, fma (nc, t0, m4 * s0));
  const R v1 = fma (g2, F1, fma (nc, t1, m4 * s1));
  const R v2 = fma (g2, F2, fma (nc, t2, m4 * s2));
  const R dE = fma (g1, dF, fma (m2, ss, m3 * tr));
  const R ee = fma (g3, dF, fma (m1, ss, m2 * tr));
  // ee d d + d V + V d = d (V + ee d / 2) + (V + ee d / 2) d
  const R he = R (0.5) * ee;
  const R w0 = fma (he, d[0], v0), w1 = fma (he, d[1], v1), w2 = fma (he, d[2], v2);
  y[6] += fma (R (2) * d[0], w0, fma (zm, Sxx, dE));
  y[7] = fma (d[0], w1, fma (d[1], w0, fma (zm, sxy, y[7])));
  y[8] = fma (d[0], w2, fma (d[2], w0, fma (zm, sxz, y[8])));
  y[9] = fma (d[1], w2, fma (d[2], w1, fma (zm, syz, y[9])));
  y[10] += fma (R (2) * d[1], w1, fma (zm, Syy, dE));
}

// the same functions in FP32 with the unit vector for d (s = 1): the closed
// forms of real_scalars_mono_ri, their combinations multiplied out and the
// polynomials shared (65 multiply-adds instead of 160).  ri = 1 / r.
template <int V>
__device__ __forceinline__ void
radial_f32 (float xi, float xisp, float r, float ri, float *f)
{
  const float x = xi * r, u = x * x, ri2 = ri * ri;
  float ec, eg;
  erfc_exp<float> (x, u, ec, eg);
  const float ex = xisp * eg, ecr = ri * ec;
  const float p1 = fmaf (u, fmaf (u, fmaf (u, 4.f, -20.f), 14.f), 1.f);
  const float p2 = fmaf (u, fmaf (u, fmaf (u, -4.f, 16.f), -2.f), -3.f);
  f[0] = fmaf (fmaf (0.5f, ri2, 0.75f), ecr, fmaf (p1, ri2, fmaf (3.f, u, -4.5f)) * ex);
  f[1] = fmaf (fmaf (-1.5f, ri2, 0.75f), ecr, fmaf (p2, ri2, fmaf (-3.f, u, 1.5f)) * ex);
  if (V == V_F) return;
  const float ecr2 = ri * ecr, ecr3 = ri2 * ecr, er = ri * ex, er2 = ri * er;
  f[2] = fmaf (-0.75f, ecr2, fmaf (u, fmaf (u, -3.f, 9.f), -1.5f) * er);
  f[3] = fmaf (-0.375f, ecr3, -0.75f * p1 * er2);
  f[4] = fmaf (1.125f, ecr3, -0.75f * p2 * er2);
  if (V == V_FT) return;
  const float p3 = fmaf (u, fmaf (u, fmaf (u, fmaf (u, -4.f, 26.f), -26.f), -2.f), -3.f);
  const float p4 = fmaf (u, fmaf (u, fmaf (u, fmaf (u, -6.4f, 32.f), -3.2f), -8.f), -12.f);
  const float p5 = fmaf (u, fmaf (u, fmaf (u, fmaf (u, fmaf (u, 9.6f, -57.6f), 4.8f), 16.8f), 42.f), 63.f);
  const float p6 = fmaf (u, fmaf (u, fmaf (u, fmaf (u, fmaf (u, -4.8f, 36.f), -38.4f), -4.8f), -12.f), -18.f);
  f[5] = fmaf (1.2f * ri2, ecr2, fmaf (-0.8f * p3, ri2, u * fmaf (3.f, u, -6.f)) * er);
  f[6] = fmaf (fmaf (-6.f, ri2, 2.25f), ecr2, fmaf (p4, ri2, fmaf (u, fmaf (u, -6.f, 3.f), 4.5f)) * er);
  f[7] = fmaf (fmaf (31.5f, ri2, -11.25f), ecr3,
               fmaf (p5, ri2, fmaf (u, fmaf (u, fmaf (u, 12.f, -6.f), -15.f), -22.5f)) * er2);
  f[8] = fmaf (fmaf (-9.f, ri2, 2.25f), ecr3,
               fmaf (p6, ri2, fmaf (u, fmaf (u, fmaf (u, -6.f, 12.f), 3.f), 4.5f)) * er2);
  f[9] = fmaf (1.8f * ri2, ecr3, fmaf (-1.2f * p3, ri2, u * fmaf (6.f, u, -12.f)) * er2);
}

}  // namespace lsg
