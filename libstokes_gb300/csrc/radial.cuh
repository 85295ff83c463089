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

}  // namespace lsg
