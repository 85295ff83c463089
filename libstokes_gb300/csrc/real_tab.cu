// real_tab.cu -- FP64 real-space pair sum of equal spheres from a table of
// its radial functions.
//
// The sum is bound by the FP64 pipe (about two lanes a clock and SM), so what
// counts is the FP64 instructions of a pair term.  Evaluated from the closed
// forms an FTS term takes about 970 of them: a square root, a division, erfc,
// exp, eleven scalars and the pair tensors.  Written in the plain
// displacement d instead of the unit vector, every coefficient is a smooth
// function of s = d.d alone (no square root, no division), and tracelessness
// leaves 2 (F), 5 (FT) or 10 (FTS) independent ones:
//
//   U = ya F + a2 (d.F) d + yb T x d - (g1 tr S + g3 dSd) d - 2 g2 S d
//   W = yb F x d + yc T + c2 (d.T) d - 2 c2 d x (S d)
//   E = (g1 d.F + m2 dSd + m3 tr S) I + (g3 d.F + m1 dSd + m2 tr S) d d
//       + d V + V d + zm S,     V = g2 F - c2 T x d + m4 S d
//   g1 = -(g3 s + 2 g2) / 3,  m2 = -(m1 s + 2 m4) / 3,  m3 = -(m2 s + zm) / 3
//
// (S the full contraction S' of ewald_device.cuh; its yh equals yc - xc).
// Each is a polynomial of degree 7 in s - s_mid per bin, RT_BINS bins per
// octave of s: 7 FMAs a function, about 200 FP64 instructions an FTS term.
// The bin and its midpoint come from the bits of s.  The truncation of such a
// bin is below 2^-53 of the function for powers s^-5.5 (bin half width over s
// at most 1/128: 2^-56 times 2^10 for the binomial and 2^-7 for Chebyshev
// nodes); the table is made on the device from the closed forms, with the
// change of basis in double-double.
//
// Far pairs.  The functions fall off as exp(-xi^2 r^2), so beyond xi r = FAR_U
// a pair contributes less than about 1e-9 of a near one, and single precision
// there costs the sum less than FP64 rounding does: 6e-8 of 1e-9 at the
// border, sqrt(300) such pairs, falling by e^-2u per 1 / xi further out, is
// 2e-16 of a near term.  About half of the pairs within the cutoff (xi r =
// 6.6) are far.  Only the relative error of s would be magnified (by u^2), so
// s and its distance to the bin's middle stay FP64 (8 instructions); the
// functions, the tensors and the sum of the far pairs are FP32.
//
// Positions are the 64-bit fixed-point fractional coordinates of the
// reciprocal sum, so the minimum image is the integer overflow and a
// displacement carries one rounding, however close the pair; the conversion
// to FP64 is done in integers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "ewald_device.cuh"
#include "radial.cuh"
#include "real_tab.h"

namespace lsg {
namespace {

constexpr int RT_T = 128;                     // threads per CTA: one target
constexpr int RT_W = RT_T / 32;               // warps
constexpr int RT_SEG = 1024;                  // accepted pairs a warp lists at a time
static_assert (32 * REAL_TAB_MAXIMG <= RT_SEG, "32 sources with every offset fit a list");

// coefficients of one bin: values at the Chebyshev nodes, then the monomial
// coefficients c_k = sum_n B[k][n] f(node n) / h^k by compensated sums
struct Basis {
  double hi[RT_DEG][RT_DEG], lo[RT_DEG][RT_DEG];
  double node[RT_DEG];
};

template <int V>
__global__ void __launch_bounds__ (RT_DEG * NFun<V>::value)
k_rt_table (Basis b, int bin0, double xi, double xisp, double *tab, float *tabf)
{
  constexpr int NF = NFun<V>::value;
  __shared__ double s_f[RT_DEG][NF];
  const int bin = bin0 + blockIdx.x, t = threadIdx.x;
  const double mid = bin_mid (bin);
  // half the bin: 2^(exponent - RT_LOG - 1)
  const double h = __hiloint2double (((bin >> RT_LOG) - RT_LOG - 1) << 20, 0);
  if (t < RT_DEG)
    {
      const double s = fma (h, b.node[t], mid);
      double f[NF];
      radial<V> (xi, xisp, sqrt (s), s, f);
      for (int q = 0; q < NF; q++) s_f[t][q] = f[q];
    }
  __syncthreads ();
  const int q = t / RT_DEG, k = t % RT_DEG;
  double sum = 0.0, err = 0.0;
  for (int n = 0; n < RT_DEG; n++)
    {
      const double f = s_f[n][q], p = b.hi[k][n] * f, pe = fma (b.hi[k][n], f, -p);
      const double v = sum + p, bb = v - sum;
      err += (sum - (v - bb)) + (p - bb) + pe + b.lo[k][n] * f;
      sum = v;
    }
  double c = sum + err;
  for (int n = 0; n < k; n++) c /= h;                   // h is a power of two
  tab[((size_t) blockIdx.x * NF + q) * RT_DEG + k] = c;
  tabf[((size_t) blockIdx.x * NF + q) * RT_DEG + k] = (float) c;
}

// pairs the table does not serve: nearer than its first bin, or under the
// rmin clamp (r raised to rm and e = d / r with the raised r,
// src/ewald.c:693-699).  At a split other than the struct's own a clamped
// pair contributes T(d / rm; s_ref(rm)) + T(d / r; s_xi(r) - s_ref(r)), the
// change of the clamp at the struct's split.
template <int V>
__device__ __noinline__ void
near_term (const RealTabArgs &a, double d0, double d1, double d2, double s, const double *x,
           double *z)
{
  const double d[3] = {d0, d1, d2};
  const double r = sqrt (s), rm = 2.0 * a.rmin;
  GenF<V, double> g;
  load_genf<V, double> (x, g);
  GenU<V, double> u;
  u.zero ();
  PairScalars<double> c;
  const double e[3] = {d[0] / r, d[1] / r, d[2] / r};
  if (r < rm)
    {
      const double ec[3] = {d[0] / rm, d[1] / rm, d[2] / rm};
      real_scalars_mono<V, double> (a.xi_ref, a.xi_ref * 0.56418958354775628, rm, c);
      pair_apply<V, double> (ec, c, g, u);
      split_diff<V, double> (a.xi_ref, a.xi, r, c);
    }
  else
    real_scalars_mono<V, double> (a.xi, a.xisp, r, c);
  pair_apply<V, double> (e, c, g, u);
#pragma unroll
  for (int q = 0; q < NComp<V>::value; q++) z[q] = u.v[q];
}

// v[0 .. P) summed over the warp, P a power of two <= 16: lane l ends up with
// the sum of element l / (32 / P).  P - 1 + 5 - log2 P additions instead of
// 5 P.
template <int P, typename R>
__device__ __forceinline__ R
warp_sums (R (&v)[P], int lane)
{
  int o = 16;
#pragma unroll
  for (int n = P / 2; n >= 1; n >>= 1, o >>= 1)
#pragma unroll
    for (int k = 0; k < n; k++)
      {
        const bool up = lane & o;
        const R keep = up ? v[k + n] : v[k], send = up ? v[k] : v[k + n];
        v[k] = keep + __shfl_xor_sync (0xffffffffu, send, o);
      }
  for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync (0xffffffffu, v[0], o);
  return v[0];
}

// One CTA per target.  Its threads test the sources (times the lattice
// offsets of a cutoff beyond half the box) in FP32 on the upper 32 bits of
// the fixed-point coordinates and list the accepted ones in shared memory (a
// segment per warp, so that the order and with it the sum is reproducible);
// then the warps take the entries of all segments 32 at a time, so that the
// FP64 pipe only sees accepted pairs and at most one partly filled warp per
// target and round.
template <int V>
__global__ void __launch_bounds__ (RT_T)
k_real_tab (RealTabArgs a)
{
  constexpr int C = NComp<V>::value, NF = NFun<V>::value;
  constexpr int P = C <= 4 ? 4 : (C <= 8 ? 8 : 16);
  __shared__ unsigned s_list[RT_W][RT_SEG];             // source | offset << 24
  __shared__ int s_n[RT_W], s_f[RT_W];                  // near entries, far entries (from the end)
  __shared__ double s_y[RT_W][P];
  const int i = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint4 qi = a.q[i];
  const ulonglong2 ua = reinterpret_cast<const ulonglong2 *> (a.u)[2 * i];
  const unsigned long long uz = a.u[4 * (size_t) i + 2];
  double y[P];
  float yf[P];
#pragma unroll
  for (int q = 0; q < P; q++)
    {
      y[q] = 0.0;
      yf[q] = 0.f;
    }
  // sources per warp and round: all of them times the offsets fit its segment
  const int per = RT_SEG / a.nimg / 32 * 32;
  for (int b0 = 0; b0 < a.np; b0 += RT_W * per)
    {
      const int j1 = min (a.np, b0 + (warp + 1) * per);
      int cnt = 0, far = 0;
      for (int jb = b0 + warp * per; jb < j1; jb += 32)
        {
          const int j = jb + lane;
          float x0 = 0.f, x1 = 0.f, x2 = 0.f;
          if (j < j1)
            {
              const uint4 qj = a.q[j];
              x0 = (float) (int) (qj.x - qi.x) * a.sf[0];
              x1 = (float) (int) (qj.y - qi.y) * a.sf[1];
              x2 = (float) (int) (qj.z - qi.z) * a.sf[2];
            }
          for (int m = 0; m < a.nimg; m++)
            {
              const float4 T = a.nimg > 1 ? a.off[m] : make_float4 (0.f, 0.f, 0.f, 0.f);
              const float dx = x0 + T.x, dy = x1 + T.y, dz = x2 + T.z;
              const float rr = dx * dx + dy * dy + dz * dz;
              const bool ok = j < j1 && (j != i || m != a.home) && rr < a.rc2;
              const bool out = ok && rr > a.far2;
              const unsigned near = __ballot_sync (0xffffffffu, ok && !out);
              const unsigned away = __ballot_sync (0xffffffffu, out), below = (1u << lane) - 1u;
              if (ok)
                s_list[warp][out ? RT_SEG - 1 - far - __popc (away & below)
                                 : cnt + __popc (near & below)]
                  = (unsigned) (j - b0) | (unsigned) m << 24;
              cnt += __popc (near);
              far += __popc (away);
            }
        }
      if (lane == 0)
        {
          s_n[warp] = cnt;
          s_f[warp] = far;
        }
      __syncthreads ();
      int n = 0, nf = 0;
#pragma unroll
      for (int w = 0; w < RT_W; w++)
        {
          n += s_n[w];
          nf += s_f[w];
        }
      // displacement of entry en in FP64
      auto displace = [&] (unsigned en, int j, double d[3]) {
        const ulonglong2 ub = reinterpret_cast<const ulonglong2 *> (a.u)[2 * (size_t) j];
        const unsigned long long vz = a.u[4 * (size_t) j + 2];
        int4 o = make_int4 (0, 0, 0, 0);
        if (a.nimg > 1) o = a.cell[en >> 24];
        // in units of 2^-60 of the box
        d[0] = int_to_double (image_diff (ua.x, ub.x) + ((long long) o.x << 60)) * a.s60[0];
        d[1] = int_to_double (image_diff (ua.y, ub.y) + ((long long) o.y << 60)) * a.s60[1];
        d[2] = int_to_double (image_diff (uz, vz) + ((long long) o.z << 60)) * a.s60[2];
      };
      for (int k = t; k < n; k += RT_T)
        {
          int w = 0, at = k;
          while (at >= s_n[w]) at -= s_n[w++];
          const unsigned en = s_list[w][at];
          const int j = b0 + (int) (en & 0xffffffu);
          double d[3];
          displace (en, j, d);
          const double s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
          const double *x = a.x + (size_t) C * j;
          const int bin = (__double2hiint (s) >> (20 - RT_LOG)) - a.bin0;
          if (bin < 0 || s < a.rm2)
            {
              // coincident points of distinct particles count as no pair
              if (s > 0.0)
                {
                  double v[C];
                  near_term<V> (a, d[0], d[1], d[2], s, x, v);
#pragma unroll
                  for (int q = 0; q < C; q++) y[q] += v[q];
                }
              continue;
            }
          double f[NF];
          table_radial<NF> (a.tab, s, bin, a.bin0, a.nbin, f);
          apply_radial<V, double> (d, s, f, x, y);
        }
      for (int k = t; k < nf; k += RT_T)
        {
          int w = 0, at = k;
          while (at >= s_f[w]) at -= s_f[w++];
          const unsigned en = s_list[w][RT_SEG - 1 - at];
          const int j = b0 + (int) (en & 0xffffffu);
          double d[3];
          displace (en, j, d);
          const double s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
          const int bin = (__double2hiint (s) >> (20 - RT_LOG)) - a.bin0;
          const float z = (float) (s - bin_mid (bin + a.bin0));
          const uint4 qj = a.q[j];
          float e[3] = {(float) (int) (qj.x - qi.x) * a.sf[0], (float) (int) (qj.y - qi.y) * a.sf[1],
                        (float) (int) (qj.z - qi.z) * a.sf[2]};
          if (a.nimg > 1)
            {
              const float4 T = a.off[en >> 24];
              e[0] += T.x; e[1] += T.y; e[2] += T.z;
            }
          const float4 *c = reinterpret_cast<const float4 *> (a.tabf)
                            + (size_t) min (bin, a.nbin - 1) * (NF * RT_DEG / 4);
          float f[NF], xj[12];
#pragma unroll
          for (int q = 0; q < NF; q++)
            {
              const float4 c1 = __ldg (c + 2 * q + 1), c0 = __ldg (c + 2 * q);
              f[q] = fmaf (fmaf (fmaf (fmaf (fmaf (c1.y, z, c1.x), z, c0.w), z, c0.z), z, c0.y), z, c0.x);
            }
          const float4 *xs = reinterpret_cast<const float4 *> (a.xf + (size_t) a.xf_ld * j);
#pragma unroll
          for (int q = 0; q < (C + 3) / 4; q++)
            {
              const float4 v = __ldg (xs + q);
              xj[4 * q] = v.x; xj[4 * q + 1] = v.y; xj[4 * q + 2] = v.z; xj[4 * q + 3] = v.w;
            }
          apply_radial<V, float> (e, e[0] * e[0] + e[1] * e[1] + e[2] * e[2], f, xj, yf);
        }
      __syncthreads ();
    }
  double v = warp_sums<P, double> (y, lane);
  // the far sum, back in its unit
  const float vf = warp_sums<P, float> (yf, lane);
  if (vf != 0.f) v += scalbn ((double) vf, *a.xtop);
  if (lane % (32 / P) == 0) s_y[warp][lane / (32 / P)] = v;
  __syncthreads ();
  if (t < C)
    {
      double r = s_y[0][t];
#pragma unroll
      for (int w = 1; w < RT_W; w++) r += s_y[w][t];
      a.out[(size_t) i * C + t] = r;
    }
}

// inverse of the Vandermonde matrix of the Chebyshev nodes, as hi + lo pairs
const Basis &
basis ()
{
  static const Basis b = [] {
    Basis r;
    long double x[RT_DEG];
    const long double pi = 3.14159265358979323846264338327950288L;
    for (int n = 0; n < RT_DEG; n++)
      {
        r.node[n] = (double) cosl (pi * (2 * n + 1) / (2 * RT_DEG));
        x[n] = r.node[n];                       // the nodes as they are used
      }
    for (int n = 0; n < RT_DEG; n++)
      {
        // Lagrange polynomial of node n: product of (x - x_m) / (x_n - x_m)
        long double c[RT_DEG] = {1.0L};
        int deg = 0;
        for (int m = 0; m < RT_DEG; m++)
          {
            if (m == n) continue;
            const long double w = 1.0L / (x[n] - x[m]);
            deg++;
            for (int k = deg; k >= 0; k--)
              c[k] = ((k ? c[k - 1] : 0.0L) - (k < deg ? c[k] * x[m] : 0.0L)) * w;
          }
        for (int k = 0; k < RT_DEG; k++)
          {
            r.hi[k][n] = (double) c[k];
            r.lo[k][n] = (double) (c[k] - (long double) r.hi[k][n]);
          }
      }
    return r;
  }();
  return b;
}

int
bin_of (double s)
{
  long long bits;
  static_assert (sizeof bits == sizeof s, "");
  __builtin_memcpy (&bits, &s, sizeof s);
  return (int) (bits >> (52 - RT_LOG));
}

}  // namespace

// the table covers r from 1 (half of contact) to a little past the cutoff
void
real_tab_range (double rc, int *bin0, int *nbin)
{
  *bin0 = bin_of (1.0);
  *nbin = std::max (1, bin_of (std::max (1.0, rc * rc * 1.0001)) - *bin0 + 1);
}

size_t
real_tab_bytes (int version, int nbin)
{
  const int nf = version == 0 ? 2 : (version == 1 ? 5 : 10);
  return (sizeof (double) + sizeof (float)) * (size_t) nbin * nf * RT_DEG;
}

size_t
real_tab_doubles (int version, int nbin)
{
  return real_tab_bytes (version, nbin) / (sizeof (double) + sizeof (float));
}

// FAR_U: 5.2 for F and FT; the stresslet functions are up to u^2 larger.  Never
// below the first bin of the table (s = 1, real_tab_range), which a split with
// xi > 5.2 reaches (a box of about one radius): the far loop takes the table
// for all of its pairs.  1e-4 above it, since the far pairs are told by FP32
// distances, within 1e-6 of the exact ones.
double
real_tab_far (int version, double xi)
{
  const double u = version == 2 ? 5.5 : 5.2;
  return std::max (1.0001, (u / xi) * (u / xi));
}

cudaError_t
launch_real_tab_build (int version, int bin0, int nbin, double xi, double *tab, float *tabf,
                       cudaStream_t st)
{
  const double xisp = xi / sqrt (M_PI);
  if (version == 0) k_rt_table<0><<<nbin, RT_DEG * 2, 0, st>>> (basis (), bin0, xi, xisp, tab, tabf);
  else if (version == 1) k_rt_table<1><<<nbin, RT_DEG * 5, 0, st>>> (basis (), bin0, xi, xisp, tab, tabf);
  else k_rt_table<2><<<nbin, RT_DEG * 10, 0, st>>> (basis (), bin0, xi, xisp, tab, tabf);
  return cudaGetLastError ();
}

cudaError_t
launch_real_tab (int version, const RealTabArgs &a, cudaStream_t st)
{
  if (version == 0) k_real_tab<0><<<a.np, RT_T, 0, st>>> (a);
  else if (version == 1) k_real_tab<1><<<a.np, RT_T, 0, st>>> (a);
  else k_real_tab<2><<<a.np, RT_T, 0, st>>> (a);
  return cudaGetLastError ();
}

}  // namespace lsg
