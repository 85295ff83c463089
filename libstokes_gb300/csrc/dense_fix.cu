// dense_fix.cu -- FP64 dense mobility matrix of equal spheres at a split of its
// own, the reciprocal part on the tensor cores.
//
// The c x c block of a pair is linear in moments sum_t scalar(t) e..e of its
// displacement r = r_j - r_i (dense_moments.cuh).  In reciprocal space 40 of
// them are independent for FTS (15 FT, 6 F): sum_k w(k) e_k..e_k cos or sin (k.r)
// with an e..e of 1 to 4 factors.  On an unsheared lattice w is even in every
// component of k, so of the eight products of cos and sin along x, y and z only
// one survives in each moment, the one whose sines are the axes with an odd
// number of factors, and one octant of k space is enough.  The pairs (i <= j
// alone: r -> -r flips the odd moments) are then evaluation points of a field
// with known coefficients: the back-projection GEMM of the FP64 product
// (k_fix_bwd: 55-bit fixed point, exact sums) with pairs for particles and, in
// four classes by the parity along y and z, moments for vector components.
//
//   k_fix_tables       functions of the particles (sincospi)
//   per chunk of pairs, so that its digit strings stay in L2:
//   k_fix_pair_tables  functions of r_j - r_i, by the addition theorem
//   k_fix_strings, k_fix_bwd
//   k_dense_tile       real-space moments of 8 x 8 pairs from the radial tables
//                      of the FP64 product (radial.cuh), the self part, and
//                      all moments -> blocks (i, j) and (j, i)
//
// Before, a warp per ordered pair summed every reciprocal vector and image of
// libstokes' own split in FP64 arithmetic, which runs at 1/64 of the FP32 rate.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "dense_moments.cuh"
#include "ewald_device.cuh"
#include "fixk.h"
#include "gpu_engine.h"
#include "radial.cuh"
#include "real_tab.h"
#include "stokes_gpu.h"

extern "C" void lsg_set_split (struct stokes *sys, double xi, double ewald_eps);

namespace lsg {

namespace {

constexpr int PT = 64;                  // pairs of a tile, 8 x 8
// tiles of a chunk, two CTAs of the last kernel per SM: its strings (about 4 KB
// a pair) stay in L2.  FTS N = 256, us: 811 at 152, 652 at 304, 632 at 608 with
// twice the scratch.
constexpr int CHUNK_TILES = 304;
constexpr int MAX_DER = 12, MAX_TERM = 8;

// a sum of at most N moments: index (-1: end) and factor
template <int N> struct Terms {
  int idx[N];
  double f[N];
};

// one reciprocal moment: scalar (0 A, 1 C, 2 M, 3 B, 4 G) times
// e_x^n[0] e_y^n[1] e_z^n[2]
struct Moment {
  int kind, n[3];
};

struct WeightArgs {
  double k0[3];
  double xi2, kmax, pivol;              // the split
  double xi2_ref, kmax_ref, pivol_ref;  // libstokes' own, for its G term
  int ref[3], fts;
  const Moment *mom;                    // [4][16]
  const int2 *blk;                      // lowest (|m2|, |m3|) of the blocks, by class
  int blk0[4];
};

// G[column][row]: the weight of one octant point in one moment, by class; and
// the largest magnitude of each column's (|m1|, moment)
__global__ void __launch_bounds__ (128)
k_dense_weights (const __grid_constant__ FixPlan p, const __grid_constant__ WeightArgs a)
{
  const int n = blockIdx.y, r = blockIdx.x * 128 + threadIdx.x;
  int cl = 0;
  while (cl < 3 && n >= p.cls[cl + 1].col0) cl++;
  const FixClass &c = p.cls[cl];
  const int nl = n - c.col0;
  double g = 0.0;
  int m1 = 0, q = 0;
  if (nl < c.ncol && r < 4 * c.nblk)
    {
      m1 = nl / c.nc;
      q = nl % c.nc;
      const int2 b = a.blk[a.blk0[cl] + r / 4];
      const int m2 = b.x + (r >> 1 & 1), m3 = b.y + (r & 1);
      const Moment mo = a.mom[16 * cl + q];
      const double k1 = a.k0[0] * m1, k2 = a.k0[1] * m2, k3 = a.k0[2] * m3;
      const double kk = k1 * k1 + k2 * k2 + k3 * k3, k = sqrt (kk);
      double ya = 0.0, yb = 0.0, yc = 0.0, yg = 0.0, ym = 0.0;
      // points with a sine of index 0 have no function
      const bool have = kk != 0.0 && m2 <= p.M[1] && m3 <= p.M[2] && (m1 || !(mo.n[0] & 1));
      if (have && k <= a.kmax)
        {
          const double k4z = kk / 4.0 / a.xi2;
          const double kexp = a.pivol * (1.0 + k4z * (1.0 + 2.0 * k4z)) / kk * exp (-k4z);
          ya = 6.0 * (1.0 - kk / 3.0) * kexp;
          yb = 3.0 * k * kexp;
          yc = 1.5 * kk * kexp;
          yg = -3.0 * (1.0 - 4.0 / 15.0 * kk) * k * kexp;
          ym = 3.0 * (1.0 - kk / 5.0) * kk * kexp;
        }
      if (have && a.fts && m1 <= a.ref[0] && m2 <= a.ref[1] && m3 <= a.ref[2]
          && (a.kmax_ref == 0.0 || k <= a.kmax_ref))
        {
          const double k4z = kk / 4.0 / a.xi2_ref;
          const double kexp = a.pivol_ref * (1.0 + k4z * (1.0 + 2.0 * k4z)) / kk * exp (-k4z);
          yg += 6.0 * (1.0 - 4.0 / 15.0 * kk) * k * kexp;
        }
      if (have)
        {
          const double ki = 1.0 / k, e[3] = {k1 * ki, k2 * ki, k3 * ki};
          const int odd = (mo.n[0] & 1) + (mo.n[1] & 1) + (mo.n[2] & 1);
          // cos (a + b + c) holds -sin sin cos, sin (-(a + b + c)) -sin cos cos and
          // +sin sin sin; the octant point stands for its sign patterns
          g = (m1 ? 2.0 : 1.0) * (m2 ? 2.0 : 1.0) * (m3 ? 2.0 : 1.0) * (odd == 1 || odd == 2 ? -1.0 : 1.0);
          g *= mo.kind == 0 ? ya : (mo.kind == 1 ? yc : (mo.kind == 2 ? ym : (mo.kind == 3 ? yb : yg)));
          for (int d = 0; d < 3; d++)
            for (int u = 0; u < mo.n[d]; u++) g *= e[d];
        }
    }
  if (r < p.Rp) ((double *) p.G)[(size_t) n * p.Rp + r] = g;
  const unsigned mx = __reduce_max_sync (0xffffffffu, (unsigned) __double2hiint (g) & 0x7fffffffu);
  if (mx && (threadIdx.x & 31) == 0 && nl < c.ncol)
    atomicMax (p.mx + cl * fix_mx_words (p) + 16 * (nl / c.nc + 1) + nl % c.nc, mx);
}

// independent real-space moments, in the plain displacement d: A0 | A2[6] |
// B1[3] | C0 | C2[6] | G2[3] | G3[10] | M4[15] | M4b[6] | zm; the others follow
// from tracelessness and yh = yc - xc (derived_real)
enum {
  R_A0 = 0, R_A2 = 1, R_B1 = 7, R_C0 = 10, R_C2 = 11, R_G2 = 17, R_G3 = 20, R_M4 = 30, R_M4B = 45,
  R_ZM = 51
};
template <int V> struct NReal;
template <> struct NReal<0> { static constexpr int value = 7; };
template <> struct NReal<1> { static constexpr int value = 17; };
template <> struct NReal<2> { static constexpr int value = 52; };



struct DenseArgs {
  const double *pos;
  const uint4 *q;                       // fractional coordinates of the particles (FixPlan)
  const unsigned long long *u;
  const int2 *tile;
  int ntile, np, ldT;
  float sf[3], rc2;                     // box / 2^32; FP32 test, a little wide
  double s60[3];                        // box / 2^60
  double xi, xisp;
  const float4 *off;                    // lattice offsets of the minimum image; indexes
  const int4 *cell;
  int noff;
  const double *tab;                    // radial functions
  int bin0, nbin;
  double self[3], same[3];              // of i = j; of distinct particles at one place
  const double *yp;
  FixClass cls[4];
  const int2 *rec;                      // class and component of a reciprocal moment
  int nrec;
  const Terms<MAX_DER> *der;            // [moment]: from the independent ones
  const Terms<MAX_TERM> *entry;         // [c c]
  double *mat;
};

constexpr int DT = 256;                 // threads: four groups of moments x 64 pairs
constexpr int WIN = 256;                // (pair, image) entries worked on at a time

// moments of group g of one pair: entries e0 .. e1 - 1 of the window, f[k][e] =
// (d, functions)
template <int V, int G>
struct RealGroup {
  static constexpr int N = G == 0 ? (V == 0 ? 7 : (V == 1 ? 14 : 15)) : G == 1 ? (V == 0 ? 0 : (V == 1 ? 3 : 16))
                           : V < 2 ? 0 : (G == 2 ? 8 : 13);
  static __device__ __forceinline__ void add (const double (*f)[WIN], int e, double (&m)[16])
  {
    const double x = f[0][e], y = f[1][e], z = f[2][e];
    if constexpr (G == 0)
      {
        const double dd[6] = {x * x, x * y, x * z, y * y, y * z, z * z};
        m[0] += f[3][e];
        const double a2 = f[4][e];
#pragma unroll
        for (int k = 0; k < 6; k++) m[1 + k] = fma (a2, dd[k], m[1 + k]);
        if constexpr (V >= 1)
          {
            m[7] += f[6][e];
            const double c2 = f[7][e];
#pragma unroll
            for (int k = 0; k < 6; k++) m[8 + k] = fma (c2, dd[k], m[8 + k]);
          }
        if constexpr (V == 2) m[14] += f[12][e];
      }
    if constexpr (G == 1 && V >= 1)
      {
        const double b = f[5][e];
        m[0] = fma (b, x, m[0]); m[1] = fma (b, y, m[1]); m[2] = fma (b, z, m[2]);
        if constexpr (V == 2)
          {
            const double g2 = f[8][e], g3 = f[9][e];
            m[3] = fma (g2, x, m[3]); m[4] = fma (g2, y, m[4]); m[5] = fma (g2, z, m[5]);
            const double gx = g3 * x, gy = g3 * y, gz = g3 * z, xx = gx * x, xy = gx * y, xz = gx * z,
                         yy = gy * y, yz = gy * z, zz = gz * z;
            m[6] = fma (xx, x, m[6]); m[7] = fma (xx, y, m[7]); m[8] = fma (xx, z, m[8]);
            m[9] = fma (xy, y, m[9]); m[10] = fma (xy, z, m[10]); m[11] = fma (xz, z, m[11]);
            m[12] = fma (yy, y, m[12]); m[13] = fma (yy, z, m[13]); m[14] = fma (yz, z, m[14]);
            m[15] = fma (zz, z, m[15]);
          }
      }
    if constexpr (G >= 2 && V == 2)
      {
        const double m1 = f[10][e];
        const double xx = x * x, xy = x * y, xz = x * z, yy = y * y, yz = y * z, zz = z * z;
        if constexpr (G == 2)
          {
            const double a = m1 * xx, b = m1 * xy;
            m[0] = fma (a, xx, m[0]); m[1] = fma (a, xy, m[1]); m[2] = fma (a, xz, m[2]);
            m[3] = fma (a, yy, m[3]); m[4] = fma (a, yz, m[4]); m[5] = fma (a, zz, m[5]);
            m[6] = fma (b, yy, m[6]); m[7] = fma (b, yz, m[7]);
          }
        else
          {
            const double a = m1 * xz, b = m1 * yy, c = m1 * zz;
            m[0] = fma (a, yz, m[0]); m[1] = fma (a, zz, m[1]);
            m[2] = fma (b, yy, m[2]); m[3] = fma (b, yz, m[3]); m[4] = fma (b, zz, m[4]);
            m[5] = fma (c, yz, m[5]); m[6] = fma (c, zz, m[6]);
            const double h = 0.5 * f[11][e];            // m4 = (ym - zm) / 2
            m[7] = fma (h, xx, m[7]); m[8] = fma (h, xy, m[8]); m[9] = fma (h, xz, m[9]);
            m[10] = fma (h, yy, m[10]); m[11] = fma (h, yz, m[11]); m[12] = fma (h, zz, m[12]);
          }
      }
  }
  // place of moment k among the real ones
  static __device__ __forceinline__ int slot (int k)
  {
    if (G == 0) return k < 7 ? R_A0 + k : (k < 14 ? R_C0 + k - 7 : R_ZM);
    if (G == 1) return k < 3 ? R_B1 + k : R_G2 + k - 3;
    return G == 2 ? R_M4 + k : R_M4 + 8 + k;
  }
};

// An 8 x 8 tile of pairs.
//
// Real space: the images of each pair's minimum-image displacement within the
// cutoff (FP32 test) are listed pair by pair; the threads evaluate the radial
// functions of WIN entries at a time, one each, then each thread adds the
// moments of its group over the entries of its pair.  Evaluated by one thread
// a pair from the closed forms this took four times the GEMM (a warp works as
// long as its pair with most images, at about 2000 FP64 instructions each).
//
// Blocks: (i, j) and its mirror image; the odd entries (velocity against torque
// or stresslet) change sign with r.
template <int V>
__global__ void __launch_bounds__ (DT, 2)
k_dense_tile (const __grid_constant__ DenseArgs a)
{
  constexpr int C = NComp<V>::value, NM = Moments<V>::N, NR = NReal<V>::value, NF = NFun<V>::value;
  extern __shared__ double sm[];
  __shared__ int s_start[PT + 1], s_warp[2];
  __shared__ unsigned short s_list[WIN];                // pair | image << 6
  double *X = sm, *mo = X + (NR + a.nrec) * PT, *out = mo + NM * PT;    // [..][PT], out [C][PT]
  double (*f)[WIN] = reinterpret_cast<double (*)[WIN]> (mo);            // (before mo is made)
  const int2 ij = a.tile[blockIdx.x];
  const int t = threadIdx.x, pr = t & (PT - 1), g = t >> 6;
  const int i = 8 * ij.x + (pr >> 3), j = 8 * ij.y + (pr & 7);
  const bool live = i < a.np && j < a.np && i <= j;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  auto scan = [&] (auto &&hit) {
    if (!live) return;
    for (int m = 0; m < a.noff; m++)
      {
        const float4 o = a.off[m];
        const float dx = fx + o.x, dy = fy + o.y, dz = fz + o.z;
        if (dx * dx + dy * dy + dz * dz < a.rc2) hit (m);
      }
  };
  if (t < PT)
    {
      if (live)
        {
          const uint4 qi = a.q[i], qj = a.q[j];
          fx = (float) (int) (qj.x - qi.x) * a.sf[0];
          fy = (float) (int) (qj.y - qi.y) * a.sf[1];
          fz = (float) (int) (qj.z - qi.z) * a.sf[2];
        }
      int n = 0;
      scan ([&] (int) { n++; });
      int pre = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
        {
          const int v = __shfl_up_sync (0xffffffffu, pre, o);
          if ((t & 31) >= o) pre += v;
        }
      s_start[t + 1] = pre;
      if ((t & 31) == 31) s_warp[t >> 5] = pre;
    }
  __syncthreads ();
  if (t >= 32 && t < PT) s_start[t + 1] += s_warp[0];
  if (t == 0) s_start[0] = 0;
  __syncthreads ();
  const int total = s_start[PT];
  double m[16];                         // of this thread's group
#pragma unroll
  for (int k = 0; k < 16; k++) m[k] = 0.0;
  for (int w0 = 0; w0 < total; w0 += WIN)
    {
      if (t < PT)
        {
          int k = s_start[t] - w0;
          scan ([&] (int m) {
            if (k >= 0 && k < WIN) s_list[k] = (unsigned short) (t | m << 6);
            k++;
          });
        }
      __syncthreads ();
      if (t < min (WIN, total - w0))
        {
          const int en = s_list[t], ep = en & (PT - 1);
          const int ei = 8 * ij.x + (ep >> 3), ej = 8 * ij.y + (ep & 7);
          const int4 o = a.cell[en >> 6];
          const unsigned long long *ui = a.u + 4 * (size_t) ei, *uj = a.u + 4 * (size_t) ej;
          double d[3], c[NF];
          d[0] = int_to_double (image_diff (ui[0], uj[0]) + ((long long) o.x << 60)) * a.s60[0];
          d[1] = int_to_double (image_diff (ui[1], uj[1]) + ((long long) o.y << 60)) * a.s60[1];
          d[2] = int_to_double (image_diff (ui[2], uj[2]) + ((long long) o.z << 60)) * a.s60[2];
          const double s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
          const int bin = radial_bin (s, a.bin0);
          if (s == 0.0)
            {
              const double *z = ei == ej ? a.self : a.same;
#pragma unroll
              for (int q = 0; q < NF; q++) c[q] = q == 0 ? z[0] : (q == 3 ? z[1] : (q == 9 ? z[2] : 0.0));
            }
          else if (bin < 0)
            radial<V> (a.xi, a.xisp, sqrt (s), s, c);
          else
            table_radial<NF> (a.tab, s, bin, a.bin0, a.nbin, c);
#pragma unroll
          for (int q = 0; q < 3; q++) f[q][t] = d[q];
#pragma unroll
          for (int q = 0; q < NF; q++) f[3 + q][t] = c[q];
        }
      __syncthreads ();
      const int e0 = max (s_start[pr] - w0, 0), e1 = min (s_start[pr + 1] - w0, WIN);
      for (int e = e0; e < e1; e++)
        {
          if (g == 0) RealGroup<V, 0>::add (f, e, m);
          else if (g == 1) RealGroup<V, 1>::add (f, e, m);
          else if (g == 2) RealGroup<V, 2>::add (f, e, m);
          else RealGroup<V, 3>::add (f, e, m);
        }
      __syncthreads ();
    }
  // a position that is not finite makes every moment of its pairs NaN
  double bad = 0.0;
  if (live)
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (!(fabs (a.pos[3 * i + k]) < 1e300 && fabs (a.pos[3 * j + k]) < 1e300))
        bad = __longlong_as_double (0x7ff8000000000000ll);
  auto put = [&] (auto r) {
    using T = decltype (r);
#pragma unroll
    for (int k = 0; k < T::N; k++) X[T::slot (k) * PT + pr] = m[k] + bad;
  };
  if (g == 0) put (RealGroup<V, 0> ());
  else if (g == 1) put (RealGroup<V, 1> ());
  else if (g == 2) put (RealGroup<V, 2> ());
  else put (RealGroup<V, 3> ());
  const size_t base = (size_t) blockIdx.x * PT;
  for (int e = t; e < a.nrec * PT; e += DT)
    {
      const int2 w = a.rec[e / PT];
      const double *y = a.yp + ((size_t) a.cls[w.x].slot0 * 16 + w.y) * a.ldT + base + e % PT;
      double v = 0.0;
      for (int k = 0; k < a.cls[w.x].nslot; k++) v += y[(size_t) k * 16 * a.ldT];
      X[NR * PT + e] = v;
    }
  __syncthreads ();
  for (int e = t; e < NM * PT; e += DT)
    {
      const int q = e % PT;
      const Terms<MAX_DER> &w = a.der[e / PT];
      double v = 0.0;
      for (int k = 0; k < MAX_DER && w.idx[k] >= 0; k++) v = fma (w.f[k], X[w.idx[k] * PT + q], v);
      mo[e] = v;
    }
  const size_t n = (size_t) C * a.np;
  for (int row = 0; row < C; row++)
    {
      __syncthreads ();
      for (int e = t; e < C * PT; e += DT)
        {
          const int q = e % PT;
          const Terms<MAX_TERM> &w = a.entry[row * C + e / PT];
          double v = 0.0;
          for (int k = 0; k < MAX_TERM && w.idx[k] >= 0; k++) v = fma (w.f[k], mo[w.idx[k] * PT + q], v);
          out[e] = v;
        }
      __syncthreads ();
      // consecutive threads write consecutive columns of the matrix
      for (int e = t; e < 2 * C * PT; e += DT)
        {
          const bool mirror = e >= C * PT;
          const int k = mirror ? e - C * PT : e;
          const int x = k / (8 * C), y = k / C % 8, col = k % C;     // row and column particle
          const int p = 8 * (mirror ? ij.y : ij.x) + x, r = 8 * (mirror ? ij.x : ij.y) + y;
          if (p >= a.np || r >= a.np) continue;
          // each block once: those of i <= j directly
          if (mirror ? p <= r : p > r) continue;
          const double v = out[col * PT + (mirror ? 8 * y + x : 8 * x + y)];
          a.mat[(size_t) (C * p + row) * n + (size_t) C * r + col]
            = mirror && (row < 3) != (col < 3) ? -v : v;
        }
    }
}

// moments of the version by class, those with a cosine along x first
std::vector<Moment>
moment_list (int version)
{
  std::vector<Moment> v;
  auto all = [&] (int kind, int order) {
    for (int x = order; x >= 0; x--)
      for (int y = order - x; y >= 0; y--) v.push_back ({kind, {x, y, order - x - y}});
  };
  all (0, 2);
  if (version >= 1)
    {
      all (1, 2);
      all (3, 1);
    }
  if (version == 2)
    {
      all (2, 4);
      all (4, 3);
    }
  return v;
}

// the reciprocal part of every moment of a pair for reciprocal moment m alone
template <int V>
void
derived (const Moment &m, double *mo)
{
  for (int q = 0; q < Moments<V>::N; q++) mo[q] = 0.0;
  int ax[4], na = 0;
  for (int d = 0; d < 3; d++)
    for (int u = 0; u < m.n[d]; u++) ax[na++] = d;
  const bool pair2 = na == 2 && ax[0] == ax[1];
  if (m.kind == 0)
    {
      mo[MO_A2 + sym2 (ax[0], ax[1])] -= 1.0;           // a2 = -ya
      if (pair2) mo[MO_A0] += 1.0;                      // ya e.e
    }
  if constexpr (V >= 1)
    {
      if (m.kind == 1)
        {
          mo[MO_C2 + sym2 (ax[0], ax[1])] -= 1.0;
          if (pair2) mo[MO_C0] += 1.0;
          if constexpr (V == 2) mo[MO_H2 + sym2 (ax[0], ax[1])] += 1.0;   // yh = yc
        }
      if (m.kind == 3) mo[MO_B1 + ax[0]] += 1.0;
    }
  if constexpr (V == 2)
    {
      // a trace over two factors is one over e.e = 1
      if (m.kind == 4)
        {
          mo[MO_G3 + sym3 (ax[0], ax[1], ax[2])] -= 2.0;                  // g3 = -2 yg
          for (int c = 0; c < 3; c++)
            if (m.n[c] >= 2)
              for (int b = 0; b < 3; b++)
                if (m.n[b] - (b == c ? 2 : 0) == 1) mo[MO_G2 + b] += 1.0; // g2 = yg
        }
      if (m.kind == 2)
        {
          mo[MO_M4 + sym4 (ax[0], ax[1], ax[2], ax[3])] -= 2.0;           // m1 = -2 ym
          for (int c = 0; c < 3; c++)
            {
              if (m.n[c] < 2) continue;
              int rest[3] = {m.n[0], m.n[1], m.n[2]}, b[2], nb = 0;
              rest[c] -= 2;
              for (int d = 0; d < 3; d++)
                for (int u = 0; u < rest[d]; u++) b[nb++] = d;
              mo[MO_M4B + sym2 (b[0], b[1])] += 0.5;                      // m4 = ym / 2
            }
        }
    }
}

// the moments of a pair for real-space moment r alone
template <int V>
void
derived_real (int r, double *mo)
{
  for (int q = 0; q < Moments<V>::N; q++) mo[q] = 0.0;
  if (r < R_B1) mo[r == R_A0 ? (int) MO_A0 : MO_A2 + r - R_A2] = 1.0;
  if constexpr (V >= 1)
    {
      if (r >= R_B1 && r < R_C0) mo[MO_B1 + r - R_B1] = 1.0;
      if (r == R_C0) mo[MO_C0] = 1.0;
      if (r >= R_C2 && r < R_G2)
        {
          mo[MO_C2 + r - R_C2] = 1.0;
          if constexpr (V == 2) mo[MO_H2 + r - R_C2] = -1.0;            // yh = yc - xc
        }
    }
  if constexpr (V == 2)
    {
      if (r >= R_G2 && r < R_G3) mo[MO_G2 + r - R_G2] = 1.0;
      if (r >= R_G3 && r < R_M4) mo[MO_G3 + r - R_G3] = 1.0;
      if (r >= R_M4 && r < R_M4B) mo[MO_M4 + r - R_M4] = 1.0;
      if (r >= R_M4B && r < R_ZM) mo[MO_M4B + r - R_M4B] = 1.0;
      if (r == R_ZM) mo[MO_M5] = 0.5;
      // g1 = -(g3 + 2 g2) / 3, m2 = -(m1 + 4 m4) / 3, m3 = -(m2 + 2 m5) / 3
      double tr2 = 0.0;
      for (int b = 0; b < 3; b++)
        {
          double t3 = 0.0;
          for (int c = 0; c < 3; c++) t3 += mo[MO_G3 + sym3 (b, c, c)];
          mo[MO_G1 + b] = -(t3 + 2.0 * mo[MO_G2 + b]) / 3.0;
          for (int d = b; d < 3; d++)
            {
              double t4 = 0.0;
              for (int c = 0; c < 3; c++) t4 += mo[MO_M4 + sym4 (b, d, c, c)];
              mo[MO_M2 + sym2 (b, d)] = -(t4 + 4.0 * mo[MO_M4B + sym2 (b, d)]) / 3.0;
            }
          tr2 += mo[MO_M2 + sym2 (b, b)];
        }
      mo[MO_M3] = -(tr2 + 2.0 * mo[MO_M5]) / 3.0;
    }
}

template <int V>
bool
make_terms (const std::vector<Moment> &rec, std::vector<Terms<MAX_DER>> &der,
            std::vector<Terms<MAX_TERM>> &entry)
{
  constexpr int NM = Moments<V>::N, C = NComp<V>::value;
  double mo[NM];
  der.assign (NM, Terms<MAX_DER> {});
  entry.assign (C * C, Terms<MAX_TERM> {});
  for (auto &t : der) t.idx[0] = -1;
  for (auto &t : entry) t.idx[0] = -1;
  bool ok = true;
  auto add = [&] (auto &t, int cap, int idx, double f) {
    int k = 0;
    while (k < cap && t.idx[k] >= 0) k++;
    if (k == cap) { ok = false; return; }
    t.idx[k] = idx;
    t.f[k] = f;
    if (k + 1 < cap) t.idx[k + 1] = -1;
  };
  constexpr int NR = NReal<V>::value;
  for (int r = 0; r < NR + (int) rec.size (); r++)
    {
      if (r < NR) derived_real<V> (r, mo);
      else derived<V> (rec[r - NR], mo);
      for (int q = 0; q < NM; q++)
        if (mo[q] != 0.0) add (der[q], MAX_DER, r, mo[q]);
    }
  for (int q = 0; q < NM; q++)
    {
      for (int k = 0; k < NM; k++) mo[k] = k == q ? 1.0 : 0.0;
      for (int e = 0; e < C * C; e++)
        {
          const double f = block_entry<V, double> (mo, e / C, e % C, false);
          if (f != 0.0) add (entry[e], MAX_TERM, q, f);
        }
    }
  return ok;
}

}  // namespace

struct DenseState {
  double key[16] = {0};
  struct stokes *ts = nullptr;
  FixPlan base, p;              // of the particles; of a chunk of pairs
  FixMaps maps;
  DenseArgs a;
  int tiles = 0, chunk = 0;     // tiles in all; of a chunk
  DevBuf arena;
  int *h_status = nullptr, *d_status = nullptr;
};

// Split of the builder: eta = xi V^(1/3).  The GEMM's work grows as eta^3, the
// images of a pair fall with it.  Measured, us at eta 5, 6, 7: FTS N = 256 656,
// 652, 752, N = 600 3315, 3394, 3876; F N = 256 261, 285, 300, but F N = 64
// (one CTA's latency) 81, 77, 63 and 65 at 8.
static double
dense_fix_eta (const struct stokes *sys)
{
  static const double env = [] {
    const char *s = getenv ("LIBSTOKES_GB300_DENSE64_ETA");
    return s ? atof (s) : -1.0;
  }();
  const double l = cbrt (sys->lx * sys->ly * sys->lz);
  const double eta = sys->version < 2 && sys->np <= 128 ? 8.0 : 6.0;
  // xi a <= 0.7, as in the product
  return std::min (env >= 0.0 ? env : eta, 0.7 * l);
}

bool
dense_fix_applies (const Ctx *c, const struct stokes *sys)
{
  const double l = cbrt (sys->lx * sys->ly * sys->lz), eta = dense_fix_eta (sys);
  const double widest = std::max (sys->lx, std::max (sys->ly, sys->lz));
  // small systems, and boxes whose eta is held down, are latency-bound in both
  // builders: k_matrix 67 us at F N = 24 (72 here), 84 at FT N = 24 (89), 163 at
  // FTS N = 16 (128)
  return sys->rmin == 0.0 && sys->a == nullptr && sys->np >= (sys->version < 2 ? 32 : 12)
         && sys->np <= 1 << 20 && eta >= 5.0 && eta > sys->xi * l
         // no more lattice offsets than an entry's 10 bits
         && widest < 3.0 * std::min (sys->lx, std::min (sys->ly, sys->lz));
}

static int
dense_setup (Ctx *c, const struct stokes *sys)
{
  if (!c->dfix) c->dfix = new DenseState ();
  DenseState *f = c->dfix;
  const bool fts = sys->version == 2;
  const double eta = dense_fix_eta (sys), l = cbrt (sys->lx * sys->ly * sys->lz);
  const double key[16] = {sys->lx, sys->ly, sys->lz, (double) sys->np, (double) sys->version, eta,
                          sys->ewald_eps, sys->xi, fts ? sys->kmax : 0.0,
                          fts ? (double) sys->kmaxx : 0.0, fts ? (double) sys->kmaxy : 0.0,
                          fts ? (double) sys->kmaxz : 0.0, 1.0};
  if (memcmp (key, f->key, sizeof key) == 0) return STOKES_GPU_OK;
  f->key[12] = 0.0;
  if (f->ts) stokes_free (f->ts);
  struct stokes *ts = f->ts = stokes_init ();
  if (!ts) return set_error (STOKES_GPU_ENOMEM, "dense split");
  ts->version = sys->version;
  ts->periodic = 1;
  stokes_set_np (ts, sys->np, sys->nm);
  stokes_set_l (ts, sys->lx, sys->ly, sys->lz);
  // FTS: tighter, as for the product
  const double eps = sys->ewald_eps > 0.0 ? sys->ewald_eps : 1e-12;
  lsg_set_split (ts, eta / l, fts ? 0.3 * eps : eps);

  FixPlan p;
  double k0[3];
  const int ref[3] = {sys->kmaxx, sys->kmaxy, sys->kmaxz};
  p.l[0] = sys->lx; p.l[1] = sys->ly; p.l[2] = sys->lz;
  for (int d = 0; d < 3; d++)
    {
      p.il[d] = 1.0 / p.l[d];
      k0[d] = 2.0 * M_PI / p.l[d];
      p.M[d] = (int) (ts->kmax / k0[d]);
      if (fts) p.M[d] = std::max (p.M[d], ref[d]);
    }
  p.nmi = 2 * p.M[0] + 1;
  p.oy = p.nmi;
  p.oz = p.oy + 2 * p.M[1] + 1;
  p.zero = p.oz + 2 * p.M[2] + 1;
  p.nT = p.zero + 1;
  // moments by class (parities along y and z), cosine along x first
  std::vector<Moment> rec = moment_list (sys->version);
  std::vector<Moment> mom (64, Moment {0, {0, 0, 0}});
  std::vector<int2> where (rec.size ());
  for (int cl = 0; cl < 4; cl++)
    {
      FixClass &w = p.cls[cl];
      w = FixClass {};
      for (int px = 0; px < 2; px++)
        for (size_t r = 0; r < rec.size (); r++)
          if ((rec[r].n[1] & 1) == cl >> 1 && (rec[r].n[2] & 1) == (cl & 1) && (rec[r].n[0] & 1) == px)
            {
              w.odd |= px << w.nc;
              where[r] = make_int2 (cl, w.nc);
              mom[16 * cl + w.nc++] = rec[r];
            }
    }
  // blocks of 2 x 2 (|m2|, |m3|) by class, by length
  auto in_set = [&] (int a, int b, int d) {
    if (b > p.M[1] || d > p.M[2]) return false;
    const double k1 = k0[0] * a, k2 = k0[1] * b, k3 = k0[2] * d;
    const double k = sqrt (k1 * k1 + k2 * k2 + k3 * k3);
    return k <= ts->kmax
           || (fts && a <= ref[0] && b <= ref[1] && d <= ref[2] && (sys->kmax == 0.0 || k <= sys->kmax));
  };
  std::vector<int2> blk;
  std::vector<int4> quart;
  std::vector<int> nqm;
  int blk0[4];
  for (int cl = 0; cl < 4; cl++)
    {
      const int p2 = cl >> 1, p3 = cl & 1;
      std::vector<std::pair<double, int2>> order;
      for (int b = p2; b <= p.M[1]; b += 2)
        for (int d = p3; d <= p.M[2]; d += 2)
          {
            bool any = false;
            for (int u = 0; u < 4; u++) any = any || in_set (0, b + (u >> 1), d + (u & 1));
            if (any)
              order.push_back ({b * b * k0[1] * k0[1] + d * d * k0[2] * k0[2], make_int2 (b, d)});
          }
      std::stable_sort (order.begin (), order.end (),
                        [] (const auto &a, const auto &b) { return a.first < b.first; });
      FixClass &w = p.cls[cl];
      w.nblk = (int) order.size ();
      w.nq0 = (int) nqm.size ();
      blk0[cl] = (int) blk.size ();
      auto row = [&] (int o, int M, int m, int sine) {
        return m > M || (sine && m == 0) ? p.zero : o + (sine ? 2 * m : (m ? 2 * m - 1 : 0));
      };
      for (const auto &o : order)
        {
          const int b = o.second.x, d = o.second.y;
          blk.push_back (o.second);
          quart.push_back (make_int4 (row (p.oy, p.M[1], b, p2), row (p.oy, p.M[1], b + 1, p2),
                                      row (p.oz, p.M[2], d, p3), row (p.oz, p.M[2], d + 1, p3)));
        }
      while (quart.size () % 8) quart.push_back (make_int4 (p.zero, p.zero, p.zero, p.zero));
      for (int a = 0; a <= p.M[0]; a++)
        {
          int n = 0;
          for (int k = w.nblk; k > 0 && n == 0; k--)
            for (int u = 0; u < 4; u++)
              if (in_set (a, order[k - 1].second.x + (u >> 1), order[k - 1].second.y + (u & 1))) n = k;
          nqm.push_back (n);
        }
      for (int a = p.M[0] - 1; a >= 0; a--)
        nqm[w.nq0 + a] = std::max (nqm[w.nq0 + a], nqm[w.nq0 + a + 1]);
    }
  // 8 x 8 tiles of pairs, on and above the diagonal
  const int nt = (sys->np + 7) / 8;
  std::vector<int2> tile;
  for (int a = 0; a < nt; a++)
    for (int b = a; b < nt; b++) tile.push_back (make_int2 (a, b));
  f->tiles = (int) tile.size ();
  const int nchunk = (f->tiles + CHUNK_TILES - 1) / CHUNK_TILES;
  f->chunk = ((f->tiles + nchunk - 1) / nchunk + 1) / 2 * 2;
  p.np = f->chunk * PT;
  p.ldT = f->chunk * PT;
  std::vector<int4> item;
  fix_plan_dense (p, nqm, item);
  FixPlan b = p;
  b.np = sys->np;
  b.c = 0;
  b.ldT = (sys->np + 127) / 128 * 128;

  std::vector<Terms<MAX_DER>> der;
  std::vector<Terms<MAX_TERM>> entry;
  const bool fit = sys->version == 0 ? make_terms<0> (rec, der, entry)
                   : sys->version == 1 ? make_terms<1> (rec, der, entry)
                                       : make_terms<2> (rec, der, entry);
  if (!fit) return set_error (STOKES_GPU_EINVAL, "dense builder: terms of an entry");
  // lattice offsets whose cell of minimum-image displacements comes within
  // the cutoff
  DenseArgs a {};
  std::vector<float4> off;
  std::vector<int4> cell;
  const double rc = sqrt (ts->rmax2);
  int no[3];
  for (int d = 0; d < 3; d++) no[d] = std::min (7, (int) ceil (rc / p.l[d] + 0.5));
  for (int a1 = -no[0]; a1 <= no[0]; a1++)
    for (int a2 = -no[1]; a2 <= no[1]; a2++)
      for (int a3 = -no[2]; a3 <= no[2]; a3++)
        {
          const int m[3] = {a1, a2, a3};
          double dd = 0.0;
          for (int d = 0; d < 3; d++)
            {
              const double gap = std::max (0.0, (fabs ((double) m[d]) - 0.5) * p.l[d]);
              dd += gap * gap;
            }
          if (dd > rc * rc * 1.0001) continue;
          off.push_back (make_float4 ((float) (a1 * p.l[0]), (float) (a2 * p.l[1]),
                                      (float) (a3 * p.l[2]), 0.f));
          cell.push_back (make_int4 (a1, a2, a3, 0));
        }
  // one allocation: host tables (one copy), what is zero where nothing writes
  // it, the rest
  std::vector<char> host;
  size_t bytes = 0;
  auto place = [&] (size_t n) {
    const size_t at = bytes;
    bytes += (std::max<size_t> (n, 16) + 255) / 256 * 256;
    return at;
  };
  auto table = [&] (const void *src, size_t n) {
    const size_t at = place (n);
    host.resize (bytes);
    if (n) memcpy (host.data () + at, src, n);
    return at;
  };
  const size_t o_quart = table (quart.data (), sizeof (int4) * quart.size ());
  const size_t o_nqm = table (nqm.data (), sizeof (int) * nqm.size ());
  const size_t o_blk = table (blk.data (), sizeof (int2) * blk.size ());
  const size_t o_mom = table (mom.data (), sizeof (Moment) * mom.size ());
  const size_t o_item = table (item.data (), sizeof (int4) * item.size ());
  const size_t o_tile = table (tile.data (), sizeof (int2) * tile.size ());
  const size_t o_rec = table (where.data (), sizeof (int2) * where.size ());
  const size_t o_der = table (der.data (), sizeof (der[0]) * der.size ());
  const size_t o_entry = table (entry.data (), sizeof (entry[0]) * entry.size ());
  const size_t o_off = table (off.data (), sizeof (float4) * off.size ());
  const size_t o_cell = table (cell.data (), sizeof (int4) * cell.size ());
  const size_t zero0 = bytes;
  const size_t o_mx = place (4 * fix_mx_words (p) * sizeof (unsigned));
  const size_t o_Tb = place (fix_bytes_T (7, b)), o_T = place (fix_bytes_T (7, p));
  const size_t o_WB = place (fix_bytes_WB (7, p));
  const size_t zero1 = bytes;
  const size_t o_G = place (fix_bytes_G (7, p));
  const size_t o_S = place (sizeof (long long) * (size_t) 4 * p.nqp * p.ldT);
  const size_t o_yp = place (sizeof (double) * (size_t) p.nbitem * 16 * p.ldT);
  int bin0, nbin;
  real_tab_range (rc, &bin0, &nbin);
  const size_t o_tab = place (real_tab_bytes (sys->version, nbin));
  const size_t o_q = place (sizeof (uint4) * b.np), o_u = place (sizeof (unsigned long long) * 4 * b.np);
  cudaStream_t st = c->stream;
  // no build of this context may still be using the tables of the last set-up
  cudaError_t e = f->arena.p ? wait_products (c) : cudaSuccess;
  if (e == cudaSuccess) e = f->arena.ensure (bytes);
  char *base = (char *) f->arena.p;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync (base, host.data (), host.size (), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync (base + zero0, 0, zero1 - zero0, st);
  if (e == cudaSuccess) e = status_word (&f->h_status, &f->d_status);
  if (e != cudaSuccess) return cuda_fail (e, "dense builder set-up");
  p.quart = (const int4 *) (base + o_quart);
  p.nqm = (const int *) (base + o_nqm);
  p.bitem = (const int4 *) (base + o_item);
  p.mx = (unsigned *) (base + o_mx);
  p.T = base + o_T; p.G = base + o_G; p.WB = base + o_WB; p.S = base + o_S; p.yp = base + o_yp;
  b.T = base + o_Tb;
  b.mx = p.mx;
  b.q = (uint4 *) (base + o_q);
  b.u = (unsigned long long *) (base + o_u);
  const int me = fix_map_wb (p, &f->maps);
  if (me) return set_error (STOKES_GPU_ECUDA, "TMA tensor map of the dense builder (%d)", me);
  WeightArgs w {};
  for (int d = 0; d < 3; d++)
    {
      w.k0[d] = k0[d];
      w.ref[d] = ref[d];
    }
  w.xi2 = ts->xi2; w.kmax = ts->kmax;
  w.pivol = M_PI / (sys->lx * sys->ly * sys->lz);
  w.xi2_ref = sys->xi2; w.kmax_ref = sys->kmax; w.pivol_ref = sys->pivol;
  w.fts = fts;
  w.mom = (const Moment *) (base + o_mom);
  w.blk = (const int2 *) (base + o_blk);
  for (int cl = 0; cl < 4; cl++) w.blk0[cl] = blk0[cl];
  k_dense_weights<<<dim3 ((p.Rp + 127) / 128, p.ncol), 128, 0, st>>> (p, w);
  e = cudaGetLastError ();
  if (e == cudaSuccess) e = launch_fix_dense_image (p, st);
  if (e == cudaSuccess)
    {
      double *tab = (double *) (base + o_tab);
      e = launch_real_tab_build (sys->version, bin0, nbin, ts->xi, tab,
                                 (float *) (tab + real_tab_doubles (sys->version, nbin)), st);
    }
  // the upload reads host vectors of this call
  if (e == cudaSuccess) e = cudaStreamSynchronize (st);
  if (e != cudaSuccess) return cuda_fail (e, "dense builder set-up");
  a.np = sys->np;
  a.ldT = p.ldT;
  for (int d = 0; d < 3; d++)
    {
      a.sf[d] = (float) (p.l[d] / 4294967296.0);
      a.s60[d] = p.l[d] / 1152921504606846976.0;
    }
  a.q = b.q;
  a.u = b.u;
  a.rc2 = (float) (ts->rmax2 * 1.00001);
  a.xi = ts->xi;
  a.xisp = ts->xi / sqrt (M_PI);
  a.off = (const float4 *) (base + o_off);
  a.cell = (const int4 *) (base + o_cell);
  a.noff = (int) off.size ();
  a.tab = (const double *) (base + o_tab);
  a.bin0 = bin0;
  a.nbin = nbin;
  // two particles at one place: libstokes leaves the pair's own image out of
  // the real space, so the result follows its split; the self terms of the
  // two splits are the difference
  const double s1[3] = {ts->self_a, ts->self_c, ts->self_m}, s0[3] = {sys->self_a, sys->self_c, sys->self_m};
  for (int d = 0; d < 3; d++)
    {
      a.self[d] = s1[d];
      a.same[d] = s1[d] - s0[d];
    }
  a.yp = (const double *) p.yp;
  for (int cl = 0; cl < 4; cl++) a.cls[cl] = p.cls[cl];
  a.rec = (const int2 *) (base + o_rec);
  a.nrec = (int) rec.size ();
  a.der = (const Terms<MAX_DER> *) (base + o_der);
  a.entry = (const Terms<MAX_TERM> *) (base + o_entry);
  a.tile = (const int2 *) (base + o_tile);
  f->a = a;
  f->p = p;
  f->base = b;
  memcpy (f->key, key, sizeof key);
  return STOKES_GPU_OK;
}

template <int V>
static cudaError_t
dense_chunk (const DenseArgs &a, cudaStream_t st, Ctx *c)
{
  // X, then mo and out; the entries of the real space lie in mo's place
  const size_t smem = sizeof (double)
                      * (PT * (size_t) (NReal<V>::value + a.nrec)
                         + std::max ((size_t) PT * (Moments<V>::N + NComp<V>::value),
                                     (size_t) WIN * (3 + NFun<V>::value)));
  static int attr_dev = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e == cudaSuccess && attr_dev != dev)
    {
      e = cudaFuncSetAttribute (k_dense_tile<V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int) smem);
      if (e == cudaSuccess) attr_dev = dev;
    }
  if (e != cudaSuccess) return e;
  k_dense_tile<V><<<a.ntile, DT, smem, st>>> (a);
  kmark (c, st, "k_dense_tile");
  return cudaGetLastError ();
}

int
matrix_fix_dev (Ctx *c, const double *d_pos, double *d_mat, cudaStream_t st)
{
  const int rc = dense_setup (c, c->sys);
  if (rc) return rc;
  DenseState *f = c->dfix;
  const int failed = earlier_failure (c, f->h_status,
                                      "a tensor-core wait of the previous dense builder ran out");
  if (failed) return failed;
  FixPlan p = f->p;
  p.stall = g_test_gemm_stall;
  int *status = f->d_status;
  kmark (c, st, nullptr);
  cudaError_t e = launch_fix_functions (f->base, d_pos, st);
  if (e != cudaSuccess) return cuda_fail (e, "function tables");
  kmark (c, st, "k_fix_tables");
  int launches = 1;
  for (int t0 = 0; t0 < f->tiles; t0 += f->chunk)
    {
      DenseArgs a = f->a;
      a.pos = d_pos;
      a.mat = d_mat;
      a.tile += t0;
      a.ntile = std::min (f->chunk, f->tiles - t0);
      if ((e = launch_fix_dense (f->base, p, f->maps, a.tile, a.ntile, status, st, c)) != cudaSuccess)
        return cuda_fail (e, "matrix kernel (reciprocal)");
      e = c->version == 0 ? dense_chunk<0> (a, st, c)
                          : (c->version == 1 ? dense_chunk<1> (a, st, c) : dense_chunk<2> (a, st, c));
      if (e != cudaSuccess) return cuda_fail (e, "matrix kernel");
      launches += 4;
    }
  c->launches = launches;
  return STOKES_GPU_OK;
}

// after the stream of a build was synchronised
int
dense_check_status (Ctx *c)
{
  DenseState *f = c->dfix;
  if (!f || !f->h_status || !*f->h_status) return STOKES_GPU_OK;
  *f->h_status = 0;
  return set_error (STOKES_GPU_ETIMEOUT, "a tensor-core wait of the dense builder ran out");
}

void
release_dense (Ctx *c)
{
  DenseState *f = c->dfix;
  if (!f) return;
  f->arena.release ();
  if (f->ts) stokes_free (f->ts);
  if (f->h_status) cudaFreeHost (f->h_status);
  delete f;
  c->dfix = nullptr;
}

}  // namespace lsg
