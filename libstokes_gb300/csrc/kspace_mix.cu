// kspace_mix.cu -- reciprocal space of the mixed product as tensor-core GEMMs.
//
// The sum is written in products of real functions of x, y and z, as in
// kspace_fix.cu (function index 0 of an axis is 1, 2 m - 1 is cos 2 pi m u, 2 m
// is sin 2 pi m u):
//
//   forward   F[n][r] = sum_j A[r][j] B[n][j],   A = f_y f_z,  B = f_x x_q
//             (k_sfac_gemm; row r = (y, z functions), column n = (mi, q))
//   operator  cosine and sine sums of the four sign patterns of (|m1|, |m2|,
//             |m3|), the Ewald weights, and back (k_kop)
//   backward  y_q(i) = sum_mi f_x(i) sum_r A[r][i] G[n][r]     (k_bp_gemm)
//
// Operands are fixed-point numbers in three 8-bit digits, exact in f16: A, |f|
// <= 1, with 24 fractional bits (the top digit up to 256); B with 25 (up to 512)
// in units of the largest entry of its column within 128 K values, so that a
// column of very different entries keeps its digits.  Six digit products (i + j
// < 3) in three accumulators; 128 K values keep every sum below 2^24, so the
// FP32 accumulation of the tensor core is exact, and each 128-wide set is
// scaled by its unit and added in FP32.  Rounding is 2^-25 for A and 2^-26 of
// the largest entry for B: with 24 bits, forces of one size lost two of theirs
// to the unit (the next power of two above the largest of 128), and products of
// some hundred unequal spheres came out up to 27% further from FP64 than with
// FP32 sums (F N = 600 1.96e-7, 2.39e-7 with 24 bits, 1.67e-7 now).  The 3xTF32 split used before carried 22 bits, had to
// be drained every 32 K values (the tensor core truncates inexact sums) and
// multiplied k and -k separately.  Kernel times between events, before and now
// (at the same split, eta 11, for N = 12001):
//                     forward            back-projection
//   FTS N = 1000      24.8 -> 16.5 us    25.0 -> 18.5 us
//   F   N = 4096      32   -> 18.5       36.8 -> 21.5
//   FTS N = 12001     168  -> 85         267  -> 104
//
// The unit of a B column comes out of the kernel that writes it: mk_prep takes
// the maxima of its 128 particles, k_kop those of its 128 rows, so no pass
// over the data comes before.
//
// One MMA takes digit i of A against the digits 0 .. 2 - i of B, which lie one
// after the other as rows of the tile (N up to 256).  What bounds the GEMMs is
// the build of A (about 20 instructions a value, 16 warps), so a tile has up to
// 128 columns for each A that is built (N = 12001 backward 117 us at 64 columns
// in two accumulator sets, 86 at 128 before the epilogue).
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "digit_gemm.cuh"
#include "ewald_device.cuh"
#include "gpu_engine.h"
#include "mixed.h"
#include "pdl.cuh"
#include "tma_host.h"

namespace lsg {
namespace {

using namespace dg;

constexpr int ND = 3;
constexpr int KT = 64;                  // K values per tile (128-byte rows)
constexpr int DK = 2;                   // tiles per set (K = 128)
constexpr int KB = DK * KT;             // K values per unit
constexpr int TN_MAX = 128;             // columns per tile at most
constexpr uint32_t A_PLANE = TM * 128;
constexpr float UNIT = 1.0f / 131072.0f;        // of a product of two top digits: 2^-8 of A, 2^-9 of B

constexpr int NS = 2;                   // stages (three leave too little L1 for the builds' loads)
constexpr uint32_t A_BYTES = ND * A_PLANE;
__host__ __device__ constexpr uint32_t b_bytes (int tn) { return ND * (uint32_t) tn * 128u; }
__host__ __device__ constexpr uint32_t stage_bytes (int tn) { return A_BYTES + b_bytes (tn); }
constexpr uint32_t SMEM_DYN = NS * stage_bytes (TN_MAX) + 1024;

// ---- digits ---------------------------------------------------------------
// a product of two 30-bit fractions (upper word: 28 fractional bits) as a
// biased string of `bits` fractional bits: bytes 0 and 1 are the lower digits
// plus 128, the upper half the top digit plus 512
constexpr int A_BITS = 24, B_BITS = 25;
template <int bits>
__device__ __forceinline__ int
biased (int hi)
{
  constexpr int sh = 28 - bits;
  return (hi + ((0x02008080 << sh) + (1 << (sh - 1)))) >> sh;
}

__device__ __forceinline__ uint32_t
half2_minus (uint32_t v, unsigned short bias)
{
  const __half2 r = __hsub2 (*reinterpret_cast<__half2 *> (&v), __half2half2 (__ushort_as_half (bias)));
  return *reinterpret_cast<const uint32_t *> (&r);
}

// the f16 pairs (digit of a, digit of b), digit by digit; 0x6400 + n is the
// f16 number 1024 + n
__device__ __forceinline__ void
digits (int a, int b, uint32_t out[ND])
{
  out[0] = half2_minus (__byte_perm (a, b, 0x7632) + 0x64006400u, 0x6600);
  out[1] = half2_minus ((__byte_perm (a, b, 0x5511) & 0x00FF00FFu) | 0x64006400u, 0x6480);
  out[2] = half2_minus ((__byte_perm (a, b, 0x4400) & 0x00FF00FFu) | 0x64006400u, 0x6480);
}

// the unit 2^E > every |v| with |v| <= the float of bits mx, and 2^-E; NaN
// for infinite or NaN entries, so that the results they enter are NaN
__device__ __forceinline__ float
unit_of (uint32_t mx, float &inverse)
{
  const int e = (int) (mx >> 23);
  if (e == 255)
    {
      inverse = 0.f;
      return __int_as_float (0x7fc00000);
    }
  const int E = max (e, 1) - 126;                       // -125 .. 128
  inverse = __int_as_float ((127 - E) << 23);           // E = 128: a denormal, 2^-128 by hand
  if (E >= 127) inverse = E == 127 ? 5.877471754111438e-39f : 2.938735877055719e-39f;
  return E == 128 ? __int_as_float (0x7f800000) : __int_as_float ((E + 127) << 23);
}

// ---- operand builders (see run_tiles in digit_gemm.cuh) --------------------
// Forward: rows r0 .. + 127, particles j0 .. + 63.  A warp makes two quarters
// (eight rows), a lane two particles.
struct BuildF {
  const int *T;
  int4 f[2];
  int j0, ldT;
  int2 v[2][4];
  __device__ __forceinline__ BuildF (const MixPlan &p, int r0, int jb) : T (p.T), ldT (p.ldT)
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    f[0] = p.quart[r0 / 4 + 2 * warp];
    f[1] = p.quart[r0 / 4 + 2 * warp + 1];
    j0 = jb + 2 * lane;
  }
  __device__ __forceinline__ void load (int t)
  {
    const size_t jo = (size_t) j0 + KT * t;
#pragma unroll
    for (int u = 0; u < 2; u++)
      {
        v[u][0] = *reinterpret_cast<const int2 *> (T + (size_t) f[u].x * ldT + jo);
        v[u][1] = *reinterpret_cast<const int2 *> (T + (size_t) f[u].y * ldT + jo);
        v[u][2] = *reinterpret_cast<const int2 *> (T + (size_t) f[u].z * ldT + jo);
        v[u][3] = *reinterpret_cast<const int2 *> (T + (size_t) f[u].w * ldT + jo);
      }
  }
  __device__ __forceinline__ void store (unsigned char *stage) const
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int b = 0; b < 4; b++)
        {
          const int2 y = v[u][b >> 1], z = v[u][2 + (b & 1)];
          uint32_t d[ND];
          digits (biased<A_BITS> (__mulhi (y.x, z.x)), biased<A_BITS> (__mulhi (y.y, z.y)), d);
          unsigned char *o = stage + chunk_off (8 * warp + 4 * u + b, lane >> 2) + (lane & 3) * 4;
#pragma unroll
          for (int q = 0; q < ND; q++) *reinterpret_cast<uint32_t *> (o + q * A_PLANE) = d[q];
        }
  }
};

// Backward: particles i0 .. + 127, one per lane, 64 rows, 16 of them (four
// quarters) per thread
struct BuildB {
  const int *T;
  const int4 *quart;
  int i, ldT;
  int v[4][4];
  __device__ __forceinline__ BuildB (const MixPlan &p, int i0, int r0) : T (p.T), ldT (p.ldT)
  {
    quart = p.quart + r0 / 4 + 4 * (threadIdx.x >> 7);
    i = i0 + (threadIdx.x & 127);
  }
  __device__ __forceinline__ void load (int t)
  {
#pragma unroll
    for (int u = 0; u < 4; u++)
      {
        const int4 f = __ldg (quart + t * (KT / 4) + u);
        v[u][0] = T[(size_t) f.x * ldT + i];
        v[u][1] = T[(size_t) f.y * ldT + i];
        v[u][2] = T[(size_t) f.z * ldT + i];
        v[u][3] = T[(size_t) f.w * ldT + i];
      }
  }
  __device__ __forceinline__ void store (unsigned char *stage) const
  {
    const int row = threadIdx.x & 127, c0 = 2 * (threadIdx.x >> 7);
#pragma unroll
    for (int h = 0; h < 2; h++)
      {
        uint32_t w[4][ND];
#pragma unroll
        for (int u = 0; u < 4; u++)
          {
            const int *f = v[2 * h + (u >> 1)];
            const int y = f[u & 1];
            digits (biased<A_BITS> (__mulhi (y, f[2])), biased<A_BITS> (__mulhi (y, f[3])), w[u]);
          }
#pragma unroll
        for (int q = 0; q < ND; q++)
          *reinterpret_cast<uint4 *> (stage + q * A_PLANE + chunk_off (row, c0 + h))
            = make_uint4 (w[0][q], w[1][q], w[2][q], w[3][q]);
      }
  }
};

// ---- the GEMM of both directions ------------------------------------------
// the MMAs of one tile: group g in TMEM columns g tn; digit i of A against the
// digits j <= 2 - i of B, as many of them as N <= 256 allows at once
__device__ __forceinline__ void
issue_tile (uint32_t a, uint32_t tmem, int tn, bool first)
{
  const uint32_t b = a + A_BYTES;
  const bool split = 3 * tn > 256;
  const uint32_t i1 = umma::idesc_f16 (TM, (uint32_t) tn), i2 = umma::idesc_f16 (TM, (uint32_t) (2 * tn)),
                 i3 = umma::idesc_f16 (TM, (uint32_t) (3 * tn));
#pragma unroll
  for (int k = 0; k < KT / 16; k++)
    {
      const uint64_t a0 = umma::smem_desc_sw128 (a + 32 * k),
                     a1 = umma::smem_desc_sw128 (a + A_PLANE + 32 * k),
                     a2 = umma::smem_desc_sw128 (a + 2 * A_PLANE + 32 * k),
                     b0 = umma::smem_desc_sw128 (b + 32 * k);
      const uint32_t add = first && k == 0 ? 0u : 1u;
      if (split)
        {
          umma::mma_f16 (tmem, a0, b0, i2, add);
          umma::mma_f16 (tmem + 2 * tn, a0, umma::smem_desc_sw128 (b + 2 * b_bytes (tn) / 3 + 32 * k), i1,
                         add);
        }
      else
        umma::mma_f16 (tmem, a0, b0, i3, add);
      umma::mma_f16 (tmem + tn, a1, b0, i2, 1u);
      umma::mma_f16 (tmem + 2 * tn, a2, b0, i1, 1u);
    }
}

// running sums of one worker: columns 16 cg .. + 15 and 64 + 16 cg .. + 15 of
// its row (cg = warp / 4).  A set of accumulators is scaled by the columns'
// units of its 128 K values: lane l holds that of the warp's column l, read a
// set ahead.
struct Sums {
  float v[2][16];
  const float *units;           // this lane's column
  float unit;
  int ld, tn, col, sets;
  uint32_t tmem;
  __device__ __forceinline__ void take (int set, int)
  {
    const float u0 = unit;
    if (set + 1 < sets) unit = units[(size_t) (set + 1) * ld];
#pragma unroll
    for (int h = 0; h < 2; h++)
      {
        if (col + 64 * h >= tn) continue;         // uniform in the warp
        float f1[16], f2[16];
        umma::tmem_ld16_issue (tmem + 64 * h + 2 * tn, f2);
        umma::tmem_ld16_issue (tmem + 64 * h + tn, f1);
        umma::tmem_ld_wait (f2);
        umma::tmem_ld_wait (f1);
#pragma unroll
        for (int u = 0; u < 16; u++) f1[u] = fmaf (f2[u], 1.0f / 256.0f, f1[u]);
        umma::tmem_ld16_issue (tmem + 64 * h, f2);
        umma::tmem_ld_wait (f2);
#pragma unroll
        for (int u = 0; u < 16; u++)
          v[h][u] = fmaf (__shfl_sync (0xffffffffu, u0, 16 * h + u), fmaf (f1[u], 1.0f / 256.0f, f2[u]),
                          v[h][u]);
      }
  }
};

// the tiles of one CTA: columns n0 .. + tn, K from k0; true when the sums are
// complete.  units: the units of B, [K / 128][ld], from the first set and the
// tile's first column.
template <class Build>
__device__ __forceinline__ bool
gemm_cta (Sync &s, unsigned char *smem, const CUtensorMap *tmB, int tn, int n0, int k0, int ntiles,
          int stall, const float *units, int ld, Build &build, Sums &acc)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem = s.tslot;
#pragma unroll
  for (int u = 0; u < 16; u++) acc.v[0][u] = acc.v[1][u] = 0.f;
  acc.col = 16 * ((warp >> 2) & 3);
  acc.ld = ld;
  acc.tn = tn;
  acc.sets = (ntiles + DK - 1) / DK;
  acc.tmem = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + (uint32_t) acc.col;
  const int mine = acc.col + (lane & 15) + 64 * (lane >> 4);
  acc.units = units + min (mine, tn - 1);
  acc.unit = acc.sets > 0 ? *acc.units : 0.f;
  const BTiles bt {tmB, k0, KT, n0, A_BYTES, b_bytes (tn)};
  return run_tiles<DK, 1, NS> (s, smem, ntiles, stage_bytes (tn), bt, stall, build, acc,
                               [=] (uint32_t a, int, bool first) { issue_tile (a, tmem, tn, first); });
}

__host__ __device__ __forceinline__ int
col_m (int n, int c)
{
  return (n / c + 1) / 2;                // |m1| of column n, c columns per function
}

// forward: a CTA takes one item (row tile, column tile, particle slice) and
// writes F[slice][column][row]; lanes are consecutive rows, so the stores
// coalesce
__global__ void __launch_bounds__ (NT, 1)
k_sfac_gemm (const __grid_constant__ CUtensorMap tmB, MixPlan p, int *status)
{
  extern __shared__ unsigned char dsm[];
  __shared__ Sync s;
  const int4 it = p.fitem[blockIdx.x];
  const int r0 = it.x * TM, n0 = it.y * p.tnf;
  unsigned char *smem = align1k (dsm);
  const int jb = it.z * p.jper, je = min (p.ldT, jb + p.jper);
  const int ntiles = je > jb ? (je - jb) / KT : 0;
  chain_next ();
  cta_setup (s);
  const uint32_t tmem = s.tslot;
  BuildF build (p, r0, jb);
  chain_wait ();
  Sums acc;
  if (gemm_cta (s, smem, &tmB, p.tnf, n0, jb, ntiles, p.stall,
                p.zs + (size_t) (jb / KB) * p.ldf + n0, p.ldf, build, acc))
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      float *F = p.F + ((size_t) it.z * p.ncolf + n0) * p.Rp + r0 + (warp & 3) * 32 + lane;
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int u = 0; u < 16; u++)
          {
            const int n = acc.col + 64 * h + u;
            if (n < p.tnf && n0 + n < p.ncolf) F[(size_t) n * p.Rp] = acc.v[h][u];
          }
    }
  cta_finish (s, tmem, status);
}

// backward: a CTA takes 128 particles and one item (column tile, first K
// tile, K tiles); the sums are parked in the freed stages and reduced over
// the x functions of the tile into the item's partial y.  POLY: the columns of
// k_kop_poly, each with its power of the particle's radius.
template <bool POLY>
__global__ void __launch_bounds__ (NT, 1)
k_bp_gemm (const __grid_constant__ CUtensorMap tmB, MixPlan p, int *status)
{
  constexpr int HLD = TN_MAX + 1;
  // parked sums and the x functions of 128 columns (three components: 44)
  static_assert ((TM * HLD + 44 * TM) * sizeof (float) <= NS * A_BYTES, "parked tile");
  extern __shared__ unsigned char dsm[];
  __shared__ Sync s;
  unsigned char *smem = align1k (dsm);
  const int4 it = p.bitem[blockIdx.y];
  const int i0 = blockIdx.x * TM, n0 = it.x * p.tnb, k0 = it.y * KT;
  cta_setup (s);
  const uint32_t tmem = s.tslot;
  BuildB build (p, i0, k0);
  Sums acc;
  float *H = reinterpret_cast<float *> (smem), *X = H + TM * HLD;
  const int cb = p.cb, ne = min (p.tnb, p.ncolb - n0), f0 = n0 / cb, nf = (n0 + ne - 1) / cb - f0 + 1;
  chain_wait ();
  // the x functions of the tile's columns, read ahead (a load per term of the
  // epilogue waited for L2 every time: 10 us at FTS N = 1000)
  constexpr int XW = 32 * WORKERS, XMAX = (44 * TM + XW - 1) / XW;
  int xr[XMAX];
  if ((int) threadIdx.x < XW)
#pragma unroll
    for (int k = 0; k < XMAX; k++)
      {
        const int e = (int) threadIdx.x + XW * k;
        xr[k] = e < nf * TM ? p.T[(size_t) (f0 + e / TM) * p.ldT + i0 + e % TM] : 0;
      }
  if (gemm_cta (s, smem, &tmB, p.tnb, n0, k0, it.z, p.stall, p.ws + (size_t) (k0 / KB) * p.ldb + n0,
                p.ldb, build, acc))
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      // the last set is drained, so every build, load and MMA is done and the
      // stages are free
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int u = 0; u < 16; u++)
          if (acc.col + 64 * h < p.tnb)
            H[((warp & 3) * 32 + lane) * HLD + acc.col + 64 * h + u] = acc.v[h][u];
#pragma unroll
      for (int k = 0; k < XMAX; k++)
        if ((int) threadIdx.x + XW * k < nf * TM) X[threadIdx.x + XW * k] = (float) xr[k];
    }
  __syncthreads ();
  if (!s.err)
    {
      const int c = p.c;
      float *yp = p.yp + (size_t) blockIdx.y * p.np * c;
      for (int e = threadIdx.x; e < TM * c; e += NT)
        {
          const int q = e / TM, r = e - q * TM, i = i0 + r;
          if (i >= p.np) continue;
          // sum of column k of the functions
          auto column = [&] (int k) {
            float y = 0.f;
            for (int n = (k + cb - n0 % cb) % cb; n < ne; n += cb)
              y = fmaf (X[((n0 + n) / cb - f0) * TM + r], H[r * HLD + n], y);
            return y;
          };
          float y;
          if constexpr (!POLY)
            y = column (q);
          else
            {
              const float a = p.rad[i], a2 = a * a;
              if (c == 3) y = a * fmaf (a2, column (3 + q), column (q));
              else
                {
                  // a^2 and a^3; then a (U) and, for FTS, a^4 (U, E), a^5 (E)
                  y = a2 * fmaf (a, column (c + 3 + q), column (3 + q));
                  if (q < 3) y = fmaf (a, column (q), y);
                  if (c == 11 && (q < 3 || q >= 6))
                    {
                      float z = column (q < 3 ? 25 + q : 22 + q);
                      if (q >= 6) z = fmaf (a, column (27 + q), z);
                      y = fmaf (a2 * a2, z, y);
                    }
                }
            }
          yp[(size_t) i * c + q] = y * 0x1p-30f;
        }
    }
  cta_finish (s, tmem, status);
}

// ---- tables and the forward image -----------------------------------------
constexpr int PREP_P = KB;              // particles per CTA: one unit
constexpr int PREP_T = 256;
constexpr int PREP_I = 4;               // (axis, m) items per CTA

// Fixed-point positions (wrapped to the primary cell, Lees-Edwards aware), x
// in FP32, the function table and the forward image.  u_d is the particle's
// fractional coordinate on axis d as a 32-bit fixed point q_d, so m u_d mod 1
// is the exact integer product m q_d mod 2^32; on a sheared lattice the
// flow-axis phase coordinate is u_x - (shift / lx) u_g.
// CTA (x, y): 128 particles, the items y, y + G, y + 2 G, y + 3 G (G =
// gridDim.y), so that the x functions, which also write the image, spread over
// the CTAs; the few operations per particle are repeated by each of them.
// Unequal radii: the image has the components x_q and then a_j^2 x_q.
__global__ void __launch_bounds__ (PREP_T)
mk_prep_tc (MixPrep a)
{
  constexpr int CMAX = 22;
  __shared__ uint32_t s_q[3][PREP_P];
  __shared__ float s_x[CMAX][PREP_P + 1];
  __shared__ uint32_t s_mx[CMAX];
  __shared__ float s_inv[CMAX];
  __shared__ int s_f[PREP_I][2][PREP_P];
  const MixPlan &p = a.p;
  const int t = threadIdx.x, jb = blockIdx.x * PREP_P, G = gridDim.y;
  const bool lead = blockIdx.y == 0;
  chain_next ();
  for (int e = t; e < PREP_P * a.c; e += PREP_T)
    {
      const int jl = e / a.c, q = e - jl * a.c, j = jb + jl;
      const float v = j < a.np ? (float) a.x[(size_t) j * a.c + q] : 0.f;
      s_x[q][jl] = v;
      if (p.cf > a.c) s_x[a.c + q][jl] = j < a.np ? a.qa[j] * v : 0.f;
      if (lead && j < a.np) a.xf[(size_t) j * ((a.c + 3) & ~3) + q] = v;
    }
  if (t < PREP_P)
    {
      const int j = jb + t;
      uint32_t q0 = 0, q1 = 0, q2 = 0, qu = 0;
      if (j < a.np)
        {
          double x = a.pos[3 * j];
          const double y = a.pos[3 * j + 1], z = a.pos[3 * j + 2];
          if (a.shear_mode == 1 || a.shear_mode == 2)
            {
              // wraps along the gradient axis shift the flow coordinate
              const long long g = __double2ll_rd ((a.shear_mode == 1 ? y * a.sy : z * a.sz));
              x = fma (-(double) (g >> 32), a.shift, x);
            }
          q0 = fixq (x * a.sx);
          q1 = fixq (y * a.sy);
          q2 = fixq (z * a.sz);
          qu = q0;
          if (a.shear_mode == 1) qu = q0 - fixq (a.sl * (double) q1);
          else if (a.shear_mode == 2) qu = q0 - fixq (a.sl * (double) q2);
          if (lead) reinterpret_cast<uint4 *> (a.qpos)[j] = make_uint4 (q0, q1, q2, 0u);
        }
      s_q[0][t] = qu; s_q[1][t] = q1; s_q[2][t] = q2;
    }
  __syncthreads ();
  // the units: one warp per component (atomics on a handful of words took 2 us)
  for (int q = t >> 5; q < p.cf; q += PREP_T / 32)
    {
      uint32_t mx = 0u;
#pragma unroll
      for (int k = 0; k < PREP_P / 32; k++)
        mx = max (mx, __float_as_uint (s_x[q][(t & 31) + 32 * k]) & 0x7fffffffu);
      mx = __reduce_max_sync (0xffffffffu, mx);
      if ((t & 31) == 0)
        {
          float inv;
          unit_of (mx, inv);
          s_mx[q] = mx;
          s_inv[q] = inv;
        }
    }
  if (lead) __syncthreads ();
  if (lead)
    for (int n = t; n < p.ldf; n += PREP_T)
      {
        float inv;
        p.zs[(size_t) blockIdx.x * p.ldf + n] = n < p.ncolf ? unit_of (s_mx[n % p.cf], inv) * UNIT : 0.f;
      }
  const int n0 = p.M[0] + 1, n1 = n0 + p.M[1] + 1, n2 = n1 + p.M[2] + 1;
  for (int k = t; k < PREP_I * PREP_P; k += PREP_T)
    {
      const int rr = k / PREP_P, jl = k - rr * PREP_P, item = blockIdx.y + rr * G;
      if (item >= n2) break;
      const int d = item < n0 ? 0 : (item < n1 ? 1 : 2);
      const int m = item - (d == 0 ? 0 : (d == 1 ? n0 : n1));
      const float2 ph = phase_of (a.rot, (uint32_t) m * s_q[d][jl]);
      const bool in = jb + jl < a.np;
      const int cs = in ? __float2int_rn (ph.x * 0x1p30f) : 0, sn = in ? __float2int_rn (ph.y * 0x1p30f) : 0;
      int *row = p.T + (size_t) ((d == 0 ? 0 : (d == 1 ? p.oy : p.oz)) + (m ? 2 * m - 1 : 0)) * p.ldT
                 + jb + jl;
      row[0] = cs;
      if (m) row[p.ldT] = sn;
      s_f[rr][0][jl] = cs;
      s_f[rr][1][jl] = sn;
    }
  __syncthreads ();
  // x functions of this CTA: digits of f_x x_q, eight particles (16 bytes per
  // digit) per thread
  int nx = 0;
  while (nx < PREP_I && (int) blockIdx.y + nx * G < n0) nx++;
  for (int e = t; e < nx * 2 * p.cf * (PREP_P / 8); e += PREP_T)
    {
      const int j8 = e % (PREP_P / 8), w = e / (PREP_P / 8), q = w % p.cf, fs = w / p.cf;
      const int rr = fs >> 1, part = fs & 1, m = blockIdx.y + rr * G;
      if (part && m == 0) continue;
      const int mi = m ? 2 * m - 1 + part : 0;
      const float inv = s_inv[q];
      uint32_t d[4][ND];
#pragma unroll
      for (int u = 0; u < 4; u++)
        {
          int v[2];
#pragma unroll
          for (int h = 0; h < 2; h++)
            {
              const int jl = 8 * j8 + 2 * u + h;
              const int xs = __float2int_rn (s_x[q][jl] * inv * 0x1p30f);
              v[h] = biased<B_BITS> (__mulhi (s_f[rr][part][jl], xs));
            }
          digits (v[0], v[1], d[u]);
        }
      uint4 *o = reinterpret_cast<uint4 *> ((__half *) p.ZF + (size_t) (mi * p.cf + q) * p.ldT + jb) + j8;
#pragma unroll
      for (int q3 = 0; q3 < ND; q3++)
        o[(size_t) q3 * p.ncolf * p.ldT / 8] = make_uint4 (d[0][q3], d[1][q3], d[2][q3], d[3][q3]);
    }
}

// ---- operators -------------------------------------------------------------
// Eight lanes per octant point.  Lane (w, b): b = 2 p2 + p3 names the row of
// the quarter, and after the transform the sign pattern (s2, s3) = (1 - 2 (b >>
// 1), 1 - 2 (b & 1)); w = 0 carries the cosine sums C and makes P, w = 1 the
// sine sums S and makes Q.  Row b enters C with its cosine column for b = 0, 3
// and its sine column for b = 1, 2, and S with the other one; G goes back the
// same way, so every lane reads and writes one column set.  Latency bounds it
// (a few thousand points): four lanes a point, each with both sums, took 13.8
// us at FTS N = 1000 (cold), this 8.1.
constexpr int KOP_T = 2 * KB;           // threads per CTA: 128 rows, one unit

struct KopLane {
  int m1, b, w, qr, row;
  bool live, sine, neg, have;           // have: its column set exists
  __device__ __forceinline__ KopLane (int nqm)
  {
    m1 = blockIdx.y;
    b = threadIdx.x & 3;
    w = (threadIdx.x >> 2) & 1;
    qr = blockIdx.x * (KOP_T / 8) + threadIdx.x / 8;
    row = 4 * qr + b;
    live = qr < nqm;
    sine = (b == 0 || b == 3) == (w == 1);
    neg = b == 3 || (w == 0 && b != 0);
    have = !(sine && m1 == 0);
  }
  // first column of this lane's x function, c columns per function
  __device__ __forceinline__ int col (int c) const
  {
    return (sine ? 2 * m1 : (m1 ? 2 * m1 - 1 : 0)) * c;
  }
};

// this lane's sums of the C components from column `first` of each function
template <int C>
__device__ __forceinline__ void
sums (const MixPlan &p, const KopLane &l, int first, float (&x)[C])
{
#pragma unroll
  for (int q = 0; q < C; q++) x[q] = 0.f;
  if (l.live && l.have)
#pragma unroll 4
    for (int s = 0; s < p.nsplit; s++)
      {
        const float *F = p.F + ((size_t) s * p.ncolf + l.col (p.cf) + first) * p.Rp + l.row;
#pragma unroll
        for (int q = 0; q < C; q++) x[q] += F[(size_t) q * p.Rp];
      }
#pragma unroll
  for (int q = 0; q < C; q++) x[q] = walsh4 (flip (x[q], l.neg), l.b);
}

// this lane's G of C components into the backward image, columns `first` on of
// its function, in the unit of the CTA's 128 rows (rows past the set but
// within its last 128 are zero)
template <int C>
__device__ __forceinline__ void
put_rows (const MixPlan &p, const KopLane &l, int first, float (&g)[C], uint32_t (*s_mx)[2])
{
  __syncthreads ();
  for (int k = threadIdx.x; k < 2 * C; k += KOP_T) (&s_mx[0][0])[k] = 0u;
  __syncthreads ();
#pragma unroll
  for (int q = 0; q < C; q++)
    {
      const float v = walsh4 (g[q], l.b);
      g[q] = l.live && l.have ? flip (v, l.neg) : 0.f;
      const uint32_t a = __float_as_uint (g[q]) & 0x7fffffffu;
      const uint32_t mc = __reduce_max_sync (0xffffffffu, l.sine ? 0u : a);
      const uint32_t ms = __reduce_max_sync (0xffffffffu, l.sine ? a : 0u);
      if ((threadIdx.x & 31) < 2) atomicMax (&s_mx[q][threadIdx.x & 1], threadIdx.x & 1 ? ms : mc);
    }
  __syncthreads ();
  const int n0 = l.col (p.cb) + first;
  if (l.have)
    {
      __half *o = (__half *) p.WB + (size_t) n0 * p.Rp + l.row;
#pragma unroll
      for (int q = 0; q < C; q++)
        {
          float inv;
          unit_of (s_mx[q][l.sine], inv);
          const int w = __float2int_rn (g[q] * inv * 0x1p25f) + 0x02008080;     // B_BITS
          uint32_t d[ND];
          digits (w, w, d);
#pragma unroll
          for (int k = 0; k < ND; k++)
            o[((size_t) k * p.ncolb + q) * p.Rp] = __ushort_as_half ((unsigned short) d[k]);
        }
    }
  // the columns' units: threads 2 q + part
  if ((int) threadIdx.x < 2 * C)
    {
      const int q = threadIdx.x >> 1, part = threadIdx.x & 1;
      float inv;
      const int n = (part ? 2 * l.m1 : (l.m1 ? 2 * l.m1 - 1 : 0)) * p.cb + first + q;
      if (!(part && l.m1 == 0))
        p.ws[(size_t) blockIdx.x * p.ldb + n] = unit_of (s_mx[q][part], inv) * UNIT;
    }
}

template <int V>
__global__ void __launch_bounds__ (KOP_T)
k_kop (MixPlan p)
{
  constexpr int C = NComp<V>::value;
  __shared__ uint32_t s_mx[C][2];
  const int nqm = p.nqm[blockIdx.y];
  chain_next ();
  if ((int) (blockIdx.x * (KOP_T / 8)) >= nqm) return;
  const KopLane l (nqm);
  const MixCoef K = p.coef[(size_t) 4 * (p.off[l.m1] + (l.live ? l.qr : 0)) + l.b];
  float x[C];
  sums<C> (p, l, 0, x);
  const float e[3] = {K.ex, K.ey, K.ez};
  Trans<V, float> own, other;
  transverse<V, float> (e, x, own);
  swap_trans<V, float> (own, other, 4);
  // P = A C - B S, Q = A S + B C
  float g[C];
  const float sg = l.w ? 1.f : -1.f;
  couple<V, float> (e, K.ya, sg * K.yb, K.yc, sg * K.yg, K.yh, K.ym, own, other, g);
  put_rows<C> (p, l, 0, g, s_mx);
}

// Unequal radii.  With a the target's radius and X, Xq the sums of x_j and a_j^2
// x_j, the weights of a pair are polynomials in a: the forward columns are X and
// Xq (2 c per function), the backward ones U, W, E by power of a
//   a    U              6 X, -k^2 Xq (A)
//   a^2  U, W, E        B and G at a = 0
//   a^3  U, W, E        -k^2 X (A); C, H and M at a = 0
//   a^4  U, E           G
//   a^5  E              M
// in this order (F: a and a^3; FT: a, a^2, a^3).  K.ya is the Ewald factor, K.yb
// and K.yc are k and k^2, K.yg the factor of G.
template <int V>
__global__ void __launch_bounds__ (KOP_T)
k_kop_poly (MixPlan p)
{
  constexpr int C = NComp<V>::value;
  __shared__ uint32_t s_mx[11][2];
  const int nqm = p.nqm[blockIdx.y];
  chain_next ();
  if ((int) (blockIdx.x * (KOP_T / 8)) >= nqm) return;
  const KopLane l (nqm);
  const MixCoef K = p.coef[(size_t) 4 * (p.off[l.m1] + (l.live ? l.qr : 0)) + l.b];
  const float e[3] = {K.ex, K.ey, K.ez};
  const float ax = K.ya, kk = K.yc, sg = l.w ? 1.f : -1.f, b3 = sg * 3.f * K.yb * ax, gk = sg * K.yb * K.yg;
  Trans<V, float> xo, xs, qo, qs;       // of X and Xq: this lane's sums, the other's
  {
    float x[C];
    sums<C> (p, l, 0, x);
    transverse<V, float> (e, x, xo);
    swap_trans<V, float> (xo, xs, 4);
    sums<C> (p, l, C, x);
    transverse<V, float> (e, x, qo);
    swap_trans<V, float> (qo, qs, 4);
  }
  float g[C], h[C];
  auto put = [&] (int first, auto n, int from) {
    constexpr int N = decltype (n)::value;
    float v[N];
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = g[N == 8 && q >= 3 ? q + 3 : from + q];
    put_rows<N> (p, l, first, v, s_mx);
  };
  using std::integral_constant;
  // a
#pragma unroll
  for (int d = 0; d < 3; d++) g[d] = ax * fmaf (-kk, qo.f[d], 6.f * xo.f[d]);
  put (0, integral_constant<int, 3> (), 0);
  if constexpr (V == V_F)
    {
#pragma unroll
      for (int d = 0; d < 3; d++) g[d] = -kk * ax * xo.f[d];
      put (3, integral_constant<int, 3> (), 0);
    }
  else
    {
      // a^2
      couple<V, float> (e, 0.f, b3, 0.f, 3.f * gk, 0.f, 0.f, xo, xs, g);
      if constexpr (V == V_FTS)
        {
          couple<V, float> (e, 0.f, 0.f, 0.f, -0.5f * kk * gk, 0.f, 0.f, qo, qs, h);
#pragma unroll
          for (int q = 0; q < C; q++) g[q] += h[q];
        }
      put (3, integral_constant<int, C> (), 0);
      // a^3
      couple<V, float> (e, -kk * ax, 0.f, 1.5f * kk * ax, 0.f, 1.5f * kk * ax, 3.f * kk * ax, xo, xs, g);
      if constexpr (V == V_FTS)
        {
          couple<V, float> (e, 0.f, 0.f, 0.f, 0.f, 0.f, -0.3f * kk * kk * ax, qo, qs, h);
#pragma unroll
          for (int q = 0; q < C; q++) g[q] += h[q];
        }
      put (C + 3, integral_constant<int, C> (), 0);
      if constexpr (V == V_FTS)
        {
          // a^4, a^5
          couple<V, float> (e, 0.f, 0.f, 0.f, -0.3f * kk * gk, 0.f, 0.f, xo, xs, g);
          put (25, integral_constant<int, 8> (), 0);
          couple<V, float> (e, 0.f, 0.f, 0.f, 0.f, 0.f, -0.3f * kk * kk * ax, xo, xs, g);
          put (33, integral_constant<int, 5> (), 6);
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
constexpr int START = 4;                // start and end of a CTA, in K tiles

// columns per tile: a multiple of 16 up to `most` that leaves the fewest unused
int
tile_cols (int ncol, int most)
{
  const int nt = (ncol + most - 1) / most;
  return (((ncol + nt - 1) / nt) + 15) / 16 * 16;
}

// time of a tile of tn columns, of one of 128: the build of A stays, B, the
// MMAs, the drain and the epilogue go with tn
double tile_time (int tn) { return (64.0 + tn) / 192.0; }

}  // namespace

// Column tiles and work items of the two GEMMs.  A column tile needs the
// quarters that its smallest |m1| uses (nqm): the forward has no item for row
// tiles past them, the backward's K ends there.  K is sliced, in units of 128,
// as evens out the SMs.
void
mix_plan_items (MixPlan &p, const std::vector<int> &nqm, std::vector<int4> &fwd,
                std::vector<int4> &bwd)
{
  p.mt = (p.np + TM - 1) / TM;
  const int kb = p.ldT / KB;
  p.tnf = tile_cols (p.ncolf, TN_MAX);
  p.nctf = (p.ncolf + p.tnf - 1) / p.tnf;
  std::vector<int> rf (p.nctf), rb;
  long long act = 0;
  for (int ct = 0; ct < p.nctf; ct++)
    {
      rf[ct] = (4 * nqm[col_m (ct * p.tnf, p.cf)] + TM - 1) / TM;
      act += rf[ct];
    }
  double best = -1;
  for (int ns = 1; ns <= std::min (16, kb); ns++)
    {
      const int per = (kb + ns - 1) / ns, used = (kb + per - 1) / per;
      // each slice is one more set of sums for the operator kernel
      const double t = (double) ((act * used + SMS - 1) / SMS) * (DK * per + START) + used / 4.0;
      if (best < 0 || t < best)
        {
          best = t;
          p.jper = per * KB;
          p.nsplit = used;
        }
    }
  p.ldf = p.nctf * p.tnf;
  fwd.clear ();
  for (int z = 0; z < p.nsplit; z++)
    for (int ct = 0; ct < p.nctf; ct++)
      for (int rt = 0; rt < rf[ct]; rt++) fwd.push_back (make_int4 (rt, ct, z, 0));
  p.nfitem = (int) fwd.size ();
  // backward: in a small system narrower tiles, more of them, end sooner (FTS N
  // = 200 48.6 -> 45.1 us a product, N = 600 61 -> 57.5); a larger one needs the
  // SMs that they take for the real space beside it (F N = 2048 65.3 -> 68.5)
  best = -1;
  int slice = 1;
  for (int most = TN_MAX; most >= (p.np <= 1024 ? 32 : TN_MAX); most /= 2)
    {
      const int tn = tile_cols (p.ncolb, most), nct = (p.ncolb + tn - 1) / tn;
      std::vector<int> sets (nct);
      for (int ct = 0; ct < nct; ct++) sets[ct] = (4 * nqm[col_m (ct * tn, p.cb)] + KB - 1) / KB;
      for (int s = 1; s <= std::max (1, sets[0]); s++)
        {
          const int l = (sets[0] + s - 1) / s;
          std::vector<int> len;
          long long sum = 0;
          for (int k : sets)
            {
              const int n = std::max (1, (k + l - 1) / l), d = DK * ((k + n - 1) / n);
              len.insert (len.end (), n, d);
              sum += (long long) n * (d + START);
            }
          if (s > 1 && len.size () > 64) break;
          // no schedule ends before the SMs' average
          if (best >= 0
              && (double) (sum * p.mt / SMS) * tile_time (tn) + len.size () / 24.0 >= best)
            continue;
          const double t = (double) makespan (len, p.mt, START) * tile_time (tn) + len.size () / 24.0;
          if (best < 0 || t < best)
            {
              best = t;
              slice = l;
              p.tnb = tn;
              p.nctb = nct;
              rb = sets;
            }
        }
    }
  p.ldb = p.nctb * p.tnb;
  bwd.clear ();
  for (int ct = 0; ct < p.nctb; ct++)
    {
      const int n = std::max (1, (rb[ct] + slice - 1) / slice);
      for (int z = 0; z < n; z++)
        {
          const int a = rb[ct] * z / n, b = rb[ct] * (z + 1) / n;
          bwd.push_back (make_int4 (ct, DK * a, DK * (b - a), 0));
        }
    }
  std::stable_sort (bwd.begin (), bwd.end (), [] (const int4 &a, const int4 &b) { return a.z > b.z; });
  p.nbitem = (int) bwd.size ();
}

int mix_poly_columns (int version) { return version == 0 ? 6 : (version == 1 ? 15 : 38); }
size_t mix_zf_bytes (const MixPlan &p) { return 2 * (size_t) ND * p.ncolf * p.ldT; }
size_t mix_wb_bytes (const MixPlan &p) { return 2 * (size_t) ND * p.ncolb * p.Rp; }
size_t mix_zs_floats (const MixPlan &p) { return (size_t) (p.ldT / KB) * p.ldf; }
size_t mix_ws_floats (const MixPlan &p) { return (size_t) (p.Rp / KB) * p.ldb; }

int
mix_maps (const MixPlan &p, MixMaps *m)
{
  int e = encode_planes_f16 (&m->zf, p.ZF, ND, p.ncolf, p.ldT, p.tnf);
  if (!e) e = encode_planes_f16 (&m->wb, p.WB, ND, p.ncolb, p.Rp, p.tnb);
  return e;
}

// the shared-memory opt-in is a per-device function attribute
static cudaError_t
gemm_attrs ()
{
  static int attr_dev = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess || attr_dev == dev) return e;
  if ((e = cudaFuncSetAttribute (k_sfac_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int) SMEM_DYN)) != cudaSuccess)
    return e;
  for (auto bp : {k_bp_gemm<false>, k_bp_gemm<true>})
    if ((e = cudaFuncSetAttribute (bp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) SMEM_DYN))
        != cudaSuccess)
      return e;
  attr_dev = dev;
  return cudaSuccess;
}

cudaError_t
launch_mix_prep (const MixPrep &a, cudaStream_t st)
{
  // fewer items a CTA while that leaves SMs idle
  const int items = a.p.M[0] + a.p.M[1] + a.p.M[2] + 3, tiles = a.p.ldT / PREP_P;
  const int g = std::max ((items + PREP_I - 1) / PREP_I, std::min (items, SMS / tiles));
  mk_prep_tc<<<dim3 (tiles, g), PREP_T, 0, st>>> (a);
  return cudaGetLastError ();
}

cudaError_t
launch_mix_forward (int version, const MixPlan &p, const MixMaps &m, int *status, cudaStream_t st,
                    Ctx *prof)
{
  cudaError_t e = gemm_attrs ();
  if (e != cudaSuccess) return e;
  e = launch_chained (k_sfac_gemm, p.nfitem, NT, SMEM_DYN, st, m.zf, p, status);
  if (e != cudaSuccess) return e;
  kmark (prof, st, "k_sfac_gemm");
  const dim3 g (p.nqp / (KOP_T / 8), p.M[0] + 1);
  if (p.rad)
    {
      if (version == 0) k_kop_poly<0><<<g, KOP_T, 0, st>>> (p);
      else if (version == 1) k_kop_poly<1><<<g, KOP_T, 0, st>>> (p);
      else k_kop_poly<2><<<g, KOP_T, 0, st>>> (p);
    }
  else if (version == 0) k_kop<0><<<g, KOP_T, 0, st>>> (p);
  else if (version == 1) k_kop<1><<<g, KOP_T, 0, st>>> (p);
  else k_kop<2><<<g, KOP_T, 0, st>>> (p);
  kmark (prof, st, "k_kop");
  return cudaGetLastError ();
}

cudaError_t
launch_mix_backward (const MixPlan &p, const MixMaps &m, int *status, cudaStream_t st, Ctx *prof)
{
  const cudaError_t e = launch_chained (p.rad ? k_bp_gemm<true> : k_bp_gemm<false>, dim3 (p.mt, p.nbitem),
                                        NT, SMEM_DYN, st, m.wb, p, status);
  // the profile's name of the back-projection of unequal radii is the same on
  // both paths: callers look for it
  kmark (prof, st, p.rad ? "mk_backproj_poly" : "k_bp_gemm");
  return e;
}

}  // namespace lsg
