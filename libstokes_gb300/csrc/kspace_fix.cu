// kspace_fix.cu -- the reciprocal Ewald sum as exact integer GEMMs on the
// tensor cores.
//
// A reciprocal vector is k = 2 pi (m1 / Lx, m2 / Ly, m3 / Lz) and every phase
// factor is a product of one function of x, y and z each.  In the basis of
// real functions f_0 = 1, f_(2m-1) = cos 2 pi m u, f_(2m) = sin 2 pi m u per
// axis (u the fractional coordinate) the sum is, with row r = (y function, z
// function) and column n = (x function mi, vector component q):
//
//   forward   F[n][r] = sum_j A[r][j] B[n][j],   A[r][j] = f_y(j) f_z(j),
//                                                B[n][j] = f_x(j) x_q(j)
//   operator  the four sign patterns of (|m1|, |m2|, |m3|): cosine and sine
//             sums C, S by a 2-bit Walsh-Hadamard transform of the eight
//             values, P, Q by the Ewald weights, G by the same transform back
//   backward  y_q(i) = sum_mi f_x(i) sum_r A[r][i] G[n][r]
//
// which is half the multiplications of the complex form (k and -k share the
// real products).
//
// Arithmetic.  FP64 runs at 1/64 of the FP32 rate here, the tensor cores
// multiply f16.  Every operand is therefore a fixed-point number cut into ND
// signed 8-bit digits, each an exact f16 integer (ND = 7: 55 fractional bits
// below the largest magnitude of its kind, where FP64 has 53 significant
// ones; |f| <= 1, x_q is scaled by a power of two per component and G by one
// per column, since G falls off with |m1| and the rounding of a column is set
// by its largest entry).
// Digit products are at most 2^14 and at most 7 x 128 of them meet in one
// accumulator, so the FP32 sums of the tensor core stay below 2^24 and are
// exact integers.  The products of digits i and j with i + j = g < ND share
// accumulator g; the dropped ones weigh less than the last digit.  Every 128
// values of K the accumulators are drained: groups 0 to 3 into 64-bit
// integers, the rest (below 2^-38 of full scale) into FP32.  The result
// carries the rounding of its inputs, about 2^-56 of full scale each, and
// none from the summation.
//
// Operands.  B comes from images of f16 digits by TMA.  A is kept as 64-bit
// digit strings [row][particle], made once per product and read by both
// GEMMs; the worker warps cut them into f16 digits in shared memory (per
// digit pair a byte permute, a mask and an f16x2 subtraction).  As f16 images
// A would be twice as large and needed in two orientations.
//
// Shared memory rows are 128 bytes: 32 K values of an even digit and of the
// next odd one side by side.  The rows of all even digits of B follow one
// another, so one MMA takes a digit of A against all of them (issue_tile).
// One MMA per digit pair (N = 64) took 78 clocks, 80 us of MMAs in the forward
// GEMM of FTS N = 1000: it reads 6 KB of shared memory for 32 clocks of tensor
// pipe.  Now a 16-wide K step is 13 MMAs that read 108 KB for 896 clocks.
#include <cuda_fp16.h>

#include <algorithm>
#include <vector>

#include "digit_gemm.cuh"
#include "ewald_device.cuh"
#include "fixk.h"
#include "gpu_engine.h"
#include "tc_umma.cuh"
#include "tma_host.h"

namespace lsg {
namespace {

using namespace dg;

// per precision: ND digits, operators in R
template <int ND> struct Cfg;
template <> struct Cfg<7> {
  using R = double;
  static constexpr int KT = 32;         // K values per tile
  static constexpr int TN = 64;         // columns per tile (7 accumulators: 448 TMEM columns)
  static constexpr int DK = 4;          // tiles per drain (K = 128)
};

// Tiles of 128-byte rows: KT = 64 values of one digit, or KT = 32 values of
// an even digit and the next one
template <int ND>
struct Geo {
  using C = Cfg<ND>;
  static constexpr int PAIR = 64 / C::KT;               // digits per row
  static constexpr int NP = (ND + PAIR - 1) / PAIR;     // planes
  static constexpr uint32_t A_PLANE = TM * 128;
  static constexpr uint32_t B_PLANE = C::TN * 128;
  static constexpr int NS = 2;                          // stages
  static constexpr uint32_t A_BYTES = NP * A_PLANE, B_BYTES = NP * B_PLANE;
  static constexpr uint32_t STAGE = A_BYTES + B_BYTES;
  static constexpr uint32_t SMEM = NS * STAGE + 1024;
  static constexpr int CPT = C::TN / 4;                 // accumulator columns per worker
  // byte offset of digit p in its row, after the plane's own offset
  static constexpr uint32_t part (int p) { return PAIR == 2 ? (uint32_t) (p & 1) * 64u : 0u; }
  static constexpr int plane (int p) { return p / PAIR; }
};

// element (digit p, row n, k) of an f16 image with `rows` rows of ld values
template <int ND>
__device__ __forceinline__ size_t
image_off (int p, size_t rows, size_t n, size_t ld, int k)
{
  using G = Geo<ND>;
  constexpr int KT = Cfg<ND>::KT;
  const size_t row = (G::plane (p) * rows + n) * ld * G::PAIR;
  return row + (size_t) (k / KT) * 64 + G::part (p) / 2 + k % KT;
}

// ---- fixed point ----------------------------------------------------------
// A table entry f (62 fractional bits) as hi 2^32 + lo with lo signed
struct Limbs {
  int hi, lo;
};
__device__ __forceinline__ Limbs
limbs (long long f)
{
  const int lo = (int) f;
  return Limbs {(int) (f >> 32) + (int) ((unsigned) lo >> 31), lo};
}

// f g as a biased string of 55 fractional bits: digit p is byte 6 - p minus
// 128 (the top one a 16-bit field).  Three 32 x 32 bit products; the dropped
// lo lo term is below 2^-61.
__device__ __forceinline__ long long
biased (Limbs f, Limbs g)
{
  const long long cross = (long long) f.hi * g.lo + (long long) f.lo * g.hi;
  const long long v = (long long) f.hi * g.hi + (cross >> 32);      // 60 fractional bits
  return (v + ((0x0080808080808080ll << 5) + 16)) >> 5;
}

// v 2^(frac - E) rounded to an integer, for |v| < 2^E: from the bits of v,
// since FP64 arithmetic and conversions run at 1/64 of the integer rate
__device__ __forceinline__ long long
to_fixed (double v, int E, int frac)
{
  const long long bits = __double_as_longlong (v);
  const int e = (int) (bits >> 52) & 0x7ff;
  long long m = bits & 0x000fffffffffffffll;
  if (e) m |= 0x0010000000000000ll;
  const int sh = 1075 - max (e, 1) - frac + E;          // >= 53 - frac
  if (sh > 54) m = 0;
  else if (sh > 0) m = (m + (1ll << (sh - 1))) >> sh;
  else m <<= -sh;
  return bits < 0 ? -m : m;
}

// the f16 pairs (digit of a, digit of b) of two biased strings, plane by plane
__device__ __forceinline__ uint32_t
f16_digits (uint32_t bytes)
{
  // 0x6400 + n is the f16 number 1024 + n
  const __half2 v = __hsub2 (*reinterpret_cast<__half2 *> (&bytes), __half2half2 (__ushort_as_half (0x6480)));
  return *reinterpret_cast<const uint32_t *> (&v);
}

__device__ __forceinline__ void
digits (long long a, long long b, uint32_t out[7])
{
  const uint32_t al = (uint32_t) a, ah = (uint32_t) ((unsigned long long) a >> 32);
  const uint32_t bl = (uint32_t) b, bh = (uint32_t) ((unsigned long long) b >> 32);
  auto pick = [] (uint32_t x, uint32_t y, uint32_t sel) {
    return f16_digits ((__byte_perm (x, y, sel) & 0x00FF00FFu) | 0x64006400u);
  };
  out[0] = f16_digits (__byte_perm (ah, bh, 0x7632) + 0x64006400u);
  out[1] = pick (ah, bh, 0x5511);
  out[2] = pick (ah, bh, 0x4400);
  out[3] = pick (al, bl, 0x7733);
  out[4] = pick (al, bl, 0x6622);
  out[5] = pick (al, bl, 0x5511);
  out[6] = pick (al, bl, 0x4400);
}

// exponent E with |v| < 2^E for every v whose high word (sign cleared) is at
// most hw; NaN and infinity: finite = false
__device__ __forceinline__ int
scale_exp (uint32_t hw, bool &finite)
{
  const int e = (int) (hw >> 20);
  finite = e != 2047;
  return e - 1022;
}

// v 2^(E - frac) as FP64, E the exponent of hw; NaN where an input was NaN or
// infinite, as a sum over it would be.  In integers, like to_fixed.
__device__ __forceinline__ double
from_fixed (long long v, uint32_t hw, int frac)
{
  bool finite;
  const int e = scale_exp (hw, finite) - frac;
  if (!finite) return __longlong_as_double (0x7ff8000000000000ll);
  const double d = int_to_double (v);
  // exponents far from the ends of the range: add e to the exponent field
  if (e > -1022 && e < 960) return v ? __longlong_as_double (__double_as_longlong (d) + ((long long) e << 52)) : 0.0;
  return scalbn (d, e);
}

__device__ __forceinline__ uint32_t
abs_hi (double v)
{
  return (uint32_t) __double2hiint (v) & 0x7fffffffu;
}

// ---- operand builders -----------------------------------------------------
// The A operand of a tile is built in two steps, so that the loads of the
// next tile are in flight while a worker waits for its stage: load() reads a
// thread's digit strings, store() cuts them and writes the stage.

// Forward: rows r0 .. r0 + 127, particles j0 .. j0 + 31.  Half a warp covers
// the 32 particles (two per lane) of four rows; the two halves of a warp write
// different halves of a 128-byte bank line (their rows differ by 4).
template <int ND>
struct BuildF {
  const long long *S;
  int ldT;
  longlong2 v[4];
  __device__ __forceinline__ BuildF (const FixPlan &p, int r0, int jb) : ldT (p.ldT)
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    S = (const long long *) p.S + (size_t) (r0 + 8 * warp + 4 * (lane >> 4)) * ldT + jb
        + 2 * (lane & 15);
  }
  __device__ __forceinline__ void load (int t)
  {
#pragma unroll
    for (int k = 0; k < 4; k++)
      v[k] = __ldg (reinterpret_cast<const longlong2 *> (S + (size_t) k * ldT + Cfg<ND>::KT * t));
  }
  __device__ __forceinline__ void store (unsigned char *stage) const
  {
    using G = Geo<ND>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jp = lane & 15;
#pragma unroll
    for (int k = 0; k < 4; k++)
      {
        const int r = 8 * warp + 4 * (lane >> 4) + k;
        uint32_t d[7];
        digits (v[k].x, v[k].y, d);
        // digits of odd number sit four chunks further
        unsigned char *o0 = stage + chunk_off (r, jp >> 2) + (jp & 3) * 4;
        unsigned char *o1 = stage + chunk_off (r, 4 + (jp >> 2)) + (jp & 3) * 4;
#pragma unroll
        for (int q = 0; q < ND; q++)
          *reinterpret_cast<uint32_t *> ((q & 1 ? o1 : o0) + G::plane (q) * G::A_PLANE) = d[q];
      }
  }
};

// Backward: particles i0 .. i0 + 127, one per lane, 32 rows, eight of them (16
// bytes per digit) per thread
template <int ND>
struct BuildB {
  const long long *S;
  int ldT, c;
  long long v[8];
  __device__ __forceinline__ BuildB (const FixPlan &p, int i0, int r0) : ldT (p.ldT)
  {
    c = threadIdx.x >> 7;
    S = (const long long *) p.S + (size_t) (r0 + 8 * c) * ldT + i0 + (threadIdx.x & 127);
  }
  __device__ __forceinline__ void load (int t)
  {
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = __ldg (S + (size_t) (t * Cfg<ND>::KT + u) * ldT);
  }
  __device__ __forceinline__ void store (unsigned char *stage) const
  {
    using G = Geo<ND>;
    uint32_t w[4][7];
#pragma unroll
    for (int u = 0; u < 4; u++) digits (v[2 * u], v[2 * u + 1], w[u]);
#pragma unroll
    for (int q = 0; q < ND; q++)
      *reinterpret_cast<uint4 *> (stage + G::plane (q) * G::A_PLANE
                                  + chunk_off (threadIdx.x & 127, (q & 1) * 4 + c))
        = make_uint4 (w[0][q], w[1][q], w[2][q], w[3][q]);
  }
};

// ---- GEMM roles -----------------------------------------------------------
// TMEM columns of accumulator group g: the even groups first, then the odd
template <int ND>
constexpr int
group_col (int g)
{
  return ((g & 1) * ((ND + 1) / 2) + g / 2) * Cfg<ND>::TN;
}

// the MMAs of one tile.  The even digits of B lie one after the other as rows
// of the tile, the odd ones likewise, and so do their groups in TMEM: one MMA
// of digit i of A with all even (or odd) digits j <= ND - 1 - i of B adds the
// products to groups i, i + 2, ... at once, with N up to 256.
template <int ND>
__device__ __forceinline__ void
issue_tile (uint32_t a, uint32_t tmem, bool first)
{
  using G = Geo<ND>;
  using C = Cfg<ND>;
  static_assert (G::PAIR == 2 && (ND + 1) / 2 * C::TN <= 256, "even digits in one MMA");
  const uint32_t b = a + G::A_BYTES;
#pragma unroll
  for (int k = 0; k < C::KT / 16; k++)
#pragma unroll
    for (int i = 0; i < ND; i++)
#pragma unroll
      for (int odd = 0; odd < 2; odd++)
        {
          const int nj = (ND - i + 1 - odd) / 2;        // digits j = odd, odd + 2, ...
          if (nj == 0) continue;
          umma::mma_f16 (tmem + (uint32_t) group_col<ND> (i + odd),
                         umma::smem_desc_sw128 (a + G::plane (i) * G::A_PLANE + G::part (i) + 32 * k),
                         umma::smem_desc_sw128 (b + G::part (odd) + 32 * k),
                         umma::idesc_f16 (TM, (uint32_t) (nj * C::TN)),
                         (first && i == 0 && k == 0) ? 0u : 1u);
        }
}

// running sums of one worker: CPT columns of one row.  Value of a column:
// (hi + lo) 2^-38; hi exact.
template <int ND> struct Acc;
template <> struct Acc<7> {
  static constexpr int CPT = Geo<7>::CPT;
  long long hi[CPT];
  float lo[CPT];
  uint32_t d;                           // TMEM address of its lanes and columns
  __device__ __forceinline__ void zero (uint32_t tmem)
  {
    d = tmem;
#pragma unroll
    for (int u = 0; u < CPT; u++) { hi[u] = 0; lo[u] = 0.f; }
  }
  __device__ __forceinline__ void take (int, int)
  {
    static_assert (CPT == 16, "one TMEM load per group");
    float f[2][16];
    umma::tmem_ld16_issue (d + group_col<7> (0), f[0]);
#pragma unroll
    for (int g = 0; g < 7; g++)
      {
        umma::tmem_ld_wait (f[g & 1]);
        if (g < 6) umma::tmem_ld16_issue (d + group_col<7> (g + 1), f[(g + 1) & 1]);
#pragma unroll
        for (int u = 0; u < 16; u++)
          {
            const float v = f[g & 1][u];
            if (g < 4) hi[u] += (long long) __float2int_rn (v) * (1 << (8 * (3 - g)));
            else lo[u] = fmaf (v, 1.0f / (float) (1u << (8 * (g - 3))), lo[u]);
          }
      }
  }
  // column u in units of 2^-fu, fu >= 38
  __device__ __forceinline__ long long fixed (int u, int fu) const
  {
    const int whole = __float2int_rn (lo[u]);
    const float rest = (lo[u] - (float) whole) * (float) (1u << (fu - 38));
    return ((hi[u] + whole) << (fu - 38)) + __float2int_rn (rest);
  }
};

// TMEM address of a worker's lanes and columns
__device__ __forceinline__ uint32_t
worker_tmem (uint32_t tmem, int cpt)
{
  const int warp = threadIdx.x >> 5;
  return tmem + ((uint32_t) ((warp & 3) * 32) << 16) + (uint32_t) ((warp >> 2) * cpt);
}

__device__ __forceinline__ int
col_m (const FixPlan &p, int n)
{
  return (n / p.c + 1) / 2;              // |m1| of column n
}

// first column of component q, of c, in the tile that starts at column n0
__device__ __forceinline__ int
first_col (int c, int n0, int q)
{
  return (q + c - n0 % c) % c;
}

constexpr int NOT_FINITE = 1 << 20;

// forward: a CTA takes one item (row tile, column tile, particle slice) and
// writes F[slice][column][row]; lanes are consecutive rows, so the stores
// coalesce
template <int ND>
__global__ void __launch_bounds__ (NT, 1)
k_fix_fwd (const __grid_constant__ CUtensorMap tmB, FixPlan p, int *status)
{
  using C = Cfg<ND>;
  using G = Geo<ND>;
  extern __shared__ unsigned char dsm[];
  __shared__ Sync s;
  const int4 it = p.fitem[blockIdx.x];
  const int r0 = it.x * TM, n0 = it.y * C::TN;
  unsigned char *smem = align1k (dsm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jb = it.z * p.jper, je = min (p.ldT, jb + p.jper);
  const int ntiles = je > jb ? (je - jb + C::KT - 1) / C::KT : 0;
  cta_setup (s);
  const uint32_t tmem = s.tslot;
  Acc<ND> acc;
  acc.zero (worker_tmem (tmem, G::CPT));
  BuildF<ND> build (p, r0, jb);
  const BTiles bt {&tmB, G::PAIR * jb, G::PAIR * C::KT, n0, G::A_BYTES, G::B_BYTES};
  if (run_tiles<C::DK, 1, G::NS> (s, smem, ntiles, G::STAGE, bt, p.stall, build, acc,
                                  [=] (uint32_t a, int, bool first) { issue_tile<ND> (a, tmem, first); }))
    {
      const int r = r0 + (warp & 3) * 32 + lane, c0 = n0 + (warp >> 2) * G::CPT;
      long long *F = (long long *) p.F + (size_t) it.z * p.ncol * p.Rp + r;
#pragma unroll
      for (int u = 0; u < G::CPT; u++)
        if (c0 + u < p.ncol) F[(size_t) (c0 + u) * p.Rp] = acc.fixed (u, p.fu);
    }
  cta_finish (s, tmem, status);
}

// backward: a CTA takes 128 particles and one item (column tile, first K
// tile, K tiles), the item number is the slot of its partial y.  The sums H are
// parked in the freed stages and reduced over the x functions of the tile in
// 128-bit integers (an FP64 operation on the 128 x 64 tile takes the FP64 pipe
// 4096 clocks, a 64 x 64 bit product of integers about a tenth): the columns'
// different units 2^E come in as a right shift of the table entry.
//
// DENSE: the moments of 128 pairs, columns and rows by class (FixClass).
template <int ND, bool DENSE>
__global__ void __launch_bounds__ (NT, 1)
k_fix_bwd (const __grid_constant__ CUtensorMap tmB, const __grid_constant__ FixPlan p, int *status)
{
  using C = Cfg<ND>;
  using G = Geo<ND>;
  constexpr int HLD = C::TN + 1;
  constexpr uint32_t H_LO = TM * HLD * sizeof (long long);
  constexpr uint32_t X_OFF = H_LO + TM * HLD * sizeof (float);
  // the parked sums and the x functions of 64 columns (a class of one
  // component: 64)
  static_assert (X_OFF + 64 * TM * sizeof (long long) <= G::NS * G::STAGE, "parked tile");
  extern __shared__ unsigned char dsm[];
  __shared__ Sync s;
  __shared__ int s_exp[C::TN], s_top[16];
  unsigned char *smem = align1k (dsm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int4 it = p.bitem[blockIdx.y];
  const int i0 = blockIdx.x * TM, n0 = it.x * C::TN;
  // columns n of the tile are column nb + n of the list (x function or |m1|,
  // component), nc components each
  int cl = 0, nb = n0, nc = p.c, ncol = p.ncol, row0 = 0;
  const unsigned *mx = p.mx;
  if constexpr (DENSE)
    {
      while (cl < 3 && n0 >= p.cls[cl + 1].col0) cl++;
      nb = n0 - p.cls[cl].col0;
      nc = p.cls[cl].nc;
      ncol = p.cls[cl].ncol;
      row0 = p.cls[cl].row0;
      mx += cl * fix_mx_words (p);
    }
  const int ne = min (C::TN, ncol - nb);
  if ((int) threadIdx.x < ne)
    {
      const int n = nb + threadIdx.x, m1 = DENSE ? n / nc : (n / nc + 1) / 2;
      bool finite;
      const int E = scale_exp (mx[16 * (m1 + 1) + n % nc], finite);
      s_exp[threadIdx.x] = finite ? E : NOT_FINITE;
    }
  const int tb = it.y, ntiles = it.z;
  cta_setup (s);
  const uint32_t tmem = s.tslot;
  // the largest unit of each component
  if ((int) threadIdx.x < nc)
    {
      int top = -2000;
      for (int n = first_col (nc, nb, threadIdx.x); n < ne; n += nc) top = max (top, s_exp[n]);
      s_top[threadIdx.x] = top;
    }
  {
    Acc<ND> acc;
    acc.zero (worker_tmem (tmem, G::CPT));
    BuildB<ND> build (p, i0, row0 + tb * C::KT);
    const BTiles bt {&tmB, G::PAIR * tb * C::KT, G::PAIR * C::KT, n0, G::A_BYTES, G::B_BYTES};
    if (run_tiles<C::DK, 1, G::NS> (s, smem, ntiles, G::STAGE, bt, p.stall, build, acc,
                                    [=] (uint32_t a, int, bool first) {
                                      issue_tile<ND> (a, tmem, first);
                                    }))
      {
        // the last set is drained, so every build, load and MMA is done and
        // the stages are free
        const int o = ((warp & 3) * 32 + lane) * HLD + (warp >> 2) * G::CPT;
        long long *Hi = reinterpret_cast<long long *> (smem) + o;
        float *Lo = reinterpret_cast<float *> (smem + H_LO) + o;
#pragma unroll
        for (int u = 0; u < G::CPT; u++)
          {
            Hi[u] = acc.hi[u];
            Lo[u] = acc.lo[u];
          }
      }
  }
  __syncthreads ();
  if (!s.err)
    {
      const long long *Hi = reinterpret_cast<const long long *> (smem);
      const float *Lo = reinterpret_cast<const float *> (smem + H_LO);
      // the x functions of the tile's columns, in one pass (a load per term
      // would wait for L2 every time)
      const int f0 = nb / nc, nf = (nb + ne - 1) / nc - f0 + 1;
      long long *X = reinterpret_cast<long long *> (smem + X_OFF);
      const long long *T = (const long long *) p.T;
      // DENSE: function k of |m1| = f0 + k / 2 where a class has both parities
      const int odd = DENSE ? p.cls[cl].odd : 0;
      const bool both = DENSE && odd != 0 && odd != (1 << nc) - 1;
      const int np2 = both ? 2 : 1;
      for (int e = threadIdx.x; e < np2 * nf * TM; e += NT)
        {
          int f = f0 + e / TM;
          if constexpr (DENSE)
            {
              const int m1 = f0 + (e / TM) / np2, sine = both ? (e / TM) & 1 : odd & 1;
              f = sine ? (m1 ? 2 * m1 : p.zero) : (m1 ? 2 * m1 - 1 : 0);
            }
          X[e] = T[(size_t) f * p.ldT + i0 + e % TM];
        }
      __syncthreads ();
      for (int e = threadIdx.x; e < TM * nc; e += NT)
        {
          const int q = e / TM, r = e - q * TM, i = i0 + r;
          if (!DENSE && i >= p.np) continue;
          const int top = s_top[q];
          __int128 y = 0;
          float yl = 0.f;
          for (int n = first_col (nc, nb, q); n < ne; n += nc)
            {
              const int sh = top - s_exp[n];
              if (sh > 62) continue;              // below the last bit
              const int k = DENSE ? np2 * ((nb + n) / nc - f0) + (both ? odd >> q & 1 : 0)
                                  : (nb + n) / nc - f0;
              const long long f = X[k * TM + r] >> sh;
              y += (__int128) f * Hi[r * HLD + n];
              yl = fmaf ((float) (int) (f >> 32), Lo[r * HLD + n], yl);
            }
          // y: 62 + 38 fractional bits, yl: 30 + 38
          const double v = (double) (long long) (y >> 64) * 0x1p-36
                           + (double) (unsigned long long) y * 0x1p-100 + (double) yl * 0x1p-68;
          double *o = (double *) p.yp;
          if constexpr (DENSE) o += ((size_t) it.w * 16 + q) * p.ldT + i;
          else o += ((size_t) blockIdx.y * p.np + i) * p.c + q;
          *o = top == NOT_FINITE ? __longlong_as_double (0x7ff8000000000000ll) : scalbn (v, top);
        }
    }
  cta_finish (s, tmem, status);
}

// ---- tables and images ----------------------------------------------------
constexpr int TAB_P = 32, TAB_R = 4;

// Function table, one (axis, m) pair of rows (cos, sin) per warp and 32
// particles.  The fractional coordinate is a 64-bit fixed-point number (the
// quotient's rounding error added back), so m u mod 1 is an exact integer
// product.  The blocks of the first group also take the maxima of |x_q|; a
// position that is not finite makes them NaN, which every result inherits.
__global__ void __launch_bounds__ (TAB_P * TAB_R)
k_fix_tables (FixPlan p, const double *pos, const double *x)
{
  __shared__ unsigned long long s_u[3][TAB_P];
  __shared__ unsigned s_mx[16];
  const int t = threadIdx.x, jb = blockIdx.x * TAB_P;
  long long *T = (long long *) p.T;
  if (t < 16) s_mx[t] = 0u;
  __syncthreads ();
  if (t < 3 * TAB_P)
    {
      const int d = t / TAB_P, jl = t % TAB_P, j = jb + jl;
      unsigned long long u = 0;
      if (j < p.np)
        {
          const double v = pos[3 * j + d], f = v * p.il[d];
          const double rest = fma (-f, p.l[d], v) * p.il[d];
          if (!(fabs (f) < 1e300) && blockIdx.y == 0) s_mx[0] = 0x7ff80000u;
          u = __double2ull_rz ((f - floor (f)) * 18446744073709551616.0)
              + (unsigned long long) __double2ll_rn (rest * 18446744073709551616.0);
        }
      s_u[d][jl] = u;
    }
  __syncthreads ();
  if (blockIdx.y == 0 && t < TAB_P && jb + t < p.np)
    {
      // the coordinates for the real space
      const unsigned long long ux = s_u[0][t], uy = s_u[1][t], uz = s_u[2][t];
      p.q[jb + t] = make_uint4 ((unsigned) (ux >> 32), (unsigned) (uy >> 32), (unsigned) (uz >> 32), 0u);
      ulonglong2 *o = reinterpret_cast<ulonglong2 *> (p.u) + 2 * (size_t) (jb + t);
      o[0] = make_ulonglong2 (ux, uy);
      o[1] = make_ulonglong2 (uz, 0ull);
    }
  const int item = blockIdx.y * TAB_R + t / TAB_P, j = jb + t % TAB_P;
  const int n0 = p.M[0] + 1, n1 = n0 + p.M[1] + 1, n2 = n1 + p.M[2] + 1;
  if (item < n2 && j < p.np)
    {
      const int d = item < n0 ? 0 : (item < n1 ? 1 : 2);
      const int m = item - (d == 0 ? 0 : (d == 1 ? n0 : n1));
      const long long ph = (long long) ((unsigned long long) m * s_u[d][t % TAB_P]);
      double sn, cs;
      sincospi ((double) ph * 1.0842021724855044e-19, &sn, &cs);     // 2^-63
      long long *row = T + (size_t) ((d == 0 ? 0 : (d == 1 ? p.oy : p.oz)) + (m ? 2 * m - 1 : 0)) * p.ldT;
      const double one = 4611686018427387904.0;                      // 2^62
      row[j] = __double2ll_rn (cs * one);
      if (m) row[p.ldT + j] = __double2ll_rn (sn * one);
    }
  if (blockIdx.y) return;
  for (int e = t; e < TAB_P * p.c; e += TAB_P * TAB_R)
    if ((size_t) jb * p.c + e < (size_t) p.np * p.c)
      atomicMax (&s_mx[e % p.c], abs_hi (x[(size_t) jb * p.c + e]));
  __syncthreads ();
  if (t < p.c) atomicMax (p.mx + t, s_mx[t]);
}

// Digit strings of the rows, S[row][particle] = f_y f_z: a thread makes the
// four rows of a quarter for two particles
__global__ void __launch_bounds__ (128)
k_fix_strings (FixPlan p)
{
  const int j2 = blockIdx.x * 32 + (threadIdx.x & 31), qd = blockIdx.y * 4 + (threadIdx.x >> 5);
  const longlong2 *T = (const longlong2 *) p.T;
  const int4 f = p.quart[qd];
  const size_t ld = p.ldT / 2;
  const longlong2 y[2] = {T[f.x * ld + j2], T[f.y * ld + j2]};
  const longlong2 z[2] = {T[f.z * ld + j2], T[f.w * ld + j2]};
  longlong2 *o = (longlong2 *) p.S + (size_t) 4 * qd * ld + j2;
#pragma unroll
  for (int b = 0; b < 4; b++)
    o[b * ld] = make_longlong2 (biased (limbs (y[b >> 1].x), limbs (z[b & 1].x)),
                                biased (limbs (y[b >> 1].y), limbs (z[b & 1].y)));
}

// Forward image: digits of f_x(j) x_q(j), 64 particles and IMG_M x functions
// per block, eight particles (16 bytes per plane) per thread
constexpr int IMG_M = 4;

__global__ void __launch_bounds__ (128)
k_fix_image (FixPlan p, const double *x)
{
  __shared__ long long s_x[11][64];
  const int t = threadIdx.x, jb = blockIdx.x * 64;
  for (int e = t; e < 64 * p.c; e += 128)
    {
      const int jl = e / p.c, q = e - jl * p.c;
      bool finite;
      const int E = scale_exp (p.mx[q], finite);
      s_x[q][jl] = jb + jl < p.np && finite ? to_fixed (x[(size_t) jb * p.c + e], E, 62) : 0ll;
    }
  __syncthreads ();
  if (blockIdx.y == 0)
    {
      // FP32 copy for the far pairs of the real space, in units of the largest
      // component (components that are not finite: their couplings are not,
      // already from the reciprocal part)
      int top = -2000;
      for (int q = 0; q < p.c; q++)
        {
          bool finite;
          const int E = scale_exp (p.mx[q], finite);
          if (finite) top = max (top, E);
        }
      for (int e = t; e < 64 * p.c; e += 128)
        {
          const int jl = e / p.c, q = e - jl * p.c;
          bool finite;
          scale_exp (p.mx[q], finite);
          if (jb + jl < p.np)
            p.xf[(size_t) (jb + jl) * XF_LD + q]
              = finite ? (float) scalbn (x[(size_t) jb * p.c + e], -top) : 0.f;
        }
      if (t == 0 && blockIdx.x == 0) *p.xtop = top;
    }
  const long long *T = (const long long *) p.T;
  for (int e = t; e < IMG_M * p.c * 8; e += 128)
    {
      const int j8 = e & 7, q = (e >> 3) % p.c, mi = blockIdx.y * IMG_M + (e >> 3) / p.c;
      if (mi >= p.nmi) continue;
      const long long *f = T + (size_t) mi * p.ldT + jb + 8 * j8;
      uint32_t w[4][7];
#pragma unroll
      for (int k = 0; k < 4; k++)
        {
          const longlong2 v = *reinterpret_cast<const longlong2 *> (f + 2 * k);
          digits (biased (limbs (v.x), limbs (s_x[q][8 * j8 + 2 * k])),
                  biased (limbs (v.y), limbs (s_x[q][8 * j8 + 2 * k + 1])), w[k]);
        }
#pragma unroll
      for (int d = 0; d < 7; d++)
        *reinterpret_cast<uint4 *> ((__half *) p.ZF
                                    + image_off<7> (d, p.ncol, mi * p.c + q, p.ldT, jb + 8 * j8))
          = make_uint4 (w[0][d], w[1][d], w[2][d], w[3][d]);
    }
}

constexpr int KOP_T = 32;               // threads per CTA: 4 octant points (FP64-bound: small CTAs
                                        // even out the SMs)

// Operators: eight lanes per octant point.  Lane (w, b): b = 2 p2 + p3 names
// the row of the quarter, and after the transform the sign pattern (s2, s3) =
// (1 - 2 (b >> 1), 1 - 2 (b & 1)); w = 0 carries the cosine sums C and makes
// P, w = 1 the sine sums S and makes Q.  Row b enters C with its cosine column
// for b = 0, 3 and its sine column for b = 1, 2, and S with the other one; G
// goes back the same way, so every lane reads and writes one column set.
template <int ND, int V>
__global__ void __launch_bounds__ (KOP_T)
k_fix_kop (FixPlan p)
{
  using R = typename Cfg<ND>::R;
  constexpr int C = NComp<V>::value;
  const int m1 = blockIdx.y, b = threadIdx.x & 3, w = (threadIdx.x >> 2) & 1;
  const int nqm = p.nqm[m1];
  if ((int) (blockIdx.x * (KOP_T / 8)) >= nqm) return;
  const int qr = blockIdx.x * (KOP_T / 8) + threadIdx.x / 8;
  const bool live = qr < nqm;
  const int row = 4 * (live ? qr : 0) + b;
  const bool sine = (b == 0 || b == 3) == (w == 1);     // this lane's columns
  const bool neg = b == 3 || (w == 0 && b != 0);        // and their sign
  const bool have = live && !(sine && m1 == 0);
  const int col = (sine ? 2 * m1 : (m1 ? 2 * m1 - 1 : 0)) * C;
  long long f[C];
#pragma unroll
  for (int q = 0; q < C; q++) f[q] = 0;
  if (have)
#pragma unroll 2
    for (int s = 0; s < p.nsplit; s++)
      {
        const long long *F = (const long long *) p.F + ((size_t) s * p.ncol + col) * p.Rp + row;
#pragma unroll
        for (int q = 0; q < C; q++) f[q] += F[(size_t) q * p.Rp];
      }
  R x[C];
#pragma unroll
  for (int q = 0; q < C; q++)
    x[q] = (R) from_fixed (walsh4 (neg ? -f[q] : f[q], b), p.mx[q], p.fu);
  const FixCoef K = p.coef[(size_t) 4 * (p.off[m1] + (live ? qr : 0)) + b];
  const R e[3] = {(R) K.ex, (R) K.ey, (R) K.ez};
  Trans<V, R> own, other;
  transverse<V, R> (e, x, own);
  swap_trans<V, R> (own, other, 4);
  // P = A C - B S, Q = A S + B C
  R g[C];
  const R sg = w ? R (1) : R (-1);
  couple<V, R> (e, (R) K.ya, sg * (R) K.yb, (R) K.yc, sg * (R) K.yg, (R) K.yh, (R) K.ym, own, other, g);
  R *G = (R *) p.G + (size_t) col * p.Rp + row;
#pragma unroll
  for (int q = 0; q < C; q++)
    {
      const R v = walsh4 (g[q], b);
      uint32_t mx = 0u;
      if (have)
        {
          G[(size_t) q * p.Rp] = neg ? -v : v;
          mx = abs_hi ((double) v);
        }
      mx = __reduce_max_sync (0xffffffffu, mx);
      if ((threadIdx.x & 31) == 0 && mx) atomicMax (p.mx + 16 * (m1 + 1) + q, mx);
    }
}

// Backward image: digits of G, eight rows per thread
template <bool DENSE>
__global__ void __launch_bounds__ (128)
k_fix_gimage (const __grid_constant__ FixPlan p)
{
  const int n = blockIdx.y, r8 = blockIdx.x * 128 + threadIdx.x;
  int m1, rows;
  const unsigned *mx = p.mx;
  if constexpr (DENSE)
    {
      int cl = 0;
      while (cl < 3 && n >= p.cls[cl + 1].col0) cl++;
      const int nl = n - p.cls[cl].col0, nc = p.cls[cl].nc;
      if (nl >= p.cls[cl].ncol) return;
      m1 = nl / nc;
      rows = 4 * p.nqm[p.cls[cl].nq0 + m1];
      mx += cl * fix_mx_words (p) + 16 * (m1 + 1) + nl % nc;
    }
  else
    {
      m1 = col_m (p, n);
      rows = 4 * p.nqm[m1];
      mx += 16 * (m1 + 1) + n % p.c;
    }
  if (8 * r8 >= rows) return;
  bool finite;
  const int E = scale_exp (*mx, finite);
  const double *g = (const double *) p.G + (size_t) n * p.Rp + 8 * r8;
  uint32_t w[4][7];
#pragma unroll
  for (int k = 0; k < 4; k++)
    {
      const double2 v = *reinterpret_cast<const double2 *> (g + 2 * k);
      const long long bias = 0x0080808080808080ll;
      digits ((finite ? to_fixed (v.x, E, 55) : 0ll) + bias,
              (finite ? to_fixed (v.y, E, 55) : 0ll) + bias, w[k]);
    }
#pragma unroll
  for (int d = 0; d < 7; d++)
    *reinterpret_cast<uint4 *> ((__half *) p.WB + image_off<7> (d, p.ncol, n, p.Rp, 8 * r8))
      = make_uint4 (w[0][d], w[1][d], w[2][d], w[3][d]);
}

// ---- dense builder --------------------------------------------------------
// f g with 62 fractional bits, both with 62
__device__ __forceinline__ long long
mul62 (Limbs f, Limbs g)
{
  const long long cross = (long long) f.hi * g.lo + (long long) f.lo * g.hi;
  return (((long long) f.hi * g.hi) << 2) + (cross >> 30);
}

// Function table of the displacements r_j - r_i of an 8 x 8 tile of pairs, by
// the addition theorem from the functions of the particles in integers: a
// thread makes the functions of one pair for one (axis, m) in four.  (sincospi
// of every pair would be 60 FP64 instructions a value.)
constexpr int PT = 64;                  // pairs of a tile
__global__ void __launch_bounds__ (4 * PT)
k_fix_pair_tables (const __grid_constant__ FixPlan a, const __grid_constant__ FixPlan p,
                   const int2 *tile)
{
  const int2 ij = tile[blockIdx.x];
  const int t = threadIdx.x & (PT - 1);
  const int i = 8 * ij.x + (t >> 3), j = 8 * ij.y + (t & 7);
  const long long *A = (const long long *) a.T;
  long long *T = (long long *) p.T + (size_t) blockIdx.x * PT + t;
  const int n0 = p.M[0] + 1, n1 = n0 + p.M[1] + 1, n2 = n1 + p.M[2] + 1;
  for (int item = blockIdx.y * 4 + (threadIdx.x >> 6); item < n2; item += 4 * gridDim.y)
    {
      const int d = item < n0 ? 0 : (item < n1 ? 1 : 2);
      const int m = item - (d == 0 ? 0 : (d == 1 ? n0 : n1));
      const int row = (d == 0 ? 0 : (d == 1 ? p.oy : p.oz)) + (m ? 2 * m - 1 : 0);
      if (m == 0)
        {
          T[(size_t) row * p.ldT] = 1ll << 62;
          continue;
        }
      const long long *r = A + (size_t) row * a.ldT;
      const Limbs ci = limbs (r[i]), si = limbs (r[a.ldT + i]);
      const Limbs cj = limbs (r[j]), sj = limbs (r[a.ldT + j]);
      T[(size_t) row * p.ldT] = mul62 (cj, ci) + mul62 (sj, si);
      T[(size_t) (row + 1) * p.ldT] = mul62 (sj, ci) - mul62 (cj, si);
    }
}

template <int ND, int V>
cudaError_t
kop_v (const FixPlan &p, cudaStream_t st)
{
  k_fix_kop<ND, V><<<dim3 (8 * p.nqp / KOP_T, p.M[0] + 1), KOP_T, 0, st>>> (p);
  return cudaGetLastError ();
}

// the shared-memory opt-in is a per-device function attribute
cudaError_t
gemm_attrs ()
{
  static int attr_dev = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);
  if (e != cudaSuccess || attr_dev == dev) return e;
  if ((e = cudaFuncSetAttribute (k_fix_fwd<7>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int) Geo<7>::SMEM)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute (k_fix_bwd<7, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int) Geo<7>::SMEM)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute (k_fix_bwd<7, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int) Geo<7>::SMEM)) != cudaSuccess)
    return e;
  attr_dev = dev;
  return cudaSuccess;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
size_t fix_bytes_T (int, const FixPlan &p) { return sizeof (long long) * (size_t) p.nT * p.ldT; }
size_t
fix_bytes_F (int, const FixPlan &p)
{
  return sizeof (long long) * (size_t) p.nsplit * p.ncol * p.Rp;
}
size_t fix_bytes_G (int, const FixPlan &p) { return sizeof (double) * (size_t) p.ncol * p.Rp; }
size_t fix_bytes_S (int, const FixPlan &p) { return sizeof (long long) * (size_t) p.Rp * p.ldT; }
static size_t image_planes () { return (size_t) Geo<7>::NP * Geo<7>::PAIR; }
size_t fix_bytes_ZF (int, const FixPlan &p) { return 2 * image_planes () * p.ncol * p.ldT; }
size_t fix_bytes_WB (int, const FixPlan &p) { return 2 * image_planes () * p.ncol * p.Rp; }
size_t
fix_bytes_yp (int, const FixPlan &p)
{
  return sizeof (double) * (size_t) p.nbitem * p.np * p.c;
}

// The time of a set of CTAs (their K tiles, longest first) on one CTA per SM,
// in K tiles; a CTA's start and end cost about START tiles (measured: a
// 4-tile forward CTA takes as long as 7 tiles of a long one).
constexpr int START = 3;               // start and end of a CTA, in K tiles

// backward items (column tile, first K tile, K tiles) from the K tiles of each
// column tile, for mt tiles of 128 particles: slices of about equal length
static void
slice_rows (const std::vector<int> &tiles, int mt, std::vector<int4> &items)
{
  long long best = -1;
  int slice = 1;
  const int most = *std::max_element (tiles.begin (), tiles.end ());
  for (int s = 1; s <= 24; s++)
    {
      const int l = std::max (1, (most + s - 1) / s);
      if (s > 1 && l < 4) break;
      std::vector<int> len;
      for (int k : tiles)
        {
          const int n = std::max (1, (k + l - 1) / l);
          for (int z = 0; z < n; z++) len.push_back ((k + n - 1) / n);
        }
      if (s > 1 && len.size () > 96) break;
      const long long t = makespan (len, mt, START);
      if (best < 0 || t < best)
        {
          best = t;
          slice = l;
        }
    }
  items.clear ();
  for (size_t ct = 0; ct < tiles.size (); ct++)
    {
      const int k = tiles[ct], n = std::max (1, (k + slice - 1) / slice);
      for (int z = 0; z < n; z++)
        {
          const int a = (int) ((long long) k * z / n), b = (int) ((long long) k * (z + 1) / n);
          items.push_back (make_int4 ((int) ct, a, b - a, 0));
        }
    }
  std::stable_sort (items.begin (), items.end (), [] (const int4 &a, const int4 &b) { return a.z > b.z; });
}

// Work items of the two GEMMs.  A column tile needs the quarters that its
// smallest |m1| uses (nqm): the forward has no item for row tiles past them,
// the backward's K ends there.  K is sliced as evens out the SMs.
void
fix_plan_items (int, FixPlan &p, const std::vector<int> &nqm, std::vector<int4> &fwd,
                std::vector<int4> &bwd)
{
  using C = Cfg<7>;
  p.nct = (p.ncol + C::TN - 1) / C::TN;
  p.mt = (p.np + TM - 1) / TM;
  std::vector<int> rows (p.nct);
  long long act = 0;
  for (int ct = 0; ct < p.nct; ct++)
    {
      rows[ct] = 4 * nqm[(ct * C::TN / p.c + 1) / 2];
      act += (rows[ct] + TM - 1) / TM;
    }
  // forward: the same number of particle slices for every tile (the operator
  // kernel adds them), of at least 128 particles
  long long best = -1;
  const int kt = p.ldT / C::KT;
  for (int ns = 1; ns <= std::min (16, p.ldT / 128); ns++)
    {
      const int per = (kt + ns - 1) / ns, used = (kt + per - 1) / per;
      const long long t = (act * used + SMS - 1) / SMS * (per + START);
      if (best < 0 || t < best)
        {
          best = t;
          p.jper = per * C::KT;
          p.nsplit = used;
        }
    }
  fwd.clear ();
  for (int z = 0; z < p.nsplit; z++)
    for (int ct = 0; ct < p.nct; ct++)
      for (int rt = 0; rt * TM < rows[ct]; rt++) fwd.push_back (make_int4 (rt, ct, z, 0));
  p.nfitem = (int) fwd.size ();
  for (int &r : rows) r = (r + C::KT - 1) / C::KT;
  slice_rows (rows, p.mt, bwd);
  p.nbitem = (int) bwd.size ();
  // |F| <= np in units of its component, and the operators add four of them
  int lg = 0;
  while ((1ll << lg) < p.ldT) lg++;
  p.fu = 60 - lg;
}

int
fix_maps (int, const FixPlan &p, FixMaps *m)
{
  using G = Geo<7>;
  int e = encode_planes_f16 (&m->zf, p.ZF, G::NP, p.ncol, (size_t) G::PAIR * p.ldT, Cfg<7>::TN);
  if (!e) e = encode_planes_f16 (&m->wb, p.WB, G::NP, p.ncol, (size_t) G::PAIR * p.Rp, Cfg<7>::TN);
  return e;
}

cudaError_t
launch_fix_tables (int, const FixPlan &p, const double *pos, const double *x, cudaStream_t st,
                   Ctx *prof)
{
  const int items = p.M[0] + p.M[1] + p.M[2] + 3;
  k_fix_tables<<<dim3 ((p.np + TAB_P - 1) / TAB_P, (items + TAB_R - 1) / TAB_R), TAB_P * TAB_R, 0,
                 st>>> (p, pos, x);
  kmark (prof, st, "k_fix_tables");
  k_fix_strings<<<dim3 (p.ldT / 64, p.nqp / 4), 128, 0, st>>> (p);
  kmark (prof, st, "k_fix_strings");
  k_fix_image<<<dim3 (p.ldT / 64, (p.nmi + IMG_M - 1) / IMG_M), 128, 0, st>>> (p, x);
  kmark (prof, st, "k_fix_image");
  return cudaGetLastError ();
}

cudaError_t
launch_fix_forward (int, int version, const FixPlan &p, const FixMaps &m, int *status,
                    cudaStream_t st, Ctx *prof)
{
  cudaError_t e = gemm_attrs ();
  if (e != cudaSuccess) return e;
  k_fix_fwd<7><<<p.nfitem, NT, Geo<7>::SMEM, st>>> (m.zf, p, status);
  kmark (prof, st, "k_fix_fwd");
  e = version == 0 ? kop_v<7, 0> (p, st) : (version == 1 ? kop_v<7, 1> (p, st) : kop_v<7, 2> (p, st));
  kmark (prof, st, "k_fix_kop");
  return e;
}

cudaError_t
launch_fix_backward (int, int, const FixPlan &p, const FixMaps &m, int *status, cudaStream_t st,
                     Ctx *prof)
{
  k_fix_gimage<false><<<dim3 ((p.Rp / 8 + 127) / 128, p.ncol), 128, 0, st>>> (p);
  kmark (prof, st, "k_fix_gimage");
  k_fix_bwd<7, false><<<dim3 (p.mt, p.nbitem), NT, Geo<7>::SMEM, st>>> (m.wb, p, status);
  kmark (prof, st, "k_fix_bwd");
  return cudaGetLastError ();
}

// ---------------------------------------------------------------------------
// dense builder
// ---------------------------------------------------------------------------
void
fix_plan_dense (FixPlan &p, const std::vector<int> &nqm, std::vector<int4> &items)
{
  using C = Cfg<7>;
  p.ncol = 0;
  int row0 = 0, most = 1;
  for (FixClass &c : p.cls)
    {
      c.col0 = p.ncol;
      c.ncol = (p.M[0] + 1) * c.nc;
      p.ncol += (c.ncol + C::TN - 1) / C::TN * C::TN;
      c.row0 = row0;
      const int rows = (4 * c.nblk + C::KT - 1) / C::KT * C::KT;
      row0 += rows;
      most = std::max (most, rows);
    }
  p.nqp = row0 / 4;
  p.Rp = most;
  p.nct = p.ncol / C::TN;
  p.mt = p.ldT / TM;
  std::vector<int> tiles (p.nct);
  for (const FixClass &c : p.cls)
    for (int n = 0; n < c.ncol; n += C::TN)
      tiles[(c.col0 + n) / C::TN] = (4 * nqm[c.nq0 + n / c.nc] + C::KT - 1) / C::KT;
  slice_rows (tiles, p.mt, items);
  p.nbitem = (int) items.size ();
  int slot = 0;
  for (FixClass &c : p.cls)
    {
      c.slot0 = slot;
      for (int4 &it : items)
        if (it.x * C::TN >= c.col0 && it.x * C::TN < c.col0 + c.ncol) it.w = slot++;
      c.nslot = slot - c.slot0;
    }
}

int
fix_map_wb (const FixPlan &p, FixMaps *m)
{
  using G = Geo<7>;
  return encode_planes_f16 (&m->wb, p.WB, G::NP, p.ncol, (size_t) G::PAIR * p.Rp, Cfg<7>::TN);
}

cudaError_t
launch_fix_functions (const FixPlan &p, const double *pos, cudaStream_t st)
{
  const int items = p.M[0] + p.M[1] + p.M[2] + 3;
  k_fix_tables<<<dim3 ((p.np + TAB_P - 1) / TAB_P, (items + TAB_R - 1) / TAB_R), TAB_P * TAB_R, 0,
                 st>>> (p, pos, nullptr);
  return cudaGetLastError ();
}

cudaError_t
launch_fix_dense_image (const FixPlan &p, cudaStream_t st)
{
  k_fix_gimage<true><<<dim3 ((p.Rp / 8 + 127) / 128, p.ncol), 128, 0, st>>> (p);
  return cudaGetLastError ();
}

cudaError_t
launch_fix_dense (const FixPlan &particles, const FixPlan &p, const FixMaps &m, const int2 *tile,
                  int ntile, int *status, cudaStream_t st, Ctx *prof)
{
  cudaError_t e = gemm_attrs ();
  if (e != cudaSuccess) return e;
  const int items = p.M[0] + p.M[1] + p.M[2] + 3;
  k_fix_pair_tables<<<dim3 (ntile, (items + 15) / 16), 4 * PT, 0, st>>> (particles, p, tile);
  kmark (prof, st, "k_fix_pair_tables");
  k_fix_strings<<<dim3 (ntile, p.nqp / 4), 128, 0, st>>> (p);
  kmark (prof, st, "k_fix_strings");
  k_fix_bwd<7, true><<<dim3 ((ntile * PT + TM - 1) / TM, p.nbitem), NT, Geo<7>::SMEM, st>>> (m.wb, p,
                                                                                            status);
  kmark (prof, st, "k_fix_bwd");
  return cudaGetLastError ();
}

}  // namespace lsg
