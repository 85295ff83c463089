// mixed.h -- data shared by the mixed-precision host code (mixed.cu) and its
// reciprocal-space tensor-core kernels (kspace_mix.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace lsg {

// floor(v) mod 2^32 for |v| < 2^62: the 32-bit fixed-point coordinate, the
// periodic wrap being the modulo
__device__ __forceinline__ uint32_t
fixq (double v)
{
  return (uint32_t) (unsigned long long) __double2ll_rd (v);
}

// one half-space reciprocal vector (64 bytes)
struct __align__ (16) MixK {
  int m1, m2, m3, pad;
  float ex, ey, ez;
  float ya, yb, yc, yg, yh, ym;
  float f0, f1, f2;
};

// e^{2 pi i p / 2^32} to FP32 accuracy from a fixed-point phase p (turns x
// 2^32): the nearest of 1024 tabulated rotations e^{2 pi i h / 1024} (rot[h]
// = (hi.re, hi.im, lo.re, lo.im), each a float pair hi + lo) times a short
// Taylor series of the remaining angle |theta| <= pi / 1024 (table-driven
// argument reduction).  Truncation errors are below 1e-14; the result
// carries one FP32 rounding (3e-8 measured over 2e6 random phases).
__device__ __forceinline__ float2
phase_of (const float4 *rot, uint32_t p)
{
  const uint32_t h = (p + (1u << 21)) >> 22;             // nearest table entry
  const int32_t r = (int32_t) (p - (h << 22));           // |r| <= 2^21
  const float th = (float) r * 1.4629180792671596e-09f;  // 2 pi / 2^32
  const float t2 = th * th;
  const float sn = th * (1.0f - t2 * (1.0f / 6.0f));     // sin th
  const float dc = t2 * (0.5f - t2 * (1.0f / 24.0f));    // 1 - cos th
  const float4 e = __ldg (rot + (h & 1023u));
  // (e.x + e.z + i (e.y + e.w)) (1 - dc + i sn), small terms first
  const float re = e.x + fmaf (-e.x, dc, fmaf (-e.y, sn, e.z));
  const float im = e.y + fmaf (-e.y, dc, fmaf (e.x, sn, e.w));
  return make_float2 (re, im);
}

// weights of one reciprocal vector on the tensor-core path: direction and the
// six scalars of recip_apply
struct __align__ (16) MixCoef {
  float ex, ey, ez, ya, yb, yc, yg, yh, ym, p0, p1, p2;
};

// plan of the tensor-core reciprocal sum (kspace_mix.cu).  Functions of an
// axis: index 0 is 1, 2 m - 1 is cos 2 pi m u, 2 m is sin 2 pi m u.
//   quarter  one (|m2|, |m3|) of the k list, sorted by length
//   row      4 quarter + 2 p2 + p3, p = 0 cosine, 1 sine: f_y f_z
//   column   mi c + q, mi the x function index, q one of c = cf (forward) or cb
//            (backward) components
struct MixPlan {
  int np, M[3];
  int c;                  // vector components
  int cf, cb;             // columns per x function, forward and backward (c; unequal
                          // radii: see k_kop_poly)
  int nmi, ncolf, ncolb;  // x functions 2 M[0] + 1; columns
  int nq, nqp, Rp;        // quarters; padded to 32; rows 4 nqp
  int ldT;                // particles padded to 128
  int oy, oz, zero, nT;   // table rows: x from 0, y, z, the zero row, total
  int tnf, nctf, ldf;     // forward columns per tile, tiles, padded columns
  int tnb, nctb, ldb;     // backward
  int mt;                 // 128-particle tiles
  int jper, nsplit;       // particles per forward slice, slices
  int nfitem, nbitem;     // work items
  int stall;              // > 0 (tests only): the MMA lane first waits that many
                          // polls on an mbarrier that nothing arrives at
  const int4 *quart;      // [nqp] table rows of (cos y, sin y, cos z, sin z)
  const int *nqm;         // [M0 + 1] quarters in use at |m1|
  const int *off;         // [M0 + 2] first octant point of |m1|
  const MixCoef *coef;    // [octant points][4 sign patterns]
  const int4 *fitem;      // forward: row tile, column tile, particle slice
  const int4 *bitem;      // backward: column tile, first K tile, K tiles
  int *T;                 // function table [nT][ldT], 30 fractional bits
  float *zs;              // units of ZF, [ldT / 128][ldf]
  float *ws;              // units of WB, [Rp / 128][ldb]
  void *ZF, *WB;          // images, f16 digits [3][columns][ldT or Rp]
  float *F;               // structure factors [nsplit][ncolf][Rp]
  float *yp;              // back-projection partials [nbitem][np][c]
  const float *rad;       // unequal radii (NULL: unit spheres)
};

// TMA descriptors of the two images
struct MixMaps {
  CUtensorMap zf, wb;
};

struct MixPrep {
  const double *pos, *x;
  int np, c;
  double sx, sy, sz;      // 2^32 / L_d
  double shift, sl;       // Lees-Edwards shift (flow axis x), shift / lx
  int shear_mode;
  const float4 *rot;      // rotations of phase_of
  const float *qa;        // unequal radii: squared radii
  uint32_t *qpos;         // [np][4] fixed-point x, y, z (+ pad)
  float *xf;              // [np][c padded to 4]
  MixPlan p;
};

void mix_plan_items (MixPlan &p, const std::vector<int> &nqm, std::vector<int4> &fwd,
                     std::vector<int4> &bwd);
// backward columns per x function of unequal radii
int mix_poly_columns (int version);
size_t mix_zf_bytes (const MixPlan &p);
size_t mix_wb_bytes (const MixPlan &p);
size_t mix_zs_floats (const MixPlan &p);
size_t mix_ws_floats (const MixPlan &p);
int mix_maps (const MixPlan &p, MixMaps *m);      // 0 on success

// prep -> forward GEMM and operators -> backward GEMM into yp
struct Ctx;
cudaError_t launch_mix_prep (const MixPrep &a, cudaStream_t st);
cudaError_t launch_mix_forward (int version, const MixPlan &p, const MixMaps &m, int *status,
                                cudaStream_t st, Ctx *prof);
cudaError_t launch_mix_backward (const MixPlan &p, const MixMaps &m, int *status, cudaStream_t st,
                                 Ctx *prof);

}  // namespace lsg
