// fixk.h -- data shared by the fixed-point tensor-core reciprocal sum
// (kspace_fix.cu) and the host code that plans it (product_fix.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace lsg {

// Weights of one reciprocal vector: its direction and the six scalars of
// recip_apply, times the weight of the vector in the sum over sign patterns.
struct __align__ (16) FixCoef {
  double ex, ey, ez, ya, yb, yc, yg, yh, ym, pad;
};

// Columns and rows of the dense builder (dense_fix.cu): the functions along y
// and z of a class have one parity each, so its K rows are products of these
// alone, in blocks of 2 x 2 (|m2|, |m3|), and its columns are (|m1|, q), q a
// pair moment of the class.  Components whose bit in `odd` is set go with
// sin(2 pi m1 x), the others with the cosine.
struct FixClass {
  int col0, ncol, nc;         // first column (a tile's), columns, components
  int row0, nblk, nq0;        // first row of S, blocks, first entry in nqm
  int odd;
  int slot0, nslot;           // its slots of partial results
};

// Plan of one reciprocal sum.  The k vectors are (m1, m2, m3) with m1 along x;
// an octant point is (|m1|, |m2|, |m3|).  Everything is expanded in products
// of real functions: function index 0 of an axis is 1, 2 m - 1 is
// cos(2 pi m u), 2 m is sin(2 pi m u), u the fractional coordinate.
//   quarter  one (|m2|, |m3|) of the set, sorted by length
//   row      4 quarter + 2 p2 + p3, p = 0 cosine, 1 sine: f_y f_z
//   column   mi c + q, mi the x function index, q the vector component
struct FixPlan {
  int np = 0, c = 0;
  double il[3] = {0, 0, 0};   // 1 / box
  double l[3] = {0, 0, 0};
  int M[3] = {0, 0, 0};       // largest |m| per axis
  int nmi = 0;                // x functions, 2 M[0] + 1
  int ncol = 0;               // nmi c
  int nq = 0, nqp = 0;        // quarters; padded to 32 (a row tile)
  int ldT = 0;                // particles padded to 128 (a backward row tile)
  int oy = 0, oz = 0, zero = 0, nT = 0;   // table rows: x from 0, y, z, the zero row, total
  int Rp = 0;                 // rows padded: 4 nqp
  int nct = 0, mt = 0;        // column tiles, 128-particle tiles
  int nsplit = 1, jper = 0;   // particle slices of the forward GEMM
  int nfitem = 0, nbitem = 0; // work items
  int fu = 0;                 // fractional bits of F
  int stall = 0;              // tests: polls of a wait that nothing completes

  const int4 *quart = nullptr;     // [nqp] table rows of (cos y, sin y, cos z, sin z)
  const int *nqm = nullptr;        // [M0 + 1] quarters in use at |m1|
  const FixCoef *coef = nullptr;   // octant points: [off[m1] + quarter][4 sign patterns]
  const int *off = nullptr;        // [M0 + 2] first octant point of |m1|
  void *T = nullptr;          // function table [nT][ldT]
  uint4 *q = nullptr;         // [np] fractional coordinates, upper 32 bits
  unsigned long long *u = nullptr;   // [np][4] the same, 64 bits
  float *xf = nullptr;        // [np][XF_LD] x / 2^xtop in FP32
  int *xtop = nullptr;
  void *S = nullptr;          // digit strings [Rp][ldT]
  void *F = nullptr;          // structure factors [nsplit][ncol][Rp], int64
  void *G = nullptr;          // operator output [ncol][Rp]
  void *ZF = nullptr;         // forward image, f16 digits of [ncol][ldT]
  void *WB = nullptr;         // backward image, f16 digits of [ncol][Rp]
  // high words of max |x_q| at [q] and of max |G| of the columns (m1, q) at
  // [16 (|m1| + 1) + q]
  unsigned *mx = nullptr;
  const int4 *fitem = nullptr;     // forward: row tile, column tile, particle slice
  const int4 *bitem = nullptr;     // backward: column tile, first K tile, K tiles
  void *yp = nullptr;         // back-projection partials [nbitem][np][c]; dense [slot][16][ldT]

  // dense builder: four classes; "particles" are the pairs of a chunk
  FixClass cls[4];
};

constexpr int XF_LD = 12;     // floats per particle of xf

struct FixMaps {
  CUtensorMap zf, wb;
};

// words of mx (a class of the dense builder; 16 (|m1| + 1) + component)
__host__ __device__ inline size_t
fix_mx_words (const FixPlan &p)
{
  return 16 * ((size_t) p.M[0] + 2);
}

// host entry points of kspace_fix.cu; ND: digits per number, 7 (FP64)
size_t fix_bytes_T (int nd, const FixPlan &p);
size_t fix_bytes_S (int nd, const FixPlan &p);
size_t fix_bytes_F (int nd, const FixPlan &p);
size_t fix_bytes_G (int nd, const FixPlan &p);
size_t fix_bytes_ZF (int nd, const FixPlan &p);
size_t fix_bytes_WB (int nd, const FixPlan &p);
size_t fix_bytes_yp (int nd, const FixPlan &p);
void fix_plan_items (int nd, FixPlan &p, const std::vector<int> &nqm, std::vector<int4> &fwd,
                     std::vector<int4> &bwd);
int fix_maps (int nd, const FixPlan &p, FixMaps *m);
struct Ctx;
// y partials of the reciprocal sum from positions and x (device), in order
// on st; p.mx is zero at the start; *status is raised when a bounded wait ran out
cudaError_t launch_fix_tables (int nd, const FixPlan &p, const double *pos, const double *x,
                               cudaStream_t st, Ctx *prof);
cudaError_t launch_fix_forward (int nd, int version, const FixPlan &p, const FixMaps &m, int *status,
                                cudaStream_t st, Ctx *prof);
cudaError_t launch_fix_backward (int nd, int version, const FixPlan &p, const FixMaps &m,
                                 int *status, cudaStream_t st, Ctx *prof);

// dense builder: columns, items and maps of its classes (cls[] holds nc, nblk
// and odd; nqm blocks in use by class and |m1|)
void fix_plan_dense (FixPlan &p, const std::vector<int> &nqm, std::vector<int4> &items);
int fix_map_wb (const FixPlan &p, FixMaps *m);
// function table of np positions (no strings or images)
cudaError_t launch_fix_functions (const FixPlan &p, const double *pos, cudaStream_t st);
// digits of G into the backward image
cudaError_t launch_fix_dense_image (const FixPlan &p, cudaStream_t st);
// partial moments of the pairs of `ntile` 8 x 8 tiles (tile[]: row, column of
// the tile) from the function table of the particles
cudaError_t launch_fix_dense (const FixPlan &particles, const FixPlan &p, const FixMaps &m,
                              const int2 *tile, int ntile, int *status, cudaStream_t st, Ctx *prof);

}  // namespace lsg
