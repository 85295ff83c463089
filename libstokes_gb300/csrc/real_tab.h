// real_tab.h -- FP64 real-space sum from radial tables (real_tab.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lsg {

struct RealTabArgs {
  const uint4 *q;                 // upper 32 bits of the fractional coordinates
  const unsigned long long *u;    // [np][4] fractional coordinates, 2^64 = the box
  const double *x;                // [np][c]
  const float *xf;                // [np][xf_ld] x / 2^*xtop, for the far pairs
  const int *xtop;
  int xf_ld;
  int np;
  // lattice offsets added to the minimum-image displacement (1: none; a cutoff
  // beyond half the box); home: the zero offset
  int nimg, home;
  const float4 *off;
  const int4 *cell;
  float sf[3];                    // box / 2^32
  double s60[3];                  // box / 2^60
  float rc2;                      // FP32 test, a little wide
  float far2;                     // pairs beyond take FP32 (see real_tab.cu)
  double xi, xisp, xi_ref;
  double rmin, rm2;               // rmin clamp: (2 rmin)^2, 0 without
  const double *tab;
  const float *tabf;              // [nbin][functions][8], FP32
  int bin0, nbin;
  double *out;                    // [np][c]
};

constexpr int REAL_TAB_MAXIMG = 32;    // offsets at most

void real_tab_range (double rc, int *bin0, int *nbin);
size_t real_tab_bytes (int version, int nbin);     // both tables
size_t real_tab_doubles (int version, int nbin);   // the first one
double real_tab_far (int version, double xi);      // squared distance of the FP32 pairs
cudaError_t launch_real_tab_build (int version, int bin0, int nbin, double xi, double *tab,
                                   float *tabf, cudaStream_t st);
cudaError_t launch_real_tab (int version, const RealTabArgs &a, cudaStream_t st);

}  // namespace lsg
