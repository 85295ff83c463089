// gpu_engine.h -- per-system device context shared by the host engine files.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <array>
#include <vector>

#include "stokes_abi.h"
#include "engine.h"

namespace lsg {

struct DevBuf {
  void *p = nullptr;
  size_t cap = 0;
  cudaError_t ensure (size_t bytes);
  void release ();
};

struct MixedState;   // mixed-precision state (mixed.cu)
struct DenseState;   // FP64 dense builder on the tensor cores (dense_fix.cu)
struct FixState;     // FP64 product with the fixed-point reciprocal sum (product_fix.cu)

struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[4] = {};
  cudaEvent_t join[2] = {};   // orders the context's stream inside the legacy default stream
  int precision = 0;

  // the end of the last product or build on another stream than `stream`
  // (note_use, wait_products); captured: one was recorded into a graph of the
  // caller's, whose replays are not seen here
  cudaEvent_t used = nullptr;
  bool used_set = false, captured = false;

  // geometry of the last prepared system
  const struct stokes *sys = nullptr;
  int version = 0, np = 0, mode = 0;
  double xi = 0, xisp = 0, rmax2 = 0, rmin = 0;
  double xi_ref = 0;      // the struct's own split (differs from xi at the tuned split)
  int nimg = 0, nk = 0;
  uint64_t fp_img = 0, fp_kt = 0, fp_pp = 0;
  std::vector<Img4> h_img;
  std::vector<double> h_kt, h_pp;

  DevBuf pos, x, y, img, kt, pp, ph, sf, yrec, partial, mat, zbuf;

  double times[3] = {0, 0, 0};
  int launches = 0;
  bool timed = false;

  // profiling window: 4 events per product (start, reciprocal done,
  // real space done, end), read back by stokes_gpu_profile_end
  bool prof_on = false;
  int prof_n = 0;
  std::vector<cudaEvent_t> prof_ev;

  // kernel profiling window: one event after each launch, tagged with the
  // kernel's name (nullptr marks the start of a product)
  bool kprof_on = false;
  // non-periodic (free-space) operator: set for systems with periodic = 0 and
  // by the *_nonewald_* entry points (force_open), src/non-ewald.c
  bool open = false, force_open = false;
  // FP64 products of an equal-sphere periodic system run at a cheaper
  // Ewald split than the reference's (prepare): a private copy of the
  // system set up at that split, its key, and whether prepare may use it
  struct stokes *tuned = nullptr;
  double tuned_key[7] = {0, 0, 0, 0, 0, 0, 0};
  bool tune = true;
  size_t kprof_n = 0;
  std::vector<cudaEvent_t> kprof_ev;
  std::vector<const char *> kprof_name;

  MixedState *mixed = nullptr;

  // the FP64 product with the fixed-point reciprocal sum (product_fix.cu);
  // use_fix: the last prepare chose it
  FixState *fix = nullptr;
  bool use_fix = false;
  const struct stokes *fix_split = nullptr;   // the tuned split of that prepare
  // the FP64 dense builder of equal spheres (dense_fix.cu), likewise
  DenseState *dfix = nullptr;
  bool use_dense = false;

  DevBuf openf;   // scratch of the mixed-precision free-space product
  DevBuf imgf;    // the images in FP32 (split-precision dense builder)
  // the thread-per-pair dense builder's split: a private copy of the system
  // at it, its key, the half-space tables (FP64 rows for the phases, floats
  // for the terms) and their count
  bool cube = false;   // the last prepare's image set is the _notbl cube
  struct stokes *dense = nullptr;
  double dense_key[7] = {0, 0, 0, 0, 0, 0, 0};
  int dense_nk = 0;
  std::vector<double> h_dkt;
  DevBuf dkt, dktf, dself;   // FP64 rows, moment coefficients, diagonal moments
  uint64_t fp_dkt = 0;

  // pinned, mapped mirror of sys->pos for the host entry points of the
  // mixed paths, whose kernels read the positions once
  // pinned buffers that small host calls pass x and y through (host_stage)
  struct Stage {
    double *p = nullptr, *dev = nullptr;      // its host and device addresses
    size_t bytes = 0;
  } hx, hy;
  double *hpos = nullptr;
  const double *hpos_dev = nullptr;   // its device address
  size_t hpos_bytes = 0;

  std::array<DevBuf *, 17> all_buffers ()
  {
    return {&pos, &x, &y, &img, &kt, &pp, &ph, &sf, &yrec, &partial, &mat, &zbuf, &openf, &imgf,
            &dkt, &dktf, &dself};
  }
};

int set_error (int code, const char *fmt, ...);
void clear_error ();
int cuda_fail (cudaError_t e, const char *where);
void dropin_failed (const char *fn, double *out, size_t nout);

Ctx *get_ctx (const struct stokes *sys, bool create);
// host tables of one system (gpu_engine.cu)
int check_sys (const struct stokes *sys, bool open = false);
// STOKES_GPU_EINVAL when a coordinate of the host positions pos[3 np] is NaN
// or infinite (the kernels would turn it into a wrong result, not an error)
int check_positions (const double *pos, int np);
void build_images (const struct stokes *sys, bool cube, std::vector<Img4> &img);
void build_ktable (const struct stokes *sys, std::vector<double> &kt);
void build_particles (const struct stokes *sys, int mode, std::vector<double> &pp,
                      bool open = false, const struct stokes *split = nullptr);
int release_ctx (const struct stokes *sys);
// u = (I + M L)^-1 M f on device buffers (krylov.cu), F and FT, the
// context's product at positions d_pos, GMRES settings from sys->it
int lub_mobility_dev (Ctx *c, struct stokes *sys, const double *d_pos, const double *d_f,
                      double *d_u, cudaStream_t st, int *iters);
// f = L u on device buffers (lub.cu): version 0 (F) or 1 (FT)
int lub_dev (const struct stokes *sys, int version, const double *d_pos, const double *d_u,
             double *d_f, cudaStream_t st);
// check sys and bring the context's device tables up to date.  tables: 1
// builds the FP64 image and reciprocal tables of the FP64 product (the
// tuned split where it applies), 2 those of the dense builder (the
// reference's split), 0 skips them (the mixed product never reads them),
// -1 chooses by the context's precision.
int prepare (Ctx *c, const struct stokes *sys, bool cube, int tables = -1);

// drops the adjoint's private copy of sys, if any (adjoint.cu)
void release_adjoint (const struct stokes *sys);
int atimes_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y,
                cudaStream_t st, bool timed);
int atimes_fp64_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y,
                     cudaStream_t st, bool timed);
// the same for equal spheres at the tuned split (product_fix.cu)
int atimes_fix_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y, cudaStream_t st,
                    bool timed);
int fix_check_status (Ctx *c);
void release_fix (Ctx *c);
// the dense matrix of equal spheres in FP64 (dense_fix.cu)
bool dense_fix_applies (const Ctx *c, const struct stokes *sys);
int matrix_fix_dev (Ctx *c, const double *d_pos, double *d_mat, cudaStream_t st);
int dense_check_status (Ctx *c);
void release_dense (Ctx *c);
void collect_times (Ctx *c);
cudaEvent_t *phase_events (Ctx *c, bool timed);
// a status word that kernels raise when a bounded wait runs out: pinned host
// memory that they write in place, so that a product needs no copy to report it
// (a copy engine's turn at its end, 2-6 us)
cudaError_t status_word (int **host, int **dev);
// STOKES_GPU_ETIMEOUT when an earlier product or build raised the word; cleared
// once those queued behind it, which may raise it again, are done
int earlier_failure (Ctx *c, int *word, const char *message);
// record a kernel-profiling mark on st when the window is open
void kmark (Ctx *c, cudaStream_t st, const char *name);

// Tables and buffers of a context are read by products that may still be queued
// on a stream of the caller's: what overwrites or frees them waits first
// (wait_products), and every function that launches such work marks its end.
cudaError_t wait_products (Ctx *c);
void note_use (Ctx *c, cudaStream_t st);
struct UseMark {
  Ctx *c;
  cudaStream_t st;
  ~UseMark () { note_use (c, st); }
};

// mixed-precision path (mixed.cu)
int atimes_mixed_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y,
                      cudaStream_t st, bool timed);
// free-space product of an open system in mixed precision (open_f32.cu)
int atimes_open_f32_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y,
                         cudaStream_t st, bool timed);
void release_mixed (Ctx *c);
// mixed-precision VJP (adjoint_f32.cu): 1 when it served the call, 0 when
// the system needs the FP64 adjoint, -status on error
int vjp_mixed (Ctx *c, const struct stokes *sys, const double *g, const double *f, double *dLdr,
               double *dLdbox);
void release_vjp_mixed (const Ctx *c);
// after the stream of a mixed product was synchronised: STOKES_GPU_ETIMEOUT
// (and the status word cleared) when a bounded wait of its tensor-core
// kernels ran out, else STOKES_GPU_OK
int mixed_check_status (Ctx *c);
// the same for whatever products and dense builds c made: every call that
// synchronises and hands back results of its own products ends with it
int check_status (Ctx *c);

// failure-injection settings of stokes_gpu_test_stall_waits (util.cu): polls
// of an extra wait of the k-space GEMMs' MMA lane on an mbarrier that nothing
// arrives at (0: no such wait), and the spin limit of the GMRES grid barrier
// (0: the default)
extern int g_test_gemm_stall;
extern long long g_test_bar_spins;

}  // namespace lsg
