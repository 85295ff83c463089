// product_fix.cu -- the FP64 product of equal spheres at the tuned split: the
// reciprocal sum as exact fixed-point GEMMs on the tensor cores
// (kspace_fix.cu), the real space on a side stream beside it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "ewald_device.cuh"
#include "fixk.h"
#include "gpu_engine.h"
#include "real_tab.h"
#include "seq_graph.h"
#include "stokes_gpu.h"

namespace lsg {

constexpr int ND = 7;

struct FixState {
  double key[16] = {0};
  uint64_t id = 0;              // counts the set-ups (part of the graph key)
  FixPlan p;
  FixMaps maps;
  double self[3] = {0, 0, 0};
  // real space: its radial table and lattice offsets; tabled: false for
  // splits with too many offsets, which the image-table kernel serves
  bool tabled = false;
  RealTabArgs real;
  DevBuf arena, partial;   // arena: every table and buffer of p and real
  int *h_status = nullptr, *d_status = nullptr;
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_end = nullptr;
  SeqGraph graph;
  bool clean = false;           // the maxima (FixPlan::mx) are zero: set-up or a whole product
};

// y = self x + real-space partials + reciprocal partials.  A CTA sums 32
// consecutive elements: warp w takes every eighth partial (coalesced), the
// eight sums meet in shared memory.
constexpr int FC_W = 8;

struct FixCombine {
  const double *x, *pr, *pk;
  int n, c, ncr, nck;
  double self[3];
  double *y;
  unsigned *mx;         // the maxima of the product, cleared for the next one
  int nmx;
};

__global__ void __launch_bounds__ (32 * FC_W)
k_fix_combine (FixCombine a)
{
  __shared__ double s_v[FC_W][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < a.nmx; k += 32 * FC_W) a.mx[k] = 0u;
  double v = 0.0;
  if (e < a.n)
    {
      for (int k = w; k < a.nck; k += FC_W) v += a.pk[(size_t) k * a.n + e];
      for (int k = w; k < a.ncr; k += FC_W) v += a.pr[(size_t) k * a.n + e];
    }
  s_v[w][lane] = v;
  __syncthreads ();
  if (w || e >= a.n) return;
#pragma unroll
  for (int k = 1; k < FC_W; k++) v += s_v[k][lane];
  const int q = e % a.c;
  // the self block is diagonal: the stresslet part (sm (S' - tr S' / 3) with
  // S' the full contraction) gives sm times the five components
  a.y[e] = fma (a.self[q < 3 ? 0 : (q < 6 ? 1 : 2)], a.x[e], v);
}

// octant points, weights and tiles of the split of ts, with libstokes' G term
// of sys's own split (FTS; the correction described at tuned_applies)
static int
fix_setup (Ctx *c, const struct stokes *sys, const struct stokes *ts)
{
  if (!c->fix) c->fix = new FixState ();
  FixState *f = c->fix;
  const bool fts = sys->version == 2;
  const double key[16] = {sys->lx, sys->ly, sys->lz, (double) sys->np, (double) sys->version,
                          ts->xi, ts->kmax, sys->xi, fts ? sys->kmax : 0.0,
                          fts ? (double) sys->kmaxx : 0.0, fts ? (double) sys->kmaxy : 0.0,
                          fts ? (double) sys->kmaxz : 0.0, 1.0};
  if (memcmp (key, f->key, sizeof key) == 0) return STOKES_GPU_OK;
  f->key[12] = 0.0;
  FixPlan p;
  p.np = sys->np;
  p.c = NCOMP (sys->version);
  p.l[0] = sys->lx; p.l[1] = sys->ly; p.l[2] = sys->lz;
  double k0[3];
  int B[3];
  const int ref[3] = {sys->kmaxx, sys->kmaxy, sys->kmaxz};
  for (int d = 0; d < 3; d++)
    {
      p.il[d] = 1.0 / p.l[d];
      k0[d] = 2.0 * M_PI / p.l[d];
      B[d] = (int) (ts->kmax / k0[d]);
      if (fts) B[d] = std::max (B[d], ref[d]);
    }
  // weights of one octant point without the direction; false: not in the set
  const double pivol = M_PI / (sys->lx * sys->ly * sys->lz);
  auto scalars = [&] (int a, int b, int d, FixCoef &w) {
    const double k1 = k0[0] * a, k2 = k0[1] * b, k3 = k0[2] * d;
    const double kk = k1 * k1 + k2 * k2 + k3 * k3, k = sqrt (kk);
    w = FixCoef {};
    if (kk == 0.0) return false;
    bool in = false;
    if (k <= ts->kmax)
      {
        const double k4z = kk / 4.0 / ts->xi2;
        const double kexp = pivol * (1.0 + k4z * (1.0 + 2.0 * k4z)) / kk * exp (-k4z);
        w.ya = 6.0 * (1.0 - kk / 3.0) * kexp;
        w.yb = 3.0 * k * kexp;
        w.yc = 1.5 * kk * kexp;
        w.yg = -3.0 * (1.0 - 4.0 / 15.0 * kk) * k * kexp;
        w.yh = 1.5 * kk * kexp;
        w.ym = 3.0 * (1.0 - kk / 5.0) * kk * kexp;
        in = true;
      }
    if (fts && a <= ref[0] && b <= ref[1] && d <= ref[2] && (sys->kmax == 0.0 || k <= sys->kmax))
      {
        const double k4z = kk / 4.0 / sys->xi2;
        const double kexp = sys->pivol * (1.0 + k4z * (1.0 + 2.0 * k4z)) / kk * exp (-k4z);
        w.yg += 6.0 * (1.0 - 4.0 / 15.0 * kk) * k * kexp;
        in = true;
      }
    w.ex = k1 / k; w.ey = k2 / k; w.ez = k3 / k;
    return in;
  };
  // quarters by length: the ones in use at |m1| are then (nearly) a prefix
  struct Quarter { int m2, m3; double kk; };
  std::vector<Quarter> qs;
  for (int b = 0; b <= B[1]; b++)
    for (int d = 0; d <= B[2]; d++)
      {
        const double k2 = k0[1] * b, k3 = k0[2] * d;
        const bool own = k2 * k2 + k3 * k3 <= ts->kmax * ts->kmax;
        const bool of_ref = fts && b <= ref[1] && d <= ref[2];
        if (own || of_ref) qs.push_back ({b, d, k2 * k2 + k3 * k3});
      }
  std::stable_sort (qs.begin (), qs.end (),
                    [] (const Quarter &a, const Quarter &b) { return a.kk < b.kk; });
  std::vector<FixCoef> coef, line (qs.size () * ((size_t) B[0] + 1));
  std::vector<int> nqm ((size_t) B[0] + 1), off ((size_t) B[0] + 2);
  for (int a = 0; a <= B[0]; a++)
    {
      nqm[a] = 0;
      for (size_t k = 0; k < qs.size (); k++)
        {
          FixCoef &w = line[(size_t) a * qs.size () + k];
          if (scalars (a, qs[k].m2, qs[k].m3, w))
            {
              nqm[a] = (int) k + 1;
              p.M[0] = a;
            }
        }
    }
  // a column tile covers the quarters of its smallest |m1|: prefixes that do
  // not grow with |m1|
  for (int a = B[0] - 1; a >= 0; a--) nqm[a] = std::max (nqm[a], nqm[a + 1]);
  const int nq = nqm[0];
  for (int a = 0; a <= B[0]; a++)
    {
      off[a] = (int) (coef.size () / 4);
      for (int k = 0; k < nqm[a]; k++)
        {
          // weight of the vector in the sum over the four sign patterns: the
          // point stands for prod (m ? 2 : 1) vectors, k and -k count alike
          const double mult = (a ? 2.0 : 1.0) * (qs[k].m2 ? 2.0 : 1.0) * (qs[k].m3 ? 2.0 : 1.0) / 4.0;
          for (int s = 0; s < 4; s++)
            {
              FixCoef w = line[(size_t) a * qs.size () + k];
              w.ey *= s & 2 ? -1.0 : 1.0;
              w.ez *= s & 1 ? -1.0 : 1.0;
              w.ya *= mult; w.yb *= mult; w.yc *= mult;
              w.yg *= mult; w.yh *= mult; w.ym *= mult;
              coef.push_back (w);
            }
        }
    }
  off[B[0] + 1] = (int) (coef.size () / 4);
  for (int k = 0; k < nq; k++)
    {
      p.M[1] = std::max (p.M[1], qs[k].m2);
      p.M[2] = std::max (p.M[2], qs[k].m3);
    }
  p.nmi = 2 * p.M[0] + 1;
  p.ncol = p.nmi * p.c;
  p.nq = nq;
  p.nqp = (std::max (nq, 1) + 31) / 32 * 32;
  p.Rp = 4 * p.nqp;
  p.ldT = (p.np + 127) / 128 * 128;
  p.oy = p.nmi;
  p.oz = p.oy + 2 * p.M[1] + 1;
  p.zero = p.oz + 2 * p.M[2] + 1;
  p.nT = p.zero + 1;
  std::vector<int4> fitem, bitem;
  fix_plan_items (ND, p, nqm, fitem, bitem);

  std::vector<int4> quart ((size_t) p.nqp, make_int4 (p.zero, p.zero, p.zero, p.zero));
  for (int k = 0; k < nq; k++)
    {
      const int b = qs[k].m2, d = qs[k].m3;
      quart[k] = make_int4 (p.oy + (b ? 2 * b - 1 : 0), b ? p.oy + 2 * b : p.zero,
                            p.oz + (d ? 2 * d - 1 : 0), d ? p.oz + 2 * d : p.zero);
    }
  // real space: lattice offsets whose cell of minimum-image displacements
  // comes within the cutoff, and the radial table
  RealTabArgs r {};
  const double rc = sqrt (ts->rmax2);
  std::vector<float4> roff;
  std::vector<int4> rcell;
  {
    int n[3];
    for (int d = 0; d < 3; d++) n[d] = std::min (7, (int) ceil (rc / p.l[d] + 0.5));
    for (int a1 = -n[0]; a1 <= n[0]; a1++)
      for (int a2 = -n[1]; a2 <= n[1]; a2++)
        for (int a3 = -n[2]; a3 <= n[2]; a3++)
          {
            const int m[3] = {a1, a2, a3};
            double dd = 0.0;
            for (int d = 0; d < 3; d++)
              {
                const double gap = std::max (0.0, (fabs ((double) m[d]) - 0.5) * p.l[d]);
                dd += gap * gap;
              }
            if (dd > rc * rc * 1.0001) continue;
            if (!a1 && !a2 && !a3) r.home = (int) roff.size ();
            roff.push_back (make_float4 ((float) (a1 * p.l[0]), (float) (a2 * p.l[1]),
                                         (float) (a3 * p.l[2]), 0.f));
            rcell.push_back (make_int4 (a1, a2, a3, 0));
          }
  }
  r.nimg = (int) roff.size ();
  f->tabled = r.nimg <= REAL_TAB_MAXIMG && rc <= 7.4 * std::min (p.l[0], std::min (p.l[1], p.l[2]));
  if (f->tabled) real_tab_range (rc, &r.bin0, &r.nbin);

  // one allocation: host tables (uploaded in one copy), then what stays zero
  // where nothing writes it (table pads, rows and columns), then the rest
  std::vector<char> host;
  size_t bytes = 0;
  auto align = [] (size_t n) { return (n + 255) / 256 * 256; };
  auto place = [&] (size_t n) {
    const size_t at = bytes;
    bytes += align (std::max<size_t> (n, 16));
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
  const size_t o_off = table (off.data (), sizeof (int) * off.size ());
  const size_t o_coef = table (coef.data (), sizeof (FixCoef) * coef.size ());
  const size_t o_fit = table (fitem.data (), sizeof (int4) * fitem.size ());
  const size_t o_bit = table (bitem.data (), sizeof (int4) * bitem.size ());
  const size_t o_roff = table (roff.data (), sizeof (float4) * roff.size ());
  const size_t o_rcell = table (rcell.data (), sizeof (int4) * rcell.size ());
  const size_t zero0 = bytes;
  const size_t o_mx = place (fix_mx_words (p) * sizeof (unsigned));
  const size_t o_T = place (fix_bytes_T (ND, p)), o_G = place (fix_bytes_G (ND, p));
  const size_t o_ZF = place (fix_bytes_ZF (ND, p)), o_WB = place (fix_bytes_WB (ND, p));
  const size_t zero1 = bytes;
  const size_t o_S = place (fix_bytes_S (ND, p)), o_F = place (fix_bytes_F (ND, p));
  const size_t o_yp = place (fix_bytes_yp (ND, p));
  const size_t o_q = place (sizeof (uint4) * p.np), o_u = place (sizeof (unsigned long long) * 4 * p.np);
  const size_t o_xf = place (sizeof (float) * XF_LD * p.np), o_top = place (sizeof (int));
  const size_t o_rt = place (f->tabled ? real_tab_bytes (sys->version, r.nbin) : 0);

  cudaStream_t st = c->stream;
  // no product of this context may still be using the tables of the last set-up
  cudaError_t e = f->id ? wait_products (c) : cudaSuccess;
  if (e == cudaSuccess) e = f->arena.ensure (bytes);
  char *base = (char *) f->arena.p;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync (base, host.data (), host.size (), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync (base + zero0, 0, zero1 - zero0, st);
  if (e == cudaSuccess && f->tabled)
    {
      r.tab = (const double *) (base + o_rt);
      r.tabf = (const float *) (r.tab + real_tab_doubles (sys->version, r.nbin));
      e = launch_real_tab_build (sys->version, r.bin0, r.nbin, ts->xi, (double *) r.tab,
                                 (float *) r.tabf, st);
    }
  // the upload reads a host vector of this call
  if (e == cudaSuccess) e = cudaStreamSynchronize (st);
  if (e != cudaSuccess) return cuda_fail (e, "FP64 product set-up");
  p.quart = (const int4 *) (base + o_quart);
  p.nqm = (const int *) (base + o_nqm);
  p.off = (const int *) (base + o_off);
  p.coef = (const FixCoef *) (base + o_coef);
  p.fitem = (const int4 *) (base + o_fit);
  p.bitem = (const int4 *) (base + o_bit);
  p.mx = (unsigned *) (base + o_mx);
  p.T = base + o_T; p.G = base + o_G; p.ZF = base + o_ZF; p.WB = base + o_WB;
  p.S = base + o_S; p.F = base + o_F; p.yp = base + o_yp;
  p.q = (uint4 *) (base + o_q);
  p.u = (unsigned long long *) (base + o_u);
  p.xf = (float *) (base + o_xf);
  p.xtop = (int *) (base + o_top);
  r.np = p.np;
  r.off = (const float4 *) (base + o_roff);
  r.cell = (const int4 *) (base + o_rcell);
  for (int d = 0; d < 3; d++)
    {
      r.sf[d] = (float) (p.l[d] / 4294967296.0);
      r.s60[d] = p.l[d] / 1152921504606846976.0;
    }
  // FP32 distances are within 1e-6 of the exact ones
  r.rc2 = (float) (ts->rmax2 * 1.00001);
  r.far2 = (float) real_tab_far (sys->version, ts->xi);
  r.xi = ts->xi;
  r.xisp = ts->xi / sqrt (M_PI);
  r.xi_ref = sys->xi;
  r.q = p.q; r.u = p.u; r.xf = p.xf; r.xtop = p.xtop;
  r.xf_ld = XF_LD;
  f->real = r;
  const int me = fix_maps (ND, p, &f->maps);
  if (me) return set_error (STOKES_GPU_ECUDA, "TMA tensor maps of the FP64 product (%d)", me);
  if ((e = status_word (&f->h_status, &f->d_status)) != cudaSuccess) return cuda_fail (e, "status");
  if (!f->side)
    {
      int lo = 0, hi = 0;
      cudaDeviceGetStreamPriorityRange (&lo, &hi);
      if (cudaStreamCreateWithPriority (&f->side, cudaStreamNonBlocking, lo) != cudaSuccess
          || cudaEventCreateWithFlags (&f->ev_fork, cudaEventDisableTiming) != cudaSuccess
          || cudaEventCreateWithFlags (&f->ev_join, cudaEventDisableTiming) != cudaSuccess
          || cudaEventCreateWithFlags (&f->ev_end, cudaEventDisableTiming) != cudaSuccess)
        return set_error (STOKES_GPU_ECUDA, "FP64 product: side stream");
    }
  f->self[0] = ts->self_a;
  f->self[1] = ts->self_c;
  f->self[2] = ts->self_m;
  f->p = p;
  f->clean = true;
  f->id++;
  memcpy (f->key, key, sizeof key);
  return STOKES_GPU_OK;
}

// source chunks per target of the real-space kernel: about 32 warps per SM
static int
real_chunks (int np)
{
  return std::max (1, std::min (std::min (np, 64), (152 * 32 + np - 1) / np));
}

int
atimes_fix_dev (Ctx *c, const double *d_pos, const double *d_x, double *d_y, cudaStream_t st,
                bool timed)
{
  const int rs = fix_setup (c, c->sys, c->fix_split);
  if (rs) return rs;
  FixState *f = c->fix;
  FixPlan p = f->p;
  p.stall = g_test_gemm_stall;
  const int np = c->np, n = np * p.c;
  const int failed = earlier_failure (c, f->h_status,
                                      "a tensor-core wait of the previous FP64 product ran out");
  if (failed) return failed;
  const int nchunk = f->tabled ? 1 : real_chunks (np);
  cudaError_t e = f->partial.ensure (sizeof (double) * (size_t) nchunk * n);
  if (e != cudaSuccess) return cuda_fail (e, "real-space scratch");

  RealArgs a;
  a.pos = d_pos;
  a.x = d_x;
  a.img = (const Img4 *) c->img.p;
  a.nimg = c->nimg;
  a.np = np;
  a.nchunk = nchunk;
  a.rmax2 = c->rmax2;
  a.rmin = c->rmin;
  a.xi = c->xi;
  a.xisp = c->xisp;
  a.rad = a.slipa = nullptr;
  a.partial = (double *) f->partial.p;
  a.open = 0;
  a.clampfix = c->rmin > 0.0 ? 1 : 0;
  a.xi_ref = c->xi_ref;
  a.xisp_ref = c->xi_ref / sqrt (M_PI);

  RealTabArgs rt = f->real;
  rt.x = d_x;
  rt.rmin = c->rmin;
  rt.rm2 = 4.0 * c->rmin * c->rmin;
  rt.far2 = std::max (rt.far2, (float) (rt.rm2 * 1.0001));     // clamped pairs are near ones
  rt.out = (double *) f->partial.p;
  auto real_space = [&] (cudaStream_t rs) {
    return f->tabled ? launch_real_tab (c->version, rt, rs)
                     : launch_real_fp64 (c->version, MODE_MONO, a, rs);
  };

  cudaEvent_t *E = phase_events (c, timed);
  const bool overlap = (!E || E == c->ev) && !c->kprof_on;
  auto sequence = [&] (bool recording) -> int {
    int *status = f->d_status;
    cudaError_t e;
    if (E && !recording) cudaEventRecord (E[0], st);
    kmark (c, st, nullptr);
    if ((e = launch_fix_tables (ND, p, d_pos, d_x, st, c)) != cudaSuccess)
      return cuda_fail (e, "reciprocal tables");
    // the real space needs the coordinates only; recorded after the forward
    // GEMM, its CTAs take what that leaves idle
    if (overlap) cudaEventRecord (f->ev_fork, st);
    if ((e = launch_fix_forward (ND, c->version, p, f->maps, status, st, c)) != cudaSuccess)
      return cuda_fail (e, "reciprocal space (forward)");
    if (overlap)
      {
        cudaStreamWaitEvent (f->side, f->ev_fork, 0);
        // nodes of the graph, so that every replay measures its real space
        const unsigned ext = recording ? cudaEventRecordExternal : cudaEventRecordDefault;
        if (E) cudaEventRecordWithFlags (E[1], f->side, ext);
        e = real_space (f->side);
        cudaEventRecord (f->ev_join, f->side);
        // beside the last kernel, which does not wait for it
        if (E)
          {
            cudaEventRecordWithFlags (E[2], f->side, ext);
            cudaEventRecord (f->ev_end, f->side);
          }
        if (e != cudaSuccess) return cuda_fail (e, "real-space kernel");
      }
    if ((e = launch_fix_backward (ND, c->version, p, f->maps, status, st, c)) != cudaSuccess)
      return cuda_fail (e, "reciprocal space (backward)");
    if (overlap)
      cudaStreamWaitEvent (st, f->ev_join, 0);
    else
      {
        if (E) cudaEventRecord (E[1], st);
        if ((e = real_space (st)) != cudaSuccess)
          return cuda_fail (e, "real-space kernel");
        kmark (c, st, f->tabled ? "k_real_tab" : "k_real");
        if (E) cudaEventRecord (E[2], st);
      }
    FixCombine cb {d_x, (const double *) f->partial.p, (const double *) p.yp, n, p.c, nchunk,
                   p.nbitem, {f->self[0], f->self[1], f->self[2]}, d_y, p.mx,
                   (int) fix_mx_words (p)};
    k_fix_combine<<<(n + 31) / 32, 32 * FC_W, 0, st>>> (cb);
    kmark (c, st, "k_fix_combine");
    if (E && overlap) cudaStreamWaitEvent (st, f->ev_end, 0);
    if (E && !recording) cudaEventRecord (E[3], st);
    if ((e = cudaGetLastError ()) != cudaSuccess) return cuda_fail (e, "FP64 product");
    return STOKES_GPU_OK;
  };
  static const bool graphs = [] {
    const char *g = getenv ("LIBSTOKES_GB300_GRAPHS");
    return !(g && strcmp (g, "0") == 0);
  }();
  uint64_t key = 1469598103934665603ull;
  uint64_t rmin_bits;
  memcpy (&rmin_bits, &a.rmin, sizeof rmin_bits);
  for (uint64_t v : {f->id, (uint64_t) (uintptr_t) d_pos, (uint64_t) (uintptr_t) d_x,
                     (uint64_t) (uintptr_t) d_y, (uint64_t) (uintptr_t) a.img, (uint64_t) a.nimg,
                     (uint64_t) (uintptr_t) a.partial, (uint64_t) (uintptr_t) E, rmin_bits})
    key = (key ^ v) * 1099511628211ull;
  const bool use = graphs && !c->kprof_on && (E == nullptr || E == c->ev) && p.stall == 0;
  // the last kernel of a product clears the maxima for the next one (a memset
  // of its own takes 2 us more); after a product that was not all launched
  // they are cleared here
  if (!f->clean)
    cudaMemsetAsync (p.mx, 0, fix_mx_words (p) * sizeof (unsigned), st);
  f->clean = false;
  const int rc = run_sequence (f->graph, key, st, E, use, sequence);
  if (rc) return rc;
  f->clean = true;
  c->launches = 9;
  c->timed = timed;
  return STOKES_GPU_OK;
}

int
fix_check_status (Ctx *c)
{
  FixState *f = c->fix;
  if (!f || !f->h_status || !*f->h_status) return STOKES_GPU_OK;
  *f->h_status = 0;
  return set_error (STOKES_GPU_ETIMEOUT, "a tensor-core wait of the FP64 product ran out");
}

void
release_fix (Ctx *c)
{
  FixState *f = c->fix;
  if (!f) return;
  for (DevBuf *b : {&f->arena, &f->partial}) b->release ();
  f->graph.release ();
  if (f->h_status) cudaFreeHost (f->h_status);
  if (f->side) cudaStreamDestroy (f->side);
  if (f->ev_fork) cudaEventDestroy (f->ev_fork);
  if (f->ev_join) cudaEventDestroy (f->ev_join);
  if (f->ev_end) cudaEventDestroy (f->ev_end);
  delete f;
  c->fix = nullptr;
}

}  // namespace lsg
