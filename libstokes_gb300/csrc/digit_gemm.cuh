// digit_gemm.cuh -- the warp roles shared by the digit GEMMs (kspace_fix.cu,
// kspace_mix.cu): operands are f16 digit planes of fixed-point numbers, B
// loaded by TMA, A built in shared memory by the worker warps, the digit
// products accumulated in TMEM and drained by the same warps.
//
// 576 threads, one CTA per SM:
//   warps 0-15  workers: build the A operand of each stage and drain the
//               accumulators; warp w reads TMEM lanes 32 (w % 4) and the
//               columns of group w / 4
//   warp 16     one lane issues the B loads of the ring of NS stages
//   warp 17     issues the MMAs
// The roles meet only at mbarriers; every wait is bounded and watches a CTA
// error flag, so a wait that runs out ends every role and raises the status
// word; the TMA lane waits for its loads in flight and the MMA warp for its
// MMAs before the CTA frees its TMEM and exits.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

#include "tc_umma.cuh"

namespace lsg {
namespace dg {

constexpr int NT = 576;
constexpr int WORKERS = 16;             // worker warps
constexpr int TMA_WARP = 16;
constexpr int MMA_WARP = 17;
constexpr int TM = 128;                 // MMA M
constexpr int MAX_NS = 3;               // stages at most
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t WAIT_LIMIT = 1u << 18;   // polls of up to ~20 us each

struct Sync {
  uint64_t afull[MAX_NS], bfull[MAX_NS], empty[MAX_NS], acc_full[2], acc_empty[2], done;
  uint64_t never;       // nothing arrives here: the wait of the failure-injection test
  uint32_t tslot;
  int err;
};

__device__ __forceinline__ unsigned char *
align1k (unsigned char *p)
{
  return p + ((1024u - (umma::smem_u32 (p) & 1023u)) & 1023u);
}

__device__ __forceinline__ void
cta_setup (Sync &s)
{
  if (threadIdx.x < 32) umma::tmem_alloc (&s.tslot, TMEM_COLS);
  if (threadIdx.x == 32)
    {
      for (int k = 0; k < MAX_NS; k++)
        {
          umma::mbar_init (&s.afull[k], WORKERS);
          umma::mbar_init (&s.bfull[k], 1);
          umma::mbar_init (&s.empty[k], 1);
        }
      for (int k = 0; k < 2; k++)
        {
          umma::mbar_init (&s.acc_full[k], 1);
          umma::mbar_init (&s.acc_empty[k], WORKERS);
        }
      umma::mbar_init (&s.done, 1);
      umma::mbar_init (&s.never, 1);
      s.err = 0;
      umma::fence_mbar_init ();
    }
  umma::fence_before_sync ();
  __syncthreads ();
  umma::fence_after_sync ();
}

__device__ __forceinline__ void
cta_finish (Sync &s, uint32_t tmem, int *status)
{
  if (threadIdx.x == 0 && s.err)
    {
      // (pinned host memory, see status_word)
      *(volatile int *) status = 1;
      __threadfence_system ();
    }
  umma::fence_before_sync ();
  __syncthreads ();
  if (threadIdx.x < 32) umma::tmem_dealloc (tmem, TMEM_COLS);
}

// byte offset of 16-byte chunk c of row r in a plane of 128-byte rows in the
// 128-byte swizzle
__device__ __forceinline__ uint32_t
chunk_off (int r, int c)
{
  return (uint32_t) (r * 128 + ((c ^ (r & 7)) << 4));
}

// one arrival per warp, after every lane's work (512 arrivals a tile took the
// barrier about 2000 clocks)
__device__ __forceinline__ void
arrive (uint64_t *bar)
{
  __syncwarp ();
  if ((threadIdx.x & 31) == 0) umma::mbar_arrive (bar);
}

// the B operand of a CTA: one box of `bytes` at x = x0 + dx t, row n0, at
// offset boff of a stage
struct BTiles {
  const CUtensorMap *map;
  int x0, dx, n0;
  uint32_t boff, bytes;
};

// All tiles of a CTA, in the role of the calling warp.  A worker builds tile t
// + NS once the MMAs of tile t are done, its loads issued a tile ahead; at the
// end of a set of DK tiles it drains first (sets alternate between NBUF
// accumulator buffers).  issue (stage address, buffer, first tile of a set)
// runs on the whole MMA warp.  True for workers whose sums are complete (false
// for the other roles and in an aborted CTA).
template <int DK, int NBUF, int NS, class Build, class Drain, class Issue>
__device__ __forceinline__ bool
run_tiles (Sync &s, unsigned char *smem, int ntiles, uint32_t stage, const BTiles &bt, int stall,
           Build &build, Drain &drain, const Issue &issue)
{
  static_assert (NS <= MAX_NS && NBUF <= 2, "ring");
  volatile int *err = &s.err, never = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == TMA_WARP)
    {
      if (lane == 0)
        {
          umma::tma_prefetch_desc (bt.map);
          int issued = 0;
          for (int t = 0; t < ntiles; t++)
            {
              const int st = t % NS;
              if (t >= NS && !umma::mbar_wait_or_abort (&s.empty[st], (t / NS - 1) & 1, WAIT_LIMIT, err))
                break;
              umma::mbar_expect_tx (&s.bfull[st], bt.bytes);
              umma::tma_load_3d (smem + (size_t) st * stage + bt.boff, bt.map, bt.x0 + bt.dx * t,
                                 bt.n0, 0, &s.bfull[st]);
              issued = t + 1;
            }
          // the last load of each stage must land before the shared memory
          // goes away
          for (int t = issued > NS ? issued - NS : 0; t < issued; t++)
            umma::mbar_wait_or_abort (&s.bfull[t % NS], (t / NS) & 1, WAIT_LIMIT, &never);
        }
      __syncwarp ();
      return false;
    }
  if (warp == MMA_WARP)
    {
      // failure injection (tests): a wait that cannot complete runs out, raises
      // the CTA error flag and ends every role before any MMA is issued
      if (stall > 0 && !umma::mbar_wait_or_abort (&s.never, 0, (uint32_t) stall, err)) ntiles = 0;
      ntiles = __shfl_sync (0xffffffffu, ntiles, 0);
      for (int t = 0; t < ntiles; t++)
        {
          const int st = t % NS, set = t / DK, b = set % NBUF;
          bool ok = umma::mbar_wait_or_abort (&s.bfull[st], (t / NS) & 1, WAIT_LIMIT, err)
                    && umma::mbar_wait_or_abort (&s.afull[st], (t / NS) & 1, WAIT_LIMIT, err);
          if (ok && t % DK == 0 && set >= NBUF)
            ok = umma::mbar_wait_or_abort (&s.acc_empty[b], (set / NBUF - 1) & 1, WAIT_LIMIT, err);
          if (!__all_sync (0xffffffffu, ok)) break;
          umma::fence_after_sync ();
          issue (umma::smem_u32 (smem) + (uint32_t) st * stage, b, t % DK == 0);
          umma::mma_commit_warp (&s.empty[st]);
          if (t % DK == DK - 1 || t == ntiles - 1) umma::mma_commit_warp (&s.acc_full[b]);
        }
      // every MMA issued so far has completed once `done` flips
      umma::mma_commit_warp (&s.done);
      umma::mbar_wait_or_abort (&s.done, 0, WAIT_LIMIT, &never);
      __syncwarp ();
      return false;
    }
  auto put = [&] (int t) {
    build.store (smem + (size_t) (t % NS) * stage);
    umma::fence_async_smem ();        // generic writes -> the MMA's async reads
    arrive (&s.afull[t % NS]);
    if (t + 1 < ntiles) build.load (t + 1);
  };
  if (ntiles > 0) build.load (0);
  for (int t = 0; t < NS && t < ntiles; t++) put (t);
  for (int t = 0; t < ntiles; t++)
    {
      if (t % DK == DK - 1 || t == ntiles - 1)
        {
          const int set = t / DK, b = set % NBUF;
          if (!umma::mbar_wait_or_abort (&s.acc_full[b], (set / NBUF) & 1, WAIT_LIMIT, err))
            return false;
          umma::fence_after_sync ();
          drain.take (set, b);
          umma::fence_before_sync ();
          arrive (&s.acc_empty[b]);
        }
      if (t + NS < ntiles)
        {
          if (!umma::mbar_wait_or_abort (&s.empty[t % NS], (t / NS) & 1, WAIT_LIMIT, err))
            return false;
          put (t + NS);
        }
    }
  return true;
}

// ---- host: how long a list of work items takes -----------------------------
constexpr int SMS = 152;

// time of `copies` CTAs of every length in len (K tiles, `start` more each),
// longest first on SMS SMs; a list of many rounds is taken as balanced to
// half its longest item
inline long long
makespan (std::vector<int> &len, int copies, int start)
{
  std::sort (len.begin (), len.end (), std::greater<int> ());
  if (len.size () * (size_t) copies > (size_t) 8 * SMS)
    {
      long long sum = 0;
      for (int l : len) sum += l + start;
      return sum * copies / SMS + (len[0] + start) / 2;
    }
  std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free;
  for (int k = 0; k < SMS; k++) free.push (0);
  long long last = 0;
  for (int l : len)
    for (int k = 0; k < copies; k++)
      {
        const long long t = free.top () + l + start;
        free.pop ();
        free.push (t);
        last = std::max (last, t);
      }
  return last;
}

}  // namespace dg
}  // namespace lsg
