// seq_graph.h -- replay of a fixed launch sequence as a CUDA graph.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "gpu_engine.h"

namespace lsg {

struct SeqGraph {
  cudaGraphExec_t exec = nullptr;
  uint64_t key = 0, cand = 0;
  void release ()
  {
    if (exec) cudaGraphExecDestroy (exec);
    exec = nullptr;
    key = cand = 0;
  }
};

// Runs `sequence (recording)` (the launches of one product on st, returning a
// status) directly the first time a configuration `key` appears, records it into a
// graph (stream capture) the second time and replays that from then on.  The
// key covers everything the recorded nodes hold: pointers, sizes, events.
// Nothing is recorded while st is itself being captured by the caller.  A
// captured cudaEventRecord is only a dependency, so the start and end events
// E[0], E[3] (E may be NULL) are recorded around a replay, and while `recording`
// the sequence makes event nodes of the others (cudaEventRecordExternal).
template <class Seq>
int
run_sequence (SeqGraph &g, uint64_t key, cudaStream_t st, cudaEvent_t *E, bool use, Seq &&sequence)
{
  if (use)
    {
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing (st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        use = false;
    }
  if (!use) return sequence (false);
  if (!g.exec || key != g.key)
    {
      if (key != g.cand)
        {
          g.cand = key;
          return sequence (false);
        }
      if (g.exec) cudaGraphExecDestroy (g.exec);
      g.exec = nullptr;
      if (cudaStreamBeginCapture (st, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        {
          cudaGetLastError ();
          return sequence (false);
        }
      const int rc = sequence (true);
      cudaGraph_t gr = nullptr;
      cudaError_t e = cudaStreamEndCapture (st, &gr);
      if (!rc && e == cudaSuccess && gr) e = cudaGraphInstantiate (&g.exec, gr, 0);
      if (gr) cudaGraphDestroy (gr);
      if (rc) return rc;
      if (e != cudaSuccess || !g.exec)
        {
          g.exec = nullptr;
          cudaGetLastError ();
          return sequence (false);             // not recorded: launch directly
        }
      g.key = key;
    }
  if (E) cudaEventRecord (E[0], st);
  const cudaError_t le = cudaGraphLaunch (g.exec, st);
  if (E) cudaEventRecord (E[3], st);
  return le == cudaSuccess ? 0 : cuda_fail (le, "product graph");
}

}  // namespace lsg
