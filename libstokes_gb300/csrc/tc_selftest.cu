// tc_selftest.cu -- known-answer checks of the tensor-core path of the digit
// GEMMs (kspace_fix.cu, kspace_mix.cu): f16 digit planes in 128-byte swizzled
// rows, one digit of A against several of B in one tcgen05.mma issued by a
// converged warp, accumulators read back from TMEM; B from hand-built planes or
// by one TMA box of all planes.  The products of digits are integers below
// 2^24, so the answer is exact.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "digit_gemm.cuh"
#include "gpu_engine.h"
#include "stokes_gpu.h"
#include "tc_umma.cuh"
#include "tma_host.h"

namespace lsg {
namespace {

constexpr int ST_ND = 3;                // digits
constexpr int ST_KT = 64, ST_NT = 2;    // values of a tile (128-byte rows), tiles
constexpr int ST_M = 128, ST_N = 32;    // rows of A, of a plane of B
constexpr int ST_NB = 24;               // rows of B; the others are zero
constexpr int ST_K = ST_KT * ST_NT;
constexpr uint32_t ST_A = ST_M * 128, ST_B = ST_N * 128;        // bytes of a plane of a tile
constexpr uint32_t ST_STAGE = ST_ND * (ST_A + ST_B);
constexpr uint32_t ST_COLS = 128;       // TMEM columns, of which ST_ND ST_N are used
constexpr uint32_t ST_LIMIT = 1u << 15; // polls of up to ~20 us each

// planes [ST_ND][rows][ST_K] of digits; D [ST_M][ST_ND ST_N]: group g sums the
// products of digits i and j with i + j = g
template <bool TMA>
__global__ void __launch_bounds__ (ST_M)
k_digit_selftest (const __grid_constant__ CUtensorMap tmB, const __half *A, const __half *B, float *D,
                  int *status)
{
  extern __shared__ unsigned char dsm[];
  __shared__ uint64_t loaded, done;
  __shared__ uint32_t tslot;
  __shared__ int err;
  const int tid = threadIdx.x, warp = tid >> 5;
  unsigned char *base = dg::align1k (dsm);
  if (warp == 0) umma::tmem_alloc (&tslot, ST_COLS);
  if (tid == 32)
    {
      umma::mbar_init (&loaded, 1);
      umma::mbar_init (&done, 1);
      err = 0;
      umma::fence_mbar_init ();
    }
  for (int t = 0; t < ST_NT; t++)
    for (int p = 0; p < ST_ND; p++)
      for (int c = 0; c < 8; c++)
        {
          unsigned char *a = base + t * ST_STAGE + p * ST_A;
          *reinterpret_cast<uint4 *> (a + dg::chunk_off (tid, c))
            = *reinterpret_cast<const uint4 *> (A + ((size_t) p * ST_M + tid) * ST_K + t * ST_KT + 8 * c);
          if (!TMA && tid < ST_N)
            *reinterpret_cast<uint4 *> (base + t * ST_STAGE + ST_ND * ST_A + p * ST_B
                                        + dg::chunk_off (tid, c))
              = tid < ST_NB ? *reinterpret_cast<const uint4 *> (B + ((size_t) p * ST_NB + tid) * ST_K
                                                                + t * ST_KT + 8 * c)
                            : make_uint4 (0u, 0u, 0u, 0u);
        }
  umma::fence_async_smem ();
  umma::fence_before_sync ();
  __syncthreads ();
  umma::fence_after_sync ();
  const uint32_t tmem = tslot;
  volatile int *e = &err, never = 0;
  if (warp == 0)
    {
      if (TMA)
        {
          if (tid == 0)
            {
              umma::mbar_expect_tx (&loaded, ST_NT * ST_ND * ST_B);
              for (int t = 0; t < ST_NT; t++)
                umma::tma_load_3d (base + t * ST_STAGE + ST_ND * ST_A, &tmB, t * ST_KT, 0, 0, &loaded);
            }
          __syncwarp ();
          // (a wait that ran out: once more before the shared memory goes away)
          if (!umma::mbar_wait_or_abort (&loaded, 0, ST_LIMIT, e))
            umma::mbar_wait_or_abort (&loaded, 0, ST_LIMIT, &never);
          __syncwarp ();
        }
      if (__all_sync (0xffffffffu, *e == 0))
        {
          umma::fence_after_sync ();
          for (int t = 0; t < ST_NT; t++)
            for (int k = 0; k < ST_KT / 16; k++)
              for (int i = 0; i < ST_ND; i++)
                {
                  const uint32_t s = umma::smem_u32 (base) + t * ST_STAGE;
                  umma::mma_f16 (tmem + i * ST_N, umma::smem_desc_sw128 (s + i * ST_A + 32 * k),
                                 umma::smem_desc_sw128 (s + ST_ND * ST_A + 32 * k),
                                 umma::idesc_f16 (ST_M, (ST_ND - i) * ST_N), t | k | i ? 1u : 0u);
                }
          umma::mma_commit_warp (&done);
          if (!umma::mbar_wait_or_abort (&done, 0, ST_LIMIT, e))
            umma::mbar_wait_or_abort (&done, 0, ST_LIMIT, &never);
        }
    }
  __syncthreads ();
  umma::fence_after_sync ();
  if (*e == 0)
    for (int c = 0; c < ST_ND * ST_N; c += 16)
      {
        float v[16];
        umma::tmem_ld16_issue (tmem + ((uint32_t) (warp * 32) << 16) + c, v);
        umma::tmem_ld_wait (v);
        for (int q = 0; q < 16; q++) D[(size_t) tid * ST_ND * ST_N + c + q] = v[q];
      }
  else if (tid == 0)
    *status = 1;
  umma::fence_before_sync ();
  __syncthreads ();
  if (warp == 0) umma::tmem_dealloc (tmem, ST_COLS);
}

template <bool TMA>
int
digit_selftest (double *max_rel_err)
{
  clear_error ();
  if (!max_rel_err) return set_error (STOKES_GPU_EINVAL, "NULL argument");
  constexpr int ND = ST_ND * ST_N;
  std::vector<__half> A ((size_t) ST_ND * ST_M * ST_K), B ((size_t) ST_ND * ST_NB * ST_K);
  std::vector<int> ia (A.size ()), ib (B.size ());
  uint32_t s = 777u;
  // digits -128 .. 127, the range ends among them
  auto digit = [&] () { s = s * 1664525u + 1013904223u; return (int) (s >> 24) - 128; };
  for (size_t k = 0; k < A.size (); k++) A[k] = __float2half ((float) (ia[k] = digit ()));
  for (size_t k = 0; k < B.size (); k++) B[k] = __float2half ((float) (ib[k] = digit ()));
  std::vector<float> D ((size_t) ST_M * ND);
  DevBuf dA, dB, dD, dS;
  cudaError_t e = dA.ensure (sizeof (__half) * A.size ());
  if (e == cudaSuccess) e = dB.ensure (sizeof (__half) * B.size ());
  if (e == cudaSuccess) e = dD.ensure (sizeof (float) * D.size ());
  if (e == cudaSuccess) e = dS.ensure (sizeof (int));
  if (e == cudaSuccess) e = cudaMemcpy (dA.p, A.data (), sizeof (__half) * A.size (), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy (dB.p, B.data (), sizeof (__half) * B.size (), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset (dS.p, 0, sizeof (int));
  if (e == cudaSuccess) e = cudaMemset (dD.p, 0xFF, sizeof (float) * D.size ());
  int status = 0, enc = 0;
  CUtensorMap map {};
  if (e == cudaSuccess && TMA) enc = encode_planes_f16 (&map, dB.p, ST_ND, ST_NB, ST_K, ST_N);
  if (e == cudaSuccess && !enc)
    {
      constexpr int smem = (int) (ST_NT * ST_STAGE) + 1024;
      e = cudaFuncSetAttribute (k_digit_selftest<TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e == cudaSuccess)
        {
          k_digit_selftest<TMA><<<1, ST_M, smem>>> (map, (const __half *) dA.p, (const __half *) dB.p,
                                                    (float *) dD.p, (int *) dS.p);
          e = cudaGetLastError ();
        }
      if (e == cudaSuccess)
        e = cudaMemcpy (D.data (), dD.p, sizeof (float) * D.size (), cudaMemcpyDeviceToHost);
      if (e == cudaSuccess) e = cudaMemcpy (&status, dS.p, sizeof (int), cudaMemcpyDeviceToHost);
    }
  for (DevBuf *b : {&dA, &dB, &dD, &dS}) b->release ();
  if (e != cudaSuccess) return cuda_fail (e, "tensor self-test");
  if (enc) return set_error (STOKES_GPU_ECUDA, "tensor self-test: tensor map encoding failed (%d)", enc);
  if (status) return set_error (STOKES_GPU_ETIMEOUT, "tensor self-test: a wait ran out");
  double worst = 0.0;
  for (int m = 0; m < ST_M; m++)
    for (int c = 0; c < ND; c++)
      {
        const int g = c / ST_N, n = c % ST_N;
        long long ref = 0, mag = 0;
        if (n < ST_NB)
          for (int i = 0; i <= g; i++)
            for (int k = 0; k < ST_K; k++)
              {
                const long long p = (long long) ia[((size_t) i * ST_M + m) * ST_K + k]
                                    * ib[((size_t) (g - i) * ST_NB + n) * ST_K + k];
                ref += p;
                mag += p < 0 ? -p : p;
              }
        const double err = fabs ((double) D[(size_t) m * ND + c] - (double) ref) / (mag > 0 ? (double) mag : 1.0);
        if (!(err <= worst)) worst = err;   // NaN-propagating max
      }
  *max_rel_err = worst;
  return STOKES_GPU_OK;
}

}  // namespace
}  // namespace lsg

extern "C" int
stokes_gpu_selftest_tensor (double *max_rel_err)
{
  return lsg::digit_selftest<false> (max_rel_err);
}

extern "C" int
stokes_gpu_selftest_tma (double *max_rel_err)
{
  return lsg::digit_selftest<true> (max_rel_err);
}
