// tma_host.h -- host-side encoding of TMA tensor maps through the driver
// entry point (no link against libcuda).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace lsg {

typedef CUresult (*EncodeTiledFn) (CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                    const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                    const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn
encode_fn ()
{
  static EncodeTiledFn fn = nullptr;
  if (!fn)
    {
      void *p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion ("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q)
            == cudaSuccess
          && q == cudaDriverEntryPointSuccess && p)
        fn = (EncodeTiledFn) p;
    }
  return fn;
}

// A [planes][rows][cols] f16 array, row-major, cols a multiple of 64, as a
// 3-d tensor map whose box is {64 columns (128 bytes), box_rows, planes}
// (every plane of a tile in one load) in the 128-byte swizzled layout; reads
// outside [rows] x [cols] fill zeros.  0 on success.
inline int
encode_planes_f16 (CUtensorMap *map, const void *base, unsigned long long planes,
                   unsigned long long rows, unsigned long long cols, unsigned box_rows)
{
  EncodeTiledFn fn = encode_fn ();
  if (!fn) return -1;
  if (cols % 64 || ((unsigned long long) base & 15ull) || box_rows == 0 || box_rows > 256
      || planes == 0 || planes > 256)
    return -2;
  const cuuint64_t dims[3] = {cols, rows, planes};
  const cuuint64_t strides[2] = {cols * 2ull, rows * cols * 2ull};
  const cuuint32_t box[3] = {64u, box_rows, (cuuint32_t) planes};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = fn (map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void *) base, dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int) r;
}

}  // namespace lsg
