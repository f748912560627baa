// tensor_map.h -- cuTensorMapEncodeTiled, looked up through the runtime once
// (no link-time dependency on libcuda); nullptr where the driver lacks it.

#ifndef CORR_GB300_TENSOR_MAP_H
#define CORR_GB300_TENSOR_MAP_H

#include <cuda.h>

namespace corrgb {

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled();

} // namespace corrgb

#endif // CORR_GB300_TENSOR_MAP_H
