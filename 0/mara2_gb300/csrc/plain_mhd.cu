// plain_mhd.cu -- the plain FP64 path's kernels for one law.
#include "plain_kernels.cuh"

namespace mara {
MARA_PLAIN_LAW(, LAW_MHD);
} // namespace mara
