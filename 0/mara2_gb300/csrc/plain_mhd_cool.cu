// plain_mhd_cool.cu -- the plain FP64 path's kernels for one law.
#include "plain_kernels.cuh"

namespace mara {
MARA_PLAIN_LAW(, LAW_MHD_COOL);
} // namespace mara
