// signature_fp32_narrow.cu -- the warp-per-letter kernels of widths 2 and 3 that
// only single calls take (a file of their own: they compile beside the others).
#include "signature_fp32.cuh"

namespace rpp_gb {

RPP_GB_LETTER_LAUNCHES(RPP_GB_LETTER_SHAPES_NARROW, _narrow)

}  // namespace rpp_gb
