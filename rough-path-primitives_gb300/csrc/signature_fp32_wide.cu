// signature_fp32_wide.cu -- the warp-per-letter kernels of widths 4, 6 and 7 that
// only single calls take (a file of their own: they compile beside the others).
#include "signature_fp32.cuh"

namespace rpp_gb {

RPP_GB_LETTER_LAUNCHES(RPP_GB_LETTER_SHAPES_WIDE, _wide)

}  // namespace rpp_gb
