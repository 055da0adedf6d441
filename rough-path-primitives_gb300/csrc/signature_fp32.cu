// signature_fp32.cu -- FP32 signatures with one warp per first letter
// (schedule bit 16, kScheduleLetterWarps): which shapes have them, and the
// launches of the shapes that the grouped launch runs too; those that only
// single calls take are in signature_fp32_narrow.cu and signature_fp32_wide.cu.
#include "signature_fp32.cuh"

namespace rpp_gb {

RPP_GB_LETTER_LAUNCHES(RPP_GB_LETTER_SHAPES, _group)
cudaError_t launch_letters_narrow(const Geometry&, const DeviceInfo&, cudaStream_t, const float*, PathBatch, float*,
                                  int64_t);
cudaError_t launch_letters_rev_narrow(const Geometry&, const DeviceInfo&, cudaStream_t, const float*, PathBatch, float*,
                                      int64_t, const float*, int64_t, float*, int);
cudaError_t launch_letters_wide(const Geometry&, const DeviceInfo&, cudaStream_t, const float*, PathBatch, float*,
                                int64_t);
cudaError_t launch_letters_rev_wide(const Geometry&, const DeviceInfo&, cudaStream_t, const float*, PathBatch, float*,
                                    int64_t, const float*, int64_t, float*, int);

namespace {

enum class LetterShapes { None, Group, Narrow, Wide };

LetterShapes letter_shapes(int width, int depth) {
#define RPP_GB_LETTER_CASE(w, d) case w * 100 + d:
    switch (width * 100 + depth) {
        RPP_GB_LETTER_SHAPES(RPP_GB_LETTER_CASE) return LetterShapes::Group;
        RPP_GB_LETTER_SHAPES_NARROW(RPP_GB_LETTER_CASE) return LetterShapes::Narrow;
        RPP_GB_LETTER_SHAPES_WIDE(RPP_GB_LETTER_CASE) return LetterShapes::Wide;
        default: return LetterShapes::None;
    }
#undef RPP_GB_LETTER_CASE
}

}  // namespace

bool letter_group_supported(int width, int depth) { return letter_shapes(width, depth) == LetterShapes::Group; }
bool letter_warps_supported(int width, int depth) { return letter_shapes(width, depth) != LetterShapes::None; }
bool letter_reverse_supported(int width, int depth) { return depth >= 3 && letter_warps_supported(width, depth); }

cudaError_t launch_signature_letters_rev(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, const float* incr,
                                         PathBatch paths, float* sig, int64_t sig_stride, const float* seed,
                                         int64_t seed_stride, float* grad, int mode) {
    switch (letter_shapes(g.width, g.depth)) {
        case LetterShapes::Group:
            return launch_letters_rev_group(g, dev, s, incr, paths, sig, sig_stride, seed, seed_stride, grad, mode);
        case LetterShapes::Narrow:
            return launch_letters_rev_narrow(g, dev, s, incr, paths, sig, sig_stride, seed, seed_stride, grad, mode);
        case LetterShapes::Wide:
            return launch_letters_rev_wide(g, dev, s, incr, paths, sig, sig_stride, seed, seed_stride, grad, mode);
        default: return cudaErrorInvalidConfiguration;
    }
}

cudaError_t launch_signature_letters(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, const float* incr,
                                     PathBatch paths, float* sig, int64_t sig_stride) {
    switch (letter_shapes(g.width, g.depth)) {
        case LetterShapes::Group: return launch_letters_group(g, dev, s, incr, paths, sig, sig_stride);
        case LetterShapes::Narrow: return launch_letters_narrow(g, dev, s, incr, paths, sig, sig_stride);
        case LetterShapes::Wide: return launch_letters_wide(g, dev, s, incr, paths, sig, sig_stride);
        default: return cudaErrorInvalidConfiguration;
    }
}

}  // namespace rpp_gb
