// axis_cols_epi_f32.cu — instantiations of fft_axis.cuh: (tile width, largest radix, most threads, CTAs per SM)
#include "fft_axis.cuh"

namespace gpufft {
namespace axis {

const Kernel kColsEpi_f32[kClasses] = {
    GPUFFT_AXIS_COLS(float, 16, 16, true, 256, 3),
    GPUFFT_AXIS_COLS(float, 16, 22, true, 352, 2),
    GPUFFT_AXIS_COLS(float, 16, 32, true, 512, 1),
    GPUFFT_AXIS_COLS(float, 8, 16, true, 640, 1),
};

}  // namespace axis
}  // namespace gpufft
