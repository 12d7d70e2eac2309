// axis_rows_f32.cu — instantiations of fft_axis.cuh: (tile width, largest radix, most threads, CTAs per SM)
#include "fft_axis.cuh"

namespace gpufft {
namespace axis {

const Kernel kRows_f32[kClasses] = {
    GPUFFT_AXIS_ROWS(float, 16, 16, 256, 3),
    GPUFFT_AXIS_ROWS(float, 16, 22, 352, 2),
    GPUFFT_AXIS_ROWS(float, 16, 32, 512, 1),
    GPUFFT_AXIS_ROWS(float, 8, 16, 640, 1),
};

}  // namespace axis
}  // namespace gpufft
