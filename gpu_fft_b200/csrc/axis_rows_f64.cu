// axis_rows_f64.cu — instantiations of fft_axis.cuh: (tile width, largest radix, most threads, CTAs per SM)
#include "fft_axis.cuh"

namespace gpufft {
namespace axis {

const Kernel kRows_f64[kClasses] = {
    GPUFFT_AXIS_ROWS(double, 8, 16, 128, 4),
    GPUFFT_AXIS_ROWS(double, 8, 22, 176, 2),
    GPUFFT_AXIS_ROWS(double, 8, 32, 256, 1),
    GPUFFT_AXIS_ROWS(double, 8, 14, 640, 1),
};

}  // namespace axis
}  // namespace gpufft
