// axis_cols_f64.cu — instantiations of fft_axis.cuh: (tile width, largest radix, most threads, CTAs per SM)
#include "fft_axis.cuh"

namespace gpufft {
namespace axis {

const Kernel kCols_f64[kClasses] = {
    GPUFFT_AXIS_COLS(double, 8, 16, false, 128, 4),
    GPUFFT_AXIS_COLS(double, 8, 22, false, 176, 2),
    GPUFFT_AXIS_COLS(double, 8, 32, false, 256, 1),
    GPUFFT_AXIS_COLS(double, 8, 14, false, 640, 1),
};

}  // namespace axis
}  // namespace gpufft
