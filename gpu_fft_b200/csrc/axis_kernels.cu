// axis_kernels.cu — the kernels of fft_axis.cuh for the lengths of
// axis_lengths.h.  Compiled once per precision (GPUFFT_AXIS_F64 0, 1) and part
// of the list (GPUFFT_AXIS_PART).
#include "axis_lengths.h"
#include "fft_axis.cuh"

namespace gpufft {
namespace axis {

#define GPUFFT_JOIN2(a, b) a##b
#define GPUFFT_JOIN(a, b) GPUFFT_JOIN2(a, b)
#if GPUFFT_AXIS_F64
using Real = double;
#define GPUFFT_AXIS_TABLE GPUFFT_JOIN(kKernels_f64_, GPUFFT_AXIS_PART)
#else
using Real = float;
#define GPUFFT_AXIS_TABLE GPUFFT_JOIN(kKernels_f32_, GPUFFT_AXIS_PART)
#endif

static const Kernels kLengths[] = {GPUFFT_JOIN(GPUFFT_AXIS_LENGTHS_, GPUFFT_AXIS_PART)(GPUFFT_AXIS_KERNELS)};
extern const KernelTable GPUFFT_AXIS_TABLE;
const KernelTable GPUFFT_AXIS_TABLE = {kLengths, sizeof(kLengths) / sizeof(kLengths[0])};

}  // namespace axis
}  // namespace gpufft
