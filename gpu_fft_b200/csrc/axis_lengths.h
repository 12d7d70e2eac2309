// axis_lengths.h — the axis lengths with kernels of their own (axis_fixed.cu):
// every length from 16 to 1024 with no prime factor above 7 that is R1 * R2
// with R1 >= R2 among the radices up to 32, R1 as small as it can be; in
// eight parts, one per compilation.
#pragma once

#define GPUFFT_AXIS_LENGTHS_0(X) \
    X(4, 4) X(8, 6) X(7, 7) X(14, 7) X(10, 10) X(14, 12) X(25, 7) X(18, 15) X(20, 14) X(27, 15) X(21, 20) X(28, 21) \
    X(25, 24) X(30, 27) X(30, 28)
#define GPUFFT_AXIS_LENGTHS_1(X) \
    X(6, 3) X(9, 5) X(10, 5) X(12, 8) X(15, 7) X(18, 9) X(15, 12) X(16, 16) X(18, 16) X(20, 20) X(24, 18) X(24, 24) \
    X(25, 25) X(32, 25) X(32, 27)
#define GPUFFT_AXIS_LENGTHS_2(X) \
    X(5, 4) X(7, 6) X(9, 6) X(10, 9) X(12, 9) X(16, 10) X(21, 9) X(18, 14) X(21, 14) X(28, 14) X(21, 21) X(27, 21) \
    X(30, 21) X(28, 28) X(32, 28)
#define GPUFFT_AXIS_LENGTHS_3(X) \
    X(7, 3) X(8, 5) X(8, 7) X(12, 7) X(14, 8) X(15, 10) X(16, 12) X(25, 10) X(20, 15) X(24, 16) X(28, 16) X(28, 20) \
    X(32, 20) X(32, 24) X(30, 30)
#define GPUFFT_AXIS_LENGTHS_4(X) \
    X(6, 4) X(6, 6) X(10, 6) X(9, 9) X(12, 10) X(21, 7) X(14, 14) X(27, 9) X(21, 15) X(21, 18) X(25, 18) X(27, 20) \
    X(27, 24) X(28, 27) X(32, 30)
#define GPUFFT_AXIS_LENGTHS_5(X) \
    X(5, 5) X(7, 5) X(9, 7) X(10, 8) X(25, 5) X(12, 12) X(20, 10) X(16, 15) X(20, 16) X(25, 15) X(24, 20) X(25, 21) \
    X(28, 24) X(30, 25) X(32, 32)
#define GPUFFT_AXIS_LENGTHS_6(X) \
    X(9, 3) X(8, 4) X(8, 8) X(15, 5) X(14, 9) X(14, 10) X(15, 14) X(15, 15) X(18, 18) X(20, 18) X(27, 18) X(32, 16) \
    X(27, 25) X(27, 27)
#define GPUFFT_AXIS_LENGTHS_7(X) \
    X(7, 4) X(6, 5) X(10, 7) X(9, 8) X(16, 8) X(15, 9) X(18, 12) X(16, 14) X(21, 16) X(25, 14) X(25, 20) X(24, 21) \
    X(28, 25) X(30, 24)
