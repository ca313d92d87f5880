// Line kernels of the FFTs (fft_pencil.cuh), lengths 18, 60, 70, 140, 160.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(18) X(60) X(70) X(140) X(160)
QBX_PENCIL_FUNCTIONS(1, QBX_LENGTHS)
