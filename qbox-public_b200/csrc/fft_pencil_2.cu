// Line kernels of the FFTs (fft_pencil.cuh), lengths 20, 56, 72, 132, 168.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(20) X(56) X(72) X(132) X(168)
QBX_PENCIL_FUNCTIONS(2, QBX_LENGTHS)
