// Line kernels of the FFTs (fft_pencil.cuh), lengths 28, 42, 88, 120, 192, 240.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(28) X(42) X(88) X(120) X(192) X(240)
QBX_PENCIL_FUNCTIONS(5, QBX_LENGTHS)
