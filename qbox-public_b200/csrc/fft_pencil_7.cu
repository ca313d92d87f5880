// Line kernels of the FFTs (fft_pencil.cuh), lengths 32, 36, 96, 110, 210, 220.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(32) X(36) X(96) X(110) X(210) X(220)
QBX_PENCIL_FUNCTIONS(7, QBX_LENGTHS)
