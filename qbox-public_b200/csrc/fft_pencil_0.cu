// Line kernels of the FFTs (fft_pencil.cuh), lengths 16, 64, 66, 144, 154.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(16) X(64) X(66) X(144) X(154)
QBX_PENCIL_FUNCTIONS(0, QBX_LENGTHS)
