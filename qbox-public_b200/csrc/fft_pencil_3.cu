// Line kernels of the FFTs (fft_pencil.cuh), lengths 22, 48, 80, 128, 176, 256.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(22) X(48) X(80) X(128) X(176) X(256)
QBX_PENCIL_FUNCTIONS(3, QBX_LENGTHS)
