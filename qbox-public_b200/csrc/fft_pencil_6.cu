// Line kernels of the FFTs (fft_pencil.cuh), lengths 30, 40, 90, 112, 198, 224.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(30) X(40) X(90) X(112) X(198) X(224)
QBX_PENCIL_FUNCTIONS(6, QBX_LENGTHS)
