// Line kernels of the FFTs (fft_pencil.cuh), lengths 24, 44, 84, 126, 180, 252.
#include "fft_pencil.cuh"

#define QBX_LENGTHS(X) X(24) X(44) X(84) X(126) X(180) X(252)
QBX_PENCIL_FUNCTIONS(4, QBX_LENGTHS)
