// The FP64 kernels of spectral_xinv.cu.
#define LES_XINV_DOUBLE
#include "spectral_xinv.cu"
