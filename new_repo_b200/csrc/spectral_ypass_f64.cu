// The FP64 kernels of spectral_ypass.cu.
#define LES_YPASS_DOUBLE
#include "spectral_ypass.cu"
