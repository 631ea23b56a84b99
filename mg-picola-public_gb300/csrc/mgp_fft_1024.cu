// Transforms of 1024^3 meshes (mgp_fft.cuh).
#include "mgp_fft.cuh"

MGP_FFT_OPS(1024)
