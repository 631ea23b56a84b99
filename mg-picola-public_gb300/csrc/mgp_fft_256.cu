// Transforms of 256^3 meshes (mgp_fft.cuh).
#include "mgp_fft.cuh"

MGP_FFT_OPS(256)
