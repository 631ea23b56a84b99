// Transforms of 64^3 and 128^3 meshes (mgp_fft.cuh).
#include "mgp_fft.cuh"

MGP_FFT_OPS(64)
MGP_FFT_OPS(128)
