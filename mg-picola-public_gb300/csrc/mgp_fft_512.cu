// Transforms of 512^3 meshes (mgp_fft.cuh).
#include "mgp_fft.cuh"

MGP_FFT_OPS(512)
