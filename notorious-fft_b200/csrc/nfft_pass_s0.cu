// One slice of the generic pass kernels (see nfft_pass_slice.cuh).
#define NFFT_PASS_SLICE 0
#include "nfft_pass_slice.cuh"
