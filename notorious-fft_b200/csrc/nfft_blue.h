// nfft_blue.h -- host interface of the single-tile Bluestein kernels
// (nfft_blue.cuh): padded lengths 2^BLUE_MIN_LOGM .. 2^BLUE_MAX_LOGM.
#pragma once

#include "nfft_engine.h"

namespace nfft {

constexpr int BLUE_MIN_LOGM = 4, BLUE_MAX_LOGM = 13;

// All of a.nlines transforms (padded length 2^a.logR, contiguous lines).
bool launch_blue(PassArgs a, cudaStream_t s);
bool blue_set_attributes();

}  // namespace nfft
