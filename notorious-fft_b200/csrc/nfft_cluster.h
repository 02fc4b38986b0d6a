// nfft_cluster.h -- host interface of the cluster pass kernels (nfft_cluster.cuh).
#pragma once

#include "nfft_engine.h"

namespace nfft {

// Longest contiguous transform done in one sweep by a pair of CTAs (log2).
constexpr int CLUSTER_ROW = sizeof(real_t) == 8 ? 13 : 14;

// Plain complex pass of radix 2^logR with column (1) or row (0) loads / stores.
bool cluster_available(int logR, int ci, int co);
bool launch_cluster(PassArgs a, int ci, int co, cudaStream_t s);
bool cluster_set_attributes();

}  // namespace nfft
