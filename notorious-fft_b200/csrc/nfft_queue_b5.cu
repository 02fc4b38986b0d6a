// nfft_queue_b5.cu -- queue kernel branches: single-tile Bluestein transforms.
#include "nfft_engine.h"
#include "nfft_queue_branches.cuh"

namespace nfft {

#define X(M, LD, ST) \
    template __device__ void qb_blue<real_t, M, LD, ST>(const QDesc*, long long, int, unsigned char*);
NFFT_QUEUE_BLUE(X)
#undef X

}  // namespace nfft
