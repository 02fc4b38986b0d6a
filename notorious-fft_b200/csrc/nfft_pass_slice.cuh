// nfft_pass_slice.cuh -- instantiates one slice of the generic pass kernels
// (NFFT_PASS_SLICE of NFFT_PASS_SLICES) so the build compiles them in parallel.
#pragma once

#include "nfft_engine.h"

namespace nfft {

using PassFn = void (*)(const PassArgs);
constexpr int NFFT_PASS_SLICES = 4;

// Valid (load, store) operator pairs.  Others are never planned.
#define NFFT_PAIRS(X)          \
    X(LD_C, ST_C)              \
    X(LD_C, ST_R)              \
    X(LD_C, ST_T2)             \
    X(LD_C, ST_T3)             \
    X(LD_C, ST_T4)             \
    X(LD_C, ST_BLUE)           \
    X(LD_T2, ST_C)             \
    X(LD_T2, ST_T2)            \
    X(LD_T3, ST_C)             \
    X(LD_T3, ST_T3)            \
    X(LD_IR, ST_C)             \
    X(LD_T4, ST_C)             \
    X(LD_T4, ST_T4)            \
    X(LD_BLUE, ST_C)           \
    X(LD_BLUE, ST_BLUE)        \
    X(LD_R2C, ST_C)            \
    X(LD_R2C, ST_R)            \
    X(LD_C, ST_C2R)            \
    X(LD_IR, ST_C2R)           \
    X(LD_FILT, ST_C)

template <bool ON, int LD, int ST>
struct PassReg {
    static void add(PassFn (*)[NUM_STORE_OPS], PassFn (*)[NUM_STORE_OPS]) {}
};
template <int LD, int ST>
struct PassReg<true, LD, ST> {
    static void add(PassFn (*t12)[NUM_STORE_OPS], PassFn (*t13)[NUM_STORE_OPS]) {
        t12[LD][ST] = pass_kernel<real_t, 12, LD, ST>;
        t13[LD][ST] = pass_kernel<real_t, 13, LD, ST>;
    }
};

#define NFFT_CAT2(a, b) a##b
#define NFFT_CAT(a, b) NFFT_CAT2(a, b)
#define X(L, S) PassReg<(__COUNTER__ % NFFT_PASS_SLICES) == NFFT_PASS_SLICE, L, S>::add(t12, t13);

void NFFT_CAT(pass_register_slice_, NFFT_PASS_SLICE)(PassFn (*t12)[NUM_STORE_OPS], PassFn (*t13)[NUM_STORE_OPS]) {
    NFFT_PAIRS(X)
}
#undef X

}  // namespace nfft
