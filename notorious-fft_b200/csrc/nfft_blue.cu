// nfft_blue.cu -- instantiation and launch of the single-tile Bluestein kernels.
#include "nfft_blue.cuh"
#include "nfft_blue.h"

namespace nfft {

namespace {
struct BlueEntry {
    void (*fn)(const PassArgs) = nullptr;
    size_t smem = 0;
    int per_sm = 1;
};
template <int LOGM> BlueEntry blue_entry() {
    return BlueEntry{blue_kernel<real_t, LOGM>, blue_smem_bytes<real_t, LOGM, blue_logt(LOGM), LD_BLUE, ST_BLUE>(),
                     lean_min_blocks<real_t, blue_logt(LOGM)>()};
}
const BlueEntry* blue_find(int logM) {
    static const BlueEntry tab[] = {blue_entry<4>(), blue_entry<5>(), blue_entry<6>(), blue_entry<7>(), blue_entry<8>(),
                                    blue_entry<9>(), blue_entry<10>(), blue_entry<11>(), blue_entry<12>(),
                                    blue_entry<13>()};
    return logM >= BLUE_MIN_LOGM && logM <= BLUE_MAX_LOGM ? &tab[logM - BLUE_MIN_LOGM] : nullptr;
}
}  // namespace

bool blue_set_attributes() {
    for (int k = BLUE_MIN_LOGM; k <= BLUE_MAX_LOGM; ++k) {
        const BlueEntry* e = blue_find(k);
        if (!cuda_ok(cudaFuncSetAttribute((const void*)e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e->smem),
                     "cudaFuncSetAttribute(Bluestein tile)"))
            return false;
    }
    return true;
}

bool launch_blue(PassArgs a, cudaStream_t s) {
    const BlueEntry* e = blue_find(a.logR);
    if (!e) {
        set_error(6, "no Bluestein tile kernel for a padded length of 2^%d", a.logR);
        return false;
    }
    const int logT = blue_logt(a.logR);
    a.logJ = logT + 4 - a.logR;
    const long long ntiles = (a.nlines + (1ll << a.logJ) - 1) >> a.logJ;
    if (ntiles <= 0) return true;
    dim3 grid((unsigned)ntiles, 1, 1);
    if (ntiles > 0x7fffffffll) grid = dim3(0x7fffffffu, (unsigned)((ntiles + 0x7fffffffll - 1) / 0x7fffffffll), 1);
    void* args[] = {(void*)&a};
    return cuda_ok(launch_dependent((const void*)e->fn, grid, 1 << logT, e->smem, args, s, e->per_sm, false),
                   "Bluestein tile kernel launch");
}

}  // namespace nfft
