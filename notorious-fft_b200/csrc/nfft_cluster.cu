// nfft_cluster.cu -- instantiation and launch of the cluster pass kernels.
#include "nfft_cluster.cuh"
#include "nfft_cluster.h"

namespace nfft {

namespace {
struct ClusterEntry {
    int logR, ci, co;
    const void* fn;
    size_t smem;
    int logJ, threads, size;
};
template <int LOGR, int LOGC, bool CI, bool CO> ClusterEntry cluster_entry() {
    using K = Cluster<real_t, LOGR, LOGC, CI, CO>;
    return ClusterEntry{LOGR, CI, CO, (const void*)cluster_kernel<real_t, LOGR, LOGC, CI, CO>,
                        cluster_smem_bytes<real_t, LOGR, LOGC, CI, CO>(), K::LOGJ, K::THREADS, K::C};
}
const std::vector<ClusterEntry>& cluster_table() {
    static const std::vector<ClusterEntry> tab = {
        cluster_entry<CLUSTER_ROW, 1, false, false>(), cluster_entry<10, 1, true, true>(), cluster_entry<11, 1, true, true>()};
    return tab;
}
const ClusterEntry* cluster_find(int logR, int ci, int co) {
    for (const ClusterEntry& e : cluster_table())
        if (e.logR == logR && e.ci == ci && e.co == co) return &e;
    return nullptr;
}
}  // namespace

bool cluster_available(int logR, int ci, int co) { return cluster_find(logR, ci, co) != nullptr; }

bool cluster_set_attributes() {
    for (const ClusterEntry& e : cluster_table())
        if (!cuda_ok(cudaFuncSetAttribute(e.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e.smem),
                     "cudaFuncSetAttribute(cluster pass)"))
            return false;
    return true;
}

bool launch_cluster(PassArgs a, int ci, int co, cudaStream_t s) {
    const ClusterEntry* e = cluster_find(a.logR, ci, co);
    if (!e) {
        set_error(6, "no cluster pass kernel for radix 2^%d", a.logR);
        return false;
    }
    a.logJ = e->logJ;
    const long long ntiles = (a.nlines + (1ll << a.logJ) - 1) >> a.logJ;
    if (ntiles <= 0) return true;
    if (ntiles * e->size > 0x7fffffffll) {
        set_error(6, "cluster pass of %lld tiles exceeds the grid", ntiles);
        return false;
    }
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)e->size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    // (two CTAs per SM: plain_launch() would keep none of these grids plain)
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ntiles * e->size), 1, 1);
    cfg.blockDim = dim3((unsigned)e->threads, 1, 1);
    cfg.dynamicSmemBytes = e->smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    void* args[] = {(void*)&a};
    note_launch();
    return cuda_ok(cudaLaunchKernelExC(&cfg, e->fn, args), "cluster pass kernel launch");
}

}  // namespace nfft
