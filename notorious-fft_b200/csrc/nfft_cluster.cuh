// nfft_cluster.cuh -- passes whose tile is shared by a cluster of CTAs.
//
// The same passes as nfft_lean.cuh (plain complex loads and stores) for the tiles
// of 128 KiB and more that one CTA can only hold alone on its SM: with one CTA
// per SM nothing overlaps its load, transform and store phases.  Here 2^LOGC CTAs
// hold a tile together, 64 KiB each, so every SM runs CTAs of two clusters and one
// tile's loads and stores overlap the other's arithmetic.
//
// A line of R points r = i + m R/16 is transformed as 16 x R/16 (decimation in
// frequency): a thread takes the 16 points of one i, does their radix-16 DFT and
// multiplies output m' by W_R^{i m'}; the R/16-point transforms over i of the 16
// sub-lines m' give the outputs k = m' + 16 k2.  CTA c of the cluster owns the
// sub-lines m' in [c 16/C, (c + 1) 16/C), so the one exchange after the first
// sub-stage crosses the cluster (distributed shared memory, (C - 1) / C of the
// points) and everything after it stays in the CTA.  Its outputs come in runs of
// 16/C consecutive points (rows) or J consecutive lines (columns).
//
// Pairs (C = 2) are what the library runs: half of the points cross, well below
// what distributed shared memory moves (about 26 bytes per ns and SM).  Bound: the
// latency of a tile's phases (two tiles per SM; L1 / shared-memory data path 52 - 57%
// busy, FP64 pipe 25 - 33%, DRAM 28 - 39%; loads and barriers are the stalls).  B200, the plain kernels
// (one CTA per SM, or two passes) -> these: FP64 8192 x 2000 165 -> 147 us, x 100
// 11.6 -> 11.3, 2048 x 2048 72 -> 66, 16 of 1024 x 1024 250 -> 225, 7 of 1024 x 128
// 18.5 -> 16; FP32 16384 x 1001 95 -> 90, 3 of 2048 x 2048 123 -> 112, 10 of
// 1024 x 1024 100 -> 89.  Clusters of four (FP64 2^14, FP32 2^15 in one sweep) lose to
// two passes on full batches (174 and 172 us, 210 and 187), and rows whose exchange
// scatters single points (a column layout for them) do too (FP32 16384 x 1001 127).
#pragma once

#include "nfft_lean.cuh"

namespace nfft {

// Cluster primitives.  A barrier's arrive releases and its wait acquires memory at
// cluster scope; cluster_addr is the address of this CTA's shared object p in CTA
// `rank`'s shared memory.
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r = 0;
#if defined(__CUDA_ARCH__)
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
#endif
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
#if defined(__CUDA_ARCH__)
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
#endif
}
__device__ __forceinline__ void cluster_wait() {
#if defined(__CUDA_ARCH__)
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
#endif
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, unsigned rank) {
    uint32_t r = 0;
#if defined(__CUDA_ARCH__)
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
#endif
    return r;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, double2 v) {
#if defined(__CUDA_ARCH__)
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
#endif
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float2 v) {
#if defined(__CUDA_ARCH__)
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
#endif
}

template <typename T, int LOGR, int LOGC, bool COL_IN, bool COL_OUT>
struct Cluster {
    static constexpr int LOGT = sizeof(T) == 8 ? 8 : 9;   // 64 KiB of points per CTA
    static constexpr int THREADS = 1 << LOGT, C = 1 << LOGC;
    using Whole = Lean<T, LOGR, LOGT + LOGC, COL_IN, COL_OUT, LD_C, ST_C>;   // the tile as one CTA's
    using Sub = Lean<T, LOGR - 4, LOGT, true, true, LD_C, ST_C>;             // the CTA's sub-lines
    static constexpr int LOGJ = Whole::LOGJ, J = Whole::J;
    static constexpr int LOGM = 4 - LOGC;                 // sub-lines of a line per CTA (log2)
    static constexpr int NS = Sub::NS;
    // column tiles [r][sub-line], pitch odd; row tiles [sub-line][r], one pad point
    // every 16 and the pitch odd: the exchange then writes runs of neighbouring
    // points into the other CTA, and both walks stay free of bank conflicts
    static constexpr int R2 = 1 << (LOGR - 4), PITCH = R2 + R2 / 16 + 1;
    static constexpr bool COLL = COL_OUT;
    static constexpr int SMEM_ELEMS = COLL ? Sub::SMEM_ELEMS : Sub::J * PITCH;
    static_assert(LOGM + LOGJ == Sub::LOGJ, "the CTA's sub-lines fill its tile");
    static_assert(NS >= 2 && NS <= 3 && J <= THREADS, "sub-stages of the sub-lines");

    // sub-line of output class m' (its low LOGM bits) of line l, and back: stores walk
    // sub-lines fastest, so rows keep m' and columns keep lines adjacent
    static NFFT_HD int sub_of(int l, int mp) {
        const int ml = mp & ((1 << LOGM) - 1);
        return COL_OUT ? (ml << LOGJ) + l : (l << LOGM) + ml;
    }
    static NFFT_HD void of_sub(int s, int& l, int& ml) {
        if constexpr (COL_OUT) { l = s & (J - 1); ml = s >> LOGJ; }
        else { ml = s & ((1 << LOGM) - 1); l = s >> LOGM; }
    }
    static NFFT_HD int at(int s, int r) {
        if constexpr (COLL) return NFFT_SM((lean_idx<true, LOGR - 4, Sub::LOGJ>(s, r)));
        else return NFFT_SM(s * PITCH + spad(r));
    }
    template <int S, bool COLMAP>
    static NFFT_HD void read(const C2<T>* sm, int t, int q, C2<T>* v, int& s, int& i) {
        constexpr int LR = LeanSched<LOGR - 4>::lr[S], lq = LOGR - 4 - LR;
        lean_map<COLMAP, Sub::LOGJ>(t + q * THREADS, lq, s, i);
#pragma unroll
        for (int m = 0; m < (1 << LR); ++m) v[m] = sm[at(s, i + (m << lq))];
    }
    template <int S>
    static NFFT_HD void write(C2<T>* sm, int s, int i, const C2<T>* v) {
#pragma unroll
        for (int m = 0; m < (1 << LeanSched<LOGR - 4>::lr[S]); ++m) sm[at(s, Sub::template out_pos<S>(i, m))] = v[m];
    }

    // Thread t of CTA c: its 16 points of one line, the radix-16 DFT and W_R^{i m'}.
    static NFFT_HD void load(const PassArgs& a, const TwTables<T>* tw, const LeanLine* lines, int c, int t, C2<T>* v,
                             int& l, int& i) {
        lean_map<COL_IN, LOGJ>((c << LOGT) + t, LOGR - 4, l, i);
        const LeanLine ln = lines[l];
        if (ln.j < 0) {
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = mkc((T)0, (T)0);
            return;
        }
        const long long rs = a.in_estride << a.logNj, s16 = rs << (LOGR - 4);
        const C2<T>* src = (const C2<T>*)a.in + ln.bin + ln.j * a.in_estride + (long long)i * rs;
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = NFFT_GLD(src + m * s16);
        if (a.conj_in) {
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m].y = -v[m].y;
        }
        Whole::pre_twiddle_dft(a, tw, ln.j, i, v);
        if constexpr (sizeof(T) == 4) {
            mul_roots<T, 4, LOGR - 4>(tw, i, v);   // W_R^{i m'}
        } else {
            // double: two roots and their products (six roots from the tables cost
            // 6% of the kernel, L1 is as busy as the FP64 pipe)
            const C2<T> w1 = table_root<T, LOGR>(tw, (uint32_t)i), w4 = table_root<T, LOGR>(tw, (uint32_t)(4 * i));
            C2<T> lo[4], hi = w4;
            lo[1] = w1;
            lo[2] = cmul(w1, w1);
            lo[3] = cmul(lo[2], w1);
#pragma unroll
            for (int m = 1; m < 4; ++m) v[m] = cmul(v[m], lo[m]);
#pragma unroll
            for (int h = 4; h < 16; h += 4) {
                v[h] = cmul(v[h], hi);
#pragma unroll
                for (int m = 1; m < 4; ++m) v[h + m] = cmul(v[h + m], cmul(hi, lo[m]));
                if (h < 12) hi = cmul(hi, w4);
            }
        }
    }
    // First sub-stage of the sub-lines: radix 16, no twiddles.
    static NFFT_HD void first(const C2<T>* sm, int t, C2<T>* v, int& s, int& i) {
        lean_map<COLL, Sub::LOGJ>(t, LOGR - 8, s, i);
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = sm[at(s, i + (m << (LOGR - 8)))];
        dft16<T>(v);
    }
    // Last sub-stage's outputs k2 of sub-line s: points k = m' + 16 k2 of its line.
    template <int S>
    static NFFT_HD void store(const PassArgs& a, const LeanLine* lines, int c, int s, int i, const C2<T>* v) {
        constexpr int RHO = 1 << LeanSched<LOGR - 4>::lr[S];
        int l, ml;
        of_sub(s, l, ml);
        const LeanLine ln = lines[l];
        if (ln.j < 0) return;
        const int logNso = a.logNs_out;
        const long long base = ((ln.j >> logNso) << (logNso + LOGR)) + (ln.j & ((1ll << logNso) - 1));
        const int k0 = (c << LOGM) + ml + (Sub::template out_pos<S>(i, 0) << 4);
        const long long rs = a.out_estride << logNso, ms = rs << (Sub::template lns_of<S>() + 4);
        C2<T>* dst = (C2<T>*)a.out + ln.bout + base * a.out_estride + (long long)k0 * rs;
        const T f = (T)a.scale, fi = a.conj_out ? -f : f;
#pragma unroll
        for (int m = 0; m < RHO; ++m) NFFT_GST(dst + m * ms, mkc(v[m].x * f, v[m].y * fi));
    }
};

template <typename T, int LOGR, int LOGC, bool COL_IN, bool COL_OUT>
constexpr size_t cluster_smem_bytes() {
    using K = Cluster<T, LOGR, LOGC, COL_IN, COL_OUT>;
    return sizeof(C2<T>) * (size_t)K::SMEM_ELEMS + sizeof(LeanLine) * (size_t)K::J;
}

template <typename T, int LOGR, int LOGC, bool COL_IN, bool COL_OUT>
__global__ void __launch_bounds__(sizeof(T) == 8 ? 256 : 512, 2) cluster_kernel(const PassArgs a) {
    using K = Cluster<T, LOGR, LOGC, COL_IN, COL_OUT>;
    using V = C2<T>;
    extern __shared__ __align__(16) unsigned char smraw[];
    V* sm = (V*)smraw;
    LeanLine* lines = (LeanLine*)(sm + K::SMEM_ELEMS);
    const TwTables<T>* tw = (const TwTables<T>*)a.tw;
    const int t = threadIdx.x;
    const int c = (int)cluster_rank();
    const long long tile = (long long)blockIdx.x >> LOGC;   // every CTA of the grid has a tile
    if (t < K::J) {
        long long tmp[3];
        line_setup(a, (tile << K::LOGJ) + t, 0, TileLines{&tmp[0], &tmp[1], &tmp[2]});
        lines[t] = LeanLine{tmp[0], tmp[1], tmp[2]};
    }
    cluster_arrive();   // every CTA of the cluster runs before any writes to its memory
    pdl_wait();
    __syncthreads();
    V v[16];
    int l, i;
    K::load(a, tw, lines, c, t, v, l, i);
    cluster_wait();
#pragma unroll
    for (int m = 0; m < 16; ++m)
        cluster_store(cluster_addr(sm, m >> K::LOGM) + (uint32_t)(sizeof(V) * K::at(K::sub_of(l, m), i)), v[m]);
    cluster_arrive();   // the sub-lines are complete; no writes to other CTAs after this
    cluster_wait();
    int s;
    K::first(sm, t, v, s, i);
    __syncthreads();
    K::template write<0>(sm, s, i, v);
    __syncthreads();
    if constexpr (K::NS >= 3) {
        constexpr int S = 1, RHO = 1 << LeanSched<LOGR - 4>::lr[S];
        V w[16];
        int ls[16 / RHO], is[16 / RHO];
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) K::template read<S, K::COLL>(sm, t, q, &w[q * RHO], ls[q], is[q]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            K::Sub::template twiddle_dft<S>(tw, is[q], &w[q * RHO]);
            K::template write<S>(sm, ls[q], is[q], &w[q * RHO]);
        }
        __syncthreads();
    }
    {
        constexpr int S = K::NS - 1, RHO = 1 << LeanSched<LOGR - 4>::lr[S];
        V w[16];
        int ls[16 / RHO], is[16 / RHO];
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) K::template read<S, true>(sm, t, q, &w[q * RHO], ls[q], is[q]);
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            K::Sub::template twiddle_dft<S>(tw, is[q], &w[q * RHO]);
            K::template store<S>(a, lines, c, ls[q], is[q], &w[q * RHO]);
        }
    }
}

}  // namespace nfft
