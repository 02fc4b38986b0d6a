// nfft_blue.cuh -- Bluestein transforms whose padded length fits one tile.
//
// One kernel does the whole convolution of n points padded to M = 2^LOGM
// (M/4 < n <= M/2): chirp premultiply, M-point FFT, filter product, M-point
// inverse FFT, window and chirp postmultiply.  Against the general pass
// kernel's two runs over the tile it keeps the spectrum in registers between
// the two FFTs: the forward sub-stages run 16 first and end on radix rho, whose
// outputs of butterfly i are the points i + m M/rho -- exactly the inputs of
// butterfly i of an inverse that starts with radix rho.  So the inverse runs
// the schedule backwards, the filter product happens in registers, and the two
// FFTs of a tile take 2 (NS - 1) exchanges through shared memory.  The upper
// half of the padded input is zero and the upper half of the output is not
// wanted: both radix-16 end stages touch 8 points of 16.
//
// Bound: the SM's L1 / shared-memory data path (84% busy in double, 93% in float, at
// 1000 points; FP64 pipe 38%, DRAM 13%): two M-point FFTs, M >= 2n, with their
// exchanges and root loads per n points of traffic.  So tiles are the smallest that
// hold a line -- 2048 points and 128 threads up to M = 2048, four (FP64) or eight (FP32)
// CTAs per SM to overlap one tile's loads with another's arithmetic.
// B200, general kernel -> this one: FP64 1000 x 2000 160 -> 58 us, 300 x 5001
// 174 -> 55 us, 3000 x 500 191 -> 76 us, 230 x 7 33 -> 7 us; FP32 17 x 219837
// 210 -> 45 us, 500 x 4000 84 -> 29 us.
#pragma once

#include "nfft_lean.cuh"

namespace nfft {

// Radix-16 DFT of points 0..7 with points 8..15 zero.
template <typename T> NFFT_HD void dft16_lower(C2<T>* a) {
    using V = C2<T>;
    V b[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        const V x0 = a[n2], x1 = a[4 + n2], r1 = mul_mi(x1);
        b[n2][0] = cadd(x0, x1);
        b[n2][1] = cadd(x0, r1);
        b[n2][2] = csub(x0, x1);
        b[n2][3] = csub(x0, r1);
    }
    const T c = K<T>::c8, s = K<T>::s8;
    b[1][1] = cmul(b[1][1], mkc(c, -s));
    b[1][2] = mul_w8_1<T>(b[1][2]);
    b[1][3] = cmul(b[1][3], mkc(s, -c));
    b[2][1] = mul_w8_1<T>(b[2][1]);
    b[2][2] = mul_mi(b[2][2]);
    b[2][3] = mul_w8_3<T>(b[2][3]);
    b[3][1] = cmul(b[3][1], mkc(s, -c));
    b[3][2] = mul_w8_3<T>(b[3][2]);
    b[3][3] = cmul(b[3][3], mkc(-c, s));
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        V x0 = b[0][k1], x1 = b[1][k1], x2 = b[2][k1], x3 = b[3][k1];
        dft4(x0, x1, x2, x3);
        a[k1] = x0; a[k1 + 4] = x1; a[k1 + 8] = x2; a[k1 + 12] = x3;
    }
}

template <typename T, int LOGM, int LOGT, int LOAD, int STORE>
struct Blue {
    static constexpr int THREADS = 1 << LOGT;
    static constexpr int M = 1 << LOGM;
    static constexpr int LOGJ = LOGT + 4 - LOGM;
    static constexpr int J = 1 << LOGJ;
    static constexpr int NS = LeanSched<LOGM>::n;
    static constexpr int SMEM_ELEMS = NS > 1 ? lean_smem_elems<false, LOGM, LOGJ>() : 0;
    static_assert(LOGJ >= 0 && LOGJ <= LOGT, "a thread per line of the tile");

    // Sub-stage radices (log2): INV runs the forward schedule backwards.
    template <int S, bool INV> static constexpr int lr() { return LeanSched<LOGM>::lr[INV ? NS - 1 - S : S]; }
    template <int S, bool INV> static constexpr int lns() {
        int s = 0;
        for (int x = 0; x < S; ++x) s += LeanSched<LOGM>::lr[INV ? NS - 1 - x : x];
        return s;
    }
    static NFFT_HD int at(int l, int r) { return NFFT_SM((lean_idx<false, LOGM, LOGJ>(l, r))); }

    // Butterfly q of thread t in a sub-stage of radix 2^LR: line l, index i.
    template <int LR> static NFFT_HD void map(int t, int q, int& l, int& i) {
        lean_map<false, LOGJ>(t + q * THREADS, LOGM - LR, l, i);
    }

    // Points i + m M/16 (m < 8) of this thread's line, chirped; then the first
    // radix-16 DFT.
    static NFFT_HD void load(const PassArgs& a, const LeanLine* lines, int t, C2<T>* v) {
        int l, i;
        map<4>(t, 0, l, i);
        const LeanLine ln = lines[l];
        const int n = ln.j < 0 ? 0 : (int)a.N;
        const C2<T>* ch = (const C2<T>*)a.chirp + i;
        C2<T> c[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int p = i + (m << (LOGM - 4));
            c[m] = p < n ? gload_keep(ch + (m << (LOGM - 4))) : mkc((T)0, (T)0);
            if constexpr (LOAD == LD_BLUE) {
                v[m] = p < n ? NFFT_GLD((const C2<T>*)a.in + ln.bin + p) : mkc((T)0, (T)0);
            } else {
                const T* x = (const T*)a.in + ln.bin;
                T r = (T)0;
                if (p < n) {
                    if constexpr (LOAD == LD_BLUE_R) r = NFFT_GLD(x + p);
                    else r = p < (n + 1) / 2 ? NFFT_GLD(x + 2 * p) : NFFT_GLD(x + 2 * n - 1 - 2 * p);
                }
                v[m] = mkc(r, (T)0);
            }
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if constexpr (LOAD == LD_BLUE) {
                if (a.conj_in) v[m].y = -v[m].y;
                v[m] = cmul(v[m], c[m]);
            } else {
                v[m] = cscale(c[m], v[m].x);
            }
        }
        dft16_lower<T>(v);
    }

    template <int S, bool INV>
    static NFFT_HD void read(const C2<T>* sm, int t, C2<T>* v) {
        constexpr int LR = lr<S, INV>(), RHO = 1 << LR, lq = LOGM - LR;
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            int l, i;
            map<LR>(t, q, l, i);
#pragma unroll
            for (int m = 0; m < RHO; ++m) v[q * RHO + m] = sm[at(l, i + (m << lq))];
        }
    }
    // Twiddles and DFTs of sub-stage S.
    template <int S, bool INV>
    static NFFT_HD void dfts(const TwTables<T>* tw, int t, C2<T>* v) {
        constexpr int LR = lr<S, INV>(), RHO = 1 << LR, LNS = lns<S, INV>();
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            int l, i;
            map<LR>(t, q, l, i);
            // up to M = 64 there are at most 4 different k: few entries per load
            if constexpr (LNS > 0 && LOGM > 6) mul_roots<T, LR, LNS>(tw, i & ((1 << LNS) - 1), v + q * RHO);
            else if constexpr (LNS > 0) mul_table<T, LR, LNS>(tw, i & ((1 << LNS) - 1), v + q * RHO);
            dft_radix<T, RHO>(v + q * RHO);
        }
    }
    template <int S, bool INV>
    static NFFT_HD void write(C2<T>* sm, int t, const C2<T>* v) {
        constexpr int LR = lr<S, INV>(), RHO = 1 << LR, LNS = lns<S, INV>();
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            int l, i;
            map<LR>(t, q, l, i);
            const int o = ((i >> LNS) << (LNS + LR)) + (i & ((1 << LNS) - 1));
#pragma unroll
            for (int m = 0; m < RHO; ++m) sm[at(l, o + (m << LNS))] = v[q * RHO + m];
        }
    }
    // The forward FFT's last outputs, point i + m M/rho of butterfly i: filter
    // product, conjugation (the inverse runs as conj(FFT(conj))), and the
    // inverse's first sub-stage (radix rho, no twiddles).
    static NFFT_HD void filter(const PassArgs& a, int t, C2<T>* v) {
        constexpr int LR = lr<NS - 1, false>(), RHO = 1 << LR, lq = LOGM - LR;
        const C2<T>* f = (const C2<T>*)a.filt;
#pragma unroll
        for (int q = 0; q < 16 / RHO; ++q) {
            int l, i;
            map<LR>(t, q, l, i);
#pragma unroll
            for (int m = 0; m < RHO; ++m)
                v[q * RHO + m] = cconj(cmul(v[q * RHO + m], gload_keep(f + i + (m << lq))));
            dft_radix<T, RHO>(v + q * RHO);
        }
    }
    // Window, chirp postmultiply and store of points i + m M/16, m < 8.
    static NFFT_HD void store(const PassArgs& a, const LeanLine* lines, int t, const C2<T>* v) {
        int l, i;
        map<4>(t, 0, l, i);
        const LeanLine ln = lines[l];
        const int n = ln.j < 0 ? 0 : (STORE == ST_BLUE_R ? (int)(a.N / 2) + 1 : (int)a.N);
        const C2<T>* ch = (const C2<T>*)a.chirp + i;
        const T f = (T)a.scale, fi = a.conj_out ? -f : f;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int p = i + (m << (LOGM - 4));
            if (p >= n) continue;
            const C2<T> w = cmul(cconj(v[m]), gload_keep(ch + (m << (LOGM - 4))));
            if constexpr (STORE == ST_BLUE_T2) {
                const C2<T> e = NFFT_GLD((const C2<T>*)a.post + p);
                NFFT_GST((T*)a.out + ln.bout + p, (T)2 * (w.x * e.x - w.y * e.y) * f);
            } else {
                NFFT_GST((C2<T>*)a.out + ln.bout + p, mkc(w.x * f, w.y * fi));
            }
        }
    }
};

template <typename T, int LOGM, int LOGT, int LOAD, int STORE>
constexpr size_t blue_smem_bytes() {
    using B = Blue<T, LOGM, LOGT, LOAD, STORE>;
    return sizeof(C2<T>) * (size_t)B::SMEM_ELEMS + sizeof(LeanLine) * (size_t)B::J;
}

// One tile (all threads of the CTA call it; uniform early exit past the last line).
template <typename T, int LOGM, int LOGT, int LOAD, int STORE, bool PDL = false>
__device__ __forceinline__ void blue_tile(const PassArgs& a, long long tile, unsigned char* smraw) {
    using B = Blue<T, LOGM, LOGT, LOAD, STORE>;
    using V = C2<T>;
    V* sm = (V*)smraw;
    LeanLine* lines = (LeanLine*)(sm + B::SMEM_ELEMS);
    const TwTables<T>* tw = (const TwTables<T>*)a.tw;
    const int t = threadIdx.x;
    const long long line0 = tile << B::LOGJ;
    if (line0 >= a.nlines) {
        if constexpr (PDL) pdl_wait();
        return;
    }
    if (t < B::J) {
        long long tmp[3];
        line_setup(a, line0 + t, 0, TileLines{&tmp[0], &tmp[1], &tmp[2]});
        lines[t] = LeanLine{tmp[0], tmp[1], tmp[2]};
    }
    if constexpr (PDL) pdl_wait();
    __syncthreads();
    V v[16];
    B::load(a, lines, t, v);
    if constexpr (B::NS >= 2) {
        B::template write<0, false>(sm, t, v);
        __syncthreads();
        if constexpr (B::NS >= 3) {
            B::template read<1, false>(sm, t, v);
            __syncthreads();
            B::template dfts<1, false>(tw, t, v);
            B::template write<1, false>(sm, t, v);
            __syncthreads();
        }
        if constexpr (B::NS >= 4) {
            B::template read<2, false>(sm, t, v);
            __syncthreads();
            B::template dfts<2, false>(tw, t, v);
            B::template write<2, false>(sm, t, v);
            __syncthreads();
        }
        B::template read<B::NS - 1, false>(sm, t, v);
        __syncthreads();
        B::template dfts<B::NS - 1, false>(tw, t, v);
    }
    B::filter(a, t, v);
    if constexpr (B::NS >= 2) {
        B::template write<0, true>(sm, t, v);
        __syncthreads();
        if constexpr (B::NS >= 3) {
            B::template read<1, true>(sm, t, v);
            __syncthreads();
            B::template dfts<1, true>(tw, t, v);
            B::template write<1, true>(sm, t, v);
            __syncthreads();
        }
        if constexpr (B::NS >= 4) {
            B::template read<2, true>(sm, t, v);
            __syncthreads();
            B::template dfts<2, true>(tw, t, v);
            B::template write<2, true>(sm, t, v);
            __syncthreads();
        }
        B::template read<B::NS - 1, true>(sm, t, v);
        B::template dfts<B::NS - 1, true>(tw, t, v);
    }
    B::store(a, lines, t, v);
}

// Threads (log2) of the kernel for padded length 2^logM: the smallest tile
// (2048 points) that holds a line.
NFFT_HD constexpr int blue_logt(int logM) { return logM <= 11 ? 7 : logM - 4; }

template <typename T, int LOGM>
__global__ void __launch_bounds__(1 << blue_logt(LOGM), (lean_min_blocks<T, blue_logt(LOGM)>()))
blue_kernel(const PassArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const long long tile = (long long)blockIdx.x + (long long)blockIdx.y * gridDim.x;
    blue_tile<T, LOGM, blue_logt(LOGM), LD_BLUE, ST_BLUE, true>(a, tile, smraw);
}

}  // namespace nfft
