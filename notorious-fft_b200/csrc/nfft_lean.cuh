// nfft_lean.cuh -- the specialized pass kernel (hot path).
//
// Same Stockham pass semantics as pass_kernel (nfft_pass.cuh), with the pass
// radix R = 2^LOGR and the tile shape fixed at compile time:
//  * the first sub-stage is radix 16 and reads its 16 points per thread
//    straight from global memory (no shared-memory staging), with the pass
//    pre-twiddle W_{Ns R}^{r k} generated per line from two table roots and
//    a depth-4 product tree;
//  * middle sub-stages exchange through shared memory;
//  * the last sub-stage writes its outputs straight to global memory, except
//    for the paired real operators, which need whole lines in shared memory.
// Thread-to-butterfly mappings are chosen per sub-stage so that global
// accesses coalesce: "column" mode walks consecutive lines (J adjacent
// Stockham lines or a unit-stride batch dim), "row" mode walks along a line.
// Column tiles are stored [r][line] with a pitch of J+1 points, row tiles
// [line][r] with one pad point every 16, which keeps both mappings free of
// shared-memory bank conflicts.
#pragma once

#include "nfft_pass.cuh"

namespace nfft {

// Sub-stage radices (log2) of a pass of radix 2^LOGR: radix 16 first.
template <int LOGR> struct LeanSched;
template <> struct LeanSched<4> { static constexpr int n = 1; static constexpr int lr[4] = {4, 0, 0, 0}; };
template <> struct LeanSched<5> { static constexpr int n = 2; static constexpr int lr[4] = {4, 1, 0, 0}; };
template <> struct LeanSched<6> { static constexpr int n = 2; static constexpr int lr[4] = {4, 2, 0, 0}; };
template <> struct LeanSched<7> { static constexpr int n = 2; static constexpr int lr[4] = {4, 3, 0, 0}; };
template <> struct LeanSched<8> { static constexpr int n = 2; static constexpr int lr[4] = {4, 4, 0, 0}; };
template <> struct LeanSched<9> { static constexpr int n = 3; static constexpr int lr[4] = {4, 3, 2, 0}; };
template <> struct LeanSched<10> { static constexpr int n = 3; static constexpr int lr[4] = {4, 4, 2, 0}; };
template <> struct LeanSched<11> { static constexpr int n = 3; static constexpr int lr[4] = {4, 4, 3, 0}; };
template <> struct LeanSched<12> { static constexpr int n = 3; static constexpr int lr[4] = {4, 4, 4, 0}; };
template <> struct LeanSched<13> { static constexpr int n = 4; static constexpr int lr[4] = {4, 4, 3, 2}; };

// Shared-memory index of point r of tile line l.
template <bool COL, int LOGR, int LOGJ>
NFFT_HD int lean_idx(int l, int r) {
    if constexpr (COL) return r * ((1 << LOGJ) + 1) + l;
    else return spad((l << LOGR) + r);
}
template <bool COL, int LOGR, int LOGJ> constexpr int lean_smem_elems() {
    return COL ? (1 << LOGR) * ((1 << LOGJ) + 1) : ((1 << (LOGR + LOGJ)) + (1 << (LOGR + LOGJ - 4)) + 1);
}

// Butterfly b of a sub-stage with B = 2^lb butterflies per line -> (line, i).
// Column mapping: lines fastest; row mapping: butterflies fastest.
template <bool COLMAP, int LOGJ>
NFFT_HD void lean_map(int b, int lb, int& l, int& i) {
    if constexpr (COLMAP) { l = b & ((1 << LOGJ) - 1); i = b >> LOGJ; }
    else { i = b & ((1 << lb) - 1); l = b >> lb; }
}

// x^0 .. x^15 by a depth-4 product tree.
template <typename T>
NFFT_HD void powers16(C2<T> x, C2<T>* p) {
    p[0] = mkc((T)1, (T)0);
    p[1] = x;
    p[2] = cmul(x, x);
    p[3] = cmul(p[2], x);
    p[4] = cmul(p[2], p[2]);
    p[8] = cmul(p[4], p[4]);
    p[12] = cmul(p[8], p[4]);
#pragma unroll
    for (int a = 4; a < 16; a += 4) {
        p[a + 1] = cmul(p[a], x);
        p[a + 2] = cmul(p[a], p[2]);
        p[a + 3] = cmul(p[a], p[3]);
    }
}

// W_{2^LOGP}^q from the tables, one entry where the order allows.
template <typename T, int LOGP>
NFFT_HD C2<T> table_root(const TwTables<T>* tw, uint32_t q) {
    if constexpr (LOGP <= TW_BITS) return twiddle_small<T>(tw, q, LOGP);
    else return twiddle<T>(tw, (uint64_t)q, LOGP);
}

// W_{2^logP}^k for a run of k that agree in their low logP - 12 bits: the factor of
// those bits is made once, each root is one entry of the first table times it, with
// the roundings of twiddle().  mirror() gives W^{K - k} for a K whose low bits are zero.
template <typename T>
struct RootRun {
    C2<T> low;
    int logP;
    bool has;
    NFFT_HD void start(const TwTables<T>* tw, long long k, int logP_) {
        logP = logP_;
        const uint64_t u = (uint64_t)k << (36 - logP);
        const uint32_t i1 = (uint32_t)(u >> TW_BITS) & (TW_SIZE - 1), i2 = (uint32_t)u & (TW_SIZE - 1);
        has = i1 || i2;
        low = i1 ? tw_load<T>(tw, 1, i1) : mkc((T)1, (T)0);
        if (i2) low = cmul(low, tw_load<T>(tw, 2, i2));
    }
    NFFT_HD uint32_t digit(long long k) const { return (uint32_t)(((uint64_t)k << (36 - logP)) >> (2 * TW_BITS)); }
    NFFT_HD C2<T> at(const TwTables<T>* tw, long long k) const {
        const C2<T> w = tw_load<T>(tw, 0, digit(k) & (TW_SIZE - 1));
        return has ? cmul(w, low) : w;
    }
    NFFT_HD C2<T> mirror(const TwTables<T>* tw, long long K, long long k) const {
        const C2<T> w = tw_load<T>(tw, 0, (digit(K) - digit(k)) & (TW_SIZE - 1));
        return has ? cmulc(w, low) : w;
    }
};

// v[m] *= W_{2^(LNS + LR)}^{m k}, m < 2^LR (the internal twiddles of a
// sub-stage): the roots of m = 1, 2, 3 and of the multiples of 4 from the
// tables (L1 hits), the others as one product of two of them -- one rounding
// more than a lookup, where a tree from the first root alone has up to four.
// Reading all of them is slower (Bluestein FP64 1000 x 2000: 84 us, 58 us so).
// The plain passes keep the tree: their tiles are bound by L1 as much as by HBM
// (B200, FP64 4096 x 256 both ways 20.5 us with the tree, 24.6 with these loads;
// FP32 8192 x 2000 79 and 92; radices below 16 alone, FP64 1024 x 1024 x 16 258
// and 266).
template <typename T, int LR, int LNS>
NFFT_HD void mul_roots(const TwTables<T>* tw, int k, C2<T>* v) {
    constexpr int RHO = 1 << LR;
    C2<T> lo[4];
#pragma unroll
    for (int m = 1; m < (RHO < 4 ? RHO : 4); ++m) {
        lo[m] = table_root<T, LNS + LR>(tw, (uint32_t)(m * k));
        v[m] = cmul(v[m], lo[m]);
    }
#pragma unroll
    for (int h = 4; h < RHO; h += 4) {
        const C2<T> w = table_root<T, LNS + LR>(tw, (uint32_t)(h * k));
        v[h] = cmul(v[h], w);
#pragma unroll
        for (int m = 1; m < 4; ++m) v[h + m] = cmul(v[h + m], cmul(w, lo[m]));
    }
}

// The same with every root from the tables: for column tiles, where the lines of a
// tile share k and a warp reads few entries at a time.
template <typename T, int LR, int LNS>
NFFT_HD void mul_table(const TwTables<T>* tw, int k, C2<T>* v) {
#pragma unroll
    for (int m = 1; m < (1 << LR); ++m) v[m] = cmul(v[m], table_root<T, LNS + LR>(tw, (uint32_t)(m * k)));
}

// Per-line state held by every thread of the line.
struct LeanLine {
    long long bin, bout, j;
};

// ---- mirror tiles: the last pass of a multi-pass realdft / DCT-2 / DST-2 ------
// The last pass of the packed N/2-point spectrum Z (M = N/2) writes, for line j
// of the ns = M / R lines of a transform, Z[j + r ns], r < R.  Bin k pairs with
// bin M - k, which lives on line ns - j (lines 0 and ns / 2 pair with
// themselves).  A mirror tile therefore holds J/2 "low" lines and their J/2
// partners: tile tt of a transform holds j = tt J/2 + l and ns - (tt J/2 + l)
// for l < J/2, except tile 0, whose first low line is j = 0 and first high line
// j = ns / 2.  The Hermitian unpack then runs inside the tile.
//
// Stockham line of local line l (of J) in tile tt of a transform.
NFFT_HD long long mirror_line(long long tt, int l, int J, long long ns) {
    const int h = J / 2;
    if (l < h) return (tt == 0 && l == 0) ? 0 : tt * h + l;
    const int u = l - h;
    if (tt == 0) return u == 0 ? ns / 2 : ns - u;
    return ns - (tt * h + u);
}
// Local line of Stockham line j in tile tt (inverse of mirror_line).
NFFT_HD int mirror_local(long long tt, long long j, int J, long long ns) {
    const int h = J / 2;
    if (tt == 0) {
        if (j == 0) return 0;
        if (j == ns / 2) return h;
        return j < ns / 2 ? (int)j : (int)(h + (ns - j));
    }
    return j < ns / 2 ? (int)(j - tt * h) : (int)(h + (ns - j - tt * h));
}
// Bin k of unpack item (l < J/2, r < R) of tile tt: every item emits bins k and
// M - k (unpack_pair), the items of a tile cover both lines of each pair.
NFFT_HD long long mirror_item_k(long long tt, int l, int r, int R, long long ns, long long lowj) {
    if (tt == 0 && l == 0) return r < R / 2 ? (long long)r * ns : ns / 2 + (long long)(r - R / 2) * ns;
    return lowj + (long long)r * ns;
}

template <typename T, int LOGR, int LOGT, bool COL_IN, bool COL_OUT, int LOAD, int STORE>
struct Lean {
    static constexpr int THREADS = 1 << LOGT;
    static constexpr int LOGTILE = LOGT + 4;
    static constexpr int LOGJ = LOGTILE - LOGR;
    static constexpr int J = 1 << LOGJ;
    static constexpr int R = 1 << LOGR;
    static constexpr int LOGR_ = LOGR;
    static constexpr bool COL_OUT_ = COL_OUT;
    static constexpr bool PAIRED = (STORE == ST_R || STORE == ST_T2);
    // shared layout: column tiles whenever either side walks lines
    static constexpr bool COLL = COL_IN || COL_OUT;
    static constexpr int NS = LeanSched<LOGR>::n;
    static constexpr int SMEM_ELEMS = lean_smem_elems<COLL, LOGR, LOGJ>();
    static_assert(LOGJ >= 0 && LOGJ <= 8, "tile must hold 1..256 lines");
    // whole lines in a column tile: a real-to-real transform along a strided
    // axis, in one pass
    static constexpr bool WHOLE_COL = COL_IN && COL_OUT && (LOAD == LD_T2 || LOAD == LD_T3 || LOAD == LD_T4);
    // paired stores need whole lines in the tile: row tiles, whole-line column
    // tiles, or mirror tiles (column in and out) for the last pass of a
    // multi-pass transform
    static constexpr bool MIRROR = PAIRED && COL_IN && COL_OUT && !WHOLE_COL;
    // DCT-3 / DST-3 and inverse real transforms: the input repack runs as a
    // paired phase into shared memory (pair_prepack_thread) and the first
    // sub-stage reads its points from there.  Row tiles and whole-line column
    // tiles hold whole lines; the first pass of a multi-pass transform (column in, row out) pairs line j
    // with line ns - j in the tile, like the mirror tiles of the last pass.
    static constexpr bool PREPACK = LOAD == LD_T3 || LOAD == LD_IR;
    static constexpr bool MIRROR_IN = PREPACK && COL_IN && !WHOLE_COL;
    static_assert(!(MIRROR_IN && (COL_OUT || LOGJ < 1)), "the repacking pass of multi-pass transforms writes rows");
    static_assert(!(PAIRED && (COL_IN != COL_OUT)), "paired operators need row tiles or mirror tiles");
    static_assert(!MIRROR || LOGJ >= 1, "mirror tiles pair lines");

    // first sub-stage (points from shared memory, then the radix-16 DFT) of PREPACK tiles
    static NFFT_HD void first_smem(const PassArgs& a, const TwTables<T>* tw, const C2<T>* sm, const LeanLine* lines,
                                   int t, C2<T>* v, int& l, int& i) {
        lean_map<COL_IN, LOGJ>(t, LOGR - 4, l, i);
        const LeanLine ln = lines[l];
        if (ln.j < 0) {
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = mkc((T)0, (T)0);
            return;
        }
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = sm[NFFT_SM((lean_idx<COLL, LOGR, LOGJ>(l, i + (m << (LOGR - 4)))))];
        pre_twiddle_dft(a, tw, ln.j, i, v);
    }

    // ---- first sub-stage: global -> registers -> radix 16 --------------------
    static NFFT_HD void first(const PassArgs& a, const TwTables<T>* tw, const LeanLine* lines, int t, C2<T>* v, int& l,
                              int& i) {
        lean_map<COL_IN, LOGJ>(t, LOGR - 4, l, i);
        const LeanLine ln = lines[l];
        if (ln.j < 0) {
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = mkc((T)0, (T)0);
            return;
        }
        if constexpr (LOAD == LD_C) {
            const long long rs = a.in_estride << a.logNj;
            const C2<T>* src = (const C2<T>*)a.in + ln.bin + ln.j * a.in_estride + (long long)i * rs;
            const long long s16 = rs << (LOGR - 4);
            if (a.hint_in == 3) {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = gload(src + m * s16, 3);
            } else if (a.hint_in) {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = gload(src + m * s16, 1);
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = NFFT_GLD(src + m * s16);
            }
            if (a.conj_in) {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m].y = -v[m].y;
            }
        } else if constexpr ((LOAD == LD_BLUE || LOAD == LD_FILT) && COL_IN) {
            // first pass of a Bluestein M-point FFT: LD_C's strided addressing
            // plus one table point per point, position p = j + (i + m R/16) Nj
            // (forward: chirp premultiply, zero pad from N on; inverse: conj of
            // the filter product).  All loads issued before any is used.
            const long long rs = a.in_estride << a.logNj;
            const C2<T>* src = (const C2<T>*)a.in + ln.bin + ln.j * a.in_estride + (long long)i * rs;
            const long long s16 = rs << (LOGR - 4);
            const long long p0 = ln.j + ((long long)i << a.logNj), ps = 1ll << (a.logNj + LOGR - 4);
            const C2<T>* tab = (const C2<T>*)(LOAD == LD_BLUE ? a.chirp : a.filt) + p0;
            // two halves of 8 points: 16 loads in flight, as for LD_C
#pragma unroll
            for (int hf = 0; hf < 16; hf += 8) {
                C2<T> c[8];
                if constexpr (LOAD == LD_BLUE) {
#pragma unroll
                    for (int m = hf; m < hf + 8; ++m) {
                        const bool in = p0 + m * ps < a.N;
                        v[m] = in ? gload(src + m * s16, a.hint_in) : mkc((T)0, (T)0);
                        c[m - hf] = in ? gload_keep(tab + m * ps) : mkc((T)0, (T)0);
                    }
#pragma unroll
                    for (int m = hf; m < hf + 8; ++m) {
                        if (a.conj_in) v[m].y = -v[m].y;
                        v[m] = cmul(v[m], c[m - hf]);
                    }
                } else {
#pragma unroll
                    for (int m = hf; m < hf + 8; ++m) {
                        v[m] = gload(src + m * s16, a.hint_in);   // queue: scratch of this launch at L2
                        c[m - hf] = gload_keep(tab + m * ps);
                    }
#pragma unroll
                    for (int m = hf; m < hf + 8; ++m) v[m] = cconj(cmul(v[m], c[m - hf]));
                }
            }
        } else if constexpr (LOAD == LD_T4 && !COL_IN) {
            // row tile of a single-pass DCT-4 / DST-4 (line j = 0): premultiply
            // e^{-i pi p / N} of p = i + m R/16 as a chain of exact steps
            // e^{-i pi (R/16) / N} = W_64 (N = 2R) from one table twiddle
            const T* x = (const T*)a.in + ln.bin;
            if (a.in_estride == 1 && ln.j == 0) {
                const long long N = a.N;
                C2<T> e = twiddle<T>(tw, (uint64_t)i, a.logN + 1);
                const C2<T> st = twiddle<T>(tw, (uint64_t)1, 6);
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const long long p = i + (m << (LOGR - 4));
                    const T xe = NFFT_GLD(&x[2 * p]), xo = NFFT_GLD(&x[N - 1 - 2 * p]);
                    if (!a.dst) v[m] = mkc(e.x * xe - e.y * xo, e.x * xo + e.y * xe);
                    else v[m] = mkc(-e.x * xe - e.y * xo, e.x * xo - e.y * xe);
                    if (m < 15) e = cmul(e, st);
                }
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m)
                    v[m] = load_elem<T, LOAD>(a, tw, ln.bin, ln.j + ((long long)(i + (m << (LOGR - 4))) << a.logNj));
            }
        } else if constexpr ((LOAD == LD_R2C || LOAD == LD_T2) && !COL_IN) {
            // row tile of a single-pass real transform (line j = 0): the packed
            // point p = i + m R/16 of the line's N = 2R reals, without the generic
            // operator's per-element branches
            const T* x = (const T*)a.in + ln.bin;
            if (a.in_estride == 1 && ln.j == 0) {
                if constexpr (LOAD == LD_R2C) {
                    if (((uintptr_t)x & (sizeof(C2<T>) - 1)) == 0) {
#pragma unroll
                        for (int m = 0; m < 16; ++m) v[m] = NFFT_GLD((const C2<T>*)x + i + (m << (LOGR - 4)));
                    } else {
#pragma unroll
                        for (int m = 0; m < 16; ++m) {
                            const long long q = 2 * (long long)(i + (m << (LOGR - 4)));
                            v[m] = mkc(NFFT_GLD(&x[q]), NFFT_GLD(&x[q + 1]));
                        }
                    }
                } else {
                    // DCT-2 / DST-2 reorder v[i] = x[2i] (i < N/2), +-x[2N-1-2i]: points
                    // m < 8 lie in the first half of the packed line, m >= 8 in the second
                    const long long N2 = 2 * a.N;
                    const T sg = a.dst ? (T)-1 : (T)1;
#pragma unroll
                    for (int m = 0; m < 16; ++m) {
                        const long long q = 4 * (long long)(i + (m << (LOGR - 4)));
                        if (m < 8) v[m] = mkc(NFFT_GLD(&x[q]), NFFT_GLD(&x[q + 2]));
                        else v[m] = mkc(sg * NFFT_GLD(&x[N2 - 1 - q]), sg * NFFT_GLD(&x[N2 - 3 - q]));
                    }
                }
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m)
                    v[m] = load_elem<T, LOAD>(a, tw, ln.bin, ln.j + ((long long)(i + (m << (LOGR - 4))) << a.logNj));
            }
        } else {
#pragma unroll
            for (int m = 0; m < 16; ++m)
                v[m] = load_elem<T, LOAD>(a, tw, ln.bin, ln.j + ((long long)(i + (m << (LOGR - 4))) << a.logNj));
        }
        pre_twiddle_dft(a, tw, ln.j, i, v);
    }

    // Pass pre-twiddle W_{Ns R}^{r k} (k = j mod Ns) of the 16 points r = i + m R/16
    // of line j held by this thread, then the first radix-16 DFT.
    static NFFT_HD void pre_twiddle_dft(const PassArgs& a, const TwTables<T>* tw, long long j, int i, C2<T>* v) {
        if (a.logNs > 0) {
            const long long k = j & ((1ll << a.logNs) - 1);
            if (k) {
                // W_{Ns R}^{(i + m R/16) k} = W_{Ns R}^{i k} * (W_{16 Ns}^{k})^m
                if (a.tw_mode == 2) {
#pragma unroll
                    for (int m = 0; m < 16; ++m)
                        v[m] = cmul(v[m], twiddle<T>(tw, (uint64_t)(i + (m << (LOGR - 4))) * (uint64_t)k, a.logNs + LOGR));
                } else if (a.tw_mode == 1) {
                    C2<T> w = twiddle<T>(tw, (uint64_t)i * (uint64_t)k, a.logNs + LOGR);
                    const C2<T> s = twiddle<T>(tw, (uint64_t)k, a.logNs + 4);
                    const C2<T> s4 = cmul(cmul(s, s), cmul(s, s));
                    // four interleaved chains w s^{4c + d}: depth 4 per chain
                    C2<T> c0 = w, c1 = cmul(w, s);
                    C2<T> c2 = cmul(c1, s), c3 = cmul(c2, s);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        v[4 * q + 0] = cmul(v[4 * q + 0], c0);
                        v[4 * q + 1] = cmul(v[4 * q + 1], c1);
                        v[4 * q + 2] = cmul(v[4 * q + 2], c2);
                        v[4 * q + 3] = cmul(v[4 * q + 3], c3);
                        if (q < 3) { c0 = cmul(c0, s4); c1 = cmul(c1, s4); c2 = cmul(c2, s4); c3 = cmul(c3, s4); }
                    }
                } else {
                    C2<T> w0 = twiddle<T>(tw, (uint64_t)i * (uint64_t)k, a.logNs + LOGR);
                    C2<T> s = twiddle<T>(tw, (uint64_t)k, a.logNs + 4);
                    C2<T> p[16];
                    powers16<T>(s, p);
#pragma unroll
                    for (int m = 0; m < 16; ++m) v[m] = cmul(v[m], (m == 0) ? w0 : cmul(w0, p[m]));
                }
            }
        }
        dft16<T>(v);
    }

    // ---- middle / last sub-stage read from shared memory ----------------------
    template <int S, bool COLMAP>
    static NFFT_HD void read(const C2<T>* sm, int t, int q, C2<T>* v, int& l, int& i) {
        constexpr int LR = LeanSched<LOGR>::lr[S];
        constexpr int RHO = 1 << LR;
        constexpr int lq = LOGR - LR;
        lean_map<COLMAP, LOGJ>(t + q * THREADS, lq, l, i);
#pragma unroll
        for (int m = 0; m < RHO; ++m) v[m] = sm[NFFT_SM((lean_idx<COLL, LOGR, LOGJ>(l, i + (m << lq))))];
    }

    // internal twiddles W_{ns RHO}^{m k} and the radix-RHO DFT (ns = 2^lns)
    template <int S>
    static NFFT_HD void twiddle_dft(const TwTables<T>* tw, int i, C2<T>* v) {
        constexpr int LR = LeanSched<LOGR>::lr[S];
        constexpr int RHO = 1 << LR;
        constexpr int lns = lns_of<S>();
        const int k = i & ((1 << lns) - 1);
        if constexpr (WHOLE_COL) {
            mul_table<T, LR, lns>(tw, k, v);
        } else if (k) {
            // W^{m k} for m < RHO from the root W^k: radix 16 by a product tree (depth
            // 4), radix 8 by a chain (a tree of depth 3 puts the result of a 128- or
            // 512-point transform 3% further off; W^{4 k} from the table 20% less far,
            // but its entries lie a cache line apart)
            C2<T> p[16];
            p[1] = table_root<T, lns + LR>(tw, (uint32_t)k);
            if constexpr (RHO == 16) {
                powers16<T>(p[1], p);
            } else {
#pragma unroll
                for (int m = 2; m < RHO; ++m) p[m] = cmul(p[m - 1], p[1]);
            }
#pragma unroll
            for (int m = 1; m < RHO; ++m) v[m] = cmul(v[m], p[m]);
        }
        dft_radix<T, RHO>(v);
    }

    template <int S> static constexpr int lns_of() {
        int s = 0;
        for (int x = 0; x < S; ++x) s += LeanSched<LOGR>::lr[x];
        return s;
    }

    // Stockham output position of sub-stage S (within the line)
    template <int S>
    static NFFT_HD int out_pos(int i, int m) {
        constexpr int LR = LeanSched<LOGR>::lr[S];
        constexpr int lns = lns_of<S>();
        const int k = i & ((1 << lns) - 1);
        return ((i >> lns) << (lns + LR)) + k + (m << lns);
    }

    template <int S>
    static NFFT_HD void write_smem(C2<T>* sm, int l, int i, const C2<T>* v) {
        constexpr int RHO = 1 << LeanSched<LOGR>::lr[S];
#pragma unroll
        for (int m = 0; m < RHO; ++m) sm[NFFT_SM((lean_idx<COLL, LOGR, LOGJ>(l, out_pos<S>(i, m))))] = v[m];
    }

    // last sub-stage: outputs straight to global memory
    template <int S>
    static NFFT_HD void write_global(const PassArgs& a, const TwTables<T>* tw, const LeanLine* lines, int l, int i,
                                     const C2<T>* v) {
        constexpr int RHO = 1 << LeanSched<LOGR>::lr[S];
        const LeanLine ln = lines[l];
        if (ln.j < 0) return;
        const int logNso = a.logNs_out;
        const long long base = ((ln.j >> logNso) << (logNso + LOGR)) + (ln.j & ((1ll << logNso) - 1));
        if constexpr (STORE == ST_C) {
            const long long rs = a.out_estride << logNso;
            C2<T>* dst = (C2<T>*)a.out + ln.bout + base * a.out_estride + (long long)out_pos<S>(i, 0) * rs;
            constexpr int lns = lns_of<S>();
            const long long sm_ = rs << lns;   // output positions step by 2^lns per m
            C2<T> x[RHO];
            if (a.scale != 1.0) {
                const T f = (T)a.scale;
                const T fi = a.conj_out ? -f : f;
#pragma unroll
                for (int m = 0; m < RHO; ++m) x[m] = mkc(v[m].x * f, v[m].y * fi);
            } else if (a.conj_out) {
#pragma unroll
                for (int m = 0; m < RHO; ++m) x[m] = mkc(v[m].x, -v[m].y);
            } else {
#pragma unroll
                for (int m = 0; m < RHO; ++m) x[m] = v[m];
            }
            if (a.hint_out == 2) {
#pragma unroll
                for (int m = 0; m < RHO; ++m) gstore(dst + m * sm_, x[m], 2);
            } else if (a.hint_out == 1) {
#pragma unroll
                for (int m = 0; m < RHO; ++m) gstore(dst + m * sm_, x[m], 1);
            } else {
#pragma unroll
                for (int m = 0; m < RHO; ++m) NFFT_GST(dst + m * sm_, x[m]);
            }
        } else if constexpr (STORE == ST_C2R) {
            // invrealdft output: each complex point is the real pair (2q, 2q+1);
            // one vector store per point when the line's reals are pair-aligned
            constexpr int lns = lns_of<S>();
            const long long q0 = base + ((long long)out_pos<S>(i, 0) << logNso), qs = 1ll << (lns + logNso);
            T* y = (T*)a.out + ln.bout;
            const T f = (T)a.scale;
            const T fi = a.conj_out ? -f : f;
            if (a.out_estride == 1 && ((uintptr_t)y & (sizeof(C2<T>) - 1)) == 0) {
                C2<T>* dst = (C2<T>*)y + q0;
#pragma unroll
                for (int m = 0; m < RHO; ++m) NFFT_GST(dst + m * qs, mkc(v[m].x * f, v[m].y * fi));
            } else {
#pragma unroll
                for (int m = 0; m < RHO; ++m)
                    store_elem<T, STORE>(a, tw, ln.bout, q0 + m * qs, v[m]);
            }
        } else if constexpr (STORE == ST_BLUE) {
            // last pass of the inverse M-point FFT: window [0, N), back from the
            // conjugated domain, chirp postmultiply, scale; positions q step by
            // 2^(lns + logNso) per m.  Table loads issued before the stores.
            constexpr int lns = lns_of<S>();
            const long long q0 = base + ((long long)out_pos<S>(i, 0) << logNso), qs = 1ll << (lns + logNso);
            const C2<T>* ch = (const C2<T>*)a.chirp + q0;
            C2<T>* dst = (C2<T>*)a.out + ln.bout + q0 * a.out_estride;
            const long long ds = qs * a.out_estride;
            C2<T> c[RHO];
#pragma unroll
            for (int m = 0; m < RHO; ++m) c[m] = q0 + m * qs < a.N ? gload_keep(ch + m * qs) : mkc((T)0, (T)0);
            const T f = (T)a.scale;
            const T fi = a.conj_out ? -f : f;
#pragma unroll
            for (int m = 0; m < RHO; ++m) {
                if (q0 + m * qs >= a.N) continue;
                const C2<T> w = cmul(cconj(v[m]), c[m]);
                NFFT_GST(dst + m * ds, mkc(w.x * f, w.y * fi));
            }
        } else {
#pragma unroll
            for (int m = 0; m < RHO; ++m)
                store_elem<T, STORE>(a, tw, ln.bout, base + ((long long)out_pos<S>(i, m) << logNso), v[m]);
        }
    }
};

template <typename T, int LOGR, int LOGT, bool COL_IN, bool COL_OUT, int LOAD, int STORE>
constexpr size_t lean_smem_bytes() {
    using L = Lean<T, LOGR, LOGT, COL_IN, COL_OUT, LOAD, STORE>;
    return sizeof(C2<T>) * (size_t)L::SMEM_ELEMS + sizeof(LeanLine) * (size_t)L::J;
}

// Mirror tile unpack, the items of thread t: (J/2 low lines) x R items, each
// emitting bins k and M - k; lines fastest, so neighbouring threads write
// neighbouring bins.  A thread's items share one line and step r by
// D = THREADS / (J/2), so k steps by D ns and the twiddles follow exactly
// known ratios: W_N^{k + D ns} = W_N^k W_{2R}^D and e^{-i pi (k + D ns) / 2N} =
// e^{-i pi k / 2N} W_{8R}^D (N = 2 ns R) -- chains of at most 8 products from
// one table twiddle.  The self-paired line 0 of tile 0 (bins r ns, then ns/2 +
// r ns) takes its twiddles from the table.
template <typename L, typename T, int STORE>
NFFT_HD void mirror_unpack_thread(const PassArgs& a, const TwTables<T>* tw, const C2<T>* sm, const LeanLine* lines,
                                  long long tile, int t) {
    using V = C2<T>;
    constexpr int LOGR = L::LOGR_;
    constexpr int R = 1 << LOGR;
    constexpr int H = L::J / 2;
    constexpr int ITEMS = H << LOGR;
    static_assert(L::THREADS % H == 0, "a thread's items share one line");
    constexpr int D = L::THREADS / H;
    const long long ns = 1ll << a.logNj, tpt = ns >> L::LOGJ;
    const long long tt = tile - (tile / tpt) * tpt;
    const long long M = ns << LOGR;
    const int l = t & (H - 1);
    const LeanLine ln = lines[l];
    auto zget = [&](long long q) {
        const long long j = q & (ns - 1);
        const int rr = (int)(q >> a.logNj);
        return sm[NFFT_SM((lean_idx<true, LOGR, L::LOGJ>(mirror_local(tt, j, L::J, ns), rr)))];
    };
    if (tt == 0 && l == 0) {
        for (int w = t; w < ITEMS; w += L::THREADS)
            unpack_pair<T, STORE>(a, tw, ln.bout, mirror_item_k(tt, l, w >> (L::LOGJ - 1), R, ns, ln.j), M, zget);
        return;
    }
    const V ws = twiddle<T>(tw, (uint64_t)D, LOGR + 1);   // W_{2R}^D
    V ts = V{};
    if constexpr (STORE == ST_T2) ts = twiddle<T>(tw, (uint64_t)D, LOGR + 3);   // W_{8R}^D
    // bin k = lowj + r ns is point r of the low line; bin M - k is point
    // R - 1 - r of its partner line ns - lowj: both local lines fixed per thread
    const int loc_lo = mirror_local(tt, ln.j, L::J, ns), loc_hi = mirror_local(tt, ns - ln.j, L::J, ns);
    auto zrow = [&](int line, int rr) { return sm[NFFT_SM((lean_idx<true, LOGR, L::LOGJ>(line, rr)))]; };
    V wk = V{}, tk = V{};
#pragma unroll
    for (int w = t; w < ITEMS; w += L::THREADS) {
        const int r = w >> (L::LOGJ - 1);
        const long long k = ln.j + (long long)r * ns;
        if (w == t) {
            wk = twiddle<T>(tw, (uint64_t)k, a.logN);
            if constexpr (STORE == ST_T2) tk = twiddle<T>(tw, (uint64_t)k, a.logN + 2);
        } else {
            wk = cmul(wk, ws);
            if constexpr (STORE == ST_T2) tk = cmul(tk, ts);
        }
        unpack_pair_tw_z<T, STORE>(a, tw, ln.bout, k, M, zrow(loc_lo, r), zrow(loc_hi, R - 1 - r), wk, tk);
    }
}

// Paired unpack of whole lines (realdft unpack / DCT-2 post pairs), the items of
// thread t: an item is the bin pair k, R - k of one line, R the packed spectrum
// length.  Row tiles: a thread takes the same k of every line of the tile (its
// twiddles serve them all); with R/2 > THREADS its k steps by THREADS (twiddles times
// the exact ratios W_N^THREADS and e^{-i pi THREADS / 2N}; a table root per pair
// instead is 3% slower at 8192 points), with a new root from the table after R/512
// pairs: the chain of a 256-thread tile, whatever the tile.
// Column tiles: lines fastest, k stepping by THREADS / J, every root from the tables
// (the lines of a tile share it).  Bin 0 (with bins M and M/2) goes through unpack_pair.
template <typename L, typename T, int STORE>
NFFT_HD void paired_unpack_thread(const PassArgs& a, const TwTables<T>* tw, const C2<T>* sm, const LeanLine* lines,
                                  int t) {
    using V = C2<T>;
    constexpr int LOGR = L::LOGR_;
    constexpr int HALF = LOGR == 0 ? 1 : (1 << (LOGR - 1));
    constexpr int ITEMS = L::J * HALF;
    auto emit = [&](int ll, int k, V wk, V tk) {
        const LeanLine ln = lines[ll];
        if (ln.j < 0) return;
        auto zget = [&](long long r) { return sm[NFFT_SM((lean_idx<L::COLL, LOGR, L::LOGJ>(ll, (int)r)))]; };
        if (k == 0) unpack_pair<T, STORE>(a, tw, ln.bout, 0, (long long)(1 << LOGR), zget);
        else unpack_pair_tw<T, STORE>(a, tw, ln.bout, k, (long long)(1 << LOGR), zget, wk, tk);
    };
    auto roots = [&](int k, V& wk, V& tk) {
        wk = twiddle<T>(tw, (uint64_t)k, a.logN);
        if constexpr (STORE == ST_T2) tk = twiddle<T>(tw, (uint64_t)k, a.logN + 2);
    };
    V wk = V{}, tk = V{};
    if constexpr (L::WHOLE_COL) {
        for (int w = t; w < ITEMS; w += L::THREADS) {
            roots(w / L::J, wk, tk);
            emit(w & (L::J - 1), w / L::J, wk, tk);
        }
    } else {
        constexpr int STEPS = HALF > L::THREADS ? HALF / L::THREADS : 1;    // pairs of a line per thread
        constexpr int EVERY = HALF > L::THREADS ? 1 : L::THREADS / HALF;    // lines of a thread
        constexpr int CHAIN = HALF < 256 ? 1 : HALF / 256;                  // pairs per table root
        V ws = V{}, ts = V{};
        if constexpr (STEPS > 1 && CHAIN > 1) {
            ws = twiddle<T>(tw, (uint64_t)L::THREADS, a.logN);
            if constexpr (STORE == ST_T2) ts = twiddle<T>(tw, (uint64_t)L::THREADS, a.logN + 2);
        }
        // whole for realdft (FP64 8192 x 1000 38.9 -> 35.4 us, one pair at a time 37.3), two
        // pairs at a time for the longer code of DCT-2: whole, it does not fit the float
        // kernel's 64 registers (4096 x 4000 50 us, 45 so), and calls that alternate
        // with DCT-3 fetch it anew (FP64 8192 x 512 both ways 68.2 us, 61.4 so)
        constexpr int UNROLL = STORE == ST_R ? STEPS : 2;
#pragma unroll UNROLL
        for (int s = 0; s < STEPS; ++s) {
            const int k = (t & (HALF - 1)) + s * L::THREADS;
            if (s % CHAIN == 0 || k == L::THREADS) {   // (bin 0 has no twiddles to go on from)
                roots(k, wk, tk);
            } else {
                wk = cmul(wk, ws);
                if constexpr (STORE == ST_T2) tk = cmul(tk, ts);
            }
            for (int ll = HALF > L::THREADS ? 0 : t / HALF; ll < L::J; ll += EVERY) emit(ll, k, wk, tk);
        }
    }
}

// Paired input repack (PREPACK): the inverse-real repack
// p -> conj(s + i e^{+2 pi i p/N} d), s / d from the bins z_p and conj z_{M-p},
// for invrealdft (z = the input bins; bins 1 .. M-1 halved for the adjoint of
// realdft) and DCT-3 / DST-3 (z = the pre-twiddled reorder zb of the reals;
// zb_0 doubled for the adjoint of DCT-2 / DST-2).  An item is a pair of bins k,
// M - k: it takes z_k and z_{M-k} once and writes both points
// (W_N^{M-k} = -conj W_N^k; in row tiles e^{-i pi (M-k)/2N} = e^{-i pi/4} conj
// e^{-i pi k/2N}, one lookup less for two roundings more), where the generic
// operators compute both members of a pair for each point.  Every thread has 8 items; all their loads are issued
// before any is used; their twiddles are the tables' roots.
// Row tiles: items walk k along a line; whole-line column tiles: lines fastest, k
// of a thread's line stepping by THREADS / J.  Mirror-in tiles: item (l, r) is bin
// j + r ns of the low line j and its partner, point R - 1 - r of line ns - j;
// the first low line of a transform's first tile (j = 0) and its high line
// (j = ns / 2) pair with themselves (mirror_item_k).  Items walk lines fastest.
// Bound by HBM like a plain pass.  B200, before (a loop of dependent loads; the
// first pass of several through the generic operator) -> now: invrealdft 2^20 x
// 16 FP64 230 -> 180 us, DCT-3 2^18 x 81 FP64 390 -> 245 us, realdft + invrealdft
// 32768 x 512 FP32 90 -> 75 us, 4096 x 2000 FP64 97 -> 80 us.
template <typename L, typename T, int LOAD>
NFFT_HD void pair_prepack_thread(const PassArgs& a, const TwTables<T>* tw, C2<T>* sm, const LeanLine* lines,
                                 long long tile, int t) {
    using V = C2<T>;
    constexpr int LOGR = L::LOGR_, R = 1 << LOGR, NI = 8;
    constexpr bool MIR = L::MIRROR_IN, WC = L::WHOLE_COL;
    constexpr int H = MIR ? L::J / 2 : R / 2;   // low lines of a tile / items of a line
    static_assert(MIR ? H * R == NI * L::THREADS : L::J * H == NI * L::THREADS, "8 items per thread");
    const long long es = a.in_estride;
    const long long ns = MIR ? 1ll << a.logNj : 1;
    const long long M = ns << LOGR, N = 2 * M;
    auto put = [&](int l, int r, V v) { sm[NFFT_SM((lean_idx<L::COLL, LOGR, L::LOGJ>(l, r)))] = v; };
    // first tile of a transform, first low line: self-paired lines
    bool self = false;
    if constexpr (MIR) self = tile % (ns >> L::LOGJ) == 0 && (t & (H - 1)) == 0;
    // item q: local lines and points of bins k and M - k, and k
    auto item = [&](int q, int& lA, int& rA, int& lB, int& rB) -> long long {
        const int w = t + q * L::THREADS;
        if constexpr (MIR) {
            const int l = w & (H - 1), r = w / H;
            if (!self) {
                lA = l; rA = r; lB = H + l; rB = R - 1 - r;
                return lines[l].j + r * ns;
            }
            if (r < R / 2) {
                lA = lB = 0; rA = r; rB = R - r;
                return r * ns;
            }
            lA = lB = H; rA = r - R / 2; rB = R - 1 - rA;
            return ns / 2 + rA * ns;
        } else {
            lA = lB = WC ? w & (L::J - 1) : w / H;
            rA = WC ? w / L::J : w & (H - 1);
            rB = R - rA;
            return rA;
        }
    };
    // the two bins of pair k as raw input values: zk, zm (LD_IR), or the reals
    // (x_k, x_{N-k}), (x_{M-k}, x_{M+k}) behind zb_k and zb_{M-k} (LD_T3)
    auto raw_k = [&](long long base, long long k) {
        if constexpr (LOAD == LD_IR) {
            return NFFT_GLD((const V*)a.in + base + k * es);
        } else {
            const T* x = (const T*)a.in + base;
            const long long iA = a.dst ? N - 1 - k : k, iB = k == 0 ? iA : (a.dst ? k - 1 : N - k);
            return mkc(NFFT_GLD(&x[iA * es]), NFFT_GLD(&x[iB * es]));
        }
    };
    auto raw_m = [&](long long base, long long k) {
        if constexpr (LOAD == LD_IR) {
            return NFFT_GLD((const V*)a.in + base + (M - k) * es);
        } else {
            const T* x = (const T*)a.in + base;
            const long long iC = a.dst ? M - 1 + k : M - k, iD = a.dst ? M - 1 - k : M + k;
            return mkc(NFFT_GLD(&x[iC * es]), NFFT_GLD(&x[iD * es]));
        }
    };
    auto pre = [&](V x, V tq) { return mkc(x.x * tq.x - x.y * tq.y, -x.x * tq.y - x.y * tq.x); };
    auto rep = [](V u, V v2, V w2) {
        const V b = cconj(v2);
        const V s2 = cadd(u, b), d = csub(u, b);
        const V od = cmulc(d, w2);
        return cconj(mkc(s2.x - od.y, s2.y + od.x));
    };
    V u[NI], v[NI], uh = V{};
    // bin M / 2 pairs with itself: one per line (row tiles) or transform
    const bool half = MIR ? self && t < H : t < L::J && lines[t].j >= 0;
#pragma unroll
    for (int q = 0; q < NI; ++q) {
        int lA, rA, lB, rB;
        const long long k = item(q, lA, rA, lB, rB);
        const LeanLine ln = lines[lA];
        u[q] = ln.j >= 0 ? raw_k(ln.bin, k) : mkc((T)0, (T)0);
        v[q] = ln.j >= 0 ? raw_m(ln.bin, k) : mkc((T)0, (T)0);
    }
    if (half) uh = raw_k(lines[MIR ? 0 : t].bin, M / 2);
    // Twiddles from the tables, pair by pair: as products of the thread's first root
    // with exact ones they cost a rounding more (DCT-3 of 8192 points and more, error
    // up to 4% larger).  The bins of a thread differ in multiples of D ns (mirror-in
    // tiles) or THREADS (row tiles), so of each root's table entries only the first
    // changes (RootRun); row tiles of short lines have the same k in every pair.
    constexpr bool SAME_K = !MIR && !WC && H <= L::THREADS;
    const int logN = MIR ? a.logN : LOGR + 1;
    RootRun<T> run_w, run_t;
    V wk = V{}, tk = V{}, tm = V{};
#pragma unroll
    for (int q = 0; q < NI; ++q) {
        int lA, rA, lB, rB;
        const long long k = item(q, lA, rA, lB, rB);
        // (a self-paired low line gives way to its high line in the middle)
        if (q == 0 || (MIR && q == NI / 2 && self)) {
            run_w.start(tw, k, logN);
            if constexpr (LOAD == LD_T3) run_t.start(tw, k, logN + 2);
        }
        if (q == 0 || !SAME_K) {
            wk = run_w.at(tw, k);
            if constexpr (LOAD == LD_T3) {
                tk = run_t.at(tw, k);
                if constexpr (MIR || WC) tm = run_t.mirror(tw, M, k);
                else tm = mkc((tk.x - tk.y) * K<T>::r2, -(tk.x + tk.y) * K<T>::r2);
            }
        }
        V zk = u[q], zm = v[q];
        if constexpr (LOAD == LD_IR) {
            if (a.vjp && k > 0) {
                zk = cscale(zk, (T)0.5);
                zm = cscale(zm, (T)0.5);
            }
        } else {
            if (k == 0) zk = mkc(a.vjp ? (T)2 * zk.x : zk.x, (T)0);
            else zk = pre(zk, tk);
            zm = pre(zm, tm);
        }
        if (k == 0) {
            put(lA, 0, mkc(zk.x + zm.x, zm.x - zk.x));
        } else {
            put(lA, rA, rep(zk, zm, wk));
            put(lB, rB, rep(zm, zk, mkc(-wk.x, wk.y)));
        }
    }
    if (half) {
        // p = M / 2: z pairs with itself and W_N^p = -i, so the point is 2 z
        V z = uh;
        if constexpr (LOAD == LD_IR) z = cscale(z, a.vjp ? (T)1 : (T)2);
        else z = cscale(pre(z, mkc(K<T>::c8, -K<T>::s8)), (T)2);
        put(MIR ? 0 : t, R / 2, z);
    }
}

// One tile of a specialized pass (all threads of the CTA call it; uniform
// early exit past the last line).
template <typename T, int LOGR, int LOGT, bool COL_IN, bool COL_OUT, int LOAD, int STORE, bool PDL = false>
__device__ __forceinline__ void lean_tile(const PassArgs& a, long long tile, unsigned char* smraw) {
    using L = Lean<T, LOGR, LOGT, COL_IN, COL_OUT, LOAD, STORE>;
    using V = C2<T>;
    V* sm = (V*)smraw;
    LeanLine* lines = (LeanLine*)(sm + L::SMEM_ELEMS);
    const TwTables<T>* tw = (const TwTables<T>*)a.tw;
    const int t = threadIdx.x;
    const long long line0 = tile << L::LOGJ;
    if (line0 >= a.nlines) {
        if constexpr (PDL) pdl_wait();
        return;
    }
    if (t < L::J) {
        long long tmp[3];
        TileLines tl{&tmp[0], &tmp[1], &tmp[2]};
        if constexpr (L::MIRROR || L::MIRROR_IN) {
            const long long ns = 1ll << a.logNj, tpt = ns >> L::LOGJ;   // lines, tiles per transform
            const long long tr = tile / tpt, tt = tile - tr * tpt;
            line_setup(a, tr * ns + mirror_line(tt, t, L::J, ns), 0, tl);
        } else {
            line_setup(a, line0 + t, 0, tl);
        }
        lines[t] = LeanLine{tmp[0], tmp[1], tmp[2]};
    }
    if constexpr (PDL) pdl_wait();
    __syncthreads();

    V v[16];
    int l, i;
    if constexpr (L::PREPACK) {
        pair_prepack_thread<L, T, LOAD>(a, tw, sm, lines, tile, t);
        __syncthreads();
        L::first_smem(a, tw, sm, lines, t, v, l, i);
        __syncthreads();   // every point read before the sub-stage writes
    } else {
        L::first(a, tw, lines, t, v, l, i);
    }
    if constexpr (L::NS == 1) {
        // single radix-16 sub-stage: the same thread stores its outputs
        if constexpr (L::PAIRED) {
            L::template write_smem<0>(sm, l, i, v);
        } else {
            L::template write_global<0>(a, tw, lines, l, i, v);
        }
    } else {
        L::template write_smem<0>(sm, l, i, v);
        __syncthreads();
        if constexpr (LOAD == LD_C && COL_IN && !L::MIRROR) {   // mirror tiles: lines are not one address run
            // every load of the tile has completed: drop the scratch lines just read
            constexpr int PER_LINE = 128 / (int)sizeof(V);
            if (a.discard_in && L::J >= PER_LINE && (l % PER_LINE) == 0) {
                const LeanLine ln = lines[l];
                if (ln.j >= 0) {
                    const V* src = (const V*)a.in + ln.bin + ln.j * a.in_estride;
                    const long long rs = a.in_estride << a.logNj;
#pragma unroll
                    for (int m = 0; m < 16; ++m) discard_l2(&src[(long long)(i + (m << (LOGR - 4))) * rs]);
                }
            }
        }
        // middle sub-stages (compile-time unrolled)
        if constexpr (L::NS >= 3) {
            constexpr int S = 1;
            constexpr int RHO = 1 << LeanSched<LOGR>::lr[S];
            V w[16];
            int ls[16 / RHO], is[16 / RHO];
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) L::template read<S, L::COLL>(sm, t, q, &w[q * RHO], ls[q], is[q]);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) {
                L::template twiddle_dft<S>(tw, is[q], &w[q * RHO]);
                L::template write_smem<S>(sm, ls[q], is[q], &w[q * RHO]);
            }
            __syncthreads();
        }
        if constexpr (L::NS >= 4) {
            constexpr int S = 2;
            constexpr int RHO = 1 << LeanSched<LOGR>::lr[S];
            V w[16];
            int ls[16 / RHO], is[16 / RHO];
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) L::template read<S, L::COLL>(sm, t, q, &w[q * RHO], ls[q], is[q]);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) {
                L::template twiddle_dft<S>(tw, is[q], &w[q * RHO]);
                L::template write_smem<S>(sm, ls[q], is[q], &w[q * RHO]);
            }
            __syncthreads();
        }
        // last sub-stage
        {
            constexpr int S = L::NS - 1;
            constexpr int RHO = 1 << LeanSched<LOGR>::lr[S];
            V w[16];
            int ls[16 / RHO], is[16 / RHO];
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) L::template read<S, COL_OUT>(sm, t, q, &w[q * RHO], ls[q], is[q]);
            if constexpr (L::PAIRED) __syncthreads();
#pragma unroll
            for (int q = 0; q < 16 / RHO; ++q) {
                L::template twiddle_dft<S>(tw, is[q], &w[q * RHO]);
                if constexpr (L::PAIRED) L::template write_smem<S>(sm, ls[q], is[q], &w[q * RHO]);
                else L::template write_global<S>(a, tw, lines, ls[q], is[q], &w[q * RHO]);
            }
        }
    }
    if constexpr (L::MIRROR) {
        __syncthreads();
        mirror_unpack_thread<L, T, STORE>(a, tw, sm, lines, tile, t);
    } else if constexpr (L::PAIRED) {
        __syncthreads();
        paired_unpack_thread<L, T, STORE>(a, tw, sm, lines, t);
    }
}

// Minimum CTAs per SM the specialized kernels are compiled for (register
// budget 65536 / (threads x CTAs)).  The passes are latency-bound, so warps per
// SM matter: the float kernels fit in 64 registers and run 8 CTAs of 128
// threads per SM (measured on B200: +11% at 2^16, +29% at 4096 over 4 CTAs);
// the double kernels need their 128.
#ifndef NFFT_LEAN_MINB_T7_F64
#define NFFT_LEAN_MINB_T7_F64 4
#endif
#ifndef NFFT_LEAN_MINB_T7_F32
#define NFFT_LEAN_MINB_T7_F32 8
#endif
#ifndef NFFT_LEAN_MINB_T8_F64
#define NFFT_LEAN_MINB_T8_F64 2
#endif
#ifndef NFFT_LEAN_MINB_T8_F32
#define NFFT_LEAN_MINB_T8_F32 4
#endif
#ifndef NFFT_LEAN_MINB_T9_F32
#define NFFT_LEAN_MINB_T9_F32 2
#endif
template <typename T, int LOGT>
constexpr int lean_min_blocks() {
    return LOGT <= 7 ? (sizeof(T) == 4 ? NFFT_LEAN_MINB_T7_F32 : NFFT_LEAN_MINB_T7_F64)
                     : (LOGT == 8 ? (sizeof(T) == 4 ? NFFT_LEAN_MINB_T8_F32 : NFFT_LEAN_MINB_T8_F64)
                                  : (sizeof(T) == 4 ? NFFT_LEAN_MINB_T9_F32 : 1));
}

// Tile order of a standalone Bluestein filter-product pass (LD_FILT): the
// batch's transforms fastest, so the filter points one tile reads are read by
// the other transforms' tiles right after it (L2 hits instead of one filter
// sweep per transform).  A permutation of [0, tiles); identity for one
// transform or other line layouts.
NFFT_HD long long lean_batch_inner(const PassArgs& a, long long tile, int logJ) {
    if (a.ndims != 2 || a.jpos != 0 || a.cnt[1] <= 1) return tile;
    const long long tpt = a.cnt[0] >> logJ, B = a.cnt[1];
    if ((tpt << logJ) != a.cnt[0] || tile >= tpt * B) return tile;
    return (tile % B) * tpt + tile / B;
}

template <typename T, int LOGR, int LOGT, bool COL_IN, bool COL_OUT, int LOAD, int STORE>
__global__ void __launch_bounds__(1 << LOGT, (lean_min_blocks<T, LOGT>()))
lean_pass_kernel(const PassArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    long long tile = (long long)blockIdx.x + (long long)blockIdx.y * gridDim.x;
    if constexpr (LOAD == LD_FILT) tile = lean_batch_inner(a, tile, Lean<T, LOGR, LOGT, COL_IN, COL_OUT, LOAD, STORE>::LOGJ);
    lean_tile<T, LOGR, LOGT, COL_IN, COL_OUT, LOAD, STORE, true>(a, tile, smraw);
}

}  // namespace nfft
