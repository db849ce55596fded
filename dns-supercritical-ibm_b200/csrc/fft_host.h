// fft_host.h -- host-side planning of the in-place DIF transforms: radix
// sequence, per-stage twiddles (extended precision, rounded once) and the
// digit-reversal position table.  Header-only so both the planned entry
// points and the no-allocation entry point fill their tables the same way,
// into caller-provided memory.
#pragma once
#include <cmath>
#include <cstring>

#include "fft_dif.cuh"
#include "fft_pass.cuh"

namespace prj {

// radices of the compile-time pass plan of length n in radix order `order` (0: the
// default of PRJ_PASS_PLANS, k >= 1: the k-th entry of n in PRJ_PASS_ALTS); 0 if none
inline int pass_radices(int n, int* fac, int cap, int order = 0) {
    int seen = 0;
#define PRJ_PASS_RADICES(N, ...)                                  \
    if (n == N && seen++ == order) {                              \
        const int r[] = {__VA_ARGS__};                            \
        const int nr = (int)(sizeof(r) / sizeof(r[0]));           \
        if (nr > cap) return -1;                                  \
        for (int i = 0; i < nr; i++) fac[i] = r[i];               \
        return nr;                                                \
    }
    PRJ_PASS_ALL(PRJ_PASS_RADICES)
#undef PRJ_PASS_RADICES
    return 0;
}

// radix orders compiled for length n (0 when n has no pass plan)
inline int pass_orders(int n) {
    int c = 0;
#define PRJ_PASS_COUNT(N, ...) \
    if (n == N) c++;
    PRJ_PASS_ALL(PRJ_PASS_COUNT)
#undef PRJ_PASS_COUNT
    return c;
}

// Fewest passes over the radices 2 .. 11 and 13 (each pass is a round trip through shared
// memory and a barrier), among those the smallest largest radix (registers), found by trying
// every multiset in descending order; -1 if n has a larger prime factor or needs more passes.
inline int short_radices(int n, int most, int left, int* fac) {
    if (n == 1) return 0;
    if (left == 0) return -1;
    static const int radices[] = {13, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    for (int r : radices) {
        if (r > most || n % r != 0) continue;
        const int got = short_radices(n / r, r, left - 1, fac + 1);
        if (got >= 0) {
            fac[0] = r;
            return got + 1;
        }
    }
    return -1;
}

// radix sequence of a length-n transform: the pass plan's radices (in radix order `order`)
// where one exists, else the fewest passes; returns the number of stages, or -1 when n has a
// prime factor above 13.  In the runtime sequence the even radices come first, 8s after them
// and odd radices last: the last pass's butterflies are R elements apart, and an odd R (or 8,
// with the padding) spreads them over the banks.
inline int fft_factorize(int n, int* fac, int cap, int order = 0) {
    const int np = pass_radices(n, fac, cap, order);
    if (np != 0) return np;
    int f[kMaxStages], best[kMaxStages], nb = -1;
    for (int left = 0; left <= kMaxStages && left <= cap && nb < 0; left++)
        for (int most = 2; most <= 13 && nb < 0; most++) {
            const int got = short_radices(n, most, left, f);
            if (got >= 0) {
                nb = got;
                std::memcpy(best, f, sizeof(f));
            }
        }
    if (nb < 0) return -1;
    auto key = [](int r) { return r % 2 ? 2 : r == 8 ? 1 : 0; };
    int c = 0;
    for (int k = 0; k < 3; k++)
        for (int i = 0; i < nb; i++)
            if (key(best[i]) == k) fac[c++] = best[i];
    return nb;
}

// true when n has an in-place plan: every prime factor at most 13
inline bool dif_supported(int n) {
    int fac[kMaxStages];
    return fft_factorize(n, fac, kMaxStages) >= 0;
}

// true when n is a product of 2, 3 and 5 (the lengths the mixed-precision and distributed
// paths accept)
inline bool smooth5(int n) {
    for (int p : {2, 3, 5})
        while (n % p == 0) n /= p;
    return n == 1;
}

// fills the stage descriptor (radix order `order` where n has a pass plan); returns the
// number of twiddles (>= 1) or -1
inline long dif_plan(int n, DifDev* f, int order = 0) {
    int fac[kMaxStages];
    const int nf = fft_factorize(n, fac, kMaxStages, order);
    if (nf < 0) return -1;
    std::memset(f, 0, sizeof(*f));
    f->n = n;
    f->nst = nf;
    long cnt = 0;
    int L = n;
    for (int s = 0; s < nf; s++) {
        const int R = fac[s];
        f->radix[s] = R;
        f->span[s] = L;
        f->twoff[s] = (int)cnt;
        f->nbdiv[s] = make_fastdiv((unsigned)(n / R));
        f->mmdiv[s] = make_fastdiv((unsigned)(L / R));
        cnt += (long)(L / R) * (R - 1);
        L /= R;
    }
    return cnt > 0 ? cnt : 1;
}

// twiddle entries of a stage descriptor (what dif_plan returned for it)
inline long dif_twiddle_count(const DifDev& f) {
    long cnt = 0;
    for (int s = 0; s < f.nst; s++) cnt += (long)(f.span[s] / f.radix[s]) * (f.radix[s] - 1);
    return cnt > 0 ? cnt : 1;
}

// twiddles (forward sign; stage s at twoff[s], entry (q-1) mm + j, so the butterflies of
// consecutive j read consecutive entries) and positions: pos[k] = slot of index k after the transform
template <typename V>
inline void dif_fill(const DifDev& f, V* tw, int* pos) {
    const long double two_pi = 6.283185307179586476925286766559005768L;
    long c = 0;
    for (int s = 0; s < f.nst; s++) {
        const int R = f.radix[s], L = f.span[s], mm = L / R;
        for (int q = 1; q < R; q++)
            for (int j = 0; j < mm; j++) {
                const long double a = two_pi * (long double)q * j / (long double)L;
                tw[c].x = (decltype(tw[c].x))cosl(a);
                tw[c].y = (decltype(tw[c].y))(-sinl(a));
                c++;
            }
    }
    if (c == 0) { tw[0].x = 1; tw[0].y = 0; }
    for (int p = 0; p < f.n; p++) {
        int rem = p, k = 0, mult = 1;
        for (int s = 0; s < f.nst; s++) {
            const int R = f.radix[s];
            const int blk = f.span[s] / R;  // slots per digit value at this stage
            const int q = rem / blk;
            rem -= q * blk;
            k += q * mult;
            mult *= R;
        }
        pos[k] = p;
    }
}

// exp(-2 pi i k / n), k = 0..m (post-processing twiddles of a real transform)
template <typename V>
inline void real_post_fill(int n, int m, V* post) {
    const long double two_pi = 6.283185307179586476925286766559005768L;
    for (int k = 0; k <= m; k++) {
        const long double a = two_pi * (long double)k / (long double)n;
        post[k].x = (decltype(post[k].x))cosl(a);
        post[k].y = (decltype(post[k].y))(-sinl(a));
    }
}

}  // namespace prj
