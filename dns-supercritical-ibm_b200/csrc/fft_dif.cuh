// fft_dif.cuh -- in-place mixed-radix decimation-in-frequency FFT for one CTA.
//
// Rows of length n live in shared memory (row stride rs).  Stage s has span
// L_s = n / (R_0 ... R_{s-1}); each butterfly takes the R_s elements
// j + r L_s/R_s of one span block, runs an R_s-point DFT and scales output q by
// exp(-+2 pi i q j / L_s), writing back to the same R_s slots.  Butterflies of a
// stage touch disjoint slots, so a stage needs one barrier and no second
// buffer.  The result is in digit-reversed order: frequency (or, for the
// inverse, time) index k sits at slot pos[k]; consumers read through `pos`.
//
// Twiddles per stage: tw[(q - 1) L/R + j] = exp(-2 pi i q j / L), j < L/R,
// 1 <= q < R.  The inverse transform uses the conjugates.  Radices 2 .. 11 and 13;
// lengths with larger prime factors use the out-of-place path of fft_device.cuh.
#pragma once
#include "fft_device.cuh"

namespace prj {

// Division by a run-time invariant d by multiply-high and shift (Granlund and
// Montgomery, "Division by invariant integers using multiplication", 1994):
// q = umulhi(x, m) >> s with s = ceil(log2 d) - 1, m = ceil(2^(31 + ceil(log2 d)) / d).
// Exact for 0 <= x < 2^22 and 1 <= d < 8200 (checked exhaustively on the host).
struct FastDiv {
    unsigned d, m, s;
};

__host__ __device__ inline FastDiv make_fastdiv(unsigned d) {
    FastDiv f{d, 0u, 0u};
    if (d > 1) {
        unsigned l = 0;
        while ((1u << l) < d) l++;
        const unsigned long long p = 31ull + l;
        f.m = (unsigned)(((1ull << p) + d - 1) / d);
        f.s = l - 1;
    }
    return f;
}

__device__ __forceinline__ int fdiv(int x, const FastDiv& f) {
    return f.d == 1 ? x : (int)(__umulhi((unsigned)x, f.m) >> f.s);
}

struct DifDev {
    int n;
    int nst;
    int radix[kMaxStages];
    int span[kMaxStages];
    int twoff[kMaxStages];
    FastDiv nbdiv[kMaxStages];  // n / radix
    FastDiv mmdiv[kMaxStages];  // span / radix
};

template <int DIR, typename V>
__device__ __forceinline__ V twiddle(V a, V w) {
    return DIR < 0 ? cmul(a, w) : cmulc(a, w);
}

// Shared-memory slot of element g.  PAD inserts one empty 16-byte slot after
// every 8 elements, so strides that are multiples of 8 elements (the late
// stages and the digit-reversal gathers) spread over all bank groups.
template <bool PAD>
__device__ __forceinline__ int sidx(int g) {
    return PAD ? g + (g >> 3) : g;
}

// elements per row buffer of n slots with optional padding
__host__ __device__ inline int padded_len(int n, bool pad) { return pad ? n + (n >> 3) + 1 : n; }

template <int DIR, int R, typename V>
__device__ __forceinline__ void dft_r(V* a) {
    if constexpr (R == 2) dft2<DIR>(a[0], a[1]);
    else if constexpr (R == 3) dft3<DIR>(a[0], a[1], a[2]);
    else if constexpr (R == 4) dft4<DIR>(a[0], a[1], a[2], a[3]);
    else if constexpr (R == 5) dft5<DIR>(a[0], a[1], a[2], a[3], a[4]);
    else if constexpr (R == 6) dft6<DIR>(a);
    else if constexpr (R == 8) dft8<DIR>(a);
    else if constexpr (R == 9) dft9<DIR>(a);
    else if constexpr (R == 10) dft10<DIR>(a);
    else {
        static_assert(R == 7 || R == 11 || R == 13, "radices 2 .. 11 and 13");
        dft_prime<DIR, R>(a);
    }
}

// a[q] *= w1^q with w1 = exp(-+2 pi i j / L) the first row of the stage table (w[j]); the
// powers come from a product tree of depth <= 4 (a few ulp), so a butterfly loads one
// twiddle instead of R-1 (the loads were the larger share of the L1 traffic of these kernels).
// For the runtime radices, loading each from the table instead took 1.5 - 5% more of a Poisson
// solve (526 -> 545 us at 360x180x250, 1090 -> 1143 at 640x100x640) and left the error against
// 64-bit transforms where it is: over 52 grids of 2, 3, 5, 7, 11 and 13 it is 0.97 times (tree)
// and 0.96 times (table) that of the radix sequences 8, 4, 2, 3, 5 used before.
template <int DIR, int R, typename V>
__device__ __forceinline__ void apply_twiddles(V* a, const V* __restrict__ w, int j) {
    V p[R];
    p[1] = w[j];
#pragma unroll
    for (int q = 2; q < R; q++) p[q] = cmul(p[q / 2], p[q - q / 2]);
#pragma unroll
    for (int q = 1; q < R; q++) a[q] = twiddle<DIR>(a[q], p[q]);
}

// One stage of radix R of the runtime-radix transform: butterflies on elements
// row rs + b L + j + q mm of buf, nb per row, spans of mm butterflies; w = the stage's twiddles.
// DIT = false: DFT, then twiddles (decimation in frequency); DIT = true: twiddles, then DFT.
// Not inlined: each radix is register-allocated on its own.
template <int DIR, bool DIT, bool PAD, int R, typename V>
__device__ __noinline__ void stage_r(V* buf, int nrows, int rs, int nb, int mm, FastDiv dnb, FastDiv dmm,
                                     const V* __restrict__ w) {
    for (int idx = threadIdx.x; idx < nb * nrows; idx += blockDim.x) {
        const int row = fdiv(idx, dnb);
        const int bi = idx - row * nb;
        const int b = fdiv(bi, dmm);
        const int j = bi - b * mm;
        const int g0 = row * rs + b * (mm * R) + j;
        V a[R];
#pragma unroll
        for (int q = 0; q < R; q++) a[q] = buf[sidx<PAD>(g0 + q * mm)];
        if (DIT && j) apply_twiddles<DIR, R>(a, w, j);
        dft_r<DIR, R>(a);
        if (!DIT && j) apply_twiddles<DIR, R>(a, w, j);
#pragma unroll
        for (int q = 0; q < R; q++) buf[sidx<PAD>(g0 + q * mm)] = a[q];
    }
}

// stage s of the plan, whatever its radix
template <int DIR, bool DIT, bool PAD, typename V>
__device__ __forceinline__ void stage_switch(V* buf, int nrows, int rs, const DifDev& f, int s, const V* __restrict__ tw) {
    const int R = f.radix[s], nb = f.n / R, mm = f.span[s] / R;
    const V* w = tw + f.twoff[s];
    const FastDiv dnb = f.nbdiv[s], dmm = f.mmdiv[s];
    switch (R) {
#define PRJ_STAGE(R_) \
    case R_: stage_r<DIR, DIT, PAD, R_>(buf, nrows, rs, nb, mm, dnb, dmm, w); break;
        PRJ_STAGE(2) PRJ_STAGE(3) PRJ_STAGE(4) PRJ_STAGE(5) PRJ_STAGE(6) PRJ_STAGE(7) PRJ_STAGE(8)
        PRJ_STAGE(9) PRJ_STAGE(10) PRJ_STAGE(11) PRJ_STAGE(13)
#undef PRJ_STAGE
    default: break;  // the host plans no other radix here (dif_supported)
    }
}

// In-place transform of `nrows` rows of n elements (row r starts at element
// r * rs; with PAD, element g of the buffer lives at slot g + g/8).  DIT = false:
// decimation in frequency, natural order in, digit-reversed out.  DIT = true:
// decimation in time with the same plan, digit-reversed in, natural out; with
// DIR = +1 it inverts the DIF transform up to the factor n.  Starts and ends
// with the CTA synchronised.
template <int DIR, bool DIT, bool PAD, typename V>
__device__ __forceinline__ void inplace_rows(V* buf, int nrows, int rs, const DifDev& f, const V* __restrict__ tw) {
    for (int t = 0; t < f.nst; t++) {
        stage_switch<DIR, DIT, PAD>(buf, nrows, rs, f, DIT ? f.nst - 1 - t : t, tw);
        __syncthreads();
    }
}

// rows of whole elements at a stride in memory, a sink of dit_rows_to
__device__ __forceinline__ void put(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void put(float2* p, double2 v) { *p = make_float2((float)v.x, (float)v.y); }
template <typename T>
struct RowStore {
    T* p;
    size_t stride;
    __device__ __forceinline__ void operator()(int r, int e, double2 v) const { put(p + r * stride + e, v); }
};

// the last stage of a decimation in time (span n), its natural-order outputs to st(row, e, value)
template <int DIR, int R, typename V, class St>
__device__ __noinline__ void stage_out_r(const V* buf, int nrows, int rs, int mm, FastDiv dmm, const V* __restrict__ w,
                                         St st) {
    for (int idx = threadIdx.x; idx < mm * nrows; idx += blockDim.x) {
        const int row = fdiv(idx, dmm), j = idx - row * mm;
        V a[R];
#pragma unroll
        for (int q = 0; q < R; q++) a[q] = buf[sidx<true>(row * rs + j + q * mm)];
        if (j) apply_twiddles<DIR, R>(a, w, j);
        dft_r<DIR, R>(a);
#pragma unroll
        for (int q = 0; q < R; q++) st(row, j + q * mm, a[q]);
    }
}

// inplace_rows with DIT = true and PAD, its result to st instead of shared memory (one round
// trip and one barrier fewer).  No barrier at the end.
template <int DIR, typename V, class St>
__device__ __forceinline__ void dit_rows_to(V* buf, int nrows, int rs, const DifDev& f, const V* __restrict__ tw, St st) {
    for (int s = f.nst - 1; s > 0; s--) {
        stage_switch<DIR, true, true>(buf, nrows, rs, f, s, tw);
        __syncthreads();
    }
    if (f.nst == 0) {  // n = 1
        for (int r = threadIdx.x; r < nrows; r += blockDim.x) st(r, 0, buf[sidx<true>(r * rs)]);
        return;
    }
    const int mm = f.span[0] / f.radix[0];
    const FastDiv dmm = f.mmdiv[0];
    switch (f.radix[0]) {
#define PRJ_STAGE(R_) \
    case R_: stage_out_r<DIR, R_>(buf, nrows, rs, mm, dmm, tw + f.twoff[0], st); break;
        PRJ_STAGE(2) PRJ_STAGE(3) PRJ_STAGE(4) PRJ_STAGE(5) PRJ_STAGE(6) PRJ_STAGE(7) PRJ_STAGE(8)
        PRJ_STAGE(9) PRJ_STAGE(10) PRJ_STAGE(11) PRJ_STAGE(13)
#undef PRJ_STAGE
    default: break;
    }
}

template <int DIR, typename V>
__device__ void dif_rows(V* buf, int nrows, int rs, const DifDev& f, const V* __restrict__ tw) {
    inplace_rows<DIR, false, false>(buf, nrows, rs, f, tw);
}

template <int DIR, typename V>
__device__ void dit_rows(V* buf, int nrows, int rs, const DifDev& f, const V* __restrict__ tw) {
    inplace_rows<DIR, true, false>(buf, nrows, rs, f, tw);
}

}  // namespace prj
