// prj_zslab.cu -- the z direction of the solve with a whole x wavenumber on chip.
//
// A cluster of C CTAs owns one x wavenumber kx: CTA c keeps the H spectral z-rows
// X[y][kx][:] of the planes y = c H .. c H + H - 1 in shared memory from the copy in to the
// store out, so the spectrum crosses the memory system twice (rows in, rows out) where the
// split kernels (prj_zsplit.cu) move it eight times and k_zline (prj_zline.cu) four times:
//
//   rows in (one TMA box, or 16-byte cp.async copies when n is no multiple of 8) and the
//   planes' pivot rows (cp.async);
//   forward z FFT of the H rows in place;
//   forward Thomas sweep of the H planes: CTA c takes d' of the plane below from CTA c - 1
//   (st.async into c's shared memory, completed on c's mbarrier) and hands its last one on;
//   c'_y = c_y / D_y over the pivot rows, once per wavenumber pair;
//   backward sweep, the values handed down from CTA c + 1 to c;
//   inverse z FFT in place, the last pass storing natural-order rows.
//
// A sweep is one dependent chain per line whichever CTA runs it, so handing the chain over
// at the CTA boundary costs no more than the hand-over itself, while the copies and both
// FFTs run on all C CTAs.  The butterflies, tables and Thomas operation order are those of
// the other z kernels (poisson_solver_multigpu.f90:401-419, round-to-nearest intrinsics,
// c_y / D_y correctly rounded as tabulated there), so the results are the same bits.
//
// Every wait on an mbarrier is bounded (a clock budget); a CTA whose wait runs out raises
// the plan's error word, waits (bounded) for its own row copy and leaves through the cluster
// barrier, so that no CTA exits while a neighbour can still write to its shared memory.  In the ordinary path a CTA's last
// incoming stores are the ones it has waited for.
#include <cuda.h>

#include "chain.cuh"
#include "cluster_util.cuh"
#include "cp_async.cuh"
#include "div_rn.cuh"
#include "fft_pass.cuh"
#include "prj_internal.h"
#include "thomas_block.cuh"
#include "zline_tiles.cuh"

namespace prj {

namespace {

struct ZSlabArgs {
    int n, ny, nh, nzh, mzp;
    int rs, H, hp;        // row stride in elements (n rounded up to 8), planes per CTA, pivot pitch
    int tma;              // rows by the tensor map (n a multiple of 8)
    FastDiv nzhdiv;
    DifDev f;             // runtime radices (RuntimeFft)
    const double2* tw;
    const double* bands;  // a, b, c, a00, b00, c00
    const double* piv;    // D[y][kx][kzs]
    const int* pair;      // pivot pair of each slot (n), then of each kz <= n/2
    double2* X;           // [y][kx][z]
    int* err;             // raised (7) when a bounded wait gives up
};

// in-place row transforms: forward natural -> slot order, inverse slot -> natural with the
// last pass handed to st(row, e, value)
template <class PL>
struct PassFft {
    static __device__ __forceinline__ void forward(double2* buf, int nr, int rs, const ZSlabArgs& a) {
        dif_passes_shared<-1, PL, 0, PL::P>(buf, nr, rs, a.tw);
    }
    template <class St>
    static __device__ __forceinline__ void inverse(double2* buf, int nr, int rs, const ZSlabArgs& a, St st) {
        dit_passes_shared<+1, PL, PL::P - 1, 0>(buf, nr, rs, a.tw);
        dit_last_pass<+1, PL>(buf, nr, rs, a.tw, st);
    }
};

// lengths without a compile-time plan: the runtime-radix passes
struct RuntimeFft {
    static __device__ __forceinline__ void forward(double2* buf, int nr, int rs, const ZSlabArgs& a) {
        inplace_rows<-1, false, true>(buf, nr, rs, a.f, a.tw);
    }
    template <class St>
    static __device__ __forceinline__ void inverse(double2* buf, int nr, int rs, const ZSlabArgs& a, St st) {
        dit_rows_to<+1>(buf, nr, rs, a.f, a.tw, st);
    }
};

// planes of a line per block of the sweeps (two blocks' values in registers)
__host__ __device__ constexpr int slab_up(int lpt) { return lpt > 1 ? 1 : 2; }
__host__ __device__ constexpr int slab_down(int lpt) { return lpt > 2 ? 1 : 4 / lpt; }

__host__ __device__ inline size_t slab_row_bytes(int rs) { return (size_t)rs * 18; }
__host__ __device__ inline size_t slab_rows_bytes(int rs, int H) { return ((size_t)H * slab_row_bytes(rs) + 127) / 128 * 128; }
// Pivots in shared memory: D_y and 1 / D_y as [pair][plane], H planes padded to whole blocks
// of four and an odd number of 16-byte pieces.  Lines in slot order meet pairs in (or against) the order of their
// numbers, so the eight lanes of a 16-byte access -- two planes of a line -- fall on eight
// bank groups.  (Rows of pivots by wavenumber, which the slots meet in digit-reversed order,
// cost 6 wavefronts per warp and plane for each of the two; the sweep then ran at 208
// cycles a plane for n = 192, 146 for n = 64.)
__host__ __device__ inline int slab_pitch(int H) { return ((H + 3) / 4 * 2 | 1) * 2; }
// 128 bytes of alignment slack and 128 of mbarriers, the rows, the pivots and their
// reciprocals, the carry row, the planes' a, a00, c and c00
inline size_t slab_smem(int n, int H) {
    return 256 + slab_rows_bytes((n + 7) & ~7, H) + (size_t)2 * (n / 2 + 1) * slab_pitch(H) * sizeof(double) +
           (size_t)n * sizeof(double2) + (size_t)4 * H * sizeof(double);
}

// planes 0 .. B - 1 of a pair (B = 1, or even and at an even plane; the pitch covers them)
template <int B>
__device__ __forceinline__ void slab_planes_of(double (&o)[B], const double* p) {
    if constexpr (B == 1) {
        o[0] = p[0];
    } else {
#pragma unroll
        for (int u = 0; u < B; u += 2) {
            const double2 v = *reinterpret_cast<const double2*>(p + u);
            o[u] = v.x;
            o[u + 1] = v.y;
        }
    }
}

// NT threads, LPT lines per thread (NT LPT >= n)
template <class FFT, int NT, int LPT>
__global__ void __launch_bounds__(NT, 512 / NT) k_zslab(const __grid_constant__ ZSlabArgs a,
                                                        const __grid_constant__ CUtensorMap tmap) {
    extern __shared__ __align__(128) unsigned char zsm[];
    chain_trigger();
    const int tid = threadIdx.x, c = (int)cluster_rank(), C = (int)gridDim.x, kx = blockIdx.y;
    const int n = a.n, ny = a.ny, nh = a.nh, rs = a.rs, H = a.H, hp = a.hp;
    const int y0 = c * H, nr = min(H, ny - y0);  // at least one plane per CTA
    unsigned char* base = align128(zsm);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base);  // [0] rows in, [1] carry in
    double2* buf = reinterpret_cast<double2*>(base + 128);
    double* dbuf = reinterpret_cast<double*>(base + 128 + slab_rows_bytes(rs, H));  // D_y, later c_y / D_y
    double* rbuf = dbuf + a.nzh * hp;                                               // 1 / D_y
    double2* carry = reinterpret_cast<double2*>(rbuf + a.nzh * hp);
    double* abuf = reinterpret_cast<double*>(carry + n);  // a, a00, c, c00
    const int rp = rs / 8 * 9;  // slots from one row to the next
    const uint32_t carry_bytes = (uint32_t)n * (uint32_t)sizeof(double2);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_fence_init();
        // the first carry: d' from below, or (CTA 0) x from above
        if (C > 1) mbar_arrive_expect_tx(&bars[1], carry_bytes);
    }
    cluster_arrive();  // this CTA's mbarriers are set up (waited for before the first st_async)
    for (int i = tid; i < 4 * nr; i += NT) {  // a, a00, c, c00 of the planes
        const int k = i / nr, r = i - k * nr;
        cp_async(abuf + k * H + r, a.bands + (size_t)((k & 1) * 3 + (k >> 1) * 2) * ny + y0 + r, 8);
    }
    cp_async_commit();
    // the pivots and their reciprocals, once per wavenumber pair and off the sweep's chain,
    // while the rows arrive; eight loads in flight
    for (int i0 = tid; i0 < nr * a.nzh; i0 += 8 * NT) {
        double D[8];
        int to[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = i0 + u * NT, r = fdiv(i, a.nzhdiv), k = i - r * a.nzh;
            if (i < nr * a.nzh) {
                D[u] = a.piv[((size_t)(y0 + r) * nh + kx) * a.mzp + k];
                to[u] = a.pair[n + k] * hp + r;
            }
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (i0 + u * NT < nr * a.nzh) {
                dbuf[to[u]] = D[u];
                rbuf[to[u]] = __drcp_rn(D[u]);
            }
        }
    }
    // this thread's lines.  A slot past n holds none: its values are zeros that no shared-memory
    // read supplies (the cells of the lines change under their own threads' sweeps, between
    // barriers), and a thread without a line takes no part in the sweeps.
    int at[LPT], piv[LPT], slot[LPT];
#pragma unroll
    for (int q = 0; q < LPT; q++) {
        slot[q] = tid + q * NT;
        const int sq = slot[q] < n ? slot[q] : 0;
        at[q] = sq + (sq >> 3);
        piv[q] = a.pair[sq] * hp;
    }
    // the rows, once the kernel that wrote them is done
    chain_wait();
    if (a.tma) {
        if (tid == 0) {
            mbar_arrive_expect_tx(&bars[0], (uint32_t)(slab_row_bytes(n) * a.H));
            tma_load_4d(buf, &tmap, 0, 0, kx, y0, &bars[0]);
        }
    } else {
        for (int r = 0; r < nr; r++) {
            const double2* src = a.X + ((size_t)(y0 + r) * nh + kx) * n;
            for (int e = tid; e < n; e += NT) cp_async(buf + (size_t)r * rp + e + (e >> 3), src + e, 16);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    bool ok = true;
    __syncthreads();  // the mbarrier is set up, the cp.async copies are in
    if (y0 == 0 && tid < 2) abuf[tid * H] = 0.0;  // a_0 plays no part (sweep_up)
    if (a.tma) ok = mbar_wait_bounded(&bars[0], 0);
    ok = !__syncthreads_or(!ok);
    cluster_wait();
    if (ok) FFT::forward(buf, nr, rs, a);  // a barrier after every pass

    uint32_t phase = 0;
    // ------------------------------------------------------------ forward sweep
    double2 prev[LPT];
#pragma unroll
    for (int q = 0; q < LPT; q++) prev[q] = make_double2(0.0, 0.0);
    if (ok && c > 0) {
        ok = mbar_wait_cluster(&bars[1], phase);
        phase ^= 1u;
        ok = !__syncthreads_or(!ok);
        if (ok) {
#pragma unroll
            for (int q = 0; q < LPT; q++)
                if (slot[q] < n) prev[q] = carry[slot[q]];
        }
        // the next carry (x from above): this CTA's part of the chain is not handed on
        // before this thread has armed it
        if (tid == 0 && c < C - 1) mbar_arrive_expect_tx(&bars[1], carry_bytes);
    }
    if (ok) {
        const uint32_t up = c < C - 1 ? cluster_map(carry, (uint32_t)(c + 1)) : 0u;
        const uint32_t upbar = c < C - 1 ? cluster_map(&bars[1], (uint32_t)(c + 1)) : 0u;
        // the loads of a block are issued a block ahead
        constexpr int B = slab_up(LPT);
        double2 below[LPT];
#pragma unroll
        for (int q = 0; q < LPT; q++) below[q] = prev[q];
        unsigned outside = 0;
        struct Block {
            double2 v[LPT][B];
            double D[LPT][B], rD[LPT][B], a[LPT][B];
        } even, odd;
        auto load = [&](Block& k, int r0) {
#pragma unroll
            for (int q = 0; q < LPT; q++) {
                slab_planes_of<B>(k.D[q], dbuf + piv[q] + r0);
                slab_planes_of<B>(k.rD[q], rbuf + piv[q] + r0);
#pragma unroll
                for (int u = 0; u < B; u++) {
                    const int r = min(r0 + u, nr - 1);
                    k.v[q][u] = slot[q] < n ? buf[at[q] + r * rp] : make_double2(0.0, 0.0);
                    k.a[q][u] = abuf[(kx == 0 && piv[q] == 0 ? H : 0) + r];
                }
            }
        };
        auto sweep = [&](Block& k, int r0) {
            const int nb = min(B, nr - r0);
            sweep_up<B, LPT>(k.v, k.D, k.rD, k.a, nb, prev, outside);
#pragma unroll
            for (int q = 0; q < LPT; q++)
#pragma unroll
                for (int u = 0; u < B; u++)
                    if (u < nb && slot[q] < n) buf[at[q] + (r0 + u) * rp] = k.v[q][u];
        };
        if (slot[0] < n) {
            load(even, 0);
            for (int r0 = 0; r0 < nr; r0 += 2 * B) {
                load(odd, min(r0 + B, nr - 1) / B * B);
                sweep(even, r0);
                if (r0 + B >= nr) break;
                load(even, min(r0 + 2 * B, nr - 1) / B * B);
                sweep(odd, r0 + B);
            }
        }
        // a quotient that may differ: the rows again from memory, which still holds them, and
        // the sweep by plain division
        if (__syncthreads_or(outside != 0)) {
            for (int r = 0; r < nr; r++)
                for (int e = tid; e < n; e += NT)
                    buf[(size_t)r * rp + e + (e >> 3)] = a.X[((size_t)(y0 + r) * nh + kx) * n + e];
            __syncthreads();
            FFT::forward(buf, nr, rs, a);
#pragma unroll
            for (int q = 0; q < LPT; q++) {
                if (slot[q] >= n) continue;
                prev[q] = below[q];
                for (int r = 0; r < nr; r++) {
                    prev[q] = step_up_safe(buf[at[q] + r * rp], dbuf[piv[q] + r],
                                           abuf[(kx == 0 && piv[q] == 0 ? H : 0) + r], prev[q]);
                    buf[at[q] + r * rp] = prev[q];
                }
            }
        }
        if (c < C - 1) {
#pragma unroll
            for (int q = 0; q < LPT; q++)
                if (slot[q] < n) st_async(up + (uint32_t)slot[q] * 16u, prev[q], upbar);
        }
        // the back-substitution factors c'_y = c_y / D_y in the pivots' place, two planes at
        // a time (c_{ny-1} / D_{ny-1} and the pad planes are not used)
        __syncthreads();
        const int np = (nr + 1) / 2;
        for (int i = tid; i < a.nzh * np; i += NT) {
            const int j = i / a.nzh, p = i - j * a.nzh;
            double2* d = reinterpret_cast<double2*>(dbuf + p * hp) + j;
            const double2 rD = reinterpret_cast<const double2*>(rbuf + p * hp)[j];
            const double* cy = abuf + (kx == 0 && p == 0 ? 3 * H : 2 * H) + 2 * j;
            const double c0 = cy[0], c1 = 2 * j + 1 < nr ? cy[1] : 0.0;
            unsigned outside = 0;
            double2 f = make_double2(div_by_recip(c0, d->x, rD.x, outside),
                                     div_by_recip(c1, d->y, rD.y, outside));
            if (outside) f = make_double2(__ddiv_rn(c0, d->x), __ddiv_rn(c1, d->y));
            *d = f;
        }
        __syncthreads();
    }
    // ----------------------------------------------------------- backward sweep
    if (ok && c < C - 1) {
        ok = mbar_wait_cluster(&bars[1], phase);
        phase ^= 1u;
        ok = !__syncthreads_or(!ok);
        if (ok) {
#pragma unroll
            for (int q = 0; q < LPT; q++)
                if (slot[q] < n) prev[q] = carry[slot[q]];
        }
    }
    if (ok) {
        const uint32_t dn = c > 0 ? cluster_map(carry, (uint32_t)(c - 1)) : 0u;
        const uint32_t dnbar = c > 0 ? cluster_map(&bars[1], (uint32_t)(c - 1)) : 0u;
        const int top = c == C - 1 ? nr - 2 : nr - 1;  // x_{ny-1} = d'_{ny-1}, still in prev
        constexpr int B = slab_down(LPT);
        struct Block {
            double2 v[LPT][B];
            double f[LPT][B];
        } even, odd;
        auto load = [&](Block& k, int r0) {
#pragma unroll
            for (int q = 0; q < LPT; q++) {
                slab_planes_of<B>(k.f[q], dbuf + piv[q] + r0);
#pragma unroll
                for (int u = 0; u < B; u++)
                    k.v[q][u] = slot[q] < n ? buf[at[q] + min(r0 + u, nr - 1) * rp] : make_double2(0.0, 0.0);
            }
        };
        auto sweep = [&](Block& k, int r0) {
            const int nb = min(B, top + 1 - r0);
            sweep_down<B, LPT>(k.v, k.f, nb, prev);
#pragma unroll
            for (int q = 0; q < LPT; q++)
#pragma unroll
                for (int u = 0; u < B; u++)
                    if (u < nb && slot[q] < n) buf[at[q] + (r0 + u) * rp] = k.v[q][u];
        };
        if (top >= 0 && slot[0] < n) {
            int r0 = top / B * B;
            load(even, r0);
            for (; r0 >= 0; r0 -= 2 * B) {
                load(odd, max(r0 - B, 0));
                sweep(even, r0);
                if (r0 < B) break;
                load(even, max(r0 - 2 * B, 0));
                sweep(odd, r0 - B);
            }
        }
        if (c > 0) {
#pragma unroll
            for (int q = 0; q < LPT; q++)
                if (slot[q] < n) st_async(dn + (uint32_t)slot[q] * 16u, prev[q], dnbar);
        }
        __syncthreads();
        FFT::inverse(buf, nr, rs, a, RowStore<double2>{a.X + ((size_t)y0 * nh + kx) * n, (size_t)nh * n});
    }
    if (!ok) {
        if (tid == 0) atomicExch(a.err, 7);
        cluster_leave(a.tma ? &bars[0] : nullptr);
    }
}

using SlabKernel = void (*)(ZSlabArgs, CUtensorMap);
constexpr int kSlabThreads = 256;
constexpr int kSlabMaxN = 512;

template <class FFT, int N>
SlabKernel slab_kernel_n() {
    if constexpr (N <= kSlabMaxN) return k_zslab<FFT, kSlabThreads, (N + kSlabThreads - 1) / kSlabThreads>;
    else return nullptr;
}

// the kernel of the plan's z length (nz <= kSlabMaxN), by the radix order in use
SlabKernel slab_kernel(const prj_plan* pl) {
    const int nz = pl->g.nz;
#define PRJ_SLAB_CASE(N, ...)                                          \
    if (nz == N && same_radices<PassList<__VA_ARGS__>>(pl->zd.f))      \
        return slab_kernel_n<PassFft<PassList<__VA_ARGS__>>, N>();
    PRJ_PASS_ALL(PRJ_SLAB_CASE)
#undef PRJ_SLAB_CASE
    return nz <= 256 ? k_zslab<RuntimeFft, kSlabThreads, 1> : k_zslab<RuntimeFft, kSlabThreads, 2>;
}

}  // namespace

// planes per CTA of the slab kernel, 0 where it does not apply: the plan's z_planes tuning, or
// the fewest CTAs per wavenumber (at most 8) with which every cluster is resident at once, up to
// nz = 512.  The kernel is one dependent pass over the planes, so a second wave of clusters doubles
// its time, and how many are resident is asked of the runtime.  Measured (Poisson solve, us, slab
// / three kernels), 20 / 29 at 48 x 32 x 24, 37 / 51 at 128 x 96 x 64, 49 / 59 at 512 x 55 x 64, 78 /
// 118 at 64 x 324 x 80, each in one wave, but 119 / 124 at 256 x 128 x 128, 155 / 123 at 32 x 256 x
// 224 and 134 / 73 at 32 x 68 x 768 in more.  With three lines per thread and more the chain
// loses in one wave too: 87 / 64 at 32 x 64 x 640, 68 / 50 at 32 x 32 x 1000; 44 / 46 at 64 x 32 x 512.
int zslab_planes(const prj_plan* pl) {
    const Geometry& g = pl->g;
    // z kernels, a row count, a ring or a stage count chosen by the plan's tuning stand
    if (!pl->z_auto || pl->zfft_rows != 0 || pl->thomas_async != -1 || pl->z_stages != 0) return 0;
    if (!pl->zd.ok || !pl->kz_of_slot || !pl->t.piv || !pl->spec || g.nz > kSlabMaxN) return 0;
    const SlabKernel kernel = slab_kernel(pl);
    auto one_wave = [&](int H) {
        const int C = (g.ny + H - 1) / H;
        if (C > 8 || H > 256) return false;  // 256 planes: a tensor-map box
        const size_t smem = slab_smem(g.nz, H);
        if (smem + 1024 > (size_t)220 * 1024) return false;
        const int per_sm = std::min((int)((size_t)228 * 1024 / (smem + 1024)), 2);  // two by registers
        return clusters_resident(kernel, kSlabThreads, smem, (unsigned)C, g.nxh, per_sm * pl->sms);
    };
    if (pl->z_planes > 0) {
        // chunks of the kernel that z_mode 1 or 3 runs by default; else planes per CTA here
        const int H = std::min(pl->z_planes, g.ny);
        return pl->zmode == 0 && one_wave(H) ? H : 0;
    }
    for (int C = 1; C <= 8 && C <= g.ny; C++) {
        const int H = (g.ny + C - 1) / C;
        if (one_wave(H)) return H;
    }
    return 0;
}

cudaError_t launch_zslab(const prj_plan* pl, cudaStream_t st) {
    const Geometry& g = pl->g;
    const int H = pl->slab_h;
    if (H <= 0) return cudaErrorNotSupported;
    ZSlabArgs a{};
    a.n = g.nz; a.ny = g.ny; a.nh = g.nxh; a.nzh = g.nzh; a.nzhdiv = make_fastdiv((unsigned)g.nzh); a.mzp = g.mzp;
    a.rs = (g.nz + 7) & ~7; a.H = H; a.hp = slab_pitch(H);
    a.f = pl->zd.f; a.tw = pl->zd.tw; a.bands = pl->t.bands; a.piv = pl->t.piv;
    a.pair = pl->kz_of_slot + g.nz; a.X = pl->spec;
    a.err = reinterpret_cast<int*>(pl->stat_buf + kStatErrSlot);
    CUtensorMap tm{};
    a.tma = zline_tmap(&tm, pl->spec, g.nz, g.nxh, g.ny, H) ? 1 : 0;
    const unsigned C = (unsigned)((g.ny + H - 1) / H);
    const size_t smem = slab_smem(g.nz, H);
    const SlabKernel kernel = slab_kernel(pl);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return e;
    return launch_chained(chained(pl), kernel, dim3(C, (unsigned)g.nxh), kSlabThreads, smem, st, C, a, tm);
}

}  // namespace prj
