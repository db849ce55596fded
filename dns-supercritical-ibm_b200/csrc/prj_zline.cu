// prj_zline.cu -- the z direction of the solve as one kernel per x wavenumber,
// built on the pass-plan butterflies (fft_pass.cuh).
//
// One CTA owns one x wavenumber kx: the ny spectral z-rows X[y][kx][:] and the nz
// Thomas lines (kx, slot) that run through them (zline_tile, zline_tiles.cuh: z FFT,
// both Thomas sweeps and the inverse z FFT, the spectrum crossing HBM four times).
// Each thread owns LPT lines (slots tid + q NT) and carries their recurrence in
// registers.  The rows of each chunk of planes arrive by one TMA copy through a 4-D
// tensor map of the spectrum (zline_tmap, encoded on the host for every launch with the
// driver's cuTensorMapEncodeTiled); a map the driver refuses sends the solve to the split
// kernels.
#include <cuda.h>

#include "chain.cuh"
#include "div_rn.cuh"
#include "fft_pass.cuh"
#include "prj_internal.h"
#include "zline_tiles.cuh"

namespace prj {

namespace {

// `tmap` (zline_tmap) is a kernel parameter: the TMA unit reads it from parameter space
template <class PL, int NS, int LPT>
__global__ void __launch_bounds__(zl_threads(PL::n, LPT), zl_minb(zl_threads(PL::n, LPT)))
    k_zline(const __grid_constant__ ZLineArgs a, const __grid_constant__ CUtensorMap tmap) {
    extern __shared__ __align__(128) unsigned char zsm[];
    zline_tile<PL, NS, LPT, zl_threads(PL::n, LPT)>(a, &tmap, blockIdx.x, zsm);
}

template <class PL, int NS, int LPT>
cudaError_t launch_zline_pl(const ZLineArgs& a, const CUtensorMap& tm, size_t smem, cudaStream_t st) {
    cudaError_t e =
        cudaFuncSetAttribute(k_zline<PL, NS, LPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_zline<PL, NS, LPT><<<a.nh, zl_threads(PL::n, LPT), smem, st>>>(a, tm);
    return cudaGetLastError();
}

// a cluster of a.C CTAs per wavenumber (two stages)
template <class PL>
__global__ void __launch_bounds__(zl_threads(PL::n, zl_lpt(PL::n)), zl_minb(zl_threads(PL::n, zl_lpt(PL::n))))
    k_zline_cluster(const __grid_constant__ ZLineArgs a, const __grid_constant__ CUtensorMap tmap) {
    extern __shared__ __align__(128) unsigned char zsm[];
    zline_tile<PL, 2, zl_lpt(PL::n), zl_threads(PL::n, zl_lpt(PL::n)), 2, true>(a, &tmap, blockIdx.x / a.C, zsm);
}

template <class PL>
cudaError_t launch_zline_ns(const ZLineArgs& a, const CUtensorMap& tm, int ns, size_t smem, cudaStream_t st) {
    constexpr int L = zl_lpt(PL::n);
    switch (ns) {
    case 2: return launch_zline_pl<PL, 2, L>(a, tm, smem, st);
    case 3: return launch_zline_pl<PL, 3, L>(a, tm, smem, st);
    default: return launch_zline_pl<PL, 4, L>(a, tm, smem, st);
    }
}


}  // namespace

bool zline_supported(const prj_plan* pl) {
    if (!pl->use_pass || !pl->zd.ok || !pl->kz_of_slot || !pl->t.pivc || !pl->spec) return false;
    CUtensorMap tm{};
    if (!zline_tmap(&tm, pl->spec, pl->g.nz, pl->g.nxh, pl->g.ny, 1)) return false;  // the driver's answer
#define PRJ_ZL_HAS(N, ...)                                                          \
    if (pl->g.nz == N && same_radices<PassList<__VA_ARGS__>>(pl->zd.f))             \
        return zline_smem(N, pl->g.mzp, 1, 2) <= (size_t)200 * 1024;
    PRJ_PASS_ALL(PRJ_ZL_HAS)
#undef PRJ_ZL_HAS
    return false;
}

ZLineArgs zline_args(const prj_plan* pl) {
    const Geometry& g = pl->g;
    ZLineArgs a{};
    a.ny = g.ny; a.nh = g.nxh; a.mzp = g.mzp;
    a.yb = pl->z_planes > 0 ? pl->z_planes : 4;
    a.tw = pl->zd.tw; a.bands = pl->t.bands; a.piv = pl->t.piv; a.pivc = pl->t.pivc;
    a.kz_of_slot = pl->kz_of_slot; a.X = pl->spec;
    a.err = reinterpret_cast<int*>(pl->stat_buf + kStatErrSlot);
    return a;
}

bool tmap_encode_f64(void* tmap128, const void* base, int rank, const uint64_t* dims, const uint64_t* strides,
                     const uint32_t* box) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode enc = []() -> Encode {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (!enc || !base || rank < 1 || rank > 5 || ((uintptr_t)base & 15u) != 0) return false;
    cuuint64_t d[5], st[4];
    cuuint32_t b[5], e[5];
    for (int i = 0; i < rank; i++) {
        d[i] = dims[i];
        b[i] = box[i];
        e[i] = 1;
        if (i + 1 < rank) st[i] = strides[i];
    }
    return enc(static_cast<CUtensorMap*>(tmap128), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t)rank,
               const_cast<void*>(base), d, st, b, e, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool zline_tmap(void* tmap128, const double2* X, int n, int nh, int ny, int yb) {
    if (n % 8 != 0 || n / 8 > 256 || yb < 1 || yb > 256) return false;
    const uint64_t dims[4] = {16, (uint64_t)(n / 8), (uint64_t)nh, (uint64_t)ny};
    const uint64_t strides[3] = {128, (uint64_t)n * 16, (uint64_t)nh * (uint64_t)n * 16};  // bytes
    const uint32_t box[4] = {18, (uint32_t)(n / 8), 1, (uint32_t)yb};
    return tmap_encode_f64(tmap128, X, 4, dims, strides, box);
}

// the cluster kernel of the plan's z length, null for the lengths that its rule leaves out
using ZClusterKernel = void (*)(ZLineArgs, CUtensorMap);
constexpr int kZClusterMaxN = 384;
template <class PL>
static ZClusterKernel zcluster_kernel_of() {
    if constexpr (PL::n <= kZClusterMaxN) return k_zline_cluster<PL>;
    else return nullptr;
}
static ZClusterKernel zcluster_kernel(const prj_plan* pl) {
#define PRJ_ZL_CASE(N, ...) \
    if (pl->g.nz == N && same_radices<PassList<__VA_ARGS__>>(pl->zd.f)) return zcluster_kernel_of<PassList<__VA_ARGS__>>();
    PRJ_PASS_ALL(PRJ_ZL_CASE)
#undef PRJ_ZL_CASE
    return nullptr;
}

// CTAs per wavenumber C and planes per chunk of the cluster form; C = 0 where it does not apply.
// The most CTAs, up to 4, whose clusters are all resident at once (as the runtime answers): a
// second wave would double the chain.  Measured (Poisson solve, us, by cluster / one CTA / three
// kernels): 102 / 118 / 124 at 256 x 128 x 128 (C = 3), 306 / 323 / 366 at 384 x 192 x 192 (C = 2),
// 212 / 287 / 244 at 96 x 300 x 256 and 79 / 150 / 79 at 48 x 105 x 384 (C = 4; 322 and 96 with 8, the
// first in two waves), 203 / 426 / 246 at 64 x 300 x 384 (238 with 8).  Lengths above 384 gain
// little or lose: 82 / 119 / 72 at 64 x 64 x 512, 598 / 1032 / 544 at 96 x 292 x 768.  So do short chains
// of the longest rows on one to one and a half CTAs per SM, where some SMs hold two and most one:
// 72 / - / 65 at 96 x 53 x 384 and 81 / - / 76 at 90 x 53 x 384, but 90 / - / 94 at 96 x 80 x 384, 74 / - /
// 75 at 128 x 53 x 384 and 54 / - / 57 at 96 x 60 x 256.
// C = 1 (k_zline) below two wavenumbers per SM, from where z_mode's default takes it: with a
// wavenumber per SM up to nz = 384 and 1.25 up to 768, 1.5 for chains below 64 planes (one CTA / three
// kernels): 412 / 426 at 400 x 72 x 512, 1054 / 1106 at 400 x 128 x 768 and 368 / 394 at 450 x 60 x 512, but
// 933 / 886 at 300 x 200 x 512, 938 / 855 at 300 x 128 x 768, 184 / 175 at 384 x 36 x 512, and with four
// and eight lines per thread 1234 / 1082 at 400 x 100 x 1024, 1061 / 830 at 300 x 60 x 1536.
void zline_cluster_shape(const prj_plan* pl, int* C_out, int* yb_out) {
    *C_out = *yb_out = 0;
    const Geometry& g = pl->g;
    // a z kernel, row count, ring, chunk or stage count chosen by the plan's tuning stands
    if (!pl->z_auto || (pl->zmode != 0 && pl->zmode != 3) || pl->zfft_rows != 0 || pl->thomas_async != -1 ||
        pl->z_stages != 0 || pl->z_planes != 0)
        return;
    if (pl->sms <= 0 || !zline_supported(pl)) return;
    const unsigned nt = (unsigned)zl_threads(g.nz, zl_lpt(g.nz));
    const ZClusterKernel kernel = zcluster_kernel(pl);
    if (kernel && g.nz > 256 && g.ny < 64 && 4 * g.nxh > pl->sms && 8 * g.nxh < 3 * pl->sms) return;
    for (int C = kernel ? 4 : 1; C >= 2; C--) {
        const int per_sm = (g.nxh * C + pl->sms - 1) / pl->sms;
        if (per_sm > zl_minb((int)nt)) continue;
        const size_t most = (size_t)228 * 1024 / per_sm - 1024;
        int yb = 8;
        while (yb > 1 && zline_cluster_smem(g.nz, g.mzp, yb, 2) > std::min(most, (size_t)220 * 1024)) yb--;
        if (yb < 2 || yb * C > g.ny) continue;
        // per_sm of them fit an SM by their shared memory, and by registers as the kernel is bound
        if (!clusters_resident(kernel, nt, zline_cluster_smem(g.nz, g.mzp, yb, 2), (unsigned)C, g.nxh, per_sm * pl->sms))
            continue;
        *C_out = C;
        *yb_out = yb;
        return;
    }
    const int quarters = g.nz <= 384 ? 4 : g.ny >= 64 ? 5 : 6;  // of a wavenumber per SM, at least
    if (g.nz <= 768 && 4 * g.nxh >= quarters * pl->sms) *C_out = 1;
}

cudaError_t launch_zline_cluster(const prj_plan* pl, cudaStream_t st) {
    const Geometry& g = pl->g;
    if (pl->zcl_c == 1) return launch_zline(pl, st);
    const ZClusterKernel kernel = zcluster_kernel(pl);
    ZLineArgs a = zline_args(pl);
    a.C = pl->zcl_c;
    a.yb = pl->zcl_yb;
    CUtensorMap tm{};
    if (a.C < 2 || !kernel || !zline_tmap(&tm, pl->spec, g.nz, g.nxh, g.ny, a.yb)) return cudaErrorNotSupported;
    const size_t smem = zline_cluster_smem(g.nz, g.mzp, a.yb, 2);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return e;
    return launch_chained(false, kernel, dim3((unsigned)(a.nh * a.C)), (unsigned)zl_threads(g.nz, zl_lpt(g.nz)), smem, st,
                          (unsigned)a.C, a, tm);
}

// cudaErrorNotSupported when nz has no pass plan (the caller runs the split kernels)
cudaError_t launch_zline(const prj_plan* pl, cudaStream_t st) {
    if (!pl->use_pass || !pl->zd.ok || !pl->kz_of_slot || !pl->t.pivc || !pl->spec) return cudaErrorNotSupported;
    const Geometry& g = pl->g;
    ZLineArgs a = zline_args(pl);
    // planes per stage and stage count: the plan's z_planes / z_stages tuning, else two stages
    // of up to 16 planes, as many as fit beside the CTAs that an SM is to hold (the wavenumbers
    // per SM, as far as registers allow).  A chunk's barriers and waits are shared
    // by its planes: 280 -> 256 us at 768 x 177 x 192 with 8 planes against 4; nz = 384 keeps
    // 4.  Measured at 768x384x384 and not kept: deeper rings at fewer CTAs per SM, and one
    // line per thread (twice the threads, spilling at the register budget of three CTAs).
    int yb = pl->z_planes > 0 ? pl->z_planes : 16, ns = pl->z_stages > 0 ? pl->z_stages : 2;
    const int sms = pl->sms > 0 ? pl->sms : 148;
    const int per_sm = std::min(zl_minb(zl_threads(g.nz, zl_lpt(g.nz))), (g.nxh + sms - 1) / sms);
    const size_t cap = std::min((size_t)228 * 1024 / per_sm - 1024, (size_t)200 * 1024);
    if (ns < 2 || ns > 4) ns = 2;
    if (yb > g.ny) yb = g.ny;
    while (yb > 1 && zline_smem(g.nz, g.mzp, yb, ns) > cap) yb--;
    const size_t smem = zline_smem(g.nz, g.mzp, yb, ns);
    if (smem > (size_t)200 * 1024) return cudaErrorNotSupported;
    a.yb = yb;
    CUtensorMap tm{};
    if (!zline_tmap(&tm, pl->spec, g.nz, g.nxh, g.ny, yb)) return cudaErrorNotSupported;  // split kernels
#define PRJ_ZL_CASE(N, ...)                                                  \
    if (g.nz == N && same_radices<PassList<__VA_ARGS__>>(pl->zd.f))          \
        return launch_zline_ns<PassList<__VA_ARGS__>>(a, tm, ns, smem, st);
    PRJ_PASS_ALL(PRJ_ZL_CASE)
#undef PRJ_ZL_CASE
    return cudaErrorNotSupported;
}

}  // namespace prj
