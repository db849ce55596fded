// thomas_block.cuh -- the forward Thomas recurrence of a block of planes, shared by the z
// kernels: d'_y = (d_y - a_y d'_{y-1}) / D_y for B planes of L lines held in registers, in
// the reference's operation order (poisson_solver_multigpu.f90:401-419, round-to-nearest
// intrinsics), the quotients correctly rounded (div_rn.cuh).
//
// The recurrence is one dependent chain per line, so its length in cycles is what a kernel
// with few warps per SM waits for.  A block runs the branch-free quotients and leaves in
// `outside` whether any may differ; the caller, which still has the block's inputs, tests it
// after a block or after many and then redoes them plane by plane with step_up_safe.  (On one
// warp, cycles per plane: 199 with a branch per quotient, 120 / 92 with one per four / eight
// planes, 68 with none in the loop, 59 without the tests.)  A y = 0 plane has a_y = 0 and
// prev = +0, which leaves d_0 as it is, its sign included.
#pragma once
#include "div_rn.cuh"

namespace prj {

// B planes of L lines: v holds d_y on entry, d'_y on exit; D, rD = RN(1/D) and a per plane;
// prev: d' of the plane below, then of plane nb - 1.  Planes nb .. B - 1 are left alone (a
// whole block runs without a test per plane).
template <int B, int L>
__device__ __forceinline__ void sweep_up(double2 (&v)[L][B], const double (&D)[L][B], const double (&rD)[L][B],
                                         const double (&a)[L][B], int nb, double2 (&prev)[L], unsigned& outside) {
    auto plane = [&](int u) {
#pragma unroll
        for (int q = 0; q < L; q++) {
            const double x = __dsub_rn(v[q][u].x, __dmul_rn(a[q][u], prev[q].x));
            const double y = __dsub_rn(v[q][u].y, __dmul_rn(a[q][u], prev[q].y));
            prev[q].x = div_by_recip(x, D[q][u], rD[q][u], outside);
            prev[q].y = div_by_recip(y, D[q][u], rD[q][u], outside);
            v[q][u] = prev[q];
        }
    };
    if (nb == B) {
#pragma unroll
        for (int u = 0; u < B; u++) plane(u);
    } else {
#pragma unroll
        for (int u = 0; u < B - 1; u++)
            if (u < nb) plane(u);
    }
}

// x_y = d'_y - (c_y / D_y) x_{y+1} of B planes from plane nb - 1 down to 0: v in and out
template <int B, int L>
__device__ __forceinline__ void sweep_down(double2 (&v)[L][B], const double (&f)[L][B], int nb, double2 (&prev)[L]) {
    auto plane = [&](int u) {
#pragma unroll
        for (int q = 0; q < L; q++) {
            prev[q].x = __dsub_rn(v[q][u].x, __dmul_rn(prev[q].x, f[q][u]));
            prev[q].y = __dsub_rn(v[q][u].y, __dmul_rn(prev[q].y, f[q][u]));
            v[q][u] = prev[q];
        }
    };
    if (nb == B) {
#pragma unroll
        for (int u = B - 1; u >= 0; u--) plane(u);
    } else {
#pragma unroll
        for (int u = B - 2; u >= 0; u--)
            if (u < nb) plane(u);
    }
}

// one step of one line by plain division, the redone block's
__device__ __forceinline__ double2 step_up_safe(double2 d, double D, double a, double2 prev) {
    return make_double2(__ddiv_rn(__dsub_rn(d.x, __dmul_rn(a, prev.x)), D),
                        __ddiv_rn(__dsub_rn(d.y, __dmul_rn(a, prev.y)), D));
}

}  // namespace prj
