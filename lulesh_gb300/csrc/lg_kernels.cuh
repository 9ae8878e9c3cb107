// lg_kernels.cuh -- FP64 kernels of the leap-frog cycle (one cycle = 4 launches).
//
// Included by lg_kernels_fp64.cu (compiled with --fmad=false: every operation
// rounds exactly as the reference's -ffp-contract=off build) and by
// lg_kernels_fma.cu (--fmad=true).  LG_NS names the namespace of each copy.
//
//   k_forces      per element: stress (IntegrateStressForElems) and
//                 Flanagan-Belytschko hourglass forces (CalcHourglassControl/
//                 CalcFBHourglassForceForElems) into the per-corner scratch
//   k_nodes       per node: ordered corner gather, a = F/m, symmetry BC,
//                 velocity with u_cut, position (LagrangeNodal)
//   k_kinematics  per element: volume, vnew, delv, arealg, vdov
//                 (CalcKinematicsForElems) and the monotonic-Q gradients
//                 (CalcMonotonicQGradientsForElems)
//   k_material    per element in region order: monotonic-Q limiter, qstop
//                 check, EOS with its repetitions, sound speed, volume
//                 update, Courant/hydro constraints with a block reduction;
//                 its last block finishes the reduction and runs the next
//                 cycle's TimeIncrement.  Small meshes run the same work as
//                 k_material_inputs (per element), k_material_eos (per
//                 repetition item) and k_material_finish (per element)
//
// The FP64 pipe issues 2 lanes per SM and clock and bounds any form of these
// kernels that lives on it, so most of their arithmetic is 64-bit integer
// arithmetic on the other pipes.
//
// The strict build keeps every operation of the reference in its order and with
// its rounding (see the oracle's lulesh_oracle.c for the line-by-line
// correspondence): products, sums of coordinates, quotients and roots as integers
// rounded to nearest even (lg_exact.cuh, lg_exact_geometry.cuh), power-of-two
// factors applied once (lg_geometry.cuh), comparisons of doubles on the integer
// pipe (dlt and friends); the results are the reference operation order's bit for
// bit.  Small meshes take lg_kernels_lanes.cuh and lg_kernels_team.cuh.
//
// The FMA build (LG_REASSOC) works in 64-bit fixed point (lg_fixed_geometry.cuh,
// lg_fixed_eos.cuh): other operations than the reference's, rounded at 2^-59 of
// the largest operand; elements the formats do not hold take FP64 forms out of
// line.
//
// Work the reference does and then discards (the shape-function B matrix that
// CalcElemNodeNormals overwrites, the off-diagonal velocity gradient terms, the
// deviatoric strains, the Courant dt of elements with vdov == 0) is not computed;
// division by refdens is skipped when refdens == 1 (x / 1.0 == x exactly).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "lg_device.h"
#include "lg_geometry.cuh"
#include "lg_fixed_geometry.cuh"
#include "lg_cycle_common.cuh"
#include "lg_exact_geometry.cuh"

#ifndef LG_NS
#error "define LG_NS"
#endif
// LG_REASSOC (the FMA build): fixed-point corner forces, nodal sums and
// kinematics.  Their FP64 forms for the elements the formats do not hold are
// algebraically equal forms of the reference's too.  forces_general: node normals
// and the volume gradient from the element's twelve edge differences
// (node_normals_x8_diff, volume_gradient_x12_diff), the hourglass_modes butterfly,
// the hourglass coefficient by the reciprocal cube root.  kinematics_general: face
// areas from the faces' diagonals (area_face_cross), the velocity-gradient trace and
// the monotonic-Q gradients from the xi/eta/zeta differences of the coordinates and
// velocities (velocity_trace_dirs, monoq_gradients_dirs), lengths by reciprocal
// square roots.  The rounding differs from the reference's operand order, as FMA
// contraction's does; the parity bar covers both.
#ifndef LG_REASSOC
#define LG_REASSOC 0
#endif

namespace lg {
namespace LG_NS {

// element geometry: lg_geometry.cuh
using namespace ::lg::geom;

// ---------------------------------------------------------------------------
// k_forces: CalcVolumeForceForElems (lulesh.cc:1062-1100)
// ---------------------------------------------------------------------------
#if LG_REASSOC
// One element in FP64: the elements the fixed-point formats below do not hold
// (flattened, folded or inverted ones, extreme scales, infinities, NaN).  The
// scratch holds one summed stress + hourglass force per corner and component.
__device__ __noinline__ void forces_general(const DevState &s, const int k, Ctl *ctl,
                                            const double hourg)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    double *const cs = s.corner;
    int nd[8];
    double x[8], y[8], z[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        nd[j] = s.nodelistT[(size_t)j * E + k];
        x[j] = s.x[nd[j]];
        y[j] = s.y[nd[j]];
        z[j] = s.z[nd[j]];
    }
    // 8 x the normals and 12 x the volume gradient from the twelve
    // differences; the 1/8 goes into sig (exact)
    double pf[3][8], gv[3][8];
    const double sig = (-s.p[k] - s.q[k]) * 0.125;
    {
        double dX[12], dY[12], dZ[12];
        elem_differences(x, dX);
        elem_differences(y, dY);
        elem_differences(z, dZ);
        node_normals_x8_diff(pf[0], pf[1], pf[2], dX, dY, dZ);
        volume_gradient_x12_diff(dX, dY, dZ, gv[0], gv[1], gv[2]);
    }
    if (jacobian_det(x, y, z) <= 0.0) raise_status(ctl, -1);  // lulesh.cc:1082-1091
    const double vk = s.v[k];
    const double determ = s.volo[k] * vk;
    if (vk <= 0.0) raise_status(ctl, -1);  // lulesh.cc:1034-1040
    const bool hg = hourg > 0.;
    double hourgam[8][4];
    {
        // 1/(12 volume) folded into the four mode sums
        const double volinv12 = (1.0 / determ) * (1.0 / 12.0);
        double hm[3][4];
        hourglass_modes(x, hm[0]);
        hourglass_modes(y, hm[1]);
        hourglass_modes(z, hm[2]);
#pragma unroll
        for (int i1 = 0; i1 < 4; ++i1) {
            const double hx = volinv12 * hm[0][i1], hy = volinv12 * hm[1][i1],
                         hz = volinv12 * hm[2][i1];
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                hourgam[kk][i1] = gam(i1, kk) - gv[0][kk] * hx - gv[1][kk] * hy - gv[2][kk] * hz;
        }
    }
    const double coefficient = (-hourg * 0.01 * s.ss[k] * s.elemMass[k]) * rcbrt(determ);
    const double *vel[3] = {s.xd, s.yd, s.zd};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double hxx[4] = {0., 0., 0., 0.};
        if (hg) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double u = vel[c][nd[j]];
#pragma unroll
                for (int i = 0; i < 4; i++) hxx[i] += hourgam[j][i] * u;
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            double f = -(sig * pf[c][j]);
            if (hg)
                f += coefficient * (hourgam[j][0] * hxx[0] + hourgam[j][1] * hxx[1] +
                                    hourgam[j][2] * hxx[2] + hourgam[j][3] * hxx[3]);
            cs[c * E8 + (size_t)j * E + k] = f;
        }
    }
}

// One element in fixed point (lg_fixed_geometry.cuh); hourg is the element's
// problem's hourglass coefficient, sm the thread's column of shared memory.
// The FP64 form of this kernel issued 648 FP64 instructions for each element at
// 2 lanes per SM and clock and was bound by them: 3,888 us at s=150.  This one
// issues about 4,700 integer instructions (128 lanes per SM and clock) and 42
// FP64 ones (conversions out, the scale factors), and one summed force for each
// corner and component instead of two: 886 us (issue slots 0.45 full, waits for its
// own results), and the gather in k_nodes 477 -> 314 us (237 with integer sums).
// s=30: 41 -> 16.6 us.  The twelve differences, the
// mode sums and the face areas live in shared memory, whose columns no other
// thread reads, so that the 32 shape terms fit the registers; the components'
// loop is not unrolled to keep the code inside the instruction cache.
template <int BS>
__device__ __forceinline__ void forces_element(const DevState &s, const int k, Ctl *ctl,
                                               const double hourg, fx::i64 *sm)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    const double vk = s.v[k];
    const double determ = s.volo[k] * vk;
    bool ok = fx::seedable(determ);
    int u[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double *p = c == 0 ? s.x : c == 1 ? s.y : s.z;
        double a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = field(&p[nd[j]]);
        ok = fx::force_component(a, c, sm, BS, u[c]) && ok;
    }
    fx::Op shape[8][4];
    ok = fx::force_shape(sm, BS, u, fx::recip(determ) * (1.0 / 12.0), shape) && ok;
    const fx::Scale k1 = fx::scale_of((s.p[k] + s.q[k]) * 0.125, ok);
    fx::Scale k2{0, -5000};
    if (hourg > 0.)
        k2 = fx::scale_of((-hourg * 0.01 * s.ss[k] * s.elemMass[k]) * fx::recip_cbrt(determ), ok);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const double *p = c == 0 ? s.xd : c == 1 ? s.yd : s.zd;
        const int uc = c == 0 ? u[0] : c == 1 ? u[1] : u[2];
        double v[8], F[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = field(&p[nd[j]]);
        ok = fx::force_corners(sm, BS, shape, c, k1, u[0] + u[1] + u[2] - uc, k2, v, F) && ok;
        double *const cs = s.corner + c * E8 + k;
#pragma unroll
        for (int j = 0; j < 8; ++j) cs[(size_t)j * E] = F[j];
    }
    if (!ok || dle(vk, 0.0)) forces_general(s, k, ctl, hourg);
}
#else
// v, negated where bit 0 of sign is set
__device__ __forceinline__ double signed_by(double v, unsigned sign)
{
    return __longlong_as_double(__double_as_longlong(v) ^ ((long long)(sign << 31) << 32));
}

// One element in FP64: the elements whose values the integer forms below do not hold
__device__ __noinline__ void forces_general(const DevState &s, const int k, Ctl *ctl,
                                            const double hourg)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    double *const cs = s.corner;

    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    double x[8], y[8], z[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = field(&s.x[nd[j]]);
        y[j] = field(&s.y[nd[j]]);
        z[j] = field(&s.z[nd[j]]);
    }

    // InitStressTermsForElems (273-286) + IntegrateStressForElems (494-587)
    {
        double pfx[8], pfy[8], pfz[8];
        // 16 x the normals, the 1/16 in sig (exact)
        const double sig = (-s.p[k] - s.q[k]) * 0.0625;
        node_normals_x16(pfx, pfy, pfz, x, y, z);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            cs[0 * E8 + (size_t)j * E + k] = -(sig * pfx[j]);
            cs[1 * E8 + (size_t)j * E + k] = -(sig * pfy[j]);
            cs[2 * E8 + (size_t)j * E + k] = -(sig * pfz[j]);
        }
        // lulesh.cc:1082-1091 uses the Jacobian determinant only for its
        // sign: an FP32 filter with a rigorous error bound settles it, and
        // the FP64 determinant is evaluated only in a warp with an element
        // the filter cannot settle (none on a valid mesh)
        const bool sure = jacobian_certainly_positive(x, y, z);
        if (__any_sync(__activemask(), !sure) && !sure && jacobian_det(x, y, z) <= 0.0)
            raise_status(ctl, -1);
    }

    // CalcHourglassControlForElems (995-1057)
    const double vk = s.v[k];
    const double determ = s.volo[k] * vk;
    if (dle(vk, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1034-1040
    if (!(hourg > 0.)) return;


    // CalcFBHourglassForceForElems (710-991), CalcElemFBHourglassForce (667-706)
    double hourgam[8][4];
    {
        double dvdx[8], dvdy[8], dvdz[8];
        volume_derivative(x, y, z, dvdx, dvdy, dvdz);
        const double volinv = rcp_op(determ);
#pragma unroll
        for (int i1 = 0; i1 < 4; ++i1) {
            const double hourmodx = x[0] * gam(i1, 0) + x[1] * gam(i1, 1) + x[2] * gam(i1, 2) +
                                    x[3] * gam(i1, 3) + x[4] * gam(i1, 4) + x[5] * gam(i1, 5) +
                                    x[6] * gam(i1, 6) + x[7] * gam(i1, 7);
            const double hourmody = y[0] * gam(i1, 0) + y[1] * gam(i1, 1) + y[2] * gam(i1, 2) +
                                    y[3] * gam(i1, 3) + y[4] * gam(i1, 4) + y[5] * gam(i1, 5) +
                                    y[6] * gam(i1, 6) + y[7] * gam(i1, 7);
            const double hourmodz = z[0] * gam(i1, 0) + z[1] * gam(i1, 1) + z[2] * gam(i1, 2) +
                                    z[3] * gam(i1, 3) + z[4] * gam(i1, 4) + z[5] * gam(i1, 5) +
                                    z[6] * gam(i1, 6) + z[7] * gam(i1, 7);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                hourgam[kk][i1] = gam(i1, kk) - volinv * (dvdx[kk] * hourmodx +
                                                          dvdy[kk] * hourmody +
                                                          dvdz[kk] * hourmodz);
        }
    }
    const double ss1 = s.ss[k];
    const double mass1 = s.elemMass[k];
    const double volume13 = cbrt(determ);
    const double coefficient = div_op(-hourg * 0.01 * ss1 * mass1, volume13);
    const double *vel[3] = {s.xd, s.yd, s.zd};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = field(&vel[c][nd[j]]);
        double hxx[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            hxx[i] = hourgam[0][i] * u[0] + hourgam[1][i] * u[1] + hourgam[2][i] * u[2] +
                     hourgam[3][i] * u[3] + hourgam[4][i] * u[4] + hourgam[5][i] * u[5] +
                     hourgam[6][i] * u[6] + hourgam[7][i] * u[7];
#pragma unroll
        for (int i = 0; i < 8; i++)
            cs[(3 + c) * E8 + (size_t)i * E + k] =
                coefficient * (hourgam[i][0] * hxx[0] + hourgam[i][1] * hxx[1] +
                               hourgam[i][2] * hxx[2] + hourgam[i][3] * hxx[3]);
    }
}

// One element; hourg is the element's problem's hourglass coefficient, sm the
// thread's column of shared memory (24 coordinates, then 24 areas, volume derivatives
// and hourglass shapes in turn).  The values are forces_general's bit for bit, with 574
// products and 264 coordinate sums on the integer pipes (lg_exact_geometry.cuh) and
// the other sums on the FP64 pipe, which bounded the FP64 form: 1,290 FP64 instructions
// for each element became 532 (0.6 of that pipe's time) of 28,400 in all: 7,786 -> 4,662
// us at s=150, 77.9 -> 67.7 at s=30, where one or two warps for each scheduler wait
// for their own results.  Faces, components and modes are loops
// that are not unrolled: with all of them unrolled inside a mode the code missed the
// instruction cache and took 6,316 us, against 4,871 with loops at that time.  Each
// corner's hourglass force accumulates over the modes in the reference's order.
template <int BS>
__device__ __forceinline__ void forces_element(const DevState &s, const int k, Ctl *ctl,
                                               const double hourg, double *sm)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    double *const cs = s.corner + k;
    fx::i64 *const n = reinterpret_cast<fx::i64 *>(sm);
    double *const w = sm + 24 * BS;

    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    unsigned bad = 0;
    int emax[3];
    {
        double x[3][8];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double *const p = c == 0 ? s.x : c == 1 ? s.y : s.z;
#pragma unroll
            for (int j = 0; j < 8; ++j) x[c][j] = field(&p[nd[j]]);
            emax[c] = fx::align8<BS>(x[c], n + 8 * c * BS, bad);
        }
        // lulesh.cc:1082-1091 uses the Jacobian determinant only for its
        // sign: an FP32 filter with a rigorous error bound settles it, and
        // the FP64 form evaluates it only for an element the filter cannot
        // settle (none on a valid mesh)
        if (!jacobian_certainly_positive(x[0], x[1], x[2])) bad = 1;
    }
    // InitStressTermsForElems (273-286) + IntegrateStressForElems (494-587)
    fx::face_areas<BS>(n, emax, 0, 6, w);
    {
        // the areas are 16 x (exact); -(sig pf) = (-sig) pf
        const fx::Factor sig = fx::factor((s.p[k] + s.q[k]) * 0.0625, bad);
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
            const unsigned code = fx::corner_faces(j);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double pf = zero_plus(w[((code & 7) * 3 + c) * BS]) +
                                  w[((code >> 3 & 7) * 3 + c) * BS] +
                                  w[((code >> 6) * 3 + c) * BS];
                cs[c * E8 + (size_t)j * E] = fx::product(fx::factor(pf, bad), sig);
            }
        }
    }
    // CalcHourglassControlForElems (995-1057)
    const double vk = s.v[k];
    if (dle(vk, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1034-1040
    if (!(hourg > 0.)) {
        if (bad) forces_general(s, k, ctl, hourg);
        return;
    }
    // CalcFBHourglassForceForElems (710-991), CalcElemFBHourglassForce (667-706)
#pragma unroll 1
    for (int c = 0; c < 3; ++c) fx::volume_derivatives<BS>(n, emax, c, w, bad);
    const double determ = s.volo[k] * vk;
    // the four modes' sums of each coordinate
    fx::Factor hm[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < 4; ++m)
            hm[c][m] = fx::factor_of(
                fx::hourglass_mode<BS>(n + 8 * c * BS, fx::mode_signs(m)), emax[c]);
    // hourgam[j][m] over the coordinates and the volume derivatives, which end here:
    // modes 0 to 2 at w[8 m + j], mode 3 at n[j]
    const fx::Factor volinv = fx::factor(rcp_op(determ), bad);
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        const fx::Factor dx = fx::factor(w[(0 + j) * BS], bad);
        const fx::Factor dy = fx::factor(w[(8 + j) * BS], bad);
        const fx::Factor dz = fx::factor(w[(16 + j) * BS], bad);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double sum = fx::product(dx, hm[0][m]) +
                               fx::product(dy, hm[1][m]) +
                               fx::product(dz, hm[2][m]);
            (m < 3 ? w + (8 * m + j) * BS : sm + j * BS)[0] =
                signed_by(1.0, fx::mode_signs(m) >> j) - fx::product(fx::factor(sum, bad), volinv);
        }
    }
    const double coefficient =
        div_op(-hourg * 0.01 * s.ss[k] * s.elemMass[k], cbrt(determ));
    const fx::Factor coef = fx::factor(coefficient, bad);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const double *const vel = c == 0 ? s.xd : c == 1 ? s.yd : s.zd;
        fx::Factor u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = fx::factor(field(&vel[nd[j]]), bad);
        double f[8];
#pragma unroll 1
        for (int m = 0; m < 4; ++m) {
            const double *const gm = m < 3 ? w + 8 * m * BS : sm;
            fx::Factor g[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = fx::factor(gm[j * BS], bad);
            double sum = fx::product(g[0], u[0]);
#pragma unroll
            for (int j = 1; j < 8; ++j) sum += fx::product(g[j], u[j]);
            const fx::Factor hx = fx::factor(sum, bad);
            double add[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) add[j] = fx::product(g[j], hx);
            int first = m;
            asm("" : "+r"(first));  // the compiler is not to peel the first mode off
            if (first == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = add[j];
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] += add[j];
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            cs[(3 + c) * E8 + (size_t)j * E] = fx::product(fx::factor(f[j], bad), coef);
    }
    if (bad) forces_general(s, k, ctl, hourg);
}
#endif

#if LG_REASSOC
// Blocks of 128 (meshes that fill the SMs): 512 resident threads per SM, 128
// registers, 6 % faster at s=150.  Smaller blocks (small meshes): 384, 168
// registers without spills, 10 to 18 % faster at s=30 and s=45, where no more
// threads are there to run.
#define LG_FORCES_MIN_BLOCKS(BS) ((BS) == 128 ? 4 : (BS) < 128 ? 384 / (BS) : 1)
#else
// 384 resident threads per SM, 168 registers: 4,662 us at s=150 (512: 4,901; 256 was
// 10 % slower than 384 in an earlier form)
#define LG_FORCES_MIN_BLOCKS(BS) (384 / (BS))
#endif
template <bool BATCHED, int BS>
__global__ void __launch_bounds__(BS, LG_FORCES_MIN_BLOCKS(BS)) k_forces(DevState s)
{
    follow_on();
#if LG_REASSOC
    extern __shared__ fx::i64 force_scratch[];
    fx::i64 *const sm = force_scratch + threadIdx.x;
#else
    extern __shared__ double force_scratch[];
    double *const sm = force_scratch + threadIdx.x;
#endif
    if (!BATCHED && !cycle_live(s.ctl)) return;
    for (int k = blockIdx.x * BS + threadIdx.x; k < s.E; k += gridDim.x * BS) {
        const int pid = BATCHED ? s.elemProb[k] : 0;
        Ctl *ctl = s.ctl + pid;
        if (BATCHED && !cycle_live(ctl)) continue;
        const double hourg = s.hgcoefs[pid];
        forces_element<BS>(s, k, ctl, hourg, sm);
    }
}

// f / m, rounded as the IEEE quotient, from rm = RN(1 / m) (the set-up's
// invMass, constant over the run) by Markstein's residual correction
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990): q0 = RN(f rm), the exact
// residual f - m q0 by one FMA, q = RN(q0 + residual rm).  Three FP64
// instructions instead of a division; equal to f / m for operands in the
// normal range whose residual does not underflow.  An exact q0 (zero
// residual) is returned as is, which keeps the sign of a zero quotient.
__device__ __forceinline__ double div_by_mass(double f, double m, double rm)
{
    const double q0 = __dmul_rn(f, rm);
    const double res = __fma_rn(-m, q0, f);
    return dnz(res) ? __fma_rn(res, rm, q0) : q0;
}

// ---------------------------------------------------------------------------
// k_nodes: corner gather (lulesh.cc:565-582, 969-986), CalcAccelerationForNodes
// (1139-1149), ApplyAccelerationBoundaryConditionsForNodes (1153-1179),
// CalcVelocityForNodes (1183-1205), CalcPositionForNodes (1209-1219)
// ---------------------------------------------------------------------------
#if LG_REASSOC
// Out of line: nodes of more than eight corners, or whose forces overflow
__device__ __noinline__ double3 corner_sums_general(const DevState &s, int b, int e)
{
    const size_t E = (size_t)s.E;
    double3 f = make_double3(0., 0., 0.);
    for (int i = b; i < e; ++i) {
        const int c = s.nodeElemCornerList[i];
        const double *p = s.corner + (size_t)(c & 7) * E + (c >> 3);
        f.x += p[0];
        f.y += p[8 * E];
        f.z += p[16 * E];
    }
    return f;
}
#endif

__device__ __forceinline__ void nodes_node(const DevState &s, const int n, const Ctl *ctl,
                                           const bool hg)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    const double *cs = s.corner;
    const int b = s.nodeElemStart[n], e = s.nodeElemStart[n + 1];
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
#if LG_REASSOC
    // The corner sums on the integer pipe: 24 additions were half of the
    // kernel's FP64 instructions, which bound it.
    bool ok = e - b <= 8;
    {
        double f[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            f[0][i] = f[1][i] = f[2][i] = 0.0;
            if (i < e - b) {
                const int c = s.nodeElemCornerList[b + i];
                const size_t idx = (size_t)(c & 7) * E + (c >> 3);
                f[0][i] = cs[0 * E8 + idx];
                f[1][i] = cs[1 * E8 + idx];
                f[2][i] = cs[2 * E8 + idx];
            }
        }
        ok = fx::sum_of(f[0], Fx) && ok;
        ok = fx::sum_of(f[1], Fy) && ok;
        ok = fx::sum_of(f[2], Fz) && ok;
    }
    if (!ok) {
        const double3 F = corner_sums_general(s, b, e);
        Fx = F.x;
        Fy = F.y;
        Fz = F.z;
    }
#else
    double hx = 0.0, hy = 0.0, hz = 0.0;
    if (b < e) {  // the first corner onto the sums' 0.0
        const int c = s.nodeElemCornerList[b];
        const size_t idx = (size_t)(c & 7) * E + (c >> 3);
        Fx = zero_plus(cs[0 * E8 + idx]);
        Fy = zero_plus(cs[1 * E8 + idx]);
        Fz = zero_plus(cs[2 * E8 + idx]);
        if (hg) {
            hx = zero_plus(cs[3 * E8 + idx]);
            hy = zero_plus(cs[4 * E8 + idx]);
            hz = zero_plus(cs[5 * E8 + idx]);
        }
    }
    for (int i = b + 1; i < e; ++i) {
        const int c = s.nodeElemCornerList[i];
        const size_t idx = (size_t)(c & 7) * E + (c >> 3);
        Fx += cs[0 * E8 + idx];
        Fy += cs[1 * E8 + idx];
        Fz += cs[2 * E8 + idx];
        if (hg) {
            hx += cs[3 * E8 + idx];
            hy += cs[4 * E8 + idx];
            hz += cs[5 * E8 + idx];
        }
    }
    if (hg) {
        Fx += hx;
        Fy += hy;
        Fz += hz;
    }
#endif
    s.fx[n] = Fx;
    s.fy[n] = Fy;
    s.fz[n] = Fz;
    const double m = s.nodalMass[n], rm = s.invMass[n];
    double xdd = div_by_mass(Fx, m, rm), ydd = div_by_mass(Fy, m, rm),
           zdd = div_by_mass(Fz, m, rm);
    const int sym = s.symm[n];
    if (sym & 1) xdd = 0.0;
    if (sym & 2) ydd = 0.0;
    if (sym & 4) zdd = 0.0;
    s.xdd[n] = xdd;
    s.ydd[n] = ydd;
    s.zdd[n] = zdd;
    const double dt = ctl->deltatime;
    const double u_cut = s.prm.u_cut;
    double xd = s.xd[n] + xdd * dt;
    if (dabs_lt(xd, u_cut)) xd = 0.0;
    double yd = s.yd[n] + ydd * dt;
    if (dabs_lt(yd, u_cut)) yd = 0.0;
    double zd = s.zd[n] + zdd * dt;
    if (dabs_lt(zd, u_cut)) zd = 0.0;
    s.xd[n] = xd;
    s.yd[n] = yd;
    s.zd[n] = zd;
    s.x[n] += xd * dt;
    s.y[n] += yd * dt;
    s.z[n] += zd * dt;
}

template <bool BATCHED, int BS>
__global__ void __launch_bounds__(BS) k_nodes(DevState s)
{
    follow_on();
    if (!BATCHED && !cycle_live(s.ctl)) return;
    for (int n = blockIdx.x * BS + threadIdx.x; n < s.N; n += gridDim.x * BS) {
        const int pid = BATCHED ? s.nodeProb[n] : 0;
        const Ctl *ctl = s.ctl + pid;
        if (BATCHED && !cycle_live(ctl)) continue;
        nodes_node(s, n, ctl, s.hgcoefs[pid] > 0.);
    }
}

// ---------------------------------------------------------------------------
// k_kinematics: CalcKinematicsForElems (lulesh.cc:1504-1568), the strain loop
// of CalcLagrangeElements (1584-1606) and CalcMonotonicQGradientsForElems
// (1613-1757)
// ---------------------------------------------------------------------------
#if LG_REASSOC
// One element in FP64: those the fixed-point formats do not hold
__device__ __noinline__ void kinematics_general(const DevState &s, const int k, Ctl *ctl)
{
    const int E = s.E;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    double x[8], y[8], z[8], xv[8], yv[8], zv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = s.x[nd[j]];
        y[j] = s.y[nd[j]];
        z[j] = s.z[nd[j]];
        xv[j] = s.xd[nd[j]];
        yv[j] = s.yd[nd[j]];
        zv[j] = s.zd[nd[j]];
    }
    const double volo = s.volo[k];
    const double volume = elem_volume(x, y, z);
    const double relativeVolume = volume / volo;
    s.vnew[k] = relativeVolume;
    s.delv[k] = relativeVolume - s.v[k];
    s.arealg[k] = char_length<double, true>(x, y, z, volume);
    // The velocity gradient's trace and the monotonic-Q gradients from the
    // xi, eta, zeta differences of the coordinates (P) and velocities (V),
    // formed once from the element's body diagonals: the half-step Jacobian
    // is P - dt/2 V (velocity_trace_dirs).
    double P[9], V[9];
    {
        double Dx[4], Dy[4], Dz[4];
        body_diagonals(x, Dx);
        body_diagonals(y, Dy);
        body_diagonals(z, Dz);
        directions3(Dx, Dy, Dz, P);
        body_diagonals(xv, Dx);
        body_diagonals(yv, Dy);
        body_diagonals(zv, Dz);
        directions3(Dx, Dy, Dz, V);
    }
    s.vdov[k] = velocity_trace_dirs(P, V, 0.5 * ctl->deltatime);
    if (dle(relativeVolume, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1598-1605

    // CalcMonotonicQGradientsForElems
    double g[6];
    monoq_gradients_dirs(P, V, volo * relativeVolume, g);
    s.delx_xi[k] = g[0];
    s.delx_eta[k] = g[1];
    s.delx_zeta[k] = g[2];
    s.delv_xi[k] = g[3];
    s.delv_eta[k] = g[4];
    s.delv_zeta[k] = g[5];
}

// One element in fixed point (lg_fixed_geometry.cuh); sm is the thread's
// column of shared memory.  Integer and 56 FP64 instructions for each element in place
// of 328 FP64 ones, which bound it: 2,007 -> 512 us at s=150, 25 -> 14 us at s=30.  The
// rates' cofactors and products keep the digits of small velocity components and small
// tilts, which costs 16 % where everything moves (s=96: 163 us with one unit for the
// three components, 189 so); warps at rest skip the rates (s=150 early on: 596 us without).
template <int BS>
__device__ __forceinline__ void kinematics_element(const DevState &s, const int k, Ctl *ctl,
                                                   fx::i64 *sm)
{
    const int E = s.E;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    fx::Op P[3][3], V[3][3];
    int u[3], lambda[3];
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double *p = c == 0 ? s.x : c == 1 ? s.y : s.z;
        double a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = field(&p[nd[j]]);
        ok = fx::kin_component(a, c, sm, BS, P[c], u[c]) && ok;
    }
    {
        double v[3][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[0][j] = field(&s.xd[nd[j]]);
            v[1][j] = field(&s.yd[nd[j]]);
            v[2][j] = field(&s.zd[nd[j]]);
        }
        ok = fx::kin_velocities(v, u, V, lambda) && ok;
    }
    fx::Kinematics r;
    ok = fx::kinematics(sm, BS, P, u, V, lambda, 0.5 * ctl->deltatime, r) && ok;
    const double volo = s.volo[k];
    const double vnew = fx::quotient(r.volume, volo);
    ok = ok && fx::seedable(volo);
    s.vnew[k] = vnew;
    s.delv[k] = vnew - s.v[k];
    s.arealg[k] = r.arealg;
    s.vdov[k] = r.vdov;
    s.delx_xi[k] = r.delx[0];
    s.delx_eta[k] = r.delx[1];
    s.delx_zeta[k] = r.delx[2];
    s.delv_xi[k] = r.delv[0];
    s.delv_eta[k] = r.delv[1];
    s.delv_zeta[k] = r.delv[2];
    if (!ok) kinematics_general(s, k, ctl);
}
#else
// One element in FP64: the elements whose values the integer forms below do not hold
__device__ __noinline__ void kinematics_general(const DevState &s, const int k, Ctl *ctl)
{
    const int E = s.E;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    double x[8], y[8], z[8], xv[8], yv[8], zv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = s.x[nd[j]];
        y[j] = s.y[nd[j]];
        z[j] = s.z[nd[j]];
        xv[j] = s.xd[nd[j]];
        yv[j] = s.yd[nd[j]];
        zv[j] = s.zd[nd[j]];
    }
    const double volo = s.volo[k];
    const double volume = elem_volume(x, y, z);
    const double relativeVolume = div_op(volume, volo);
    s.vnew[k] = relativeVolume;
    s.delv[k] = relativeVolume - s.v[k];
    s.arealg[k] = char_length(x, y, z, volume);
    {
        const double dt2 = 0.5 * ctl->deltatime;
        double xh[8], yh[8], zh[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            xh[j] = x[j] - dt2 * xv[j];
            yh[j] = y[j] - dt2 * yv[j];
            zh[j] = z[j] - dt2 * zv[j];
        }
        // 64 x the determinant and 64 x B, whose factors cancel exactly in
        // inv_detJ * (B . v)
        double bx[4], by[4], bz[4];
        const double inv_detJ = rcp_op(shape_derivs_x64(xh, yh, zh, bx, by, bz));
        const double dxx = inv_detJ * (bx[0] * (xv[0] - xv[6]) + bx[1] * (xv[1] - xv[7]) +
                                       bx[2] * (xv[2] - xv[4]) + bx[3] * (xv[3] - xv[5]));
        const double dyy = inv_detJ * (by[0] * (yv[0] - yv[6]) + by[1] * (yv[1] - yv[7]) +
                                       by[2] * (yv[2] - yv[4]) + by[3] * (yv[3] - yv[5]));
        const double dzz = inv_detJ * (bz[0] * (zv[0] - zv[6]) + bz[1] * (zv[1] - zv[7]) +
                                       bz[2] * (zv[2] - zv[4]) + bz[3] * (zv[3] - zv[5]));
        s.vdov[k] = dxx + dyy + dzz;
    }
    if (dle(relativeVolume, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1598-1605

    // CalcMonotonicQGradientsForElems
    double g[6];
    monoq_gradients<double, true>(x, y, z, xv, yv, zv, volo * relativeVolume, g);
    s.delx_xi[k] = g[0];
    s.delx_eta[k] = g[1];
    s.delx_zeta[k] = g[2];
    s.delv_xi[k] = g[3];
    s.delv_eta[k] = g[4];
    s.delv_zeta[k] = g[5];
}

// One element; sm is the thread's column of shared memory (24 coordinates, then the
// half step's Jacobian and the gradients' differences of the coordinates and velocities,
// nine each; the cofactors go over the coordinates).  kinematics_general's values bit
// for bit with 212 products and 180 coordinate sums on the integer pipes
// (lg_exact_geometry.cuh) instead of the FP64 pipe, which bounded that form: 695 FP64
// instructions for each element became 321, 4,064 -> 2,585 us at s=150 and 43.4 -> 38.9 at
// s=30.
template <int BS>
__device__ __forceinline__ void kinematics_element(const DevState &s, const int k, Ctl *ctl,
                                                   double *sm)
{
    const int E = s.E;
    fx::i64 *const n = reinterpret_cast<fx::i64 *>(sm);
    double *const cof = sm, *const jac = sm + 24 * BS, *const grad = sm + 33 * BS,
                 *const vgrad = sm + 42 * BS;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    unsigned bad = 0;
    int emax[3];
    const fx::Factor dt2 = fx::factor(0.5 * ctl->deltatime, bad);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const double *const px = c == 0 ? s.x : c == 1 ? s.y : s.z;
        const double *const pv = c == 0 ? s.xd : c == 1 ? s.yd : s.zd;
        double x[8], v[8], h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = px[nd[j]];
            v[j] = pv[nd[j]];
            h[j] = x[j] - fx::product(fx::factor(v[j], bad), dt2);
        }
        const int ec = fx::align8<BS>(x, n + 8 * c * BS, bad);
        if (c == 0) emax[0] = ec;
        if (c == 1) emax[1] = ec;
        if (c == 2) emax[2] = ec;
        fx::gradient_sums<BS>(n + 8 * c * BS, ec, grad + 3 * c * BS);
        const double D0 = h[6] - h[0], D1 = h[5] - h[3], D2 = h[7] - h[1], D3 = h[4] - h[2];
        jac[(3 * c + 0) * BS] = D0 + D1 - D2 - D3;
        jac[(3 * c + 1) * BS] = D0 - D1 + D2 - D3;
        jac[(3 * c + 2) * BS] = D0 + D1 + D2 + D3;
#define LG_S4(a, b, c, d) (v[a] + v[b] + v[c] + v[d])
        vgrad[(3 * c + 0) * BS] = LG_S4(1, 2, 6, 5) - LG_S4(0, 3, 7, 4);
        vgrad[(3 * c + 1) * BS] = signed_by(LG_S4(0, 1, 5, 4) - LG_S4(3, 2, 6, 7), 1);
        vgrad[(3 * c + 2) * BS] = LG_S4(4, 5, 6, 7) - LG_S4(0, 1, 2, 3);
#undef LG_S4
    }
    const double volo = s.volo[k];
    double volume = 0.0;
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const double triple = fx::volume_triple<BS>(n, emax, i, bad);
        volume = i ? volume + triple : triple;
    }
    volume = fx::product(fx::factor(volume, bad), fx::factor(1.0 / 12.0, bad));
    const double relativeVolume = div_op(volume, volo);
    s.vnew[k] = relativeVolume;
    s.delv[k] = relativeVolume - s.v[k];
    s.arealg[k] = div_op(fx::times_pow2<2>(volume),
                         sqrt_op(fx::largest_area_face<BS>(n, emax, 0, 6, bad)));
    // 64 x the cofactors: cof[c][d] of the rows c + 1, c + 2 and columns d + 1, d + 2
    double det = 0.0;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const double *const j1 = jac + (c == 2 ? 0 : 3 * (c + 1)) * BS,
                            *const j2 = jac + (c == 0 ? 6 : 3 * (c - 1)) * BS;
        fx::Factor r1[3];
        fx::Factor r2[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            r1[d] = fx::factor(j1[d * BS], bad);
            r2[d] = fx::factor(j2[d * BS], bad);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
            const double v = fx::product(r1[d1], r2[d2]) - fx::product(r1[d2], r2[d1]);
            cof[(3 * c + d) * BS] = v;
            if (d == 1) {
                const double t = fx::product(fx::factor(v, bad),
                                             fx::factor(jac[(3 * c + 1) * BS], bad));
                det = c ? det + t : t;
            }
        }
    }
    const fx::Factor inv_detJ = fx::factor(rcp_op(det), bad);
    double vdov = 0.0;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const double *const pv = c == 0 ? s.xd : c == 1 ? s.yd : s.zd;
        const double ci = cof[(3 * c + 0) * BS], ce = cof[(3 * c + 1) * BS],
                     cz = cof[(3 * c + 2) * BS];
        const double ic = ci + ce, id = ci - ce;
        const fx::Factor b0 = fx::factor(-ic - cz, bad), b1 = fx::factor(id - cz, bad),
                         b2 = fx::factor(ic - cz, bad), b3 = fx::factor(-id - cz, bad);
        const double sum =
            fx::product(b0, fx::factor(pv[nd[0]] - pv[nd[6]], bad)) +
            fx::product(b1, fx::factor(pv[nd[1]] - pv[nd[7]], bad)) +
            fx::product(b2, fx::factor(pv[nd[2]] - pv[nd[4]], bad)) +
            fx::product(b3, fx::factor(pv[nd[3]] - pv[nd[5]], bad));
        const double rate = fx::product(fx::factor(sum, bad), inv_detJ);
        vdov = c ? vdov + rate : rate;
    }
    s.vdov[k] = vdov;

    // CalcMonotonicQGradientsForElems: direction d from the differences of the other two
    const double vol = fx::product(fx::factor(volo, bad), fx::factor(relativeVolume, bad));
    const fx::Factor norm =
        fx::factor(fx::times_pow2<-6>(rcp_op(vol + 1.e-36)), bad);
    const double vol16 = fx::times_pow2<4>(vol);
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        const int p = d == 2 ? 0 : d + 1, q = d == 0 ? 2 : d - 1;
        fx::Factor a[3];
        fx::Factor b[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a[c] = fx::factor(grad[(3 * c + p) * BS], bad);
            b[c] = fx::factor(grad[(3 * c + q) * BS], bad);
        }
        double size = 0.0, rate = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
            const fx::Factor x =
                fx::factor(fx::product(a[c1], b[c2]) - fx::product(a[c2], b[c1]), bad);
            const double xx = fx::product(x, x);
            const double xv = fx::product(fx::factor(fx::product(x, norm), bad),
                                          fx::factor(vgrad[(3 * c + d) * BS], bad));
            size = c ? size + xx : xx;
            rate = c ? rate + xv : xv;
        }
        double *const ox = d == 0 ? s.delx_xi : d == 1 ? s.delx_eta : s.delx_zeta;
        double *const ov = d == 0 ? s.delv_xi : d == 1 ? s.delv_eta : s.delv_zeta;
        ox[k] = div_op(vol16, sqrt_op(size + 256.e-36));
        ov[k] = rate;
    }
    if (bad)
        kinematics_general(s, k, ctl);
    else if (dle(relativeVolume, 0.0))
        raise_status(ctl, -1);  // lulesh.cc:1598-1605
}
#endif

#if LG_REASSOC
// 512 resident threads per SM: 616 -> 590 us at s=150 against 384, the same at
// s=30 and s=45; 640 656 us
#define LG_KIN_THREADS 512
#define LG_KIN_MIN_BLOCKS(BS) (LG_KIN_THREADS / (BS) > 0 ? LG_KIN_THREADS / (BS) : 1)
#else
// 512 resident threads per SM: 2,585 us at s=150 (384: 2,642)
#define LG_KIN_MIN_BLOCKS(BS) (512 / (BS))
#endif
template <bool BATCHED, int BS>
__global__ void __launch_bounds__(BS, LG_KIN_MIN_BLOCKS(BS)) k_kinematics(DevState s)
{
    follow_on();
#if LG_REASSOC
    extern __shared__ fx::i64 kin_scratch[];
    fx::i64 *const sm = kin_scratch + threadIdx.x;
#else
    extern __shared__ double kin_scratch[];
    double *const sm = kin_scratch + threadIdx.x;
#endif
    if (!BATCHED && !cycle_live(s.ctl)) return;
    for (int k = blockIdx.x * BS + threadIdx.x; k < s.E; k += gridDim.x * BS) {
        Ctl *ctl = s.ctl + (BATCHED ? s.elemProb[k] : 0);
        if (BATCHED && !cycle_live(ctl)) continue;
        kinematics_element<BS>(s, k, ctl, sm);
    }
}

#if LG_REASSOC
// monoq_phi with one product by the reciprocal of the element's own gradient:
// min(mult d-, mult d+, (d- + d+) / 2) of the unscaled neighbour gradients, their
// order turned round where the divisor is negative.  6 FP64 instructions for
// each direction instead of 12; the rounding differs from the reference's.
__device__ __forceinline__ double monoq_phi_fma(const Params &P, const double *dv, int ielem,
                                                int bc, int msymm, int mfree, int mmask, int psymm,
                                                int pfree, int pmask, int nbm, int nbp)
{
    const double self = dv[ielem], div = self + 1.e-36;
    if (!fx::seedable(fabs(div)))
        return monoq_phi(P.monoq_limiter_mult, P.monoq_max_slope, dv, ielem, bc, msymm, mfree,
                         mmask, psymm, pfree, pmask, nbm, nbp);
    const int bm = bc & mmask, bp = bc & pmask;
    double dm = 0., dp = 0.;
    if (bm == msymm)
        dm = self;
    else if (bm == 0 || bm == (mmask & ~(msymm | mfree)))
        dm = dv[nbm];
    if (bp == psymm)
        dp = self;
    else if (bp == 0 || bp == (pmask & ~(psymm | pfree)))
        dp = dv[nbp];
    const bool flip = __double2hiint(div) < 0;
    const double lo = P.monoq_limiter_mult * (dlt(dp, dm) != flip ? dp : dm);
    const double mid = 0.5 * (dm + dp);
    double phi = (dlt(lo, mid) != flip ? lo : mid) * fx::recip(div);
    if (dlt(phi, 0.)) phi = 0.;
    if (dlt(P.monoq_max_slope, phi)) phi = P.monoq_max_slope;
    return phi;
}
#endif

#if !LG_REASSOC
#include "lg_kernels_lanes.cuh"
#include "lg_kernels_team.cuh"
#endif

// One element of the material phase: its id and EOS repetitions (work item
// t of k_material, region order: regPerm[t], regRep[t]; every such item is
// its element's writer), its limiter results, clamped volumes and EOS
// inputs.  Every repetition computes the same values from the same inputs,
// so any repetition's results are the update; the split kernels for small
// meshes rely on that too.
struct MatItem {
    int ielem, reps;
    bool writer;
    double qlin, qquad, q_old, vnewc, vnew, e, delv, p;
};

// The element part of phase 1, reads only: monotonic-Q limiter, qstop check
// and the material clamps of element ielem.
__device__ __forceinline__ void material_inputs(const DevState &s, const int ielem, Ctl *ctl,
                                                MatItem &m)
{
    const Params &P = s.prm;
    // CalcMonotonicQRegionForElems, lulesh.cc:1761-1921
    const int bc = s.elemBC[ielem];
#if LG_REASSOC
#define LG_PHI(dv, ...) monoq_phi_fma(P, dv, __VA_ARGS__)
#else
#define LG_PHI(dv, ...) monoq_phi(P.monoq_limiter_mult, P.monoq_max_slope, dv, __VA_ARGS__)
#endif
    const double phixi = LG_PHI(s.delv_xi, ielem, bc, XI_M_SYMM, XI_M_FREE, XI_M, XI_P_SYMM,
                                XI_P_FREE, XI_P, s.lxim[ielem], s.lxip[ielem]);
    const double phieta = LG_PHI(s.delv_eta, ielem, bc, ETA_M_SYMM, ETA_M_FREE, ETA_M, ETA_P_SYMM,
                                 ETA_P_FREE, ETA_P, s.letam[ielem], s.letap[ielem]);
    const double phizeta = LG_PHI(s.delv_zeta, ielem, bc, ZETA_M_SYMM, ZETA_M_FREE, ZETA_M,
                                  ZETA_P_SYMM, ZETA_P_FREE, ZETA_P, s.lzetam[ielem],
                                  s.lzetap[ielem]);
#undef LG_PHI
    const double vnew = s.vnew[ielem];
    const double vdov = s.vdov[ielem];
    double qlin, qquad;
    if (dlt(0., vdov)) {
        qlin = 0.;
        qquad = 0.;
    } else {
        double delvxxi = s.delv_xi[ielem] * s.delx_xi[ielem];
        double delvxeta = s.delv_eta[ielem] * s.delx_eta[ielem];
        double delvxzeta = s.delv_zeta[ielem] * s.delx_zeta[ielem];
        if (dlt(0., delvxxi)) delvxxi = 0.;
        if (dlt(0., delvxeta)) delvxeta = 0.;
        if (dlt(0., delvxzeta)) delvxzeta = 0.;
        const double vol = s.volo[ielem] * vnew;
#if LG_REASSOC
        const double rho = fx::seedable(vol) ? fx::quotient(s.elemMass[ielem], vol)
                                             : s.elemMass[ielem] / vol;
#else
        const double rho = div_op(s.elemMass[ielem], vol);
#endif
        qlin = -P.qlc_monoq * rho *
               (delvxxi * (1. - phixi) + delvxeta * (1. - phieta) +
                delvxzeta * (1. - phizeta));
        qquad = P.qqc_monoq * rho *
                (delvxxi * delvxxi * (1. - phixi * phixi) +
                 delvxeta * delvxeta * (1. - phieta * phieta) +
                 delvxzeta * delvxzeta * (1. - phizeta * phizeta));
    }
    m.qlin = qlin;
    m.qquad = qquad;

    // qstop check on the previous cycle's q, lulesh.cc:1993-2008
    m.q_old = s.q[ielem];
    if (dlt(P.qstop, m.q_old)) ctl->err_qstop = 1;

    // ApplyMaterialPropertiesForElems, lulesh.cc:2328-2406
    double vnewc = vnew;
    if (dnz(P.eosvmin) && dlt(vnewc, P.eosvmin)) vnewc = P.eosvmin;
    if (dnz(P.eosvmax) && dlt(P.eosvmax, vnewc)) vnewc = P.eosvmax;
    double vc = s.v[ielem];
    if (dnz(P.eosvmin) && dlt(vc, P.eosvmin)) vc = P.eosvmin;
    if (dnz(P.eosvmax) && dlt(P.eosvmax, vc)) vc = P.eosvmax;
    if (dle(vc, 0.)) ctl->err_matvol = 1;
    m.vnewc = vnewc;
    m.vnew = vnew;
    m.e = s.e[ielem];
    m.delv = s.delv[ielem];
    m.p = s.p[ielem];
}

// Phase 1 of item t: its element, repetitions and role, and (MODE != 1) the
// element's inputs.  False for an item without an element.
template <int MODE>
__device__ __forceinline__ bool material_load(const DevState &s, const int t, Ctl *ctl,
                                              MatItem &m)
{
    const int ielem = s.regPerm[t];
    if (ielem < 0) return false;
    const int r = s.regRep[t];
    m.ielem = ielem;
    m.writer = r > 0;
    m.reps = r > 0 ? r : -r;
    if (MODE != 1) material_inputs(s, ielem, ctl, m);
    return true;
}

// The writer's part of phase 2: the element's update from the results o of
// its repetitions (MODE != 1) and its Courant/hydro candidates (MODE != 0).
template <int MODE>
__device__ __forceinline__ void material_finish(const DevState &s, const MatItem &m,
                                                const EosOut &o, double &dtc, double &dth)
{
    const Params &P = s.prm;
    const int ielem = m.ielem;
    if (MODE != 1) {
        s.qq[ielem] = m.qquad;
        s.ql[ielem] = m.qlin;
        s.p[ielem] = o.p;
        s.e[ielem] = o.e;
        s.q[ielem] = o.q;
        s.ss[ielem] = eos_sound_speed(P, o, m.vnewc);

        // UpdateVolumesForElems, lulesh.cc:2410-2427
        double tmpV = m.vnew;
        if (dabs_lt(tmpV - 1.0, P.v_cut)) tmpV = 1.0;
        s.v[ielem] = tmpV;
    }
    if (MODE != 0) {
        // CalcCourantConstraintForElems (2447-2513) and
        // CalcHydroConstraintForElems (2517-2572) for one element.  The
        // reference evaluates the Courant dt of every element but keeps it
        // only where vdov != 0; a warp of elements at rest skips it (the
        // barriers keep the compiler from hoisting that work above the vote).
        double vdov = s.vdov[ielem];
        const bool moving = dnz(vdov);
        if (__any_sync(__activemask(), moving) && moving) {
            const double qqc2 = 64.0 * P.qqc * P.qqc;
            double ssv = s.ss[ielem];
            double arealg = s.arealg[ielem];
            opaque(vdov); opaque(ssv); opaque(arealg);
            double dtf = ssv * ssv;
            if (dlt(vdov, 0.)) dtf = dtf + qqc2 * arealg * arealg * vdov * vdov;
            double rate = fabs(vdov) + 1.e-20;
#if LG_REASSOC
            dtf = fx::seedable(dtf) ? arealg * fx::recip_sqrt(dtf) : arealg / sqrt(dtf);
            const double dtdvov = fx::seedable(rate) ? fx::quotient(P.dvovmax, rate)
                                                     : P.dvovmax / rate;
#else
            dtf = div_op(arealg, sqrt_op(dtf));
            const double dtdvov = div_op(P.dvovmax, rate);
#endif
            if (dlt(dtf, dtc)) dtc = dtf;
            if (dlt(dtdvov, dth)) dth = dtdvov;
        }
    }
}

// Phase 2: the item's EOS repetitions (MODE != 1); the writer finishes the
// element.
template <int MODE>
__device__ __forceinline__ void material_update(const DevState &s, const MatItem &m,
                                                double &dtc, double &dth)
{
    EosOut o{};
    if (MODE != 1)
        o = eos_reps(s.prm, m.e, m.delv, m.p, m.q_old, m.qquad, m.qlin, m.vnewc, m.reps);
    if (m.writer) material_finish<MODE>(s, m, o, dtc, dth);
}

// The split material phase (DevState::matSplit, small meshes): three
// kernels instead of one, so that every FP64 instruction runs with full
// warps.  k_material_inputs (one thread per element, natural order): the
// monotonic-Q limiter, qstop check and clamps, staging the EOS inputs;
// k_material_eos (one thread per repetition item, equal shares per warp):
// the item's share of the EOS repetitions, the writer staging the results;
// k_material_finish (one thread per element): sound speed, stores, volume
// update, Courant/hydro candidates and the block reduction whose last block
// runs the next TimeIncrement.  The staging area is the per-corner scratch,
// which k_nodes has consumed and the next k_forces overwrites: eight inputs
// and five results per element, SoA.  Each element's arithmetic is that of
// the one-kernel path.
namespace matstage {
enum { E_OLD, DELV, P_OLD, Q_OLD, QQ, QL, VNEWC, VNEW, N_IN };
enum { P_NEW = N_IN, E_NEW, Q_NEW, BVC, PBVC, N_ALL };
}  // namespace matstage

template <int MODE, int BS>
__global__ void __launch_bounds__(BS) k_material_inputs(DevState s)
{
    follow_on();
    if (!cycle_live(s.ctl)) return;
    const int k = blockIdx.x * BS + threadIdx.x;
    if (k >= s.E) return;
    MatItem m;
    material_inputs(s, k, s.ctl, m);
    double *st = s.corner;
    const size_t E = (size_t)s.E;
    st[matstage::E_OLD * E + k] = m.e;
    st[matstage::DELV * E + k] = m.delv;
    st[matstage::P_OLD * E + k] = m.p;
    st[matstage::Q_OLD * E + k] = m.q_old;
    st[matstage::QQ * E + k] = m.qquad;
    st[matstage::QL * E + k] = m.qlin;
    st[matstage::VNEWC * E + k] = m.vnewc;
    st[matstage::VNEW * E + k] = m.vnew;
}

// M: the strict build's meshes with eight lanes for each element, which run less than
// a warp for each scheduler here and wait for the products' 22 instructions, keep
// FP64 products (IeeeOps): 52.5 us a cycle at s=10 against 53.3; s=30 143 against 148
template <int BS, class M = CycleOps>
__global__ void __launch_bounds__(BS, LG_EOS_MIN_BLOCKS(BS)) k_material_eos(DevState s)
{
    follow_on();
    if (!cycle_live(s.ctl)) return;
    const int t = blockIdx.x * BS + threadIdx.x;
    if (t >= s.nItems) return;
    const int k = s.regPerm[t], r = s.regRep[t];
    double *st = s.corner;
    const size_t E = (size_t)s.E;
    const EosOut o = eos_reps<M>(s.prm, st[matstage::E_OLD * E + k], st[matstage::DELV * E + k],
                                 st[matstage::P_OLD * E + k], st[matstage::Q_OLD * E + k],
                                 st[matstage::QQ * E + k], st[matstage::QL * E + k],
                                 st[matstage::VNEWC * E + k], r > 0 ? r : -r);
    if (r > 0) {
        st[matstage::P_NEW * E + k] = o.p;
        st[matstage::E_NEW * E + k] = o.e;
        st[matstage::Q_NEW * E + k] = o.q;
        st[matstage::BVC * E + k] = o.bvc;
        st[matstage::PBVC * E + k] = o.pbvc;
    }
}

template <int MODE, int BS>
__global__ void __launch_bounds__(BS) k_material_finish(DevState s)
{
    follow_on();
    if (!cycle_live(s.ctl)) return;
    double dtc = 1.0e+20, dth = 1.0e+20;
    const int k = blockIdx.x * BS + threadIdx.x;
    if (k < s.E) {
        MatItem m;
        m.ielem = k;
        m.writer = true;
        EosOut o{};
        if (MODE != 1) {
            const double *st = s.corner;
            const size_t E = (size_t)s.E;
            m.qquad = st[matstage::QQ * E + k];
            m.qlin = st[matstage::QL * E + k];
            m.vnewc = st[matstage::VNEWC * E + k];
            m.vnew = st[matstage::VNEW * E + k];
            o = {st[matstage::P_NEW * E + k], st[matstage::E_NEW * E + k],
                 st[matstage::Q_NEW * E + k], st[matstage::BVC * E + k],
                 st[matstage::PBVC * E + k]};
        }
        material_finish<MODE>(s, m, o, dtc, dth);
    }
    if (MODE != 0)
        finish_dt<BS, true>(s, dtc, dth, MODE == 2);
    else
        finish_material_flags(s);
}

template <int MODE, bool BATCHED, int BS>
__global__ void __launch_bounds__(BS, LG_MAT_MIN_BLOCKS(BS)) k_material(DevState s)
{
    follow_on();
    if (!BATCHED && !cycle_live(s.ctl)) return;
    double dtc = 1.0e+20, dth = 1.0e+20;
    if (!BATCHED) {
        // one item per element (nItems == E); small meshes run the split
        // kernels above
        const int t = blockIdx.x * BS + threadIdx.x;
        MatItem m;
        if (t < s.nItems && material_load<MODE>(s, t, s.ctl, m))
            material_update<MODE>(s, m, dtc, dth);
        if (MODE != 0)
            finish_dt<BS, true>(s, dtc, dth, MODE == 2);
        else
            finish_material_flags(s);
        return;
    }
    for (int t0 = blockIdx.x * BS; t0 < s.E; t0 += gridDim.x * BS) {
        const int t = t0 + threadIdx.x;
        int pid = -1;
        dtc = 1.0e+20;
        dth = 1.0e+20;
        if (t < s.E) {
            pid = s.elemProb[s.regPerm[t]];
            Ctl *ctl = s.ctl + pid;
            MatItem m;
            if (cycle_live(ctl) && material_load<2>(s, t, ctl, m))
                material_update<2>(s, m, dtc, dth);
        }
        batched_dt_candidates(s, pid, dtc, dth);
    }
    finish_batched(s);
}

}  // namespace LG_NS
}  // namespace lg
