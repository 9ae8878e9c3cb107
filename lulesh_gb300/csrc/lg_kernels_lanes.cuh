// lg_kernels_lanes.cuh -- the strict build's element kernels with eight lanes for each
// element, one for each corner, for meshes too small to fill the SMs.
//
// An SM's four schedulers each issue one FP64 warp instruction per 64 clocks, so a
// warp of 32 elements takes 64 x 1,272 clocks (39 us) for the corner forces
// however few warps there are: at s=10, 32 warps on 608 schedulers.  Here four elements
// share a warp.  The lanes divide the faces, corners, modes and directions of
// their element and exchange results through shared memory: about 240 FP64
// instructions deep instead of 1,272 (forces), 155 instead of 600 (kinematics).
// Every value is formed by the same operations in the same order as in k_forces and
// k_kinematics, so the results are the same bits.  Included inside namespace lg::LG_NS.
#pragma once

// tables indexed by lane
__constant__ signed char kFaces[8][4] = {{0, 1, 2, 3}, {0, 4, 5, 1}, {1, 5, 6, 2}, {2, 6, 7, 3},
                                         {3, 7, 4, 0}, {4, 7, 6, 5}, {0, 1, 2, 3}, {0, 1, 2, 3}};
// the three faces of each corner, in the order their areas are added
__constant__ signed char kCornerFaces[8][3] = {{0, 1, 4}, {0, 1, 2}, {0, 2, 3}, {0, 3, 4},
                                               {1, 4, 5}, {1, 2, 5}, {2, 3, 5}, {3, 4, 5}};
// CalcElemVolumeDerivative's neighbours (volume_derivative)
__constant__ signed char kVolu[8][6] = {{1, 2, 3, 4, 5, 7}, {2, 3, 0, 5, 6, 4}, {3, 0, 1, 6, 7, 5},
                                        {0, 1, 2, 7, 4, 6}, {7, 6, 5, 0, 3, 1}, {4, 7, 6, 1, 0, 2},
                                        {5, 4, 7, 2, 1, 3}, {6, 5, 4, 3, 2, 0}};
// CalcElemCharacteristicLength's faces (char_length)
__constant__ signed char kLengthFaces[8][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 1, 5, 4},
                                               {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 0, 4, 7},
                                               {0, 1, 2, 3}, {0, 1, 2, 3}};
// CalcElemVolume's three triple products a . (b x c): a = r0 - r1 + (r2 - r3),
// b = r4 - r5, c = r6 - r7
__constant__ signed char kTriple[3][8] = {{3, 1, 7, 2, 6, 3, 2, 0}, {4, 3, 5, 7, 6, 4, 7, 0},
                                          {1, 4, 2, 5, 6, 1, 5, 0}};
// CalcMonotonicQGradientsForElems' node sums: direction i = (first four) - (last
// four); j is negated
__constant__ signed char kGrad[3][8] = {{1, 2, 6, 5, 0, 3, 7, 4}, {0, 1, 5, 4, 3, 2, 6, 7},
                                        {4, 5, 6, 7, 0, 1, 2, 3}};

// v with its sign turned when flip (exact, off the FP64 pipe)
__device__ __forceinline__ double signed_of(double v, bool flip)
{
    return __longlong_as_double(__double_as_longlong(v) ^
                                (flip ? (long long)0x8000000000000000ULL : 0LL));
}

struct LaneForces {
    double x[3][8], u[3][8], area[3][8], mode[3][4], hg[4][8], hx[12];
};

template <int BS>
__global__ void __launch_bounds__(BS) k_forces_lanes(DevState s)
{
    follow_on();
    if (!cycle_live(s.ctl)) return;
    __shared__ LaneForces sm[BS / 8];
    LaneForces &m = sm[threadIdx.x >> 3];
    const int j = threadIdx.x & 7, E = s.E;
    const size_t E8 = 8 * (size_t)E;
    const int k0 = (blockIdx.x * BS + threadIdx.x) >> 3;
    const bool live = k0 < E;  // the lanes past the last element repeat it
    const int k = live ? k0 : E - 1;
    Ctl *ctl = s.ctl;
    const double hourg = s.hgcoefs[0];
    double *const cs = s.corner;

    const int nd = __ldg(&s.nodelistT[(size_t)j * E + k]);
    m.x[0][j] = s.x[nd];
    m.x[1][j] = s.y[nd];
    m.x[2][j] = s.z[nd];
    m.u[0][j] = s.xd[nd];
    m.u[1][j] = s.yd[nd];
    m.u[2][j] = s.zd[nd];
    const double sig = (-s.p[k] - s.q[k]) * 0.0625;  // the areas are 16 x
    const double vk = s.v[k];
    const double determ = s.volo[k] * vk;
    __syncwarp();

    // one face for each lane, then the corner's three
    {
        double ax, ay, az;
        face_area_x16(m.x[0], m.x[1], m.x[2], kFaces[j][0], kFaces[j][1], kFaces[j][2],
                      kFaces[j][3], ax, ay, az);
        m.area[0][j] = ax;
        m.area[1][j] = ay;
        m.area[2][j] = az;
    }
    // one mode for each lane: x and y (lanes 0..3), z (lanes 4..7)
    {
        const int i1 = j & 3;
        const double *a = j < 4 ? m.x[0] : m.x[2];
        double p = signed_of(a[0], gam(i1, 0) < 0.), q = signed_of(m.x[1][0], gam(i1, 0) < 0.);
#pragma unroll
        for (int n = 1; n < 8; ++n) {
            p = p + signed_of(a[n], gam(i1, n) < 0.);
            q = q + signed_of(m.x[1][n], gam(i1, n) < 0.);
        }
        m.mode[j < 4 ? 0 : 2][i1] = p;
        if (j < 4) m.mode[1][i1] = q;
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double pf = zero_plus(m.area[c][kCornerFaces[j][0]]) +
                          m.area[c][kCornerFaces[j][1]] + m.area[c][kCornerFaces[j][2]];
        if (live) cs[c * E8 + (size_t)j * E + k] = -(sig * pf);
    }
    {
        const bool sure = jacobian_certainly_positive(m.x[0], m.x[1], m.x[2]);
        if (!sure && live && j == 0 && jacobian_det(m.x[0], m.x[1], m.x[2]) <= 0.0)
            raise_status(ctl, -1);
    }
    if (live && j == 0 && dle(vk, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1034-1040
    if (!(hourg > 0.)) return;

    double dvdx, dvdy, dvdz;
    {
        double x[6], y[6], z[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            x[i] = m.x[0][kVolu[j][i]];
            y[i] = m.x[1][kVolu[j][i]];
            z[i] = m.x[2][kVolu[j][i]];
        }
        volu_der(x, y, z, 0, 1, 2, 3, 4, 5, dvdx, dvdy, dvdz);
    }
    const double volinv = rcp_op(determ);
    double h[4];
#pragma unroll
    for (int i1 = 0; i1 < 4; ++i1) {
        h[i1] = signed_of(1.0, gam(i1, j) < 0.) -
                volinv * (dvdx * m.mode[0][i1] + dvdy * m.mode[1][i1] + dvdz * m.mode[2][i1]);
        m.hg[i1][j] = h[i1];
    }
    const double volume13 = cbrt(determ);
    const double coefficient = div_op(-hourg * 0.01 * s.ss[k] * s.elemMass[k], volume13);
    __syncwarp();
    // the twelve mode amplitudes: lane l takes l and, where there is one, l + 8
    for (int t = j; t < 12; t += 8) {
        const double *g = m.hg[t & 3], *u = m.u[t >> 2];
        m.hx[t] = g[0] * u[0] + g[1] * u[1] + g[2] * u[2] + g[3] * u[3] + g[4] * u[4] +
                  g[5] * u[5] + g[6] * u[6] + g[7] * u[7];
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double *x = m.hx + 4 * c;
        const double f = coefficient * (h[0] * x[0] + h[1] * x[1] + h[2] * x[2] + h[3] * x[3]);
        if (live) cs[(3 + c) * E8 + (size_t)j * E + k] = f;
    }
}

struct LaneKinematics {
    double x[3][8], u[3][8], h[3][8], area[8], triple[4], jac[3][3], cof[3][3], rate[4],
        grad[6][3];
};

template <int BS>
__global__ void __launch_bounds__(BS) k_kinematics_lanes(DevState s)
{
    follow_on();
    if (!cycle_live(s.ctl)) return;
    __shared__ LaneKinematics sm[BS / 8];
    LaneKinematics &m = sm[threadIdx.x >> 3];
    const int j = threadIdx.x & 7, E = s.E;
    const int k0 = (blockIdx.x * BS + threadIdx.x) >> 3;
    const bool live = k0 < E;
    const int k = live ? k0 : E - 1;
    Ctl *ctl = s.ctl;
    const int nd = __ldg(&s.nodelistT[(size_t)j * E + k]);
    const double dt2 = 0.5 * ctl->deltatime;
    {
        const double *const px[3] = {s.x, s.y, s.z}, *const pu[3] = {s.xd, s.yd, s.zd};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double x = px[c][nd], u = pu[c][nd];
            m.x[c][j] = x;
            m.u[c][j] = u;
            m.h[c][j] = x - dt2 * u;
        }
    }
    const double volo = s.volo[k];
    __syncwarp();

    // CalcElemVolume: a triple product for each of three lanes
    {
        const signed char *T = kTriple[j < 3 ? j : 0];
        double a[3], b[3], c[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double *r = m.x[d];
            a[d] = (r[T[0]] - r[T[1]]) + (r[T[2]] - r[T[3]]);
            b[d] = r[T[4]] - r[T[5]];
            c[d] = r[T[6]] - r[T[7]];
        }
        const double t = a[0] * (b[1] * c[2] - c[1] * b[2]) + a[1] * (c[0] * b[2] - b[0] * c[2]) +
                         a[2] * (b[0] * c[1] - c[0] * b[1]);
        if (j < 3) m.triple[j] = t;
    }
    m.area[j] = area_face(m.x[0], m.x[1], m.x[2], kLengthFaces[j][0], kLengthFaces[j][1],
                          kLengthFaces[j][2], kLengthFaces[j][3]);
    // 8 x the half-step Jacobian: nine sums, lane 0 takes the last as well
    for (int t = j; t < 9; t += 8) {
        const int d = t % 3;
        const double *r = m.h[t / 3];
        const double D1 = r[5] - r[3], D2 = r[7] - r[1], D3 = r[4] - r[2];
        // xi: + - -, eta: - + -, zeta: + + +
        m.jac[t / 3][d] = (r[6] - r[0]) + signed_of(D1, d == 1) + signed_of(D2, d == 0) +
                          signed_of(D3, d < 2);
    }
    // the Q gradients' differences of the coordinates and velocities
    for (int t = j; t < 18; t += 8) {
        const int d = t % 3;
        const double *r = t < 9 ? m.x[t / 3] : m.u[t / 3 - 3];
        const signed char *T = kGrad[d];
        const double g = (r[T[0]] + r[T[1]] + r[T[2]] + r[T[3]]) -
                         (r[T[4]] + r[T[5]] + r[T[6]] + r[T[7]]);
        m.grad[t / 3][d] = signed_of(g, d == 1);
    }
    __syncwarp();
    double volume = m.triple[0] + m.triple[1] + m.triple[2];
    volume *= 1.0 / 12.0;
    const double relativeVolume = div_op(volume, volo);
    double cl = 0.0;
#pragma unroll
    for (int f = 0; f < 6; ++f) cl = lt(m.area[f], cl) ? cl : m.area[f];
    // 64 x the cofactors: cof[c][d] of the rows c + 1, c + 2 and columns d + 1, d + 2
    for (int t = j; t < 9; t += 8) {
        const int c1 = (t / 3 + 1) % 3, c2 = (t / 3 + 2) % 3, d1 = (t % 3 + 1) % 3,
                  d2 = (t % 3 + 2) % 3;
        m.cof[t / 3][t % 3] = m.jac[c1][d1] * m.jac[c2][d2] - m.jac[c2][d1] * m.jac[c1][d2];
    }
    __syncwarp();
    {
        // a row of B against the velocity differences for each of three lanes
        const int c = j < 3 ? j : 0;
        const double ci = m.cof[c][0], ce = m.cof[c][1], cz = m.cof[c][2];
        const double b0 = -ci - ce - cz, b1 = ci - ce - cz, b2 = ci + ce - cz, b3 = -ci + ce - cz;
        const double det = m.jac[0][1] * m.cof[0][1] + m.jac[1][1] * m.cof[1][1] +
                           m.jac[2][1] * m.cof[2][1];
        const double inv_detJ = rcp_op(det);
        const double *u = m.u[c];
        const double d = inv_detJ * (b0 * (u[0] - u[6]) + b1 * (u[1] - u[7]) + b2 * (u[2] - u[4]) +
                                     b3 * (u[3] - u[5]));
        if (j < 3) m.rate[j] = d;
    }
    // a direction of the Q gradients for each of three lanes
    double delx, delv;
    {
        const double vol = volo * relativeVolume;
        const double norm = rcp_op(vol + 1.e-36) * 0.015625;
        const int d = j < 3 ? j : 0, p = (d + 1) % 3, q = (d + 2) % 3;
        const double px = m.grad[0][p], py = m.grad[1][p], pz = m.grad[2][p];
        const double qx = m.grad[0][q], qy = m.grad[1][q], qz = m.grad[2][q];
        double ax = py * qz - pz * qy, ay = pz * qx - px * qz, az = px * qy - py * qx;
        delx = div_op(16.0 * vol, sqrt_op(ax * ax + ay * ay + az * az + 256.e-36));
        ax *= norm;
        ay *= norm;
        az *= norm;
        delv = ax * m.grad[3][d] + ay * m.grad[4][d] + az * m.grad[5][d];
    }
    __syncwarp();
    if (!live) return;
    if (j == 0) {
        s.vnew[k] = relativeVolume;
        s.delv[k] = relativeVolume - s.v[k];
        s.arealg[k] = div_op(4.0 * volume, sqrt_op(cl));
        s.vdov[k] = m.rate[0] + m.rate[1] + m.rate[2];
        if (dle(relativeVolume, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1598-1605
    }
    if (j < 3) {
        double *const ox = j == 0 ? s.delx_xi : j == 1 ? s.delx_eta : s.delx_zeta;
        double *const ov = j == 0 ? s.delv_xi : j == 1 ? s.delv_eta : s.delv_zeta;
        ox[k] = delx;
        ov[k] = delv;
    }
}
