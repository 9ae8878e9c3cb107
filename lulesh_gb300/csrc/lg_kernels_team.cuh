// lg_kernels_team.cuh -- the strict build's corner forces and kinematics with three warps
// for 32 elements, warp c with their component c.
//
// On meshes of up to about two warps of elements for each scheduler the one-thread form
// (forces_element: 28,400 instructions in one chain) waits for its own results:
// s=30 68 us whether a scheduler has one warp or two.  Here every warp has a third of the
// faces, derivatives, corners and directions, and the three exchange the rest through
// shared memory: k_forces 68 -> 59 us, k_kinematics 39 -> 35 and a cycle 138 -> 125 at
// s=30; s=21 104 -> 74 (there against the FP64 form).  The same operations in the same
// order, so the same bits.  Larger meshes fill the schedulers without it and would pay
// for the work that all three repeat and for the barriers: s=31 143 us a cycle with one
// thread, 149 so; s=150, with a dearer product, 4,871 and 2,746 us against 6,500 and
// 2,970.  Included inside namespace lg::LG_NS.
#pragma once

constexpr int kTeam = 3;       // threads for an element, one for each component
constexpr int kTeamElems = 32;  // elements of a block, one for each lane of a warp
struct ForceSlots {  // words of an element's column
    enum { N = 0, W = 24, H = 48, COUNT = 60 };
};
struct KinSlots {
    enum { N = 0, JAC = 24, GRAD = 33, VGRAD = 42, COF = 51, COUNT = 60 };
};
// bytes of a block's shared memory: the elements' columns, a word of them kTeamElems
// apart, then three exponents and three flags for each element
constexpr int kTeamSmem = kTeamElems * (60 * 8 + 6 * 4);

// One element's component c by one thread, with two others of the same block; hourg is
// the element's problem's hourglass coefficient, sm the element's column (coordinates;
// areas, volume derivatives and hourglass shapes in turn; mode sums).  live: the
// element is there and its cycle runs (every thread takes the barriers).
template <int BS>
__device__ __forceinline__ void forces_team(const DevState &s, const int k, const bool live,
                                            Ctl *ctl, const double hourg, double *sm, int *em,
                                            const int c)
{
    const int E = s.E;
    const size_t E8 = 8 * (size_t)E;
    double *const cs = s.corner + k;
    fx::i64 *const n = reinterpret_cast<fx::i64 *>(sm);
    double *const w = sm + ForceSlots::W * BS, *const h = sm + ForceSlots::H * BS;

    int nd[8];
    unsigned bad = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    {
        const double *const p = c == 0 ? s.x : c == 1 ? s.y : s.z;
        double a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = field(&p[nd[j]]);
        em[c * BS] = fx::align8<BS>(a, n + 8 * c * BS, bad);
        if (c == 2) {
            // lulesh.cc:1082-1091 uses the Jacobian determinant only for its
            // sign: an FP32 filter with a rigorous error bound settles it, and
            // the FP64 form evaluates it only for an element the filter cannot
            // settle (none on a valid mesh)
            double x[8], y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                x[j] = field(&s.x[nd[j]]);
                y[j] = field(&s.y[nd[j]]);
            }
            if (!jacobian_certainly_positive(x, y, a)) bad = 1;
        }
    }
    __syncthreads();
    const int emax[3] = {em[0], em[BS], em[2 * BS]};
    // InitStressTermsForElems (273-286) + IntegrateStressForElems (494-587)
    fx::face_areas<BS>(n, emax, 2 * c, 2, w);
    __syncthreads();
    {
        // the areas are 16 x (exact); -(sig pf) = (-sig) pf
        const fx::Factor sig = fx::factor((s.p[k] + s.q[k]) * 0.0625, bad);
#pragma unroll 2
        for (int j = 0; j < 8; ++j) {
            const unsigned code = fx::corner_faces(j);
            const double pf = zero_plus(w[((code & 7) * 3 + c) * BS]) +
                              w[((code >> 3 & 7) * 3 + c) * BS] + w[((code >> 6) * 3 + c) * BS];
            const double f = fx::product(fx::factor(pf, bad), sig);
            if (live) cs[c * E8 + (size_t)j * E] = f;
        }
    }
    // CalcHourglassControlForElems (995-1057)
    const double vk = s.v[k];
    if (live && c == 0 && dle(vk, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1034-1040
    const bool hg = hourg > 0.;
    // CalcFBHourglassForceForElems (710-991), CalcElemFBHourglassForce (667-706)
    int *const flags = em + kTeam * BS;
    if (!__syncthreads_or(hg)) {
        flags[c * BS] = (int)bad;
        __syncthreads();
        if (c == 0 && live && (flags[0] | flags[BS] | flags[2 * BS]))
            forces_general(s, k, ctl, hourg);
        return;
    }
    fx::volume_derivatives<BS>(n, emax, c, w, bad);
#pragma unroll
    for (int m = 0; m < 4; ++m)
        h[(4 * c + m) * BS] =
            fx::double_of(fx::hourglass_mode<BS>(n + 8 * c * BS, fx::mode_signs(m)), em[c * BS]);
    __syncthreads();
    // hourgam[j][m] over the coordinates and the volume derivatives, which end here:
    // modes 0 to 2 at w[8 m + j], mode 3 at n[j]
    const double determ = s.volo[k] * vk;
    {
        const fx::Factor volinv = fx::factor(rcp_op(determ), bad);
        fx::Factor hm[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int m = 0; m < 4; ++m) hm[i][m] = fx::factor(h[(4 * i + m) * BS], bad);
#pragma unroll 1
        for (int j = c; j < 8; j += kTeam) {
            const fx::Factor dx = fx::factor(w[(0 + j) * BS], bad);
            const fx::Factor dy = fx::factor(w[(8 + j) * BS], bad);
            const fx::Factor dz = fx::factor(w[(16 + j) * BS], bad);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const double sum = fx::product(dx, hm[0][m]) + fx::product(dy, hm[1][m]) +
                                   fx::product(dz, hm[2][m]);
                (m < 3 ? w + (8 * m + j) * BS : sm + j * BS)[0] =
                    signed_by(1.0, fx::mode_signs(m) >> j) -
                    fx::product(fx::factor(sum, bad), volinv);
            }
        }
    }
    const double coefficient =
        div_op(-hourg * 0.01 * s.ss[k] * s.elemMass[k], cbrt(determ));
    __syncthreads();
    {
        const fx::Factor coef = fx::factor(coefficient, bad);
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
        if (live && hg) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                cs[(3 + c) * E8 + (size_t)j * E] = fx::product(fx::factor(f[j], bad), coef);
        }
    }
    flags[c * BS] = (int)bad;
    __syncthreads();
    if (c == 0 && live && (flags[0] | flags[BS] | flags[2 * BS])) forces_general(s, k, ctl, hourg);
}

// six blocks of an SM: 112 registers; one wave at the largest mesh that comes here
constexpr int kTeamBlocks = 6;

template <bool BATCHED>
__global__ void __launch_bounds__(kTeam *kTeamElems, kTeamBlocks) k_forces_team(DevState s)
{
    follow_on();
    constexpr int BS = kTeamElems;
    extern __shared__ double force_scratch[];
    const int lane = threadIdx.x % BS, c = threadIdx.x / BS;
    int *const em = reinterpret_cast<int *>(force_scratch + ForceSlots::COUNT * BS) + lane;
    // one answer for the block: an element of another may end the cycle meanwhile
    if (!BATCHED && !__syncthreads_or(cycle_live(s.ctl))) return;
    for (int k0 = blockIdx.x * BS; k0 < s.E; k0 += gridDim.x * BS) {
        const int k = k0 + lane < s.E ? k0 + lane : s.E - 1;
        const int pid = BATCHED ? s.elemProb[k] : 0;
        Ctl *ctl = s.ctl + pid;
        const bool live = k0 + lane < s.E && (!BATCHED || cycle_live(ctl));
        if (BATCHED && !__syncthreads_or(live)) continue;
        forces_team<BS>(s, k, live, ctl, s.hgcoefs[pid], force_scratch + lane, em, c);
        if (BATCHED) __syncthreads();
    }
}

// One element's component c by one thread, with two others of the same block (see
// forces_team); sm is the element's column (coordinates; the half step's Jacobian; the
// gradients' differences of the coordinates and velocities; cofactors).
template <int BS>
__device__ __forceinline__ void kinematics_team(const DevState &s, const int k, const bool live,
                                                Ctl *ctl, double *sm, int *em, const int c)
{
    const int E = s.E;
    fx::i64 *const n = reinterpret_cast<fx::i64 *>(sm);
    double *const jac = sm + KinSlots::JAC * BS, *const grad = sm + KinSlots::GRAD * BS,
                 *const vgrad = sm + KinSlots::VGRAD * BS, *const cof = sm + KinSlots::COF * BS;
    int nd[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) nd[j] = __ldg(&s.nodelistT[(size_t)j * E + k]);
    unsigned bad = 0;
    double v[8];
    {
        const fx::Factor dt2 = fx::factor(0.5 * ctl->deltatime, bad);
        const double *const px = c == 0 ? s.x : c == 1 ? s.y : s.z;
        const double *const pv = c == 0 ? s.xd : c == 1 ? s.yd : s.zd;
        double x[8], h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = px[nd[j]];
            v[j] = pv[nd[j]];
        }
        const int ec = fx::align8<BS>(x, n + 8 * c * BS, bad);
        em[c * BS] = ec;
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = x[j] - fx::product(fx::factor(v[j], bad), dt2);
        const double D0 = h[6] - h[0], D1 = h[5] - h[3], D2 = h[7] - h[1], D3 = h[4] - h[2];
        jac[(3 * c + 0) * BS] = D0 + D1 - D2 - D3;
        jac[(3 * c + 1) * BS] = D0 - D1 + D2 - D3;
        jac[(3 * c + 2) * BS] = D0 + D1 + D2 + D3;
        fx::gradient_sums<BS>(n + 8 * c * BS, ec, grad + 3 * c * BS);
#define LG_S4(a, b, c, d) (v[a] + v[b] + v[c] + v[d])
        vgrad[(3 * c + 0) * BS] = LG_S4(1, 2, 6, 5) - LG_S4(0, 3, 7, 4);
        vgrad[(3 * c + 1) * BS] = signed_by(LG_S4(0, 1, 5, 4) - LG_S4(3, 2, 6, 7), 1);
        vgrad[(3 * c + 2) * BS] = LG_S4(4, 5, 6, 7) - LG_S4(0, 1, 2, 3);
#undef LG_S4
    }
    __syncthreads();
    const int emax[3] = {em[0], em[BS], em[2 * BS]};
    const double triple = fx::volume_triple<BS>(n, emax, c, bad);
    const double largest = fx::largest_area_face<BS>(n, emax, 2 * c, 2, bad);
    // 64 x the cofactors q of row c: of the rows c + 1, c + 2 and columns d + 1, d + 2
    double part;
    {
        const double *const j1 = jac + (c == 2 ? 0 : 3 * (c + 1)) * BS,
                            *const j2 = jac + (c == 0 ? 6 : 3 * (c - 1)) * BS;
        fx::Factor r1[3];
        fx::Factor r2[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            r1[d] = fx::factor(j1[d * BS], bad);
            r2[d] = fx::factor(j2[d * BS], bad);
        }
        double q[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
            q[d] = fx::product(r1[d1], r2[d2]) - fx::product(r1[d2], r2[d1]);
        }
        part = fx::product(fx::factor(q[1], bad), fx::factor(jac[(3 * c + 1) * BS], bad));
        const double ic = q[0] + q[1], id = q[0] - q[1];
        const double sum =
            fx::product(fx::factor(-ic - q[2], bad), fx::factor(v[0] - v[6], bad)) +
            fx::product(fx::factor(id - q[2], bad), fx::factor(v[1] - v[7], bad)) +
            fx::product(fx::factor(ic - q[2], bad), fx::factor(v[2] - v[4], bad)) +
            fx::product(fx::factor(-id - q[2], bad), fx::factor(v[3] - v[5], bad));
        cof[(0 + c) * BS] = part;
        cof[(3 + c) * BS] = triple;
        cof[(6 + c) * BS] = largest;
        part = sum;
    }
    __syncthreads();
    const double volo = s.volo[k];
    const double volume =
        fx::product(fx::factor(cof[3 * BS] + cof[4 * BS] + cof[5 * BS], bad),
                    fx::factor(1.0 / 12.0, bad));
    const double relativeVolume = div_op(volume, volo);
    const double inv_detJ = rcp_op(cof[0] + cof[BS] + cof[2 * BS]);
    const double rate = fx::product(fx::factor(part, bad), fx::factor(inv_detJ, bad));

    // CalcMonotonicQGradientsForElems: direction c from the differences of the other two
    {
        const double vol = fx::product(fx::factor(volo, bad), fx::factor(relativeVolume, bad));
        const fx::Factor norm = fx::factor(fx::times_pow2<-6>(rcp_op(vol + 1.e-36)), bad);
        const int p = c == 2 ? 0 : c + 1, q = c == 0 ? 2 : c - 1;
        fx::Factor a[3];
        fx::Factor b[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = fx::factor(grad[(3 * i + p) * BS], bad);
            b[i] = fx::factor(grad[(3 * i + q) * BS], bad);
        }
        double size = 0.0, slope = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
            const fx::Factor x =
                fx::factor(fx::product(a[i1], b[i2]) - fx::product(a[i2], b[i1]), bad);
            const double xx = fx::product(x, x);
            const double xv = fx::product(fx::factor(fx::product(x, norm), bad),
                                          fx::factor(vgrad[(3 * i + c) * BS], bad));
            size = i ? size + xx : xx;
            slope = i ? slope + xv : xv;
        }
        double *const ox = c == 0 ? s.delx_xi : c == 1 ? s.delx_eta : s.delx_zeta;
        double *const ov = c == 0 ? s.delv_xi : c == 1 ? s.delv_eta : s.delv_zeta;
        const double length = div_op(fx::times_pow2<4>(vol), sqrt_op(size + 256.e-36));
        if (live) {
            ox[k] = length;
            ov[k] = slope;
        }
    }
    jac[c * BS] = rate;  // the Jacobian has been read
    int *const flags = em + kTeam * BS;
    flags[c * BS] = (int)bad;
    __syncthreads();
    if (!live || c != 0) return;
    if (flags[0] | flags[BS] | flags[2 * BS]) {
        kinematics_general(s, k, ctl);
        return;
    }
    double area = cof[6 * BS];
    area = lt(cof[7 * BS], area) ? area : cof[7 * BS];
    area = lt(cof[8 * BS], area) ? area : cof[8 * BS];
    s.vnew[k] = relativeVolume;
    s.delv[k] = relativeVolume - s.v[k];
    s.arealg[k] = div_op(fx::times_pow2<2>(volume), sqrt_op(area));
    s.vdov[k] = jac[0] + jac[BS] + jac[2 * BS];
    if (dle(relativeVolume, 0.0)) raise_status(ctl, -1);  // lulesh.cc:1598-1605
}

template <bool BATCHED>
__global__ void __launch_bounds__(kTeam *kTeamElems, kTeamBlocks) k_kinematics_team(DevState s)
{
    follow_on();
    constexpr int BS = kTeamElems;
    extern __shared__ double kin_scratch[];
    const int lane = threadIdx.x % BS, c = threadIdx.x / BS;
    int *const em = reinterpret_cast<int *>(kin_scratch + KinSlots::COUNT * BS) + lane;
    // one answer for the block: an element of another may end the cycle meanwhile
    if (!BATCHED && !__syncthreads_or(cycle_live(s.ctl))) return;
    for (int k0 = blockIdx.x * BS; k0 < s.E; k0 += gridDim.x * BS) {
        const int k = k0 + lane < s.E ? k0 + lane : s.E - 1;
        Ctl *ctl = s.ctl + (BATCHED ? s.elemProb[k] : 0);
        const bool live = k0 + lane < s.E && (!BATCHED || cycle_live(ctl));
        if (BATCHED && !__syncthreads_or(live)) continue;
        kinematics_team<BS>(s, k, live, ctl, kin_scratch + lane, em, c);
        if (BATCHED) __syncthreads();
    }
}
