// lg_adjoint.cu -- checkpointed reverse-mode adjoint of the FP64 leap-frog
// cycle with the time-step sequence frozen.
//
// The cycle c maps the state S_c = (x, y, z, xd, yd, zd, e, p, q, v, ss) to
// S_{c+1} with the frozen step dt_c.  Its adjoint runs the forward phases
// backwards, one kernel per phase, each element or node recomputing the
// forward values it needs (lg_adjoint_math.h) from stored states:
//   ka_material   EOS (one repetition: the repetitions recompute identical
//                 values) and monotonic-Q limiter, from the adjoints of
//                 e, p, q, ss, v of S_{c+1}
//   ka_qslots     the limiter's neighbour reads, transposed into a gather
//   ka_kinematics Q gradients and the element volume (vnew = V / volo)
//   ka_nodes      position/velocity update, a = F / m, boundary conditions
//   ka_forces     stress and FB hourglass forces
//   ka_gather     the element -> node corner sums of the two element phases
// Scatter adjoints become gathers through the corner scratch and the node
// corner lists, as in the forward path: no atomics, deterministic sums.
// S_c is checkpointed every k cycles in a first forward pass; each segment is
// recomputed from its checkpoint storing S_c and the per-cycle temporaries
// (vnew, vdov and the six Q gradients), then swept backwards.
// The reverse kernels are bound by the FP64 pipe: quotients and roots are the integer
// pipes' (the same bits)
#define LG_EXACT_OPS 1

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "lg_adjoint.h"
#include "lg_adjoint_cycle.h"
#include "lg_exact.cuh"
#include "lg_device.h"
#include "lg_kernelset.h"

namespace lg {
int record_error(int code, const char *msg);
}

#include "lulesh_gb300.h"

namespace {

constexpr int kB = 128;
using namespace ::lg::adj;

__global__ void __launch_bounds__(kB) ka_material(lg::DevState s, AdjArgs a)
{
    const int k = blockIdx.x * kB + threadIdx.x;
    if (k < s.E) adj_material(s, a, k);
}

__global__ void __launch_bounds__(kB) ka_qslots(lg::DevState s, AdjArgs a)
{
    const int k = blockIdx.x * kB + threadIdx.x;
    if (k < s.E) adj_qslots(s, a, k);
}

__global__ void __launch_bounds__(kB) ka_kinematics(lg::DevState s, AdjArgs a)
{
    const int k = blockIdx.x * kB + threadIdx.x;
    if (k < s.E) adj_kinematics(s, a, k);
}

__global__ void __launch_bounds__(kB) ka_nodes(lg::DevState s, AdjArgs a)
{
    const int n = blockIdx.x * kB + threadIdx.x;
    if (n < s.N) adj_nodes(s, a, n);
}

__global__ void __launch_bounds__(kB) ka_forces(lg::DevState s, AdjArgs a)
{
    const int k = blockIdx.x * kB + threadIdx.x;
    const double hgb = (k < s.E) ? adj_forces(s, a, k) : 0.;
    // block sum of the hourglass-coefficient adjoint (fixed order)
    __shared__ double red[kB];
    red[threadIdx.x] = hgb;
    __syncthreads();
    for (int w = kB / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) a.hgPart[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(kB) ka_gather(lg::DevState s, AdjArgs a)
{
    const int n = blockIdx.x * kB + threadIdx.x;
    if (n < s.N) adj_gather(s, a, n);
}

// Copies up to 19 arrays in one launch (blockIdx.y: the array).  A cycle's
// state and temporaries went as 19 device-to-device copies, 2 to 3 us each:
// more than the forward cycle's own kernels on small meshes.
constexpr int kCopies = 19;
struct Copies {
    double *dst[kCopies];
    const double *src[kCopies];
    unsigned n[kCopies];
};
__global__ void __launch_bounds__(256) ka_copy(Copies c)
{
    const unsigned i = blockIdx.x * 256 + threadIdx.x, a = blockIdx.y;
    if (i < c.n[a]) c.dst[a][i] = c.src[a][i];
}

// Adds the per-block hourglass-coefficient partials of one reverse cycle to
// acc: one block, each thread summing a strided subset in index order, then
// a pairwise tree in shared memory.  The order is fixed, so the sum is the
// same on every run; one thread reading them in turn waited on each load.
__global__ void __launch_bounds__(kB) ka_hg_sum(const double *part, int nparts, double *acc)
{
    __shared__ double red[kB];
    double t = 0.;
    for (int i = threadIdx.x; i < nparts; i += kB) t += part[i];
    red[threadIdx.x] = t;
    __syncthreads();
    for (int w = kB / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *acc += red[0];
}

int err(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    return lg::record_error(code, buf);
}

#define AD_CUDA(call)                                                                    \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return err(LG_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_),     \
                       __FILE__, __LINE__);                                              \
    } while (0)

}  // namespace

namespace lg {

// Handles keep their sweeps' memory between calls up to this size, all of them together;
// a sweep that would exceed it gives its own back (the allocation costs a large one
// nothing in comparison)
constexpr size_t kKeepBytes = (size_t)256 << 20;
std::atomic<size_t> g_kept{0};

int AdjointWork::reserve(size_t bytes, char **out)
{
    if (bytes > held) {
        free_arena();
        if (cudaMalloc(&arena, bytes) != cudaSuccess) {
            (void)cudaGetLastError();
            arena = nullptr;
            return err(LG_ERR_NOMEM, "adjoint: cudaMalloc(%zu bytes) failed", bytes);
        }
        held = bytes;
    }
    *out = arena;
    return LG_OK;
}

void AdjointWork::free_arena()
{
    if (kept) g_kept -= held;
    if (arena) cudaFree(arena);
    arena = nullptr;
    held = 0;
    kept = false;
}

void AdjointWork::release()
{
    size_t k = g_kept.load();
    while (!kept && k + held <= kKeepBytes) kept = g_kept.compare_exchange_weak(k, k + held);
    if (!kept) free_arena();
}

void AdjointWork::drop_map()
{
    if (revStart) cudaFree(revStart);
    revStart = revEntry = nullptr;
}

void AdjointWork::drop()
{
    drop_map();
    free_arena();
}

// The limiter's reverse neighbour map (element j reads element k), by counting:
// each list in ascending j.  It depends on the topology alone and is kept until
// that changes.
int AdjointWork::reverse_map(const AdjointIO &io, int E, cudaStream_t st)
{
    if (revStart) return LG_OK;
    const std::vector<int> *nb[6] = {io.lxim, io.lxip, io.letam, io.letap, io.lzetam, io.lzetap};
    const int mask[6] = {XI_M, XI_P, ETA_M, ETA_P, ZETA_M, ZETA_P};
    const int sym[6] = {XI_M_SYMM, XI_P_SYMM, ETA_M_SYMM, ETA_P_SYMM, ZETA_M_SYMM, ZETA_P_SYMM};
    const int fr[6] = {XI_M_FREE, XI_P_FREE, ETA_M_FREE, ETA_P_FREE, ZETA_M_FREE, ZETA_P_FREE};
    auto uses = [&](int bits, int f) {
        const int b = bits & mask[f];
        return b == 0 || (b != sym[f] && b != fr[f] && b == (mask[f] & ~(sym[f] | fr[f])));
    };
    std::vector<int> start((size_t)E + 1, 0), entry;
    for (int f = 0; f < 6; ++f)
        for (int j = 0; j < E; ++j)
            if (uses((*io.elemBC)[j], f)) ++start[(*nb[f])[j] + 1];
    for (int k = 0; k < E; ++k) start[k + 1] += start[k];
    entry.assign(std::max(1, start[E]), 0);
    {
        std::vector<int> at(start.begin(), start.end() - 1);
        for (int j = 0; j < E; ++j)
            for (int f = 0; f < 6; ++f)
                if (uses((*io.elemBC)[j], f)) entry[at[(*nb[f])[j]]++] = j * 6 + f;
    }
    int *d = nullptr;
    if (cudaMalloc(&d, sizeof(int) * (start.size() + entry.size())) != cudaSuccess) {
        (void)cudaGetLastError();
        return err(LG_ERR_NOMEM, "adjoint: no memory for the neighbour map");
    }
    revStart = d;
    revEntry = d + start.size();
    cudaError_t e = cudaMemcpyAsync(revStart, start.data(), sizeof(int) * start.size(),
                                    cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(revEntry, entry.data(), sizeof(int) * entry.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        drop_map();
        return err(LG_ERR_CUDA, "adjoint: %s", cudaGetErrorString(e));
    }
    return LG_OK;
}

int adjoint_run(const AdjointIO &io, double *J, double *dJdhg)
{
    const DevState &S = *io.ds;
    const int E = S.E, N = S.N;
    const int K = std::max(1, std::min(io.ckpt_k, io.ncycles));
    const int nseg = (io.ncycles + K - 1) / K;
    const size_t snapD = 6 * (size_t)N + 5 * (size_t)E, tempD = 8 * (size_t)E;
    cudaStream_t st = io.stream;

    // one arena for checkpoints, the segment store and the adjoint arrays
    const int eb = (E + kB - 1) / kB, nbk = (N + kB - 1) / kB;
    const size_t dbl = (size_t)(nseg + 1) * snapD + (size_t)(K + 1) * snapD + (size_t)K * tempD +
                       6 * (size_t)N + 5 * (size_t)E + 7 * (size_t)E + 6 * (size_t)E +
                       48 * (size_t)E + 3 * (size_t)N + eb + 1;
    char *arena = nullptr;
    const size_t bytes = dbl * sizeof(double);
    int rc;
    if ((rc = io.work->reverse_map(io, E, st)) || (rc = io.work->reserve(bytes, &arena))) return rc;
    struct Free {
        AdjointWork *w;
        ~Free() { w->release(); }
    } guard{io.work};
    double *p = reinterpret_cast<double *>(arena);
    auto take = [&](size_t n) {
        double *r = p;
        p += n;
        return r;
    };
    double *ckpt = take((size_t)(nseg + 1) * snapD);
    double *seg = take((size_t)(K + 1) * snapD);
    double *tmp = take((size_t)K * tempD);
    double *nbar = take(6 * (size_t)N);
    double *ebar = take(5 * (size_t)E);
    double *vnewb = take(E), *dxb = take(3 * (size_t)E), *dvb = take(3 * (size_t)E);
    double *slot = take(6 * (size_t)E), *corner = take(48 * (size_t)E), *fb = take(3 * (size_t)N);
    double *hgPart = take(eb), *hgAcc = take(1);

    double *const live_n[6] = {S.x, S.y, S.z, S.xd, S.yd, S.zd};
    double *const live_e[5] = {S.e, S.p, S.q, S.v, S.ss};
    double *const live_t[8] = {S.vnew, S.vdov, S.delx_xi, S.delx_eta, S.delx_zeta,
                               S.delv_xi, S.delv_eta, S.delv_zeta};
    auto snap_at = [&](double *base) {
        Snap s;
        for (int i = 0; i < 6; ++i) s.n[i] = base + (size_t)i * N;
        for (int i = 0; i < 5; ++i) s.el[i] = base + 6 * (size_t)N + (size_t)i * E;
        return s;
    };
    const unsigned cb_x = (unsigned)((std::max(E, N) + 255) / 256);
    // the live state into a snapshot, and a cycle's temporaries when given
    auto save = [&](double *base, double *temps) -> int {
        const Snap s = snap_at(base);
        Copies c{};
        for (int i = 0; i < 6; ++i) c.dst[i] = s.n[i], c.src[i] = live_n[i], c.n[i] = (unsigned)N;
        for (int i = 0; i < 5; ++i)
            c.dst[6 + i] = s.el[i], c.src[6 + i] = live_e[i], c.n[6 + i] = (unsigned)E;
        for (int i = 0; temps && i < 8; ++i)
            c.dst[11 + i] = temps + (size_t)i * E, c.src[11 + i] = live_t[i], c.n[11 + i] = (unsigned)E;
        ka_copy<<<dim3(cb_x, temps ? 19 : 11), 256, 0, st>>>(c);
        AD_CUDA(cudaGetLastError());
        return LG_OK;
    };
    auto restore = [&](const double *base) -> int {
        const Snap s = snap_at(const_cast<double *>(base));
        Copies c{};
        for (int i = 0; i < 6; ++i) c.dst[i] = live_n[i], c.src[i] = s.n[i], c.n[i] = (unsigned)N;
        for (int i = 0; i < 5; ++i)
            c.dst[6 + i] = live_e[i], c.src[6 + i] = s.el[i], c.n[6 + i] = (unsigned)E;
        ka_copy<<<dim3(cb_x, 11), 256, 0, st>>>(c);
        AD_CUDA(cudaGetLastError());
        return LG_OK;
    };
    auto read_ctl = [&](Ctl *out) -> int {
        AD_CUDA(cudaMemcpyAsync(io.h_ctl, S.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, st));
        AD_CUDA(cudaStreamSynchronize(st));
        *out = *io.h_ctl;
        return LG_OK;
    };
    auto write_ctl = [&](const Ctl &c) -> int {
        *io.h_ctl = c;
        AD_CUDA(cudaMemcpyAsync(S.ctl, io.h_ctl, sizeof(Ctl), cudaMemcpyHostToDevice, st));
        AD_CUDA(cudaStreamSynchronize(st));
        return LG_OK;
    };
    auto cycle = [&]() -> int {
        AD_CUDA(cudaGraphLaunch(io.cycle, st));
        return LG_OK;
    };

    // forward pass: checkpoints at cycles 0, K, 2K, ...
    std::vector<Ctl> ckctl(nseg + 1);
    Ctl c0;
    if ((rc = read_ctl(&c0))) return rc;
    c0.cycle_limit = c0.cycle + io.ncycles;
    if ((rc = write_ctl(c0))) return rc;
    io.ks->begin(S.ctl, st);
    for (int c = 0; c < io.ncycles; ++c) {
        if (c % K == 0) {
            if ((rc = save(ckpt + (size_t)(c / K) * snapD, nullptr))) return rc;
            if ((rc = read_ctl(&ckctl[c / K]))) return rc;
        }
        if ((rc = cycle())) return rc;
    }
    AD_CUDA(cudaGetLastError());
    Ctl cend;
    if ((rc = read_ctl(&cend))) return rc;
    if (cend.status != 0) return cend.status;
    if ((rc = save(ckpt + (size_t)nseg * snapD, nullptr))) return rc;

    // the adjoint of the final state: the masked terminal energy sum(e * volo)
    // seeds e with volo on the masked elements; otherwise the caller's seeds
    AD_CUDA(cudaMemsetAsync(nbar, 0, 8 * 6 * (size_t)N, st));
    AD_CUDA(cudaMemsetAsync(ebar, 0, 8 * 5 * (size_t)E, st));
    AD_CUDA(cudaMemsetAsync(hgAcc, 0, 8, st));
    if (io.mask) {
        std::vector<double> e(E), volo(E);
        AD_CUDA(cudaMemcpyAsync(e.data(), S.e, 8 * (size_t)E, cudaMemcpyDeviceToHost, st));
        AD_CUDA(cudaMemcpyAsync(volo.data(), S.volo, 8 * (size_t)E, cudaMemcpyDeviceToHost, st));
        AD_CUDA(cudaStreamSynchronize(st));
        double j = 0.;
        std::vector<double> eb0(E, 0.);
        for (int i = 0; i < E; ++i)
            if (io.mask[i]) {
                j += e[i] * volo[i];
                eb0[i] = volo[i];
            }
        if (J) *J = j;
        AD_CUDA(cudaMemcpyAsync(ebar, eb0.data(), 8 * (size_t)E, cudaMemcpyHostToDevice, st));
    } else {
        for (int f = 0; f < kAdjFields; ++f) {
            if (!io.seed || !io.seed[f]) continue;
            double *dst = f < 6 ? nbar + (size_t)f * N : ebar + (size_t)(f - 6) * E;
            AD_CUDA(cudaMemcpyAsync(dst, io.seed[f], 8 * (size_t)(f < 6 ? N : E),
                                    cudaMemcpyHostToDevice, st));
        }
        AD_CUDA(cudaStreamSynchronize(st));  // the seeds are the caller's memory
    }

    AdjArgs A;
    for (int i = 0; i < 6; ++i) A.nb[i] = nbar + (size_t)i * N;
    A.eb = ebar;
    A.pb = ebar + E;
    A.qb = ebar + 2 * (size_t)E;
    A.vb = ebar + 3 * (size_t)E;
    A.ssb = ebar + 4 * (size_t)E;
    A.vnewb = vnewb;
    for (int d = 0; d < 3; ++d) {
        A.delxb[d] = dxb + (size_t)d * E;
        A.delvb[d] = dvb + (size_t)d * E;
    }
    A.slot = slot;
    A.corner = corner;
    A.fb = fb;
    A.hgPart = hgPart;
    A.revStart = io.work->revStart;
    A.revEntry = io.work->revEntry;
    A.hg = io.hgcoef;

    // backward over segments
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int cb = sg * K, ce = std::min(cb + K, io.ncycles);
        if ((rc = restore(ckpt + (size_t)sg * snapD))) return rc;
        Ctl cs = ckctl[sg];
        cs.cycle_limit = c0.cycle + ce;  // absolute, like the cycle counter
        if ((rc = write_ctl(cs))) return rc;
        if ((rc = save(seg, nullptr))) return rc;
        for (int c = cb; c < ce; ++c) {
            if ((rc = cycle())) return rc;
            if ((rc = save(seg + (size_t)(c - cb + 1) * snapD, tmp + (size_t)(c - cb) * tempD)))
                return rc;
        }
        Ctl cr;
        if ((rc = read_ctl(&cr))) return rc;
        if (cr.status != 0 || cr.cycle != c0.cycle + ce)
            return err(LG_ERR_STATE, "adjoint: the recomputed segment ended at cycle %d (status %d), "
                                     "not %d", cr.cycle, cr.status, c0.cycle + ce);
        for (int c = ce - 1; c >= cb; --c) {
            A.s0 = snap_at(seg + (size_t)(c - cb) * snapD);
            A.s1 = snap_at(seg + (size_t)(c - cb + 1) * snapD);
            for (int t = 0; t < 8; ++t) A.tc.t[t] = tmp + (size_t)(c - cb) * tempD + (size_t)t * E;
            A.dt = io.dts[c];
            ka_material<<<eb, kB, 0, st>>>(S, A);
            ka_qslots<<<eb, kB, 0, st>>>(S, A);
            ka_kinematics<<<eb, kB, 0, st>>>(S, A);
            ka_nodes<<<nbk, kB, 0, st>>>(S, A);
            ka_forces<<<eb, kB, 0, st>>>(S, A);
            ka_gather<<<nbk, kB, 0, st>>>(S, A);
            ka_hg_sum<<<1, kB, 0, st>>>(hgPart, eb, hgAcc);
        }
        AD_CUDA(cudaGetLastError());
    }
    for (int f = 0; f < kAdjFields; ++f) {
        if (!io.grad || !io.grad[f]) continue;
        const double *src = f < 6 ? nbar + (size_t)f * N : ebar + (size_t)(f - 6) * E;
        AD_CUDA(cudaMemcpyAsync(io.grad[f], src, 8 * (size_t)(f < 6 ? N : E),
                                cudaMemcpyDeviceToHost, st));
    }
    AD_CUDA(cudaMemcpyAsync(dJdhg, hgAcc, 8, cudaMemcpyDeviceToHost, st));
    // leave the handle in the final forward state
    if ((rc = restore(ckpt + (size_t)nseg * snapD))) return rc;
    if ((rc = write_ctl(cend))) return rc;
    AD_CUDA(cudaStreamSynchronize(st));
    return LG_OK;
}

}  // namespace lg
