// sfgpu_group.cu -- kernels and launches of the cluster engine
// (sfgpu_group.cuh): a residual evaluation or a whole Pure_DIIS iteration
// (SFNewton::PlainLBFGSDIIS, sfnewton.cpp:566-664) of a first-order 1D or 2D
// system per thread-block cluster.
#include <algorithm>
#include <cmath>
#include <cstring>
#include "sfgpu_group.cuh"
#include "sfgpu_group.h"

using namespace sfg;

namespace {

struct GroupArgs {
    const InstDesc *descs;
    int n, *queue;
    const double *x;            // residual mode: x -> f of descs[0]
    double *f;
    int m, maxit;
    double eta, tol;
    int *status, *iters;
    double *errs;
    int smem_doubles;
};

__device__ __forceinline__ Grp group_here() {
    Grp g;
    uint32_t r, s;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(s));
    g.rank = (int)r;
    g.size = (int)s;
    g.gt = g.rank * blockDim.x + threadIdx.x;
    g.gn = g.size * blockDim.x;
    return g;
}

__device__ __forceinline__ void load_desc(const InstDesc *src, InstDesc &I) {
    const int *s = reinterpret_cast<const int *>(src);
    int *d = reinterpret_cast<int *>(&I);
    for (int i = threadIdx.x; i < (int)(sizeof(InstDesc) / sizeof(int)); i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

// residual of the system in I at x (a 2D system's halo barriers: parity)
template <int kDim, int J, bool kCurved>
__device__ __forceinline__ void evaluate(const InstDesc &I, const double *x, double *f, const Grp &g, GShared &sh,
                                         double *sm, uint32_t &parity, const Local1 &loc) {
    if constexpr (kDim == 2) residual2d<J, kCurved>(I, x, f, g, sh, parity);
    else residual1d<kCurved>(I, x, f, g, sh, loc);
}

template <int kDim, int J, bool kCurved, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) group_residual_kernel(GroupArgs a) {
    double *sm = dyn_smem();
    __shared__ InstDesc I;
    __shared__ GShared sh;
    const Grp g = group_here();
    uint32_t parity = 0;
    group_init(sh);
    load_desc(a.descs, I);
    gsync(g);
    Local1 loc = {};
    if constexpr (kDim == 1) loc = localize1d(I, a.descs, sm, a.smem_doubles, 0);
    evaluate<kDim, J, kCurved>(I, a.x, a.f, g, sh, sm, parity, loc);
    if constexpr (kDim == 1) write_back1d(I, a.descs, loc, 0);
}

template <int kDim, int J, bool kCurved, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) group_diis_kernel(GroupArgs a) {
    double *sm = dyn_smem();
    __shared__ InstDesc I;
    __shared__ GShared sh;
    const Grp g = group_here();
    uint32_t parity = 0;
    const int m = a.m;
    group_init(sh);
    gsync(g);
    for (;;) {
        if (g.rank == 0 && threadIdx.x == 0) {
            const int q = atomicAdd(a.queue, 1);
            for (int r = 0; r < g.size; r++) st_peer(peer(smem_u32(&sh.inst), r), q);
        }
        gsync(g);
        const int inst = sh.inst;
        if (inst >= a.n) break;
        load_desc(a.descs + inst, I);
        const long long iv = I.nvar;
        double *x = I.x, *gr = I.g, *XR = I.XR, *XX0 = I.XX0;
        Local1 loc = {};
        if constexpr (kDim == 1) {
            loc = localize1d(I, a.descs + inst, sm, a.smem_doubles, m);
            x = loc.x; gr = loc.g; XR = loc.XR; XX0 = loc.XX0;
        }
        // first step: x = -eta * g(x_initial)  (sfnewton.cpp:578-584)
        evaluate<kDim, J, kCurved>(I, x, gr, g, sh, sm, parity, loc);
        gsync(g);
        double part[kHist + 1];
        int slot[kHist + 1];
#pragma unroll
        for (int i = 0; i <= kHist; i++) { part[i] = 0; slot[i] = -1; }
        slot[kHist] = 0;
        for (long long r = g.gt; r < iv; r += g.gn) {
            const double v = 0.0 - gr[r] * a.eta;
            XX0[r] = v - x[r];
            XR[r] = v;
            x[r] = v;
            part[kHist] += gr[r] * gr[r];
        }
        gsum(part, slot, 1, g, sh);
        double err = sqrt(sh.val[0]);
        int k = 0, it = 0, kd = 1, st = SFGPU_OK;
        for (int i = threadIdx.x; i < kHist * kHist; i += blockDim.x) sh.gram[i] = 0;
        gsync(g);
        while (a.tol < err && it < a.maxit) {
            it++;
            evaluate<kDim, J, kCurved>(I, x, gr, g, sh, sm, parity, loc);
            gsync(g);
            k = it % m;
            kd = min(kd + 1, m);
            double *xr = XR + (size_t)k * iv, *xx = XX0 + (size_t)k * iv;
            // x -= eta*g; XR[k] = x; XX0[k] = x - x0; Gram row and |g|^2 in one pass
#pragma unroll
            for (int i = 0; i <= kHist; i++) {
                part[i] = 0;
                slot[i] = (i < kd) ? i : (i == kHist ? kd : -1);
            }
            for (long long r = g.gt; r < iv; r += g.gn) {
                const double x0 = x[r], gv = gr[r];
                const double v = x0 - gv * a.eta;
                const double d = v - x0;
                double h[kHist];
#pragma unroll
                for (int i = 0; i < kHist; i++) {
                    if (i >= kd - 1) continue;      // the newest is d itself
                    int posi = k - kd + 1 + i;
                    if (posi < 0) posi += m;
                    h[i] = XX0[(size_t)posi * iv + r];
                }
                xr[r] = v;
                xx[r] = d;
                part[kHist] += gv * gv;
#pragma unroll
                for (int i = 0; i < kHist; i++) {
                    if (i >= kd) continue;
                    part[i] += (i == kd - 1 ? d : h[i]) * d;
                }
            }
            gsum(part, slot, kd + 1, g, sh);
            if (threadIdx.x < 32) {
                const int lane = threadIdx.x;
                // shift out the oldest row and column when the memory is full
                // (sfnewton.cpp:624-628), then the new row: the Gram entries
                // (i, j) of the kd kept steps, oldest first
                if (it >= m) {
                    // row by row: row i takes row i + 1, shifted by a column
#pragma unroll 1
                    for (int i = 0; i + 1 < m; i++) {
                        const double v = (lane + 1 < m) ? sh.gram[m * (i + 1) + lane + 1] : 0.0;
                        __syncwarp();
                        if (lane + 1 < m) sh.gram[m * i + lane] = v;
                        __syncwarp();
                    }
                }
                if (lane < kd) sh.gram[lane + m * (kd - 1)] = sh.gram[kd - 1 + m * lane] = sh.val[lane];
                __syncwarp();
                // until the memory is full the oldest step's own product is
                // 0 (the first step's is never formed, sfnewton.cpp:602-628):
                // that row goes last in the elimination
                const int first = (kd > 1 && sh.gram[0] == 0) ? 1 : 0;
#pragma unroll 1
                for (int e = lane; e < kd * kd; e += 32) {
                    const int i = (e / kd + first) % kd, j = (e % kd + first) % kd;
                    sh.A[e] = sh.gram[i + m * j];
                }
                __syncwarp();
                const bool ok = coeff_ldl_warp(kd, sh.A, sh.Q, sh.work);
                __syncwarp();
                if (ok) {
                    if (lane < kd) sh.coef[(lane + first) % kd] = sh.Q[lane];
                    __syncwarp();
                } else {
                    for (int e = lane; e < kd * kd; e += 32) sh.A[e] = sh.gram[(e % kd) + m * (e / kd)];
                    __syncwarp();
                    sfb::diis_coeff_warp(kd, sh.A, sh.Q, sh.coef);
                }
                double nc = 0;
#pragma unroll 1
                for (int i = 0; i < kd; i++) nc += sh.coef[i];
                __syncwarp();
                if (lane < kd) {
                    sh.coef[lane] = sh.coef[lane] / nc;
                    int posi = k - kd + 1 + lane;
                    if (posi < 0) posi += m;
                    sh.pos[lane] = posi;
                }
            }
            __syncthreads();
            for (long long r = g.gt; r < iv; r += g.gn) {
                double v = 0;
#pragma unroll
                for (int i = 0; i < kHist; i++) {
                    if (i >= kd) continue;
                    const double w = sh.coef[i] * XR[(size_t)sh.pos[i] * iv + r];
                    v = (i == 0) ? w : v + w;
                }
                x[r] = v;
            }
            err = sqrt(sh.val[kd]);
            gsync(g);
            if (!isfinite(err)) { st = SFGPU_ERR_NONFINITE; break; }
        }
        if (st == SFGPU_OK && !(err <= a.tol)) st = SFGPU_ERR_NOTCONVERGED;
        if constexpr (kDim == 1) write_back1d(I, a.descs + inst, loc, m);
        if (g.rank == 0 && threadIdx.x == 0) {
            a.status[inst] = st;
            a.iters[inst] = it;
            a.errs[inst] = err;
        }
        __syncthreads();
    }
}

using Kernel = void (*)(GroupArgs);

template <int kDim, int J, bool kCurved, int kThreads>
Kernel pick_mode(bool diis) {
    return diis ? (Kernel)group_diis_kernel<kDim, J, kCurved, kThreads>
                : (Kernel)group_residual_kernel<kDim, J, kCurved, kThreads>;
}

Kernel pick(const GroupShape &s, bool diis) {
    if (s.dim == 1 && s.threads <= 256)
        return s.curved ? pick_mode<1, 1, true, 256>(diis) : pick_mode<1, 1, false, 256>(diis);
    if (s.dim == 1) return s.curved ? pick_mode<1, 1, true, 512>(diis) : pick_mode<1, 1, false, 512>(diis);
    switch (s.J) {
        case 1: return s.curved ? pick_mode<2, 1, true, 512>(diis) : pick_mode<2, 1, false, 512>(diis);
        case 2: return s.curved ? pick_mode<2, 2, true, 512>(diis) : pick_mode<2, 2, false, 512>(diis);
        case 4: return s.curved ? pick_mode<2, 4, true, 512>(diis) : pick_mode<2, 4, false, 512>(diis);
        default: return s.curved ? pick_mode<2, 8, true, 512>(diis) : pick_mode<2, 8, false, 512>(diis);
    }
}

int cuda_fail(cudaError_t e, const char *what) {
    sfgpu_set_error(e, what, __FILE__, __LINE__);
    return SFGPU_ERR_CUDA;
}

}  // namespace

constexpr size_t kSmemMax = 204 * 1024;   // dynamic shared memory a block may take beside GShared and InstDesc

bool group_eligible(const sfgpu_system *s) {
    const DLat &L = s->H.L;
    if (s->K != 1 || L.order != 1 || L.grad > 2 || s->logmode || s->charged) return false;
    if (s->nseg > sfb::kResMax || s->nclass > sfb::kResMax || s->nmol > sfb::kMaxMol) return false;
    for (int d = 0; d < L.grad; d++)
        if (L.Md[d] - 2 < 3) return false;      // boundary copies of boundary copies: the general path
    for (const auto &o : s->mols)
        if (o.dend || o.tree || o.ring || o.force != 0 || s->primal_checkpointed(o)) return false;
    if (L.grad == 1) {
        // a periodic lattice's ends are neighbours: not in a warp's run of sites
        if (L.bc_lo[0] == SFGPU_BOUND_PERIODIC || L.bc_hi[0] == SFGPU_BOUND_PERIODIC) return false;
        return warps1d(L.Md[0] - 2) <= kMaxWarps1;
    }
    return true;
}

// what a 1D system asks of shared memory: exchange lines and the ring, its
// working arrays, and the stored slices of its longest chain
struct Doubles1 { size_t always, arrays, chain; };
static Doubles1 doubles1(const sfgpu_system *s) {
    const int n = s->H.L.Md[0] - 2;
    int nonfrozen = 0, pinned = 0, molphis = 0;
    Doubles1 q = {line1d(n) + kRing1 * slice1d(n), 0, 0};
    for (int i = 0; i < s->nseg; i++) {
        nonfrozen += s->freedom[i] != SFGPU_SEG_FROZEN;
        pinned += s->freedom[i] == SFGPU_SEG_PINNED;
    }
    for (const auto &o : s->mols) {
        molphis += (int)o.used.size();
        if (o.type != 0) q.chain = std::max(q.chain, (size_t)(o.sym ? o.N / 2 : o.N) * slice1d(n));
    }
    q.arrays = local1d_doubles(s->M, s->nseg, nonfrozen, pinned, molphis, s->nmol);
    return q;
}

// as localize1d decides it
size_t group_slices(const sfgpu_system *s, const GroupShape &g) {
    if (g.dim != 1) return 0;
    const Doubles1 q = doubles1(s);
    return q.always + q.arrays + q.chain <= g.smem / sizeof(double) ? 0 : q.chain;
}

// Blocks per cluster, rows per thread and threads of one system when `blocks`
// blocks at most work on it.  Rows per thread: the fewest whose threads stay
// within `threads`, so that a block's steps have many warps to hide their
// latencies behind (128 x 128 over 16 blocks: 0.43 us a step with 512 threads
// of 2 rows, 0.88 with 256 of 4).
bool group_shape(const sfgpu_system *s, int blocks, int threads, int m, GroupShape *out) {
    const DLat &L = s->H.L;
    GroupShape g;
    g.dim = L.grad;
    g.curved = L.cyl != 0;
    if (L.grad == 1) {
        const int n = L.Md[0] - 2;
        g.C = 1;
        g.J = 1;
        // the phases between the chains want a thread per site (one system alone,
        // n = 200: 3.30 ms a solve with 128 threads, 2.95 with 256).  In a large
        // batch two blocks of 128 share an SM where the largest instance leaves
        // them the room: up to 96 KB each beside 17 KB of static shared memory
        g.threads = std::max(blocks > 1 ? 256 : 128, 32 * warps1d(n));
        // what localize1d takes, in its order; the last ones only where they fit
        const Doubles1 need = doubles1(s);
        size_t d = need.always;
        const size_t most = kSmemMax / sizeof(double) / (blocks > 1 ? 1 : 2);
        if (d + need.arrays <= most) {
            d += need.arrays;
            if (d + need.chain <= most) d += need.chain;
            const size_t nv = s->nvar;
            if (m > 0 && d + 2 * nv <= most) {
                d += 2 * nv;
                if (d + 2 * nv * m <= most) d += 2 * nv * m;
            }
        }
        g.smem = sizeof(double) * ((d + 1) / 2 * 2);
        if (g.smem > kSmemMax) return false;
        *out = g;
        return true;
    }
    const int nx = L.Md[0] - 2, ny = L.Md[1] - 2;
    int C = std::max(1, std::min(std::min(blocks, kMaxCluster), nx));
    const int R = (nx + C - 1) / C;
    C = (nx + R - 1) / R;
    g.C = C;
    for (int J : {1, 2, 4, 8}) {
        const long t = ((long)ny * ((R + J - 1) / J) + 31) / 32 * 32;
        if (t > threads && J < 8) continue;
        if (t > 512) return false;
        g.J = J;
        g.threads = (int)t;
        break;
    }
    g.smem = sizeof(double) * (2 * (size_t)(R + 2) * L.Md[1] + 2 * (size_t)R);
    if (g.smem > kSmemMax) return false;
    *out = g;
    return true;
}

int group_prepare(const GroupShape &s, bool diis) {
    Kernel k = pick(s, diis);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute");
    if (s.C > 8 && (e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
        return cuda_fail(e, "cudaFuncSetAttribute");
    return SFGPU_OK;
}

static void config(const GroupShape &s, int clusters, cudaStream_t st, cudaLaunchConfig_t *cfg,
                   cudaLaunchAttribute *attr) {
    *cfg = {};
    cfg->gridDim = dim3(s.C * clusters);
    cfg->blockDim = dim3(s.threads);
    cfg->dynamicSmemBytes = s.smem;
    cfg->stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = s.C;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = s.C > 1 ? 1 : 0;
}

int group_max_clusters(const GroupShape &s, bool diis) {
    int rc = group_prepare(s, diis);
    if (rc) { cudaGetLastError(); return 0; }
    int n = 0;
    if (s.C == 1) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pick(s, diis), s.threads, s.smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n * sms;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(s, 1, nullptr, &cfg, &attr);
    if (cudaOccupancyMaxActiveClusters(&n, pick(s, diis), &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}

int group_residual(const GroupShape &s, const sfb::InstDesc *desc, const double *x, double *f, cudaStream_t st) {
    GroupArgs a = {};
    a.descs = desc;
    a.n = 1;
    a.x = x;
    a.f = f;
    a.smem_doubles = (int)(s.smem / sizeof(double));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(s, 1, st, &cfg, &attr);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, pick(s, false), a);
    return e == cudaSuccess ? SFGPU_OK : cuda_fail(e, "cudaLaunchKernelEx");
}

int group_diis(const GroupShape &s, const sfb::InstDesc *descs, int n, int clusters, int *queue, int m, double eta,
               double tol, int maxit, int *status, int *iters, double *errs, cudaStream_t st) {
    GroupArgs a = {};
    a.descs = descs;
    a.n = n;
    a.queue = queue;
    a.m = m;
    a.eta = eta;
    a.tol = tol;
    a.maxit = maxit;
    a.status = status;
    a.iters = iters;
    a.errs = errs;
    a.smem_doubles = (int)(s.smem / sizeof(double));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(s, clusters, st, &cfg, &attr);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, pick(s, true), a);
    return e == cudaSuccess ? SFGPU_OK : cuda_fail(e, "cudaLaunchKernelEx");
}
