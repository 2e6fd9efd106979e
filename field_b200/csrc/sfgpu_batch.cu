// sfgpu_batch.cu -- persistent batched solver: many independent SF-SCF
// instances (a Vary-style sweep, Vary.cpp:127 / SF_Box.cpp:145-177) solved by
// Pure_DIIS in ONE kernel launch.  Blocks take instances from an atomic work
// queue, so uneven instances (different lattices and chain lengths) balance
// across the SMs; each block iterates its instance to convergence on device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "sfgpu_batch_kernel.cuh"
#include "sfgpu_group.h"

using namespace sfb;

struct sfgpu_batch {
    std::vector<sfgpu_system *> sys;
    std::vector<InstDesc> desc_h;
    InstDesc *d_desc = nullptr;
    int *d_queue = nullptr, *d_status = nullptr, *d_iters = nullptr;
    double *d_err = nullptr, *d_xall = nullptr;
    std::vector<long long> offset;      // start of each instance in the concatenated x
    long long total = 0;
    int m = 10, block = 256;
    size_t stage_bytes = 0;         // dynamic shared memory per block (staged G)
    bool wide = false;              // some instance needs batch_diis_kernel_t<true>
    bool grouped = false;           // every instance runs in the cluster engine, with this shape
    GroupShape shape;
    int clusters = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<void *> allocs;
    ~sfgpu_batch() {
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        for (void *p : allocs) cudaFree(p);
        for (auto *s : sys) delete s;
        if (own_stream && stream) cudaStreamDestroy(stream);
    }
};

static int balloc(sfgpu_batch *b, void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes ? bytes : 8);
    if (e != cudaSuccess) { sfgpu_set_error(e, "cudaMalloc", __FILE__, __LINE__); return SFGPU_ERR_NOMEM; }
    b->allocs.push_back(*p);
    return SFGPU_OK;
}

// ---------------------------------------------------------------------------
// Shared-memory staging of each instance: G of the running segment where
// the lattice fits next to the kernel's static shared memory, and on 1D
// symmetric homopolymers also the running slices, phi and the ring of
// stored slices.  allow = false stages nothing (more blocks per SM).
static BatchKernel batch_kernel(const sfgpu_batch *b) {
    return b->wide ? batch_kernel_wide() : batch_diis_kernel_t<false>;
}

static int configure_stage(sfgpu_batch *b, bool allow) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, batch_kernel(b)) != cudaSuccess)
        return SFGPU_ERR_CUDA;
    const size_t fixed = fa.sharedSizeBytes + 1024;   // 1 KB the system reserves per block
    const size_t room = (size_t)optin > fixed ? (size_t)optin - fixed : 0;
    size_t need = 0;
    const int n = (int)b->sys.size();
    for (int i = 0; i < n; i++) {
        const size_t bytes = sizeof(double) * (size_t)b->sys[i]->M;
        b->desc_h[i].gstage = (allow && bytes <= room) ? 1 : 0;
        if (b->desc_h[i].gstage) need = std::max(need, bytes);
        // 1D symmetric homopolymers: G, two running slices, phi and the
        // ring of stored slices, when these 4 + kRing lattice vectors fit
        // in 48 KB (M <= 768), a budget that keeps several blocks
        // resident per SM
        const auto *sy = b->sys[i];
        bool sym1d = allow && sy->H.L.grad == 1;
        bool any_sym = false;
        for (const auto &o : sy->mols) any_sym |= o.sym != 0;
        const size_t vecs = (4 + sfb::kRing) * bytes;
        sym1d = sym1d && any_sym && vecs <= 48 * 1024 && vecs <= room;
        b->desc_h[i].small1d = sym1d ? 1 : 0;
        if (sym1d) need = std::max(need, vecs);
    }
    if (cudaMemcpyAsync(b->d_desc, b->desc_h.data(), sizeof(InstDesc) * n, cudaMemcpyHostToDevice, b->stream) !=
            cudaSuccess ||
        cudaFuncSetAttribute(batch_kernel(b), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need) !=
            cudaSuccess)
        return SFGPU_ERR_CUDA;
    b->stage_bytes = need;
    return SFGPU_OK;
}

// The cluster engine takes a batch whose instances it all accepts on lattices
// of one kind.  2D blocks per instance: with enough instances to fill the
// chip, about 2048 sites a block (fewer blocks idle less in halo exchanges,
// more let two blocks share an SM and hide them).  296 cylinders of 128 x 128
// to 1e-11: 172 ms with 8 blocks of 256 threads, 176 with 4 of 512, 218 with 16
// of 256, and 231 in the one-block-per-instance kernel; these with the engine as
// it was before the phases that run once an iteration were shortened, with
// which the 8 blocks take 159.  With fewer instances
// the SMs left over go to their clusters.
static void configure_group(sfgpu_batch *b) {
    const sfgpu_system *s0 = b->sys[0];
    const int n = (int)b->sys.size();
    long sites = 1;
    for (auto *s : b->sys) {
        const DLat &L = s->H.L;
        if (!group_eligible(s) || L.grad != s0->H.L.grad || (L.cyl != 0) != (s0->H.L.cyl != 0)) return;
        if (L.grad == 2) sites = std::max(sites, (long)(L.Md[0] - 2) * (L.Md[1] - 2));
    }
    int C = 1, threads = 256;
    if (s0->H.L.grad == 2) {
        while (C < 8 && sites > 2048L * C) C *= 2;
        const int base = C;
        while (C < 16 && 2L * C * n <= 148) C *= 2;
        if (C > base) threads = 512;
    } else if (n <= 148) {
        C = 2;   // 1D: one block an SM, whose shared memory the chain's slices may fill
    }
    GroupShape big;
    for (auto *s : b->sys) {
        GroupShape g;
        if (!group_shape(s, C, threads, b->m, &g)) return;
        big.J = std::max(big.J, g.J);
    }
    for (auto *s : b->sys) {
        GroupShape g;
        group_shape(s, C, threads, b->m, &g);
        big.dim = g.dim;
        big.curved = g.curved;
        big.C = std::max(big.C, g.C);
        big.threads = std::max(big.threads, g.threads);
        big.smem = std::max(big.smem, g.smem);
    }
    const int most = group_max_clusters(big, true);
    if (most < 1) return;
    b->shape = big;
    b->clusters = std::min(n, most);
    b->grouped = true;
}

// Tables and working memory of all instances, in one allocation each and one copy
// (256 uneven 1D systems of up to 400 layers and 1000 segments: 78 ms to create
// and 116 MiB; with allocations and copies per instance, and slices beside d_gi,
// 112 ms and 176 MiB).  chains[i]: instance i's chain tables.
static int upload_tables(sfgpu_batch *b, std::vector<const int *> *chains) {
    const size_t n = b->sys.size();
    std::vector<int> tables;
    std::vector<size_t> maps(n), at(n), part(n), slices(n);
    size_t doubles = 0;
    auto take = [&](size_t k) { const size_t r = doubles; doubles += (k + 1) / 2 * 2; return r; };   // 16-byte aligned
    for (size_t i = 0; i < n; i++) {
        sfgpu_system *s = b->sys[i];
        maps[i] = tables.size();
        if (b->grouped) {
            s->site_maps(&tables);
            part[i] = take((size_t)s->nmol * ((s->M + 255) / 256));
            slices[i] = take(group_slices(s, b->shape));
        }
        std::vector<int>().swap(s->jmap_h);
        at[i] = tables.size();
        s->chain_tables(&tables);
    }
    int *d = nullptr, rc;
    double *w = nullptr;
    if ((rc = balloc(b, (void **)&d, sizeof(int) * tables.size()))) return rc;
    if (b->grouped && (rc = balloc(b, (void **)&w, sizeof(double) * doubles))) return rc;
    SFGPU_CUDA_TRY(cudaMemcpy(d, tables.data(), sizeof(int) * tables.size(), cudaMemcpyHostToDevice));
    for (size_t i = 0; i < n; i++) {
        sfgpu_system *s = b->sys[i];
        (*chains)[i] = d + at[i];
        if (!b->grouped) continue;
        s->d_smap = d + maps[i];
        s->d_jall = s->d_smap + s->M;
        s->d_wpart = w + part[i];
        s->d_slices1 = w + slices[i];
        if ((rc = s->clear_profiles())) return rc;
    }
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_create(int n, const sfgpu_system_desc *descs, int m, sfgpu_batch **out) {
    if (!out || !descs || n < 1) return SFGPU_ERR_INVALID;
    *out = nullptr;
    if (m < 1 || m > kMaxHist) return SFGPU_ERR_INVALID;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return SFGPU_ERR_NODEVICE; }
    sfgpu_batch *b = new sfgpu_batch();
    b->m = m;
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) { delete b; return SFGPU_ERR_CUDA; }
    b->own_stream = true;
    int rc = SFGPU_OK;
    int maxM = 1;
    b->offset.resize(n);
    for (int i = 0; i < n && !rc; i++) {
        if (descs[i].lattice.order != 1) { rc = fail_unsupported("batched second-order lattices"); break; }
        if (descs[i].overflow_protection) { rc = fail_unsupported("batched systems with overflow protection"); break; }
        for (int q = 0; q < descs[i].n_segments && !rc; q++)
            if (descs[i].segments[q].valence != 0) rc = fail_unsupported("batched charged systems");
        if (rc) break;
        for (int q = 0; q < descs[i].n_molecules && !rc; q++) {
            if (descs[i].molecules[q].n_generations > 0 || descs[i].molecules[q].bond_parent ||
                descs[i].molecules[q].ring)
                rc = fail_unsupported("batched dendrimers, branched molecules and rings");
            if (descs[i].molecules[q].force != 0) b->wide = true;
        }
        if (rc) break;
        if (descs[i].lattice.gradients == 3 && descs[i].lattice.lattice_type != SFGPU_LATTICE_STANDARD) b->wide = true;
        sfgpu_system *s = new sfgpu_system();
        s->stream = b->stream;
        rc = s->setup(&descs[i], false);
        if (!rc && (s->nseg > kResMax || s->nclass > kResMax)) rc = SFGPU_ERR_UNSUPPORTED;   // site_residual registers
        if (rc) { delete s; break; }
        b->sys.push_back(s);
        b->offset[i] = b->total;
        b->total += (long long)s->nvar;
        maxM = std::max(maxM, s->M);
    }
    if (rc) { delete b; return rc; }
    configure_group(b);
    // chain storage: the engine keeps a 1D chain in slices of its own, everything
    // else in d_gi
    for (auto *s : b->sys)
        if (!rc && !(b->grouped && s->H.L.grad == 1)) rc = s->alloc_chains();
    std::vector<const int *> chains(n);
    if (!rc) rc = upload_tables(b, &chains);
    if (rc) { delete b; return rc; }
    // concatenated iteration variables and per-instance DIIS work
    if ((rc = balloc(b, (void **)&b->d_xall, sizeof(double) * b->total))) { delete b; return rc; }
    b->desc_h.resize(n);
    for (int i = 0; i < n && !rc; i++) {
        sfgpu_system *s = b->sys[i];
        InstDesc &I = b->desc_h[i];
        fill_inst_desc(s, &I);
        s->point_chains(chains[i], &I);
        {   // force ensembles: step weights per molecule
            std::vector<sfk::ForceW> fw(2 * s->nmol);
            I.fmask = 0;
            for (int q = 0; q < s->nmol; q++)
                if (s->mols[q].force != 0) {
                    I.fmask |= 1 << q;
                    fw[2 * q] = force_weights(s->H.L, s->mols[q].force);
                    fw[2 * q + 1] = force_weights(s->H.L, -s->mols[q].force);
                }
            sfk::ForceW *dfw = nullptr;
            if (I.fmask) {
                if ((rc = balloc(b, (void **)&dfw, sizeof(sfk::ForceW) * fw.size()))) break;
                if (cudaMemcpy(dfw, fw.data(), sizeof(sfk::ForceW) * fw.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
                    rc = SFGPU_ERR_CUDA;
                    break;
                }
            }
            I.fw = dfw;
        }
        const size_t iv = s->nvar;
        I.x = b->d_xall + b->offset[i];
        if ((rc = balloc(b, (void **)&I.x0, sizeof(double) * iv)) || (rc = balloc(b, (void **)&I.g, sizeof(double) * iv)) ||
            (rc = balloc(b, (void **)&I.XR, sizeof(double) * iv * m)) || (rc = balloc(b, (void **)&I.XX0, sizeof(double) * iv * m)))
            break;
    }
    if (!rc) rc = balloc(b, (void **)&b->d_desc, sizeof(InstDesc) * n);
    if (!rc) rc = balloc(b, (void **)&b->d_queue, sizeof(int));
    if (!rc) rc = balloc(b, (void **)&b->d_status, sizeof(int) * n);
    if (!rc) rc = balloc(b, (void **)&b->d_iters, sizeof(int) * n);
    if (!rc) rc = balloc(b, (void **)&b->d_err, sizeof(double) * n);
    if (rc) { delete b; return rc; }
    // threads per block by the largest lattice (timed on the 2D cylinder and
    // on the uneven 1D sweep, where 384 beat 256 by 4.5 % and 32..128 lost)
    b->block = maxM >= 4096 ? 1024 : (maxM >= 1024 ? 512 : (maxM >= 384 ? 384 : 256));
    if ((rc = configure_stage(b, true))) { delete b; return rc; }
    if ((rc = sfgpu_after_setup(b->stream))) { delete b; return rc; }
    *out = b;
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_destroy(sfgpu_batch *b) {
    if (!b) return SFGPU_OK;
    cudaStreamSynchronize(b->stream);
    delete b;
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_info(sfgpu_batch *b, int *n, long long *total_nvar, long long *offsets) {
    if (!b) return SFGPU_ERR_INVALID;
    if (n) *n = (int)b->sys.size();
    if (total_nvar) *total_nvar = b->total;
    if (offsets) for (size_t i = 0; i < b->sys.size(); i++) offsets[i] = b->offset[i];
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_set_stream(sfgpu_batch *b, void *stream) {
    if (!b) return SFGPU_ERR_INVALID;
    SFGPU_CUDA_TRY(cudaStreamSynchronize(b->stream));
    if (b->own_stream) cudaStreamDestroy(b->stream);
    b->own_stream = false;
    b->stream = (cudaStream_t)stream;
    for (auto *s : b->sys) s->stream = b->stream;
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_cluster(sfgpu_batch *b, int *blocks, int *threads) {
    if (!b) return SFGPU_ERR_INVALID;
    if (blocks) *blocks = b->grouped ? b->shape.C : 0;
    if (threads) *threads = b->grouped ? b->shape.threads : b->block;
    return SFGPU_OK;
}

// Launch shape of the persistent kernel: threads per block (32..1024, a
// multiple of 32) and whether instances stage G (and the 1D slices) in
// shared memory.  By default 1024/512/256 threads by lattice size and
// staging on.  Batches of the cluster engine keep the engine's own shape.
extern "C" int sfgpu_batch_set_launch(sfgpu_batch *b, int threads, int stage) {
    if (!b || threads < 32 || threads > 1024 || threads % 32) return SFGPU_ERR_INVALID;
    SFGPU_CUDA_TRY(cudaStreamSynchronize(b->stream));
    b->block = threads;
    return configure_stage(b, stage != 0);
}

// Load the concatenated initial guesses (host) into the device iterate.
extern "C" int sfgpu_batch_load(sfgpu_batch *b, const double *x) {
    if (!b || !x) return SFGPU_ERR_INVALID;
    SFGPU_CUDA_TRY(cudaMemcpyAsync(b->d_xall, x, sizeof(double) * b->total, cudaMemcpyHostToDevice, b->stream));
    SFGPU_CUDA_TRY(cudaStreamSynchronize(b->stream));
    return SFGPU_OK;
}

// Solve every instance by Pure_DIIS starting from the device-resident
// iterate: one persistent kernel launch, queued asynchronously on the batch
// stream and bracketed by CUDA events (sfgpu_batch_kernel_ms).
extern "C" int sfgpu_batch_solve_resident(sfgpu_batch *b, double tol, int maxit, double eta) {
    if (!b || maxit < 0 || !(eta > 0)) return SFGPU_ERR_INVALID;
    const int n = (int)b->sys.size();
    cudaStream_t st = b->stream;
    SFGPU_CUDA_TRY(cudaMemsetAsync(b->d_queue, 0, sizeof(int), st));
    int dev = 0, nsm = 148;
    SFGPU_CUDA_TRY(cudaGetDevice(&dev));
    SFGPU_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int per_sm = 1;
    SFGPU_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel(b), b->block, b->stage_bytes));
    int grid = std::max(1, std::min(n, nsm * std::max(1, per_sm)));
    if (!b->ev0) {
        SFGPU_CUDA_TRY(cudaEventCreate(&b->ev0));
        SFGPU_CUDA_TRY(cudaEventCreate(&b->ev1));
    }
    SFGPU_CUDA_TRY(cudaEventRecord(b->ev0, st));
    if (b->grouped) {
        const int rc = group_diis(b->shape, b->d_desc, n, b->clusters, b->d_queue, b->m, eta, tol, maxit, b->d_status,
                                  b->d_iters, b->d_err, st);
        if (rc) return rc;
        SFGPU_CUDA_TRY(cudaEventRecord(b->ev1, st));
        return SFGPU_OK;
    }
    batch_kernel(b)<<<grid, b->block, b->stage_bytes, st>>>(b->d_desc, n, b->d_queue, b->m, eta, tol, maxit,
                                                  b->d_status, b->d_iters, b->d_err);
    SFGPU_CUDA_TRY(cudaGetLastError());
    SFGPU_CUDA_TRY(cudaEventRecord(b->ev1, st));
    return SFGPU_OK;
}

// Copy out the per-instance results (and the iterates when x != NULL).
extern "C" int sfgpu_batch_results(sfgpu_batch *b, double *x, int *status, int *iterations, double *errors) {
    if (!b) return SFGPU_ERR_INVALID;
    const int n = (int)b->sys.size();
    cudaStream_t st = b->stream;
    if (x) SFGPU_CUDA_TRY(cudaMemcpyAsync(x, b->d_xall, sizeof(double) * b->total, cudaMemcpyDeviceToHost, st));
    std::vector<int> s_h(n), it_h(n);
    std::vector<double> e_h(n);
    SFGPU_CUDA_TRY(cudaMemcpyAsync(s_h.data(), b->d_status, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    SFGPU_CUDA_TRY(cudaMemcpyAsync(it_h.data(), b->d_iters, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    SFGPU_CUDA_TRY(cudaMemcpyAsync(e_h.data(), b->d_err, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
    SFGPU_CUDA_TRY(cudaStreamSynchronize(st));
    for (int i = 0; i < n; i++) {
        if (status) status[i] = s_h[i];
        if (iterations) iterations[i] = it_h[i];
        if (errors) errors[i] = e_h[i];
    }
    return SFGPU_OK;
}

extern "C" int sfgpu_batch_kernel_ms(sfgpu_batch *b, double *ms) {
    if (!b || !b->ev0) return SFGPU_ERR_INVALID;
    SFGPU_CUDA_TRY(cudaEventSynchronize(b->ev1));
    float v = 0;
    SFGPU_CUDA_TRY(cudaEventElapsedTime(&v, b->ev0, b->ev1));
    *ms = v;
    return SFGPU_OK;
}

// Host convenience: load guesses x_in, solve, read back the iterates into
// x_out (may be NULL) and the per-instance results.
extern "C" int sfgpu_batch_solve(sfgpu_batch *b, const double *x_in, double *x_out, double tol, int maxit,
                                 double eta, int *status, int *iterations, double *errors) {
    if (!b || !x_in) return SFGPU_ERR_INVALID;
    cudaStream_t st = b->stream;
    SFGPU_CUDA_TRY(cudaMemcpyAsync(b->d_xall, x_in, sizeof(double) * b->total, cudaMemcpyHostToDevice, st));
    int rc = sfgpu_batch_solve_resident(b, tol, maxit, eta);
    if (rc) return rc;
    return sfgpu_batch_results(b, x_out, status, iterations, errors);
}

// results of instance i after a solve (its last residual evaluation)
extern "C" int sfgpu_batch_get_phi(sfgpu_batch *b, int inst, int seg, double *phi) {
    if (!b || inst < 0 || inst >= (int)b->sys.size()) return SFGPU_ERR_INVALID;
    sfgpu_system *s = b->sys[inst];
    if (seg < 0 || seg >= s->nseg) return SFGPU_ERR_INVALID;
    SFGPU_CUDA_TRY(cudaMemcpyAsync(phi, s->d_phi[seg], sizeof(double) * s->M, cudaMemcpyDeviceToHost, b->stream));
    SFGPU_CUDA_TRY(cudaStreamSynchronize(b->stream));
    return SFGPU_OK;
}
