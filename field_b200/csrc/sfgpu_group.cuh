// sfgpu_group.cuh -- one first-order 1D or 2D system evaluated, or iterated
// to convergence, by ONE thread-block cluster in one launch.
//
// A chain of N segments is 2N dependent steps over a lattice that fits on
// chip, so a launch per step leaves the chip waiting on launches.  Here the
// cluster keeps the running propagator slice in shared memory (2D) or
// registers (1D) for the whole chain, G and phi of the running segment in
// registers, and streams only the stored forward slices; a step costs an
// exchange of edge rows between neighbouring blocks (2D) or two warp shuffles
// (1D).  Everything else of a residual evaluation (segment weights,
// normalisation, contact averages) and of Pure_DIIS runs in the same launch,
// with cluster barriers between the phases.
//
// What bounds it is latency, not traffic.  Measured on a B200 against the
// launch-per-step path (microseconds; both builds in turn on one box):
//   residual, 1D n = 100, N = 100            222 -> 26.6  (0.09 a step, of which 0.045
//                                                          are the shuffle and the step's
//                                                          six dependent FP64 operations)
//   residual, 2D cylinder 128 x 128, N = 40  335 -> 71    (0.43 a step)
//   Pure_DIIS, 1D n = 200, N = 200         40053 -> 3067
//   Pure_DIIS, 2D cylinder 128 x 128       18289 -> 4121
// Of an issued instruction's 11 cycles in the 2D residual 2.6 are barriers, 2.1
// fixed latencies, 1.7 loads and 1.2 instruction fetches.
//
// Every value is formed by the operations, in the order, of the
// single-system kernels (stencil1, finalize_phi, residual) and lnGN sums run
// over the same 256-element trees, so a residual is bit-identical to the
// launch-per-step path.
#pragma once
#include "sfgpu_group.h"

namespace sfg {
using sfb::InstDesc;
using sfb::IMol;
using sfk::MolScal;

constexpr int kMaxCluster = 16;
constexpr int kHist = sfb::kMaxHist;
constexpr int kVals = kHist + 2;

struct GShared {
    double red[32 * kVals];                 // per-warp partial sums
    double part[kMaxCluster][kVals];        // block partial sums by rank (written by every block)
    double val[kVals];
    MolScal scal[sfb::kMaxMol];
    double phib[SFGPU_MAX_SEG], chib[SFGPU_MAX_SEG];
    double gram[kHist * kHist], A[kHist * kHist], Q[kHist * kHist], coef[kHist], work[kHist];
    int pos[kHist];
    int inst;
    unsigned long long mbar[2];             // halo rows arrived, by buffer of the running slice
};

// ---- the group: the blocks of one cluster ---------------------------------
struct Grp {
    int rank, size;      // block in the cluster, blocks
    int gt, gn;          // thread in the cluster, threads
};
__device__ __forceinline__ void cl_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { __syncwarp(); asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void gsync(const Grp &g) {
    if (g.size == 1) { __syncthreads(); return; }
    cl_arrive();
    cl_wait();
}
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// shared-memory address of block `rank` that corresponds to this block's `a`
__device__ __forceinline__ uint32_t peer(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t a, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// remote store that completes 8 bytes of transaction on the peer's barrier
__device__ __forceinline__ void st_async(uint32_t a, double v, uint32_t mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a), "d"(v), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
// waits for the phase of the given parity; false when the (generous) limit of
// tries ran out, which only a lost peer could cause
__device__ __forceinline__ bool mbar_wait(uint32_t b, uint32_t parity) {
    for (int i = 0; i < (1 << 22); i++) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\n"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(b), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}
// barriers of the halo rows: initialised once per kernel, before any use
__device__ __forceinline__ void group_init(GShared &sh) {
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&sh.mbar[0]));
        mbar_init(smem_u32(&sh.mbar[1]));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// Sums over the whole group in a fixed order: sh.val[slot[i]] = sum of v[i].
// Two calls in a row need a group barrier between them (every caller has
// one: the residual's phases lie between two sums).
template <int NMAX>
__device__ __forceinline__ void gsum(const double (&v)[NMAX], const int (&slot)[NMAX], int nv, const Grp &g,
                                     GShared &sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NMAX; i++) {
        if (slot[i] < 0) continue;
        double a = v[i];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sh.red[slot[i] * 32 + warp] = a;
    }
    __syncthreads();
    if (g.size == 1) {
        if (threadIdx.x < nv) {
            double a = 0;
            for (int w = 0; w < nw; w++) a += sh.red[threadIdx.x * 32 + w];
            sh.val[threadIdx.x] = a;
        }
        __syncthreads();
        return;
    }
    // thread (i, r): this block's partial sum i goes to block r
    for (int q = threadIdx.x; q < nv * g.size; q += blockDim.x) {
        const int i = q % nv, r = q / nv;
        double a = 0;
        for (int w = 0; w < nw; w++) a += sh.red[i * 32 + w];
        st_peer(peer(smem_u32(&sh.part[g.rank][i]), r), a);
    }
    gsync(g);
    if (threadIdx.x < nv) {
        double a = 0;
        for (int r = 0; r < g.size; r++) a += sh.part[r][threadIdx.x];
        sh.val[threadIdx.x] = a;
    }
    __syncthreads();
}

// ---- 2D chains -------------------------------------------------------------
// Block `rank` owns rows x0 .. x0 + mine - 1.  A thread owns a strip of J rows
// of one column: its values stay in registers, the two column neighbours and
// the rows above and below the strip are read from shared memory, so a site
// costs 2 + 2/J shared loads instead of 5.  Rows carry their two boundary
// columns (the copies SetBoundaries makes) and the block the two rows next
// to its own.  The owning block sends those with st.async, which completes
// transactions on an mbarrier of the receiving block: a block waits for its
// neighbours' rows only, and its stores of forward slices to global memory
// are not part of any step's release (a cluster barrier per step waited for
// them: 1.3 us a step at 128 x 128 instead of 0.6).
//
// Two buffers and an mbarrier each suffice: a block sends rows of slice t + 1
// only after it has received slice t's from its neighbours, whose edge threads
// have by then read slice t - 1's halo.
struct Rows2 {
    int R;                  // rows per block (the last blocks may own fewer)
    int x0, mine;           // first row (1-based) and number of rows of this block
};
__device__ __forceinline__ Rows2 rows_of(const DLat &L, const Grp &g) {
    Rows2 q;
    const int nx = L.Md[0] - 2;
    q.R = (nx + g.size - 1) / g.size;
    q.x0 = g.rank * q.R + 1;
    q.mine = max(0, min(q.R, nx - g.rank * q.R));
    return q;
}
// a thread's strip
template <int J>
struct Strip {
    int x, k, valid, MY, site;   // first row, column, rows that exist, lattice row width, first site
    __device__ __forceinline__ Strip(const DLat &L, const Rows2 &q) {
        const int ny = L.Md[1] - 2, s = threadIdx.x / ny;
        MY = L.Md[1];
        k = threadIdx.x - s * ny + 1;
        x = q.x0 + s * J;
        valid = max(0, min(J, q.mine - s * J));
        site = x * MY + k;
    }
};

extern __shared__ double2 g_sm2[];      // the kernels' dynamic shared memory
__device__ __forceinline__ double *dyn_smem() { return reinterpret_cast<double *>(g_sm2); }

// kFull: every strip of the block has all its J rows
template <int J, bool kCyl, bool kFull>
struct Chain2 {
    Strip<J> st;
    int src, dst;           // the strip's first site in the buffer a step reads / writes
    int PW;
    // where the strip's values are copies or halo rows: a boundary column
    // (offset from the site, 0 for none), and the block and barrier that take
    // the first / last row (0 for none); `many`: more than that (rows or
    // columns that several boundaries copy), taken from cols and push
    int col;
    uint32_t pa0, pb0, pa1, pb1;
    bool many;
    int cols[2];
    uint32_t push;          // 4 bits per row: 1 previous block, 2 next block, 4 block 0's upper, 8 the last block's lower halo
    uint32_t pa[4], pb[4];
    uint32_t po;            // byte offset of the written buffer, 0 or a buffer's size
    bool edge;              // reads a halo row another block sends
    uint32_t mbar, expect;  // this block's barriers; bytes it receives per step
    uint32_t parity;        // bit b: parity of barrier b's current phase
    int left;               // steps left in the sweep
    double l1, l0;
    static constexpr bool kLamReg = kCyl && J <= 4;     // lambda of the strip's rows in registers, else in shared memory
    static constexpr int kG = J < 4 ? J : 4;            // rows whose neighbours are loaded at a time
    double lmr[kLamReg ? J : 1], lpr[kLamReg ? J : 1];
    int lam, lamrows;       // shared memory: lambda- of the strip's rows, lambda+ lamrows further
    double v[J], g[J], ph[J], gf[J];

    __device__ __forceinline__ Chain2(const DLat &L, const Rows2 &q, const Grp &gr, GShared &sh)
        : st(L, q) {
        const int ny = L.Md[1] - 2, nx = L.Md[0] - 2;
        PW = st.MY;
        const int bufsz = (q.R + 2) * PW;
        l1 = L.l1;
        l0 = 1 - 4 * L.l1;
        const int i0 = st.x - q.x0;
        const uint32_t b0 = smem_u32(dyn_smem()), m0 = smem_u32(&sh.mbar[0]);
        src = (i0 + 1) * PW + st.k;
        dst = src + bufsz;
        po = 8u * bufsz;
        lam = 2 * bufsz + i0;
        lamrows = q.R;
        if (kLamReg) {
#pragma unroll
            for (int j = 0; j < J; j++) {
                lmr[j] = (j < st.valid) ? L.lam_m[st.x + j] : 0.0;
                lpr[j] = (j < st.valid) ? L.lam_p[st.x + j] : 0.0;
            }
        }
        cols[0] = (st.k == L.map_lo[1]) ? -st.k : 0;
        cols[1] = (st.k == L.map_hi[1]) ? PW - 1 - st.k : 0;
        const int lastb = (nx + q.R - 1) / q.R - 1;             // last block that owns rows
        const int lastrows = nx - lastb * q.R;
        mbar = m0;
        const int to[4] = {max(gr.rank - 1, 0), min(gr.rank + 1, gr.size - 1), 0, lastb};
        const uint32_t ha[4] = {b0 + 8u * ((q.R + 1) * PW + st.k), b0 + 8u * st.k, b0 + 8u * st.k,
                                b0 + 8u * ((lastrows + 1) * PW + st.k)};
#pragma unroll
        for (int e = 0; e < 4; e++) { pa[e] = peer(ha[e], to[e]); pb[e] = peer(m0, to[e]); }
        push = 0;
        pa0 = pb0 = pa1 = pb1 = 0;
        int n0 = 0, n1 = 0, other = 0;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const int x = st.x + j;
            uint32_t p = 0;
            if (j < st.valid) {
                if (gr.rank > 0 && x == q.x0) p |= 1;
                if (gr.rank < lastb && x == q.x0 + q.mine - 1) p |= 2;
                if (x == L.map_lo[0]) p |= 4;
                if (x == L.map_hi[0]) p |= 8;
            }
            push |= p << (4 * j);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (!((p >> e) & 1)) continue;
                if (j == 0 && n0 == 0) { pa0 = pa[e]; pb0 = pb[e]; n0++; }
                else if (j == J - 1 && n1 == 0) { pa1 = pa[e]; pb1 = pb[e]; n1++; }
                else other++;
            }
        }
        col = cols[0] ? cols[0] : cols[1];
        many = other || (cols[0] && cols[1]);
        if (many) { pa0 = pa1 = 0; col = 0; }
        // halo rows that come from other blocks (or from this one's own st.async)
        int in = 0;
        if (q.mine > 0) {
            if (gr.rank > 0 || L.map_lo[0] > 0) in++;
            if (gr.rank < lastb || L.map_hi[0] <= nx) in++;
        }
        expect = 8u * ny * in;
        edge = st.valid > 0 && in > 0 && (i0 == 0 || i0 + st.valid == q.mine);
    }
    __device__ __forceinline__ bool row_in(int j) const { return kFull ? st.valid > 0 : j < st.valid; }
    // before a sweep of n steps, the first from buffer 0 to buffer 1; one
    // thread arms the barriers
    __device__ __forceinline__ void begin(int n) {
        left = n;
        if (po == 0) turn();
        if (threadIdx.x == 0 && expect) {
            if (n > 0) mbar_expect(mbar + 8, expect);
            if (n > 1) mbar_expect(mbar, expect);
        }
    }
    __device__ __forceinline__ void turn() {
        const int t = src;
        const int bufsz = dst > src ? dst - src : src - dst;
        src = dst;
        dst = t;
        po = po ? 0u : 8u * bufsz;
    }
    // one step: reads the src buffer (and v), leaves the new values in v and dst
    __device__ __forceinline__ void step() {
        if (st.valid == 0) return;
        const double *s = dyn_smem() + src;
        double *d = dyn_smem() + dst;
        double old = s[-PW];                              // the row above, before this step
        const double below = s[(kFull ? J : st.valid) * PW];
#pragma unroll
        for (int j0 = 0; j0 < J; j0 += kG) {
            double a[kG], c[kG], lm[kCyl ? kG : 1], lp[kCyl ? kG : 1];
#pragma unroll
            for (int u = 0; u < kG; u++) {
                const int j = j0 + u;
                a[u] = c[u] = 0;
                if (kFull || j < st.valid) { a[u] = s[j * PW - 1]; c[u] = s[j * PW + 1]; }
                if (kLamReg) { lm[u] = lmr[j]; lp[u] = lpr[j]; }
                else if (kCyl) {
                    // the table ends with the block's rows, the last strip may not
                    const bool in = kFull || j < st.valid;
                    lm[u] = in ? dyn_smem()[lam + j] : 0.0;
                    lp[u] = in ? dyn_smem()[lam + lamrows + j] : 0.0;
                }
            }
#pragma unroll
            for (int u = 0; u < kG; u++) {
                const int j = j0 + u;
                const double b = v[j], up = old;
                double dn = below;
                if (j + 1 < J) dn = (kFull || j + 1 < st.valid) ? v[j + 1] : below;
                if (kCyl) v[j] = g[j] * (b + lm[u] * (up - b) + lp[u] * (dn - b) + l1 * (a[u] + c[u] - b - b));
                else v[j] = g[j] * (l0 * b + l1 * (a[u] + c[u]) + l1 * (up + dn));
                old = b;
                if (kFull || j < st.valid) d[j * PW] = v[j];
            }
        }
        if (pa0) st_async(pa0 + po, v[0], pb0 + (po ? 8 : 0));
        if (pa1) st_async(pa1 + po, v[J - 1], pb1 + (po ? 8 : 0));
        if (col) {
#pragma unroll
            for (int j = 0; j < J; j++)
                if (row_in(j)) d[j * PW + col] = v[j];
        }
        if (many) {
#pragma unroll
            for (int j = 0; j < J; j++) {
                if (!row_in(j)) continue;
                if (cols[0]) d[j * PW + cols[0]] = v[j];
                if (cols[1]) d[j * PW + cols[1]] = v[j];
                const uint32_t p = (push >> (4 * j)) & 15;
                if (!p) continue;
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if ((p >> e) & 1) st_async(pa[e] + po, v[j], pb[e] + (po ? 8 : 0));
            }
        }
    }
    // after the step's other work: the written buffer is complete for this thread's reads
    __device__ __forceinline__ void settle() {
        __syncthreads();
        left--;
        if (expect) {
            const int d = po ? 1 : 0;
            if (edge || threadIdx.x == 0) {
                if (!mbar_wait(mbar + 8 * d, (parity >> d) & 1)) {
#pragma unroll
                    for (int j = 0; j < J; j++) v[j] = __longlong_as_double(0x7ff8000000000000LL);
                }
                if (threadIdx.x == 0 && left > 1) mbar_expect(mbar + 8 * d, expect);
            }
            parity ^= 1u << d;
        }
        turn();
    }
    // the strip's values of a lattice vector; p points at its first site
    __device__ __forceinline__ void load(double (&r)[J], const double *p) const {
#pragma unroll
        for (int j = 0; j < J; j++) {
            r[j] = row_in(j) ? *p : 0.0;
            p += PW;
        }
    }
    __device__ __forceinline__ void store(const double (&r)[J], double *p) const {
#pragma unroll
        for (int j = 0; j < J; j++) {
            if (row_in(j)) *p = r[j];
            p += PW;
        }
    }
};

// propagation and raw composition (sum of Gf Gb, before the division by G)
// of molecule m into its phi; the end-point distribution goes to I.ginv0.
// G of every segment is complete on interior sites of the whole lattice.
// parity: the halo barriers' phases, carried from chain to chain.
template <int J, bool kCyl, bool kFull>
__device__ __noinline__ void chain2d(const InstDesc &I, int m, const Grp &gr, GShared &sh, uint32_t &parity) {
    const IMol &o = I.mol[m];
    const DLat &L = I.L;
    const int M = I.M, N = o.N, sym = o.sym;
    const int *seg = o.seg, *runf = o.runf, *runb = o.runb;
    const Rows2 q = rows_of(L, gr);
    Chain2<J, kCyl, kFull> c(L, q, gr, sh);
    c.parity = parity;
    double *sm = dyn_smem();
    const int site = c.st.site, MY = c.st.MY, bufsz = (q.R + 2) * MY;
    if (kCyl) {
        double *lam = sm + 2 * bufsz;
        for (int i = threadIdx.x; i < q.mine; i += blockDim.x) {
            lam[i] = L.lam_m[q.x0 + i];
            lam[q.R + i] = L.lam_p[q.x0 + i];
        }
    }
    // the start slice with its boundary copies (surface layers 0); the other
    // buffer's entries that no step writes hold 0
    auto fill = [&](const double *G) {
        const int rows = (q.mine > 0) ? q.mine + 2 : 0;
        __syncthreads();                   // the last sweep's halo rows have arrived
        // a warp takes rows, its lanes the columns, four loads at a time
        for (int row = threadIdx.x >> 5; row < q.R + 2; row += blockDim.x >> 5) {
            const int x = lat_mapc(L, 0, min(q.x0 - 1 + row, L.Md[0] - 1));
            const bool in = row < rows && x >= 1 && x <= L.Md[0] - 2;
            for (int c0 = threadIdx.x & 31; c0 < MY; c0 += 128) {
                double e[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int col = c0 + 32 * u, y = lat_mapc(L, 1, col);
                    e[u] = (in && col < MY && y >= 1 && y <= L.Md[1] - 2) ? G[x * MY + y] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (c0 + 32 * u < MY) {
                        sm[row * MY + c0 + 32 * u] = e[u];
                        sm[bufsz + row * MY + c0 + 32 * u] = 0.0;
                    }
            }
        }
    };
    const double zero[J] = {};
    for (int a = 0; a < o.nused; a++) c.store(zero, o.phi[o.used[a]] + site);
    int held = seg[0];                     // segment whose G (and phi) the registers hold
    c.load(c.g, I.gseg[held] + site);
#pragma unroll
    for (int j = 0; j < J; j++) { c.v[j] = c.g[j]; c.ph[j] = 0; }
    fill(I.gseg[held]);
    double *gp = I.gi + site;              // the strip in the stored slice a step writes or reads
    c.store(c.v, gp);
    const int nf = sym ? N / 2 : N;        // forward slices
    // a symmetric chain runs on from its forward half; others start again at the other end
    const int sp0 = (N + 3) / 2, nback = sym ? N - sp0 + 1 : N - 1;
    c.begin(sym ? nf - 1 + N % 2 + nback : nf - 1);
    gsync(gr);
    for (int t = 1; t < nf;) {             // runs of equal segments
        const int sg = seg[t], e = min(runf[t], nf);
        if (sg != held) { c.load(c.g, I.gseg[sg] + site); held = sg; }
        for (; t < e; t++) {
            c.step();
            gp += M;
            c.store(c.v, gp);
            c.settle();
        }
    }
    int t = N - 2;                         // slice the next backward step composes with
    if (sym) {
        if (N % 2 == 1) {
            c.step();
#pragma unroll
            for (int j = 0; j < J; j++) c.ph[j] = (c.ph[j] + c.v[j] * c.v[j]) * 0.5;
            c.settle();
        }
        t = N - sp0;
    } else {
        const int sN = seg[N - 1];
        c.load(c.gf, gp);
        if (sN != held) { c.load(c.g, I.gseg[sN] + site); held = sN; }
        fill(I.gseg[sN]);
#pragma unroll
        for (int j = 0; j < J; j++) { c.v[j] = c.g[j]; c.ph[j] += c.g[j] * c.gf[j]; }
        c.begin(nback);
        gsync(gr);
    }
    gp = I.gi + site + (size_t)t * M;
    c.load(c.gf, gp);
    while (t >= 0) {
        const int sg = seg[t], e = sym ? -1 : runb[t];
        if (sg != held) {
            c.store(c.ph, o.phi[held] + site);
            c.load(c.ph, o.phi[sg] + site);
            c.load(c.g, I.gseg[sg] + site);
            held = sg;
        }
        for (; t > e; t--) {
            c.step();
#pragma unroll
            for (int j = 0; j < J; j++) c.ph[j] = c.ph[j] + c.v[j] * c.gf[j];
            if (t > 0) { gp -= M; c.load(c.gf, gp); }
            c.settle();
        }
    }
    c.store(c.ph, o.phi[held] + site);
    c.store(c.v, I.ginv0 + site);
    parity = c.parity;
}

// ---- 1D chains -------------------------------------------------------------
// A warp keeps 32 * kJ1 consecutive positions in registers, kJ1 per lane, so a
// step exchanges one value with each neighbour lane and needs no barrier.
// Position 0 is the first register of some lane of warp 0 and position n + 1
// lies in the last warp; G is 0 there, so a surface layer's value stays 0 and
// only mirrors need a rule.  Lattices wider than one warp are cut into runs of
// kOwn1 positions, with kHalo1 + 1 further ones below and kHalo1 - 1 above that a
// warp recomputes (position 0 has to be some lane's first register).  A step
// makes one more position at either end wrong, so after kHalo1 - 1 steps the
// warps exchange their values once through shared memory.
//
// One warp walks the chain alone, so a step is a latency: the loops are short
// and free of branches (an eight-fold unrolled form with a rule per boundary
// kind took 720 cycles a step, 120 instructions of which most waited for
// instruction fetches and branches).  kM2: some side is a mirror2.
template <bool kCurved, bool kM2>
struct Chain1 {
    int p0;                 // lattice position of the lane's first register
    int own;                // bit j: register j is the warp's own
    int jhi;                // register at position n of an upper mirror, or -1
    bool lom, lo2, hi2;     // the first register is position 0 below a mirror; mirror2 below / above
    double l1;
    double lm[kCurved ? kJ1 : 1], lp[kCurved ? kJ1 : 1];
    double v[kJ1], g[kJ1], ph[kJ1];
    __device__ __forceinline__ Chain1(const DLat &L, int warp, int lane) {
        const int n = L.Md[0] - 2, nw = warps1d(n);
        p0 = (nw == 1 ? 0 : warp * kOwn1 - kHalo1) + lane * kJ1;
        lom = p0 == 0 && L.bc_lo[0] != SFGPU_BOUND_SURFACE;
        lo2 = L.bc_lo[0] == SFGPU_BOUND_MIRROR2;
        hi2 = L.bc_hi[0] == SFGPU_BOUND_MIRROR2;
        jhi = -1;
        own = 0;
        l1 = L.l1;
        const int first = (nw == 1) ? 1 : warp * kOwn1 + 1, last = (nw == 1) ? n : min(n, first + kOwn1 - 1);
#pragma unroll
        for (int j = 0; j < kJ1; j++) {
            const int p = p0 + j;
            if (p == n && L.bc_hi[0] != SFGPU_BOUND_SURFACE) jhi = j;
            if (p >= first && p <= last) own |= 1 << j;
            if (kCurved) {
                const bool in = p >= 1 && p <= n;
                lm[j] = in ? L.lam_m[p] : 0.0;
                lp[j] = in ? L.lam_p[p] : 0.0;
            }
        }
    }
    __device__ __forceinline__ void step() {
        const unsigned full = 0xffffffffu;
        const double left = __shfl_up_sync(full, v[kJ1 - 1], 1);      // lane 0's is not used: position 0 or a halo's end
        const double right = __shfl_down_sync(full, v[0], 1);
        double o[kJ1];
#pragma unroll
        for (int j = 0; j < kJ1; j++) {
            const double b = v[j];
            double a = (j == 0) ? left : v[j - 1];
            double c = (j == kJ1 - 1) ? right : v[j + 1];
            if (j == 1) a = lom ? (kM2 && lo2 ? v[2] : b) : a;
            c = (j == jhi) ? (kM2 && hi2 ? a : b) : c;
            if (kCurved) o[j] = g[j] * (b + lm[j] * (a - b) + lp[j] * (c - b));
            else o[j] = g[j] * (b + l1 * (a - b - b + c));
        }
#pragma unroll
        for (int j = 0; j < kJ1; j++) v[j] = o[j];
    }
    // values of positions 1..n (0 elsewhere) of a lattice vector
    __device__ __forceinline__ void load(double (&r)[kJ1], const double *p, int n) const {
#pragma unroll
        for (int j = 0; j < kJ1; j++) {
            const int z = p0 + j;
            r[j] = (z >= 1 && z <= n) ? p[z] : 0.0;
        }
    }
    __device__ __forceinline__ void store(const double (&r)[kJ1], double *p) const {
#pragma unroll
        for (int j = 0; j < kJ1; j++)
            if ((own >> j) & 1) p[p0 + j] = r[j];
    }
};

// as chain2d, on one block.  store: the stored slices, [slice][warp][lane][j],
// each lane reading back its own: in shared memory, or (ring != nullptr) in
// global memory, from where they return through a ring of kRing1 slices in
// shared memory by asynchronous copies issued kRing1 steps ahead.  line: 2
// lattice vectors in shared memory for the warps' exchanges.  Only the warps
// that hold positions take part and no block barrier is met inside.
template <bool kCurved, bool kM2>
__device__ __noinline__ void chain1d(const InstDesc &I, int m, double *line, double *store, double *ring) {
    const IMol &o = I.mol[m];
    const DLat &L = I.L;
    const int N = o.N, n = L.Md[0] - 2, nw = warps1d(n), sym = o.sym;
    const int *seg = o.seg;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= nw) return;
    Chain1<kCurved, kM2> c(L, warp, lane);
    const size_t SL = slice1d(n);
    store += ((size_t)warp * 32 + lane) * kJ1;
    ring += ring ? ((size_t)warp * 32 + lane) * kJ1 : 0;
    double *sp = store;                     // slice the next put writes
    auto put = [&]() {
        double2 *d = reinterpret_cast<double2 *>(sp);
        d[0] = make_double2(c.v[0], c.v[1]);
        d[1] = make_double2(c.v[2], c.v[3]);
        sp += SL;
    };
    auto get = [&](double (&r)[kJ1], const double *p) {
        const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
        r[0] = a.x; r[1] = a.y; r[2] = b.x; r[3] = b.y;
    };
    int held = seg[0], lb = 0;
    int since = nw > 1 ? 0 : -(1 << 30);    // steps since the halos were exchanged
    auto exchange = [&]() {
        double *l = line + lb * (n + 2);
        lb ^= 1;
        c.store(c.v, l);
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"r"(nw * 32) : "memory");
#pragma unroll
        for (int j = 0; j < kJ1; j++) {
            const int z = c.p0 + j;
            if (!((c.own >> j) & 1) && z >= 1 && z <= n) c.v[j] = l[z];
        }
        since = 0;
    };
    auto step = [&]() {
        if (since == kHalo1 - 1) exchange();
        since++;
        c.step();
    };
    const double zero[kJ1] = {};
    for (int a = 0; a < o.nused; a++) c.store(zero, o.phi[o.used[a]]);
    c.load(c.g, I.gseg[held], n);
#pragma unroll
    for (int j = 0; j < kJ1; j++) { c.v[j] = c.g[j]; c.ph[j] = 0; }
    put();
    const int nf = sym ? N / 2 : N;
    for (int t = 1; t < nf;) {              // runs of equal segments
        const int sg = seg[t], e = min(o.runf[t], nf);
        if (sg != held) { c.load(c.g, I.gseg[sg], n); held = sg; }
        for (; t < e; t++) {
            step();
            put();
        }
    }
    // backward: slice `last` first, then down to 0
    int last, sg;
    if (sym) {
        if (N % 2 == 1) {
            step();
#pragma unroll
            for (int j = 0; j < kJ1; j++) c.ph[j] = (c.ph[j] + c.v[j] * c.v[j]) * 0.5;
        }
        last = N - (N + 3) / 2;
    } else {
        const int sN = seg[N - 1];
        if (sN != held) { c.load(c.g, I.gseg[sN], n); held = sN; }
        double gf[kJ1];
        get(gf, store + (size_t)(N - 1) * SL);
#pragma unroll
        for (int j = 0; j < kJ1; j++) { c.v[j] = c.g[j]; c.ph[j] += c.g[j] * gf[j]; }
        if (nw > 1) since = 0;
        last = N - 2;
    }
    auto run = [&](int t) {                 // position t's segment into the registers; where its run ends
        sg = seg[t];
        if (sg != held) {
            c.store(c.ph, o.phi[held]);
            c.load(c.ph, o.phi[sg], n);
            c.load(c.g, I.gseg[sg], n);
            held = sg;
        }
        return sym ? -1 : o.runb[t];
    };
    const double *gp = store + (size_t)last * SL;
    if (!ring) {
        double gf[kJ1];
        get(gf, gp);
        for (int t = last; t >= 0;) {
            const int e = run(t);
            for (; t > e; t--) {
                step();
#pragma unroll
                for (int j = 0; j < kJ1; j++) c.ph[j] = c.ph[j] + c.v[j] * gf[j];
                gp -= (t > 0) ? SL : 0;
                get(gf, gp);
            }
        }
    } else {
        auto issue = [&](int t, int slot) {  // slice t (gp) into the ring, always one group
            if (t >= 0) {
                double *d = ring + (size_t)slot * SL;
                __pipeline_memcpy_async(d, gp, 16);
                __pipeline_memcpy_async(d + 2, gp + 2, 16);
                gp -= SL;
            }
            __pipeline_commit();
        };
        for (int q = 0; q < kRing1; q++) issue(last - q, q);
        int slot = 0;
        for (int t = last; t >= 0;) {
            const int e = run(t);
            for (; t > e; t--) {
                step();
                __pipeline_wait_prior(kRing1 - 1);
                double gf[kJ1];
                get(gf, ring + (size_t)slot * SL);
#pragma unroll
                for (int j = 0; j < kJ1; j++) c.ph[j] = c.ph[j] + c.v[j] * gf[j];
                issue(t - kRing1, slot);
                slot = (slot + 1) & (kRing1 - 1);
            }
        }
        __pipeline_wait_prior(0);
    }
    c.store(c.ph, o.phi[held]);
    c.store(c.v, I.ginv0);
}

// One copy of the logarithm and of the exponential in a kernel whose phases run
// once an evaluation: such code is bound by instruction fetches, and the
// functions are called from a dozen places.
__device__ __noinline__ double log1(double v) { return log(v); }
__device__ __noinline__ double exp1(double v) { return exp(v); }

// ---- lnGN sums -------------------------------------------------------------
// Partial sums of w * g over 256-element blocks of the lattice vector, each in
// the order of wsum_partial's shared-memory tree, into part[0 .. ceil(M/256)).
__device__ __forceinline__ void wsum_blocks(int M, const double *g, const double *w, double *part, const Grp &gr) {
    const int lane = threadIdx.x & 31, nb = (M + 255) / 256;
    for (int b = gr.gt >> 5; b < nb; b += gr.gn >> 5) {
        double e[8], ww[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int r = min(b * 256 + q * 32 + lane, M - 1);
            ww[q] = w[r];
            e[q] = g[r];
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const bool in = b * 256 + q * 32 + lane < M && ww[q] != 0;
            e[q] = in ? 0.0 + ww[q] * e[q] : 0.0;
        }
#pragma unroll
        for (int s = 4; s > 0; s >>= 1)
#pragma unroll
            for (int q = 0; q < s; q++) e[q] += e[q + s];
        double a = e[0];
        for (int s = 16; s > 0; s >>= 1) a += __shfl_down_sync(0xffffffffu, a, s);
        if (lane == 0) part[b] = a;
    }
}

// mol_scalars (sfgpu_kernels.cuh) for a first-order molecule
__device__ __noinline__ MolScal mol_scalars_of(const IMol &o, const MolScal *scal, int m, int nmol, double wsum) {
    MolScal s;
    s.lngn = log1(wsum);
    double phib = o.phibulk;
    if (o.solvent) {
        phib = 1.0;
        for (int q = 0; q < nmol; q++)
            if (q != m) phib -= scal[q].phibulk;
    }
    const double N = (double)o.N;
    const double gn = exp1(s.lngn);
    if (o.freedom == SFGPU_MOL_RESTRICTED) {
        if (o.type == 0) { s.lnc = log1(o.theta) - s.lngn; s.norm = o.theta / gn; }
        else {
            s.lnc = log1(o.theta) - s.lngn - log1(1.0 * o.N);
            s.norm = (o.sym ? 2 * o.theta / N : o.theta / N) / gn;
        }
        s.phibulk = o.theta / gn;
    } else {
        s.phibulk = phib;
        if (o.type == 0) { s.lnc = log1(phib); s.norm = phib; }
        else { s.lnc = log1(phib / N); s.norm = o.sym ? 2 * phib / N : phib / N; }
    }
    if (o.pinned) s.phibulk = 0;
    return s;
}

// lnGN sums, molecule scalars and the bulk terms once every chain's
// end-point distribution has been summed into I.wpart
__device__ inline void scalars_group(const InstDesc &I, const Grp &gr, GShared &sh) {
    const int nb = (I.M + 255) / 256;
    // a warp per molecule takes the sum over the partials, serially as
    // mol_scalars does: 32 at a time from its lanes
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int q = threadIdx.x >> 5; q < I.nmol; q += nw) {
        const double *p = I.wpart + (size_t)q * nb;
        double v = 0;
        for (int b = 0; b < nb; b += 128) {
            double e[4];
#pragma unroll
            for (int u = 0; u < 4; u++) e[u] = p[min(b + 32 * u + lane, nb - 1)];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                sh.red[(q & 15) * 32 + lane] = e[u];
                __syncwarp();
                if (lane == 0) {
                    const int n = min(32, nb - b - 32 * u);
#pragma unroll 8
                    for (int i = 0; i < n; i++) v += sh.red[(q & 15) * 32 + i];
                }
                __syncwarp();
            }
        }
        if (lane == 0) {
            sh.val[q] = v;
            if (q != I.solvent) sh.scal[q] = mol_scalars_of(I.mol[q], sh.scal, q, I.nmol, v);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        sh.scal[I.solvent] = mol_scalars_of(I.mol[I.solvent], sh.scal, I.solvent, I.nmol, sh.val[I.solvent]);
        for (int i = 0; i < I.nseg; i++) {
            double v = 0;
            for (int q = 0; q < I.nmol; q++) v += sh.scal[q].phibulk * I.frac[i * SFGPU_MAX_SEG + q];
            sh.phib[i] = v;
        }
        for (int c = 0; c < I.nclass; c++) {
            const int st = I.rep[c];
            double v = 0;
            for (int j = 0; j < I.nseg; j++) {
                const double xx = I.ct.chi[st * SFGPU_MAX_SEG + j];
                if (xx != 0) v += xx * sh.phib[j];
            }
            sh.chib[c] = v;
        }
        if (gr.rank == 0 && I.scal_out) {
            for (int q = 0; q < I.nmol; q++) I.scal_out[q] = sh.scal[q];
            for (int i = 0; i < I.nseg; i++) I.phib_out[i] = sh.phib[i];
            for (int c = 0; c < I.nclass; c++) I.chib_out[c] = sh.chib[c];
        }
    }
    __syncthreads();
}

// f of one site from its total volume fraction, contact averages (by segment)
// and G (by class): the sums of residual in sfgpu_kernels.cuh, in its order.
// Rolled loops over local arrays: short code, fetched once.
__device__ __noinline__ void put_residual(const InstDesc &I, const double *chib, double phit, const double *rho,
                                          const double *g, double *f) {
    const int ncl = I.nclass, nseg = I.nseg;
    double u[sfb::kResMax];
    double av = 0;
#pragma unroll 1
    for (int c = 0; c < ncl; c++) {
        const double *chi = I.ct.chi + I.rep[c] * SFGPU_MAX_SEG;
        double v = -log1(g[c]);
        double ci = 0;
#pragma unroll 1
        for (int i = 0; i < nseg; i++) {
            const double xx = chi[i];
            if (xx != 0) ci += xx * rho[i];
        }
        v -= ci / phit;
        v += chib[c];
        u[c] = v;
        av += v;
    }
    av /= ncl;
    const double t = -1.0 + 1.0 / phit;
#pragma unroll 1
    for (int c = 0; c < ncl; c++) f[c] = t + u[c] - av;
}

// f on a thread's strip; NS bounds the segment types and classes.  Every load of
// a site is issued before the first use (a segment that is not there or does
// not interact reads its neighbour in the list again).
template <int J, bool kCyl, int NS>
__device__ __noinline__ void sites_residual2d(const InstDesc &I, double *f, const Strip<J> &st, const double *chib) {
    const DLat &L = I.L;
    const int nseg = I.nseg, ncl = I.nclass, MY = st.MY;
    const int dl = (st.k == 1) ? L.map_lo[1] - 1 : -1, dr = (st.k == MY - 2) ? L.map_hi[1] - st.k : 1;
    const double l = L.l1chi;
    for (int j = 0; j < st.valid; j++) {
        const int x = st.x + j, z = st.site + j * MY;
        const int jj = I.jall[z];
        const int du = (lat_mapc(L, 0, x - 1) - x) * MY, dd = (lat_mapc(L, 0, x + 1) - x) * MY;
        const double lm = kCyl ? L.lam_m[x] : l, lp = kCyl ? L.lam_p[x] : l;
        double e[NS][5], g[NS];
#pragma unroll
        for (int i = 0; i < NS; i++) {
            const double *p = I.phi[min(i, nseg - 1)];
            e[i][0] = p[z];
            e[i][1] = p[z + dl];
            e[i][2] = p[z + dr];
            e[i][3] = p[z + du];
            e[i][4] = p[z + dd];
        }
#pragma unroll
        for (int c = 0; c < NS; c++) g[c] = I.gfull[I.rep[min(c, ncl - 1)]][z];
        double phit = 0, rho[NS];
#pragma unroll
        for (int i = 0; i < NS; i++) {
            const double b = e[i][0], a = e[i][1], c = e[i][2], u = e[i][3], d = e[i][4];
            if (i < nseg) phit += b;
            double v;
            if (kCyl) v = b + lp * (d - b) + lm * (u - b) + l * (a + c - b - b);
            else v = (1 - 2 * l - lm - lp) * b + l * (u + d) + l * (a + c);
            rho[i] = (i < nseg && ((I.need >> i) & 1)) ? v : 0.0;
        }
        if (jj >= 0) put_residual(I, chib, phit, rho, g, f + (size_t)jj * ncl);
    }
}

// ---- x -> f (SF_Solve::residuals, SF_Solve.cpp:647-651) ----------------------
// 2D: every phase runs on the strips of the chains, so a thread meets only
// its own values from G to the state profiles; neighbours' values are needed
// by the chains and by the contact averages.  Boundary entries (copies) of G
// and of the profiles are written for the readers after this kernel and read
// by nobody in it.
template <int J, bool kCyl>
__device__ inline void residual2d(const InstDesc &I, const double *x, double *f, const Grp &gr, GShared &sh,
                                  uint32_t &parity) {
    const DLat &L = I.L;
    const int M = I.M, nseg = I.nseg, nmol = I.nmol, ncl = I.nclass;
    const Rows2 q = rows_of(L, gr);
    const Strip<J> st(L, q);
    {
        int jx[J];
#pragma unroll
        for (int j = 0; j < J; j++) jx[j] = (j < st.valid) ? I.jall[st.site + j * st.MY] : -1;
        for (int i = 0; i < nseg; i++) {
            const int fr = I.freedom[i];
            if (fr == SFGPU_SEG_FROZEN) continue;
            const int cls = I.class_of[i];
            double xv[J];
#pragma unroll
            for (int j = 0; j < J; j++) xv[j] = (jx[j] >= 0) ? x[(size_t)jx[j] * ncl + cls] : 0.0;
            double *gf = I.gfull[i], *gs = I.gseg[i];
            const double *range = I.range[i];
#pragma unroll
            for (int j = 0; j < J; j++) {
                if (j >= st.valid) continue;
                const int z = st.site + j * st.MY;
                const double v = (jx[j] >= 0) ? exp1(-xv[j]) : 0.0;
                gf[z] = v;
                if (fr == SFGPU_SEG_PINNED) gs[z] = range[z] > 0 ? v : 0.0;
            }
        }
    }
    gsync(gr);
    const int nb = (M + 255) / 256;
    for (int m = 0; m < nmol; m++) {
        const IMol &o = I.mol[m];
        if (o.type != 0) {
            if (q.mine % J == 0) chain2d<J, kCyl, true>(I, m, gr, sh, parity);
            else chain2d<J, kCyl, false>(I, m, gr, sh, parity);
            gsync(gr);
        }
        wsum_blocks(M, o.type == 0 ? I.gseg[o.seg[0]] : I.ginv0, I.w_gn, I.wpart + (size_t)m * nb, gr);
        if (o.type != 0 && m + 1 < nmol) gsync(gr);        // ginv0 is the next chain's too
    }
    gsync(gr);
    scalars_group(I, gr, sh);
    for (int i = 0; i < nseg; i++) {
        if (I.freedom[i] == SFGPU_SEG_FROZEN) continue;
        const double *G = I.gseg[i];
        double acc[J];
#pragma unroll
        for (int j = 0; j < J; j++) acc[j] = 0;
        for (int m = 0; m < nmol; m++) {
            double *phi = I.mol[m].phi[i];
            if (!phi) continue;
            const bool mono = I.mol[m].type == 0;
            const double norm = sh.scal[m].norm;
            double p[J], g[J];
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int z = st.site + j * st.MY;
                g[j] = (j < st.valid) ? G[z] : 0.0;
                p[j] = (j < st.valid && !mono) ? phi[z] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < J; j++) {
                if (j >= st.valid) continue;
                const double v = (mono ? g[j] : (g[j] > 0 ? p[j] / g[j] : 0.0)) * norm;
                phi[st.site + j * st.MY] = v;
                acc[j] += v;
            }
        }
#pragma unroll
        for (int j = 0; j < J; j++)
            if (j < st.valid) I.phi[i][st.site + j * st.MY] = acc[j];
    }
    gsync(gr);
    // boundary copies, and f on the strips
    const int MX = L.Md[0], MY = L.Md[1];
    for (int e = gr.gt; e < 2 * (MX + MY); e += gr.gn) {
        // the first and last row, then the first and last column
        const int r = e < MY ? e : e < 2 * MY ? (MX - 1) * MY + e - MY : e < 2 * MY + MX ? (e - 2 * MY) * MY
                                                                                    : (e - 2 * MY - MX) * MY + MY - 1;
        const int t = I.smap[r];
        for (int i = 0; i < nseg; i++) {
            if (I.freedom[i] == SFGPU_SEG_FROZEN) continue;
            double *gf = I.gfull[i], *gs = I.gseg[i], *ph = I.phi[i];
            const int tx = t / st.MY, ty = t - tx * st.MY;
            const bool in = tx != 0 && tx != L.Md[0] - 1 && ty != 0 && ty != L.Md[1] - 1;
            gf[r] = in ? gf[t] : 0.0;
            if (gs != gf) gs[r] = in ? gs[t] : 0.0;
            ph[r] = in ? ph[t] : 0.0;
            for (int m = 0; m < nmol; m++) {
                double *p = I.mol[m].phi[i];
                if (p) p[r] = in ? p[t] : 0.0;
            }
        }
    }
    if (nseg <= 4 && ncl <= 4) sites_residual2d<J, kCyl, 4>(I, f, st, sh.chib);
    else sites_residual2d<J, kCyl, sfb::kResMax>(I, f, st, sh.chib);
}

// where a 1D system's arrays lie (localize1d)
struct Local1 {
    double *line, *store, *ring;   // exchange lines, stored slices and their ring (nullptr: they lie in shared memory)
    double *x, *g, *XR, *XX0;      // Pure_DIIS's vectors
    bool on;                       // the working arrays lie in shared memory
};
// 1D: one block; the descriptor's working arrays may lie in shared memory
template <bool kCurved>
__device__ inline void residual1d(const InstDesc &I, const double *x, double *f, const Grp &gr, GShared &sh,
                                  const Local1 &loc) {
    const DLat &L = I.L;
    const int M = I.M, nseg = I.nseg, nmol = I.nmol, ncl = I.nclass;
    for (int r = threadIdx.x; r < M; r += blockDim.x) {
        const int j = I.jall[r];
        for (int i = 0; i < nseg; i++) {
            if (I.freedom[i] == SFGPU_SEG_FROZEN) continue;
            const double v = (j >= 0) ? exp1(-x[(size_t)j * ncl + I.class_of[i]]) : 0.0;
            I.gfull[i][r] = v;
            if (I.freedom[i] == SFGPU_SEG_PINNED) I.gseg[i][r] = I.range[i][I.smap[r]] > 0 ? v : 0.0;
        }
    }
    __syncthreads();
    const int nb = (M + 255) / 256;
    for (int m = 0; m < nmol; m++) {
        const IMol &o = I.mol[m];
        if (o.type != 0) {
            if (L.bc_lo[0] == SFGPU_BOUND_MIRROR2 || L.bc_hi[0] == SFGPU_BOUND_MIRROR2)
                chain1d<kCurved, true>(I, m, loc.line, loc.store, loc.ring);
            else
                chain1d<kCurved, false>(I, m, loc.line, loc.store, loc.ring);
            __syncthreads();
        }
        wsum_blocks(M, o.type == 0 ? I.gseg[o.seg[0]] : I.ginv0, I.w_gn, I.wpart + (size_t)m * nb, gr);
        if (o.type != 0 && m + 1 < nmol) __syncthreads();   // ginv0 is the next chain's too
    }
    __syncthreads();
    scalars_group(I, gr, sh);
    // a boundary entry's profile is its mapped site's: formed there from the
    // same operands, so no barrier separates the copies
    for (int r = threadIdx.x; r < M; r += blockDim.x) {
        if (r == 0 || r == M - 1) continue;
        for (int i = 0; i < nseg; i++) {
            if (I.freedom[i] == SFGPU_SEG_FROZEN) continue;
            const double g = I.gseg[i][r];
            double acc = 0;
            for (int m = 0; m < nmol; m++) {
                double *phi = I.mol[m].phi[i];
                if (!phi) continue;
                const double v = ((I.mol[m].type == 0) ? g : (g > 0 ? phi[r] / g : 0.0)) * sh.scal[m].norm;
                phi[r] = v;
                acc += v;
                if (r == L.map_lo[0]) phi[0] = v;
                if (r == L.map_hi[0]) phi[M - 1] = v;
            }
            I.phi[i][r] = acc;
            if (r == L.map_lo[0]) I.phi[i][0] = acc;
            if (r == L.map_hi[0]) I.phi[i][M - 1] = acc;
            // surface layers: 0
            if (r == 1 && L.map_lo[0] == 0) {
                I.phi[i][0] = 0;
                for (int m = 0; m < nmol; m++) if (I.mol[m].phi[i]) I.mol[m].phi[i][0] = 0;
            }
            if (r == M - 2 && L.map_hi[0] == M - 1) {
                I.phi[i][M - 1] = 0;
                for (int m = 0; m < nmol; m++) if (I.mol[m].phi[i]) I.mol[m].phi[i][M - 1] = 0;
            }
        }
    }
    __syncthreads();
    const double l = L.l1chi;
    for (int z = threadIdx.x + 1; z < M - 1; z += blockDim.x) {
        const int jj = I.jall[z];
        if (jj < 0) continue;
        double phit = 0, rho[sfb::kResMax], g[sfb::kResMax];
#pragma unroll 1
        for (int i = 0; i < nseg; i++) {
            const double *p = I.phi[i];
            const double a = p[z - 1], b = p[z], c = p[z + 1];
            phit += b;
            double v;
            if (kCurved) v = b + L.lamc_p[z] * (c - b) + L.lamc_m[z] * (a - b);
            else v = b + l * (a - b - b + c);
            rho[i] = ((I.need >> i) & 1) ? v : 0.0;
        }
#pragma unroll 1
        for (int c = 0; c < ncl; c++) g[c] = I.gfull[I.rep[c]][z];
        put_residual(I, sh.chib, phit, rho, g, f + (size_t)jj * ncl);
    }
}

// ---- 1D systems in shared memory ---------------------------------------------
// A 1D system's working arrays are a few KB each, and every phase of an
// evaluation is one dependent pass over them: from shared memory a pass costs
// tens of cycles, from L2 hundreds.  The descriptor's pointers are redirected
// to shared memory where the arrays fit, and the profiles and segment weights
// written back when the kernel is done with the system.
// doubles of the exchange lines, an even number
__host__ __device__ inline size_t line1d(int n) { return (2 * (size_t)(n + 2) + 1) / 2 * 2; }
__host__ __device__ inline size_t local1d_doubles(int M, int nseg, int nonfrozen, int pinned, int molphis, int nmol) {
    return (size_t)M * (nonfrozen + pinned + nseg + molphis + 3) + (size_t)nmol * ((M + 255) / 256);
}
template <class T>
__device__ __forceinline__ void copy_in(T *dst, const T *src, long long n) {
    for (long long i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}
__device__ inline Local1 localize1d(InstDesc &I, const InstDesc *src, double *sm, size_t room, int m) {
    const int M = I.M, n = I.L.Md[0] - 2, nseg = I.nseg, nmol = I.nmol;
    Local1 q;
    q.line = sm;
    q.store = I.slices1;
    q.ring = sm + line1d(n);
    q.x = I.x; q.g = I.g; q.XR = I.XR; q.XX0 = I.XX0;
    size_t at = line1d(n) + kRing1 * slice1d(n);
    int nonfrozen = 0, pinned = 0, molphis = 0;
    size_t chain = 0;
    for (int i = 0; i < nseg; i++) {
        if (I.freedom[i] != SFGPU_SEG_FROZEN) nonfrozen++;
        if (I.freedom[i] == SFGPU_SEG_PINNED) pinned++;
    }
    for (int k = 0; k < nmol; k++) {
        molphis += I.mol[k].nused;
        const int N = I.mol[k].N;
        if (I.mol[k].type != 0) {
            const size_t c = (size_t)(I.mol[k].sym ? N / 2 : N) * slice1d(n);
            chain = c > chain ? c : chain;
        }
    }
    const size_t need = local1d_doubles(M, nseg, nonfrozen, pinned, molphis, nmol);
    q.on = at + need <= room;
    if (!q.on) return q;
    const InstDesc &G = *src;   // the global arrays
    __syncthreads();
    double *p = sm + at;
    auto take = [&](size_t k) { double *r = p; p += k; return r; };
    double *w = take(M), *end = take(M), *part = take((size_t)nmol * ((M + 255) / 256));
    int *ints = (int *)take(M);
    copy_in(w, G.w_gn, M);
    copy_in(ints, G.smap, M);
    copy_in(ints + M, G.jall, M);
    for (int i = 0; i < nseg; i++) {
        const bool fr = I.freedom[i] == SFGPU_SEG_FROZEN, pin = I.freedom[i] == SFGPU_SEG_PINNED;
        double *ph = take(M);
        double *gf = fr ? nullptr : take(M);
        double *gs = pin ? take(M) : gf;
        if (fr) copy_in(ph, G.phi[i], M);
        if (threadIdx.x == 0) { I.phi[i] = ph; I.gfull[i] = gf; I.gseg[i] = gs; }
    }
    for (int k = 0; k < nmol; k++)
        for (int a = 0; a < I.mol[k].nused; a++) {
            double *ph = take(M);
            if (threadIdx.x == 0) I.mol[k].phi[I.mol[k].used[a]] = ph;
        }
    if (threadIdx.x == 0) { I.w_gn = w; I.smap = ints; I.jall = ints + M; I.wpart = part; I.ginv0 = end; }
    size_t left = room - (size_t)(p - sm);
    if (chain <= left) {
        q.store = sm + room - chain;    // slices are 16-byte aligned: so is the end of the room
        q.ring = nullptr;
        left -= chain;
    }
    if (m > 0) {
        const size_t nv = (size_t)I.nvar;
        if (2 * nv <= left) {
            q.x = take(nv);
            q.g = take(nv);
            left -= 2 * nv;
            copy_in(q.x, G.x, I.nvar);
            if (2 * nv * m <= left) { q.XR = take(nv * m); q.XX0 = take(nv * m); }
        }
    }
    __syncthreads();
    return q;
}
__device__ inline void write_back1d(const InstDesc &I, const InstDesc *src, const Local1 &q, int m) {
    if (!q.on) return;
    const InstDesc &G = *src;
    __syncthreads();
    for (int i = 0; i < I.nseg; i++) {
        if (I.freedom[i] == SFGPU_SEG_FROZEN) continue;
        copy_in(G.phi[i], (const double *)I.phi[i], I.M);
        copy_in(G.gfull[i], (const double *)I.gfull[i], I.M);
        if (I.gseg[i] != I.gfull[i]) copy_in(G.gseg[i], (const double *)I.gseg[i], I.M);
        for (int k = 0; k < I.nmol; k++)
            if (I.mol[k].phi[i]) copy_in(G.mol[k].phi[i], (const double *)I.mol[k].phi[i], I.M);
    }
    if (m > 0 && q.x != G.x) copy_in(G.x, (const double *)q.x, I.nvar);
    __syncthreads();
}

// ---- DIIS coefficients --------------------------------------------------------
// c = A^-1 1 for the symmetric Gram matrix by eliminating the augmented system
// in one warp: per column one division a row and a rank-one update shared by
// the lanes, where the Jacobi rotations of diis_coeff_warp take n (n - 1) / 2
// serial square roots and divisions a sweep (m = 10: 400 k cycles a call; 8 k
// here).  The loops stay rolled on purpose: this runs once an iteration, and
// unrolled over registers it took 50 k cycles, nearly all of them instruction
// fetches.  A is n x n in shared memory, overwritten; c and w hold n values.
// Returns false, with c unset, when a pivot keeps less than 1e-14 of the terms
// it is the sum of: down to there the Gram matrix's own rounding limits either
// method alike, below it the stored steps are linearly dependent to rounding
// and the eigen-decomposition's pseudo-inverse decides.
__device__ __noinline__ bool coeff_ldl_warp(int n, double *A, double *c, double *w) {
    const int lane = threadIdx.x & 31;
    double mag = (lane < n) ? fabs(A[lane * n + lane]) : 0.0;   // of the terms of this row's pivot
    double rhs = 1.0;                       // row `lane` of the right-hand side
#pragma unroll 1
    for (int k = 0; k < n; k++) {
        const double piv = A[k * n + k];
        if (!(fabs(piv) > 1e-14 * __shfl_sync(0xffffffffu, mag, k))) return false;
        const double mul = (lane > k && lane < n) ? A[lane * n + k] / piv : 0.0;
        rhs -= mul * __shfl_sync(0xffffffffu, rhs, k);
        if (lane < n) {
            w[lane] = mul;
            mag += fabs(mul * A[k * n + lane]);
        }
        __syncwarp();
        // the trailing block: half a warp a row
        const int j = k + 1 + (lane & 15);
        if (j < n) {
            const double p = A[k * n + j];
#pragma unroll 1
            for (int i = k + 1 + (lane >> 4); i < n; i += 2) A[i * n + j] -= w[i] * p;
        }
        __syncwarp();
    }
#pragma unroll 1
    for (int k = n - 1; k >= 0; k--) {
        const double x = __shfl_sync(0xffffffffu, rhs, k) / A[k * n + k];
        if (lane == 0) c[k] = x;
        if (lane < k) rhs -= A[lane * n + k] * x;
    }
    __syncwarp();
    return true;
}

}  // namespace sfg
