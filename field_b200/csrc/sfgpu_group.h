// sfgpu_group.h -- host side of the cluster engine (sfgpu_group.cuh).
#pragma once
#include "sfgpu_batch.cuh"
#include "sfgpu_system.h"

namespace sfg {
// 1D chains: a warp's sites per lane, and its own ones; it recomputes kHalo1 + 1
// sites below them and kHalo1 - 1 above, which are right for as many steps.
// Stored slices are whole warps of lanes.
constexpr int kJ1 = 4, kHalo1 = 12, kOwn1 = 32 * kJ1 - 2 * kHalo1;
static_assert(kHalo1 % kJ1 == 0, "position 0 is the first register of a lane");
static_assert(32 * kJ1 - (kHalo1 + 1) - kOwn1 >= kHalo1 - 1, "sites above a warp's own, one for each step between exchanges");
constexpr int kMaxWarps1 = 16;
constexpr int kRing1 = 8;       // stored slices on their way back from global memory (a power of two)
__host__ __device__ inline int warps1d(int n) { return n <= 32 * kJ1 - 2 ? 1 : (n + kOwn1 - 1) / kOwn1; }
__host__ __device__ inline size_t slice1d(int n) { return (size_t)warps1d(n) * 32 * kJ1; }
}  // namespace sfg

// launch shape: lattice dimension, curved lattice, blocks per cluster, rows
// per thread (2D), threads per block, dynamic shared memory
struct GroupShape {
    int dim = 0, C = 1, J = 1, threads = 0;
    bool curved = false;
    size_t smem = 0;
};

bool group_eligible(const sfgpu_system *s);
// blocks: most blocks a system may take (1D: more than one lets the chain's
// slices fill shared memory); threads: most threads a 2D block should take
// m: Pure_DIIS's memory, 0 for a residual evaluation
bool group_shape(const sfgpu_system *s, int blocks, int threads, int m, GroupShape *out);
// doubles of stored slices that a 1D system keeps in global memory under the
// shape: 0 where its chains fit into shared memory
size_t group_slices(const sfgpu_system *s, const GroupShape &shape);
int group_prepare(const GroupShape &s, bool diis);
int group_max_clusters(const GroupShape &s, bool diis);
int group_residual(const GroupShape &s, const sfb::InstDesc *desc, const double *x, double *f, cudaStream_t st);
int group_diis(const GroupShape &s, const sfb::InstDesc *descs, int n, int clusters, int *queue, int m, double eta,
               double tol, int maxit, int *status, int *iters, double *errs, cudaStream_t st);
// the descriptor of a system's buffers and tables (iteration vectors unset)
void fill_inst_desc(const sfgpu_system *s, sfb::InstDesc *I);
