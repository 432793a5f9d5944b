// Gauss-Seidel smoothers on the device.
//
// A sweep visits the groups of a Schedule in order; the rows of one group are
// updated concurrently.  Row i reads the NEW value of a neighbour j when
// rank[j] < rank[i] and the value at sweep start (a copy, `vt`) otherwise --
// exactly what a sequential sweep in rank order reads.  With the level
// schedule of the natural ordering (rank = i forward, n-1-i backward) this
// reproduces the reference's sequential sweeps bit for bit; with a
// multicolour schedule (rank = colour) it is Gauss-Seidel in colour order.
//
// * gs_sweep:  jxf_PAMGRelax6 with relax_weight = omega = 1 at one rank and
//   one thread (jxfpamg-0220/csrc/operation/relaxations/par_relax_6.c:226-270):
//   u_i = (f_i - sum_{j != i} a_ij u_j) / a_ii, skipped when a_ii == 0.
// * hgs_sweep: jxf_ParBSRHGSRelax (jxfpamg-0220/csrc/amg/par_relax_bsr.c:193-573)
//   with its Kahan-compensated block products (seq_bsr_matrix.c:841-872) and
//   2x2 / 3x3 diagonal-block solves (:945-1100).
//
// Execution: schedules of narrow groups are swept by one block from a stream
// in schedule order (exact_sweep.cu).  The others (wide groups; patterns the
// stream does not cover) run here: one persistent cooperative kernel per
// sweep, groups separated by a grid barrier whose wait is bounded (a timeout
// raises the error flag and every CTA leaves), or, for small systems, a single
// CTA with __syncthreads between groups.
#include <cooperative_groups.h>

#include "amg.cuh"
#include "block_ops.cuh"
#include "common.cuh"
#include "grid_sync.cuh"

namespace jxcpr {

// ---------------------------------------------------------------------------
// scalar Gauss-Seidel row update
// ---------------------------------------------------------------------------
__device__ __forceinline__ void gs_row(int i, const int *__restrict__ ia, const int *__restrict__ ja,
                                       const double *__restrict__ a, const int *__restrict__ rank,
                                       const double *__restrict__ f, double *u, const double *__restrict__ vt) {
    const int d = ia[i];
    if (d == ia[i + 1]) return;
    const double diag = a[d];
    if (diag == 0.0) return;
    const int ri = rank[i];
    double res = f[i];
    for (int k = d + 1; k < ia[i + 1]; ++k) {
        const int j = ja[k];
        const double uj = (rank[j] < ri) ? ((volatile const double *)u)[j] : vt[j];
        res = res - a[k] * uj;
    }
    u[i] = res / diag;
}

__global__ void gs_sweep_grid_kernel(int ngroups, const int *__restrict__ gptr, const int *__restrict__ perm,
                                     const int *__restrict__ ia, const int *__restrict__ ja,
                                     const double *__restrict__ a, const int *__restrict__ rank,
                                     const double *__restrict__ f, double *u, const double *__restrict__ vt,
                                     GridBarrier *bar, int *err) {
    const int nthreads = gridDim.x * blockDim.x;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (int g = 0; g < ngroups; ++g) {
        const int r0 = gptr[g], r1 = gptr[g + 1];
        for (int t = r0 + tid; t < r1; t += nthreads) gs_row(perm[t], ia, ja, a, rank, f, u, vt);
        if (g + 1 < ngroups) {
            __threadfence();
            if (!grid_barrier(bar, gridDim.x, err)) return;
        }
    }
}

__global__ void gs_sweep_block_kernel(int ngroups, const int *__restrict__ gptr, const int *__restrict__ perm,
                                      const int *__restrict__ ia, const int *__restrict__ ja,
                                      const double *__restrict__ a, const int *__restrict__ rank,
                                      const double *__restrict__ f, double *u, const double *__restrict__ vt) {
    // ngroups == 1: any number of CTAs; otherwise a single CTA (barrier = __syncthreads)
    const int stride = gridDim.x * blockDim.x;
    for (int g = 0; g < ngroups; ++g) {
        const int r0 = gptr[g], r1 = gptr[g + 1];
        for (int t = r0 + blockIdx.x * blockDim.x + threadIdx.x; t < r1; t += stride)
            gs_row(perm[t], ia, ja, a, rank, f, u, vt);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// block hybrid Gauss-Seidel row update
// ---------------------------------------------------------------------------
// vt: the iterate at the start of the pass (read for neighbours not yet
// updated in it); vt2: the vector of the res2 term (vt for HGS, the CPR's work
// vector for HSGS).
template <int BS>
__device__ __forceinline__ void hgs_row(int i, const int *__restrict__ ia, const int *__restrict__ ja,
                                        const double *__restrict__ a, const int *__restrict__ rank,
                                        const double *__restrict__ b, double *x, const double *__restrict__ vt,
                                        const double *__restrict__ vt2, double w, double omega, bool plain) {
    constexpr int B2 = BS * BS;
    const int ri = rank[i];
    const long long d = ia[i], e = ia[i + 1];
    double res[BS], out[BS];
#pragma unroll
    for (int k = 0; k < BS; ++k) res[k] = b[(long long)i * BS + k];
    if (plain) {
        for (long long jj = d + 1; jj < e; ++jj) {
            const int j = ja[jj];
            double xj[BS];
            const bool fresh = rank[j] < ri;
#pragma unroll
            for (int k = 0; k < BS; ++k)
                xj[k] = fresh ? ((volatile const double *)x)[(long long)j * BS + k] : vt[(long long)j * BS + k];
            blk_matvec_stable<BS>(-1.0, a + jj * B2, xj, res);
        }
        blk_inv_matvec<BS>(a + d * B2, res, out);
#pragma unroll
        for (int k = 0; k < BS; ++k) x[(long long)i * BS + k] = out[k];
        return;
    }
    double res0[BS], res2[BS], tmp[BS];
#pragma unroll
    for (int k = 0; k < BS; ++k) {
        res0[k] = 0.0;
        res2[k] = 0.0;
    }
    for (long long jj = d + 1; jj < e; ++jj) {
        const int j = ja[jj];
        double xj[BS], vj[BS];
        const bool fresh = rank[j] < ri;
#pragma unroll
        for (int k = 0; k < BS; ++k) {
            vj[k] = vt2[(long long)j * BS + k];
            xj[k] = fresh ? ((volatile const double *)x)[(long long)j * BS + k] : vt[(long long)j * BS + k];
        }
        blk_matvec_stable<BS>(-1.0, a + jj * B2, xj, res0);
        blk_matvec_stable<BS>(1.0, a + jj * B2, vj, res2);
    }
    const double prod = 1.0 - w * omega, omo = 1.0 - omega;
#pragma unroll
    for (int k = 0; k < BS; ++k) tmp[k] = omega * res[k] + res0[k] + omo * res2[k];
    blk_inv_matvec<BS>(a + d * B2, tmp, out);
#pragma unroll
    for (int k = 0; k < BS; ++k) {
        double xv = x[(long long)i * BS + k];
        xv *= prod;
        xv += w * out[k];
        x[(long long)i * BS + k] = xv;
    }
}

template <int BS>
__global__ void hgs_sweep_grid_kernel(int ngroups, const int *__restrict__ gptr, const int *__restrict__ perm,
                                      const int *__restrict__ ia, const int *__restrict__ ja,
                                      const double *__restrict__ a, const int *__restrict__ rank,
                                      const double *__restrict__ b, double *x, const double *__restrict__ vt,
                                      const double *__restrict__ vt2, double w, double omega, int plain,
                                      GridBarrier *bar, int *err) {
    const int nthreads = gridDim.x * blockDim.x;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (int g = 0; g < ngroups; ++g) {
        const int r0 = gptr[g], r1 = gptr[g + 1];
        for (int t = r0 + tid; t < r1; t += nthreads)
            hgs_row<BS>(perm[t], ia, ja, a, rank, b, x, vt, vt2, w, omega, plain);
        if (g + 1 < ngroups) {
            __threadfence();
            if (!grid_barrier(bar, gridDim.x, err)) return;
        }
    }
}

template <int BS>
__global__ void hgs_sweep_block_kernel(int ngroups, const int *__restrict__ gptr, const int *__restrict__ perm,
                                       const int *__restrict__ ia, const int *__restrict__ ja,
                                       const double *__restrict__ a, const int *__restrict__ rank,
                                       const double *__restrict__ b, double *x, const double *__restrict__ vt,
                                       const double *__restrict__ vt2, double w, double omega, int plain) {
    const int stride = gridDim.x * blockDim.x;
    for (int g = 0; g < ngroups; ++g) {
        const int r0 = gptr[g], r1 = gptr[g + 1];
        for (int t = r0 + blockIdx.x * blockDim.x + threadIdx.x; t < r1; t += stride)
            hgs_row<BS>(perm[t], ia, ja, a, rank, b, x, vt, vt2, w, omega, plain);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
namespace {
constexpr int kSweepThreads = 256;
constexpr int kSmallRows = 12288;

// The grid barrier of a cooperative sweep lives beside the hierarchy's error flag (err[0]) in the
// same per-hierarchy allocation (err[2..3]), so exact-order sweeps of different solvers on
// concurrent streams never share a barrier.
GridBarrier *barrier_of(int *err) { return reinterpret_cast<GridBarrier *>(err + 2); }

template <typename K>
int coop_grid(K kernel) {
    int per_sm = 0;
    JX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSweepThreads, 0));
    if (per_sm < 1) per_sm = 1;
    return per_sm * sm_count();
}
}  // namespace

void gs_sweep(const CsrView<double> &A, const Schedule &sch, const double *f, double *u, const int *rank,
              double *vt, int *err, cudaStream_t s) {
    const int n = A.nrows;
    if (n == 0 || sch.ngroups == 0) return;
    JX_CUDA(cudaMemcpyAsync(vt, u, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    if (n <= kSmallRows || sch.ngroups == 1) {
        const int threads = sch.ngroups == 1 ? 256 : 1024;
        const int blocks = sch.ngroups == 1 ? div_up(n, 256) : 1;
        gs_sweep_block_kernel<<<blocks, threads, 0, s>>>(sch.ngroups, sch.group_ptr.get(), sch.perm.get(), A.ia,
                                                         A.ja, A.a, rank, f, u, vt);
        JX_LAUNCH_CHECK();
        return;
    }
    static int grid = 0;
    if (!grid) grid = coop_grid(gs_sweep_grid_kernel);
    const int blocks = std::min(grid, div_up(sch.max_group, kSweepThreads));
    GridBarrier *bar = barrier_of(err);
    JX_CUDA(cudaMemsetAsync(bar, 0, sizeof(GridBarrier), s));
    int ng = sch.ngroups;
    const int *gp = sch.group_ptr.get(), *pm = sch.perm.get();
    const int *aia = A.ia, *aja = A.ja;
    const double *aa = A.a;
    void *args[] = {&ng, &gp, &pm, &aia, &aja, &aa, &rank, &f, &u, &vt, &bar, &err};
    JX_CUDA(cudaLaunchCooperativeKernel((void *)gs_sweep_grid_kernel, blocks, kSweepThreads, args, 0, s));
    count_launch();
}

namespace {
// One pass of the block point update along `sch` (vt already holds the iterate at the pass start).
void hgs_pass(const BsrView<double> &A, const Schedule &sch, const double *b, double *x, const int *rank,
              const double *vt, const double *vt2, double w, double omega, int plain, int *err, cudaStream_t s) {
    const int nb = A.nb;
    if (nb <= kSmallRows || sch.ngroups == 1) {
        const int threads = sch.ngroups == 1 ? 256 : 1024;
        const int blocks = sch.ngroups == 1 ? div_up(nb, 256) : 1;
        if (A.bs == 2)
            hgs_sweep_block_kernel<2><<<blocks, threads, 0, s>>>(sch.ngroups, sch.group_ptr.get(), sch.perm.get(),
                                                                 A.ia, A.ja, A.a, rank, b, x, vt, vt2, w, omega,
                                                                 plain);
        else
            hgs_sweep_block_kernel<3><<<blocks, threads, 0, s>>>(sch.ngroups, sch.group_ptr.get(), sch.perm.get(),
                                                                 A.ia, A.ja, A.a, rank, b, x, vt, vt2, w, omega,
                                                                 plain);
        JX_LAUNCH_CHECK();
        return;
    }
    static int grid2 = 0, grid3 = 0;
    if (!grid2) grid2 = coop_grid(hgs_sweep_grid_kernel<2>);
    if (!grid3) grid3 = coop_grid(hgs_sweep_grid_kernel<3>);
    const int grid = A.bs == 2 ? grid2 : grid3;
    const int blocks = std::min(grid, div_up(sch.max_group, kSweepThreads));
    GridBarrier *bar = barrier_of(err);
    JX_CUDA(cudaMemsetAsync(bar, 0, sizeof(GridBarrier), s));
    int ng = sch.ngroups;
    const int *gp = sch.group_ptr.get(), *pm = sch.perm.get();
    const int *aia = A.ia, *aja = A.ja;
    const double *aa = A.a;
    void *args[] = {&ng, &gp, &pm, &aia, &aja, &aa, &rank, &b, &x, &vt, &vt2, &w, &omega, &plain, &bar, &err};
    void *fn = A.bs == 2 ? (void *)hgs_sweep_grid_kernel<2> : (void *)hgs_sweep_grid_kernel<3>;
    JX_CUDA(cudaLaunchCooperativeKernel(fn, blocks, kSweepThreads, args, 0, s));
    count_launch();
}

int plain_weights(double w, double omega) {
    const double eps = 2.220446049250313e-16;
    return (fabs(w - 1) < eps && fabs(omega - 1) < eps) ? 1 : 0;
}
}  // namespace

void hgs_sweep(const BsrView<double> &A, const Schedule &sch, const SweepStream &stream, const double *b, double *x,
               const int *rank, double *vt, double w, double omega, int *err, cudaStream_t s) {
    const int nb = A.nb;
    if (nb == 0 || sch.ngroups == 0) return;
    if (stream.ready()) {
        hgs_stream(A, stream, b, x, x, w, omega, plain_weights(w, omega), err, s);
        return;
    }
    JX_CUDA(cudaMemcpyAsync(vt, x, sizeof(double) * nb * A.bs, cudaMemcpyDeviceToDevice, s));
    hgs_pass(A, sch, b, x, rank, vt, vt, w, omega, plain_weights(w, omega), err, s);
}

void hsgs_sweep(const BsrView<double> &A, const Schedule &fwd, const Schedule &bwd, const SweepStream &sfwd,
                const SweepStream &sbwd, const double *b, double *x, double *vt, double *work, double w, double omega,
                int *err, cudaStream_t s) {
    const int nb = A.nb;
    if (nb == 0 || fwd.ngroups == 0 || bwd.ngroups == 0) return;
    const int plain = plain_weights(w, omega);
    // the reference refreshes only the first nb (block-row count) entries of its work vector
    if (!plain) JX_CUDA(cudaMemcpyAsync(work, x, sizeof(double) * nb, cudaMemcpyDeviceToDevice, s));
    if (sfwd.ready() && sbwd.ready()) {
        hgs_stream(A, sfwd, b, x, work, w, omega, plain, err, s);
        hgs_stream(A, sbwd, b, x, work, w, omega, plain, err, s);
        return;
    }
    JX_CUDA(cudaMemcpyAsync(vt, x, sizeof(double) * nb * A.bs, cudaMemcpyDeviceToDevice, s));
    hgs_pass(A, fwd, b, x, fwd.rank.get(), vt, work, w, omega, plain, err, s);
    JX_CUDA(cudaMemcpyAsync(vt, x, sizeof(double) * nb * A.bs, cudaMemcpyDeviceToDevice, s));
    hgs_pass(A, bwd, b, x, bwd.rank.get(), vt, work, w, omega, plain, err, s);
}

}  // namespace jxcpr
