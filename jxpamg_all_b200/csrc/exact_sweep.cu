// Exact-order Gauss-Seidel sweeps of narrow schedules by one block.
//
// In natural order a sweep is a chain of groups (level schedule): 68 on the finest level of an 8,000-cell
// grid, 150 to 370 of 3 to 60 rows on the levels below.  What bounds it is the latency from one group to
// the next, not bandwidth: with the rows read from the CSR arrays where they lie, each entry is a chain
// column -> rank -> value from L2 (5 to 15 us per group).  Here the matrix is laid out in schedule order at
// setup and streamed through a ring of shared-memory stages by bulk (TMA) copies issued several groups
// ahead, the iterate stays in shared memory, and a group costs its arithmetic and a block barrier.
// Everything that does not depend on the sweep's own updates is done before it by the whole GPU: the
// right-hand side is put in schedule order, and in the block sweep the Kahan products with the iterate at
// the start of the pass (the res2 term, and the contributions of rows not yet updated) are formed per entry,
// so that the chain keeps the products with updated rows only.  Of an 8,000-cell system: a block sweep of 68
// groups 650 -> 218 us, four sweeps of the level below (150 groups) 8,310 -> 558 us, an application of the
// preconditioner 15.1 -> 2.6 ms (of an 85,184-cell one 340 -> 35, of 264,000 cells 553 -> 82); the setups, which
// lay the streams out, 6.3 -> 7.8 ms (24.8 -> 32.2, 54 -> 94).
// The order of operations of every row is the sequential sweep's (jxf_PAMGRelax6,
// jxfpamg-0220/csrc/operation/relaxations/par_relax_6.c:226-270; jxf_ParBSRHGSRelax,
// jxfpamg-0220/csrc/amg/par_relax_bsr.c:193-573): results are bit-identical.
#include <string.h>

#include <algorithm>

#include "block_ops.cuh"
#include "exact_sweep.cuh"
#include "ptx.cuh"

namespace jxcpr {

namespace {
constexpr int kSweepChunkBytes = 16 * 1024;
constexpr int kSweepThreads = 256;                // the threads that compute; one more warp issues the copies
constexpr int kSweepSmem = 220 * 1024;
constexpr int kSweepMaxStages = 8;
// bytes: a double per entry of the fullest chunk (12 bytes each); the stages behind it need their 128-byte boundary
constexpr int kSweepProducts = ((kSweepChunkBytes / 12 + 1) * 8 + 127) / 128 * 128;
static_assert(kSweepProducts % 128 == 0, "bulk copies land on 16-byte boundaries");
// Mean rows per group above which a grid of blocks does the sweep (one SM's bandwidth then bounds the stream).
// An application with level 0 and stage 2 streamed / swept by a grid, their groups of 655, 913, 1,380 rows:
// 36.4 / 35.1, 57.5 / 50.9, 105.2 / 84.4 ms; the levels below, narrower, are streamed in both.
constexpr int kSweepGroupRows = 512;
constexpr unsigned kOld = 1u << 31;   // column word: the neighbour is read as at the start of the pass
constexpr unsigned kSweepWait = 1u << 22;

__host__ __device__ __forceinline__ int al16(int b) { return (b + 15) & ~15; }

// The matrix part: SweepHead, rows[nrows], ptr[nrows + 1], cols[nent], bs > 1: newptr[nrows + 1] (entries
// of rows updated earlier), newcol[nnew] (their columns); then on a 16-byte boundary the diagonal (bs^2 per
// row), its reciprocal (scalar) or 1 / det (2x2; 3x3: unused), one per row, and the values: scalar every
// entry, blocks the entries of rows updated earlier.
struct SweepHead {
    int nrows, nent, nnew, pad;
};
__host__ __device__ __forceinline__ int sweep_ints(int bs, int nrows, int nent, int nnew) {
    return al16(16 + 4 * (nrows + nrows + 1 + nent + (bs > 1 ? nrows + 1 + nnew : 0)));
}
__host__ __device__ __forceinline__ int sweep_mat_bytes(int bs, int nrows, int nent, int nnew) {
    return sweep_ints(bs, nrows, nent, nnew) +
           al16(8 * (nrows + bs * bs * (nrows + (bs > 1 ? nnew : nent))));
}
// The part written by each call: scalar f (1 per row); blocks omega b, (1 - omega) res2 (bs per row each) and
// the products with rows not yet updated (bs per entry).
__host__ __device__ __forceinline__ int sweep_dyn_bytes(int bs, int nrows, int nent, int nnew) {
    return al16(8 * (bs > 1 ? bs * (2 * nrows + nent - nnew) : nrows));
}

struct SweepView {
    int nrows, nent, nnew;
    int *rows, *ptr, *cols, *newptr, *newcol;
    double *diag, *recip, *vals;
    __host__ __device__ __forceinline__ SweepView(unsigned char *p, int bs, int nr, int ne, int nn)
        : nrows(nr), nent(ne), nnew(nn) {
        rows = reinterpret_cast<int *>(p + 16);
        ptr = rows + nr;
        cols = ptr + nr + 1;
        newptr = cols + ne;
        newcol = newptr + nr + 1;
        diag = reinterpret_cast<double *>(p + sweep_ints(bs, nr, ne, nn));
        recip = diag + bs * bs * nr;
        vals = recip + nr;
    }
};
}  // namespace

bool build_sweep_stream_host(int n, const int *ia, const int *ja, int bs, const std::vector<int> &perm,
                             const std::vector<int> &gptr, bool forward, SweepStreamHost &out) {
    const int ng = (int)gptr.size() - 1;
    if (n <= 0 || ng <= 0 || (long long)n > (long long)kSweepGroupRows * ng) return false;
    auto updated = [&](int i, int j) { return forward ? j < i : j > i; };
    if (bs == 1) {
        // one copy of the iterate serves both reads: a neighbour not yet updated must come in a later group
        std::vector<int> grp(n);
        for (int g = 0; g < ng; ++g)
            for (int t = gptr[g]; t < gptr[g + 1]; ++t) grp[perm[t]] = g;
        for (int i = 0; i < n; ++i)
            for (int k = ia[i] + 1; k < ia[i + 1]; ++k) {
                const int j = ja[k];
                if (j != i && !updated(i, j) && grp[j] <= grp[i]) return false;
            }
    }
    out = SweepStreamHost();
    long long mat = 0;
    auto close = [&](int t0, int t1) {
        SweepChunk d{};
        d.nrows = t1 - t0;
        for (int t = t0; t < t1; ++t) {
            const int i = perm[t];
            d.nent += std::max(0, ia[i + 1] - ia[i] - 1);
            for (int k = ia[i] + 1; k < ia[i + 1]; ++k) d.nnew += updated(i, ja[k]) ? 1 : 0;
        }
        d.mat = mat;
        d.dyn = out.dyn;
        d.mat_bytes = sweep_mat_bytes(bs, d.nrows, d.nent, d.nnew);
        d.dyn_bytes = sweep_dyn_bytes(bs, d.nrows, d.nent, d.nnew);
        mat += d.mat_bytes;
        out.dyn += d.dyn_bytes;
        out.max_mat = std::max(out.max_mat, d.mat_bytes);
        out.max_dyn = std::max(out.max_dyn, d.dyn_bytes);
        out.desc.push_back(d);
    };
    std::vector<int> first;
    for (int g = 0; g < ng; ++g) {
        int t0 = gptr[g], ne = 0;
        for (int t = t0; t < gptr[g + 1]; ++t) {
            const int e = std::max(0, ia[perm[t] + 1] - ia[perm[t]] - 1);
            // an upper bound of the matrix part: every entry with its value
            if (sweep_mat_bytes(bs, 1, e, e) > kSweepChunkBytes) return false;
            if (t > t0 && sweep_mat_bytes(bs, t - t0 + 1, ne + e, ne + e) > kSweepChunkBytes) {
                first.push_back(t0);
                close(t0, t);
                t0 = t;
                ne = 0;
            }
            ne += e;
        }
        if (gptr[g + 1] > t0) {
            first.push_back(t0);
            close(t0, gptr[g + 1]);
        }
    }
    out.mat.assign((size_t)mat, 0);
    for (size_t c = 0; c < out.desc.size(); ++c) {
        const SweepChunk &d = out.desc[c];
        unsigned char *p = out.mat.data() + d.mat;
        const SweepHead h{d.nrows, d.nent, d.nnew, 0};
        memcpy(p, &h, sizeof h);
        SweepView V(p, bs, d.nrows, d.nent, d.nnew);
        int e = 0, m = 0;
        for (int r = 0; r < d.nrows; ++r) {
            const int i = perm[first[c] + r];
            V.rows[r] = i;
            V.ptr[r] = e;
            if (bs > 1) V.newptr[r] = m;
            for (int k = ia[i] + 1; k < ia[i + 1]; ++k) {
                const bool up = updated(i, ja[k]);
                V.cols[e++] = (int)((unsigned)ja[k] | (bs > 1 && !up ? kOld : 0u));
                if (bs > 1 && up) V.newcol[m] = ja[k];
                m += up ? 1 : 0;
            }
        }
        V.ptr[d.nrows] = e;
        if (bs > 1) V.newptr[d.nrows] = m;
    }
    return true;
}

// the values of one chunk per block: diag (0 for an empty row), entries in stored order
__global__ void sweep_values_kernel(const SweepChunk *__restrict__ desc, unsigned char *__restrict__ mat, int bs,
                                    const int *__restrict__ ia, const double *__restrict__ a) {
    const SweepChunk d = desc[blockIdx.x];
    SweepView V(mat + d.mat, bs, d.nrows, d.nent, d.nnew);
    const int b2 = bs * bs;
    for (int r = threadIdx.x; r < d.nrows; r += blockDim.x) {
        const int i = V.rows[r];
        const long long k0 = ia[i];
        const bool empty = ia[i] == ia[i + 1];
        for (int q = 0; q < b2; ++q) V.diag[r * b2 + q] = empty ? 0.0 : a[k0 * b2 + q];
        V.recip[r] = bs == 1 ? 1.0 / V.diag[r] : bs == 2 ? blk2_inv_det(V.diag + r * b2) : 0.0;
        int m = bs > 1 ? V.newptr[r] : V.ptr[r];
        for (int e = V.ptr[r]; e < V.ptr[r + 1]; ++e) {
            if (bs > 1 && ((unsigned)V.cols[e] & kOld)) continue;
            const long long k = k0 + 1 + (e - V.ptr[r]);
            for (int q = 0; q < b2; ++q) V.vals[(long long)m * b2 + q] = a[k * b2 + q];
            ++m;
        }
    }
}

void upload_sweep_stream(const SweepStreamHost &h, int bs, const int *ia, const double *a, SweepStream &S,
                         cudaStream_t s) {
    S.bs = bs;
    S.nchunks = (int)h.desc.size();
    S.max_mat = h.max_mat;
    S.max_dyn = h.max_dyn;
    S.desc.alloc(h.desc.size());
    S.desc.upload(h.desc.data(), h.desc.size(), s);
    S.mat.alloc(h.mat.size());
    S.mat.upload(h.mat.data(), h.mat.size(), s);
    S.dyn.alloc((size_t)h.dyn);
    sweep_values_kernel<<<S.nchunks, 128, 0, s>>>(S.desc.get(), S.mat.get(), bs, ia, a);
    JX_LAUNCH_CHECK();
    JX_CUDA(cudaStreamSynchronize(s));  // the host arrays may go
}

// ---------------------------------------------------------------------------
// the ring of stages
// ---------------------------------------------------------------------------
namespace {
struct SweepArgs {
    const SweepChunk *desc[2];  // forward, backward (or the one pass)
    const unsigned char *mat[2];
    unsigned char *dyn[2];
    int nchunks[2];
    int nsweeps;  // sweep s uses stream s & 1
    int nstages, mat_cap, stage_bytes, u_bytes;  // u_bytes 0: the iterate stays in global memory
};

// The issuing warp's side of the ring: the chunks of all sweeps in turn.  Lane l holds the descriptor of chunk
// base + l and, read ahead, that of base + 32 + l: with one descriptor read per chunk the load's latency, not
// the computing threads, set the pace (0.9 us a chunk).
struct SweepProducer {
    SweepChunk cur, ahead;
    int q = 0, total = 0, stage = 0;
    __device__ __forceinline__ void fetch(const SweepArgs &A, int i, SweepChunk &d) const {
        if (i >= total) return;
        const int r = i % (A.nchunks[0] + A.nchunks[1]), w = r >= A.nchunks[0];
        d = A.desc[w][w ? r - A.nchunks[0] : r];
    }
    __device__ __forceinline__ void start(const SweepArgs &A, int lane) {
        total = 0;
        for (int s = 0; s < A.nsweeps; ++s) total += A.nchunks[s & 1];
        fetch(A, lane, cur);
        fetch(A, 32 + lane, ahead);
    }
    __device__ __forceinline__ void issue(const SweepArgs &A, unsigned char *stages, uint64_t *bars, int lane) {
        if (q >= total) return;
        const int src = q & 31;
        const long long mat = __shfl_sync(0xffffffffu, cur.mat, src), dyn = __shfl_sync(0xffffffffu, cur.dyn, src);
        const int mb = __shfl_sync(0xffffffffu, cur.mat_bytes, src), db = __shfl_sync(0xffffffffu, cur.dyn_bytes, src);
        if (lane == 0) {
            const int w = q % (A.nchunks[0] + A.nchunks[1]) >= A.nchunks[0];
            unsigned char *p = stages + (size_t)stage * A.stage_bytes;
            ptx::mbar_arrive_expect_tx(&bars[stage], (uint32_t)(mb + db));
            ptx::bulk_g2s(p, A.mat[w] + mat, (uint32_t)mb, &bars[stage]);
            ptx::bulk_g2s(p + A.mat_cap, A.dyn[w] + dyn, (uint32_t)db, &bars[stage]);
        }
        stage = stage + 1 == A.nstages ? 0 : stage + 1;
        if ((++q & 31) == 0) {
            cur = ahead;
            fetch(A, q + 32 + lane, ahead);
        }
    }
};

// barrier among the computing threads
__device__ __forceinline__ void sweep_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(kSweepThreads) : "memory");
}

// Runs body(matrix part, call part) on every chunk of every sweep in turn (threads 0 .. kSweepThreads - 1), a
// block barrier after each; the last warp issues the copies.  Returns false (in every thread) when a
// copy did not arrive: the error flag is raised and the copies in flight have been waited for, with a limit
// as well.
template <typename F>
__device__ __forceinline__ bool sweep_chunks(const SweepArgs &A, unsigned char *smem, int *err, F &&body) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    unsigned char *stages = smem + 128 + A.u_bytes + kSweepProducts;
    const bool producer = threadIdx.x >= kSweepThreads;
    const int lane = threadIdx.x & 31;
    SweepProducer P;
    if (producer) {
        P.start(A, lane);
        if (lane == 0) {
            for (int q = 0; q < A.nstages; ++q) ptx::mbar_init(&bars[q], 1);
            ptx::fence_mbar_init();
        }
        __syncwarp();
        for (int q = 0; q < A.nstages; ++q) P.issue(A, stages, bars, lane);
    }
    __syncthreads();  // the barriers are initialised, the iterate is in place
    int stage = 0;
    uint32_t parity = 0;
    for (int s = 0; s < A.nsweeps; ++s)
        for (int c = 0; c < A.nchunks[s & 1]; ++c) {
            bool ok = true;
            if (!producer) {
                ok = ptx::mbar_wait_bounded(&bars[stage], parity, kSweepWait);
                // a thread that gave up still takes part in the body's barriers; nothing it leaves is used
                unsigned char *p = stages + (size_t)stage * A.stage_bytes;
                body(ok, p, reinterpret_cast<const double *>(p + A.mat_cap));
            }
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == kSweepThreads) {
                    atomicExch(err, 1);
                    for (int q = 0; q < A.nstages; ++q)
                        ptx::mbar_wait_bounded(&bars[q], q < stage ? parity ^ 1u : parity, kSweepWait >> 4);
                }
                return false;
            }
            if (producer) P.issue(A, stages, bars, lane);
            if (++stage == A.nstages) {
                stage = 0;
                parity ^= 1u;
            }
        }
    return true;
}

// Stages and shared memory for an iterate of u_bytes; the iterate goes to global memory where fewer than
// two stages would be left beside it.
size_t sweep_plan(SweepArgs &A, int max_mat, int max_dyn, size_t u_bytes) {
    A.mat_cap = max_mat;
    A.stage_bytes = (max_mat + max_dyn + 127) & ~127;
    const size_t u = (u_bytes + 127) & ~(size_t)127;
    const int fixed = 128 + kSweepProducts;
    A.u_bytes = u + fixed + 2 * (size_t)A.stage_bytes <= (size_t)kSweepSmem ? (int)u : 0;
    A.nstages = std::min(kSweepMaxStages, (kSweepSmem - fixed - A.u_bytes) / A.stage_bytes);
    return fixed + (size_t)A.u_bytes + (size_t)A.nstages * A.stage_bytes;
}
}  // namespace

// ---------------------------------------------------------------------------
// scalar sweeps
// ---------------------------------------------------------------------------
__global__ void sweep_rhs_kernel(const SweepChunk *__restrict__ desc, unsigned char *__restrict__ mat,
                                 unsigned char *__restrict__ dyn, const double *__restrict__ f) {
    const SweepChunk d = desc[blockIdx.x];
    const SweepView V(mat + d.mat, 1, d.nrows, d.nent, d.nnew);
    double *o = reinterpret_cast<double *>(dyn + d.dyn);
    for (int r = threadIdx.x; r < d.nrows; r += blockDim.x) o[r] = f[V.rows[r]];
}

// Per chunk: every product a_ij u_j at once (a group's neighbours are all final), then each row's sum in stored
// order.  The products have a place of their own: writing them over the stage would need a proxy fence before
// the next copy.
__global__ void __launch_bounds__(kSweepThreads + 32, 1) sgs_stream_kernel(SweepArgs A, int n, double *u, int *err) {
    extern __shared__ __align__(128) unsigned char sweep_smem[];
    double *us = A.u_bytes ? reinterpret_cast<double *>(sweep_smem + 128) : u;
    double *prod = reinterpret_cast<double *>(sweep_smem + 128 + A.u_bytes);
    if (A.u_bytes)
        for (int i = threadIdx.x; i < n; i += blockDim.x) us[i] = u[i];
    const bool ok = sweep_chunks(A, sweep_smem, err, [&](bool arrived, unsigned char *p, const double *f) {
        const SweepHead h = arrived ? *reinterpret_cast<const SweepHead *>(p) : SweepHead{0, 0, 0, 0};
        const SweepView V(p, 1, h.nrows, h.nent, h.nnew);
        for (int e = threadIdx.x; e < h.nent; e += 4 * kSweepThreads) {
            double t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (e + q * kSweepThreads < h.nent)
                    t[q] = V.vals[e + q * kSweepThreads] * us[V.cols[e + q * kSweepThreads]];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (e + q * kSweepThreads < h.nent) prod[e + q * kSweepThreads] = t[q];
        }
        sweep_sync();
        for (int r = threadIdx.x; r < h.nrows; r += kSweepThreads) {
            const double diag = V.diag[r], recip = V.recip[r];
            double res = f[r];
            int e = V.ptr[r];
            const int e1 = V.ptr[r + 1];
            for (; e + 7 < e1; e += 8) {
                double t[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) t[q] = prod[e + q];
#pragma unroll
                for (int q = 0; q < 8; ++q) res = res - t[q];
            }
            double t[7];
#pragma unroll
            for (int q = 0; q < 7; ++q)
                if (e + q < e1) t[q] = prod[e + q];
#pragma unroll
            for (int q = 0; q < 7; ++q)
                if (e + q < e1) res = res - t[q];
            if (diag != 0.0) us[V.rows[r]] = div_known(res, diag, recip);
        }
    });
    if (ok && A.u_bytes)
        for (int i = threadIdx.x; i < n; i += blockDim.x) u[i] = us[i];
}

void sgs_stream(int n, const SweepStream &fwd, const SweepStream &bwd, int apps, const double *f, double *u, int *err,
                cudaStream_t s) {
    SweepArgs A{};
    for (int w = 0; w < 2; ++w) {
        const SweepStream &S = w ? bwd : fwd;
        sweep_rhs_kernel<<<S.nchunks, 128, 0, s>>>(S.desc.get(), S.mat.get(), S.dyn.get(), f);
        JX_LAUNCH_CHECK();
        A.desc[w] = S.desc.get();
        A.mat[w] = S.mat.get();
        A.dyn[w] = S.dyn.get();
        A.nchunks[w] = S.nchunks;
    }
    A.nsweeps = 2 * apps;
    const size_t smem = sweep_plan(A, std::max(fwd.max_mat, bwd.max_mat), std::max(fwd.max_dyn, bwd.max_dyn),
                                   sizeof(double) * (size_t)n);
    JX_CUDA(cudaFuncSetAttribute(sgs_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSweepSmem));
    sgs_stream_kernel<<<1, kSweepThreads + 32, smem, s>>>(A, n, u, err);
    JX_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// block sweeps
// ---------------------------------------------------------------------------
// Per row: omega b (plain: b), (1 - omega) res2 with res2 = sum A_ij vt2_j, and per entry whose row is not
// updated yet the product A_ij x_j; every block product Kahan-compensated, sums in stored order.
template <int BS>
__global__ void hgs_before_kernel(const SweepChunk *__restrict__ desc, unsigned char *__restrict__ mat,
                                  unsigned char *__restrict__ dyn, const int *__restrict__ ia,
                                  const int *__restrict__ ja, const double *__restrict__ a,
                                  const double *__restrict__ b, const double *__restrict__ x,
                                  const double *__restrict__ vt2, double omega, int plain) {
    const SweepChunk d = desc[blockIdx.x];
    const SweepView V(mat + d.mat, BS, d.nrows, d.nent, d.nnew);
    double *p1 = reinterpret_cast<double *>(dyn + d.dyn), *c2 = p1 + BS * d.nrows, *so = c2 + BS * d.nrows;
    const double omo = 1.0 - omega;
    for (int r = threadIdx.x; r < d.nrows; r += blockDim.x) {
        const int i = V.rows[r];
        double res2[BS];
#pragma unroll
        for (int q = 0; q < BS; ++q) res2[q] = 0.0;
        int m = V.ptr[r] - V.newptr[r];
        for (int e = V.ptr[r]; e < V.ptr[r + 1]; ++e) {
            const unsigned cw = (unsigned)V.cols[e];
            const int j = (int)(cw & ~kOld);
            const double *blk = a + ((long long)ia[i] + 1 + (e - V.ptr[r])) * (BS * BS);
            double v[BS], k[BS];
            if (cw & kOld) {
#pragma unroll
                for (int q = 0; q < BS; ++q) v[q] = x[(long long)j * BS + q];
                blk_kahan<BS>(blk, v, k);
#pragma unroll
                for (int q = 0; q < BS; ++q) so[m * BS + q] = k[q];
                ++m;
            }
            if (!plain) {
#pragma unroll
                for (int q = 0; q < BS; ++q) v[q] = vt2[(long long)j * BS + q];
                blk_kahan<BS>(blk, v, k);
#pragma unroll
                for (int q = 0; q < BS; ++q) res2[q] += 1.0 * k[q];
            }
        }
#pragma unroll
        for (int q = 0; q < BS; ++q) {
            const double bq = b[(long long)i * BS + q];
            p1[r * BS + q] = plain ? bq : omega * bq;
            c2[r * BS + q] = omo * res2[q];
        }
    }
}

// Per chunk: the Kahan products with updated rows all at once, then each row's sum
// in stored order and its block solve.
template <int BS>
__global__ void __launch_bounds__(kSweepThreads + 32, 1) hgs_stream_kernel(SweepArgs A, int nb, double *x, double w,
                                                                           double omega, int plain, int *err) {
    extern __shared__ __align__(128) unsigned char sweep_smem[];
    constexpr int B2 = BS * BS;
    double *xs = A.u_bytes ? reinterpret_cast<double *>(sweep_smem + 128) : x;
    const int n = nb * BS;
    if (A.u_bytes)
        for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = x[i];
    double *prod = reinterpret_cast<double *>(sweep_smem + 128 + A.u_bytes);
    const double keep = 1.0 - w * omega;
    const bool ok = sweep_chunks(A, sweep_smem, err, [&](bool arrived, unsigned char *p, const double *dy) {
        const SweepHead h = arrived ? *reinterpret_cast<const SweepHead *>(p) : SweepHead{0, 0, 0, 0};
        const SweepView V(p, BS, h.nrows, h.nent, h.nnew);
        const double *p1 = dy, *c2 = p1 + BS * h.nrows, *so = c2 + BS * h.nrows;
        for (int m = threadIdx.x; m < h.nnew; m += kSweepThreads) {
            double v[BS], k[BS];
            const double *xj = xs + (long long)V.newcol[m] * BS;
#pragma unroll
            for (int q = 0; q < BS; ++q) v[q] = xj[q];
            blk_kahan<BS>(V.vals + m * B2, v, k);
#pragma unroll
            for (int q = 0; q < BS; ++q) prod[m * BS + q] = k[q];
        }
        sweep_sync();
        for (int r = threadIdx.x; r < h.nrows; r += kSweepThreads) {
            double res[BS], out[BS];
#pragma unroll
            for (int q = 0; q < BS; ++q) res[q] = plain ? p1[r * BS + q] : 0.0;
            const int e0 = V.ptr[r], e1 = V.ptr[r + 1];
            int m = V.newptr[r], o = e0 - m;
            for (int e = e0; e < e1; ++e) {
                const bool old = ((unsigned)V.cols[e] & kOld) != 0u;
                const double *k = old ? so + o * BS : prod + m * BS;
                o += old ? 1 : 0;
                m += old ? 0 : 1;
#pragma unroll
                for (int q = 0; q < BS; ++q) res[q] += -1.0 * k[q];
            }
            if (!plain)
#pragma unroll
                for (int q = 0; q < BS; ++q) res[q] = p1[r * BS + q] + res[q] + c2[r * BS + q];
            const double *D = V.diag + r * B2;
            const double inv_det = V.recip[r];
            if (BS == 2 && inv_det == inv_det) {  // blk_inv_matvec's products with the factor formed at setup
                out[0] = (D[3] * res[0] - D[1] * res[1]) * inv_det;
                out[1] = (-D[2] * res[0] + D[0] * res[1]) * inv_det;
            } else {
                blk_inv_matvec<BS>(D, res, out);
            }
            double *xi = xs + (long long)V.rows[r] * BS;
#pragma unroll
            for (int q = 0; q < BS; ++q) {
                if (plain) {
                    xi[q] = out[q];
                } else {
                    double xv = xi[q];
                    xv *= keep;
                    xv += w * out[q];
                    xi[q] = xv;
                }
            }
        }
    });
    if (ok && A.u_bytes)
        for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] = xs[i];
}

template <int BS>
static void hgs_stream_t(const BsrView<double> &A, const SweepStream &S, const double *b, double *x, const double *vt2,
                         double w, double omega, int plain, int *err, cudaStream_t s) {
    hgs_before_kernel<BS><<<S.nchunks, 128, 0, s>>>(S.desc.get(), S.mat.get(), S.dyn.get(), A.ia, A.ja, A.a, b, x, vt2,
                                                    omega, plain);
    JX_LAUNCH_CHECK();
    SweepArgs R{};
    R.desc[0] = R.desc[1] = S.desc.get();
    R.mat[0] = R.mat[1] = S.mat.get();
    R.dyn[0] = R.dyn[1] = S.dyn.get();
    R.nchunks[0] = R.nchunks[1] = S.nchunks;
    R.nsweeps = 1;
    const size_t smem = sweep_plan(R, S.max_mat, S.max_dyn, sizeof(double) * (size_t)A.nb * BS);
    JX_CUDA(cudaFuncSetAttribute(hgs_stream_kernel<BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSweepSmem));
    hgs_stream_kernel<BS><<<1, kSweepThreads + 32, smem, s>>>(R, A.nb, x, w, omega, plain, err);
    JX_LAUNCH_CHECK();
}

void hgs_stream(const BsrView<double> &A, const SweepStream &S, const double *b, double *x, const double *vt2, double w,
                double omega, int plain, int *err, cudaStream_t s) {
    if (A.bs == 2) hgs_stream_t<2>(A, S, b, x, vt2, w, omega, plain, err, s);
    else hgs_stream_t<3>(A, S, b, x, vt2, w, omega, plain, err, s);
}

}  // namespace jxcpr
