// Exact-order Gauss-Seidel sweeps fed from a stream in schedule order (exact_sweep.cu).
#pragma once

#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace jxcpr {

// A piece of a group: consecutive rows of the schedule, at most kSweepChunkBytes of matrix.
struct alignas(16) SweepChunk {
    long long mat, dyn;        // byte offsets of its matrix part and of its part written by each call
    int mat_bytes, dyn_bytes;  // multiples of 16
    int nrows, nent, nnew;     // rows, off-diagonal entries, of these the ones updated earlier in the sweep
    int pad[3];
};

// The matrix in schedule order.  bs 1: scalar operator, 2 / 3: block operator.
struct SweepStream {
    int bs = 0, nchunks = 0, max_mat = 0, max_dyn = 0;
    DevBuf<SweepChunk> desc;
    DevBuf<unsigned char> mat, dyn;
    bool ready() const { return nchunks > 0; }
};

// Host: the chunks and the integer part of the stream of a schedule (perm, gptr; forward: rows of lower
// index are read updated, else of higher index).  False where the sweep needs the general kernels: a
// scalar row reads a not yet updated neighbour of its own or an earlier group, a row is longer than a
// chunk, or the groups are wide enough to keep many blocks busy.
struct SweepStreamHost {
    std::vector<SweepChunk> desc;
    std::vector<unsigned char> mat;
    int max_mat = 0, max_dyn = 0;
    long long dyn = 0;
};
bool build_sweep_stream_host(int n, const int *ia, const int *ja, int bs, const std::vector<int> &perm,
                             const std::vector<int> &gptr, bool forward, SweepStreamHost &out);
// Uploads it and adds the values (a: n rows of blocks or scalars, diagonal first).
void upload_sweep_stream(const SweepStreamHost &h, int bs, const int *ia, const double *a, SweepStream &S,
                         cudaStream_t s);

// `apps` symmetric applications (a forward, then a backward sweep) of u_i = (f_i - sum a_ij u_j) / a_ii.
void sgs_stream(int n, const SweepStream &fwd, const SweepStream &bwd, int apps, const double *f, double *u, int *err,
                cudaStream_t s);
// One pass of the block update (jxf_ParBSRHGSRelax) along S; vt2: the vector of the res2 term (x: the
// iterate at the start of the pass).
void hgs_stream(const BsrView<double> &A, const SweepStream &S, const double *b, double *x, const double *vt2, double w,
                double omega, int plain, int *err, cudaStream_t s);

}  // namespace jxcpr
