// BSR sparse matrix-vector product y = alpha*A*x + beta*y for b x b blocks
// (b = 2, 3), the hot kernel of the CPR-GMRES path.
//
// Semantics follow jxf_BSRMatrixMatvec (jxfpamg-0220/csrc/operation/mvops/
// seq_bsr_matvec.c:22-140): y <- (beta/alpha) y (0 if beta/alpha == 0,
// untouched if 1), then for each block of the row in stored order and each
// block column in order  y_i += A_ij x_j, then y <- alpha y.  Each output
// component is accumulated by one thread in exactly that order with separate
// multiply and add (the library is compiled with --fmad=false), so results
// are bit-identical to the reference CPU loop.
//
// staged == 0, the solves' choice: the slab or the direct kernel below; else the persistent TMA kernel.
//
// TMA kernel: a CTA owns a tile of ROWS consecutive block rows, one thread
// per output component.  The tile's block values and column indices are a
// contiguous slab of global memory [ia[r0], ia[r1]); a single elected thread
// streams each slab into shared memory with the 1-D bulk TMA copy
// (cp.async.bulk, completion on an mbarrier) while the CTA computes the
// previous tile, STAGES slabs deep.  CTAs are persistent (grid = 2 x SMs) and
// walk tiles with a grid stride.  x is gathered through the read-only path
// (it is L2-resident: 18 MB for 1.12 M 2x2 rows).  A tile whose slab does not
// fit a stage, or whose 16-byte-rounded copy would run past the end of the
// arrays, is computed with direct global loads instead; results are the same.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace jxcpr {

template <int BS, typename V>
struct SpmvTileCfg {
    static constexpr int ROWS = (BS == 2) ? 128 : 64;
    static constexpr int THREADS = ROWS * BS;
    static constexpr int STAGES = 3;
    static constexpr int CAP_BLOCKS = ROWS * ((BS == 2) ? 8 : 7);
    static constexpr int VAL_BYTES = CAP_BLOCKS * BS * BS * (int)sizeof(V) + 32;
    static constexpr int COL_BYTES = CAP_BLOCKS * 4 + 32;
    static constexpr int STAGE_BYTES = ((VAL_BYTES + 15) / 16 + (COL_BYTES + 15) / 16) * 16;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 128;
};

struct SlabPlan {
    long long v_src;  // byte offset of the 16-aligned copy start in a[]
    int v_bytes;      // copy size (multiple of 16)
    int v_pre;        // bytes between copy start and the first block of the tile
    long long c_src;
    int c_bytes;
    int c_pre;
    bool staged;
};

template <int BS, typename V>
__device__ __forceinline__ SlabPlan plan_slab(long long k0, long long k1, long long nnzb) {
    using Cfg = SpmvTileCfg<BS, V>;
    SlabPlan p;
    const long long vb = (long long)BS * BS * sizeof(V);
    long long vs = k0 * vb, ve = k1 * vb;
    long long vs16 = vs & ~15LL, ve16 = (ve + 15) & ~15LL;
    long long cs = k0 * 4, ce = k1 * 4;
    long long cs16 = cs & ~15LL, ce16 = (ce + 15) & ~15LL;
    p.v_src = vs16;
    p.v_bytes = (int)(ve16 - vs16);
    p.v_pre = (int)(vs - vs16);
    p.c_src = cs16;
    p.c_bytes = (int)(ce16 - cs16);
    p.c_pre = (int)(cs - cs16);
    p.staged = (k1 > k0) && (p.v_bytes <= Cfg::VAL_BYTES) && (p.c_bytes <= Cfg::COL_BYTES) &&
               (ve16 <= nnzb * vb) && (ce16 <= nnzb * 4);
    return p;
}

template <int BS, typename X>
__device__ __forceinline__ void gather_x(const X *__restrict__ x, int c, X (&xv)[BS]) {
#pragma unroll
    for (int j = 0; j < BS; ++j) xv[j] = __ldg(x + (long long)c * BS + j);
}

template <>
__device__ __forceinline__ void gather_x<2, double>(const double *__restrict__ x, int c, double (&xv)[2]) {
    double2 v = __ldg(reinterpret_cast<const double2 *>(x) + c);
    xv[0] = v.x;
    xv[1] = v.y;
}

// init_mode: 0 -> start from 0, 1 -> start from y, 2 -> start from y*scale_y.
template <int BS, typename V, typename X>
__device__ __forceinline__ X row_init(const X *y, long long idx, int init_mode, X scale_y) {
    if (init_mode == 0) return X(0);
    X v = y[idx];
    return init_mode == 1 ? v : v * scale_y;
}


// Accumulates one output component of a block row in stored block order.
template <int BS, typename V, typename X, bool SMEM>
__device__ __forceinline__ X row_accumulate(X acc, long long kb, long long ke, long long kbase,
                                            const V *__restrict__ vals, const int *__restrict__ cols,
                                            const X *__restrict__ x, int comp) {
    for (long long k = kb; k < ke; ++k) {
        const long long kk = k - kbase;
        const int c = SMEM ? cols[kk] : __ldg(cols + kk);
        X xv[BS];
        gather_x<BS, X>(x, c, xv);
#pragma unroll
        for (int j = 0; j < BS; ++j) {
            const V v = SMEM ? vals[kk * (BS * BS) + comp * BS + j] : __ldg(vals + kk * (BS * BS) + comp * BS + j);
            acc = acc + (X)v * xv[j];
        }
    }
    return acc;
}

template <int BS, typename V, typename X>
__global__ void __launch_bounds__(SpmvTileCfg<BS, V>::THREADS)
    bsr_spmv_tma_kernel(int nb, long long nnzb, const int *__restrict__ ia, const int *__restrict__ ja,
                        const V *__restrict__ a, const X *__restrict__ x, X *__restrict__ y, int init_mode,
                        X scale_y, X alpha, int *__restrict__ err) {
    using Cfg = SpmvTileCfg<BS, V>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
    unsigned char *stages = smem_raw + 128;
    const int tid = threadIdx.x;
    const int tiles = (nb + Cfg::ROWS - 1) / Cfg::ROWS;
    const unsigned char *a_bytes = reinterpret_cast<const unsigned char *>(a);
    const unsigned char *j_bytes = reinterpret_cast<const unsigned char *>(ja);

    if (tid == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) ptx::mbar_init(&bars[s], 1);
        ptx::fence_mbar_init();
    }
    __syncthreads();

    auto issue = [&](int t, int s) {
        long long r0 = (long long)t * Cfg::ROWS;
        long long r1 = min((long long)nb, r0 + Cfg::ROWS);
        long long k0 = ia[r0], k1 = ia[r1];
        SlabPlan p = plan_slab<BS, V>(k0, k1, nnzb);
        unsigned char *st = stages + (size_t)s * Cfg::STAGE_BYTES;
        if (p.staged) {
            ptx::mbar_arrive_expect_tx(&bars[s], (uint32_t)(p.v_bytes + p.c_bytes));
            ptx::bulk_g2s(st, a_bytes + p.v_src, (uint32_t)p.v_bytes, &bars[s]);
            ptx::bulk_g2s(st + ((Cfg::VAL_BYTES + 15) / 16) * 16, j_bytes + p.c_src, (uint32_t)p.c_bytes,
                          &bars[s]);
        } else {
            ptx::mbar_arrive_expect_tx(&bars[s], 0u);
        }
    };

    if (tid == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) {
            int t = blockIdx.x + s * gridDim.x;
            if (t < tiles) issue(t, s);
        }
    }

    bool aborted = false;
    int iter = 0;
    int t = blockIdx.x;
    for (; t < tiles; t += gridDim.x, ++iter) {
        const int s = iter % Cfg::STAGES;
        const uint32_t parity = (uint32_t)((iter / Cfg::STAGES) & 1);
        const long long r0 = (long long)t * Cfg::ROWS;
        const long long r1 = min((long long)nb, r0 + Cfg::ROWS);
        const long long k0 = ia[r0], k1 = ia[r1];
        const SlabPlan p = plan_slab<BS, V>(k0, k1, nnzb);
        const int failed = ptx::mbar_wait_bounded(&bars[s], parity, 1u << 26) ? 0 : 1;
        if (__syncthreads_or(failed)) {  // uniform decision: every thread leaves together
            if (tid == 0) atomicExch(err, 1);
            aborted = true;
            break;
        }
        const unsigned char *st = stages + (size_t)s * Cfg::STAGE_BYTES;
        const V *vs = reinterpret_cast<const V *>(st + p.v_pre);
        const int *cs = reinterpret_cast<const int *>(st + ((Cfg::VAL_BYTES + 15) / 16) * 16 + p.c_pre);
        const long long row = r0 + tid / BS;
        const int comp = tid % BS;
        if (row < r1) {
            const long long kb = ia[row], ke = ia[row + 1];
            const long long oidx = row * BS + comp;
            X acc = row_init<BS, V, X>(y, oidx, init_mode, scale_y);
            if (p.staged)
                acc = row_accumulate<BS, V, X, true>(acc, kb, ke, k0, vs, cs, x, comp);
            else
                acc = row_accumulate<BS, V, X, false>(acc, kb, ke, 0, a, ja, x, comp);
            y[oidx] = (alpha == X(1)) ? acc : acc * alpha;
        }
        __syncthreads();  // every thread is done with stage s
        if (tid == 0) {
            int nt = t + Cfg::STAGES * gridDim.x;
            if (nt < tiles) issue(nt, s);
        }
    }
    if (aborted && tid == 0) {
        // drain copies still in flight into this CTA's shared memory (bounded)
        int it2 = iter;
        for (int tt = t; tt < tiles && it2 < iter + Cfg::STAGES; tt += gridDim.x, ++it2) {
            int s = it2 % Cfg::STAGES;
            ptx::mbar_wait_bounded(&bars[s], (uint32_t)((it2 / Cfg::STAGES) & 1), 1u << 22);
        }
    }
}

// Slab kernel (2x2 FP64 blocks): a block of threads owns kSlabRows consecutive block rows, one thread per output
// component, and first copies their blocks -- one contiguous range -- to shared memory with 16-byte
// asynchronous copies.  Read where they lie, the rows' blocks cost one cache line each: a warp's load of the 16
// rows' k-th blocks touches 16 lines 224 bytes apart, and the L1's line rate, not the memory, bounds the 2x2
// product (1.12 M 2x2 rows in FP64: 65.0 us, 0.75 of the copy rate; this kernel 61).  While the copies are in
// flight the threads read their rows' first columns and gather x: what then bounds a block is the chain
// row pointer -> column -> x beside the copy.  ALONE, the product that a caller asks for by itself, is held to 40
// registers and six blocks per SM (60.7 us, with five 63.0).  Inside a solve five run (44 to 48 registers): a
// solve is the same with either, but of 64 systems at once other kernels run beside it, and its shared
// memory counts (82.2 ms; 85.7 with six blocks in the restarts' products, 91.4 in all).  The copies need no
// wait that could hang, and start before the kernel ahead has finished (no kernel of a solve writes the matrix).  A
// block whose range does not fit (rows of more than 8 blocks in the mean) reads it from global memory.
// XV: the type x is stored in (float where the caller's vector is FP32; widened before the product).
constexpr int kSlabThreads = 256, kSlabRows = kSlabThreads / 2;
constexpr int kSlabCap = kSlabRows * 8;                                   // blocks
constexpr int kSlabBytes = kSlabCap * 4 * (int)sizeof(double) + 16;       // 16: a range that starts off a boundary

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_addr(dst)), "l"(src) : "memory");
}

// Copies count values from src to dst + (src mod 16); the whole 16-byte pieces asynchronously, the ends value by
// value (src is aligned to 8).
__device__ __forceinline__ void slab_copy(unsigned char *dst, const double *src, int count) {
    const uintptr_t s0 = reinterpret_cast<uintptr_t>(src), s1 = s0 + (uintptr_t)count * sizeof(double);
    const uintptr_t base = s0 & ~(uintptr_t)15, a0 = (s0 + 15) & ~(uintptr_t)15, a1 = s1 & ~(uintptr_t)15;
    for (uintptr_t p = a0 + 16 * (uintptr_t)threadIdx.x; p < a1; p += 16 * kSlabThreads)
        cp_async16(dst + (p - base), reinterpret_cast<const void *>(p));
    // a whole number of blocks: both ends are off a boundary, or neither
    if (a0 != s0 && threadIdx.x < 2 && count > 0) {
        const int i = threadIdx.x ? count - 1 : 0;
        *reinterpret_cast<double *>(dst + (s0 - base) + i * sizeof(double)) = src[i];
    }
}

template <int BS, typename X, typename XV>
__device__ __forceinline__ void gather_wide(const XV *x, int c, X (&xv)[BS]) {
    if constexpr (BS == 2 && std::is_same<XV, double>::value) {
        const double2 v = reinterpret_cast<const double2 *>(x)[c];
        xv[0] = v.x;
        xv[1] = v.y;
    } else if constexpr (BS == 2 && !std::is_same<X, XV>::value) {
        const float2 v = reinterpret_cast<const float2 *>(x)[c];
        xv[0] = (X)v.x;
        xv[1] = (X)v.y;
    } else {
#pragma unroll
        for (int j = 0; j < BS; ++j) xv[j] = (X)x[(long long)c * BS + j];
    }
}

// Row `comp` of 2x2 block k.  PAIR: both values in one load, which needs them on a 16-byte boundary (the
// caller's array may start off one).
template <bool PAIR>
__device__ __forceinline__ void load_block_row(const double *a, long long k, int comp, double (&v)[2]) {
    const double *p = a + k * 4 + comp * 2;
    if constexpr (PAIR) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x;
        v[1] = t.y;
    } else {
        v[0] = p[0];
        v[1] = p[1];
    }
}

// NB entries of a row: their columns, and the x they name.
template <typename XV>
struct SlabBatch {
    static constexpr int NB = 4;
    int c[NB];
    double x[NB][2];
    __device__ __forceinline__ void columns(const int *__restrict__ ja, int k, int ke) {
#pragma unroll
        for (int t = 0; t < NB; ++t)
            if (k + t < ke) c[t] = __ldg(ja + k + t);
    }
    __device__ __forceinline__ void gather(const XV *xv, int k, int ke) {
#pragma unroll
        for (int t = 0; t < NB; ++t)
            if (k + t < ke) gather_wide<2, double, XV>(xv, c[t], x[t]);
    }
};

// One component of the row's entries [k, ke), in stored order, vals[0] the value of entry 0 of [kv, ...): the
// first batch's x is in B.
template <bool PAIR, typename XV>
__device__ __forceinline__ double slab_row(double acc, int k, int ke, int kv, const double *vals,
                                           const int *__restrict__ ja, const XV *x, int comp, SlabBatch<XV> &B) {
    constexpr int NB = SlabBatch<XV>::NB;
    while (k < ke) {
#pragma unroll
        for (int t = 0; t < NB; ++t)
            if (k + t < ke) {
                double v[2];
                load_block_row<PAIR>(vals, k - kv + t, comp, v);
#pragma unroll
                for (int j = 0; j < 2; ++j) acc = acc + v[j] * B.x[t][j];
            }
        k += NB;
        B.columns(ja, k, ke);
        B.gather(x, k, ke);
    }
    return acc;
}

// KeepX<ZT>: the product's x is also stored, as ZT, in vector Z[*i] (the flexible GMRES keeps its directions).
template <typename ZT>
struct KeepX {
    ZT *const *Z;
    const int *i;
};
struct NoKeep {};

// ALONE: see above (0: no bound of its own).
template <typename XV, class Keep, bool ALONE>
__global__ void __launch_bounds__(kSlabThreads, ALONE ? 6 : 0)
    bsr_spmv_slab_kernel(int nb, const int *__restrict__ ia, const int *__restrict__ ja, const double *__restrict__ a,
                         const XV *x, double *y, int init_mode, double scale_y, double alpha, Keep keep) {
    __shared__ __align__(16) unsigned char slab[kSlabBytes];
    const int tid = threadIdx.x, comp = tid % 2;
    const int r0 = blockIdx.x * kSlabRows, r1 = min(nb, r0 + kSlabRows);
    const int row = r0 + tid / 2;
    const bool live = row < r1;
    const int k0 = __ldg(ia + r0), k1 = __ldg(ia + r1);
    const int kb = live ? __ldg(ia + row) : 0, ke = live ? __ldg(ia + row + 1) : 0;
    const bool staged = k1 - k0 <= kSlabCap;
    const double *vs = a + (long long)k0 * 4;
    if (staged) {
        slab_copy(slab, vs, (k1 - k0) * 4);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    SlabBatch<XV> B;
    B.columns(ja, kb, ke);
    grid_dep_wait();
    B.gather(x, kb, ke);
    const long long oidx = (long long)row * 2 + comp;
    double acc = 0;
    if (live) {
        if constexpr (!std::is_same<Keep, NoKeep>::value) {
            using ZT = typename std::remove_reference<decltype(keep.Z[0][0])>::type;
            keep.Z[*keep.i][oidx] = (ZT)x[oidx];
        }
        acc = row_init<2, double, double>(y, oidx, init_mode, scale_y);
    }
    if (staged) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (!live) return;
    if (staged) {
        vs = reinterpret_cast<const double *>(slab + (reinterpret_cast<uintptr_t>(vs) & 15));
        if ((reinterpret_cast<uintptr_t>(vs) & 15) == 0)
            acc = slab_row<true, XV>(acc, kb, ke, k0, vs, ja, x, comp, B);
        else
            acc = slab_row<false, XV>(acc, kb, ke, k0, vs, ja, x, comp, B);
    } else {
        acc = slab_row<false, XV>(acc, kb, ke, k0, vs, ja, x, comp, B);
    }
    y[oidx] = alpha == 1.0 ? acc : acc * alpha;
}

template <typename X>
__global__ void scale_kernel(long long n, X beta, X *y) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = y[i] * beta;
}

// Direct kernel: one thread per output component, its row's blocks read where they lie.  Three values of a
// 3x3 block's row, or FP32 values, fill more of the lines that a warp's loads touch, and the slab's copy then costs
// more than it saves (slab / this, 1.12 M rows: 3x3 FP64 123 / 111 us, 3x3 FP32 96 / 86, 2x2 FP32 50.4 / 46.8; 2x2
// FP64 61 / 65.0).  x may be what the kernel ahead wrote: plain loads.
template <int BS, typename V, typename X, typename XV, class Keep>
__global__ void __launch_bounds__(256)
    bsr_spmv_direct_kernel(int nb, const int *__restrict__ ia, const int *__restrict__ ja, const V *__restrict__ a,
                           const XV *x, X *y, int init_mode, X scale_y, X alpha, Keep keep) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long row = gid / BS;
    const int comp = (int)(gid % BS);
    grid_dep_wait();
    if (row >= nb) return;
    const int kb = __ldg(ia + row), ke = __ldg(ia + row + 1);
    const long long oidx = row * BS + comp;
    if constexpr (!std::is_same<Keep, NoKeep>::value) {
        using ZT = typename std::remove_reference<decltype(keep.Z[0][0])>::type;
        keep.Z[*keep.i][oidx] = (ZT)x[oidx];
    }
    X acc = row_init<BS, V, X>(y, oidx, init_mode, scale_y);
    for (int k = kb; k < ke; ++k) {
        X xv[BS];
        gather_wide<BS, X, XV>(x, __ldg(ja + k), xv);
        const V *v = a + (long long)k * (BS * BS) + comp * BS;
#pragma unroll
        for (int j = 0; j < BS; ++j) acc = acc + (X)__ldg(v + j) * xv[j];
    }
    y[oidx] = (alpha == X(1)) ? acc : acc * alpha;
}

// staged == 0: the slab kernel for 2x2 FP64 blocks, else the direct one.
template <int BS, typename V, typename X, typename XV, class Keep>
static void launch_unstaged(const BsrView<V> &A, const XV *x, X *y, int init_mode, X scale_y, X alpha, Keep keep,
                            cudaStream_t stream, bool alone = false) {
    if constexpr (BS == 2 && sizeof(V) == 8) {
        auto kernel = bsr_spmv_slab_kernel<XV, Keep, false>;
        if constexpr (std::is_same<Keep, NoKeep>::value)
            if (alone) kernel = bsr_spmv_slab_kernel<XV, Keep, true>;
        launch_dep(kernel, dim3(div_up(A.nb, kSlabRows)), dim3(kSlabThreads), stream, A.nb, A.ia, A.ja, A.a, x, y,
                   init_mode, scale_y, alpha, keep);
    } else {
        launch_dep(bsr_spmv_direct_kernel<BS, V, X, XV, Keep>, dim3(div_up((long long)A.nb * BS, 256)), dim3(256), stream,
                   A.nb, A.ia, A.ja, A.a, x, y, init_mode, scale_y, alpha, keep);
    }
}

template <int BS, typename V, typename X>
static void launch_spmv(const BsrView<V> &A, X alpha, const X *x, X beta, X *y, int *err, cudaStream_t stream,
                        bool staged, bool alone) {
    const long long n = (long long)A.nb * BS;
    if (A.nb == 0) return;
    if (alpha == X(0)) {
        scale_kernel<X><<<div_up(n, 256), 256, 0, stream>>>(n, beta, y);
        JX_LAUNCH_CHECK();
        return;
    }
    X temp = beta / alpha;
    int init_mode = (temp == X(0)) ? 0 : (temp == X(1) ? 1 : 2);
    if (staged && err != nullptr) {
        using Cfg = SpmvTileCfg<BS, V>;
        static bool attr_set[64] = {};
        int dev = 0;
        JX_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64 || !attr_set[dev]) {
            JX_CUDA(cudaFuncSetAttribute(bsr_spmv_tma_kernel<BS, V, X>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg::SMEM_BYTES));
            if (dev >= 0 && dev < 64) attr_set[dev] = true;
        }
        int tiles = div_up(A.nb, Cfg::ROWS);
        int grid = std::min(tiles, 2 * sm_count());
        bsr_spmv_tma_kernel<BS, V, X><<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(
            A.nb, A.nnzb, A.ia, A.ja, A.a, x, y, init_mode, temp, alpha, err);
    } else {
        launch_unstaged<BS, V, X, X>(A, x, y, init_mode, temp, alpha, NoKeep{}, stream, alone);
    }
    JX_LAUNCH_CHECK();
}

template <typename V, typename X>
void bsr_spmv(const BsrView<V> &A, X alpha, const X *x, X beta, X *y, int *err, cudaStream_t stream, bool staged,
              bool alone) {
    switch (A.bs) {
        case 2: launch_spmv<2, V, X>(A, alpha, x, beta, y, err, stream, staged, alone); break;
        case 3: launch_spmv<3, V, X>(A, alpha, x, beta, y, err, stream, staged, alone); break;
        default:
            set_error("bsr_spmv: unsupported block size %d", A.bs);
            throw CudaError{cudaErrorInvalidValue, "block size"};
    }
}

template <int BS, typename ZT>
static void launch_keep(const BsrView<double> &A, const float *x, double *y, ZT *const *Z, const int *i,
                        cudaStream_t stream) {
    if (A.nb == 0) return;
    launch_unstaged<BS, double, double, float>(A, x, y, 0, 0.0, 1.0, KeepX<ZT>{Z, i}, stream);
    JX_LAUNCH_CHECK();
}

template <typename ZT>
void bsr_spmv_keep(const BsrView<double> &A, const float *x, double *y, ZT *const *Z, const int *i,
                   cudaStream_t stream) {
    if (A.bs == 2) launch_keep<2>(A, x, y, Z, i, stream);
    else launch_keep<3>(A, x, y, Z, i, stream);
}

template void bsr_spmv_keep<float>(const BsrView<double> &, const float *, double *, float *const *, const int *,
                                   cudaStream_t);
template void bsr_spmv_keep<double>(const BsrView<double> &, const float *, double *, double *const *, const int *,
                                    cudaStream_t);
template void bsr_spmv<double, double>(const BsrView<double> &, double, const double *, double, double *, int *,
                                       cudaStream_t, bool, bool);
template void bsr_spmv<float, double>(const BsrView<float> &, double, const double *, double, double *, int *,
                                      cudaStream_t, bool, bool);
template void bsr_spmv<float, float>(const BsrView<float> &, float, const float *, float, float *, int *,
                                     cudaStream_t, bool, bool);

}  // namespace jxcpr
