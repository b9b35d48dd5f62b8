/*
 * kernels_fast.cu -- TBS_ALGO_FP64 / TBS_ALGO_MIXED kernels for sm_100a,
 * plus the norm / permutation helpers every algorithm uses.
 *
 * The LIJ sweep of the reference (src/main.cxx:207-229) is
 *     dU = -M^-1 R ;  U += dU ;  R = rhs + J U
 * with M the block-tridiagonal part of J along each line.  Writing
 * J = M + O (O = couplings between different lines) and using M dU = -R,
 *     R_new = R + J dU = O dU,
 * so after the first sweep only the cross-line blocks are read to update
 * the residual.  The line solve is rewritten with explicit inverses:
 *     b_k  = -Dinv_k R_k                         (fast_resid, all cells)
 *     y_k  = b_k - G_k y_{k-1},   G_k = Dinv_k A_k (fast_thomas forward)
 *     dU_k = y_k - Gam_k dU_{k+1}, Gam_k = Dinv_k C_k (backward)
 * where Dinv_k = (D_k - A_k Gam_{k-1})^-1 is the inverse of the block-Thomas
 * pivot of src/okl/lineLU_v2.okl:58-182.  The recurrence on each line is
 * then one 9x9 matvec per cell; everything else is data parallel.
 *
 * Data are "position" ordered: cells in line order, each line starting at a
 * multiple of 4 positions, so that runs of cells are 16-byte aligned for
 * cp.async.bulk in FP64 and FP32 alike.
 */
#include "device_common.cuh"
#include "recip.cuh"
#include "tbs_internal.hxx"
#include "thomas.cuh"
#include "tma.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace tbs {

constexpr int NV = 9;
constexpr int NB = 81;
constexpr unsigned FULL = 0xffffffffu;

/* ================================================================ helpers */

__global__ void zero_kernel(double *p, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        p[t] = 0.0;
}

static int grid_for(long long n, int threads, int cap = 148 * 8) {
    long long b = (n + threads - 1) / threads;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int launch_zero(cudaStream_t st, double *p, long long n) {
    zero_kernel<<<grid_for(n, 256), 256, 0, st>>>(p, n);
    return (int)cudaGetLastError();
}

/* block b sums v[b*chunk : (b+1)*chunk)^2 in a fixed order */
__global__ void norm_partials_kernel(const double *__restrict__ v, long long n, long long chunk,
                                     double *__restrict__ partials) {
    const long long lo = blockIdx.x * chunk;
    long long hi = lo + chunk;
    if (hi > n) hi = n;
    double s = 0.0;
    for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) s += v[t] * v[t];
    __shared__ double red[8];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        partials[blockIdx.x] = tot;
    }
}

int launch_norm_partials(cudaStream_t st, const double *v, long long n, double *partials,
                         int npart) {
    long long chunk = (n + npart - 1) / npart;
    if (chunk < 1) chunk = 1;
    norm_partials_kernel<<<npart, 256, 0, st>>>(v, n, chunk, partials);
    return (int)cudaGetLastError();
}

/* threads of the one-CTA norm sum (its order: thread t adds partials t,
 * t + REDUCE_THREADS, ..., then the warps' sums in order) */
constexpr int REDUCE_THREADS = 1024;

/* Sum the partials in a fixed order, record the norm and decide whether the
 * solve goes on.  The decision feeds the CUDA graph's while-node, so the
 * sweep loop never returns to the host.  n == 0 re-records the latest norm
 * (state->last) as the start of a new sweep sequence; is_start ==
 * NORM_CHECK records a converged solve's true residual. */
__global__ void reduce_norm_kernel(const double *__restrict__ partials, int n, SolveState *state,
                                   double *hist, int is_start,
                                   cudaGraphConditionalHandle handle, int use_cond,
                                   cudaGraphConditionalHandle handle2, int use2) {
    __shared__ double red[REDUCE_THREADS / 32];
    double acc = strided_sum(partials, n, REDUCE_THREADS);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(FULL, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < REDUCE_THREADS / 32; ++w) tot += red[w];
        const double nrm = n > 0 ? sqrt(tot) : state->last;
        if (is_start == NORM_CHECK) {
            /* the true residual of a solve whose recursive residual passed:
             * both conditions (the loop's, and the IF node that makes the
             * restart's input) say whether the solve goes on */
            const bool go = record_check(state, hist, nrm);
            if (use_cond) cudaGraphSetConditional(handle, go ? 1u : 0u);
            if (use2) cudaGraphSetConditional(handle2, go ? 1u : 0u);
            return;
        }
        if (is_start) {
            state->sweep = 0;
            state->norm0 = nrm;
            state->true_norm = -1.0;
            state->checks = 0;
            state->restarts = 0;
        } else {
            state->sweep += 1;
        }
        const int sw = state->sweep;
        if (sw < state->hist_cap) hist[sw] = nrm;
        state->last = nrm;
        const bool go = isfinite(nrm) && nrm > state->tol * state->norm0 && sw < state->max_sweeps;
        if (use_cond) cudaGraphSetConditional(handle, go ? 1u : 0u);
        if (use2) cudaGraphSetConditional(handle2, go ? 1u : 0u);
    }
}

int launch_reduce_norm(cudaStream_t st, const double *partials, int n, SolveState *state,
                       double *hist, int is_start, unsigned long long cond_handle, int use_cond,
                       unsigned long long cond_handle2, int use2) {
    reduce_norm_kernel<<<1, REDUCE_THREADS, 0, st>>>(partials, n, state, hist, is_start,
                                                     (cudaGraphConditionalHandle)cond_handle, use_cond,
                                                     (cudaGraphConditionalHandle)cond_handle2, use2);
    return (int)cudaGetLastError();
}

/* Vectors between element and position order (src, dst by word; grid row r:
 * vector r).  Bound by HBM once a word's element costs little: with a 64-bit
 * division by nv a word 1200x1280 took 59 us, with 32-bit word numbers, nv a
 * constant where it is 9, 55.  NVC 0: any nv.  Eight vectors of 360x384 in one
 * launch: 40 us, 97 in eight. */
template <int NVC, bool TO_POS, typename I>
__global__ void permute_kernel(int nv_, long long n_, const int *__restrict__ pos_of_elem,
                               const double *__restrict__ src, double *__restrict__ dst, long long src_stride,
                               long long dst_stride) {
    const I nv = NVC > 0 ? NVC : nv_, n = (I)n_;
    src += blockIdx.y * src_stride;
    dst += blockIdx.y * dst_stride;
    for (I t = blockIdx.x * (I)blockDim.x + threadIdx.x; t < n; t += (I)gridDim.x * blockDim.x) {
        const I e = t / nv;
        const long long p = (long long)pos_of_elem[e] * nv + (t - e * nv);
        if (TO_POS) dst[p] = src[t];
        else dst[t] = src[p];
    }
}

template <bool TO_POS>
static int launch_permute(cudaStream_t st, int nv, int nelem, const int *pos, const double *src, double *dst,
                          int count, long long ss, long long ds) {
    const long long n = (long long)nv * nelem;
    const dim3 grid(grid_for(n, 256), count);
    if (n >= (1LL << 31)) /* word numbers and strides past 32 bits */
        permute_kernel<0, TO_POS, long long><<<grid, 256, 0, st>>>(nv, n, pos, src, dst, ss, ds);
    else if (nv == 9)
        permute_kernel<9, TO_POS, unsigned><<<grid, 256, 0, st>>>(nv, n, pos, src, dst, ss, ds);
    else
        permute_kernel<0, TO_POS, unsigned><<<grid, 256, 0, st>>>(nv, n, pos, src, dst, ss, ds);
    return (int)cudaGetLastError();
}

int launch_permute_to_pos(cudaStream_t st, int nv, int nelem, const int *pos_of_elem, const double *src_elem,
                          double *dst_pos, int count, long long src_stride, long long dst_stride) {
    return launch_permute<true>(st, nv, nelem, pos_of_elem, src_elem, dst_pos, count, src_stride, dst_stride);
}

int launch_permute_to_elem(cudaStream_t st, int nv, int nelem, const int *pos_of_elem, const double *src_pos,
                           double *dst_elem, int count, long long src_stride, long long dst_stride) {
    return launch_permute<false>(st, nv, nelem, pos_of_elem, src_pos, dst_elem, count, src_stride, dst_stride);
}

__global__ void permute_f32_to_elem_kernel(int nv, int nelem, const int *__restrict__ pos_of_elem,
                                           const float *__restrict__ src,
                                           double *__restrict__ dst) {
    long long n = (long long)nv * nelem;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        int e = (int)(t / nv), i = (int)(t - (long long)e * nv);
        dst[t] = (double)src[(long long)pos_of_elem[e] * nv + i];
    }
}

int launch_permute_f32_to_elem(cudaStream_t st, int nv, int nelem, const int *pos_of_elem,
                               const float *src_pos, double *dst_elem) {
    permute_f32_to_elem_kernel<<<grid_for((long long)nv * nelem, 256), 256, 0, st>>>(
        nv, nelem, pos_of_elem, src_pos, dst_elem);
    return (int)cudaGetLastError();
}

template <typename T>
__global__ void axpy_same_kernel(const T *__restrict__ d, T *__restrict__ U, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        U[t] += d[t];
}

__global__ void cast_kernel(const double *__restrict__ s, float *__restrict__ d, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        d[t] = (float)s[t];
}

int launch_cast_f64_f32(cudaStream_t st, const double *src, float *dst, long long n) {
    cast_kernel<<<grid_for(n, 256), 256, 0, st>>>(src, dst, n);
    return (int)cudaGetLastError();
}

__global__ void axpy_kernel(const float *__restrict__ d, double *__restrict__ U, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        U[t] += (double)d[t];
}

int launch_axpy_f32_f64(cudaStream_t st, const float *d, double *U, long long n) {
    axpy_kernel<<<grid_for(n, 256), 256, 0, st>>>(d, U, n);
    return (int)cudaGetLastError();
}

__global__ void axpy2_kernel(const float *__restrict__ c, const float *__restrict__ d,
                             double *__restrict__ U, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        U[t] += (double)c[t] + (double)d[t];
}

int launch_axpy_f64(cudaStream_t st, const double *d, double *U, long long n) {
    axpy_same_kernel<double><<<grid_for(n, 256), 256, 0, st>>>(d, U, n);
    return (int)cudaGetLastError();
}

int launch_axpy2_f32_f64(cudaStream_t st, const float *c, const float *d, double *U, long long n) {
    axpy2_kernel<<<grid_for(n, 256), 256, 0, st>>>(c, d, U, n);
    return (int)cudaGetLastError();
}

/* ====================================================== line factorization
 * Twisted block Thomas.  Each line is split into a top chain (cells
 * 0..m-1, eliminated downward as in src/okl/lineLU_v2.okl:58-182), a
 * bottom chain (cells n-1 down to m+1, the same elimination run upward) and
 * the twist cell m.  For chain step s >= 1 with A = block(row c_s, col
 * c_{s-1}) and C = block(row c_{s-1}, col c_s), both from the in-line face
 * between them (picked as in lineLU_v2.okl:116-117):
 *   Gam_{s-1} = Dinv_{s-1} C
 *   W         = D_s - A Gam_{s-1}          (block-Thomas pivot)
 *   Dinv_s    = W^-1   (in-place Gauss-Jordan, no pivoting, as the
 *                        reference's LU has none: lineLU_v2.okl:17-27)
 *   G_s       = Dinv_s A
 * and the chain's last Gam couples it to the twist cell, for which
 *   Dinv_tw = (D_m - A_tw Gam_top - C_tw Gam_bot)^-1
 * and Dinv_tw A_tw / Dinv_tw C_tw go in the G / Gam slots of the twist
 * position.  All are stored column-major like the input blocks.  The FP32
 * arrays, when given, are the FP64 results rounded once.
 *
 * What bounds it is the step along the chain (nine dependent pivots and two
 * products; a warp issues an FP64 operation every 4 cycles at best and a
 * reciprocal takes about 70) where lines are few, and the shuffles and
 * shared-memory reads of all the chains of an SM where they are many; the
 * bytes (six blocks a cell) come last.  So a warp runs three chains, nine
 * lanes each, a lane holding a 3x3 tile of its block: 54 reads for the 81
 * multiply-adds of three products and 14 shuffles for three pivots, where 27
 * lanes per chain took 108 and 48.  A CTA takes three lines: one such warp
 * for their top chains, one for the bottom chains, and beside each a helper
 * warp that copies the coming cells' blocks into shared memory, forms G (no
 * step waits for it) and writes the results, so that the chain warps run
 * nothing but the chain.
 * Few lines (at most seven for four SMs) leave the SM's pipes idle and the
 * step's latency counts alone; there 27 lanes per chain are faster (27
 * multiply-adds a product, a pivot's chain shorter by a fifth), one CTA per
 * line: fast_factor_few_kernel.  Measured with the cross-line copy (us; few /
 * this / a warp per chain doing everything and the copy behind it, the form
 * before): 100 lines of 256 cells 160 / 215 / 240, 255 of 256 199 / 219, 290 of
 * 256 234 / 216 / 279, 440 of 256 273 / 218 / 332, 600 of 640 920 / 777 / 1,020,
 * 1200 of 1280 4,210 / 2,840 / 3,750.
 */

struct FactorOut {
    double *Dinv, *G, *Gam;
    float *Dinv32, *G32, *Gam32;
    __device__ void put_dinv(size_t q, double v) const {
        if (Dinv) Dinv[q] = v;
        if (Dinv32) Dinv32[q] = (float)v;
    }
    __device__ void put_g(size_t q, double v) const {
        if (G) G[q] = v;
        if (G32) G32[q] = (float)v;
    }
    __device__ void put_gam(size_t q, double v) const {
        if (Gam) Gam[q] = v;
        if (Gam32) Gam32[q] = (float)v;
    }
};

/* X[q] = cross-line block of slot q = s*np16 + p (slot-major), or zeros: work
 * that needs nothing of the factorization, done by CTAs behind its own in the
 * same launch.  A chain leaves most of the memory system idle, so the copy
 * (235 us by itself at 600x640, 15 at 120x128) runs under it. */
struct XCopy {
    const int *xsrc;
    double *X; /* null: no copy */
    long long nslots;
    int first; /* the first CTA that copies */
};

/* a warp's share: four blocks at a time, their loads before their stores */
__device__ __forceinline__ void xcopy_part(const XCopy &xc, const double *__restrict__ O1,
                                           const double *__restrict__ O2) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const long long warps = (long long)(gridDim.x - xc.first) * nw;
    const long long w = (long long)(blockIdx.x - xc.first) * nw + (threadIdx.x >> 5);
    for (long long q0 = 4 * w; q0 < xc.nslots; q0 += 4 * warps) {
        double v[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int src = q0 + k < xc.nslots ? xc.xsrc[q0 + k] : -1;
            const double *x = ((src & 1) ? O2 : O1) + (size_t)(src >> 1) * NB + lane;
#pragma unroll
            for (int r = 0; r < 3; ++r) v[k][r] = (src >= 0 && lane + 32 * r < NB) ? __ldcs(x + 32 * r) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double *d = xc.X + (q0 + k) * NB + lane;
#pragma unroll
            for (int r = 0; r < 3; ++r)
                if (q0 + k < xc.nslots && lane + 32 * r < NB) d[32 * r] = v[k][r];
        }
    }
}

/* In-place Gauss-Jordan inverse of a 9x9 block distributed by columns:
 * lane j < 9 holds column j in w[0..8].  Pivot column p is broadcast with
 * shuffles; no pivoting, as the reference's LU has none. */
__device__ __forceinline__ void gj_invert_cols(double (&w)[NV], int j, unsigned *status) {
#pragma unroll
    for (int p = 0; p < NV; ++p) {
        double colp[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) colp[i] = __shfl_sync(FULL, w[i], p);
        const double piv = colp[p];
        if (threadIdx.x == 0 && !(fabs(piv) > 0.0 && isfinite(piv))) atomicOr(status, ST_PIVOT);
        const double r = __drcp_rn(piv);
        const bool isp = (j == p);
        const double t = w[p] * r;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (i != p) w[i] = isp ? -colp[i] * r : w[i] - colp[i] * t;
        w[p] = isp ? r : t;
    }
}

/* Gauss-Jordan inverse of a 9x9 block held by 27 lanes: lane j + 9g
 * (column j, row group g) holds rows 3g..3g+2 of column j in w[0..2].  For
 * pivot p, the pivot column's entries of this lane's rows come from lane
 * p + 9g, the pivot row's entry of this column from row group p / 3, and
 * the three entries that make the next pivot from their lanes; all lanes
 * then know the next pivot two operations after the reciprocal of this one.
 * Each entry is updated with the operations of gj_invert_cols (the pivot
 * column as 0 - column * r); no pivoting, as the reference's LU has none.
 * No branch stands in the chain: a pivot for which rcp_newton does not hold
 * (rcp_exception) is noted, and the block is then done again with the general
 * reciprocal.  Returns whether a pivot was zero or not finite. */
template <bool GENERAL>
__device__ __forceinline__ bool gj_pass_27(double (&w)[3], int j, int g) {
    bool bad = false;
    double piv = __shfl_sync(FULL, w[0], 0);
#pragma unroll
    for (int p = 0; p < NV; ++p) {
        const int pg = p / 3, pr = p % 3;
        const int n = p + 1 < NV ? p + 1 : p, ng = n / 3, nr = n % 3;
        const double dn = __shfl_sync(FULL, w[nr], n + 9 * ng);
        const double cn = __shfl_sync(FULL, w[nr], p + 9 * ng);
        const double rn = __shfl_sync(FULL, w[pr], n + 9 * pg);
        double colp[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) colp[k] = __shfl_sync(FULL, w[k], p + 9 * g);
        double t = __shfl_sync(FULL, w[pr], j + 9 * pg);
        if (j == p) {
            t = 1.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) w[k] = 0.0;
        }
        if (GENERAL)
            bad |= !(fabs(piv) > 0.0 && isfinite(piv));
        else
            bad |= rcp_exception(piv);
        const double r = GENERAL ? __drcp_rn(piv) : rcp_newton(piv);
        piv = dn - cn * (rn * r);
        t *= r;
#pragma unroll
        for (int k = 0; k < 3; ++k) w[k] -= colp[k] * t;
        if (g == pg) w[pr] = t;
    }
    return bad;
}

__device__ __noinline__ bool gj_general_27(double &a, double &b, double &c, int j, int g) {
    double w[3] = {a, b, c};
    const bool bad = gj_pass_27<true>(w, j, g);
    a = w[0];
    b = w[1];
    c = w[2];
    return bad;
}

__device__ __forceinline__ bool gj_invert_27(double (&w)[3], int j, int g) {
    double a = w[0], b = w[1], c = w[2];
    if (!gj_pass_27<false>(w, j, g)) return false; /* the pivots are the same in every lane */
    const bool bad = gj_general_27(a, b, c, j, g);
    w[0] = a;
    w[1] = b;
    w[2] = c;
    return bad;
}

/* the lane's three entries of c +- x y, x and y 9x9 blocks in shared memory
 * (r0 = 3g), the sum over q = 0..8 in order */
template <bool NEG>
__device__ __forceinline__ void product_27(double (&c)[3], const double *x, const double *y, int j, int r0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double v = y[q + NV * j];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (NEG)
                c[k] -= x[r0 + k + NV * q] * v;
            else
                c[k] += x[r0 + k + NV * q] * v;
        }
    }
}

__device__ __forceinline__ void entries_27(double (&c)[3], const double *x, int j, int r0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = x[r0 + k + NV * j];
}

__device__ __forceinline__ void put_27(const double (&c)[3], double *x, int j, int r0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) x[r0 + k + NV * j] = c[k];
}

/* shared memory of one chain: FEW_STAGES cells (A, C, D), two Dinv, two Gam
 * and the helper's G */
constexpr int FEW_STAGES = 6;
constexpr int FEW_WORDS = (3 * FEW_STAGES + 5) * NB;

/* The factorization of few lines (launch_fast_factor): one CTA per line,
 * warps 0 / 1 on its top / bottom chain, warp 2 helping both; the three meet
 * once per cell.  In step s a chain warp eliminates cell s (Gam_{s-1},
 * Dinv_s), the helper starts the copies of cell s + 4, forms and writes
 * G_{s-1}, Dinv_{s-1} and Gam_{s-2}, and waits for cell s + 1. */
__global__ void __launch_bounds__(96) fast_factor_few_kernel(
    int nline, const int *__restrict__ line_start, const int *__restrict__ line_len,
    const int *__restrict__ line_twist, const int *__restrict__ fsrc,
    const double *__restrict__ jacD, const double *__restrict__ O1, const double *__restrict__ O2,
    FactorOut out, XCopy xc, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int stages = FEW_STAGES, ahead = stages - 2;
    const int line = blockIdx.x;
    if (line >= nline) {
        xcopy_part(xc, O1, O2);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ps = line_start[line], n = line_len[line], m = line_twist[line];
    const int ptw = ps + n - 1;
    const int lens[2] = {m, n - 1 - m};
    const int maxlen = max(lens[0], lens[1]);
    auto base = [&](int chain) { return reinterpret_cast<double *>(smem) + chain * FEW_WORDS; };
    /* block `which` (0: A, 1: C, 2: D) of a cell's slot; the last Dinv, Gam */
    auto blk = [&](int chain, int slot, int which) { return base(chain) + (slot * 3 + which) * NB; };
    auto sM = [&](int chain, int s) { return base(chain) + (3 * stages + (s & 1)) * NB; };
    auto sGm = [&](int chain, int s) { return base(chain) + (3 * stages + 2 + (s & 1)) * NB; };
    auto turn = [&](int slot) { return slot + 1 == stages ? 0 : slot + 1; };
    /* lanes 27..31 repeat lanes 18..22 and store nothing */
    const bool act = lane < 27;
    const int j = act ? lane % 9 : lane - 27;
    const int g = act ? lane / 9 : 2, r0 = 3 * g;

    if (warp == 2) {
        /* the layout's row of a chain's cell c, entry `lane` of five (loaded in
         * one step, used in the next).  The cell after a chain's last (c ==
         * len) has C alone, which couples the chain to the twist; after the
         * longer chain's, the top slot takes the twist cell's own blocks (the
         * CTA's last phase). */
        auto row = [&](int chain, int c) {
            const int p = c < lens[chain] ? ps + (chain ? m : 0) + c : ptw;
            return lane < 5 ? fsrc[5 * p + lane] : 0;
        };
        auto copy = [&](int chain, int c, int slot, int v) {
            const int len = lens[chain];
            const int e = __shfl_sync(FULL, v, 0);
            const int f1 = __shfl_sync(FULL, v, 1), s1 = __shfl_sync(FULL, v, 2);
            const int f2 = __shfl_sync(FULL, v, 3), s2 = __shfl_sync(FULL, v, 4);
            const bool twist = c == maxlen + 1 && chain == 0;
            const double *q[3] = {nullptr, nullptr, nullptr};
            if (c < len || twist) q[2] = jacD + (size_t)e * NB;
            if (twist) {
                if (f1 >= 0) q[0] = (s1 ? O2 : O1) + (size_t)f1 * NB;
                if (f2 >= 0) q[1] = (s2 ? O2 : O1) + (size_t)f2 * NB;
            } else if (c < len && c > 0) {
                q[0] = (s1 ? O2 : O1) + (size_t)f1 * NB;
                q[1] = (s1 ? O1 : O2) + (size_t)f1 * NB;
            } else if (c == len && len > 0) {
                q[1] = ((chain ? s2 : s1) ? O1 : O2) + (size_t)(chain ? f2 : f1) * NB;
            }
            double *d = blk(chain, slot, 0) + lane;
#pragma unroll
            for (int which = 0; which < 3; ++which, d += NB) {
                if (q[which]) {
                    const double *x = q[which] + lane;
                    cp_async8(d, x);
                    cp_async8(d + 32, x + 32);
                    if (lane < NB - 64) cp_async8(d + 64, x + 64);
                } else if (twist) { /* a line's end without a neighbour */
                    d[0] = d[32] = 0.0;
                    if (lane < NB - 64) d[64] = 0.0;
                }
            }
        };
        for (int c = 0; c < ahead; ++c) {
            const int v0 = row(0, c), v1 = row(1, c);
            copy(0, c, c, v0);
            copy(1, c, c, v1);
            cp_async_commit();
        }
        int v0 = row(0, ahead), v1 = row(1, ahead);
        int into = ahead, done = stages - 1; /* slots of cells s + ahead and s - 1 */
        cp_async_wait<ahead - 1>(); /* cell 0 has landed */
        __syncthreads();
        for (int s = 0; s <= maxlen + 2; ++s) {
            copy(0, s + ahead, into, v0);
            copy(1, s + ahead, into, v1);
            cp_async_commit();
            into = turn(into);
            v0 = row(0, s + ahead + 1);
            v1 = row(1, s + ahead + 1);
            const int c = s - 1; /* the cell whose Dinv is done; Gam's is c - 1 */
            /* both chains' products side by side; what lies beyond a chain's
             * cells is not written out */
            double gt[2][3];
#pragma unroll
            for (int chain = 0; chain < 2; ++chain) {
                gt[chain][0] = gt[chain][1] = gt[chain][2] = 0.0;
                product_27<false>(gt[chain], sM(chain, c), blk(chain, done, 0), j, r0);
            }
#pragma unroll
            for (int chain = 0; chain < 2; ++chain) {
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (c == 0) gt[chain][k] = 0.0;
                if (act) put_27(gt[chain], base(chain) + (3 * stages + 4) * NB, j, r0);
            }
            __syncwarp();
#pragma unroll
            for (int chain = 0; chain < 2; ++chain) {
                const int len = lens[chain];
                const size_t q = (size_t)(ps + (chain ? m : 0) + c) * NB;
                const double *go = base(chain) + (3 * stages + 4) * NB, *di = sM(chain, c);
                if (c >= 0 && c < len) {
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        const int e = lane + 32 * r;
                        if (e < NB) {
                            out.put_dinv(q + e, di[e]);
                            out.put_g(q + e, go[e]);
                        }
                    }
                }
                if (c >= 1 && c - 1 < len) {
                    const double *gm = sGm(chain, c);
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        const int e = lane + 32 * r;
                        if (e < NB) out.put_gam(q - NB + e, gm[e]);
                    }
                }
            }
            __syncwarp();
            done = turn(done);
            cp_async_wait<ahead - 1>(); /* cell s + 1 */
            __syncthreads();
        }
        cp_async_wait<0>();
        __syncthreads(); /* the twist's blocks for warp 0 */
        return;
    }

    const int len = lens[warp];
    bool bad = false;
    int slot = 0; /* of cell s */
    __syncthreads();
    for (int s = 0; s <= maxlen + 2; ++s) {
        if (s <= len) {
            if (s > 0) {
                double gm[3] = {0.0, 0.0, 0.0};
                product_27<false>(gm, sM(warp, s - 1), blk(warp, slot, 1), j, r0);
                if (act) put_27(gm, sGm(warp, s), j, r0);
                __syncwarp();
            }
            if (s < len) {
                double w[3];
                entries_27(w, blk(warp, slot, 2), j, r0);
                if (s > 0) product_27<true>(w, blk(warp, slot, 0), sGm(warp, s), j, r0);
                bad = gj_invert_27(w, j, g) || bad;
                if (act) put_27(w, sM(warp, s), j, r0);
                __syncwarp();
            }
        }
        slot = turn(slot);
        __syncthreads();
    }
    __syncthreads(); /* the twist's blocks have landed */
    /* ---------------- the twist cell: warp 0, the chains' last Gam where their
     * step s = len left it */
    if (warp == 0) {
        const int tw = (maxlen + 1) % stages;
        const double *A = blk(0, tw, 0), *C = blk(0, tw, 1);
        double w[3];
        entries_27(w, blk(0, tw, 2), j, r0);
        if (lens[0] > 0) product_27<true>(w, A, sGm(0, lens[0]), j, r0);
        if (lens[1] > 0) product_27<true>(w, C, sGm(1, lens[1]), j, r0);
        bad = gj_invert_27(w, j, g) || bad;
        double *inv = sM(0, 0);
        if (act) put_27(w, inv, j, r0);
        __syncwarp();
        double ga[3] = {0.0, 0.0, 0.0}, gc[3] = {0.0, 0.0, 0.0};
        product_27<false>(ga, inv, A, j, r0);
        product_27<false>(gc, inv, C, j, r0);
        if (act) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const size_t q = (size_t)ptw * NB + r0 + k + NV * j;
                out.put_dinv(q, w[k]);
                out.put_g(q, ga[k]);
                out.put_gam(q, gc[k]);
            }
        }
    }
    if (bad && lane == 0) atomicOr(status, ST_PIVOT);
}

/* Gauss-Jordan inverse of three 9x9 blocks by 27 lanes: lane (a, b) of the
 * nine from `base` holds rows 3a..3a+2, columns 3b..3b+2 of its block.  For
 * pivot p each lane takes the pivot, the pivot column's entries of its rows
 * and the pivot row's of its columns.  Each entry is updated with the
 * operations of gj_invert_cols (the pivot column as 0 - column * r); no
 * pivoting, as the reference's LU has none.  No branch stands in the chain: a
 * pivot for which rcp_newton does not hold (rcp_exception) is noted, and the
 * blocks are then done again with the general reciprocal.  Returns
 * whether a pivot of the lane's block was zero or not finite. */
template <bool GENERAL>
__device__ __forceinline__ bool gj_pass(double (&w)[3][3], int a, int b, int base) {
    bool bad = false;
#pragma unroll
    for (int p = 0; p < NV; ++p) {
        const int pa = p / 3, pk = p % 3;
        const double piv = __shfl_sync(FULL, w[pk][pk], base + 4 * pa);
        double colp[3], t[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) colp[k] = __shfl_sync(FULL, w[k][pk], base + 3 * a + pa);
#pragma unroll
        for (int l = 0; l < 3; ++l) t[l] = __shfl_sync(FULL, w[pk][l], base + 3 * pa + b);
        if (GENERAL)
            bad |= !(fabs(piv) > 0.0 && isfinite(piv));
        else
            bad |= rcp_exception(piv);
        const double r = GENERAL ? __drcp_rn(piv) : rcp_newton(piv);
        if (b == pa) {
            t[pk] = 1.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) w[k][pk] = 0.0;
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) t[l] *= r;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l) w[k][l] -= colp[k] * t[l];
        if (a == pa) {
#pragma unroll
            for (int l = 0; l < 3; ++l) w[pk][l] = t[l];
        }
    }
    return bad;
}

/* a block's tiles through memory, out of line: x[9] per lane */
__device__ __noinline__ bool gj_general(double *x, int a, int b, int base) {
    double w[3][3];
#pragma unroll
    for (int k = 0; k < 9; ++k) w[k / 3][k % 3] = x[k];
    const bool bad = gj_pass<true>(w, a, b, base);
#pragma unroll
    for (int k = 0; k < 9; ++k) x[k] = w[k / 3][k % 3];
    return bad;
}

/* W from the lane's tile in shared memory form: `again` rebuilds the tile
 * (the general pass starts from the block itself); `use`: the lane's chain
 * has a block here (the lanes of the others take part in the shuffles) */
template <typename Build>
__device__ __forceinline__ bool gj_invert_tile(double (&w)[3][3], int a, int b, int base, bool use,
                                               Build &&again) {
    const bool odd = gj_pass<false>(w, a, b, base);
    if (!__any_sync(FULL, use && odd)) return false;
    again(w);
    double x[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) x[k] = w[k / 3][k % 3];
    const bool bad = gj_general(x, a, b, base);
#pragma unroll
    for (int k = 0; k < 9; ++k) w[k / 3][k % 3] = x[k];
    return use && bad;
}

/* lane (a, b)'s 3x3 tile of c +- x y; x and y are 9x9 blocks in shared
 * memory, the sum over q = 0..8 in order */
template <bool NEG>
__device__ __forceinline__ void tile_product(double (&c)[3][3], const double *x, const double *y, int a,
                                             int b) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        double r[3], s[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            r[k] = x[3 * a + k + NV * q];
            s[k] = y[q + NV * (3 * b + k)];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                if (NEG)
                    c[k][l] -= r[k] * s[l];
                else
                    c[k][l] += r[k] * s[l];
            }
    }
}

__device__ __forceinline__ void tile_zero(double (&c)[3][3]) {
#pragma unroll
    for (int k = 0; k < 9; ++k) c[k / 3][k % 3] = 0.0;
}

__device__ __forceinline__ void tile_load(double (&c)[3][3], const double *x, int a, int b) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) c[k][l] = x[3 * a + k + NV * (3 * b + l)];
}

__device__ __forceinline__ void tile_store(const double (&c)[3][3], double *x, int a, int b) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) x[3 * a + k + NV * (3 * b + l)] = c[k][l];
}

/* blocks of a group of three lie FB words apart (81 and 8 of padding), so
 * that the nine rows (or columns) that the 27 lanes read at once lie in
 * different banks */
constexpr int FB = NB + 8;
/* shared memory of three chains: `stages` cells (A, C, D), two Dinv, two Gam
 * and the helper's G */
__host__ __device__ constexpr int fac_pair_words(int stages) { return (3 * stages + 5) * 3 * FB; }

/* CTA: lines 3 * blockIdx.x + g, g = 0..2; warps 0 / 1 run their top / bottom
 * chains, warps 2 / 3 help them; a pair of warps meets at its own barrier
 * once per cell.  In step s the chain warp eliminates cell s (Gam_{s-1},
 * Dinv_s), the helper starts the copies of cell s + stages - 2, forms and
 * writes G_{s-1}, Dinv_{s-1} and Gam_{s-2}, and waits for cell s + 1. */
__global__ void __launch_bounds__(128, 3) fast_factor_kernel(
    int nline, int stages, int nsm, const int *__restrict__ line_start, const int *__restrict__ line_len,
    const int *__restrict__ line_twist, const int *__restrict__ fsrc,
    const double *__restrict__ jacD, const double *__restrict__ O1, const double *__restrict__ O2,
    FactorOut out, XCopy xc, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    if ((int)blockIdx.x * 3 >= nline) {
        xcopy_part(xc, O1, O2);
        return;
    }
    /* a warp's scheduler goes by its number in the CTA: every other CTA of an
     * SM (they come round every nsm) has its chain warps on the schedulers
     * where the others' helpers are */
    const int warp = (threadIdx.x >> 5) ^ ((blockIdx.x / nsm & 1) << 1), lane = threadIdx.x & 31;
    const int chain = warp & 1; /* 0: top, 1: bottom */
    /* lanes 27..31 repeat lanes 18..22 and write nothing */
    const bool lact = lane < 27;
    const int ln = lact ? lane : lane - 9;
    const int g = ln / 9, l9 = ln % 9, a = l9 / 3, b = l9 % 3;
    const int line = 3 * blockIdx.x + g;
    const bool have = line < nline, act = lact && have;
    const int lc = have ? line : nline - 1;
    const int ps = line_start[lc], n = line_len[lc], m = line_twist[lc];
    const int ptw = ps + n - 1;
    const int len = have ? (chain ? n - 1 - m : m) : 0;
    const int cs = ps + (chain ? m : 0);
    int maxlen = len;
#pragma unroll
    for (int k = 0; k < 3; ++k) maxlen = max(maxlen, __shfl_sync(FULL, len, 9 * k));
    double *pair = reinterpret_cast<double *>(smem) + chain * fac_pair_words(stages) + g * FB;
    /* block `which` (0: A, 1: C, 2: D) of a cell's slot; the last Dinv, Gam */
    auto blk = [&](int slot, int which) { return pair + (slot * 3 + which) * 3 * FB; };
    auto sM = [&](int s) { return pair + (3 * stages + (s & 1)) * 3 * FB; };
    auto sGm = [&](int s) { return pair + (3 * stages + 2 + (s & 1)) * 3 * FB; };
    auto turn = [&](int slot) { return slot + 1 == stages ? 0 : slot + 1; };
    auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + chain) : "memory"); };

    if (warp >= 2) {
        const int ahead = stages - 2;
        double *sGo = pair + (3 * stages + 4) * 3 * FB;
        /* the layout's row of the chain's cell c (loaded in one step, used in
         * the next).  The cell after a chain's last (c == len) has C alone,
         * which couples the chain to the twist; after the longest chain's, the
         * top slots take the twist cells' own blocks (the CTA's last phase). */
        struct Src {
            int e, f1, s1, f2, s2;
        };
        auto row = [&](int c) {
            const int *q = fsrc + 5 * (c < len ? cs + c : ptw);
            return Src{q[0], q[1], q[2], q[3], q[4]};
        };
        auto copy = [&](int c, int slot, const Src &r) {
            const bool twist = c == maxlen + 1 && chain == 0 && have;
            const double *q[3] = {nullptr, nullptr, nullptr};
            if (c < len || twist) q[2] = jacD + (size_t)r.e * NB;
            if (twist) {
                if (r.f1 >= 0) q[0] = (r.s1 ? O2 : O1) + (size_t)r.f1 * NB;
                if (r.f2 >= 0) q[1] = (r.s2 ? O2 : O1) + (size_t)r.f2 * NB;
            } else if (c < len && c > 0) {
                q[0] = (r.s1 ? O2 : O1) + (size_t)r.f1 * NB;
                q[1] = (r.s1 ? O1 : O2) + (size_t)r.f1 * NB;
            } else if (c == len && len > 0) {
                q[1] = ((chain ? r.s2 : r.s1) ? O1 : O2) + (size_t)(chain ? r.f2 : r.f1) * NB;
            }
            if (lact) {
#pragma unroll
                for (int which = 0; which < 3; ++which) {
                    double *d = blk(slot, which) + l9;
                    if (q[which]) {
#pragma unroll
                        for (int k = 0; k < NV; ++k) cp_async8(d + NV * k, q[which] + l9 + NV * k);
                    } else if (twist) { /* a line's end without a neighbour */
#pragma unroll
                        for (int k = 0; k < NV; ++k) d[NV * k] = 0.0;
                    }
                }
            }
            cp_async_commit();
        };
        auto wait_next = [&]() { /* all but the newest ahead - 1 cells */
            if (ahead == 4)
                cp_async_wait<3>();
            else
                cp_async_wait<1>();
        };
        for (int c = 0; c < ahead; ++c) copy(c, c, row(c));
        Src nxt = row(ahead);
        int into = ahead, done = stages - 1; /* slots of cells s + ahead and s - 1 */
        wait_next();
        meet();
        for (int s = 0; s <= maxlen + 2; ++s) {
            copy(s + ahead, into, nxt);
            into = turn(into);
            nxt = row(s + ahead + 1);
            const int c = s - 1; /* the cell whose Dinv is done; Gam's is c - 1 */
            double gt[3][3];
            tile_zero(gt);
            if (c > 0) tile_product<false>(gt, sM(c), blk(done, 0), a, b);
            if (lact) tile_store(gt, sGo, a, b);
            __syncwarp();
            if (act && c >= 0 && c < len) {
                const size_t q = (size_t)(cs + c) * NB + l9;
                const double *di = sM(c) + l9, *go = sGo + l9;
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    out.put_dinv(q + NV * k, di[NV * k]);
                    out.put_g(q + NV * k, go[NV * k]);
                }
            }
            if (act && c >= 1 && c - 1 < len) {
                const size_t q = (size_t)(cs + c - 1) * NB + l9;
                const double *gm = sGm(c) + l9;
#pragma unroll
                for (int k = 0; k < NV; ++k) out.put_gam(q + NV * k, gm[NV * k]);
            }
            __syncwarp();
            done = turn(done);
            wait_next();
            meet();
        }
        cp_async_wait<0>();
        __syncthreads(); /* the twists' blocks for warp 0 */
        return;
    }

    bool bad = false;
    int slot = 0; /* of cell s */
    meet();
    for (int s = 0; s <= maxlen + 2; ++s) {
        if (s <= maxlen) {
            if (s > 0) {
                double gm[3][3];
                tile_zero(gm);
                tile_product<false>(gm, sM(s - 1), blk(slot, 1), a, b);
                if (lact && s <= len) tile_store(gm, sGm(s), a, b);
                __syncwarp();
            }
            double w[3][3];
            auto pivot = [&](double(&x)[3][3]) {
                tile_load(x, blk(slot, 2), a, b);
                if (s > 0) tile_product<true>(x, blk(slot, 0), sGm(s), a, b);
            };
            pivot(w);
            bad = gj_invert_tile(w, a, b, 9 * g, have && s < len, pivot) || bad;
            if (lact && s < len) tile_store(w, sM(s), a, b);
            __syncwarp();
        }
        slot = turn(slot);
        meet();
    }
    __syncthreads(); /* both chains are done, the twists' blocks have landed */
    /* ---------------- the twist cells: warp 0, the chains' last Gam where
     * their step s = len left it */
    if (warp == 0) {
        const int tw = (maxlen + 1) % stages, lenb = have ? n - 1 - m : 0;
        const double *A = blk(tw, 0), *C = blk(tw, 1), *gt = sGm(len);
        const double *gb = pair + fac_pair_words(stages) + (3 * stages + 2 + (lenb & 1)) * 3 * FB;
        double w[3][3];
        auto pivot = [&](double(&x)[3][3]) {
            tile_load(x, blk(tw, 2), a, b);
            if (len > 0) tile_product<true>(x, A, gt, a, b);
            if (lenb > 0) tile_product<true>(x, C, gb, a, b);
        };
        pivot(w);
        __syncwarp();
        bad = gj_invert_tile(w, a, b, 9 * g, have, pivot) || bad;
        double *inv = pair + (3 * stages + 4) * 3 * FB; /* the helper is done with it */
        if (lact) tile_store(w, inv, a, b);
        __syncwarp();
        double ga[3][3], gc[3][3];
        tile_zero(ga);
        tile_zero(gc);
        tile_product<false>(ga, inv, A, a, b);
        tile_product<false>(gc, inv, C, a, b);
        if (act) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const size_t q = (size_t)ptw * NB + 3 * a + k + NV * (3 * b + l);
                    out.put_dinv(q, w[k][l]);
                    out.put_g(q, ga[k][l]);
                    out.put_gam(q, gc[k][l]);
                }
        }
    }
    if (bad && act) atomicOr(status, ST_PIVOT);
}

/* The factorization of many short lines: one warp per line, its top chain, its
 * bottom chain and its twist cell one after the other, the blocks in registers
 * a cell ahead.  Nothing has to be filled or drained, and 20 lines an SM hide
 * each other's latencies, where the pairs of warps above spend three steps a
 * line at the ends of their chains and hold nine. */
__global__ void __launch_bounds__(32) fast_factor_short_kernel(
    int nline, const int *__restrict__ line_start, const int *__restrict__ line_len,
    const int *__restrict__ line_twist, const int *__restrict__ fsrc,
    const double *__restrict__ jacD, const double *__restrict__ O1, const double *__restrict__ O2,
    FactorOut out, XCopy xc, unsigned *status) {
    __shared__ double sM[NB], sA[NB], sC[NB], sGm[2][NB];
    const int line = blockIdx.x;
    if (line >= nline) {
        xcopy_part(xc, O1, O2);
        return;
    }
    const int lane = threadIdx.x;
    /* lanes 27..31 repeat lanes 18..22 and store nothing */
    const bool act = lane < 27;
    const int j = act ? lane % 9 : lane - 27;
    const int g = act ? lane / 9 : 2, r0 = 3 * g;
    const int ps = line_start[line], n = line_len[line], m = line_twist[line];
    const int ptw = ps + n - 1;
    double an[3], cn[3], dn[3];
    auto load = [&](double (&v)[3], const double *x) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = x[r0 + k + NV * j];
    };
    auto clear = [&](double (&v)[3]) { v[0] = v[1] = v[2] = 0.0; };
    /* the blocks of step s of a chain: A, C and D of its cell, C alone (the
     * coupling to the twist) behind the last cell */
    auto fetch = [&](int chain, int cs, int len, int s) {
        const int *q = fsrc + 5 * (s < len ? cs + s : ptw);
        const int at = s < len || !chain ? 1 : 3;
        const size_t f = (size_t)q[at] * NB;
        const bool second = q[at + 1] != 0;
        load(cn, (second ? O1 : O2) + f);
        if (s < len) {
            load(an, (second ? O2 : O1) + f);
            load(dn, jacD + (size_t)q[0] * NB);
        }
    };
    auto put = [&](const double (&v)[3], size_t p, auto &&store) {
        if (act) {
#pragma unroll
            for (int k = 0; k < 3; ++k) store(p * NB + r0 + k + NV * j, v[k]);
        }
    };
    auto dinv = [&](size_t q, double v) { out.put_dinv(q, v); };
    auto gq = [&](size_t q, double v) { out.put_g(q, v); };
    auto gamq = [&](size_t q, double v) { out.put_gam(q, v); };
    bool bad = false;
    for (int chain = 0; chain < 2; ++chain) {
        const int len = chain ? n - 1 - m : m, cs = ps + (chain ? m : 0);
        if (len == 0) continue;
        double w[3], x[3];
        load(w, jacD + (size_t)fsrc[5 * cs] * NB);
        fetch(chain, cs, len, 1);
        for (int s = 0;; ++s) {
            if (s > 0) {
                const double d[3] = {dn[0], dn[1], dn[2]};
                if (act) {
                    put_27(cn, sC, j, r0);
                    put_27(an, sA, j, r0);
                }
                if (s < len) fetch(chain, cs, len, s + 1);
                __syncwarp();
                clear(x);
                product_27<false>(x, sM, sC, j, r0);
                put(x, cs + s - 1, gamq);
                if (act) put_27(x, sGm[chain], j, r0);
                __syncwarp();
                if (s == len) break;
#pragma unroll
                for (int k = 0; k < 3; ++k) w[k] = d[k];
                product_27<true>(w, sA, sGm[chain], j, r0);
            }
            bad = gj_invert_27(w, j, g) || bad;
            if (act) put_27(w, sM, j, r0);
            put(w, cs + s, dinv);
            __syncwarp();
            clear(x);
            if (s > 0) product_27<false>(x, sM, sA, j, r0);
            put(x, cs + s, gq);
            __syncwarp(); /* sA and sC are written again */
        }
        __syncwarp(); /* and sM */
    }
    /* ---------------- the twist cell */
    const int *q = fsrc + 5 * ptw;
    double w[3];
    load(w, jacD + (size_t)q[0] * NB);
    clear(an);
    clear(cn);
    if (q[1] >= 0) load(an, (q[2] ? O2 : O1) + (size_t)q[1] * NB);
    if (q[3] >= 0) load(cn, (q[4] ? O2 : O1) + (size_t)q[3] * NB);
    if (act) {
        put_27(an, sA, j, r0);
        put_27(cn, sC, j, r0);
    }
    __syncwarp();
    if (m > 0) product_27<true>(w, sA, sGm[0], j, r0);
    if (n - 1 - m > 0) product_27<true>(w, sC, sGm[1], j, r0);
    bad = gj_invert_27(w, j, g) || bad;
    if (act) put_27(w, sM, j, r0);
    __syncwarp();
    double ga[3] = {0.0, 0.0, 0.0}, gc[3] = {0.0, 0.0, 0.0};
    product_27<false>(ga, sM, sA, j, r0);
    product_27<false>(gc, sM, sC, j, r0);
    put(w, ptw, dinv);
    put(ga, ptw, gq);
    put(gc, ptw, gamq);
    if (bad && lane == 0) atomicOr(status, ST_PIVOT);
}

/* cells in shared memory per pair of warps: six (copies four steps ahead)
 * where the CTAs of three lines are at most two per SM, else four, which
 * keeps three CTAs resident */
static int fac_stages(const FastLayout &L, int nsm) { return (L.nline + 2) / 3 <= 2 * nsm ? 6 : 4; }

/* Whether the lines are short: sixteen cells on average, and the longest, at
 * 1.65 us a cell on its one warp, done while the others are (0.3 us a cell and
 * SM) or before a chain of half as many cells and its ends would be.  Measured
 * (us, with the cross-line copy; this / three lines a CTA / a warp per chain, a
 * launch for the twists and one for the copy, the form before): 30000x1 99 /
 * 212 / 206, 50000x3 300 / 552 / 474, 600x3 12 / 16 / 25, 20000x8 320 / 401 /
 * 377, 3000x13 92 / 99 / 123, 9000 lines of 1 to 11 117 / 181 / 164; 3000x50
 * 328 / 307 / 364, one line of 500 and 9000 of 3 824 / 425 / 462. */
static bool fac_short(const FastLayout &L, int nsm) {
    const double longest = L.max_len, cells = L.cells;
    return cells <= 16.0 * L.nline && 1.65 * longest <= std::max(0.3 * cells / nsm, 1.7 * (0.5 * longest + 3.0));
}

int launch_fast_factor(cudaStream_t st, const FastLayout &L, const double *jacD, const double *O1,
                       const double *O2, double *Dinv, double *G, double *Gam, float *Dinv32,
                       float *G32, float *Gam32, double *X, unsigned *status) {
    if (L.nv != NV) return (int)cudaErrorInvalidValue;
    FactorOut out{Dinv, G, Gam, Dinv32, G32, Gam32};
    XCopy xc{L.xsrc, X, (long long)L.np16 * L.nx, 0};
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (nsm < 1) nsm = 148;
    /* CTAs that copy, each with at least a few blocks.  While the
     * factorization's CTAs are at most one per SM: one per SM, so that all are
     * resident at once and the chains stay spread over the SMs (360x384: 1.07
     * of the time with half as many, 1.5 with twice as many, which fill the SMs
     * and put two factorizing CTAs on one; 120x128: 1.01 and 1.2).  Else four
     * per SM, which take their places as they come free (600x640: 0.88 of the
     * time with one per SM, 1200x640: 0.75). */
    const bool few = 4 * (long long)L.nline <= 7 * (long long)nsm;
    const int nfac = (L.nline + 2) / 3;
    const int most = few || nfac <= nsm ? nsm : 4 * nsm;
    const int copiers = X ? (int)std::min<long long>(most, (xc.nslots + 63) / 64) : 0;
    if (fac_short(L, nsm)) {
        xc.first = L.nline;
        const int warps = X ? (int)std::min<long long>(32LL * nsm, (xc.nslots + 15) / 16) : 0;
        fast_factor_short_kernel<<<L.nline + warps, 32, 0, st>>>(L.nline, L.line_start, L.line_len, L.line_twist,
                                                                 L.fsrc, jacD, O1, O2, out, xc, status);
        return (int)cudaGetLastError();
    }
    if (few) {
        xc.first = L.nline;
        fast_factor_few_kernel<<<L.nline + copiers, 96, 2 * FEW_WORDS * sizeof(double), st>>>(
            L.nline, L.line_start, L.line_len, L.line_twist, L.fsrc, jacD, O1, O2, out, xc, status);
        return (int)cudaGetLastError();
    }
    const int stages = fac_stages(L, nsm);
    const size_t smem = 2 * (size_t)fac_pair_words(stages) * sizeof(double);
    const int rc = smem_raise((const void *)fast_factor_kernel, smem);
    if (rc) return rc;
    xc.first = nfac;
    fast_factor_kernel<<<xc.first + copiers, 128, smem, st>>>(L.nline, stages, nsm, L.line_start, L.line_len,
                                                              L.line_twist, L.fsrc, jacD, O1, O2, out, xc,
                                                              status);
    return (int)cudaGetLastError();
}

/* DX[q] = Dinv(p) X(q) for slot q = s*np16 + p, rounded once to FP32, from
 * the FP64 inverse and the original FP64 face block; one warp per slot */
__global__ void __launch_bounds__(256) fast_dx_kernel(long long nslots, int np16,
                                                      const int *__restrict__ xsrc,
                                                      const double *__restrict__ Dinv,
                                                      const double *__restrict__ O1,
                                                      const double *__restrict__ O2,
                                                      float *__restrict__ DX) {
    __shared__ double sm[8][2 * NB];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    double *sD = sm[wb], *sX = sm[wb] + NB;
    for (long long q = w0; q < nslots; q += nw) {
        const int src = xsrc[q];
        const long long p = q % np16;
        __syncwarp();
        for (int t = lane; t < NB; t += 32) {
            sD[t] = Dinv[p * NB + t];
            sX[t] = src >= 0 ? ((src & 1) ? O2 : O1)[(size_t)(src >> 1) * NB + t] : 0.0;
        }
        __syncwarp();
        for (int t = lane; t < NB; t += 32) {
            const int i = t % NV, j = t / NV;
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < NV; ++k) acc += sD[i + NV * k] * sX[k + NV * j];
            DX[q * NB + t] = (float)acc;
        }
    }
}

int launch_fast_dx(cudaStream_t st, const FastLayout &L, const double *Dinv, const double *O1,
                   const double *O2, float *DX) {
    const long long nslots = (long long)L.np16 * L.nx;
    if (nslots == 0) return 0;
    fast_dx_kernel<<<grid_for(nslots * 32, 256), 256, 0, st>>>(nslots, L.np16, L.xsrc, Dinv, O1, O2, DX);
    return (int)cudaGetLastError();
}

/* ================================================ residual -> Thomas RHS
 * Tiles of RES_TILE positions, each staged by one phase of the CTA's bulk
 * copy barrier; the single-system launches are persistent (as many CTAs
 * as fit, tiles round-robin per CTA).  Per tile:
 *   mode 0:  R = Rsrc (a residual already in position order)
 *   mode 1:  R = sum over slots X_slot dU[xnbr_slot]   (R_new = O dU)
 * then b = -Dinv R.  Thread t < 144 owns (cell c = t % 16, row i = t / 16):
 * with blocks 81 doubles apart, the 16 cells of a half-warp hit 16
 * distinct bank pairs, so the shared-memory reads are conflict-free.
 * X and xnbr are slot-major ([slot][position]) for the same reason.
 * Every tile writes its sum R^2; the last CTA to finish (atomic ticket)
 * adds the partials in tile order and, when asked, records the norm, the
 * sweep count and the graph's loop condition.
 */
constexpr int RES_THREADS_FAST = 160;

int fast_resid_grid(int np16) { return np16 / RES_TILE > 0 ? np16 / RES_TILE : 1; }

template <typename T>
__host__ __device__ inline size_t resid_smem_bytes(int nx) {
    const int nxa = nx > 0 ? nx : 1;
    return 128 + (size_t)RES_TILE * NB * sizeof(T) * (1 + nx) +
           (size_t)nxa * RES_TILE * NV * sizeof(T) + (size_t)RES_TILE * NV * sizeof(T) * 2;
}

/* The residual kernels' staging barrier sits at the start of the dynamic
 * shared memory; it is initialised once per CTA, and each tile the CTA
 * processes completes one phase of it. */
__device__ __forceinline__ uint64_t *resid_bar_init() {
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    return bar;
}

/* The products of a row of a block (column-major, at its entry of column 0)
 * with a vector, in three sums: a_j takes products j, j + 3, j + 6.
 * open_sums: the first six, products j and j + 3 opening a_j, the latter
 * rounded by itself.  (The sums as an array: the batch residual spilled.) */
template <typename T>
__device__ __forceinline__ void open_sums(T &a0, T &a1, T &a2, const T *row, const T *v) {
    a0 = fma_rn(row[0], v[0], mul_rn(row[27], v[3]));
    a1 = fma_rn(row[9], v[1], mul_rn(row[36], v[4]));
    a2 = fma_rn(row[18], v[2], mul_rn(row[45], v[5]));
}

/* the last three products */
template <typename T>
__device__ __forceinline__ void close_sums(T &a0, T &a1, T &a2, const T *row, const T *v) {
    a0 = fma_rn(row[54], v[6], a0);
    a1 = fma_rn(row[63], v[7], a1);
    a2 = fma_rn(row[72], v[8], a2);
}

/* all nine */
template <typename T>
__device__ __forceinline__ void add_products(T &a0, T &a1, T &a2, const T *row, const T *v) {
    a0 = fma_rn(row[0], v[0], a0);
    a1 = fma_rn(row[9], v[1], a1);
    a2 = fma_rn(row[18], v[2], a2);
    a0 = fma_rn(row[27], v[3], a0);
    a1 = fma_rn(row[36], v[4], a1);
    a2 = fma_rn(row[45], v[5], a2);
    close_sums(a0, a1, a2, row, v);
}

/* -(row of Dinv) . R for one (cell, row): dr points at entry (row, 0) of
 * the cell's column-major block, rv at the cell's R; three accumulators,
 * the order every b = -Dinv R of this file uses */
template <typename T>
__device__ __forceinline__ T neg_dinv_row(const T *dr, const T *rv) {
    T a0, a1, a2;
    open_sums(a0, a1, a2, dr, rv);
    close_sums(a0, a1, a2, dr, rv);
    return -(a0 + (a1 + a2));
}

/* One tile (positions blk*RES_TILE ..) with the staging barrier's phase of
 * the given parity.  Returns false (status set, copies landed) when the
 * wait for the tile's bulk copies ran out of time. */
template <typename T>
__device__ __forceinline__ bool fast_resid_body(
    int nx, int np16, int mode, const T *__restrict__ Dinv, const T *__restrict__ X,
    const int *__restrict__ xnbr, const T *__restrict__ dU, const T *__restrict__ Rsrc,
    T *__restrict__ b, T *__restrict__ Uacc, const NormSink &ns, unsigned *status, int blk,
    uint64_t *bar, uint32_t parity, const int *nbr_pre = nullptr, const T *__restrict__ Uin = nullptr) {
    extern __shared__ __align__(128) unsigned char smem[];
    T *sD = reinterpret_cast<T *>(smem + 128);
    T *sX = sD + RES_TILE * NB;
    const int nxa = nx > 0 ? nx : 1;
    T *sg = sX + nx * RES_TILE * NB;
    T *sr = sg + nxa * RES_TILE * NV;
    T *sb = sr + RES_TILE * NV;
    const int p0 = blk * RES_TILE;
    const int tid = threadIdx.x;
    const int c = tid % RES_TILE, i = tid / RES_TILE;
    const bool act = tid < RES_TILE * NV;
    const uint32_t szD = RES_TILE * NB * sizeof(T), szR = RES_TILE * NV * sizeof(T);

    if (tid == 0) {
        const uint64_t pol = policy_evict_first();
        const bool noD = mode == 3 || mode == 4;
        const uint32_t bytes = (noD ? 0u : szD) + (mode >= 1 ? nx * szD : szR);
        mbar_arrive_expect_tx(bar, bytes);
        if (!noD) bulk_g2s_hint(sD, Dinv + (size_t)p0 * NB, szD, bar, pol);
        if (mode >= 1) {
            for (int s = 0; s < nx; ++s)
                bulk_g2s_hint(sX + s * RES_TILE * NB, X + ((size_t)s * np16 + p0) * NB, szD, bar, pol);
        } else {
            bulk_g2s(sr, Rsrc + (size_t)p0 * NV, szR, bar);
        }
    }
    if (act && Uacc) {
        /* modes 1, 3: U += dU of this tile (the Thomas kernel leaves U to
         * this kernel), the previous U read from Uin when set; mode 0:
         * U = 0, the start of a sweep sequence */
        const size_t q = (size_t)p0 * NV + tid;
        Uacc[q] = (mode >= 1) ? (Uin ? Uin[q] : Uacc[q]) + dU[q] : T(0);
    }
    if (mode >= 1 && act) {
        /* neighbour dU gathers overlap the bulk copies (their indices
         * loaded during the previous tile when the caller prefetched them) */
        if (nbr_pre) {
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if (s < nx) {
                    const int nb = nbr_pre[s];
                    sg[(s * RES_TILE + c) * NV + i] = (nb >= 0) ? dU[(size_t)nb * NV + i] : T(0);
                }
            }
        } else {
            for (int s = 0; s < nx; ++s) {
                const int nb = xnbr[(size_t)s * np16 + p0 + c];
                sg[(s * RES_TILE + c) * NV + i] = (nb >= 0) ? dU[(size_t)nb * NV + i] : T(0);
            }
        }
    }
    const bool ok = mbar_wait(bar, parity);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicOr(status, ST_TIMEOUT);
            mbar_wait(bar, parity, 1LL << 28); /* let the copies land before the CTA retires */
        }
        return false;
    }
    T r = T(0);
    if (mode >= 1) {
        if (act) {
            T a0 = T(0), a1 = T(0), a2 = T(0);
            for (int s = 0; s < nx; ++s) {
                const T *xr = sX + (s * RES_TILE + c) * NB + i;
                const T *g = sg + (s * RES_TILE + c) * NV;
                add_products(a0, a1, a2, xr, g);
            }
            r = a0 + (a1 + a2);
            sr[c * NV + i] = r;
        }
        __syncthreads();
    } else if (act) {
        r = sr[c * NV + i];
    }
    double sq = act ? mul_rn((double)r, (double)r) : 0.0;
    if (mode == 3) {
        /* X held Dinv X: r is already Dinv R */
        if (act) sb[c * NV + i] = -r;
    } else if (mode == 4) {
        /* R = v + J z after the line solves, so J z = R - v */
        if (act) sb[c * NV + i] = r - Rsrc[(size_t)p0 * NV + c * NV + i];
    } else if (act) {
        sb[c * NV + i] = neg_dinv_row<T>(sD + c * NB + i, sr + c * NV);
    }
    __syncthreads();
    if (act) b[(size_t)p0 * NV + tid] = sb[tid]; /* contiguous tile store */
    if (ns.partials) {
        __shared__ double red[RES_THREADS_FAST / 32];
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
        if ((tid & 31) == 0) red[tid >> 5] = sq;
        __syncthreads();
        if (tid == 0) {
            double tot = 0.0;
            for (int w = 0; w < RES_THREADS_FAST / 32; ++w) tot += red[w];
            ns.partials[blk] = tot; /* the tile's sum R^2; totals by finalize_total */
        }
    }
    return true;
}

/* The single-system residual launches are persistent: CTA k takes tiles
 * k, k + grid, ...; each tile completes one phase of the CTA's barrier and
 * writes its partial; finalize_total then sums the tiles' partials in tile
 * order (the order of the batched norm kernel with 160 threads). */
template <typename T>
__device__ __forceinline__ bool resid_tiles(int nx, int np16, int mode, const T *Dinv, const T *X,
                                            const int *xnbr, const T *dU, const T *Rsrc, T *b,
                                            T *Uacc, const NormSink &ns, unsigned *status,
                                            int u_tile0 = 0, const T *Uin = nullptr) {
    timer_launch_start(ns.timer);
    uint64_t *bar = resid_bar_init();
    const int ntiles = np16 / RES_TILE;
    uint32_t parity = 0;
    /* the neighbour indices of a CTA's next tile are loaded while it works
     * on the current one, so that a tile's gathers wait for one memory
     * round trip, not two */
    constexpr int PRE = 4;
    const bool pre = mode >= 1 && nx <= PRE && threadIdx.x < RES_TILE * NV;
    const int c = threadIdx.x % RES_TILE;
    int nbr[PRE], nxt[PRE];
#pragma unroll
    for (int s = 0; s < PRE; ++s) nbr[s] = (pre && s < nx && blockIdx.x < ntiles)
                                               ? xnbr[(size_t)s * np16 + blockIdx.x * RES_TILE + c] : -1;
    for (int w = blockIdx.x; w < ntiles; w += gridDim.x) {
        const int wn = w + gridDim.x;
#pragma unroll
        for (int s = 0; s < PRE; ++s)
            nxt[s] = (pre && s < nx && wn < ntiles) ? xnbr[(size_t)s * np16 + wn * RES_TILE + c] : -1;
        const bool ok = fast_resid_body<T>(nx, np16, mode, Dinv, X, xnbr, dU, Rsrc, b,
                                           w >= u_tile0 ? Uacc : nullptr, ns, status, w, bar, parity,
                                           pre ? nbr : nullptr, Uin);
        parity ^= 1u;
        if (!ok) break;
#pragma unroll
        for (int s = 0; s < PRE; ++s) nbr[s] = nxt[s];
        __syncthreads(); /* the next tile's copies overwrite the stages */
    }
    /* a line partition's norm covers its owned lines, which come first */
    return finalize_total(ns, (ns.ntiles > 0 && ns.ntiles < ntiles) ? ns.ntiles : ntiles);
}

/* mode 1 (R = sum X dU over the cross-line slots); U += dU (Uacc = Uin +
 * dU when Uin is set) for the tiles from u_tile0 on: a line partition's
 * halo tiles, whose line solves leave U alone */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST) fast_resid_kernel(
    int nx, int np16, const T *__restrict__ Dinv, const T *__restrict__ X,
    const int *__restrict__ xnbr, const T *__restrict__ dU, T *__restrict__ b,
    T *__restrict__ Uacc, NormSink ns, unsigned *status, int u_tile0, const T *__restrict__ Uin) {
    resid_tiles<T>(nx, np16, 1, Dinv, X, xnbr, dU, nullptr, b, Uacc, ns, status, u_tile0, Uin);
}

/* mode 3 (b = -sum (Dinv X) dU: premultiplied cross-line blocks, no norm) */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST) fast_resid_dx_kernel(
    int nx, int np16, const T *__restrict__ DX, const int *__restrict__ xnbr,
    const T *__restrict__ dU, T *__restrict__ b, T *__restrict__ Uacc, unsigned *status) {
    resid_tiles<T>(nx, np16, 3, nullptr, DX, xnbr, dU, nullptr, b, Uacc, NormSink{}, status);
}

/* mode 4 (the product with J of a preconditioned direction: R = sum X dU
 * is the residual of v + J z after the line solves, so w = R - v; no
 * Dinv, no norm) */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST) fast_resid_jv_kernel(
    int nx, int np16, const T *__restrict__ X, const int *__restrict__ xnbr,
    const T *__restrict__ dU, const T *__restrict__ v, T *__restrict__ w, T *__restrict__ Uacc,
    unsigned *status) {
    resid_tiles<T>(nx, np16, 4, nullptr, X, xnbr, dU, v, w, Uacc, NormSink{}, status);
}

/* mode 0 (R given in position order) */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST) fast_resid_rhs_kernel(
    int np16, const T *__restrict__ Dinv, const T *__restrict__ Rsrc, T *__restrict__ b,
    T *__restrict__ Uzero, NormSink ns, unsigned *status) {
    resid_tiles<T>(0, np16, 0, Dinv, nullptr, nullptr, nullptr, Rsrc, b, Uzero, ns, status);
}

/* CTAs of a persistent single-system residual launch: as many as fit */
static int resid_grid_persistent(const void *fn, size_t smem, int ntiles) {
    int dev = 0, nsm = 148, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, RES_THREADS_FAST, smem) != cudaSuccess ||
        per < 1)
        per = 1;
    const int g = per * nsm;
    return ntiles < g ? (ntiles > 0 ? ntiles : 1) : g;
}

template <typename T>
int launch_fast_resid(cudaStream_t st, const FastLayout &L, int mode, const T *Dinv, const T *X,
                      const T *dU, const T *Rsrc, T *b, const NormSink &ns, unsigned *status,
                      T *Uacc, int u_tile0, const T *Uin) {
    if (L.nv != NV) return (int)cudaErrorInvalidValue;
    const int grid = fast_resid_grid(L.np16);
    if (mode == 4) {
        /* nx == 0 runs the kernel too: no slot is read, w = -v */
        if (!Rsrc) return (int)cudaErrorInvalidValue;
        const size_t smem4 = resid_smem_bytes<T>(L.nx);
        fast_resid_jv_kernel<T><<<resid_grid_persistent((const void *)fast_resid_jv_kernel<T>, smem4, grid),
                                  RES_THREADS_FAST, smem4, st>>>(L.nx, L.np16, X, L.xnbr, dU, Rsrc, b,
                                                                 Uacc, status);
        return (int)cudaGetLastError();
    }
    if (mode >= 1 && L.nx == 0) {
        /* a mesh that is one line: the line solve is exact, R_new = 0 */
        if (Uacc) {
            const long long n = (long long)L.np16 * NV;
            axpy_same_kernel<T><<<grid_for(n, 256), 256, 0, st>>>(dU, Uacc, n);
        }
        cudaMemsetAsync(b, 0, (size_t)L.np16 * NV * sizeof(T), st);
        if (mode == 3) return (int)cudaGetLastError(); /* no norm wanted */
        /* run the kernel on a zero residual (read from b itself) so that the
         * norm bookkeeping happens */
        mode = 0;
        Rsrc = b;
        Uacc = nullptr;
    }
    if (mode == 0 && !Rsrc) return (int)cudaErrorInvalidValue;
    const size_t smem = resid_smem_bytes<T>(mode >= 1 ? L.nx : 0);
    if (mode == 3)
        fast_resid_dx_kernel<T><<<resid_grid_persistent((const void *)fast_resid_dx_kernel<T>, smem, grid),
                                  RES_THREADS_FAST, smem, st>>>(L.nx, L.np16, X, L.xnbr, dU, b, Uacc,
                                                                status);
    else if (mode == 1)
        fast_resid_kernel<T><<<resid_grid_persistent((const void *)fast_resid_kernel<T>, smem, grid),
                               RES_THREADS_FAST, smem, st>>>(L.nx, L.np16, Dinv, X, L.xnbr, dU, b, Uacc,
                                                             ns, status, u_tile0, Uin);
    else
        fast_resid_rhs_kernel<T><<<resid_grid_persistent((const void *)fast_resid_rhs_kernel<T>, smem, grid),
                                   RES_THREADS_FAST, smem, st>>>(L.np16, Dinv, Rsrc, b, Uacc, ns, status);
    return (int)cudaGetLastError();
}

template int launch_fast_resid<double>(cudaStream_t, const FastLayout &, int, const double *,
                                       const double *, const double *, const double *, double *,
                                       const NormSink &, unsigned *, double *, int, const double *);
template int launch_fast_resid<float>(cudaStream_t, const FastLayout &, int, const float *,
                                      const float *, const float *, const float *, float *,
                                      const NormSink &, unsigned *, float *, int, const float *);

/* =========================================================== line Thomas
 * thomas.cuh holds the line solve; here are its launches at block size 9. */
constexpr int THOMAS_P = 8;

template <typename T>
constexpr uint32_t thomas_stage() { return thomas_stage_bytes<T, NV, THOMAS_P>(); }

/* one CTA (one warp) per line */
/* lines from nacc on leave U alone (accumulate 2) */
template <typename T, int P, bool YS>
__global__ void __launch_bounds__(32) fast_thomas_kernel(
    int nline, int NS, int accumulate, int nacc, const int *__restrict__ line_start,
    const int *__restrict__ line_len, const int *__restrict__ line_twist, const T *__restrict__ G,
    const T *__restrict__ Gam, const T *__restrict__ b, T *__restrict__ y, T *__restrict__ dU,
    T *__restrict__ U, const T *__restrict__ Uin, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int l = blockIdx.x;
    if (l >= nline) return;
    thomas_init_bars(smem, NS);
    const uint64_t pol = threadIdx.x == 0 ? policy_evict_first() : 0;
    uint32_t pbase = 0;
    thomas_line<T, NV, P, YS>(NS, l < nacc ? accumulate : 2, line_start[l], line_len[l], line_twist[l], G,
                          Gam, b, y, dU, U, status, smem, pbase, pol, Uin);
}

/* Warp-specialised form, one CTA of two warps per line: warp 1 issues the
 * staging copies, warp 0 runs the chains with the same arithmetic as
 * fast_thomas_kernel, so its results are bit-identical; the chain warp no
 * longer stops every chunk to issue the next copies. */
template <typename T, int P, bool YS>
__global__ void __launch_bounds__(64) fast_thomas_ws_kernel(
    int nline, int NS, int accumulate, int nacc, const int *__restrict__ line_start,
    const int *__restrict__ line_len, const int *__restrict__ line_twist, const T *__restrict__ G,
    const T *__restrict__ Gam, const T *__restrict__ b, T *__restrict__ y, T *__restrict__ dU,
    T *__restrict__ U, const T *__restrict__ Uin, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int l = blockIdx.x;
    if (l >= nline) return;
    if (threadIdx.x == 0) thomas_init_ws(smem, NS);
    __syncthreads();
    const uint64_t pol = threadIdx.x == 32 ? policy_evict_first() : 0;
    uint32_t pbase = 0;
    thomas_line<T, NV, P, YS, true>(NS, l < nacc ? accumulate : 2, line_start[l], line_len[l],
                                line_twist[l], G, Gam, b, y, dU, U, status, smem, pbase, pol, Uin);
}

/* Persistent form over many systems: each CTA (one warp) takes (system,
 * line) items from a device work queue, in the order of `work` (longest
 * lines first, so that the long lines do not start last), and skips the
 * lines of systems that have converged.  queue[0] is the next item,
 * queue[1] counts retired CTAs; the last CTA to retire resets both for the
 * next launch.  U is left to the residual kernel (accumulate = 2). */
template <typename T, int P>
__global__ void __launch_bounds__(32) fast_thomas_batch_kernel(
    const ThomasSys<T> *__restrict__ sys, const WorkItem *__restrict__ work,
    const int *__restrict__ nwork_p, const int *__restrict__ active, unsigned *queue, int NS,
    unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int nwork = *nwork_p;
    thomas_init_bars(smem, NS);
    const uint64_t pol = lane == 0 ? policy_evict_first() : 0;
    uint32_t pbase = 0;
    for (;;) {
        int w = 0;
        if (lane == 0) w = (int)atomicAdd(queue, 1u);
        w = __shfl_sync(FULL, w, 0);
        if (w >= nwork) break;
        const WorkItem it = work[w];
        if (active && !active[it.sys]) continue;
        const ThomasSys<T> S = sys[it.sys];
        const int l = it.unit;
        if (!thomas_line<T, NV, P, false>(NS, 2, S.line_start[l], S.line_len[l], S.line_twist[l], S.G,
                                      S.Gam, S.b, S.y, S.dU, nullptr, status, smem, pbase, pol))
            break;
    }
    if (lane == 0) {
        __threadfence();
        if (atomicAdd(queue + 1, 1u) == gridDim.x - 1) {
            queue[0] = 0u;
            queue[1] = 0u;
            __threadfence();
        }
    }
}

/* The same persistent loop with two warps per CTA: warp 1 issues every
 * line's staging copies, warp 0 runs its chains (thomas_line's
 * warp-specialised form, bit-identical results).  Thread 0 takes the next
 * item for both warps; the staging barriers' parities carry across lines
 * in `pbase`, kept the same in both warps. */
template <typename T, int P>
__global__ void __launch_bounds__(64) fast_thomas_batch_ws_kernel(
    const ThomasSys<T> *__restrict__ sys, const WorkItem *__restrict__ work,
    const int *__restrict__ nwork_p, const int *__restrict__ active, unsigned *queue, int NS,
    unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_item, s_stop;
    const int nwork = *nwork_p;
    if (threadIdx.x == 0) {
        thomas_init_ws(smem, NS);
        s_stop = 0;
    }
    __syncthreads();
    const uint64_t pol = threadIdx.x == 32 ? policy_evict_first() : 0;
    uint32_t pbase = 0;
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(queue, 1u);
        __syncthreads();
        const int w = s_item;
        __syncthreads(); /* s_item is read before thread 0 takes the next item */
        if (w >= nwork) break;
        const WorkItem it = work[w];
        if (active && !active[it.sys]) continue;
        const ThomasSys<T> S = sys[it.sys];
        const int l = it.unit;
        const bool ok = thomas_line<T, NV, P, false, true>(NS, 2, S.line_start[l], S.line_len[l],
                                                       S.line_twist[l], S.G, S.Gam, S.b, S.y, S.dU,
                                                       nullptr, status, smem, pbase, pol);
        if (!ok && (threadIdx.x & 31) == 0) s_stop = 1;
        __syncthreads();
        if (s_stop) break;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(queue + 1, 1u) == gridDim.x - 1) {
            queue[0] = 0u;
            queue[1] = 0u;
            __threadfence();
        }
    }
}

struct ThomasCfg {
    int NS;
    bool ys;
    size_t smem;
};

template <typename T, bool WS = false>
static ThomasCfg thomas_cfg(const FastLayout &L) {
    const size_t sb = thomas_stage<T>();
    /* lines resident per SM in one wave, and the shared memory each may use
     * so that they all are: the SM's capacity over them, less the per-CTA
     * reservation.  The deeper the copy ring, the more of the DRAM latency
     * the chain steps hide. */
    int dev = 0, nsm = 148, smem_sm = 228 * 1024, reserved = 1024;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (nsm < 1) nsm = 148;
    const int per_sm = (L.nline + nsm - 1) / nsm;
    const long long budget = smem_share(smem_sm, per_sm, reserved);
    const size_t ys_bytes = (size_t)((L.max_len + 3) & ~3) * NV * sizeof(T);
    const size_t fixed = thomas_hdr<WS>() + BCAST<T, NV> * sizeof(T);
    ThomasCfg c;
    c.ys = (long long)(fixed + ys_bytes + 3 * sb) <= budget;
    long long left = budget - (long long)fixed - (c.ys ? (long long)ys_bytes : 0);
    long long ns = left / (long long)sb;
    if (ns > 8) ns = 8;
    if (ns < 2) ns = 2;
    c.NS = (int)ns;
    c.smem = fixed + (size_t)c.NS * sb + (c.ys ? ys_bytes : 0);
    return c;
}

/* Which single-system line solve: the warp-specialised kernel (a copy
 * warp beside each chain warp) where few lines share an SM -- there the
 * launch is bound by the chain's step latency, and taking the copy issue
 * off the chain warp shortens every step (360 lines: 53 -> 45 us); the
 * one-warp kernel where many lines share an SM, whose warps hide each
 * other's latency and which holds more lines per SM in its registers
 * (1,200 lines: 419 us one-warp, 569 us warp-specialised).  At 600 lines
 * (5 per SM) the copy warp still pays: 128 -> 124 us (FP64), 91 -> 82 us
 * (FP32).  The environment variable TBS_THOMAS_WS=0 / 1 forces one or the
 * other. */
static bool thomas_ws(const FastLayout &L) {
    static const int forced = [] {
        const char *e = getenv("TBS_THOMAS_WS");
        return e && e[0] ? (e[0] == '0' ? 0 : 1) : -1;
    }();
    if (forced >= 0) return forced == 1;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (nsm < 1) nsm = 148;
    return (L.nline + nsm - 1) / nsm <= 5;
}

template <typename T, bool WS, bool YS>
static const void *thomas_fn() {
    return WS ? (const void *)fast_thomas_ws_kernel<T, THOMAS_P, YS>
              : (const void *)fast_thomas_kernel<T, THOMAS_P, YS>;
}

template <typename T, bool WS>
static const void *thomas_fn(bool ys) {
    return ys ? thomas_fn<T, WS, true>() : thomas_fn<T, WS, false>();
}

template <typename T>
int launch_fast_thomas(cudaStream_t st, const FastLayout &L, const T *G, const T *Gam, const T *b,
                       T *y, T *dU, T *U, unsigned *status, int accumulate, int nacc, const T *Uin) {
    if (L.nv != NV) return (int)cudaErrorInvalidValue;
    const bool ws = thomas_ws(L);
    const ThomasCfg c = ws ? thomas_cfg<T, true>(L) : thomas_cfg<T>(L);
    const void *fn = ws ? thomas_fn<T, true>(c.ys) : thomas_fn<T, false>(c.ys);
    int ns = c.NS, nline = L.nline;
    if (nacc < 0 || nacc > nline) nacc = nline;
    const int *ls = L.line_start, *ll = L.line_len, *lt = L.line_twist;
    void *args[] = {&nline, &ns,  &accumulate, &nacc, &ls, &ll, &lt,
                    &G,     &Gam, &b,          &y,    &dU, &U,  &Uin, &status};
    return (int)cudaLaunchKernel(fn, dim3(L.nline), dim3(ws ? 64 : 32), args, c.smem, st);
}

template int launch_fast_thomas<double>(cudaStream_t, const FastLayout &, const double *,
                                        const double *, const double *, double *, double *,
                                        double *, unsigned *, int, int, const double *);
template int launch_fast_thomas<float>(cudaStream_t, const FastLayout &, const float *,
                                       const float *, const float *, float *, float *, float *,
                                       unsigned *, int, int, const float *);

static int smem_limit(const void *fn) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, fn);
    return optin - (int)fa.sharedSizeBytes;
}

int smem_raise(const void *fn, size_t need) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess && (size_t)fa.maxDynamicSharedSizeBytes >= need)
        return 0;
    return (int)cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
}

static int set_smem(const void *fn, size_t need) {
    if ((long long)need > smem_limit(fn)) return (int)cudaErrorInvalidConfiguration;
    if (need <= 48 * 1024) return 0;
    return smem_raise(fn, need);
}

/* Called before any launch (and outside stream capture) once the layout is
 * known: opts the streaming kernels into the shared memory they need. */
int fast_prepare(const FastLayout &L) {
    int rc = set_smem((const void *)fast_resid_kernel<double>, resid_smem_bytes<double>(L.nx));
    if (!rc) rc = set_smem((const void *)fast_resid_jv_kernel<double>, resid_smem_bytes<double>(L.nx));
    if (!rc) rc = set_smem((const void *)fast_resid_kernel<float>, resid_smem_bytes<float>(L.nx));
    const ThomasCfg c64 = thomas_cfg<double>(L), c32 = thomas_cfg<float>(L);
    const ThomasCfg w64 = thomas_cfg<double, true>(L), w32 = thomas_cfg<float, true>(L);
    if (!rc) rc = set_smem(thomas_fn<double, false>(c64.ys), c64.smem);
    if (!rc) rc = set_smem(thomas_fn<float, false>(c32.ys), c32.smem);
    if (!rc) rc = set_smem(thomas_fn<double, true>(w64.ys), w64.smem);
    if (!rc) rc = set_smem(thomas_fn<float, true>(w32.ys), w32.smem);
    return rc;
}

/* ==================================================== many sweeps, one launch
 * TBS_ALGO_FP64 sweeps of a system of few lines as one cooperative launch: a
 * CTA per line (and more, to share the tiles), per sweep
 *   line solves (warps 0 and 1, thomas_line's warp-specialised form)
 *   -- all CTAs meet --
 *   residual tiles (mode 1 of fast_resid_body: same operations and order),
 *   each CTA's first tiles' blocks copied before the meeting
 *   -- all CTAs meet --
 *   every CTA adds the tiles' partials (finalize_total's order) and decides
 * until the tolerance, the sweep limit or a norm that is not finite.  The
 * results, the history and the decisions are those of the launches per sweep,
 * bit for bit.
 * What it saves is what bounds a small system: two launches' start and end
 * and the graph's loop and condition nodes, about 11 us a sweep, against two
 * meetings of 1.2 us (60x64: 28 us a sweep before).  Vectors that other CTAs
 * wrote are read past the L1; what bulk copies read or wrote is fenced from
 * the ordinary accesses. */
constexpr int SMALL_THREADS = RES_THREADS_FAST;
constexpr int SMALL_NS = 6;   /* ring stages of the line solve; two residual tiles lie in the ring */
constexpr int SMALL_HDR = 256;

struct SmallSweeps {
    int nline, nx, np16, max_len, longest;
    const int *line_start, *line_len, *line_twist, *xnbr;
    const double *G, *Gam, *Dinv, *X;
    double *b, *y, *dU, *U, *partials, *hist;
    SolveState *state;
    unsigned *meet; /* grid_meet's words */
    unsigned *status;
    unsigned long long *timer;
    unsigned long long loop, check; /* condition handles */
    int use_check;
    int keep; /* the blocks fit in the L2 and are read to stay there */
    MeetTest test;
};

static size_t small_smem(const FastLayout &L) {
    return SMALL_HDR + SMALL_NS * (size_t)thomas_stage<double>() + BCAST<double, NV> * sizeof(double) +
           (size_t)((L.max_len + 3) & ~3) * NV * sizeof(double) +
           (size_t)(L.nx + 2) * RES_TILE * NV * sizeof(double);
}

/* tiles whose blocks fit in the ring at once */
__host__ __device__ inline int small_bufs(int nx) {
    return (int)(SMALL_NS * 2 * THOMAS_P * (NB + NV) * sizeof(double)) / ((1 + nx) * RES_TILE * NB * 8) >= 2 ? 2 : 1;
}

__global__ void __launch_bounds__(SMALL_THREADS, 2) small_sweeps_kernel(SmallSweeps A) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int nx = A.nx, np16 = A.np16, ntiles = np16 / RES_TILE, nbuf = small_bufs(nx);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    uint64_t *rbar = bars + 18; /* behind thomas_line's two counters */
    volatile int *s_ok = reinterpret_cast<volatile int *>(smem + 160);
    double *red = reinterpret_cast<double *>(smem + 168); /* one per warp, then the norm */
    unsigned char *ring = smem + SMALL_HDR;
    double *aux = reinterpret_cast<double *>(ring + SMALL_NS * thomas_stage<double>()) + BCAST<double, NV> +
                  ((A.max_len + 3) & ~3) * NV;
    double *sg = aux, *sr = aux + nx * RES_TILE * NV, *sb = sr + RES_TILE * NV;
    if (tid == 0) {
        mbar_init(&rbar[0], 1);
        mbar_init(&rbar[1], 1);
        thomas_init_ws(smem, SMALL_NS);
    }
    __syncthreads();
    const SolveState *S = A.state;
    const double norm0 = S->norm0, tol = S->tol;
    const int max_sweeps = S->max_sweeps, hist_cap = S->hist_cap;
    int sw = S->sweep;
    double nrm = 0.0;
    const bool away = (int)blockIdx.x == A.test.absent;
    bool met = false, ok = !away;
    const bool mine = (int)blockIdx.x < A.nline && !away;
    const int ls = mine ? A.line_start[blockIdx.x] : 0, ll = mine ? A.line_len[blockIdx.x] : 0,
              lt = mine ? A.line_twist[blockIdx.x] : 0;
    const uint64_t pol = A.keep ? policy_evict_last() : policy_evict_first();
    uint32_t pbase = 0, rpar = 0;
    unsigned round = 0;
    const int c = tid % RES_TILE, i = tid / RES_TILE;
    const bool act = tid < RES_TILE * NV;
    const uint32_t szD = RES_TILE * NB * sizeof(double);
    auto meet = [&](auto &&meanwhile) { return grid_meet(A.meet, ++round, s_ok, A.test.budget, meanwhile); };
    auto tile_of = [&](int k) { return (int)blockIdx.x + k * (int)gridDim.x; };
    auto blocks = [&](int k) { return reinterpret_cast<double *>(ring) + (size_t)(k % nbuf) * (1 + nx) * RES_TILE * NB; };
    auto issue = [&](int k) { /* thread 0: the k-th tile's blocks */
        const int p0 = tile_of(k) * RES_TILE;
        if (tile_of(k) >= ntiles) return;
        uint64_t *bar = &rbar[k % nbuf];
        double *d = blocks(k);
        mbar_arrive_expect_tx(bar, (1 + nx) * szD);
        bulk_g2s_hint(d, A.Dinv + (size_t)p0 * NB, szD, bar, pol);
        for (int s = 0; s < nx; ++s)
            bulk_g2s_hint(d + (1 + s) * RES_TILE * NB, A.X + ((size_t)s * np16 + p0) * NB, szD, bar, pol);
    };
    /* the neighbours of this thread's cell of the k-th tile, and their dU */
    auto neighbours = [&](int k, int (&nb)[4]) {
#pragma unroll
        for (int s = 0; s < 4; ++s)
            nb[s] = (act && s < nx && tile_of(k) < ntiles) ? A.xnbr[(size_t)s * np16 + tile_of(k) * RES_TILE + c] : -1;
    };
    auto gather = [&](const int (&nb)[4], double (&g)[4]) {
#pragma unroll
        for (int s = 0; s < 4; ++s) g[s] = nb[s] >= 0 ? __ldcg(A.dU + (size_t)nb[s] * NV + i) : 0.0;
    };
    /* the sums of the partials that threads 32 v .. 32 v + 31 (and 32 v1 ..)
     * of finalize_total would make, loads of both in flight together */
    auto norm_part = [&](int v, int v1) {
        constexpr int B = 6;
        double acc[2] = {0.0, 0.0};
        const int q0 = 32 * v + (tid & 31), d = 32 * (v1 - v);
        for (int r = 0; r * SMALL_THREADS < ntiles; r += B) {
            double x[2][B];
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const int q = q0 + (r + k) * SMALL_THREADS;
                x[0][k] = q < ntiles ? __ldcg(A.partials + q) : 0.0;
                x[1][k] = d > 0 && q + d < ntiles ? __ldcg(A.partials + q + d) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < B; ++k) { /* sums of squares: adding 0.0 changes none */
                acc[0] += x[0][k];
                acc[1] += x[1][k];
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            acc[0] += __shfl_down_sync(FULL, acc[0], o);
            acc[1] += __shfl_down_sync(FULL, acc[1], o);
        }
        if ((tid & 31) == 0) {
            red[v] = acc[0];
            if (d > 0) red[v1] = acc[1];
        }
    };
    static_assert(SMALL_THREADS == 160, "the counts of barriers 2 and 3");
    auto line = [&](auto phase) {
        return thomas_line<double, NV, THOMAS_P, true, true, decltype(phase)::value>(
            SMALL_NS, 1, ls, ll, lt, A.G, A.Gam, A.b, A.y, A.dU, A.U, A.status, smem, pbase, pol, nullptr, true);
    };
    /* b, as the others stored it, for this warp's bulk copies */
    auto start_vecs = [&]() {
        if (tid == 32) fence_async_all();
        line(std::integral_constant<int, PH_VECS>{});
    };
    int nb0[4], nb1[4]; /* the first two tiles' neighbours, the same in every sweep */
    neighbours(0, nb0);
    neighbours(1, nb1);
    if (mine && warp == 1) {
        line(std::integral_constant<int, PH_BLOCKS>{});
        start_vecs();
    }
    while (ok) {
        /* ---------------- line solves */
        if (mine && warp < 2) ok = line(std::integral_constant<int, PH_RUN>{});
        ok = __syncthreads_and(ok); /* the ring is free */
        if (!ok) break;
        unsigned long long t0 = 0;
        if (A.timer && (int)blockIdx.x == A.longest && tid == 0) t0 = globaltimer_ns();
        if (tid == 0)
            for (int k = 0; k < nbuf; ++k) issue(k);
        const bool came = meet([]() {});
        /* ---------------- residual: R = sum X dU, b = -Dinv R; the next tile's
         * neighbours' dU is read while a tile is worked on */
        double g[4], gn[4];
        int nn[4];
        gather(nb0, g);
        for (int k = 0; ok && tile_of(k) < ntiles; ++k) {
            const int blk = tile_of(k), p0 = blk * RES_TILE;
            if (act) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    if (s < nx) sg[(s * RES_TILE + c) * NV + i] = g[s];
            }
            if (k == 0)
                gather(nb1, gn);
            else
                gather(nn, gn);
            neighbours(k + 2, nn);
            const bool landed = mbar_wait(&rbar[k % nbuf], (rpar >> (k % nbuf)) & 1u);
            rpar ^= 1u << (k % nbuf);
            if (__syncthreads_or(!landed)) {
                if (tid == 0)
                    for (int q = k; q < k + nbuf; ++q) /* let the copies land before the CTA retires */
                        if (tile_of(q) < ntiles)
                            mbar_wait(&rbar[q % nbuf], ((rpar >> (q % nbuf)) & 1u) ^ (q == k ? 1u : 0u), 1LL << 28);
                ok = false;
                break;
            }
            const double *sD = blocks(k), *sX = sD + RES_TILE * NB;
            double r = 0.0;
            if (act) {
                double a0 = 0.0, a1 = 0.0, a2 = 0.0;
                for (int s = 0; s < nx; ++s) {
                    const double *xr = sX + (s * RES_TILE + c) * NB + i;
                    const double *q = sg + (s * RES_TILE + c) * NV;
                    add_products(a0, a1, a2, xr, q);
                }
                r = a0 + (a1 + a2);
                sr[c * NV + i] = r;
            }
            __syncthreads();
            double sq = act ? mul_rn(r, r) : 0.0;
            if (act) sb[c * NV + i] = neg_dinv_row<double>(sD + c * NB + i, sr + c * NV);
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
            if ((tid & 31) == 0) red[warp] = sq;
            __syncthreads();
            if (act) A.b[(size_t)p0 * NV + tid] = sb[tid];
            if (tid == 0) {
                double tot = 0.0;
                for (int w = 0; w < SMALL_THREADS / 32; ++w) tot += red[w];
                A.partials[blk] = tot;
                issue(k + nbuf); /* every thread is done with this buffer */
            }
            /* red, sg, sr and sb are next written behind another barrier */
#pragma unroll
            for (int s = 0; s < 4; ++s) g[s] = gn[s];
        }
        if (!ok) break;
        /* the next solves' first blocks go into the ring, which is free again;
         * their b follows the meeting and lands under the norm */
        ok = meet([&]() {
                 if (mine) line(std::integral_constant<int, PH_BLOCKS>{});
             }) && came;
        bool more = false;
        if (ok) {
            if (A.timer && (int)blockIdx.x == A.longest && tid == 0) {
                atomicAdd(A.timer + 1, globaltimer_ns() - t0);
                atomicAdd(A.timer + 2, 1ull);
            }
            /* ---------------- the norm, by every CTA: warp 1 starts the copies
             * of b, the others add the partials in finalize_total's order
             * (that of SMALL_THREADS threads, warp 0 taking warp 1's part too) */
            if (warp == 1) {
                if (mine) start_vecs();
                asm volatile("bar.sync 3, 160;" ::: "memory");
            } else {
                norm_part(warp, warp == 0 ? 1 : warp);
                asm volatile("bar.arrive 3, 160;" ::: "memory");
                asm volatile("bar.sync 2, 128;" ::: "memory");
            }
            double tot = 0.0;
            for (int w = 0; w < SMALL_THREADS / 32; ++w) tot += red[w];
            nrm = sqrt(tot);
            ++sw;
            if (blockIdx.x == 0 && tid == 0 && sw < hist_cap) A.hist[sw] = nrm;
            met = isfinite(nrm) && nrm <= tol * norm0;
            more = isfinite(nrm) && !met && sw < max_sweeps;
        }
        if (!more) {
            if (mine && warp == 1) {
                if (!ok) start_vecs(); /* the copies that the barriers count on */
                line(std::integral_constant<int, PH_DROP>{});
            }
            break;
        }
    }
    if (!ok && !away && tid == 0) atomicOr(A.status, ST_TIMEOUT);
    __syncthreads();
    if (tid == 0) {
        if (grid_leave(A.meet)) { /* every CTA has left the meetings */
            A.state->sweep = sw;
            A.state->last = nrm;
            cudaGraphSetConditional((cudaGraphConditionalHandle)A.loop, 0u);
            if (A.use_check) cudaGraphSetConditional((cudaGraphConditionalHandle)A.check, ok && met ? 1u : 0u);
        }
    }
}

/* CTAs of a launch of all sweeps; 0: the system is not for it.
 * One a line at least, and one a tile up to half an SM count of them, where
 * several such launches fit beside each other in any case.  More tiles go
 * nbuf to a CTA while there are places (the second tile's blocks are copied
 * under the first), so that the launches of several threads' contexts fit:
 * 60x64 takes 12.9 us a sweep with 120 CTAs and 12.3 with 240, and four
 * threads with a system each 59 us a solve in all, 98 with 240, 66 with a
 * launch per kernel.
 * Where a CTA's place is an SM (lines beyond 537 cells), a launch per kernel,
 * with six CTAs an SM on the tiles, is faster from some 48 blocks of 16
 * positions a CTA on (this / that, us a sweep: 60x600 72 / 74 at 46 blocks,
 * 36x1000 104 / 104 at 46, 20x2000 180 / 179 at 51, 60x800 93 / 91 at 61, 100x600
 * 85 / 83 at 76, 148x1000 162 / 139 at 187; three and four neighbours off the
 * line: 10x2x1500 147 / 144 at 51, 5x5x1000 107 / 109 at 53, 7x7x700 92 / 90 at
 * 72); with two CTAs an SM it is not, up to the 100 that their lines allow
 * (296x530 103 / 109; 17x17x500 133 / 145 at 153). */
constexpr int SMALL_BLOCKS = 48;

int small_sweeps_grid(const FastLayout &L) {
    if (L.nv != NV || L.nx < 1 || L.nx > 4) return 0;
    const size_t smem = small_smem(L);
    if ((long long)smem > smem_limit((const void *)small_sweeps_kernel)) return 0;
    if (smem_raise((const void *)small_sweeps_kernel, smem)) return 0;
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)small_sweeps_kernel, SMALL_THREADS,
                                                      smem) != cudaSuccess)
        return 0;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int cap = std::min(per, 2) * nsm;
    if (L.nline > cap) return 0;
    const int ntiles = L.np16 / RES_TILE, nbuf = small_bufs(L.nx);
    if (per == 1 && (long long)ntiles * (1 + L.nx) > (long long)SMALL_BLOCKS * nsm) return 0;
    const int share = std::max((ntiles + nbuf - 1) / nbuf, std::min(ntiles, nsm / 2));
    return std::max(L.nline, std::min(share, cap));
}

int launch_small_sweeps(cudaStream_t st, const FastLayout &L, const double *G, const double *Gam,
                        const double *Dinv, const double *X, double *b, double *y, double *dU, double *U,
                        const NormSink &ns, unsigned *meet, unsigned *status, MeetTest test) {
    const int grid = small_sweeps_grid(L);
    if (grid < 1) return (int)cudaErrorInvalidValue;
    SmallSweeps A{L.nline,  L.nx, L.np16, L.max_len, L.longest, L.line_start, L.line_len, L.line_twist, L.xnbr,
                  G,        Gam,  Dinv,   X,         b,            y,          dU,           U,
                  ns.partials, ns.hist, ns.state, meet, status, ns.timer, ns.handle, ns.check_handle,
                  ns.use_check,
                  (long long)L.np16 * (3 + L.nx) * NB * (long long)sizeof(double) <= (96LL << 20),
                  MeetTest{test.absent, test.budget > 0 ? test.budget : MEET_BUDGET}};
    void *args[] = {&A};
    return (int)cudaLaunchCooperativeKernel((const void *)small_sweeps_kernel, dim3(grid), dim3(SMALL_THREADS),
                                            args, small_smem(L), st);
}

int fast_kernels_init() { return 0; }

/* one CTA per line of the pack; the descriptor travels as a kernel parameter */
__global__ void __launch_bounds__(256) line_pack_kernel(LinePack lp, double *__restrict__ vec,
                                                        double *__restrict__ buf, int to_line) {
    const int k = blockIdx.x;
    if (k >= lp.n) return;
    const long long n = (long long)lp.len[k] * NV;
    double *v = vec + (long long)lp.start[k] * NV;
    double *b = buf + lp.off[k];
    for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        if (to_line)
            v[t] = b[t];
        else
            b[t] = v[t];
    }
}

int launch_line_pack(cudaStream_t st, const LinePack &lp, double *vec, double *buf, int to_line) {
    if (lp.n <= 0) return 0;
    line_pack_kernel<<<lp.n, 256, 0, st>>>(lp, vec, buf, to_line);
    return (int)cudaGetLastError();
}

/* ============================================ true residual, any ordering
 * R(pos(e)) = rhs(e) + D_e U(pos(e)) + sum_{faces} offJ U(pos(nbr)) with the
 * original FP64 blocks (face rule of linesmoothLU_TriBlock_v3.okl:299-328),
 * output in position order as T, plus fixed-order per-block sum R^2.
 * Used for the FP64 outer residual of TBS_ALGO_MIXED, for a non-zero
 * starting solution, and for tbs_true_residual_norm / tbs_get_residual. */
constexpr int FULLRES_THREADS = 288;

template <typename T>
__device__ __forceinline__ void full_resid_body(
    int nelem, const int *__restrict__ epoint, const int *__restrict__ ef,
    const int *__restrict__ fc, const int *__restrict__ pos_of_elem,
    const double *__restrict__ D, const double *__restrict__ O1, const double *__restrict__ O2,
    const double *__restrict__ rhs, const double *__restrict__ Up, T *__restrict__ Rp,
    double *__restrict__ partials, int blk) {
    const int epb = FULLRES_THREADS / NV;
    const int le = threadIdx.x / NV;
    const int i = threadIdx.x - le * NV;
    const int e = blk * epb + le;
    double sq = 0.0;
    if (e < nelem) {
        const int pe = pos_of_elem[e];
        const double *u = Up + (size_t)pe * NV;
        const double *dr = D + (size_t)e * NB + i;
        double a0, a1, a2;
        open_sums(a0, a1, a2, dr, u);
        close_sums(a0, a1, a2, dr, u);
        for (int k2 = epoint[e]; k2 < epoint[e + 1]; ++k2) {
            const int f = ef[k2];
            if (f >= 0) {
                const int e1 = fc[2 * f], e2 = fc[2 * f + 1];
                const double *o = ((e == e1) ? O2 : O1) + (size_t)f * NB + i;
                const double *un = Up + (size_t)pos_of_elem[(e == e1) ? e2 : e1] * NV;
                add_products(a0, a1, a2, o, un);
            }
        }
        const double r = (rhs ? rhs[(size_t)e * NV + i] : 0.0) + (a0 + (a1 + a2));
        Rp[(size_t)pe * NV + i] = (T)r;
        sq = mul_rn(r, r);
    }
    __shared__ double red[FULLRES_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < FULLRES_THREADS / 32; ++w) tot += red[w];
        partials[blk] = tot;
    }
}

template <typename T>
__global__ void __launch_bounds__(FULLRES_THREADS) full_resid_kernel(
    int nelem, const int *__restrict__ epoint, const int *__restrict__ ef,
    const int *__restrict__ fc, const int *__restrict__ pos_of_elem,
    const double *__restrict__ D, const double *__restrict__ O1, const double *__restrict__ O2,
    const double *__restrict__ rhs, const double *__restrict__ Up, T *__restrict__ Rp,
    double *__restrict__ partials) {
    full_resid_body<T>(nelem, epoint, ef, fc, pos_of_elem, D, O1, O2, rhs, Up, Rp, partials,
                       blockIdx.x);
}

int full_resid_blocks(int nelem) { return (nelem + (FULLRES_THREADS / NV) - 1) / (FULLRES_THREADS / NV); }

template <typename T>
int launch_full_resid(cudaStream_t st, int nelem, const int *epoint, const int *ef, const int *fc,
                      const int *pos_of_elem, const double *D, const double *O1, const double *O2,
                      const double *rhs, const double *Up, T *Rp, double *partials) {
    full_resid_kernel<T><<<full_resid_blocks(nelem), FULLRES_THREADS, 0, st>>>(
        nelem, epoint, ef, fc, pos_of_elem, D, O1, O2, rhs, Up, Rp, partials);
    return (int)cudaGetLastError();
}

template int launch_full_resid<double>(cudaStream_t, int, const int *, const int *, const int *,
                                       const int *, const double *, const double *,
                                       const double *, const double *, const double *, double *,
                                       double *);
template int launch_full_resid<float>(cudaStream_t, int, const int *, const int *, const int *,
                                      const int *, const double *, const double *,
                                      const double *, const double *, const double *, float *,
                                      double *);


/* ============================================ full residual, position order
 * Dp = D blocks by position, XF[s][p] = the block of interior face s of the
 * cell (ef order) in the cell's row; both from the original FP64 arrays,
 * zero where absent.  One warp per block. */
__global__ void fullpos_layout_kernel(long long nblk, int np16, const int *__restrict__ elem_of_pos,
                                      const int *__restrict__ xsrcf, const double *__restrict__ D,
                                      const double *__restrict__ O1, const double *__restrict__ O2,
                                      double *__restrict__ Dp, double *__restrict__ XF) {
    const int lane = threadIdx.x & 31;
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long q = w0; q < nblk; q += nw) {
        const double *src = nullptr;
        double *dst;
        if (q < np16) {
            const int e = elem_of_pos[q];
            if (e >= 0) src = D + (size_t)e * NB;
            dst = Dp + q * NB;
        } else {
            const long long k = q - np16; /* slot-major index s*np16 + p */
            const int f = xsrcf[k];
            if (f >= 0) src = ((f & 1) ? O2 : O1) + (size_t)(f >> 1) * NB;
            dst = XF + k * NB;
        }
        for (int tt = lane; tt < NB; tt += 32) dst[tt] = src ? src[tt] : 0.0;
    }
}

int launch_fullpos_layout(cudaStream_t st, const FastLayout &L, const double *jacD,
                          const double *O1, const double *O2, double *Dp, double *XF) {
    const long long nblk = (long long)L.np16 * (1 + L.nxf);
    fullpos_layout_kernel<<<grid_for(nblk * 32, 256), 256, 0, st>>>(nblk, L.np16, L.elem_of_pos,
                                                                    L.xsrcf, jacD, O1, O2, Dp, XF);
    return (int)cudaGetLastError();
}

__host__ __device__ inline size_t fullpos_smem_bytes(int nxf) {
    return 128 + (size_t)RES_TILE * NB * sizeof(double) * (1 + nxf) +
           (size_t)(nxf + 1) * RES_TILE * NV * sizeof(double) + (size_t)RES_TILE * NV * sizeof(double) +
           (size_t)RES_TILE * NB * sizeof(float) + 2 * (size_t)RES_TILE * NV * sizeof(float);
}

/* b = -Dinv R of one cell row in FP32, the operation order of the FP32
 * mode-0 residual (fast_resid_body): dr = column-major block row i, rv = R */

/* One tile of 16 positions (160 threads; thread t < 144 owns cell t % 16,
 * row t / 16).  R = rhs + D u + sum over faces (ef order) offJ u_nbr with
 * the accumulation pattern of full_resid_body; R32 out, partials[blk] =
 * the tile's sum R^2 (fixed order).  With Dinv32: also the next inner
 * solve's right-hand side b32 = -Dinv32 R32 and c32 = 0. */
__device__ __forceinline__ bool full_resid_pos_body(
    int nxf, int np16, const double *__restrict__ Dp, const double *__restrict__ XF,
    const int *__restrict__ xnbrf, const double *__restrict__ rhsp, const double *__restrict__ Up,
    float *__restrict__ R32, double *__restrict__ partials, const float *__restrict__ Dinv32,
    float *__restrict__ b32, float *__restrict__ c32, unsigned *status, int blk, uint64_t *bar,
    uint32_t parity, const int *nbr_pre = nullptr) {
    extern __shared__ __align__(128) unsigned char smem[];
    double *sD = reinterpret_cast<double *>(smem + 128);
    double *sX = sD + RES_TILE * NB;
    double *sg = sX + nxf * RES_TILE * NB;      /* [1 + nxf][16][9]: own u, then neighbours */
    double *sr = sg + (nxf + 1) * RES_TILE * NV; /* rhs tile */
    float *sDi = reinterpret_cast<float *>(sr + RES_TILE * NV); /* Dinv32 tile */
    float *so = sDi + RES_TILE * NB;
    float *sb = so + RES_TILE * NV;
    const int p0 = blk * RES_TILE;
    const int tid = threadIdx.x;
    const int c = tid % RES_TILE, i = tid / RES_TILE;
    const bool act = tid < RES_TILE * NV;
    const uint32_t szD = RES_TILE * NB * sizeof(double), szR = RES_TILE * NV * sizeof(double);
    const uint32_t szDi = RES_TILE * NB * sizeof(float);
    if (tid == 0) {
        const uint64_t pol = policy_evict_first();
        mbar_arrive_expect_tx(bar, szD * (1 + nxf) + szR + (Dinv32 ? szDi : 0u));
        bulk_g2s_hint(sD, Dp + (size_t)p0 * NB, szD, bar, pol);
        for (int s = 0; s < nxf; ++s)
            bulk_g2s_hint(sX + s * RES_TILE * NB, XF + ((size_t)s * np16 + p0) * NB, szD, bar, pol);
        bulk_g2s(sr, rhsp + (size_t)p0 * NV, szR, bar);
        if (Dinv32) bulk_g2s_hint(sDi, Dinv32 + (size_t)p0 * NB, szDi, bar, pol);
    }
    if (act && c32) c32[(size_t)p0 * NV + tid] = 0.0f;
    if (act) {
        sg[c * NV + i] = Up[(size_t)(p0 + c) * NV + i];
        if (nbr_pre) { /* indices loaded during the previous tile */
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if (s < nxf) {
                    const int nb = nbr_pre[s];
                    sg[((s + 1) * RES_TILE + c) * NV + i] = (nb >= 0) ? Up[(size_t)nb * NV + i] : 0.0;
                }
            }
        } else {
            for (int s = 0; s < nxf; ++s) {
                const int nb = xnbrf[(size_t)s * np16 + p0 + c];
                sg[((s + 1) * RES_TILE + c) * NV + i] = (nb >= 0) ? Up[(size_t)nb * NV + i] : 0.0;
            }
        }
    }
    const bool ok = mbar_wait(bar, parity);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicOr(status, ST_TIMEOUT);
            mbar_wait(bar, parity, 1LL << 28); /* let the copies land before the CTA retires */
        }
        return false;
    }
    double sq = 0.0;
    if (act) {
        const double *dr = sD + c * NB + i;
        const double *u = sg + c * NV;
        double a0, a1, a2;
        open_sums(a0, a1, a2, dr, u);
        close_sums(a0, a1, a2, dr, u);
        for (int s = 0; s < nxf; ++s) {
            const double *o = sX + (s * RES_TILE + c) * NB + i;
            const double *un = sg + ((s + 1) * RES_TILE + c) * NV;
            add_products(a0, a1, a2, o, un);
        }
        const double r = sr[c * NV + i] + (a0 + (a1 + a2));
        so[c * NV + i] = (float)r;
        sq = mul_rn(r, r);
    }
    __syncthreads();
    if (act) R32[(size_t)p0 * NV + tid] = so[tid]; /* contiguous tile store */
    if (Dinv32) {
        if (act) sb[c * NV + i] = neg_dinv_row<float>(sDi + c * NB + i, so + c * NV);
        __syncthreads();
        if (act) b32[(size_t)p0 * NV + tid] = sb[tid];
    }
    __shared__ double red[RES_THREADS_FAST / 32];
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
    if ((tid & 31) == 0) red[tid >> 5] = sq;
    __syncthreads();
    if (tid == 0) {
        double tot = 0.0;
        for (int w = 0; w < RES_THREADS_FAST / 32; ++w) tot += red[w];
        partials[blk] = tot;
    }
    return true;
}

/* persistent: CTA k takes tiles k, k + grid, ... */
__global__ void __launch_bounds__(RES_THREADS_FAST) full_resid_pos_kernel(
    int nxf, int np16, const double *__restrict__ Dp, const double *__restrict__ XF,
    const int *__restrict__ xnbrf, const double *__restrict__ rhsp, const double *__restrict__ Up,
    float *__restrict__ R32, double *__restrict__ partials, const float *__restrict__ Dinv32,
    float *__restrict__ b32, float *__restrict__ c32, unsigned *status) {
    uint64_t *bar = resid_bar_init();
    const int ntiles = np16 / RES_TILE;
    uint32_t parity = 0;
    /* the next tile's neighbour indices load during the current one */
    const bool pre = nxf >= 1 && nxf <= 4 && threadIdx.x < RES_TILE * NV;
    const int c = threadIdx.x % RES_TILE;
    int nbr[4], nxt[4];
#pragma unroll
    for (int s = 0; s < 4; ++s)
        nbr[s] = (pre && s < nxf && (int)blockIdx.x < ntiles)
                     ? xnbrf[(size_t)s * np16 + blockIdx.x * RES_TILE + c] : -1;
    for (int w = blockIdx.x; w < ntiles; w += gridDim.x) {
        const int wn = w + gridDim.x;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            nxt[s] = (pre && s < nxf && wn < ntiles) ? xnbrf[(size_t)s * np16 + wn * RES_TILE + c] : -1;
        const bool ok = full_resid_pos_body(nxf, np16, Dp, XF, xnbrf, rhsp, Up, R32, partials, Dinv32,
                                            b32, c32, status, w, bar, parity, pre ? nbr : nullptr);
        parity ^= 1u;
        if (!ok) break;
#pragma unroll
        for (int s = 0; s < 4; ++s) nbr[s] = nxt[s];
        __syncthreads(); /* the next tile's copies overwrite the stages */
    }
}

int launch_full_resid_pos(cudaStream_t st, const FastLayout &L, const double *Dp, const double *XF,
                          const double *rhsp, const double *Up, float *R32, double *partials,
                          const float *Dinv32, float *b32, float *c32, unsigned *status) {
    if (L.nxf < 0 || L.nxf > 4) return (int)cudaErrorInvalidValue;
    const size_t smem = fullpos_smem_bytes(L.nxf);
    const int grid = resid_grid_persistent((const void *)full_resid_pos_kernel, smem,
                                           fast_resid_grid(L.np16));
    full_resid_pos_kernel<<<grid, RES_THREADS_FAST, smem, st>>>(L.nxf, L.np16, Dp, XF, L.xnbrf, rhsp,
                                                                Up, R32, partials, Dinv32, b32, c32,
                                                                status);
    return (int)cudaGetLastError();
}

/* ================================================ mixed-precision prime
 * Per tile of RES_TILE positions (160 threads, 144 active): U = 0, the
 * FP32 copy of the residual R = rhs, and the tile's sum rhs^2 in a fixed
 * order (lane order within a warp, then warps in order). */
__device__ __forceinline__ void mixed_prime_body(const double *__restrict__ rhsp,
                                                 float *__restrict__ R32, double *__restrict__ Up,
                                                 double *__restrict__ partials,
                                                 const float *__restrict__ Dinv32,
                                                 float *__restrict__ b32, float *__restrict__ c32,
                                                 int blk) {
    const int tid = threadIdx.x;
    const bool act = tid < RES_TILE * NV;
    __shared__ float sR[RES_TILE * NV];
    __shared__ float4 sDi[RES_TILE * NB / 4];
    double sq = 0.0;
    /* HBM bounds it: the tile's Dinv32 in 16-byte words, all on their way
     * before anything waits (600x640: 58 us in 4-byte words, 46 now) */
    constexpr int WORDS = (RES_TILE * NB / 4 + RES_THREADS_FAST - 1) / RES_THREADS_FAST;
    float4 di[WORDS];
    if (Dinv32) {
        const float4 *src = reinterpret_cast<const float4 *>(Dinv32) + (size_t)blk * (RES_TILE * NB / 4);
#pragma unroll
        for (int k = 0; k < WORDS; ++k)
            if (tid + k * RES_THREADS_FAST < RES_TILE * NB / 4) di[k] = __ldg(src + tid + k * RES_THREADS_FAST);
    }
    if (act) {
        const size_t q = (size_t)blk * RES_TILE * NV + tid;
        const double v = rhsp[q];
        R32[q] = (float)v;
        sR[tid] = (float)v;
        Up[q] = 0.0;
        if (c32) c32[q] = 0.0f;
        sq = mul_rn(v, v);
    }
    if (Dinv32) {
        /* the first inner solve's right-hand side b32 = -Dinv32 R32 */
#pragma unroll
        for (int k = 0; k < WORDS; ++k)
            if (tid + k * RES_THREADS_FAST < RES_TILE * NB / 4) sDi[tid + k * RES_THREADS_FAST] = di[k];
        __syncthreads();
        if (act) {
            const int c = tid / NV, i = tid % NV;
            b32[(size_t)blk * RES_TILE * NV + tid] =
                neg_dinv_row<float>(reinterpret_cast<const float *>(sDi) + c * NB + i, sR + c * NV);
        }
    }
    __shared__ double red[RES_THREADS_FAST / 32];
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
    if ((tid & 31) == 0) red[tid >> 5] = sq;
    __syncthreads();
    if (tid == 0) {
        double tot = 0.0;
        for (int w = 0; w < RES_THREADS_FAST / 32; ++w) tot += red[w];
        partials[blk] = tot;
    }
}

/* one CTA per tile (measured faster than a persistent loop here) */
__global__ void __launch_bounds__(RES_THREADS_FAST) mixed_prime_kernel(
    const double *__restrict__ rhsp, float *__restrict__ R32, double *__restrict__ Up,
    double *__restrict__ partials, const float *__restrict__ Dinv32, float *__restrict__ b32,
    float *__restrict__ c32) {
    mixed_prime_body(rhsp, R32, Up, partials, Dinv32, b32, c32, blockIdx.x);
}

int launch_mixed_prime(cudaStream_t st, const FastLayout &L, const double *rhsp, float *R32,
                       double *Up, double *partials, const float *Dinv32, float *b32, float *c32) {
    mixed_prime_kernel<<<fast_resid_grid(L.np16), RES_THREADS_FAST, 0, st>>>(rhsp, R32, Up, partials,
                                                                             Dinv32, b32, c32);
    return (int)cudaGetLastError();
}

/* ================================================================ batches
 * Every batched kernel reads its work count from device memory (a field of
 * the launch sequence's BatchCtl), so one instantiated graph serves any set
 * of members; all but the per-member norm kernel are persistent, with grids
 * sized to the SMs. */

/* Item w of a group index (layout in tbs_internal.hxx): the group by
 * binary search over the prefix sums, then unit-major within the group. */
__device__ __forceinline__ WorkItem group_item(const int *__restrict__ gi, int w) {
    const int ng = gi[0];
    const int *base = gi + 1;
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    const int *nmem = base + ng + 1, *moff = nmem + ng, *mlist = moff + ng;
    const int off = w - base[lo], r = nmem[lo];
    return WorkItem{mlist[moff[lo] + off % r], off / r};
}

__device__ __forceinline__ int group_items(const int *__restrict__ gi) { return gi[1 + gi[0]]; }

/* group_item for a CTA that visits items in increasing order: the group of
 * the last item (its range [lo, hi) and index g) is kept, so the binary
 * search runs only when the item leaves it */
struct GroupCursor {
    int lo = 0, hi = 0, g = -1;
    int r = 1, mo = 0, m0 = 0; /* the group's member count, list offset, first member */
};

__device__ __forceinline__ WorkItem group_item_next(const int *__restrict__ gi, int w, GroupCursor &c) {
    const int ng = gi[0];
    const int *base = gi + 1;
    const int *nmem = base + ng + 1, *moff = nmem + ng, *mlist = moff + ng;
    if (c.g < 0 || w < c.lo || w >= c.hi) {
        int lo = 0, hi = ng - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (base[mid] <= w) lo = mid;
            else hi = mid - 1;
        }
        c.g = lo;
        c.lo = base[lo];
        c.hi = base[lo + 1];
        c.r = nmem[lo];
        c.mo = moff[lo];
        c.m0 = mlist[c.mo];
    }
    const int off = w - c.lo;
    if (c.r == 1) return WorkItem{c.m0, off};
    return WorkItem{mlist[c.mo + off % c.r], off / c.r};
}

static int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

template <typename T>
size_t thomas_batch_smem(int stages, int warps) {
    return (warps == 2 ? thomas_hdr<true>() : thomas_hdr<false>()) +
           (size_t)stages * 2 * THOMAS_P * (NB + NV) * sizeof(T) + BCAST<T, NV> * sizeof(T);
}

template <typename T>
int thomas_batch_fit(int stages, int warps) {
    int n = 0;
    const size_t smem = thomas_batch_smem<T>(stages, warps);
    const void *fn = warps == 2 ? (const void *)fast_thomas_batch_ws_kernel<T, THOMAS_P>
                                : (const void *)fast_thomas_batch_kernel<T, THOMAS_P>;
    if (smem_raise(fn, smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 32 * warps, smem) != cudaSuccess)
        return 0;
    return n;
}

template <typename T>
int launch_thomas_batch(cudaStream_t st, const BatchSched &bs, const ThomasSys<T> *sys,
                        const WorkItem *work, const int *nwork, const int *active, unsigned *queue,
                        unsigned *status) {
    if (bs.stages < 2 || bs.stages > 8 || bs.ctas_per_sm < 1 || (bs.warps != 1 && bs.warps != 2))
        return (int)cudaErrorInvalidValue;
    const size_t smem = thomas_batch_smem<T>(bs.stages, bs.warps);
    const int grid = bs.ctas_per_sm * sm_count();
    if (bs.warps == 2)
        fast_thomas_batch_ws_kernel<T, THOMAS_P><<<grid, 64, smem, st>>>(sys, work, nwork, active,
                                                                          queue, bs.stages, status);
    else
        fast_thomas_batch_kernel<T, THOMAS_P><<<grid, 32, smem, st>>>(sys, work, nwork, active,
                                                                       queue, bs.stages, status);
    return (int)cudaGetLastError();
}

/* The tiles [unit * chunk, ...) of a member: the units of a group index
 * are single tiles (chunk 1) or chunks of BATCH_CHUNK tiles, which pay the
 * item's decode and descriptor load once for several tiles */
__device__ __forceinline__ int chunk_end(int unit, int chunk, int ntiles) {
    const int e = (unit + 1) * chunk;
    return e < ntiles ? e : ntiles;
}

/* persistent residual over (member, tile) items: CTA k takes items k,
 * k + grid, ...; each tile completes one phase of the CTA's barrier and writes
 * its own partial */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST, 8) fast_resid_batch_kernel(
    const ResidSys<T> *__restrict__ sys, const int *__restrict__ groups, int mode,
    const int *__restrict__ active, unsigned *status) {
    uint64_t *bar = resid_bar_init();
    const int nwork = group_items(groups);
    uint32_t parity = 0;
    GroupCursor gc;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = group_item_next(groups, w, gc);
        if (active && !active[it.sys]) continue;
        const ResidSys<T> S = sys[it.sys];
        NormSink ns{};
        ns.partials = (mode == 3) ? nullptr : S.partials; /* no counter: partials only */
        if (!fast_resid_body<T>(mode == 0 ? 0 : S.nx, S.np16, mode, S.Dinv, S.X, S.xnbr, S.dU, S.Rsrc, S.b,
                                S.Uacc, ns, status, it.unit, bar, parity))
            return;
        parity ^= 1u;
        __syncthreads(); /* the next tile's copies overwrite the stages */
    }
}

/* A CTA's tiles of those of the active members of `groups` (one member a
 * group, units of single tiles): run(member, first tile, tile behind the last)
 * for each piece, until one returns false.  Full waves give each CTA
 * BATCH_CHUNK consecutive tiles, the tiles left over are dealt equally to a
 * tile.  (Equal consecutive shares of all tiles spread the CTAs' reads over
 * the whole of memory: 8 systems of 600x640 took 15.4 ms, not 14.0.)  All
 * threads take part; each warp makes the prefix sums for itself. */
template <typename F>
__device__ __forceinline__ void active_share(const int *__restrict__ groups, const int *__restrict__ active,
                                             F &&run) {
    const int ng = groups[0];
    const int *base = groups + 1, *mlist = base + (ng + 1) + 2 * ng;
    const int lane = threadIdx.x & 31;
    auto tiles = [&](int g, int &m) {
        m = g < ng ? mlist[g] : -1;
        return m >= 0 && active[m] ? base[g + 1] - base[g] : 0;
    };
    int total = 0, m;
    for (int g = lane; g - lane < ng; g += 32) total += tiles(g, m);
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(FULL, total, o);
    const int wave = gridDim.x * BATCH_CHUNK;
    for (int w0 = 0; w0 < total;) {
        const int left = total - w0, deal = left < wave ? left : wave;
        const int s = w0 + (int)((long long)deal * blockIdx.x / gridDim.x);
        const int e = w0 + (int)((long long)deal * (blockIdx.x + 1) / gridDim.x);
        w0 += deal;
        int before = 0;
        for (int g = lane; g - lane < ng && before < e; g += 32) {
            const int n = tiles(g, m);
            int pre = n;
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(FULL, pre, o);
                if (lane >= o) pre += x;
            }
            pre += before;
            before = __shfl_sync(FULL, pre, 31);
            pre -= n;
            for (unsigned hit = __ballot_sync(FULL, pre < e && pre + n > s); hit; hit &= hit - 1) {
                const int j = __ffs(hit) - 1;
                const int p = __shfl_sync(FULL, pre, j), nj = __shfl_sync(FULL, n, j);
                if (!run(__shfl_sync(FULL, m, j), max(s - p, 0), min(e - p, nj))) return;
            }
        }
    }
}

/* The sweep residual (mode 1) of the members alone in their system.  HBM
 * bounds it, as the single-system launch, when every CTA has the same work:
 * dealt in chunks of 8 tiles, 12 systems of 117 000 cells together gave 37 of
 * 888 CTAs a second chunk and took 66 us for 53 now. */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST, 6) fast_resid_solo_kernel(
    const ResidSys<T> *__restrict__ sys, const int *__restrict__ groups, const int *__restrict__ active,
    unsigned *status) {
    uint64_t *bar = resid_bar_init();
    uint32_t parity = 0;
    active_share(groups, active, [&](int member, int tb, int t1) {
        const ResidSys<T> S = sys[member];
        NormSink ns{};
        ns.partials = S.partials; /* no counter: partials only */
        /* the next tile's neighbour indices load during the current tile */
        const bool pre = S.nx >= 1 && S.nx <= 4 && threadIdx.x < RES_TILE * NV;
        const int c = threadIdx.x % RES_TILE;
        int nbr[4], nxt[4];
#pragma unroll
        for (int s = 0; s < 4; ++s)
            nbr[s] = (pre && s < S.nx) ? S.xnbr[(size_t)s * S.np16 + tb * RES_TILE + c] : -1;
        for (int t = tb; t < t1; ++t) {
#pragma unroll
            for (int s = 0; s < 4; ++s)
                nxt[s] = (pre && s < S.nx && t + 1 < t1) ? S.xnbr[(size_t)s * S.np16 + (t + 1) * RES_TILE + c]
                                                         : -1;
            const bool ok = fast_resid_body<T>(S.nx, S.np16, 1, S.Dinv, S.X, S.xnbr, S.dU, S.Rsrc, S.b, S.Uacc,
                                               ns, status, t, bar, parity, pre ? nbr : nullptr);
            parity ^= 1u;
            if (!ok) return false;
#pragma unroll
            for (int s = 0; s < 4; ++s) nbr[s] = nxt[s];
            __syncthreads(); /* the next tile's copies overwrite the stages */
        }
        return true;
    });
}

/* Item w of a unit index (the group index layout with base[] the prefix
 * sums of each group's units, not units x members): (group, unit). */
__device__ __forceinline__ int2 group_unit(const int *__restrict__ gi, int w) {
    const int ng = gi[0];
    const int *base = gi + 1;
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    return make_int2(lo, w - base[lo]);
}

/* The sweep residual (mode 1) of the members of one system together: an
 * item is (system group, chunk of tiles); per tile the CTA stages the
 * system's Dinv and cross-line blocks once and then runs every active
 * member (one right-hand side each) over them, with fast_resid_body's
 * arithmetic, in its order, for each: U += dU, neighbour gathers, R, b,
 * the tile's partial.  The members' blocks are read from HBM once per tile
 * instead of once per member. */
template <typename T>
__global__ void __launch_bounds__(RES_THREADS_FAST) fast_resid_group_kernel(
    const ResidSys<T> *__restrict__ sys, const int *__restrict__ gunits, int chunk,
    const int *__restrict__ active, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[RES_THREADS_FAST / 32];
    uint64_t *bar = resid_bar_init();
    const int ng = gunits[0];
    const int nwork = gunits[1 + ng];
    const int *nmem = gunits + 2 + ng, *moff = nmem + ng, *mlist = moff + ng;
    const int tid = threadIdx.x;
    const int c = tid % RES_TILE, i = tid / RES_TILE;
    const bool act = tid < RES_TILE * NV;
    uint32_t parity = 0;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int2 gu = group_unit(gunits, w);
        const int *ml = mlist + moff[gu.x];
        const int r = nmem[gu.x];
        const ResidSys<T> S0 = sys[ml[0]];
        const int nx = S0.nx, np16 = S0.np16;
        const int nxa = nx > 0 ? nx : 1;
        T *sD = reinterpret_cast<T *>(smem + 128);
        T *sX = sD + RES_TILE * NB;
        T *sg = sX + nx * RES_TILE * NB;
        T *sr = sg + nxa * RES_TILE * NV;
        T *sb = sr + RES_TILE * NV;
        const uint32_t szD = RES_TILE * NB * sizeof(T);
        const int t1 = chunk_end(gu.y, chunk, np16 / RES_TILE);
        const int tb = gu.y * chunk;
        /* a tile's neighbour indices serve every member; the next tile's
         * load while this one is worked on */
        int nb[4], nbn[4];
#pragma unroll
        for (int s = 0; s < 4; ++s)
            nb[s] = (act && s < nx && tb < t1) ? S0.xnbr[(size_t)s * np16 + tb * RES_TILE + c] : -1;
        for (int t = tb; t < t1; ++t) {
            const int p0 = t * RES_TILE;
            if (tid == 0) {
                const uint64_t pol = policy_evict_first();
                mbar_arrive_expect_tx(bar, (1 + nx) * szD);
                bulk_g2s_hint(sD, S0.Dinv + (size_t)p0 * NB, szD, bar, pol);
                for (int s = 0; s < nx; ++s)
                    bulk_g2s_hint(sX + s * RES_TILE * NB, S0.X + ((size_t)s * np16 + p0) * NB, szD, bar,
                                  pol);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s)
                nbn[s] = (act && s < nx && t + 1 < t1) ? S0.xnbr[(size_t)s * np16 + (t + 1) * RES_TILE + c]
                                                       : -1;
            /* members in a software pipeline: the next active member's
             * loads (its U and dU, its neighbour gathers) are issued before
             * the current one's products, so they overlap them */
            const size_t q = (size_t)p0 * NV + tid;
            auto next_active = [&](int k) {
                while (k < r && active && !active[ml[k]]) ++k;
                return k;
            };
            auto load_member = [&](const ResidSys<T> &S, T &u, T &d, T (&g)[4]) {
                u = d = T(0);
#pragma unroll
                for (int s = 0; s < 4; ++s) g[s] = T(0);
                if (!act) return;
                d = S.dU[q];
                if (S.Uacc) u = S.Uacc[q];
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    if (s < nx && nb[s] >= 0) g[s] = S.dU[(size_t)nb[s] * NV + i];
            };
            bool staged = false;
            int k = next_active(0);
            ResidSys<T> Sc{};
            T cu, cd, cg[4];
            if (k < r) {
                Sc = sys[ml[k]];
                load_member(Sc, cu, cd, cg);
            }
            while (k < r) {
                if (act && Sc.Uacc) Sc.Uacc[q] = cu + cd;
                if (act) {
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        if (s < nx) sg[(s * RES_TILE + c) * NV + i] = cg[s];
                }
                const int kn = next_active(k + 1);
                ResidSys<T> Sn{};
                T nu = T(0), nd = T(0), ngv[4] = {T(0), T(0), T(0), T(0)};
                if (kn < r) {
                    Sn = sys[ml[kn]];
                    load_member(Sn, nu, nd, ngv);
                }
                if (!staged) {
                    const bool ok = mbar_wait(bar, parity);
                    parity ^= 1u;
                    staged = true;
                    if (__syncthreads_or(!ok)) {
                        if (tid == 0) {
                            atomicOr(status, ST_TIMEOUT);
                            mbar_wait(bar, parity ^ 1u, 1LL << 28);
                        }
                        return;
                    }
                } else {
                    __syncthreads();
                }
                T rr = T(0);
                if (act) {
                    T a0 = T(0), a1 = T(0), a2 = T(0);
                    for (int s = 0; s < nx; ++s) {
                        const T *xr = sX + (s * RES_TILE + c) * NB + i;
                        const T *g = sg + (s * RES_TILE + c) * NV;
                        add_products(a0, a1, a2, xr, g);
                    }
                    rr = a0 + (a1 + a2);
                    sr[c * NV + i] = rr;
                }
                __syncthreads();
                double sq = act ? mul_rn((double)rr, (double)rr) : 0.0;
                if (act) sb[c * NV + i] = neg_dinv_row<T>(sD + c * NB + i, sr + c * NV);
                __syncthreads();
                if (act) Sc.b[(size_t)p0 * NV + tid] = sb[tid];
                for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(FULL, sq, o);
                if ((tid & 31) == 0) red[tid >> 5] = sq;
                __syncthreads();
                if (tid == 0) {
                    double tot = 0.0;
                    for (int ww = 0; ww < RES_THREADS_FAST / 32; ++ww) tot += red[ww];
                    Sc.partials[t] = tot;
                }
                __syncthreads(); /* the next member overwrites sg, sr, sb and red */
                Sc = Sn;
                cu = nu;
                cd = nd;
#pragma unroll
                for (int s = 0; s < 4; ++s) cg[s] = ngv[s];
                k = kn;
            }
            if (!staged) { /* no member active: the tile's copies still land */
                const bool ok = mbar_wait(bar, parity);
                parity ^= 1u;
                if (__syncthreads_or(!ok)) {
                    if (tid == 0) {
                        atomicOr(status, ST_TIMEOUT);
                        mbar_wait(bar, parity ^ 1u, 1LL << 28);
                    }
                    return;
                }
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) nb[s] = nbn[s];
            __syncthreads(); /* the next tile's copies overwrite the stages */
        }
    }
}

static int resid_batch_grid(size_t smem, const void *fn) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, RES_THREADS_FAST, smem) != cudaSuccess ||
        per < 1)
        per = 1;
    return per * sm_count();
}

template <typename T>
int launch_resid_batch(cudaStream_t st, int mode, int max_nx, const ResidSys<T> *sys,
                       const int *groups, const int *active, unsigned *status) {
    if (mode != 0 && mode != 3) return (int)cudaErrorInvalidValue;
    const size_t smem = resid_smem_bytes<T>(mode == 0 ? 0 : max_nx);
    const int grid = resid_batch_grid(smem, (const void *)fast_resid_batch_kernel<T>);
    fast_resid_batch_kernel<T><<<grid, RES_THREADS_FAST, smem, st>>>(sys, groups, mode, active, status);
    return (int)cudaGetLastError();
}

int launch_resid_solo(cudaStream_t st, int max_nx, const ResidSys<double> *sys, const int *groups,
                      const int *active, unsigned *status) {
    const size_t smem = resid_smem_bytes<double>(max_nx);
    const int grid = resid_batch_grid(smem, (const void *)fast_resid_solo_kernel<double>);
    fast_resid_solo_kernel<double><<<grid, RES_THREADS_FAST, smem, st>>>(sys, groups, active, status);
    return (int)cudaGetLastError();
}

__global__ void __launch_bounds__(FULLRES_THREADS) full_resid_batch_kernel(
    const FullResSys *__restrict__ sys, const int *__restrict__ groups,
    const int *__restrict__ active) {
    const int nwork = group_items(groups);
    GroupCursor gc;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = group_item_next(groups, w, gc);
        if (active && !active[it.sys]) continue;
        const FullResSys S = sys[it.sys];
        full_resid_body<float>(S.nelem, S.epoint, S.ef, S.fc, S.pos_of_elem, S.D, S.O1, S.O2,
                               S.rhs, S.Up, S.R32, S.partials, it.unit);
        __syncthreads(); /* the block sum's shared array is reused */
    }
}

static int plain_batch_grid(const void *fn, int threads) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, 0) != cudaSuccess || per < 1)
        per = 1;
    return per * sm_count();
}

int launch_full_resid_batch(cudaStream_t st, const FullResSys *sys, const int *groups,
                            const int *active) {
    const int grid = plain_batch_grid((const void *)full_resid_batch_kernel, FULLRES_THREADS);
    full_resid_batch_kernel<<<grid, FULLRES_THREADS, 0, st>>>(sys, groups, active);
    return (int)cudaGetLastError();
}

__global__ void __launch_bounds__(RES_THREADS_FAST) mixed_prime_batch_kernel(
    const VecSys *__restrict__ sys, const int *__restrict__ groups) {
    const int nwork = group_items(groups);
    GroupCursor gc;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = group_item_next(groups, w, gc);
        const VecSys S = sys[it.sys];
        mixed_prime_body(S.rhsp, S.R32, S.Up, S.partials, S.Dinv32, S.b32, S.c32, it.unit);
        __syncthreads();
    }
}

int launch_mixed_prime_batch(cudaStream_t st, const VecSys *sys, const int *groups) {
    const int grid = plain_batch_grid((const void *)mixed_prime_batch_kernel, RES_THREADS_FAST);
    mixed_prime_batch_kernel<<<grid, RES_THREADS_FAST, 0, st>>>(sys, groups);
    return (int)cudaGetLastError();
}

/* U += c + d over one tile (elementwise: the same values as axpy2_kernel) */
__global__ void __launch_bounds__(RES_THREADS_FAST) axpy2_batch_kernel(
    const VecSys *__restrict__ sys, const int *__restrict__ groups,
    const int *__restrict__ active) {
    const int nwork = group_items(groups);
    GroupCursor gc;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = group_item_next(groups, w, gc);
        if (active && !active[it.sys]) continue;
        if (threadIdx.x >= RES_TILE * NV) continue;
        const VecSys S = sys[it.sys];
        const size_t q = (size_t)it.unit * RES_TILE * NV + threadIdx.x;
        S.Up[q] += (double)S.c32[q] + (double)S.d32[q];
    }
}

int launch_axpy2_batch(cudaStream_t st, const VecSys *sys, const int *groups, const int *active) {
    const int grid = plain_batch_grid((const void *)axpy2_batch_kernel, RES_THREADS_FAST);
    axpy2_batch_kernel<<<grid, RES_THREADS_FAST, 0, st>>>(sys, groups, active);
    return (int)cudaGetLastError();
}

__global__ void __launch_bounds__(RES_THREADS_FAST) full_resid_pos_batch_kernel(
    const FullPosSys *__restrict__ sys, const int *__restrict__ groups, int chunk,
    const int *__restrict__ active, unsigned *status) {
    uint64_t *bar = resid_bar_init();
    const int nwork = group_items(groups);
    uint32_t parity = 0;
    GroupCursor gc;
    bool ok = true;
    for (int w = blockIdx.x; w < nwork && ok; w += gridDim.x) {
        const WorkItem it = group_item_next(groups, w, gc);
        if (active && !active[it.sys]) continue;
        const FullPosSys S = sys[it.sys];
        const int t1 = chunk_end(it.unit, chunk, S.np16 / RES_TILE);
        /* the next tile's neighbour indices load during the current one */
        const bool pre = chunk > 1 && S.nxf >= 1 && S.nxf <= 4 && threadIdx.x < RES_TILE * NV;
        const int c = threadIdx.x % RES_TILE;
        int nbr[4], nxt[4];
        const int tb = it.unit * chunk;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            nbr[s] = (pre && s < S.nxf && tb < t1) ? S.xnbrf[(size_t)s * S.np16 + tb * RES_TILE + c] : -1;
        for (int t = tb; t < t1; ++t) {
#pragma unroll
            for (int s = 0; s < 4; ++s)
                nxt[s] = (pre && s < S.nxf && t + 1 < t1)
                             ? S.xnbrf[(size_t)s * S.np16 + (t + 1) * RES_TILE + c] : -1;
            ok = full_resid_pos_body(S.nxf, S.np16, S.Dp, S.XF, S.xnbrf, S.rhsp, S.Up, S.R32,
                                     S.partials, S.Dinv32, S.b32, S.c32, status, t, bar, parity,
                                     pre ? nbr : nullptr);
            parity ^= 1u;
            if (!ok) break;
#pragma unroll
            for (int s = 0; s < 4; ++s) nbr[s] = nxt[s];
            __syncthreads(); /* the next tile's copies overwrite the stages */
        }
    }
}

template <typename T>
int launch_resid_group(cudaStream_t st, int max_nx, const ResidSys<T> *sys, const int *gunits, int chunk,
                       const int *active, unsigned *status) {
    const size_t smem = resid_smem_bytes<T>(max_nx);
    const int grid = resid_batch_grid(smem, (const void *)fast_resid_group_kernel<T>);
    fast_resid_group_kernel<T><<<grid, RES_THREADS_FAST, smem, st>>>(sys, gunits, chunk, active, status);
    return (int)cudaGetLastError();
}
template int launch_resid_group<double>(cudaStream_t, int, const ResidSys<double> *, const int *, int,
                                        const int *, unsigned *);

int launch_full_resid_pos_batch(cudaStream_t st, int max_nxf, const FullPosSys *sys,
                                const int *groups, int chunk, const int *active, unsigned *status) {
    const size_t smem = fullpos_smem_bytes(max_nxf);
    const int grid = resid_batch_grid(smem, (const void *)full_resid_pos_batch_kernel);
    full_resid_pos_batch_kernel<<<grid, RES_THREADS_FAST, smem, st>>>(sys, groups, chunk, active,
                                                                      status);
    return (int)cudaGetLastError();
}

/* One CTA per descriptor (grid = capacity; CTAs beyond *nred only take
 * their ticket).  The last CTA to finish decides whether the graph's loop
 * goes on: some member is active, the sweep limit of the launch is not
 * reached and, when asked, no member stopped during the launch. */
__global__ void batch_reduce_kernel(const ReduceSys *__restrict__ sys, const int *__restrict__ nred_p,
                                    int is_start, int *active, BatchCtl *ctl, unsigned *counter,
                                    cudaGraphConditionalHandle handle, int use_cond,
                                    cudaGraphConditionalHandle handle2, int use2) {
    __shared__ double red[32];
    __shared__ unsigned ticket;
    const int s = blockIdx.x;
    if (s < *nred_p) {
        const ReduceSys R = sys[s];
        const int m = R.member;
        if (is_start || active[m]) {
            double acc = strided_sum(R.partials, R.n, (int)blockDim.x);
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(FULL, acc, o);
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
            __syncthreads();
            if (threadIdx.x == 0) {
                double tot = 0.0;
                for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) tot += red[w];
                const double nrm = sqrt(tot);
                SolveState *S = R.state;
                if (is_start) {
                    S->sweep = 0;
                    S->norm0 = nrm;
                } else {
                    S->sweep += 1;
                }
                const int sw = S->sweep;
                if (sw < S->hist_cap) R.hist[sw] = nrm;
                S->last = nrm;
                const bool go = isfinite(nrm) && nrm > S->tol * S->norm0 && sw < S->max_sweeps;
                active[m] = go ? 1 : 0;
                if (!go) ctl->finished = 1;
            }
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        ticket = atomicAdd(counter, 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0 && ticket == gridDim.x - 1) {
        __threadfence();
        int any = 0;
        const int n = ctl->nsys;
        for (int k = 0; k < n; ++k) any |= __ldcg(active + k);
        bool go = any != 0;
        if (!is_start && ctl->chunk_limit > 0) {
            ctl->chunk += 1;
            if (ctl->chunk >= ctl->chunk_limit) go = false;
        }
        if (ctl->stop_on_finish && __ldcg(&ctl->finished)) go = false;
        if (use_cond) cudaGraphSetConditional(handle, go ? 1u : 0u);
        if (use2) cudaGraphSetConditional(handle2, go ? 1u : 0u);
        *counter = 0u;
    }
}

int launch_reduce_batch(cudaStream_t st, int threads, const ReduceSys *sys, const int *nred,
                        int cap, int is_start, int *active, BatchCtl *ctl, unsigned *counter,
                        unsigned long long cond_handle, int use_cond,
                        unsigned long long cond_handle2, int use2) {
    if (cap <= 0) return 0;
    if (threads != RES_THREADS_FAST && threads != REDUCE_THREADS) return (int)cudaErrorInvalidValue;
    batch_reduce_kernel<<<cap, threads, 0, st>>>(sys, nred, is_start, active, ctl, counter,
                                                 (cudaGraphConditionalHandle)cond_handle, use_cond,
                                                 (cudaGraphConditionalHandle)cond_handle2, use2);
    return (int)cudaGetLastError();
}

/* member blockIdx.x's state and the norms of its history to host rows of
 * `stride` norms */
__global__ void batch_collect_kernel(const ReduceSys *__restrict__ sys, SolveState *states, double *hist,
                                     int stride) {
    const ReduceSys R = sys[blockIdx.x];
    const int n = min(R.state->sweep + 1, stride);
    if (threadIdx.x == 0) states[blockIdx.x] = *R.state;
    for (int k = threadIdx.x; k < n; k += blockDim.x) hist[(size_t)blockIdx.x * stride + k] = R.hist[k];
}

int launch_batch_collect(cudaStream_t st, const ReduceSys *sys, int n, SolveState *states, double *hist,
                         int stride) {
    if (n <= 0) return 0;
    batch_collect_kernel<<<n, 64, 0, st>>>(sys, states, hist, stride);
    return (int)cudaGetLastError();
}

/* opt the batched kernels into the shared memory of the widest member
 * (outside stream capture) */
int batch_prepare(int max_nx) {
    int rc = set_smem((const void *)fast_resid_batch_kernel<double>, resid_smem_bytes<double>(max_nx));
    if (!rc) rc = set_smem((const void *)fast_resid_solo_kernel<double>, resid_smem_bytes<double>(max_nx));
    if (!rc) rc = set_smem((const void *)fast_resid_batch_kernel<float>, resid_smem_bytes<float>(max_nx));
    if (!rc)
        rc = set_smem((const void *)fast_resid_group_kernel<double>, resid_smem_bytes<double>(max_nx));

    if (!rc) rc = set_smem((const void *)full_resid_pos_batch_kernel, fullpos_smem_bytes(4));
    return rc;
}

int fullpos_prepare(const FastLayout &L) {
    return set_smem((const void *)full_resid_pos_kernel, fullpos_smem_bytes(L.nxf));
}

template size_t thomas_batch_smem<double>(int, int);
template size_t thomas_batch_smem<float>(int, int);
template int thomas_batch_fit<double>(int, int);
template int thomas_batch_fit<float>(int, int);
template int launch_thomas_batch<double>(cudaStream_t, const BatchSched &, const ThomasSys<double> *,
                                         const WorkItem *, const int *, const int *, unsigned *,
                                         unsigned *);
template int launch_thomas_batch<float>(cudaStream_t, const BatchSched &, const ThomasSys<float> *,
                                        const WorkItem *, const int *, const int *, unsigned *,
                                        unsigned *);
template int launch_resid_batch<double>(cudaStream_t, int, int, const ResidSys<double> *, const int *,
                                        const int *, unsigned *);
template int launch_resid_batch<float>(cudaStream_t, int, int, const ResidSys<float> *, const int *,
                                        const int *, unsigned *);


/* ============================================== several right-hand sides
 * nr <= MULTI_MAX right-hand sides of one factored system swept together
 * (TBS_ALGO_FP64): the line blocks (G, Gam, Dinv, X) are read once per
 * sweep for all of them.  Vectors are RHS-major: right-hand side r of a
 * vector v starts at v + r * vs, vs = np16 * 9.  A right-hand side whose
 * solve has ended (active[r] == 0) is skipped by every kernel, so its
 * solution stays the one of its last sweep, and the per-element arithmetic
 * is the single-system kernels' own: every right-hand side's iterates,
 * norms and sweep count are bit-identical to a solve of it alone. */

/* Forward / backward chunk steps of thomas_line's chains for MULTI_RPW
 * right-hand sides at once: the row of G (Gam) is loaded once per step and
 * feeds one dot product per right-hand side, each with row_dot's own
 * expression, so every right-hand side's values are those of fwd_chunk /
 * bwd_chunk.  Right-hand side j reads its b chunk at sB[j], publishes its
 * vector through bc[j] and writes y (dU) through yg[j] (dUl[j]); only the
 * first `nown` of them write. */
constexpr int MULTI_RPW = 2;

/* AHEAD: the vectors of both right-hand sides of a warp are read before either
 * product; else each before its own, which takes 36 registers fewer.  The
 * kernel of one system has room for them (8 right-hand sides at 360x384: 155 us
 * for 161); the one that reads its lines' addresses from memory has not (it
 * spilled: 2 right-hand sides 111 us, 83 without). */
template <int P, bool CHECK, bool AHEAD>
__device__ __forceinline__ void fwd_chunk_m(const double *sG, const double *const *sB,
                                            double *const *bc, double *const *yg, int nown,
                                            int kbase, int len, int cpos, int i) {
    Row<double, NV> cur_row, next_row;
    load_row(cur_row, sG, i, 0);
    double cur_b[MULTI_RPW], next_b[MULTI_RPW];
#pragma unroll
    for (int j = 0; j < MULTI_RPW; ++j) cur_b[j] = sB[j][i];
#pragma unroll
    for (int q = 0; q < P; ++q) {
        StepVec<double, NV> v[MULTI_RPW];
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j) {
            if (AHEAD) v[j].load(bc[j] + (q & 1) * 10, i, 0);
            next_b[j] = 0.0;
        }
        if (q + 1 < P) {
            load_row(next_row, sG + (q + 1) * NB, i, 0);
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) next_b[j] = sB[j][(q + 1) * NV + i];
        }
        double yi[MULTI_RPW];
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j) {
            if (!AHEAD) v[j].load(bc[j] + (q & 1) * 10, i, 0);
            yi[j] = row_dot(cur_row, v[j], cur_b[j]);
        }
        /* lanes 9..15 repeat lane 8's row, value and address: no divergence */
        if (!CHECK || kbase + q < len) {
            const int pos = cpos + kbase + q;
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) {
                if (j < nown) {
                    bc[j][((q & 1) ^ 1) * 10 + i] = yi[j];
                    yg[j][(size_t)pos * NV + i] = yi[j];
                }
            }
        }
        __syncwarp();
        cur_row = next_row;
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j) cur_b[j] = next_b[j];
    }
}

template <int P, bool CHECK, bool AHEAD>
__device__ __forceinline__ void bwd_chunk_m(const double *sG, double *const *bc,
                                            const double (*yv)[P], double *const *dUl, int nown,
                                            int kbase, int len, int cpos, int i) {
    Row<double, NV> cur_row, next_row;
    load_row(cur_row, sG + (P - 1) * NB, i, 0);
#pragma unroll
    for (int q = P - 1; q >= 0; --q) {
        const int f = (P - 1 - q) & 1;
        StepVec<double, NV> v[MULTI_RPW];
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j)
            if (AHEAD) v[j].load(bc[j] + f * 10, i, 0);
        if (q > 0) load_row(next_row, sG + (q - 1) * NB, i, 0);
        const bool valid = !CHECK || (kbase + q >= 0 && kbase + q < len);
        const int pos = cpos + kbase + q;
        double d[MULTI_RPW];
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j) {
            if (!AHEAD) v[j].load(bc[j] + f * 10, i, 0);
            d[j] = row_dot(cur_row, v[j], valid ? yv[j][q] : 0.0);
        }
        if (valid) { /* lanes 9..15 repeat lane 8's row, value and address */
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) {
                if (j < nown) {
                    bc[j][(f ^ 1) * 10 + i] = d[j];
                    dUl[j][(size_t)pos * NV + i] = d[j];
                }
            }
        }
        __syncwarp();
        cur_row = next_row;
    }
}

/* Thomas: one CTA per line; warp w solves the active right-hand sides
 * 2w and 2w+1 (in active order) with the chains of thomas_line (y in
 * global memory).  Thread 0 streams the jobs through an NS-stage ring; a
 * forward stage holds, for either chain, a chunk of G rows followed by the
 * chunks of b of the active right-hand sides, a backward stage a chunk of
 * Gam rows.  All warps have consumed a stage before it is refilled (one
 * CTA barrier per chunk). */
template <int P, bool AHEAD>
__device__ __forceinline__ void multi_thomas_line(const MultiLine &S, int l, int NS,
                                                  const int *__restrict__ active, unsigned *status) {
    using T = double;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned amask_s;
    __shared__ int rid[MULTI_MAX];
    /* the right-hand sides' vectors, indexed by slot */
    __shared__ const T *sbp[MULTI_MAX];
    __shared__ T *syp[MULTI_MAX], *sdp[MULTI_MAX];
    const int nr = S.nr;
    const int *__restrict__ line_start = S.line_start;
    const int *__restrict__ line_len = S.line_len;
    const int *__restrict__ line_twist = S.line_twist;
    const T *__restrict__ G = S.G;
    const T *__restrict__ Gam = S.Gam;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    if (tid == 0) {
        unsigned am = 0;
        int k = 0;
#pragma unroll
        for (int r = 0; r < MULTI_MAX; ++r) {
            sbp[r] = S.b[r];
            syp[r] = S.y[r];
            sdp[r] = S.dU[r];
            if (r < nr && active[S.aid[r]]) {
                am |= 1u << r;
                rid[k++] = r;
            }
        }
        amask_s = am;
        for (int s = 0; s < NS; ++s) mbar_init(&bars[s], 1);
        mbar_fence_init();
    }
    __syncthreads();
    const unsigned amask = amask_s;
    if (amask == 0u) return;
    const int nact = __popc(amask);
    const int k0 = w * MULTI_RPW;                  /* this warp's first active slot */
    const int nown = max(0, min(MULTI_RPW, nact - k0));
    const bool mine = nown > 0;
    const uint32_t halfb = P * (NB + nr * NV) * sizeof(T);
    const uint32_t stage = 2 * halfb;
    unsigned char *st0 = smem + 128;
    T *bcw = reinterpret_cast<T *>(st0 + (size_t)NS * stage) + w * MULTI_RPW * BCAST<T, NV>;
    const int ps = line_start[l], n = line_len[l], m = line_twist[l];
    const int h = lane >> 4, li = lane & 15;
    const int i = li < NV ? li : NV - 1;
    const int nb = n - 1 - m;
    const int len = h ? nb : m;
    const int cpos = h ? m : 0;
    const int nchT = (m + P - 1) / P, nchB = (nb + P - 1) / P;
    const int nch = h ? nchB : nchT;
    const int nf = nchT > nchB ? nchT : nchB;
    const int njobs = 2 * nf;
    /* per owned right-hand side: its broadcast buffers (this half), y, dU
     * and b (slots beyond nown alias slot 0 and never write) */
    T *bc[MULTI_RPW], *yl[MULTI_RPW], *dUl[MULTI_RPW];
    const T *bg[MULTI_RPW];
    int slot[MULTI_RPW];
#pragma unroll
    for (int j = 0; j < MULTI_RPW; ++j) {
        const int jj = j < nown ? j : 0;
        slot[j] = mine ? k0 + jj : 0;
        const int rr = mine ? rid[k0 + jj] : 0;
        bc[j] = bcw + j * BCAST<T, NV> + h * 20;
        yl[j] = syp[rr] + (size_t)ps * NV;
        dUl[j] = sdp[rr] + (size_t)ps * NV;
        bg[j] = sbp[rr] + (size_t)ps * NV;
    }
    const uint64_t pol = tid == 0 ? policy_evict_first() : 0;
    for (int t = lane; t < MULTI_RPW * BCAST<T, NV>; t += 32) bcw[t] = T(0);
    __syncwarp();

    auto cells = [&](int ln, int c) { return ((min(P, ln - c * P) + 3) & ~3); };
    auto issue = [&](int job, int s) {
        unsigned char *base = st0 + (size_t)s * stage;
        uint32_t bytes = 0;
        if (job < nf) {
            if (job < nchT) bytes += cells(m, job) * (NB + nact * NV) * sizeof(T);
            if (job < nchB) bytes += cells(nb, job) * (NB + nact * NV) * sizeof(T);
        } else {
            const int jb = job - nf;
            if (nchT - 1 - jb >= 0) bytes += cells(m, nchT - 1 - jb) * NB * sizeof(T);
            if (nchB - 1 - jb >= 0) bytes += cells(nb, nchB - 1 - jb) * NB * sizeof(T);
        }
        mbar_arrive_expect_tx(&bars[s], bytes);
        for (int hh = 0; hh < 2; ++hh) {
            const int ln = hh ? nb : m, nc = hh ? nchB : nchT, cp = hh ? m : 0;
            unsigned char *hb = base + hh * halfb;
            if (job < nf) {
                const int c = job;
                if (c >= nc) continue;
                const int cnt = cells(ln, c);
                const size_t p = (size_t)(ps + cp + c * P);
                bulk_g2s_hint(hb, G + p * NB, cnt * NB * sizeof(T), &bars[s], pol);
                for (int k = 0; k < nact; ++k)
                    bulk_g2s(hb + (size_t)(P * NB + k * P * NV) * sizeof(T), sbp[rid[k]] + p * NV,
                             cnt * NV * sizeof(T), &bars[s]);
            } else {
                const int c = nc - 1 - (job - nf);
                if (c < 0) continue;
                const int cnt = cells(ln, c);
                bulk_g2s_hint(hb, Gam + (size_t)(ps + cp + c * P) * NB, cnt * NB * sizeof(T),
                              &bars[s], pol);
            }
        }
    };
    int issued = 0;
    if (tid == 0) {
        for (; issued < NS && issued < njobs; ++issued) issue(issued, issued);
    }
    int consumed = 0;
    bool timed_out = false;
    const int both_full = (m < nb ? m : nb) / P;

    /* ---------------- forward */
    for (int c = 0; c < nf; ++c) {
        const int s = c % NS;
        const bool ok = __all_sync(FULL, mbar_wait(&bars[s], (uint32_t)(c / NS) & 1u));
        if (ok && mine) {
            const T *sG = reinterpret_cast<const T *>(st0 + (size_t)s * stage + h * halfb);
            const T *sB[MULTI_RPW];
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) sB[j] = sG + P * NB + slot[j] * P * NV;
            if (c < both_full)
                fwd_chunk_m<P, false, AHEAD>(sG, sB, bc, yl, nown, c * P, len, cpos, i);
            else
                fwd_chunk_m<P, true, AHEAD>(sG, sB, bc, yl, nown, c * P, len, cpos, i);
            __syncwarp();
        }
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        ++consumed;
        if (tid == 0 && issued < njobs) {
            issue(issued, s);
            ++issued;
        }
    }

    if (!timed_out) {
        /* ---------------- twist: x_m = b_m - G_tw y_top - Gam_tw y_bot */
        const int ptw = n - 1;
        T xm[MULTI_RPW];
#pragma unroll
        for (int j = 0; j < MULTI_RPW; ++j) xm[j] = T(0);
        if (mine && lane < NV) {
            const T *gr = G + (size_t)(ps + ptw) * NB + lane;
            const T *cr = Gam + (size_t)(ps + ptw) * NB + lane;
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) {
                const T *base = bcw + j * BCAST<T, NV>;
                const T *ytop = base + (m & 1) * 10;
                const T *ybot = base + 20 + (nb & 1) * 10;
                T acc = bg[j][(size_t)ptw * NV + lane];
#pragma unroll
                for (int jj = 0; jj < NV; ++jj) acc -= fma_rn(gr[NV * jj], ytop[jj], mul_rn(cr[NV * jj], ybot[jj]));
                xm[j] = acc;
            }
        }
        __syncwarp();
        if (mine && lane < NV) {
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j) {
                if (j < nown) {
                    T *base = bcw + j * BCAST<T, NV>;
                    for (int t = 0; t < 4; ++t) base[t * 10 + lane] = xm[j];
                    dUl[j][(size_t)ptw * NV + lane] = xm[j];
                }
            }
        }
        __syncwarp();

        /* ---------------- backward */
        T yv[MULTI_RPW][P], nyv[MULTI_RPW][P];
        auto load_chunk = [&](int c, T (*yy)[P]) {
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j)
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    const int k = c * P + q;
                    yy[j][q] = T(0);
                    if (j < nown && c >= 0 && k < len) /* lanes 9..15: lane 8's values */
                        yy[j][q] = yl[j][(size_t)(cpos + k) * NV + i];
                }
        };
        load_chunk(nch - 1, yv);
        for (int jb = 0; jb < nf; ++jb) {
            const int job = nf + jb;
            const int c = nch - 1 - jb;
            load_chunk(c - 1, nyv);
            const int s = job % NS;
            const bool ok = __all_sync(FULL, mbar_wait(&bars[s], (uint32_t)(job / NS) & 1u));
            if (ok && mine) {
                const T *sG = reinterpret_cast<const T *>(st0 + (size_t)s * stage + h * halfb);
                const bool full = (nchT - 1 - jb) * P + P <= m && (nchB - 1 - jb) * P + P <= nb &&
                                  nchT - 1 - jb >= 0 && nchB - 1 - jb >= 0;
                if (full)
                    bwd_chunk_m<P, false, AHEAD>(sG, bc, yv, dUl, nown, c * P, len, cpos, i);
                else
                    bwd_chunk_m<P, true, AHEAD>(sG, bc, yv, dUl, nown, c * P, len, cpos, i);
                __syncwarp();
            }
            if (__syncthreads_or(!ok)) {
                timed_out = true;
                break;
            }
            ++consumed;
            if (tid == 0 && issued < njobs) {
                issue(issued, s);
                ++issued;
            }
#pragma unroll
            for (int j = 0; j < MULTI_RPW; ++j)
#pragma unroll
                for (int q = 0; q < P; ++q) yv[j][q] = nyv[j][q];
        }
    }
    if (timed_out && tid == 0) {
        atomicOr(status, ST_TIMEOUT);
        for (int job = consumed; job < issued; ++job)
            mbar_wait(&bars[job % NS], (uint32_t)(job / NS) & 1u, 1LL << 28);
    }
}

/* one line of one system per CTA: the context's solve (tbs_solve_multi) */
template <int P>
__global__ void __launch_bounds__(32 * MULTI_MAX / MULTI_RPW) multi_thomas_kernel(
    int nline, int NS, MultiLine S, const int *__restrict__ active, unsigned *status) {
    if ((int)blockIdx.x >= nline) return;
    multi_thomas_line<P, true>(S, blockIdx.x, NS, active, status);
}

/* the batch engine: item k = (group of one system's members, line) */
template <int P>
__global__ void __launch_bounds__(32 * MULTI_MAX / MULTI_RPW) multi_thomas_items_kernel(
    const MultiLine *__restrict__ sys, const WorkItem *__restrict__ items, const int *__restrict__ nitems,
    int NS, const int *__restrict__ active, unsigned *status) {
    if ((int)blockIdx.x >= *nitems) return;
    const WorkItem it = items[blockIdx.x];
    multi_thomas_line<P, false>(sys[it.sys], it.unit, NS, active, status);
}

static int multi_thomas_warps(int nr) { return (nr + MULTI_RPW - 1) / MULTI_RPW; }

static size_t multi_thomas_stage(int nr) {
    return 2 * (size_t)THOMAS_P * (NB + nr * NV) * sizeof(double);
}

static size_t multi_thomas_smem(int nr, int NS) {
    return 128 + (size_t)NS * multi_thomas_stage(nr) +
           (size_t)multi_thomas_warps(nr) * MULTI_RPW * BCAST<double, NV> * sizeof(double);
}

/* ring depth: the shared memory each of the SM's resident lines may use (the
 * kernel's static arrays come out of it), at least 3 and at most 8 stages */
static int multi_thomas_ns(const FastLayout &L, int nr) {
    int dev = 0, nsm = 148, smem_sm = 228 * 1024, reserved = 1024;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (nsm < 1) nsm = 148;
    int per_sm = (L.nline + nsm - 1) / nsm;
    const int by_threads = 2048 / (32 * multi_thomas_warps(nr));
    if (per_sm > by_threads) per_sm = by_threads;
    if (per_sm < 1) per_sm = 1;
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, (const void *)multi_thomas_kernel<THOMAS_P>);
    const long long budget = smem_share(smem_sm, per_sm, reserved) - (long long)fa.sharedSizeBytes;
    long long ns = (budget - (long long)multi_thomas_smem(nr, 0)) / (long long)multi_thomas_stage(nr);
    if (ns > 8) ns = 8;
    if (ns < 3) ns = 3;
    return (int)ns;
}

int launch_multi_thomas(cudaStream_t st, const FastLayout &L, int nr, const double *G,
                        const double *Gam, const double *b, double *y, double *dU,
                        const int *active, unsigned *status) {
    if (L.nv != NV || nr < 1 || nr > MULTI_MAX) return (int)cudaErrorInvalidValue;
    const int NS = multi_thomas_ns(L, nr);
    const long long vs = (long long)L.np16 * NV;
    MultiLine S{};
    S.line_start = L.line_start;
    S.line_len = L.line_len;
    S.line_twist = L.line_twist;
    S.G = G;
    S.Gam = Gam;
    S.nr = nr;
    for (int r = 0; r < MULTI_MAX; ++r) {
        const int rr = r < nr ? r : 0;
        S.aid[r] = rr;
        S.b[r] = b + (size_t)rr * vs;
        S.y[r] = y + (size_t)rr * vs;
        S.dU[r] = dU + (size_t)rr * vs;
    }
    multi_thomas_kernel<THOMAS_P><<<L.nline, 32 * multi_thomas_warps(nr), multi_thomas_smem(nr, NS), st>>>(
        L.nline, NS, S, active, status);
    return (int)cudaGetLastError();
}

/* ring depth of the engine's multi-RHS line solves (their shared memory
 * is sized for MULTI_MAX right-hand sides) */
constexpr int MULTI_ITEMS_NS = 3;

int multi_items_prepare() {
    return set_smem((const void *)multi_thomas_items_kernel<THOMAS_P>,
                    multi_thomas_smem(MULTI_MAX, MULTI_ITEMS_NS));
}

int launch_multi_thomas_items(cudaStream_t st, int grid, const MultiLine *sys, const WorkItem *items,
                              const int *nitems, const int *active, unsigned *status) {
    if (grid < 1) return 0;
    multi_thomas_items_kernel<THOMAS_P>
        <<<grid, 32 * multi_thomas_warps(MULTI_MAX), multi_thomas_smem(MULTI_MAX, MULTI_ITEMS_NS), st>>>(
            sys, items, nitems, MULTI_ITEMS_NS, active, status);
    return (int)cudaGetLastError();
}

/* Residual of several right-hand sides per tile: Dinv and the cross-line
 * blocks are staged once, then for every active right-hand side r
 *   mode 0 (the start):  R = Rsrc_r (staged), U_r = 0
 *   mode 1 (a sweep):    R = sum X dU_r, U_r += dU_r
 * followed by b_r = -Dinv R and the tile's sum R^2 for r, each with the
 * expressions (and summation order) of fast_resid_body.  The last CTA to
 * finish adds every active r's partials in tile order (finalize_total's
 * order), records the norms, retires the right-hand sides whose solve has
 * ended and keeps the graph's loop running while any is active.
 *
 * HBM would take 90 us for 8 right-hand sides at 360x384; shared memory is
 * what bounds it.  A thread per (cell, row) that loads a block's row once and
 * each right-hand side's vector for itself reads ten words for nine products
 * and took 214 us at three quarters of the L1's throughput.  Here a thread has
 * three rows (i0, i0 + 3, i0 + 6) of a cell for three right-hand sides, six
 * words for nine products, without a branch for each; a cell's vectors arrive
 * by asynchronous copies of adjacent words, the sums of squares of eight
 * right-hand sides go down the lanes together (nine exchanges for forty), and
 * R takes the place of the blocks it was made of, so that four CTAs fit an
 * SM: 150 us. */
constexpr int MULTI_KG = 3;                                    /* right-hand sides of a thread */
static_assert(3 * MULTI_KG >= MULTI_MAX && RES_TILE * 9 <= RES_THREADS_FAST, "three groups of threads");

static size_t multi_resid_smem(int nx, int nr) {
    const int nxa = nx > 0 ? nx : 1;
    const size_t vec = (size_t)nr * RES_TILE * NV, blk = (size_t)RES_TILE * NB;
    return 128 + (blk + std::max(nx * blk, vec) + nxa * vec) * sizeof(double);
}

/* rows i0, i0 + 3, i0 + 6 of a block times the vectors at v0 + off[k], in
 * fast_resid_body's order */
struct MultiAcc {
    double a[MULTI_KG][3][3];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < MULTI_KG; ++k)
#pragma unroll
            for (int q = 0; q < 3; ++q) a[k][q][0] = a[k][q][1] = a[k][q][2] = 0.0;
    }
    __device__ __forceinline__ void add(const double *row, const double *v0, const int (&off)[MULTI_KG]) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const double x0 = row[9 * j], x1 = row[9 * j + 3], x2 = row[9 * j + 6];
#pragma unroll
            for (int k = 0; k < MULTI_KG; ++k) {
                const double v = v0[off[k] + j];
                a[k][0][j % 3] += x0 * v;
                a[k][1][j % 3] += x1 * v;
                a[k][2][j % 3] += x2 * v;
            }
        }
    }
    /* the same in neg_dinv_row's order */
    __device__ __forceinline__ void set(const double *row, const double *v0, const int (&off)[MULTI_KG]) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            double x[3][3];
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int q = 0; q < 3; ++q) x[m][q] = row[9 * (j + 3 * m) + 3 * q];
#pragma unroll
            for (int k = 0; k < MULTI_KG; ++k) {
                const double *v = v0 + off[k] + j;
                const double u0 = v[0], u1 = v[3], u2 = v[6];
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    a[k][q][j] = fma_rn(x[2][q], u2, fma_rn(x[0][q], u0, mul_rn(x[1][q], u1)));
            }
        }
    }
    __device__ __forceinline__ double sum(int k, int q) const { return a[k][q][0] + (a[k][q][1] + a[k][q][2]); }
};

/* the warp's sums of v[0..8) (SQ: squared), each with the pairs of a shfl_down
 * tree; lane 4 k has that of v[k] */
template <bool SQ>
__device__ __forceinline__ double warp_sums8(const double (&v)[8]) {
    const int lane = threadIdx.x & 31;
    double w[4], x[2], y;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double keep = lane & 16 ? v[k + 4] : v[k], give = lane & 16 ? v[k] : v[k + 4];
        const double got = __shfl_xor_sync(FULL, give, 16);
        w[k] = SQ ? mul_rn(keep, keep) + mul_rn(got, got) : keep + got;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double keep = lane & 8 ? w[k + 2] : w[k], give = lane & 8 ? w[k] : w[k + 2];
        x[k] = keep + __shfl_xor_sync(FULL, give, 8);
    }
    {
        const double keep = lane & 4 ? x[1] : x[0], give = lane & 4 ? x[0] : x[1];
        y = keep + __shfl_xor_sync(FULL, give, 4);
    }
    y += __shfl_xor_sync(FULL, y, 2);
    y += __shfl_xor_sync(FULL, y, 1);
    return y;
}

template <int MODE>
__global__ void __launch_bounds__(RES_THREADS_FAST, 4) multi_resid_kernel(
    MultiSys M, const double *__restrict__ Dinv, const double *__restrict__ X,
    const int *__restrict__ xnbr, const double *__restrict__ Rsrc, unsigned long long handle,
    int use_cond, unsigned *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned amask_s, ticket;
    __shared__ double red[MULTI_MAX][RES_THREADS_FAST / 32];
    const int tid = threadIdx.x;
    const int nx = MODE == 1 ? M.nx : 0;
    const int nxa = nx > 0 ? nx : 1;
    const int nr = M.nr;
    const long long vs = (long long)M.np16 * NV;
    const int ntiles = M.np16 / RES_TILE;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    double *sD = reinterpret_cast<double *>(smem + 128);
    double *sg = sD + RES_TILE * NB; /* [k][s][c][i] gathers, then b; mode 0: R */
    double *sX = sg + (size_t)nr * nxa * RES_TILE * NV;
    double *sr = sX; /* [k][c][i] R, in the place of the blocks it was made of; mode 0: b */
    __shared__ int rid[MULTI_MAX]; /* the k-th active right-hand side */
    if (tid == 0) {
        unsigned am = 0;
        int k = 0;
        for (int r = 0; r < nr; ++r)
            if (MODE == 0 || M.active[r]) {
                am |= 1u << r;
                rid[k++] = r;
            }
        amask_s = am;
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    const unsigned amask = amask_s;
    const int nact = __popc(amask);
    const bool act = tid < RES_TILE * NV;
    /* products: a cell, three of its rows, a group of right-hand sides */
    const int c = tid % RES_TILE, i0 = (tid / RES_TILE) % 3;
    const int k0 = tid / RES_TILE / 3 * MULTI_KG;
    const int ng = act ? max(0, min(MULTI_KG, nact - k0)) : 0;
    /* (a group that is not full repeats its last one and does not store it) */
    int offg[MULTI_KG], offr[MULTI_KG];
#pragma unroll
    for (int k = 0; k < MULTI_KG; ++k) {
        const int kk = max(0, min(k0 + k, nact - 1));
        offg[k] = kk * nx * RES_TILE * NV;
        offr[k] = kk * RES_TILE * NV;
    }
    /* loads: a word of a cell's vectors; the norm: (cell, row) as
     * fast_resid_body deals them */
    const int lc = tid / NV, li = tid % NV;
    const int nat = c * NV + tid / RES_TILE;
    const uint32_t szD = RES_TILE * NB * sizeof(double), szR = RES_TILE * NV * sizeof(double);
    uint32_t parity = 0;
    bool failed = false;
    /* the neighbour indices of the CTA's next tile load during the current one */
    int pnbr[MULTI_NX];
#pragma unroll
    for (int s = 0; s < MULTI_NX; ++s)
        pnbr[s] = (MODE == 1 && act && s < nx && (int)blockIdx.x < ntiles)
                      ? __ldg(xnbr + (size_t)s * M.np16 + blockIdx.x * RES_TILE + lc) : -1;
    for (int blk = blockIdx.x; blk < ntiles && nact > 0; blk += gridDim.x) {
        const int p0 = blk * RES_TILE;
        const int bn = blk + gridDim.x;
        if (tid == 0) {
            const uint64_t pol = policy_evict_first();
            mbar_arrive_expect_tx(bar, szD + (MODE == 1 ? nx * szD : nact * szR));
            bulk_g2s_hint(sD, Dinv + (size_t)p0 * NB, szD, bar, pol);
            if (MODE == 1) {
                for (int s = 0; s < nx; ++s)
                    bulk_g2s_hint(sX + s * RES_TILE * NB, X + ((size_t)s * M.np16 + p0) * NB, szD,
                                  bar, pol);
            } else {
                int k = 0;
                for (int r = 0; r < nr; ++r) {
                    if (!((amask >> r) & 1u)) continue;
                    bulk_g2s(sg + (size_t)k * RES_TILE * NV, Rsrc + (size_t)r * vs + (size_t)p0 * NV,
                             szR, bar);
                    ++k;
                }
            }
        }
        if (act) {
            const size_t q = (size_t)p0 * NV + tid;
            if (MODE == 1) {
                for (int k = 0; k < nact; ++k) {
                    const double *d = M.dU + (size_t)rid[k] * vs + li;
#pragma unroll
                    for (int s = 0; s < MULTI_NX; ++s)
                        if (s < nx) {
                            double *to = sg + (size_t)(k * nx + s) * RES_TILE * NV + tid;
                            if (pnbr[s] >= 0) cp_async8(to, d + (size_t)pnbr[s] * NV);
                            else *to = 0.0;
                        }
                }
                cp_async_commit();
                /* every load is issued before the first store */
                double uv[MULTI_MAX], dv[MULTI_MAX];
#pragma unroll
                for (int k = 0; k < MULTI_MAX; ++k) {
                    uv[k] = dv[k] = 0.0;
                    if (k < nact) {
                        const size_t ro = (size_t)rid[k] * vs;
                        uv[k] = M.U[ro + q];
                        dv[k] = __ldg(M.dU + ro + q);
                    }
                }
#pragma unroll
                for (int s = 0; s < MULTI_NX; ++s)
                    pnbr[s] = (s < nx && bn < ntiles)
                                  ? __ldg(xnbr + (size_t)s * M.np16 + bn * RES_TILE + lc) : -1;
#pragma unroll
                for (int k = 0; k < MULTI_MAX; ++k)
                    if (k < nact) M.U[(size_t)rid[k] * vs + q] = uv[k] + dv[k];
                cp_async_wait<0>();
            } else {
                for (int k = 0; k < nact; ++k) M.U[(size_t)rid[k] * vs + q] = 0.0;
            }
        }
        const bool ok = mbar_wait(bar, parity);
        parity ^= 1u;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(status, ST_TIMEOUT);
                mbar_wait(bar, parity ^ 1u, 1LL << 28);
            }
            failed = true;
            break;
        }
        MultiAcc acc;
        if (MODE == 1) {
            acc.clear();
            if (ng > 0)
                for (int s = 0; s < nx; ++s)
                    acc.add(sX + (s * RES_TILE + c) * NB + i0, sg + (s * RES_TILE + c) * NV, offg);
            __syncthreads(); /* the blocks are read */
#pragma unroll
            for (int k = 0; k < MULTI_KG; ++k)
                if (k < ng) {
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        sr[(size_t)(k0 + k) * RES_TILE * NV + c * NV + i0 + 3 * q] = acc.sum(k, q);
                }
            __syncthreads();
        }
        /* b = -Dinv R for every active r (into sg, free now), and R^2 */
        const double *rsrc = MODE == 1 ? sr : sg;
        double *sb = MODE == 1 ? sg : sr;
        if (ng > 0) acc.set(sD + c * NB + i0, rsrc + c * NV, offr);
#pragma unroll
        for (int k = 0; k < MULTI_KG; ++k)
            if (k < ng) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    sb[(size_t)(k0 + k) * RES_TILE * NV + c * NV + i0 + 3 * q] = -acc.sum(k, q);
            }
        /* the tile's sum R^2 per r, in fast_resid_body's order */
        double rr[MULTI_MAX];
#pragma unroll
        for (int k = 0; k < MULTI_MAX; ++k)
            rr[k] = act && k < nact ? rsrc[(size_t)k * RES_TILE * NV + nat] : 0.0;
        const double ws = warp_sums8<true>(rr);
        if ((tid & 3) == 0) red[(tid & 31) >> 2][tid >> 5] = ws;
        __syncthreads();
        if (act)
            for (int k = 0; k < nact; ++k)
                M.b[(size_t)rid[k] * vs + (size_t)p0 * NV + tid] = sb[(size_t)k * RES_TILE * NV + tid];
        if (tid < nact) {
            double tot = 0.0;
            for (int w = 0; w < RES_THREADS_FAST / 32; ++w) tot += red[tid][w];
            M.partials[(size_t)rid[tid] * ntiles + blk] = tot;
        }
        if (MODE == 1) fence_async_smem(); /* R was stored where blocks are copied to */
        __syncthreads(); /* the next tile's copies overwrite the stages */
    }
    (void)failed;

    /* ---------------- the last CTA: norms of every active r */
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        ticket = atomicAdd(M.counter, 1u);
    }
    __syncthreads();
    if (ticket != gridDim.x - 1) return;
    __threadfence();
    /* per r the order of strided_sum, all r side by side: one r after the other
     * (each waits for its loads twelve times at 8640 tiles) a launch took 12 to
     * 27 us longer */
    double acc[MULTI_MAX];
#pragma unroll
    for (int r = 0; r < MULTI_MAX; ++r) acc[r] = 0.0;
    {
        constexpr int AHEAD = 3;
        const double *p = M.partials + tid;
        int t = tid;
        for (; t + (AHEAD - 1) * RES_THREADS_FAST < ntiles; t += AHEAD * RES_THREADS_FAST, p += AHEAD * RES_THREADS_FAST) {
            double v[AHEAD][MULTI_MAX];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
                for (int r = 0; r < MULTI_MAX; ++r)
                    v[u][r] = r < nr ? __ldcg(p + (size_t)r * ntiles + u * RES_THREADS_FAST) : 0.0;
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
                for (int r = 0; r < MULTI_MAX; ++r) acc[r] += v[u][r];
        }
        for (; t < ntiles; t += RES_THREADS_FAST, p += RES_THREADS_FAST) {
#pragma unroll
            for (int r = 0; r < MULTI_MAX; ++r)
                if (r < nr) acc[r] += __ldcg(p + (size_t)r * ntiles);
        }
    }
    const double ws = warp_sums8<false>(acc);
    if ((tid & 3) == 0) red[(tid & 31) >> 2][tid >> 5] = ws;
    __syncthreads();
    bool go = false;
    if (tid < nr && ((amask >> tid) & 1u)) {
        double tot = 0.0;
        for (int w = 0; w < RES_THREADS_FAST / 32; ++w) tot += red[tid][w];
        const double nrm = sqrt(tot);
        SolveState *S = M.state + tid;
        if (MODE == 0) {
            S->sweep = 0;
            S->norm0 = nrm;
        } else {
            S->sweep += 1;
        }
        const int sw = S->sweep;
        if (sw < S->hist_cap) M.hist[(size_t)tid * M.hist_stride + sw] = nrm;
        S->last = nrm;
        go = isfinite(nrm) && nrm > S->tol * S->norm0 && sw < S->max_sweeps;
        M.active[tid] = go ? 1 : 0;
    }
    const int any_go = __syncthreads_or(go);
    if (tid == 0) {
        if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)handle, any_go ? 1u : 0u);
        *M.counter = 0u;
    }
}

int launch_multi_resid(cudaStream_t st, const FastLayout &L, int mode, const MultiSys &M,
                       const double *Dinv, const double *X, const double *Rsrc,
                       unsigned long long cond_handle, int use_cond, unsigned *status) {
    if (L.nv != NV || M.nr < 1 || M.nr > MULTI_MAX || (mode != 0 && mode != 1))
        return (int)cudaErrorInvalidValue;
    const int ntiles = L.np16 / RES_TILE;
    if (mode == 1) {
        const size_t smem = multi_resid_smem(L.nx, M.nr);
        multi_resid_kernel<1><<<resid_grid_persistent((const void *)multi_resid_kernel<1>, smem, ntiles),
                                RES_THREADS_FAST, smem, st>>>(M, Dinv, X, L.xnbr, nullptr,
                                                              cond_handle, use_cond, status);
    } else {
        const size_t smem = multi_resid_smem(0, M.nr);
        multi_resid_kernel<0><<<resid_grid_persistent((const void *)multi_resid_kernel<0>, smem, ntiles),
                                RES_THREADS_FAST, smem, st>>>(M, Dinv, nullptr, nullptr, Rsrc,
                                                              cond_handle, use_cond, status);
    }
    return (int)cudaGetLastError();
}

/* opt the multi-RHS kernels into the shared memory of nr right-hand sides
 * (outside stream capture) */
int multi_prepare(const FastLayout &L, int nr) {
    if (nr < 1 || nr > MULTI_MAX) return (int)cudaErrorInvalidValue;
    int rc = set_smem((const void *)multi_thomas_kernel<THOMAS_P>,
                      multi_thomas_smem(nr, multi_thomas_ns(L, nr)));
    if (!rc) rc = set_smem((const void *)multi_resid_kernel<1>, multi_resid_smem(L.nx, nr));
    if (!rc) rc = set_smem((const void *)multi_resid_kernel<0>, multi_resid_smem(0, nr));
    return rc;
}


/* ================================================ point-implicit Jacobi
 * TBS_ALGO_PIJ: the sweep dU = -D^-1 R, U += dU, R = rhs + J U with the
 * diagonal block alone as the implicit operator (every cell its own
 * line).  As for the line form, D dU = -R makes the new residual
 * R + J dU = sum over the interior faces of offJ dU_nbr, so one sweep is
 * one streaming launch of the residual kernel over the position-ordered
 * face blocks (slot s = the s-th interior face of the cell in ef order):
 *     U += dU;  R = sum_s XF_s dU_nbr(s);  b = -Dinv R  (= the next dU)
 * with dU and b in two buffers that swap every sweep.  The buffer parity
 * lives in SolveState::pad, flipped by the launch's last CTA, so graph and
 * eager sweep sequences agree on where the latest update is. */

/* Dinv = D^-1 per position, in place (Gauss-Jordan without pivoting, as
 * the reference's LU has none); pads stay zero.  One warp per position. */
__global__ void __launch_bounds__(32) pij_invert_kernel(int np16, const int *__restrict__ elem_of_pos,
                                                        double *__restrict__ D, unsigned *status) {
    const int j = threadIdx.x;
    for (int p = blockIdx.x; p < np16; p += gridDim.x) {
        if (elem_of_pos[p] < 0) continue;
        double w[NV];
        double *blk = D + (size_t)p * NB;
#pragma unroll
        for (int i = 0; i < NV; ++i) w[i] = j < NV ? blk[NV * j + i] : (i == j ? 1.0 : 0.0);
        gj_invert_cols(w, j, status);
        if (j < NV) {
#pragma unroll
            for (int i = 0; i < NV; ++i) blk[NV * j + i] = w[i];
        }
        __syncwarp();
    }
}

int launch_pij_invert(cudaStream_t st, const FastLayout &L, double *D, unsigned *status) {
    const int grid = L.np16 < 148 * 32 ? (L.np16 > 0 ? L.np16 : 1) : 148 * 32;
    pij_invert_kernel<<<grid, 32, 0, st>>>(L.np16, L.elem_of_pos, D, status);
    return (int)cudaGetLastError();
}

__global__ void __launch_bounds__(RES_THREADS_FAST) pij_sweep_kernel(
    int nxf, int np16, const double *__restrict__ Dinv, const double *__restrict__ XF,
    const int *__restrict__ xnbrf, double *bufA, double *bufB, double *__restrict__ Up,
    NormSink ns, unsigned *status) {
    /* read before any CTA can finish: the last CTA flips it after every
     * CTA has taken its ticket */
    const int odd = ns.state->pad & 1;
    const double *dU = odd ? bufB : bufA;
    double *b = odd ? bufA : bufB;
    const bool last = resid_tiles<double>(nxf, np16, 1, Dinv, XF, xnbrf, dU, nullptr, b, Up, ns, status);
    if (last && threadIdx.x == 0) ns.state->pad = odd ^ 1;
}

int launch_pij_sweep(cudaStream_t st, const FastLayout &L, const double *Dinv, const double *XF,
                     double *bufA, double *bufB, double *Up, const NormSink &ns, unsigned *status) {
    /* nxf == 0 (no interior faces): no slot is read and R_new = 0 */
    if (L.nv != NV || L.nxf > 4 || !ns.state || !ns.partials) return (int)cudaErrorInvalidValue;
    const size_t smem = resid_smem_bytes<double>(L.nxf);
    pij_sweep_kernel<<<resid_grid_persistent((const void *)pij_sweep_kernel, smem, L.np16 / RES_TILE),
                       RES_THREADS_FAST, smem, st>>>(L.nxf, L.np16, Dinv, XF, L.xnbrf, bufA, bufB, Up,
                                                     ns, status);
    return (int)cudaGetLastError();
}

int pij_prepare(const FastLayout &L) {
    return set_smem((const void *)pij_sweep_kernel, resid_smem_bytes<double>(L.nxf));
}


/* =============================================== bounded-wait self-test
 * One thread arms an mbarrier for 16 bytes that no copy will deliver (no
 * copy is issued) and waits on it with the given clock budget, the wait
 * every staging pipeline uses: it must give up, and the status bit it then
 * records is the one the kernels record on a stalled copy. */
__global__ void selftest_timeout_kernel(long long budget, unsigned *status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    mbar_fence_init();
    mbar_arrive_expect_tx(&bar, 16);
    if (!mbar_wait(&bar, 0, budget)) atomicOr(status, ST_TIMEOUT);
}

int launch_selftest_timeout(cudaStream_t st, long long budget_cycles, unsigned *status) {
    if (budget_cycles < 0) return (int)cudaErrorInvalidValue;
    selftest_timeout_kernel<<<1, 32, 0, st>>>(budget_cycles, status);
    return (int)cudaGetLastError();
}

}  // namespace tbs
