/*
 * kernels_ref.cu -- TBS_ALGO_REFERENCE: the reference's arithmetic, in its
 * operation order, on the GPU.  Built with -fmad=false so that every
 * multiply and add rounds separately, exactly like the CPU oracle built with
 * -ffp-contract=off; U, dU and R then agree bit for bit.
 *
 *   ref_line_lu      src/okl/lineLU_v2.okl:58-182 (LU 17-27, solveLU 30-52)
 *   ref_assemble_A   src/Jacobian.cxx:76-117 (done on the device here)
 *   ref_solve_du     src/okl/linesmoothLU_TriBlock_v3.okl:92-226
 *   ref_add_copy     src/okl/linesmoothLU_v5.okl:75-103 (addAtoB + copyAtoB)
 *   ref_line_res     src/okl/linesmoothLU_TriBlock_v3.okl:228-336
 *
 * Parallel decomposition differs from the reference (one warp per line,
 * rows spread over lanes; one thread per (element,row) for the residual)
 * but each scalar is produced by the same sequence of roundings: rows of
 * the Doolittle update are independent once the pivot row is final, the
 * nv columns of D'^-1 C are independent solves, and every dot product is
 * summed from 0.0 in ascending j as in the OKL loops.
 */
#include "recip.cuh"
#include "tbs_internal.hxx"
#include "tma.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace tbs {

constexpr int REF_MAXNV = 32;

#define MIDX(i, j, nv) ((i) + (nv) * (j))

/* x = (LU)^-1 b for one lane; A in shared memory, column-major.
 * lineLU_v2.okl:30-52 / linesmoothLU_TriBlock_v3.okl:23-45 */
template <int NV>
__device__ __forceinline__ void solve_lu_lane(const double *A, const double *b, double *x,
                                              int nv_rt) {
    const int nv = NV ? NV : nv_rt;
    double y[NV ? NV : REF_MAXNV];
#pragma unroll
    for (int i = 0; i < nv; ++i) {
        double tot = 0.0;
#pragma unroll
        for (int j = 0; j < i; ++j) tot += A[MIDX(i, j, nv)] * y[j];
        y[i] = b[i] - tot;
    }
#pragma unroll
    for (int i = nv - 1; i >= 0; --i) {
        double tot = 0.0;
#pragma unroll
        for (int j = i + 1; j < nv; ++j) tot += A[MIDX(i, j, nv)] * x[j];
        x[i] = (y[i] - tot) / A[MIDX(i, i, nv)];
    }
}

/* In-place no-pivot Doolittle on a shared-memory block, rows over lanes.
 * Row j is final when step j starts and only rows i > j change in it, so
 * lane i applying its own row's updates reproduces lineLU_v2.okl:17-27. */
template <int NV>
__device__ __forceinline__ void lu_rows(double *A, int lane, int nv_rt, unsigned *status) {
    const int nv = NV ? NV : nv_rt;
    for (int j = 0; j < nv; ++j) {
        __syncwarp();
        const double ajj = A[MIDX(j, j, nv)];
        if (lane == 0 && !(fabs(ajj) > 0.0 && isfinite(ajj))) atomicOr(status, ST_PIVOT);
        const double pivot = 1.0 / ajj;
        if (lane > j && lane < nv) {
            const double lij = A[MIDX(lane, j, nv)] * pivot;
            A[MIDX(lane, j, nv)] = lij;
            for (int k = j + 1; k < nv; ++k) A[MIDX(lane, k, nv)] -= lij * A[MIDX(j, k, nv)];
        }
    }
    __syncwarp();
}

template <int NV>
__global__ void __launch_bounds__(32) ref_line_lu_kernel(
    int nv_rt, int nline, const int *__restrict__ fc, const int *__restrict__ linesize,
    const int *__restrict__ linepoint, const int *__restrict__ lines,
    const int *__restrict__ lineface, double *__restrict__ Dia, const double *__restrict__ O1,
    const double *__restrict__ O2, double *__restrict__ DinvC, unsigned *status) {
    const int nv = NV ? NV : nv_rt;
    const int l = blockIdx.x;
    if (l >= nline) return;
    const int lane = threadIdx.x;
    const size_t bs = (size_t)nv * nv;
    extern __shared__ double sm[];
    double *sGamma = sm;
    double *sC = sGamma + bs;
    double *sAT = sC + bs;
    double *sDe = sAT + bs;
    double *sDl = sDe + bs;

    const int n = linesize[l];
    const int m0 = linepoint[l];
    int e = lines[m0];
    if (lane < nv)
        for (int j = 0; j < nv; ++j) sDe[MIDX(lane, j, nv)] = Dia[MIDX(lane, j, nv) + bs * e];
    lu_rows<NV>(sDe, lane, nv, status);
    if (lane < nv)
        for (int j = 0; j < nv; ++j) Dia[MIDX(lane, j, nv) + bs * e] = sDe[MIDX(lane, j, nv)];

    for (int k = 1; k < n; ++k) {
        const int m = m0 + k;
        const int elast = e;
        e = lines[m];
        const int f = lineface[m];
        const int e1 = fc[2 * f];
        const double *A = (e == e1) ? O2 : O1;
        const double *C = (e == e1) ? O1 : O2;
        __syncwarp();
        if (lane < nv) {
            for (int j = 0; j < nv; ++j) {
                /* D'_{k-1} is the block factored in the previous step; the
                 * reference re-reads it from global memory, same bits */
                sDl[MIDX(lane, j, nv)] = sDe[MIDX(lane, j, nv)];
            }
        }
        __syncwarp();
        if (lane < nv) {
            for (int j = 0; j < nv; ++j) {
                sC[MIDX(lane, j, nv)] = C[MIDX(lane, j, nv) + bs * f];
                sAT[MIDX(j, lane, nv)] = A[MIDX(lane, j, nv) + bs * f];
                sDe[MIDX(lane, j, nv)] = Dia[MIDX(lane, j, nv) + bs * e];
            }
        }
        __syncwarp();
        /* Gamma(:,i) = D'_{k-1}^-1 C(:,i)  (lineLU_v2.okl:142-144) */
        if (lane < nv) solve_lu_lane<NV>(sDl, &sC[MIDX(0, lane, nv)], &sGamma[MIDX(0, lane, nv)], nv);
        __syncwarp();
        /* D_k - A_k Gamma  (lineLU_v2.okl:147-161) */
        if (lane < nv) {
            for (int kk = 0; kk < nv; ++kk) {
                double tot = 0.0;
                for (int j = 0; j < nv; ++j) tot += sAT[MIDX(j, lane, nv)] * sGamma[MIDX(j, kk, nv)];
                sDe[MIDX(lane, kk, nv)] -= tot;
            }
        }
        lu_rows<NV>(sDe, lane, nv, status);
        if (lane < nv) {
            for (int j = 0; j < nv; ++j) {
                Dia[MIDX(lane, j, nv) + bs * e] = sDe[MIDX(lane, j, nv)];
                DinvC[MIDX(lane, j, nv) + bs * elast] = sGamma[MIDX(lane, j, nv)];
            }
        }
    }
}

/* ------------------------------------------------- block size 9, quickly
 * The same scalars, each by the same sequence of roundings, with the chain
 * kept short: solveLU's divisions by a diagonal whose reciprocal is known
 * beforehand, every lane of a warp computing the whole vector (no exchange
 * inside a triangular solve), a second warp copying the coming cells' blocks
 * into shared memory. */

/* a divisor left to the general division (rcp_newton, ref_div) */
__device__ __forceinline__ bool ref_plain_divisor(double d) {
    return (int)!within_pow2(d, 500) | (int)ones_significand(d);
}

/* RN(n / d) from r = RN(1 / d) and rl, the rest of 1 / d to twice the
 * precision: q is within an ulp, the remainder exact and the last step
 * rounds correctly (Markstein, as for rcp_newton).  Holds for |d| within 2^-500 ..
 * 2^500 and |n| within 2^-400 .. 2^400; the caller checks both. */
__device__ __forceinline__ double ref_div(double n, double d, double r, double rl) {
    const double q = fma(n, r, n * rl);
    return fma(fma(-q, d, n), r, q);
}

constexpr int RC = 4;                        /* cells of one copy job */
constexpr int RS = 3;                        /* jobs in shared memory */
constexpr int RCELL = 81 + 81 + 9 + 9 + 9 + 1; /* D', A, R, 1/U_ii (r, rl), flag */

/* x = (LU)^-1 s, all of it in every lane; D: the block in shared memory
 * (column-major), rc: r and rl of its diagonal.  The sums start from 0.0 and
 * take j in ascending order, as solveLU's: forward by columns (each row's
 * terms still come in order), backward by rows, from products formed as the
 * x_j come.  A first term is rounded once by fma(a, b, 0.0) (0.0 + a*b).
 * plain: the diagonal or a numerator may be out of ref_div's range (decided by
 * the caller), so divide. */
__device__ __forceinline__ bool ref_solve9(const double *D, const double *rc, const double (&s)[9],
                                           double (&x)[9]) {
    double tot[9], y[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        y[j] = j == 0 ? s[0] - 0.0 : s[j] - tot[j];
#pragma unroll
        for (int i = j + 1; i < 9; ++i)
            tot[i] = j == 0 ? fma(D[i], y[0], 0.0) : tot[i] + D[i + 9 * j] * y[j];
    }
    double p[9][9];
    bool ok = true;
#pragma unroll
    for (int i = 8; i >= 0; --i) {
        double t = 0.0;
#pragma unroll
        for (int j = i + 1; j < 9; ++j) t = j == i + 1 ? p[i][j] : t + p[i][j];
        const double n = y[i] - t;
        ok = ok && within_pow2(n, 400);
        x[i] = ref_div(n, D[10 * i], rc[i], rc[9 + i]);
#pragma unroll
        for (int k = 0; k < i; ++k) p[k][i] = k + 1 == i ? fma(D[k + 9 * i], x[i], 0.0) : D[k + 9 * i] * x[i];
    }
    return ok;
}

/* In-place no-pivot Doolittle (lineLU_v2.okl:17-27) of a block held by 27
 * lanes, lane i + 9g row i, columns 3g..3g+2.  Step j: l_ij = a_ij * (1/a_jj),
 * a_ik -= l_ij a_jk, each operation rounded by itself; every lane forms the
 * next pivot from three entries fetched while this one's reciprocal is on its
 * way.  rc[0..8], rc[9..17]: r and rl of the diagonal (ref_div), rc[18]: not 0
 * when a pivot is not for ref_div (and, unless PLAIN, the result not valid).
 * Returns whether a pivot was zero or not finite (PLAIN) or has to be done by
 * the general division. */
template <bool PLAIN>
__device__ __forceinline__ bool ref_lu27(double (&w)[3], int i, int g, bool first, double *rc) {
    bool odd = false, bad = false;
    double a = __shfl_sync(0xffffffffu, w[0], 0);
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        const int jg = j / 3, jk = j % 3, n = j < 8 ? j + 1 : j, ng = n / 3, nk = n % 3;
        const double dn = __shfl_sync(0xffffffffu, w[nk], n + 9 * ng);
        const double cn = __shfl_sync(0xffffffffu, w[jk], n + 9 * jg);
        const double rn = __shfl_sync(0xffffffffu, w[nk], j + 9 * ng);
        double l = __shfl_sync(0xffffffffu, w[jk], i + 9 * jg);
        double u[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = __shfl_sync(0xffffffffu, w[k], j + 9 * g);
        if (PLAIN) bad |= !(fabs(a) > 0.0 && isfinite(a));
        odd |= ref_plain_divisor(a);
        const double r = PLAIN ? 1.0 / a : rcp_newton(a);
        if (first && i == j) {
            rc[j] = r;
            rc[9 + j] = fma(-a, r, 1.0) * r;
        }
        l = l * r;
        a = dn - (cn * r) * rn;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int c = 3 * g + k;
            const double v = w[k] - l * u[k];
            if (i > j) w[k] = c > j ? v : (c == j ? l : w[k]);
        }
    }
    if (first && i == 0) rc[18] = odd ? 1.0 : 0.0;
    return PLAIN ? bad : odd;
}

__device__ __noinline__ bool ref_lu27_plain(double *v, int i, int g, bool first, double *rc) {
    double w[3] = {v[0], v[1], v[2]};
    const bool bad = ref_lu27<true>(w, i, g, first, rc);
    v[0] = w[0];
    v[1] = w[1];
    v[2] = w[2];
    return bad;
}

constexpr int LS = 4;                /* cells in shared memory */
constexpr int LCELL = 3 * 81;        /* D, A, C */

/* ref_line_lu_kernel for block size 9, and the packing of the lower blocks
 * (ref_assemble_A_kernel): one CTA of two warps per line, warp 0 on the chain
 * (Gamma: a column per lane; D - A Gamma and the LU: 27 lanes), warp 1 copying
 * the cells two steps ahead into shared memory and writing D', D'^-1 C and A
 * out.  ref_line_lu_kernel, which loads as it goes and divides 18 times a
 * cell, took 9,900 cycles a cell; 360x384: 1,960 us and 95 for the packing,
 * 657 together here. */
__global__ void __launch_bounds__(64) ref_line_lu9_kernel(
    int nline, const int *__restrict__ fc, const int *__restrict__ linesize,
    const int *__restrict__ linepoint, const int *__restrict__ lines,
    const int *__restrict__ lineface, double *Dia, const double *__restrict__ O1,
    const double *__restrict__ O2, double *__restrict__ DinvC, double *__restrict__ Aout,
    unsigned *status) {
    __shared__ __align__(16) double stage[LS][LCELL];
    __shared__ __align__(16) double sL[2][81], sG[2][81], rc[19];
    const int l = blockIdx.x;
    if (l >= nline) return;
    const int lane = threadIdx.x & 31;
    const int n = linesize[l], m0 = linepoint[l];
    if (threadIdx.x >= 32) {
        auto elem = [&](int c) { return c >= 0 && c < n ? lines[m0 + c] : 0; };
        auto face = [&](int c) { return c >= 1 && c < n ? lineface[m0 + c] : 0; };
        auto first = [&](int c, int f) { return c >= 1 && c < n ? fc[2 * f] : 0; };
        /* copies of cell c (element e, face f, whose first element is e1) */
        auto copy = [&](int c, int e, int f, int e1) {
            if (c < n) {
                const double *pD = Dia + 81 * (size_t)e;
                const double *pA = (e == e1 ? O2 : O1) + 81 * (size_t)f;
                const double *pC = (e == e1 ? O1 : O2) + 81 * (size_t)f;
                double *d = stage[c % LS];
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const int t = lane + 32 * r;
                    if (t < 81) {
                        cp_async8(d + t, pD + t);
                        if (c > 0) {
                            cp_async8(d + 81 + t, pA + t);
                            cp_async8(d + 162 + t, pC + t);
                        }
                    }
                }
            }
            cp_async_commit();
        };
        auto put = [&](double *dst, const double *src) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int t = lane + 32 * r;
                if (t < 81) dst[t] = src[t];
            }
        };
        int ep2 = 0, ep1 = 0, e0 = elem(0), e1 = elem(1), e2 = elem(2), e3 = elem(3);
        int f2 = face(2), f3 = face(3), a2;
        {
            const int f1 = face(1);
            copy(0, e0, 0, 0);
            copy(1, e1, f1, first(1, f1));
        }
        a2 = first(2, f2);
        cp_async_wait<1>();
        __syncthreads();
        for (int s = 0; s <= n + 1; ++s) {
            copy(s + 2, e2, f2, a2);
            const int en = elem(s + 4), fn = face(s + 4), an = first(s + 3, f3);
            if (s >= 1 && s < n) put(Aout + 81 * (size_t)e0, stage[s % LS] + 81);
            if (s >= 1 && s - 1 < n) put(Dia + 81 * (size_t)ep1, sL[(s - 1) & 1]);
            if (s >= 2 && s - 1 < n) put(DinvC + 81 * (size_t)ep2, sG[(s - 1) & 1]);
            ep2 = ep1;
            ep1 = e0;
            e0 = e1;
            e1 = e2;
            e2 = e3;
            e3 = en;
            f2 = f3;
            f3 = fn;
            a2 = an;
            cp_async_wait<1>();
            __syncthreads();
        }
        cp_async_wait<0>();
        return;
    }
    /* lanes 27..31 repeat lanes 18..22 and store nothing */
    const bool act = lane < 27;
    const int ln = act ? lane : lane - 9;
    const int i = ln % 9, g = ln / 9;
    const int col = lane < 9 ? lane : 8;
    bool bad = false;
    __syncthreads();
    for (int s = 0; s <= n + 1; ++s) {
        if (s < n) {
            const double *D = stage[s % LS], *A = D + 81, *C = D + 162;
            double w[3];
            if (s > 0) {
                /* Gamma(:, col) = D'_{s-1}^-1 C(:, col) (lineLU_v2.okl:142-144) */
                double v[9], x[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) v[k] = C[k + 9 * col];
                const double *L = sL[(s - 1) & 1];
                const bool ok = ref_solve9(L, rc, v, x);
                if (!ok || rc[18] != 0.0) solve_lu_lane<9>(L, v, x, 9);
                if (lane < 9) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) sG[s & 1][k + 9 * col] = x[k];
                }
                __syncwarp();
            }
            /* D_s - A Gamma (lineLU_v2.okl:147-161) */
            auto pivot = [&]() {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int c = 3 * g + k;
                    w[k] = D[i + 9 * c];
                    if (s > 0) {
                        const double *G = sG[s & 1] + 9 * c;
                        double tot = fma(A[i], G[0], 0.0);
#pragma unroll
                        for (int j = 1; j < 9; ++j) tot += A[i + 9 * j] * G[j];
                        w[k] = w[k] - tot;
                    }
                }
            };
            pivot();
            if (ref_lu27<false>(w, i, g, act && g == 0, rc)) { /* the same in every lane */
                pivot();
                double v[3] = {w[0], w[1], w[2]};
                __syncwarp();
                bad = ref_lu27_plain(v, i, g, act && g == 0, rc) || bad;
#pragma unroll
                for (int k = 0; k < 3; ++k) w[k] = v[k];
            }
            if (act) {
#pragma unroll
                for (int k = 0; k < 3; ++k) sL[s & 1][i + 9 * (3 * g + k)] = w[k];
            }
            __syncwarp();
        }
        __syncthreads();
    }
    if (bad && lane == 0) atomicOr(status, ST_PIVOT);
}

/* Jacobian.cxx:76-117: A[e] = (e == fc[2f]) ? O2[f] : O1[f], f = lineface[m],
 * for every line cell after the first.  One warp per line cell. */
__global__ void ref_assemble_A_kernel(int nv, int nline, const int *__restrict__ fc,
                                      const int *__restrict__ linesize,
                                      const int *__restrict__ linepoint,
                                      const int *__restrict__ lines,
                                      const int *__restrict__ lineface,
                                      const double *__restrict__ O1,
                                      const double *__restrict__ O2, double *__restrict__ A) {
    const int l = blockIdx.x;
    if (l >= nline) return;
    const size_t bs = (size_t)nv * nv;
    const int n = linesize[l];
    for (int k = 1 + threadIdx.y; k < n; k += blockDim.y) {
        const int m = linepoint[l] + k;
        const int f = lineface[m];
        const int e = lines[m];
        const double *src = (e == fc[2 * f]) ? &O2[bs * f] : &O1[bs * f];
        for (int t = threadIdx.x; t < (int)bs; t += 32) A[bs * e + t] = src[t];
    }
}

/* Block size 9: whether the kernels of two warps a line are the faster ones.
 * They are where the longest line's chain sets the time or four lines an SM
 * (their registers allow no more) take them all in a few rounds; the kernels
 * of one warp a line, slower along a chain, hold all of an SM's lines at once
 * and have nothing to fill before the first cell.  Estimates, in us: two
 * warps, `step` a cell and line and two cells' worth (the factorization) or
 * three to start a line, in rounds of four lines an SM; one warp, a cell
 * `alone` and `more` for each line that shares the SM, or `flow` a cell and SM.
 * Measured (two warps / one, us): solve 592x16 23 / 38, 1200x100 288 / 299,
 * 1800x100 384 / 317, 700x8 24 / 22, 592x3 11 / 11, 20000x16 588 / 364, 20000x1
 * 82 / 23; factorization 592x16 37 / 87, 1200x16 84 / 105,
 * 1800x100 682 / 714, 2500x16 148 / 138, 20000x3 221 / 154. */
struct RefRate {
    double step, start, alone, more, flow;
};
constexpr RefRate REF_LU{1.74, 2.0, 5.2, 0.16, 0.385}, REF_DU{1.0, 3.0, 2.6, 0.05, 0.17};

static bool ref_two_warps(const RefRate &r, int nline, long long cells, int longest) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (nsm < 1) nsm = 148;
    const double rounds = (nline + 4 * nsm - 1) / (4 * nsm), mean = (double)cells / nline;
    const double two = r.step * std::max(longest + r.start, rounds * (mean + r.start));
    const double one = std::max(longest * (r.alone + r.more * nline / nsm), r.flow * (double)cells / nsm);
    return two < one;
}


/* the line factorization (DLU in place, DinvC) and the packed lower blocks */
int launch_ref_line_lu(cudaStream_t st, int nv, int nline, long long cells, int longest, const int *fc,
                       const int *linesize, const int *linepoint, const int *lines, const int *lineface, double *DLU,
                       const double *O1, const double *O2, double *DinvC, double *A, unsigned *status) {
    if (nv < 1 || nv > REF_MAXNV) return (int)cudaErrorInvalidValue;
    if (nv == 9 && ref_two_warps(REF_LU, nline, cells, longest)) {
        ref_line_lu9_kernel<<<nline, 64, 0, st>>>(nline, fc, linesize, linepoint, lines, lineface, DLU, O1,
                                                  O2, DinvC, A, status);
        return (int)cudaGetLastError();
    }
    const size_t smem = 5 * (size_t)nv * nv * sizeof(double);
    if (smem > 48 * 1024) {
        const int e = smem_raise((const void *)ref_line_lu_kernel<0>, smem);
        if (e != 0) return e;
    }
    ref_assemble_A_kernel<<<nline, dim3(32, 8), 0, st>>>(nv, nline, fc, linesize, linepoint, lines,
                                                         lineface, O1, O2, A);
    if (nv == 9)
        ref_line_lu_kernel<9><<<nline, 32, smem, st>>>(nv, nline, fc, linesize, linepoint, lines, lineface,
                                                       DLU, O1, O2, DinvC, status);
    else
        ref_line_lu_kernel<0><<<nline, 32, smem, st>>>(nv, nline, fc, linesize, linepoint, lines, lineface,
                                                       DLU, O1, O2, DinvC, status);
    return (int)cudaGetLastError();
}

/* ref_solve_du_kernel for block size 9: one CTA of two warps per line.
 * What bounds it is the dependent chain of a cell -- 9 multiply-adds and
 * subtractions forward, 28 additions, 9 subtractions and 9 divisions
 * backward, in solveLU's order -- about 1,100 cycles; lane 0 solving alone
 * and loading what it needs as it goes (ref_solve_du_kernel) took 5,300.
 * 360x384: 1,053 -> 382 us. */
__global__ void __launch_bounds__(64) ref_solve_du9_kernel(
    int nline, const int *__restrict__ linesize, const int *__restrict__ linepoint,
    const int *__restrict__ lines, const double *__restrict__ Dia, const double *__restrict__ DinvC,
    const double *__restrict__ A, double *__restrict__ dU, const double *__restrict__ R) {
    __shared__ __align__(16) double stage[RS][RC][RCELL];
    __shared__ __align__(16) double vec[2][10];
    const int l = blockIdx.x;
    if (l >= nline) return;
    const int lane = threadIdx.x & 31;
    const int n = linesize[l], m0 = linepoint[l];
    const int nf = (n + RC - 1) / RC, nb = (n - 1 + RC - 1) / RC, njobs = nf + nb;
    /* forward job c: cells 4c..; backward job c: cells n-2-4c, n-3-4c, .. */
    auto cell = [&](int job, int q) { return job < nf ? job * RC + q : n - 2 - ((job - nf) * RC + q); };
    auto valid = [&](int job, int q) {
        const int k = cell(job, q);
        return job < njobs && k >= 0 && k < (job < nf ? n : n - 1);
    };
    if (threadIdx.x >= 32) {
        auto index = [&](int job) { return lane < RC && valid(job, lane) ? lines[m0 + cell(job, lane)] : 0; };
        auto copy = [&](int job, int es) {
#pragma unroll
            for (int q = 0; q < RC; ++q) {
                const size_t e = __shfl_sync(0xffffffffu, es, q);
                if (!valid(job, q)) continue;
                double *d = stage[job % RS][q];
                const double *b0 = (job < nf ? Dia : DinvC) + 81 * e, *b1 = A + 81 * e;
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const int t = lane + 32 * r;
                    if (t < 81) {
                        cp_async8(d + t, b0 + t);
                        if (job < nf) cp_async8(d + 81 + t, b1 + t);
                    }
                }
                if (job < nf && lane < 9) cp_async8(d + 162 + lane, R + 9 * e + lane);
            }
            cp_async_commit();
        };
        /* the reciprocals of a landed forward job's diagonals */
        auto recips = [&](int job) {
            __syncwarp();
            if (job >= nf) return;
            if (lane < RC) stage[job % RS][lane][189] = 0.0;
            __syncwarp();
            for (int t = lane; t < 9 * RC; t += 32) {
                const int q = t / 9, i = t % 9;
                double *d = stage[job % RS][q];
                const double u = d[10 * i], r = rcp_newton(u);
                d[171 + i] = r;
                d[180 + i] = fma(-u, r, 1.0) * r;
                if (ref_plain_divisor(u)) d[189] = 1.0;
            }
        };
        copy(0, index(0));
        copy(1, index(1));
        int es = index(2);
        cp_async_wait<1>();
        recips(0);
        __syncthreads();
        for (int job = 0; job < njobs; ++job) {
            copy(job + 2, es);
            es = index(job + 3);
            cp_async_wait<1>();
            recips(job + 1);
            __syncthreads();
        }
        cp_async_wait<0>();
        return;
    }
    const int i = lane < 9 ? lane : 8;
    double x[9];
    __syncthreads();
    for (int job = 0; job < nf; ++job) {
        int es[RC];
#pragma unroll
        for (int q = 0; q < RC; ++q) es[q] = valid(job, q) ? lines[m0 + cell(job, q)] : 0;
#pragma unroll 1
        for (int q = 0; q < RC; ++q) {
            if (!valid(job, q)) break;
            const double *d = stage[job % RS][q];
            /* lane i: s_i = -R_i - (A dU_{k-1})_i */
            double si = -d[162 + i];
            if (job > 0 || q > 0) {
                double tot = fma(d[81 + i], x[0], 0.0);
#pragma unroll
                for (int j = 1; j < 9; ++j) tot += d[81 + i + 9 * j] * x[j];
                si = si - tot;
            }
            double s[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) s[j] = __shfl_sync(0xffffffffu, si, j);
            const bool ok = ref_solve9(d, d + 171, s, x);
            if (!ok || d[189] != 0.0) solve_lu_lane<9>(d, s, x, 9); /* the same in every lane */
            double mine = x[0];
#pragma unroll
            for (int j = 1; j < 9; ++j) mine = i == j ? x[j] : mine;
            const int e = q == 0 ? es[0] : q == 1 ? es[1] : q == 2 ? es[2] : es[3];
            if (lane < 9) dU[9 * (size_t)e + i] = mine;
        }
        __syncthreads();
    }
    /* back substitution: dU_k -= DinvC_k dU_{k+1}, the vector through shared
     * memory (lanes 9.. repeat lane 8); a job's dU is read (by the lanes that
     * wrote it) one job ahead */
    {
        double mine = x[0];
#pragma unroll
        for (int j = 1; j < 9; ++j) mine = i == j ? x[j] : mine;
        vec[0][i] = mine;
        __syncwarp();
    }
    double u[RC], nu[RC];
    int es[RC], ns[RC];
    auto fetch = [&](int job, double *v, int *ee) {
#pragma unroll
        for (int q = 0; q < RC; ++q) {
            ee[q] = valid(job, q) ? lines[m0 + cell(job, q)] : 0;
            v[q] = valid(job, q) ? dU[9 * (size_t)ee[q] + i] : 0.0;
        }
    };
    if (nb > 0) fetch(nf, u, es);
    for (int job = nf; job < njobs; ++job) {
        fetch(job + 1, nu, ns);
#pragma unroll
        for (int q = 0; q < RC; ++q) {
            if (valid(job, q)) {
                const double *d = stage[job % RS][q];
                const double2 *v = reinterpret_cast<const double2 *>(vec[q & 1]);
                const double2 v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
                const double v8 = vec[q & 1][8];
                double tot = fma(d[i], v0.x, 0.0);
                tot += d[i + 9] * v0.y;
                tot += d[i + 18] * v1.x;
                tot += d[i + 27] * v1.y;
                tot += d[i + 36] * v2.x;
                tot += d[i + 45] * v2.y;
                tot += d[i + 54] * v3.x;
                tot += d[i + 63] * v3.y;
                tot += d[i + 72] * v8;
                const double mine = u[q] - tot;
                vec[(q & 1) ^ 1][i] = mine;
                if (lane < 9) dU[9 * (size_t)es[q] + i] = mine;
                __syncwarp();
            }
        }
#pragma unroll
        for (int q = 0; q < RC; ++q) {
            u[q] = nu[q];
            es[q] = ns[q];
        }
        __syncthreads();
    }
}

/* linesmoothLU_TriBlock_v3.okl:92-226, any block size.  Lane 0 runs solveLU as the
 * reference does (its `if(i==0)` guard, :154/:192); the other lanes do the
 * row-parallel matvecs and prefetch the next cell's blocks meanwhile. */
template <int NV>
__global__ void __launch_bounds__(32) ref_solve_du_kernel(
    int nv_rt, int nline, const int *__restrict__ linesize, const int *__restrict__ linepoint,
    const int *__restrict__ lines, const double *__restrict__ Dia,
    const double *__restrict__ DinvC, const double *__restrict__ A, double *__restrict__ dU,
    const double *__restrict__ R) {
    const int nv = NV ? NV : nv_rt;
    const int l = blockIdx.x;
    if (l >= nline) return;
    const int lane = threadIdx.x;
    const size_t bs = (size_t)nv * nv;
    extern __shared__ double sm[];
    double *sDia = sm;
    double *sAT = sDia + bs;
    double *sS = sAT + bs;
    double *sdU = sS + REF_MAXNV;

    const int n = linesize[l];
    const int m0 = linepoint[l];
    int e = lines[m0];
    if (lane < nv) {
        sS[lane] = -R[lane + (size_t)nv * e];
        for (int j = 0; j < nv; ++j) sDia[MIDX(lane, j, nv)] = Dia[MIDX(lane, j, nv) + bs * e];
    }
    __syncwarp();
    if (lane == 0) solve_lu_lane<NV>(sDia, sS, sdU, nv);
    __syncwarp();
    if (lane < nv) dU[lane + (size_t)nv * e] = sdU[lane];

    for (int k = 1; k < n; ++k) {
        e = lines[m0 + k];
        __syncwarp();
        if (lane < nv) {
            for (int j = 0; j < nv; ++j) {
                sAT[MIDX(j, lane, nv)] = A[MIDX(lane, j, nv) + bs * e];
                sDia[MIDX(lane, j, nv)] = Dia[MIDX(lane, j, nv) + bs * e];
            }
        }
        __syncwarp();
        if (lane < nv) {
            double tot = 0.0;
            for (int j = 0; j < nv; ++j) tot += sAT[MIDX(j, lane, nv)] * sdU[j];
            sS[lane] = -R[lane + (size_t)nv * e] - tot;
        }
        __syncwarp();
        if (lane == 0) solve_lu_lane<NV>(sDia, sS, sdU, nv);
        __syncwarp();
        if (lane < nv) dU[lane + (size_t)nv * e] = sdU[lane];
    }
    /* back substitution: dU_k -= DinvC_k dU_{k+1}; sdU holds dU of the
     * last cell, the value the reference reloads from global memory */
    for (int k = n - 2; k >= 0; --k) {
        e = lines[m0 + k];
        double mine = 0.0;
        if (lane < nv) {
            double tot = 0.0;
            for (int j = 0; j < nv; ++j) tot += DinvC[MIDX(lane, j, nv) + bs * e] * sdU[j];
            mine = dU[lane + (size_t)nv * e] - tot;
            dU[lane + (size_t)nv * e] = mine;
        }
        __syncwarp();
        if (lane < nv) sdU[lane] = mine;
        __syncwarp();
    }
}

int launch_ref_solve_du(cudaStream_t st, int nv, int nline, long long cells, int longest,
                        const int *linesize, const int *linepoint, const int *lines, const double *DLU,
                        const double *DinvC, const double *A, double *dU, const double *R) {
    if (nv < 1 || nv > REF_MAXNV) return (int)cudaErrorInvalidValue;
    const size_t smem = (2 * (size_t)nv * nv + 2 * REF_MAXNV) * sizeof(double);
    if (nv == 9 && ref_two_warps(REF_DU, nline, cells, longest))
        ref_solve_du9_kernel<<<nline, 64, 0, st>>>(nline, linesize, linepoint, lines, DLU, DinvC, A, dU, R);
    else if (nv == 9)
        ref_solve_du_kernel<9><<<nline, 32, smem, st>>>(nv, nline, linesize, linepoint, lines, DLU, DinvC, A,
                                                        dU, R);
    else
        ref_solve_du_kernel<0><<<nline, 32, smem, st>>>(nv, nline, linesize, linepoint, lines, DLU, DinvC, A,
                                                        dU, R);
    return (int)cudaGetLastError();
}

/* addAtoB (U += dU) and copyAtoB (R = rhs), linesmoothLU_v5.okl:75-103 */
__global__ void ref_add_copy_kernel(long long n, const double *__restrict__ dU,
                                    double *__restrict__ U, const double *__restrict__ rhs,
                                    double *__restrict__ R) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        U[t] += dU[t];
        R[t] = rhs[t];
    }
}

int launch_ref_add_copy(cudaStream_t st, long long n, const double *dU, double *U,
                        const double *rhs, double *R) {
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    ref_add_copy_kernel<<<(int)blocks, 256, 0, st>>>(n, dU, U, rhs, R);
    return (int)cudaGetLastError();
}

/* linesmoothLU_TriBlock_v3.okl:228-336, one thread per (element, row):
 * R(i,e) += [D U](i) + sum over faces in ef order of [offJ U_nbr](i).
 * Each block also writes the sum of R^2 over its entries (fixed-order tree)
 * for the residual norm the reference does not compute. */
constexpr int RES_THREADS = 288;

__global__ void __launch_bounds__(RES_THREADS) ref_line_res_kernel(
    int nv, int nelem, const int *__restrict__ epoint, const int *__restrict__ ef,
    const int *__restrict__ fc, const double *__restrict__ D, const double *__restrict__ O1,
    const double *__restrict__ O2, const double *__restrict__ U, double *__restrict__ R,
    double *__restrict__ partials) {
    const int epb = RES_THREADS / nv;
    const int le = threadIdx.x / nv;
    const int i = threadIdx.x - le * nv;
    const int e = blockIdx.x * epb + le;
    const size_t bs = (size_t)nv * nv;
    double sq = 0.0;
    if (le < epb && e < nelem) {
        double tot = 0.0;
        for (int j = 0; j < nv; ++j) tot += D[MIDX(i, j, nv) + bs * e] * U[j + (size_t)nv * e];
        double sR = tot;
        for (int k2 = epoint[e]; k2 < epoint[e + 1]; ++k2) {
            const int f = ef[k2];
            if (f >= 0) {
                const int e1 = fc[2 * f + 0];
                const int e2 = fc[2 * f + 1];
                const double *offJ = (e == e1) ? O2 : O1;
                const int nb = (e == e1) ? e2 : e1;
                double t2 = 0.0;
                for (int j = 0; j < nv; ++j) t2 += offJ[MIDX(i, j, nv) + bs * f] * U[j + (size_t)nv * nb];
                sR += t2;
            }
        }
        const double r = R[i + (size_t)nv * e] + sR;
        R[i + (size_t)nv * e] = r;
        sq = r * r;
    }
    /* deterministic block sum */
    __shared__ double red[RES_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < RES_THREADS / 32; ++w) s += red[w];
        partials[blockIdx.x] = s;
    }
}

int ref_line_res_partials(int nelem) { return (nelem + 31) / 32; }

int launch_ref_line_res(cudaStream_t st, int nv, int nline, int nelem, const int *epoint,
                        const int *ef, const int *fc, const int *linesize, const int *linepoint,
                        const int *lines, const double *D, const double *O1, const double *O2,
                        const double *U, double *R, double *partials, int *npartials_out) {
    (void)nline;
    (void)linesize;
    (void)linepoint;
    (void)lines;
    if (nv < 1 || nv > REF_MAXNV) return (int)cudaErrorInvalidValue;
    const int epb = RES_THREADS / nv;
    const int blocks = (nelem + epb - 1) / epb;
    if (npartials_out) *npartials_out = blocks;
    ref_line_res_kernel<<<blocks, RES_THREADS, 0, st>>>(nv, nelem, epoint, ef, fc, D, O1, O2, U, R,
                                                        partials);
    return (int)cudaGetLastError();
}

}  // namespace tbs
