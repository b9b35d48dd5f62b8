/*
 * thomas.cuh -- the line solve (block Thomas on explicit inverses) of one
 * line by one warp, or by a chain warp with a copy warp beside it, shared by
 * kernels_fast.cu (block size 9, FP64 and FP32) and kernels_nv.cu (the other
 * block sizes, FP64).
 */
#ifndef TBS_THOMAS_CUH
#define TBS_THOMAS_CUH

#include "device_common.cuh"
#include "tbs_internal.hxx"
#include "tma.cuh"

#include <cuda_runtime.h>

namespace tbs {

/* =========================================================== line Thomas
 * One warp per line, twisted (block size NV <= 16; 9 in the figures): lanes
 * 0..NV-1 run the top chain and lanes 16..16+NV-1 the bottom chain of the line with the same instruction stream, so
 * a line of n cells takes n+1 dependent steps instead of 2n.  Lane 0 (or a
 * copy warp) streams "jobs" through an NS-stage bulk-copy ring, each stage
 * holding one chunk of P cells per chain: jobs 0..nf-1 forward chunks (G
 * blocks and b), jobs nf..2nf-1 backward chunks in reverse (Gam blocks).
 * Chain forward:  y_s = b_s - G_s y_{s-1};  twist:  x_m = b_m - G_tw y_top
 * - Gam_tw y_bot;  chain backward:  x_s = y_s - Gam_s x_{s+1} (s+1 toward
 * the twist).
 *
 * What bounds it where few lines share an SM is the step: publish the
 * 9-vector in shared memory, read it back, a 9-term dot product.  On a warp
 * alone, rows held in registers, that is 86 cycles; so everything else is
 * kept off the chain.  Lane i owns row i; the row of the NEXT cell is read
 * into registers behind the current step's vector reads, across chunk
 * boundaries too: the next chunk's barrier is tested early in a chunk and
 * the result looked at a few steps later (testing it between chunks and
 * reading the row after it cost about 300 cycles per 8-cell chunk).  The
 * blocks are column-major, so that the nine lanes read a column of nine
 * neighbouring words: no bank conflicts and one copy of the vector (with
 * row-major blocks: two copies, lane-dependent offsets, 122 cycles a step
 * against 106; rows as aligned pairs of columns: 111).  The dot product is
 * three partial sums, so that no more than four roundings follow one another
 * (two sums: six, and an error 3 to 4 % larger); the vector's words arrive
 * one after the other, and the last of them joins the sum that starts from
 * the right-hand side, two operations from the result: as fast as two sums
 * to 1 % (45 us and 46 at 360x384, 32.9 and 32.8 at 181x301).
 * YS: the line's y and x live in shared memory, and dU / U are written after
 * the line is solved: dU by one bulk copy, and in FP64 U += dU by one bulk
 * add (the L2 adds, so the warp does not wait for U); otherwise y goes to
 * global memory (read back one chunk ahead) and dU / U per step, U read
 * one chunk ahead with y (one-warp form) or staged behind the backward
 * chunk's Gam blocks by the copy warp (warp-specialised form).
 *   accumulate = 0:  U = dU
 *   accumulate = 1:  U += dU (the FP64 sweeps of a context; U read from a
 *                    second buffer Uin when one is given: line partitions)
 *   accumulate = 2:  U untouched (the residual kernel that follows adds
 *                    dU to U for its tile, with coalesced tile accesses:
 *                    the batch engine)
 */
template <typename T, int NV, int P>
__host__ __device__ constexpr uint32_t thomas_stage_bytes() {
    return (uint32_t)(2 * P * (NV * NV + NV) * sizeof(T));
}

/* The vector a step reads and the row it multiplies.
 * FP64: lane i's row in column order, and one copy of the vector read as
 * four pairs and a single.
 * FP32: the vector in two copies (y_j at j and at 11 + j), so that a lane
 * whose row number and cell have different parity starts its pairs at
 * column 1; the order of the sum by lane is kept as it was first written,
 * since the outer refinement's history shows a change of FP32 rounding. */
template <typename T, int NV> struct StepVec;

template <int NV>
struct StepVec<double, NV> {
    static constexpr int BUF = (NV + 1) & ~1; /* words of one buffer */
    double v[NV];
    __device__ __forceinline__ void load(const double *b, int, int) {
        const double2 *q = reinterpret_cast<const double2 *>(b);
#pragma unroll
        for (int c = 0; c < NV / 2; ++c) {
            const double2 d = q[c];
            v[2 * c] = d.x;
            v[2 * c + 1] = d.y;
        }
        if (NV & 1) v[NV - 1] = b[NV - 1];
    }
    static __device__ __forceinline__ void put(double *buf, int i, double y) { buf[i] = y; }
};

template <>
struct StepVec<float, 9> {
    static constexpr int BUF = 20;
    float2 p[4];
    float s;
    __device__ __forceinline__ void load(const float *v, int i, int odd) {
        const int par = (i + odd) & 1;
        const float2 *q = reinterpret_cast<const float2 *>(v + (par ? 12 : 0));
#pragma unroll
        for (int c = 0; c < 4; ++c) p[c] = q[c];
        s = v[par ? 0 : 8];
    }
    static __device__ __forceinline__ void put(float *buf, int i, float y) {
        buf[i] = y;
        buf[11 + i] = y;
    }
};

/* row i of a block, in the order StepVec gives the vector: FP64 columns in
 * order; FP32 the single's column, then the pairs' */
template <typename T, int NV>
struct Row {
    T r[NV];
};

template <int NV>
__device__ __forceinline__ void load_row(Row<double, NV> &R, const double *blk, int i, int) {
#pragma unroll
    for (int j = 0; j < NV; ++j) R.r[j] = blk[NV * j + i];
}

__device__ __forceinline__ void load_row(Row<float, 9> &R, const float *blk, int i, int odd) {
    const int par = (i + odd) & 1;
    const float *q = blk + i - (par ? 0 : 9);
    R.r[0] = blk[par ? i : 72 + i];
#pragma unroll
    for (int j = 1; j < 9; ++j) R.r[j] = q[9 * j];
}

/* init - row . vec in three partial sums: the terms j with NV - 1 - j
 * divisible by three go to the one that starts from init, each of the others
 * opens with its second product, rounded, and the first */
template <int NV>
__device__ __forceinline__ double row_dot(const Row<double, NV> &R, const StepVec<double, NV> &V, double init) {
    double a[3] = {init, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = (NV - 1 - j) % 3;
        if (c == 0)
            a[0] = fma_rn(-R.r[j], V.v[j], a[0]);
        else if (j < 3)
            a[c] = j + 3 < NV ? fma_rn(R.r[j], V.v[j], mul_rn(R.r[j + 3], V.v[j + 3])) : mul_rn(R.r[j], V.v[j]);
        else if (j >= 6)
            a[c] = fma_rn(R.r[j], V.v[j], a[c]);
    }
    return a[0] - (NV > 2 ? a[1] + a[2] : a[1]);
}

__device__ __forceinline__ float row_dot(const Row<float, 9> &R, const StepVec<float, 9> &V, float init) {
    float a0 = fma_rn(-R.r[0], V.s, init);
    float a1 = fma_rn(R.r[1], V.p[0].x, mul_rn(R.r[4], V.p[1].y));
    float a2 = fma_rn(R.r[2], V.p[0].y, mul_rn(R.r[5], V.p[2].x));
    a0 = fma_rn(-R.r[3], V.p[1].x, a0);
    a0 = fma_rn(-R.r[6], V.p[2].y, a0);
    a1 = fma_rn(R.r[7], V.p[3].x, a1);
    a2 = fma_rn(R.r[8], V.p[3].y, a2);
    return a0 - (a1 + a2);
}

/* The next chunk's stage is taken two steps before its first row is read, so
 * that the barrier's answer is there; where blocks of 13 and more leave the
 * ring two stages, at that step: a stage is refilled when its chunk is done,
 * and what is taken early was asked for late (900x1100, nvar 13 529 / 520 us, 15
 * 830 / 817, 16 878 / 867; smaller blocks and deeper rings lose up to 3 %). */
template <int NV, bool YS>
constexpr bool LATE = NV >= 13 && !YS;

/* words of the broadcast vectors: 2 halves x 2 alternating buffers */
template <typename T, int NV>
constexpr int BCAST = 4 * StepVec<T, NV>::BUF;

/* Forward steps kbase..kbase+P-1 of this half's chain (length len, first
 * position cpos relative to the line start), the chunk's blocks at sG and
 * its b behind them; `row` / `bi` hold the first cell's row and b, and are
 * left holding those of the next chunk, whose stage next() gives (null:
 * none; probe() has asked for it).  CHECK: some steps of the warp may lie
 * beyond one chain's end; those compute but write nothing, and beyond the
 * longer chain's (`last` cells: no chunk follows) none are made: 50,000 lines
 * of three cells 186 us a line solve, 169 so, FP32 118 and 101. */
template <typename T, int NV, int P, bool CHECK, bool YS, typename Probe, typename Next>
__device__ __forceinline__ void fwd_chunk(const T *sG, Row<T, NV> &row, T &bi, T *bc, T *ys, T *yg,
                                          int kbase, int len, int last, int cpos, int i, uint64_t ypol,
                                          Probe &&probe, Next &&next) {
    constexpr int NB = NV * NV, VB = StepVec<T, NV>::BUF;
    const T *sB = sG + P * NB;
    const T *sN = sG;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        if (CHECK && q > 0 && kbase + q >= last) break; /* both chains have ended: the last chunk */
        Row<T, NV> nrow;
        StepVec<T, NV> v;
        T nb = T(0);
        if (LATE<NV, YS> && q == P - 1) {
            const T *n = next();
            if (n) sN = n;
        }
        v.load(bc + (q & 1) * VB, i, q & 1);
        if (q + 1 < P) {
            load_row(nrow, sG + (q + 1) * NB, i, (q + 1) & 1);
            nb = sB[(q + 1) * NV + i];
        } else { /* no next chunk: some cell of this one, not used */
            load_row(nrow, sN, i, 0);
            nb = sN[P * NB + i];
        }
        if (q == 1) probe();
        if (!LATE<NV, YS> && q == P - 3) {
            const T *n = next();
            if (n) sN = n;
        }
        const T yi = row_dot(row, v, bi);
        /* lanes 9..15 of a half compute row 8 from the same inputs as lane
         * 8 and store the same value to the same address: no divergence */
        if (!CHECK || kbase + q < len) {
            StepVec<T, NV>::put(bc + ((q & 1) ^ 1) * VB, i, yi);
            const int pos = cpos + kbase + q;
            if (YS)
                ys[pos * NV + i] = yi;
            else /* kept in L2 for the backward chain (the blocks stream evict-first) */
                st_hint(yg + (size_t)pos * NV + i, yi, ypol);
        }
        __syncwarp();
        row = nrow;
        bi = nb;
    }
}

/* Backward steps kbase+P-1..kbase, `row` holding the row of the first of
 * them (and left holding the next chunk's).  YS: y and x in ys, `yk` the y
 * of the first step, left holding the next chunk's; otherwise the chunk's
 * y in yv.  uv: U of the chunk's cells read ahead in registers, or sU (when
 * set): the chunk's U staged behind its Gam blocks */
template <typename T, int NV, int P, bool CHECK, bool YS, typename Probe, typename Next>
__device__ __forceinline__ void bwd_chunk(const T *sG, Row<T, NV> &row, T &yk, T *bc, T *ys, const T *yv,
                                          const T *uv, T *dUl, T *Ul, int kbase, int len, int cpos,
                                          int i, const T *sU, Probe &&probe, Next &&next) {
    constexpr int NB = NV * NV, VB = StepVec<T, NV>::BUF;
    const T *sN = sG;
#pragma unroll
    for (int q = P - 1; q >= 0; --q) {
        const int f = (P - 1 - q) & 1; /* buffer alternates per step */
        Row<T, NV> nrow;
        StepVec<T, NV> v;
        if (LATE<NV, YS> && q == 0) {
            const T *n = next();
            if (n) sN = n;
        }
        v.load(bc + f * VB, i, q & 1);
        load_row(nrow, q > 0 ? sG + (q - 1) * NB : sN + (P - 1) * NB, i, (q + P - 1) & 1);
        if (q == P - 2) probe();
        if (!LATE<NV, YS> && q == 2) {
            const T *n = next();
            if (n) sN = n;
        }
        const int k = kbase + q;
        const bool valid = !CHECK || (k >= 0 && k < len);
        const int pos = cpos + k;
        T nyk = T(0);
        if (YS && ((CHECK || q == 0) ? (k >= 1 && k - 1 < len) : true)) nyk = ys[(pos - 1) * NV + i];
        const T d = row_dot(row, v, YS ? yk : (valid ? yv[q] : T(0)));
        if (valid) { /* lanes 9..15 repeat lane 8's row, value and address */
            StepVec<T, NV>::put(bc + (f ^ 1) * VB, i, d);
            if (YS) {
                ys[pos * NV + i] = d;
            } else {
                dUl[(size_t)pos * NV + i] = d;
                if (Ul) Ul[(size_t)pos * NV + i] = (sU ? sU[q * NV + i] : uv[q]) + d;
            }
        }
        __syncwarp();
        row = nrow;
        yk = nyk;
    }
}

/* Solve one line (start ps, n cells, twist m) with the warp of the calling
 * CTA.  The staging barriers live at the start of `smem` and stay
 * initialised across the lines that a persistent CTA solves: bit s of
 * `pbase` is the parity with which barrier s completes its next phase.
 * Returns false when a staging wait ran out of time; the status bit is
 * then set and the copies in flight have landed. */
/* bytes before the first staging buffer: the barriers (and, in the
 * warp-specialised form, the producer's counters) */
template <bool WS>
__host__ __device__ constexpr int thomas_hdr() { return WS ? 256 : 128; }

/* the two warps of a warp-specialised line solve (the CTA may hold more) */
__device__ __forceinline__ void ws_meet() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

/* accumulate = 1 reads U from Uin when it is set (a second buffer: the
 * previous U stays intact), else from U itself.  drain (YS): dU has been
 * written when the call returns, not only read from shared memory (for kernels
 * that go on to read it), U before the next call writes it.  b and U are read
 * past the L1, which may hold an earlier sweep's. */
/* PH 0: the whole line.  The other phases split it (WS; the copy warp's lane
 * 0 acts in all but the third): PH_BLOCKS starts the copies of the first jobs'
 * blocks, while others still write b; PH_VECS those of their b; PH_RUN is the
 * line after both; PH_DROP waits for the copies when no line follows. */
enum { PH_ALL = 0, PH_BLOCKS, PH_VECS, PH_RUN, PH_DROP };

template <typename T, int NV, int P, bool YS, bool WS = false, int PH = PH_ALL>
__device__ __forceinline__ bool thomas_line(
    int NS, int accumulate, int ps, int n, int m, const T *__restrict__ G,
    const T *__restrict__ Gam, const T *__restrict__ b, T *__restrict__ y, T *__restrict__ dU,
    T *__restrict__ U, unsigned *status, unsigned char *smem, uint32_t &pbase, uint64_t pol,
    const T *__restrict__ Uin = nullptr, bool drain = false) {
    constexpr int NB = NV * NV;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    /* WS (warp-specialised CTA of two warps): bars[0..NS) complete when a
     * stage's copies have landed, bars[8..8+NS) when warp 0 has consumed
     * it; warp 1 lane 0 issues the copies, warp 0 runs the chains */
    uint64_t *empty = bars + 8;
    volatile int *ws_issued = reinterpret_cast<volatile int *>(smem + 128);
    volatile int *ws_abort = ws_issued + 1;
    const uint32_t stage = thomas_stage_bytes<T, NV, P>();
    const uint32_t half = stage / 2;
    unsigned char *st0 = smem + thomas_hdr<WS>();
    T *bcall = reinterpret_cast<T *>(st0 + (size_t)NS * stage);
    constexpr int VB = StepVec<T, NV>::BUF;
    T *ys = bcall + BCAST<T, NV>;
    const int lane = threadIdx.x & 31;
    const int h = lane >> 4, li = lane & 15;
    const int i = li < NV ? li : NV - 1;
    const int nb = n - 1 - m;
    const int len = h ? nb : m;      /* this half's chain length */
    const int cpos = h ? m : 0;      /* its first position, relative to ps */
    const int nchT = (m + P - 1) / P, nchB = (nb + P - 1) / P;
    const int nch = h ? nchB : nchT;
    const int nf = nchT > nchB ? nchT : nchB;
    const int njobs = 2 * nf;
    T *bc = bcall + h * 2 * VB;
    T *yl = y + (size_t)ps * NV;
    T *dUl = dU + (size_t)ps * NV;
    T *Ul = U ? U + (size_t)ps * NV : nullptr;
    const T *Uil = Uin ? Uin + (size_t)ps * NV : Ul;

    const bool producer = WS && (threadIdx.x >> 5) == 1;
    /* warp-specialised form: the copy warp also stages U behind the
     * backward chunks' Gam blocks (where the forward stages hold b), so the
     * chain warp reads it from shared memory */
    const bool stage_u = WS && !YS && accumulate == 1 && Ul != nullptr;
    __syncwarp(); /* the previous line's readers of the stages are done */
    if (!producer && (PH == PH_ALL || PH == PH_RUN))
        for (int t = lane; t < BCAST<T, NV>; t += 32) bcall[t] = T(0);
    __syncwarp();

    /* copy size of chunk c of a chain of length ln, rounded up to 4 cells
     * (16-byte multiple); the extra cells stay inside the line's range */
    auto cells = [&](int ln, int c) { return ((min(P, ln - c * P) + 3) & ~3); };
    auto issue = [&](int job, int s, bool blocks = true, bool vecs = true) {
        unsigned char *base = st0 + (size_t)s * stage;
        uint32_t bytes = 0;
        if (job < nf) {
            const int c = job;
            if (c < nchT) bytes += cells(m, c) * (NB + NV) * sizeof(T);
            if (c < nchB) bytes += cells(nb, c) * (NB + NV) * sizeof(T);
        } else {
            const int jb = job - nf, bw = NB + (stage_u ? NV : 0);
            if (nchT - 1 - jb >= 0) bytes += cells(m, nchT - 1 - jb) * bw * sizeof(T);
            if (nchB - 1 - jb >= 0) bytes += cells(nb, nchB - 1 - jb) * bw * sizeof(T);
        }
        if (blocks) mbar_arrive_expect_tx(&bars[s], bytes);
        for (int hh = 0; hh < 2; ++hh) {
            const int ln = hh ? nb : m, nc = hh ? nchB : nchT, cp = hh ? m : 0;
            unsigned char *hb = base + hh * half;
            if (job < nf) {
                const int c = job;
                if (c >= nc) continue;
                const int cnt = cells(ln, c);
                if (blocks)
                    bulk_g2s_hint(hb, G + (size_t)(ps + cp + c * P) * NB, cnt * NB * sizeof(T), &bars[s], pol);
                if (vecs)
                    bulk_g2s(hb + P * NB * sizeof(T), b + (size_t)(ps + cp + c * P) * NV, cnt * NV * sizeof(T),
                             &bars[s]);
            } else if (blocks) {
                const int c = nc - 1 - (job - nf);
                if (c < 0) continue;
                const int cnt = cells(ln, c);
                bulk_g2s_hint(hb, Gam + (size_t)(ps + cp + c * P) * NB, cnt * NB * sizeof(T), &bars[s], pol);
                if (stage_u)
                    bulk_g2s(hb + P * NB * sizeof(T), Uil + (size_t)(cp + c * P) * NV, cnt * NV * sizeof(T),
                             &bars[s]);
            }
        }
    };
    /* Each full barrier completes one phase per job landed in its stage,
     * each empty barrier one per job consumed from it: `pbase` gives the
     * parity of the first of them (carried across lines by a persistent
     * CTA), RingPos the rest, without divisions */
    struct RingPos {
        int s = 0;
        uint32_t wrap = 0;
        __device__ void next(int NS) {
            if (++s == NS) {
                s = 0;
                wrap ^= 1u;
            }
        }
    };
    auto parity = [&](const RingPos &r) { return ((pbase >> r.s) ^ r.wrap) & 1u; };
    /* after the line, every job was waited for: barrier s completed one
     * phase per job j = s, s+NS, ... below njobs */
    auto close_phases = [&]() {
        for (int s = 0; s < NS && s < njobs; ++s) {
            const int cnt = (njobs - 1 - s) / NS + 1;
            pbase ^= (uint32_t)(cnt & 1) << s;
        }
    };
    /* YS: U += x by the loads and stores of the warps (FP32, or U read from
     * another buffer) waits for a round of loads after another: both warps of
     * a line share it (600x640 FP32: a line solve of 82 us with the chain
     * warp alone and 8 loads a lane in flight, 78) */
    const bool share = WS && YS && PH == PH_ALL && accumulate == 1 && !(sizeof(T) == 8 && !Uin);
    auto add_to_u = [&](int first, int w, int warps) {
        constexpr int B = 16;
        const int nv = n * NV, nbulk = (n & ~3) * NV;
        for (int t0 = first + w * 32 + lane; t0 < nv; t0 += 32 * warps * B) {
            T u[B];
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const int t = t0 + 32 * warps * k;
                u[k] = (accumulate == 1 && t < nv) ? __ldcg(Uil + t) : T(0);
            }
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const int t = t0 + 32 * warps * k;
                if (t < nv) {
                    const T x = ys[t];
                    if (t >= nbulk) dUl[t] = x;
                    if (accumulate < 2) Ul[t] = u[k] + x;
                }
            }
        }
    };
    if (producer) {
        /* every job as soon as the consumer has released its stage: job
         * j >= NS waits for the consumption of job j - NS */
        if (PH == PH_BLOCKS || PH == PH_VECS || PH == PH_DROP) {
            if (lane == 0)
                for (int job = 0; job < NS && job < njobs; ++job) {
                    if (PH == PH_DROP)
                        mbar_wait(&bars[job], (pbase >> job) & 1u, 1LL << 28);
                    else
                        issue(job, job, PH == PH_BLOCKS, PH == PH_VECS);
                }
            return true;
        }
        if (lane == 0) {
            RingPos r, e; /* e: the consumed job's place, NS jobs behind */
            for (int job = 0; job < njobs; ++job) {
                if (*ws_abort) break;
                if (job >= NS) {
                    if (!mbar_wait(&empty[e.s], parity(e))) {
                        atomicOr(status, ST_TIMEOUT);
                        break;
                    }
                    e.next(NS);
                }
                if (PH == PH_ALL || job >= NS) issue(job, r.s);
                r.next(NS);
                *ws_issued = job + 1;
            }
        }
        __syncwarp();
        if (share) {
            ws_meet(); /* x is in ys, or the chains have given up */
            if (*ws_abort) return true;
            add_to_u(0, 1, 2);
        }
        ws_meet();
        close_phases();
        return true;
    }
    int issued = 0;
    if (!WS && lane == 0) {
        for (; issued < NS && issued < njobs; ++issued) issue(issued, issued);
    }
    int consumed = 0; /* jobs waited for */
    bool timed_out = false;
    const int both_full = (m < nb ? m : nb) / P; /* jobs where both chains run P steps */
    /* y, written by the forward chains and read once by the backward ones */
    const uint64_t ypol_last = YS ? 0ull : policy_evict_last();
    const uint64_t ypol_first = YS ? 0ull : policy_evict_first();

    RingPos rd; /* the next job to wait for */
    bool landed = false;
    auto probe = [&]() { landed = mbar_test(&bars[rd.s], parity(rd)); };
    /* the next job's stage (this half's part of it), waited for when probe()
     * did not find it landed; null when the wait ran out of time */
    auto take = [&]() -> const T * {
        const T *p = reinterpret_cast<const T *>(st0 + (size_t)rd.s * stage + h * half);
        if (__any_sync(0xffffffffu, !landed)) {
            if (__any_sync(0xffffffffu, !mbar_wait(&bars[rd.s], parity(rd)))) {
                timed_out = true;
                return nullptr;
            }
        }
        ++consumed;
        rd.next(NS);
        return p;
    };
    /* the stage of the chunk just finished may be refilled */
    int rel = 0;
    auto release = [&]() {
        if (WS) {
            mbar_arrive_if(&empty[rel], lane == 0);
        } else if (lane == 0 && issued < njobs) {
            issue(issued, rel);
            ++issued;
        }
        if (++rel == NS) rel = 0;
    };

    /* ---------------- forward */
    const T *sG = nullptr, *sN = nullptr;
    Row<T, NV> row;
    T bi = T(0);
    if (nf > 0) {
        sG = take();
        if (sG) {
            load_row(row, sG, i, 0);
            bi = sG[P * NB + i];
        }
    }
    for (int c = 0; c < nf && !timed_out; ++c) {
        auto next = [&]() -> const T * { return sN = (c + 1 < nf ? take() : nullptr); };
        if (c < both_full)
            fwd_chunk<T, NV, P, false, YS>(sG, row, bi, bc, ys, yl, c * P, len, m > nb ? m : nb, cpos, i, ypol_last, probe,
                                       next);
        else
            fwd_chunk<T, NV, P, true, YS>(sG, row, bi, bc, ys, yl, c * P, len, m > nb ? m : nb, cpos, i, ypol_last, probe,
                                      next);
        release();
        sG = sN;
    }

    if (!timed_out) {
        /* ---------------- twist: x_m = b_m - G_tw y_top - Gam_tw y_bot */
        const int ptw = n - 1; /* relative to ps */
        const T *ytop = bcall + (m & 1) * VB;
        const T *ybot = bcall + (2 + (nb & 1)) * VB;
        T xm = T(0);
        if (lane < NV) {
            const T *gr = G + (size_t)(ps + ptw) * NB + lane;
            const T *cr = Gam + (size_t)(ps + ptw) * NB + lane;
            T acc = __ldcg(b + (size_t)(ps + ptw) * NV + lane);
#pragma unroll
            for (int j = 0; j < NV; ++j) acc -= fma_rn(gr[NV * j], ytop[j], mul_rn(cr[NV * j], ybot[j]));
            xm = acc;
        }
        __syncwarp();
        if (lane < NV) {
            for (int t = 0; t < 4; ++t) StepVec<T, NV>::put(bcall + t * VB, lane, xm);
            if (YS)
                ys[ptw * NV + lane] = xm;
            else {
                dUl[(size_t)ptw * NV + lane] = xm;
                if (accumulate < 2)
                    Ul[(size_t)ptw * NV + lane] = (accumulate ? Uil[(size_t)ptw * NV + lane] : T(0)) + xm;
            }
        }
        __syncwarp();

        /* ---------------- backward */
        T yv[P], uv[P], nyv[P], nuv[P];
        auto load_chunk = [&](int c, T *yy, T *uu) {
#pragma unroll
            for (int q = 0; q < P; ++q) {
                const int k = c * P + q;
                yy[q] = T(0);
                uu[q] = T(0);
                if (!YS && c >= 0 && k < len) { /* lanes 9..15: lane 8's values */
                    yy[q] = ld_hint(yl + (size_t)(cpos + k) * NV + i, ypol_first);
                    if (accumulate == 1 && !stage_u) uu[q] = Uil[(size_t)(cpos + k) * NV + i];
                }
            }
        };
        if (!YS) load_chunk(nch - 1, yv, uv);
        T yk = T(0);
        if (nf > 0) {
            probe();
            sG = take();
            if (sG) load_row(row, sG + (P - 1) * NB, i, (P - 1) & 1);
            const int k = nch * P - 1;
            if (YS && k >= 0 && k < len) yk = ys[(cpos + k) * NV + i];
        }
        for (int jb = 0; jb < nf && !timed_out; ++jb) {
            const int c = nch - 1 - jb; /* this half's chunk (may be < 0) */
            if (!YS) load_chunk(c - 1, nyv, nuv);
            const bool full = (nchT - 1 - jb) * P + P <= m && (nchB - 1 - jb) * P + P <= nb &&
                              nchT - 1 - jb >= 0 && nchB - 1 - jb >= 0;
            const T *sU = stage_u ? sG + P * NB : nullptr;
            T *Uw = accumulate < 2 ? Ul : nullptr;
            auto next = [&]() -> const T * { return sN = (jb + 1 < nf ? take() : nullptr); };
            if (full)
                bwd_chunk<T, NV, P, false, YS>(sG, row, yk, bc, ys, yv, uv, dUl, Uw, c * P, len, cpos, i, sU,
                                           probe, next);
            else
                bwd_chunk<T, NV, P, true, YS>(sG, row, yk, bc, ys, yv, uv, dUl, Uw, c * P, len, cpos, i, sU,
                                          probe, next);
            release();
            sG = sN;
            if (!YS) {
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    yv[q] = nyv[q];
                    uv[q] = nuv[q];
                }
            }
        }
        if (YS && !timed_out) {
            /* dU = x (and U = x or U += x) for the line's n cells.  The whole
             * groups of 4 cells (16-byte multiples) of dU go by one bulk
             * copy, and in FP64 those of U by one bulk add (U + x rounded
             * once, as the loop would); what is left, and the forms that
             * read another buffer, by the loop, whose U loads of a batch are
             * issued together so that their latencies overlap */
            const int nbulk = (n & ~3) * NV;
            const bool ub = accumulate == 0 || (accumulate == 1 && sizeof(T) == 8 && !Uin);
            fence_async_smem();
            __syncwarp();
            if (lane == 0 && nbulk > 0) {
                bulk_s2g(dUl, ys, nbulk * sizeof(T));
                if (drain) {
                    bulk_s2g_commit();
                    /* an earlier line's add to U is complete: the older group */
                    bulk_s2g_wait_but<1>();
                }
                if (accumulate == 0) bulk_s2g(Ul, ys, nbulk * sizeof(T));
                if (accumulate == 1 && ub) bulk_add_s2g(Ul, ys, nbulk * sizeof(T));
                bulk_s2g_commit();
            }
            if (share) ws_meet();
            add_to_u(accumulate < 2 && !ub ? 0 : nbulk, 0, share ? 2 : 1);
            if (lane == 0 && nbulk > 0) {
                if (drain) bulk_s2g_wait_but<1>(); /* dU */
                bulk_s2g_wait_read(); /* before the CTA's memory goes */
            }
            __syncwarp();
        }
    }
    if (timed_out) {
        if (WS) {
            /* stop the producer (its own waits are bounded), then wait for
             * the copies it issued */
            if (lane == 0) *ws_abort = 1;
            __syncwarp();
            ws_meet();
            issued = *ws_issued;
        }
        if (lane == 0) {
            atomicOr(status, ST_TIMEOUT);
            RingPos r = rd;
            for (int job = consumed; job < issued; ++job) {
                mbar_wait(&bars[r.s], parity(r), 1LL << 28);
                r.next(NS);
            }
        }
        __syncwarp();
        return false;
    }
    if (WS) ws_meet();
    close_phases();
    return true;
}

__device__ __forceinline__ void thomas_init_bars(unsigned char *smem, int NS) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    if ((threadIdx.x & 31) == 0) {
        for (int s = 0; s < NS; ++s) mbar_init(&bars[s], 1);
        mbar_fence_init();
    }
    __syncwarp();
}

/* the staging barriers of a warp-specialised CTA (thread 0; the CTA's barrier
 * follows) */
__device__ __forceinline__ void thomas_init_ws(unsigned char *smem, int NS) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    for (int s = 0; s < NS; ++s) {
        mbar_init(&bars[s], 1);
        mbar_init(&bars[8 + s], 1);
    }
    int *cnt = reinterpret_cast<int *>(smem + 128);
    cnt[0] = 0;
    cnt[1] = 0;
    mbar_fence_init();
}

}  // namespace tbs

#endif /* TBS_THOMAS_CUH */
