// k_sweep.cu — fused implicit line sweeps of the ADI step.
//
// A line's sweep does what the reference spreads over five kernels and global scratch
// (UZSolver_calculate_preindex/_abcd/_matrix_coeff, tridiagSolver,
// UZSolver_extract_solution, UVZSolver_multithread.cu:881-943 and the VZ twins 818-879;
// Scan_FS*/tridiagSolver/FS*_extract_solution, Sediment_Transport.cu:570-617).
// Only the wet segments of the line are touched: their cells and their tridiagonal rows
// are packed one segment after another, so a line with a few wet cells costs a few rows
// however long it is.
//   A  continuity coefficients a2, c2, d2 of every wet cell (those of the segment ends
//      kept for D)
//   B  momentum coefficients and the interleaved rows of every segment's system
//   C  all segments of the line solved as one block-decoupled tridiagonal system by a
//      partitioned method: each thread eliminates a chunk of rows, the chunk-end
//      unknowns are solved by parallel cyclic reduction, each thread substitutes back
//      (replaces the reference's serial Thomas sweep, UVZSolver_multithread.cu:203-228)
//   D  the solution scattered to t_z / t_u (t_v) with the reference's boundary formulas.
//
// One persistent kernel per sweep: a 512-thread CTA per SM takes every G-th line, 16 at a time,
// one warp setting up each.  The lines are then swept side by side by teams of warps, a
// team's share of the 16 warps by its line's rows, as many lines at once as their rows fit
// the shared memory (a global scratch region per CTA for a line that does not fit at all).
// How a line is solved depends on its rows alone, not on its team: up to about 480 rows 32
// chunks eliminated by one warp whose chunk ends are solved by shuffle-only cyclic reduction,
// beyond that a level more (up to 256 chunks, then one warp on the chunk-end system as
// above); so a line's values are the same bits in every launch shape.
// In the column sweeps the cell-local coefficients come precomputed, stored column-major
// so that a column reads them contiguously (k_coef_bnd<0>, k_coef_fsj).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "hydist_dev.cuh"

namespace {

constexpr int kTL = 512;         // threads of a sweep CTA
constexpr int kWL = kTL / 32;    // lines per group (one warp sets up each)
// Shared memory asked for beyond the longest line: `wide`, room for every line of a group with
// up to kRowW rows side by side; else up to kRowSlice rows (more of the SM's on-chip memory
// left to L1).
constexpr int kRowW = 288;
constexpr int kRowSlice = 96;
// continuity coefficients (a, c, d) of the first and last cell of every segment of a
// hydrodynamic line, kept for the extraction: 6 values per segment
constexpr int kEnds = 6 * HYD_SEGL;

// A warp's threads setting up a line.  exchange() gives lane t the values v of lanes t - h (lo)
// and t + h (hi).
struct WarpG {
    static constexpr int size = 32;
    __device__ static __forceinline__ int rank() { return threadIdx.x & 31; }
    __device__ static __forceinline__ void sync() { __syncwarp(); }
    template <class R>
    __device__ static __forceinline__ void exchange(const R (&v)[6], int h, R (&lo)[6], R (&hi)[6]) {
#pragma unroll
        for (int k = 0; k < 6; k++) {
            lo[k] = __shfl_up_sync(0xffffffffu, v[k], h);
            hi[k] = __shfl_down_sync(0xffffffffu, v[k], h);
        }
    }
};

// The threads that sweep one line: a warp by itself, or a team.
struct WarpTeam {
    static constexpr int size = 32;
    const int rank = threadIdx.x & 31;
    __device__ __forceinline__ void sync() const { __syncwarp(); }
};

// The warps [first, first + size / 32) of the CTA sweeping one line.  Teams of several warps
// meet at a hardware barrier of their own (1 + first / 2: two teams of two warps or more start
// at least two warps apart; barrier 0 is the CTA's).
struct Team {
    int size, rank, bar;
    __device__ __forceinline__ Team(int first, int warps)
        : size(32 * warps), rank((int)threadIdx.x - 32 * first), bar(1 + first / 2) {}
    __device__ __forceinline__ void sync() const {
        if (size == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(size) : "memory");
    }
};

// Chunk length for R rows over T threads: at least 3 and odd (odd strides keep the
// chunk-strided shared-memory accesses free of bank conflicts).
__host__ __device__ inline int chunk_len(int R, int T) {
    int m = (int)((unsigned)(R + T - 1) / (unsigned)T);
    if (m < 3) m = 3;
    if ((m & 1) == 0) m++;
    return m;
}

// Partitioned tridiagonal solve.  Row r: A[r] x[r-1] + B[r] x[r] + C[r] x[r+1] = D[r];
// A[0] and C[last] are ignored.  Thread t owns the chunk of rows [t*m, t*m+m) (m >= 3).
//
// chunk_reduce: downward elimination inside the chunk (x_i + c'_i x_{i+1} + a'_i x_s =
// d'_i), then upward (x_i = d''_i - a''_i x_s - c''_i x_e for s < i < e), leaving the two
// chunk-end rows of the reduced system on the chunk-end unknowns, ordered (x_s, x_e)
// chunk after chunk and scaled to a unit diagonal: row 2t is (v[0], 1, v[1] | v[2]), row
// 2t+1 is (v[3], 1, v[4] | v[5]) as (lower, diagonal, upper | right-hand side).
// Every solver function is a template on the arithmetic type R: double for the FP64 form,
// float for the mixed form (the FP64 instantiation is the same code with R = double).
template <class R>
__device__ __forceinline__ void chunk_reduce(R* A, R* B, R* C, R* D, int s, int e, R (&v)[6]) {
    {
        int i = s + 1;
        R r = R(1) / B[i];
        R cp = C[i] * r, dp = D[i] * r, ap = A[i] * r;
        A[i] = ap;
        C[i] = cp;
        D[i] = dp;
        for (i = s + 2; i <= e; i++) {
            const R ai = A[i];
            r = R(1) / (B[i] - ai * cp);
            cp = C[i] * r;
            dp = (D[i] - ai * dp) * r;
            ap = -(ai * ap) * r;
            A[i] = ap;
            C[i] = cp;
            D[i] = dp;
        }
    }
    {
        R an = A[e - 1], cn = C[e - 1], dn = D[e - 1];
        for (int i = e - 2; i >= s + 1; i--) {
            const R ci = C[i];
            dn = D[i] - ci * dn;
            an = A[i] - ci * an;
            cn = -ci * cn;
            A[i] = an;
            C[i] = cn;
            D[i] = dn;
        }
    }
    const R cs = C[s];
    const R ib = R(1) / (B[s] - cs * A[s + 1]);
    v[0] = A[s] * ib;
    v[1] = -cs * C[s + 1] * ib;
    v[2] = (D[s] - cs * D[s + 1]) * ib;
    v[3] = A[e];
    v[4] = C[e];
    v[5] = D[e];
}

// The chunk's inner unknowns from its end values; x goes to B.
template <class R>
__device__ __forceinline__ void chunk_back(R* A, R* B, R* C, R* D, int s, int e, R xs, R xe) {
    for (int i = s + 1; i < e; i++) B[i] = D[i] - A[i] * xs - C[i] * xe;
    B[s] = xs;
    B[e] = xe;
}

// Parallel cyclic reduction of the 64-row reduced system of a warp (two unit-diagonal
// rows per lane, in registers, exchanged by shuffles): at distance d row r eliminates rows
// r - d and r + d, every row rescaled to a unit diagonal (one reciprocal per row and
// level).  On return v[2] = x_s and v[5] = x_e of the lane's chunk.
template <class R>
__device__ __forceinline__ void pcr_warp(R (&v)[6]) {
    constexpr int T = 32, n = 2 * T;
    const int t = threadIdx.x & 31;
    for (int d = 1; d < n; d <<= 1) {
        R lo[6], hi[6];
        const int h = d == 1 ? 1 : d >> 1;
        WarpG::exchange(v, h, lo, hi);
        R la[2], lc[2], ld[2], ha[2], hc[2], hd[2];
        bool lv[2], hv[2];
        if (d == 1) {
            // row 2t: lo = row 2t-1 (lane t-1, second row), hi = row 2t+1 (own second row)
            la[0] = lo[3]; lc[0] = lo[4]; ld[0] = lo[5]; lv[0] = t >= 1;
            ha[0] = v[3]; hc[0] = v[4]; hd[0] = v[5]; hv[0] = true;
            // row 2t+1: lo = row 2t (own first row), hi = row 2t+2 (lane t+1, first row)
            la[1] = v[0]; lc[1] = v[1]; ld[1] = v[2]; lv[1] = true;
            ha[1] = hi[0]; hc[1] = hi[1]; hd[1] = hi[2]; hv[1] = t + 1 < T;
        } else {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                la[q] = lo[3 * q]; lc[q] = lo[3 * q + 1]; ld[q] = lo[3 * q + 2]; lv[q] = t - h >= 0;
                ha[q] = hi[3 * q]; hc[q] = hi[3 * q + 1]; hd[q] = hi[3 * q + 2]; hv[q] = t + h < T;
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const R a = v[3 * q], c = v[3 * q + 1];
            R nA = R(0), nC = R(0), nB = R(1), nD = v[3 * q + 2];
            if (lv[q]) {
                nA = -la[q] * a;
                nB -= lc[q] * a;
                nD -= ld[q] * a;
            }
            if (hv[q]) {
                nC = -hc[q] * c;
                nB -= ha[q] * c;
                nD -= hd[q] * c;
            }
            const R ib = R(1) / nB;
            v[3 * q] = nA * ib;
            v[3 * q + 1] = nC * ib;
            v[3 * q + 2] = nD * ib;
        }
    }
}

// One warp: rows [0, 32 m), chunks of m rows per lane, the reduced system by pcr_warp.
// On return B[r] holds x[r].
template <class R>
__device__ __forceinline__ void solve_warp(R* A, R* B, R* C, R* D, int m) {
    const int t = threadIdx.x & 31;
    const int s = t * m, e = s + m - 1;
    R v[6];
    chunk_reduce(A, B, C, D, s, e, v);
    pcr_warp(v);
    chunk_back(A, B, C, D, s, e, v[2], v[5]);
    __syncwarp();
}

// How R rows are solved: t1 chunks of m rows.  t1 == 32: one warp (solve_warp).  t1 > 32: two
// levels (solve_two): the 2 t1 chunk-end rows form a tridiagonal system that one warp solves
// in chunks of m2 = chunk_len(2 t1, 32) rows.  The plan minimises the serial depth, about
// 3 m + 6 for one warp and 3 m + 3 m2 + 10 for two levels (their two barriers counted as two
// steps each).
struct SolvePlan {
    int t1, m;
    __host__ __device__ int rows() const { return t1 * m; }                                   // padded
    __host__ __device__ int red() const { return t1 > 32 ? 32 * chunk_len(2 * t1, 32) : 0; }  // reduced rows
};
constexpr int kRedRows = 32 * 17;  // reduced rows of the largest two-level plan (t1 = 256)
__host__ __device__ inline SolvePlan solve_plan(int R, int max_t1) {
    SolvePlan best{32, chunk_len(R, 32)};
    int depth = 3 * best.m + 6;
#pragma unroll
    for (int t1 = 64; t1 <= 256; t1 <<= 1) {  // unrolled: the divisions become shifts
        if (t1 > max_t1) break;
        const int m1 = chunk_len(R, t1), m2 = chunk_len(2 * t1, 32);
        const int d = 3 * m1 + 3 * m2 + 10;
        if (d < depth) {
            depth = d;
            best = SolvePlan{t1, m1};
        }
    }
    return best;
}

// Two-level solve by a team (rows [0, t1 m)); red holds 4 red() values.  Every thread of the
// team calls it.  On return B[r] holds x[r].
template <class R, class TM>
__device__ __forceinline__ void solve_two(R* A, R* B, R* C, R* D, SolvePlan pl, R* red, const TM& tm) {
    const int nr = pl.red();
    R *rA = red, *rB = red + nr, *rC = red + 2 * nr, *rD = red + 3 * nr;
    for (int t = tm.rank; t < pl.t1; t += tm.size) {
        const int s = t * pl.m, e = s + pl.m - 1;
        R v[6];
        chunk_reduce(A, B, C, D, s, e, v);
        rA[2 * t] = v[0];
        rB[2 * t] = R(1);
        rC[2 * t] = v[1];
        rD[2 * t] = v[2];
        rA[2 * t + 1] = v[3];
        rB[2 * t + 1] = R(1);
        rC[2 * t + 1] = v[4];
        rD[2 * t + 1] = v[5];
    }
    for (int r = 2 * pl.t1 + tm.rank; r < nr; r += tm.size) {  // identity rows
        rA[r] = R(0);
        rB[r] = R(1);
        rC[r] = R(0);
        rD[r] = R(0);
    }
    tm.sync();
    if (tm.rank < 32) solve_warp(rA, rB, rC, rD, nr / 32);
    tm.sync();
    for (int t = tm.rank; t < pl.t1; t += tm.size) {
        const int s = t * pl.m, e = s + pl.m - 1;
        chunk_back(A, B, C, D, s, e, rB[2 * t], rB[2 * t + 1]);
    }
    tm.sync();
}

// Serial Thomas over the packed rows by the team's first thread, in the reference's
// operation order (tridiag, UVZSolver_multithread.cu:203-228); decoupled segments solve
// exactly as separate systems.  Used to check the partitioned solver.
template <class R, class TM>
__device__ __forceinline__ void solve_thomas(R* A, R* B, R* C, R* D, int rows, const TM& tm) {
    if (tm.rank == 0 && rows > 0) {
        R Ap = -C[0] / B[0], Bp = D[0] / B[0];
        C[0] = Ap;
        D[0] = Bp;
        for (int i = 1; i < rows; i++) {
            const R ep = A[i] * Ap + B[i];
            Ap = -C[i] / ep;
            Bp = (D[i] - (A[i] * Bp)) / ep;
            C[i] = Ap;
            D[i] = Bp;
        }
        R x = D[rows - 1];
        B[rows - 1] = x;
        for (int i = rows - 2; i >= 0; i--) {
            x = D[i] + (C[i] * x);
            B[i] = x;
        }
    }
    tm.sync();
}

// Solve of a line's packed system (rows padded with identity rows to pl.rows()) by a team.
template <int SOLVER, class R, class TM>
__device__ __forceinline__ void solve_line(R* A, R* B, R* C, R* D, SolvePlan pl, int rows, R* red, const TM& tm) {
    constexpr bool one = std::is_same<TM, WarpTeam>::value;  // its lines are never long enough for two levels
    if (SOLVER == 0) {
        if (one || pl.t1 == 32) {
            if (tm.rank < 32) solve_warp(A, B, C, D, pl.m);
            if (tm.size > 32) tm.sync();
        } else {
            solve_two(A, B, C, D, pl, red, tm);
        }
    } else {
        solve_thomas(A, B, C, D, rows, tm);
    }
}

struct LineShared {
    int first[HYD_SEGL], last[HYD_SEGL];
    int br1[HYD_SEGL], br2[HYD_SEGL];
    int typeR[HYD_SEGL];     // rows start with continuity (bienrandau) rather than momentum (bienlongdau)
    int sn[HYD_SEGL];        // last row index of the segment's system (the reference's SN)
    int lastKind[HYD_SEGL];  // 0 wall end, 1 discharge end, 2 stage end
    int co[HYD_SEGL + 1];    // packed cell offset of each segment
    int ro[HYD_SEGL + 1];    // packed row offset of each segment
    double tzl[HYD_SEGL], tzr[HYD_SEGL];
    double zl[HYD_SEGL], zr[HYD_SEGL];  // mixed form: z at the segment ends (the increments' base)
    int nseg, R, C;
};

// The segment holding packed cell (seg_of) or packed row (seg_of_row) c: the last s with
// off[s] <= c (binary search over at most 20 offsets).
__device__ __forceinline__ int seg_search(const int* off, int nseg, int c) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int seg_of(const LineShared& sg, int c) { return seg_search(sg.co, sg.nseg, c); }
__device__ __forceinline__ int seg_of_row(const LineShared& sg, int c) { return seg_search(sg.ro, sg.nseg, c); }

// ---- hydrodynamic sweeps ----------------------------------------------------------
// DIR 0: UZ, line = column j, cells i (t_u, ubt/ubp, bienQ[2]/[3]).
// DIR 1: VZ, line = row i, cells j (t_v, vbd/vbt, bienQ[1]/[0]).

// Segments of the line, their system sizes (_calculate_matrix_coeff,
// UVZSolver_multithread.cu:515-592) and packed offsets, into sg.
template <int DIR, class G, bool MIX>
__device__ __forceinline__ void hydro_setup(const DevGrid& g, const DevParams& p, int line, LineShared& sg) {
    const int tid = G::rank();
    const int L = DIR == 0 ? g.N : g.M;
    const int along = DIR == 0 ? g.P : 1;
    const int base = DIR == 0 ? line : line * g.P;
    const int Q1 = DIR == 0 ? g.bienQ[2] : g.bienQ[1];  // dkBienQ_1
    const int Q2 = DIR == 0 ? g.bienQ[3] : g.bienQ[0];  // dkBienQ_2
    const int nseg = DIR == 0 ? g.mocj[line] : g.moci[line];
    if (tid < nseg) {
        const int f = DIR == 0 ? g.dauj[line * HYD_SEGL + tid] : g.daui[line * HYD_SEGL + tid];
        const int l = DIR == 0 ? g.cuoij[line * HYD_SEGL + tid] : g.cuoii[line * HYD_SEGL + tid];
        int b1, b2;
        if (DIR == 0) seg_flags_u(g, p, line, f, l, b1, b2);
        else seg_flags_v(g, p, line, f, l, b1, b2);
        const int Ls = l - f;
        const int tR = b1 || (Q1 && f == 2);
        const int qEnd = Q1 && l == L;
        int sn, kind;
        if (b1) {
            if (!b2) {
                if (Q2 && l == L) { sn = 2 * Ls; kind = 1; }
                else { sn = 2 * Ls - 1; kind = 2; }
            } else { sn = 2 * Ls; kind = 0; }
        } else if (tR) {
            if (!b2) {
                if (qEnd) { sn = 2 * Ls; kind = 1; }
                else { sn = 2 * Ls - 1; kind = 2; }
            } else { sn = 2 * Ls; kind = 0; }
        } else {
            if (!b2) {
                if (qEnd) { sn = 2 * Ls - 1; kind = 1; }
                else { sn = 2 * Ls - 2; kind = 2; }
            } else { sn = 2 * Ls - 1; kind = 0; }
        }
        sg.first[tid] = f;
        sg.last[tid] = l;
        sg.br1[tid] = b1;
        sg.br2[tid] = b2;
        sg.typeR[tid] = tR;
        sg.sn[tid] = sn;
        sg.lastKind[tid] = kind;
        sg.tzl[tid] = g.t_z[base + f * along];
        sg.tzr[tid] = g.t_z[base + l * along];
        if (MIX) {
            sg.zl[tid] = g.z[base + f * along];
            sg.zr[tid] = g.z[base + l * along];
        }
    }
    G::sync();
    if (tid == 0) {
        int c = 0, r = 0;
        for (int s = 0; s < nseg; s++) {
            sg.co[s] = c;
            sg.ro[s] = r;
            c += sg.last[s] - sg.first[s] + 1;
            if (sg.sn[s] >= 0) r += sg.sn[s] + 1;
            else flag_status(g, HYD_ST_DEGENERATE);  // single-cell segment on an open edge
        }
        sg.co[nseg] = c;
        sg.ro[nseg] = r;
        sg.C = c;
        sg.R = r;
        sg.nseg = nseg;
    }
    G::sync();
}

// Phases A-D of one line by a team.  Rows A, B, Cc, D hold at least pl.rows() entries, ends
// kEnds; red: the two-level solve's reduced rows.
// R = float: the mixed form.  Its coefficients (k_coef_bnd's FP32 arrays) are those of the
// level increment dz = z' - z: the continuity right-hand side d2 - z and the momentum
// f5 - f4 (z_k - z_k+1), so that the same rows solve for (dz, u) in FP32; the prescribed
// levels enter as increments, and the new level is z + dz in FP64.
template <int DIR, int SOLVER, class R, class TM>
__device__ __forceinline__ void hydro_body(const DevGrid& g, const DevParams& p, int line, const LineShared& sg,
                                           R* A, R* B, R* Cc, R* D, R* ends, R* red, SolvePlan pl, const TM& tm) {
    constexpr bool MIX = sizeof(R) == sizeof(float);
    const int T = tm.size;
    const int tid = tm.rank;
    const int N = g.N, M = g.M, P = g.P;
    const int L = DIR == 0 ? N : M;
    (void)M;
    const int along = DIR == 0 ? P : 1;  // offset to the next cell of the line
    const int base = DIR == 0 ? line : line * P;
    double* tvel = DIR == 0 ? g.t_u : g.t_v;
    const R bq_first = R(DIR == 0 ? g.ubt[line] : g.vbd[line]);  // ubt_or_vbd
    const R bq_last = R(DIR == 0 ? g.ubp[line] : g.vbt[line]);   // ubp_or_vbt
    const int nseg = sg.nseg;
    const int C = sg.C, Rn = sg.R;

    // ---- A + B1, one pass over the cells: the continuity coefficients of the cell and of
    // the next one (preindex, UVZSolver_multithread.cu:402-406 / 345-349), the momentum
    // coefficients (preindex f1..f5, _calculate_abcd 409-466) and the rows.  The continuity
    // coefficients of each segment's first and last cell are kept for the extraction.
    auto cont = [&](int k, R& a, R& c, R& d) {
        if (DIR == 0) {
            const size_t t = (size_t)line * g.LT + k;  // precomputed by k_coef_bnd<0>
            a = colTr<R>(g, 0)[t];
            c = colTr<R>(g, 1)[t];
            d = colTr<R>(g, 2)[t];
        } else {
            const int pos = base + k * along;  // precomputed by k_coef_bnd<1>
            a = rowCr<R>(g, 0)[pos];
            c = rowCr<R>(g, 1)[pos];
            d = rowCr<R>(g, 2)[pos];
        }
    };
    for (int r = Rn + tid; r < pl.rows(); r += T) {  // identity rows up to the solver's rows
        A[r] = R(0);
        B[r] = R(1);
        Cc[r] = R(0);
        D[r] = R(0);
    }
    const R f4 = R(DIR == 0 ? 2 * p.g * p.dTchia2dX : 2 * p.g * p.dTchia2dY);
    for (int c = tid; c < C; c += T) {
        const int sI = seg_of(sg, c);
        const int f = sg.first[sI], l = sg.last[sI];
        const int k = f + (c - sg.co[sI]);
        const int Ls = l - f;
        const int tR = sg.typeR[sI];
        const int b1f = sg.br1[sI], b2f = sg.br2[sI];
        const int sn = sg.sn[sI];
        const int r0 = sg.ro[sI];
        const int rel = 2 * (k - f);  // row 2k relative to the segment's first row 2f
        // every coefficient the cell may need, loaded at once (the next cell's and f1..f5
        // are in bounds even where unused: k + 1 <= L + 1 inside the padded line)
        R ac, cc, dc, an, cn, dn, f1, f2, f3, f5;
        cont(k, ac, cc, dc);
        cont(k + 1, an, cn, dn);
        if (DIR == 0) {
            const size_t t = (size_t)line * g.LT + k;
            f1 = colTr<R>(g, 3)[t];
            f2 = colTr<R>(g, 4)[t];
            f3 = colTr<R>(g, 5)[t];
            f5 = colTr<R>(g, 6)[t];
        } else {
            const int pos = base + k * along;
            f1 = rowCr<R>(g, 3)[pos];
            f2 = rowCr<R>(g, 4)[pos];
            f3 = rowCr<R>(g, 5)[pos];
            f5 = rowCr<R>(g, 6)[pos];
        }
        if (k == f) {
            ends[6 * sI] = ac;
            ends[6 * sI + 1] = cc;
            ends[6 * sI + 2] = dc;
        }
        if (k == l) {
            ends[6 * sI + 3] = ac;
            ends[6 * sI + 4] = cc;
            ends[6 * sI + 5] = dc;
        }
        if (tR && rel <= sn) {
            A[r0 + rel] = ac;
            B[r0 + rel] = R(1);
            Cc[r0 + rel] = cc;
            D[r0 + rel] = dc;
        }
        if (k == l) continue;
        if (Ls <= 1 && k != f) continue;
        const int rm = tR ? rel + 1 : rel;  // the momentum row of this cell
        if (rm > sn) continue;
        R ra, rb, rc, rd;
        if (Ls >= 2) {
            if (k == f && b1f) {
                ra = f4;
                rb = f2 - (f3 * an / cn);
                rc = -f4 - (f3 / cn);
                rd = f5 - (f3 * dn / cn);
            } else if (k == l - 1 && b2f) {
                ra = f4 - f1 / ac;
                rb = f2 - (f1 * cc / ac);
                rc = -f4;
                rd = f5 - (f1 * dc / ac);
            } else {
                ra = f4 - f1 / ac;
                rc = -f4 - (f3 / cn);
                rb = f2 - (f1 * cc / ac) - (f3 * an / cn);
                rd = f5 - (f1 * dc / ac) - (f3 * dn / cn);
            }
        } else {
            ra = f4;
            rb = f2;
            rd = f5;
            rc = -f4;
        }
        A[r0 + rm] = ra;
        B[r0 + rm] = rb;
        Cc[r0 + rm] = rc;
        D[r0 + rm] = rd;
        if (!tR && rel + 1 <= sn) {
            A[r0 + rel + 1] = an;
            B[r0 + rel + 1] = R(1);
            Cc[r0 + rel + 1] = cn;
            D[r0 + rel + 1] = dn;
        }
    }
    tm.sync();

    // ---- B2: segment end rows (_calculate_matrix_coeff 469-592) and decoupling
    if (tid < nseg && sg.sn[tid] >= 0) {
        const int sn = sg.sn[tid];
        const int rowF = sg.ro[tid], rowL = rowF + sn;
        const R oA = A[rowL], oB = B[rowL], oC = Cc[rowL], oD = D[rowL];
        // the prescribed end levels (increments over z in the mixed form)
        const R tzl = MIX ? R(sg.tzl[tid] - sg.zl[tid]) : R(sg.tzl[tid]);
        const R tzr = MIX ? R(sg.tzr[tid] - sg.zr[tid]) : R(sg.tzr[tid]);
        if (!sg.br1[tid]) {
            if (sg.typeR[tid]) D[rowF] = D[rowF] - A[rowF] * bq_first;
            else D[rowF] = D[rowF] - A[rowF] * tzl;
        }
        // the end-row statement always rewrites AA, BB, DD of the last row; for a
        // single-row system that undoes the first-row override (UVZSolver_multithread.cu:574-590)
        A[rowL] = oA;
        B[rowL] = oB;
        const int kind = sg.lastKind[tid];
        if (kind == 1) D[rowL] = oD - oC * bq_last;
        else if (kind == 2) D[rowL] = oD - oC * tzr;
        else D[rowL] = oD;
        A[rowF] = R(0);
        Cc[rowL] = R(0);
    }
    tm.sync();

    // ---- C: solve
    solve_line<SOLVER, R>(A, B, Cc, D, pl, Rn, red, tm);

    // ---- D: extract (_uzSolver_extract_solution 668-723 / _vzSolver_extract_solution 595-665)
    const R* x = B;
    // a solved level: the unknown itself, or z + the increment in FP64 (mixed form); a
    // prescribed level as the rows use it
    auto put_z = [&](int pos, R xz) { g.t_z[pos] = MIX ? g.z[pos] + (double)xz : (double)xz; };
    auto row_z = [&](int pos) { return MIX ? R(g.t_z[pos] - g.z[pos]) : R(g.t_z[pos]); };
    const int QF = DIR == 0 ? g.bienQ[2] : g.bienQ[1];
    const int QL = DIR == 0 ? g.bienQ[3] : g.bienQ[0];
    for (int c = tid; c < C; c += T) {
        const int sI = seg_of(sg, c);
        const int f = sg.first[sI], l = sg.last[sI];
        const int k = f + (c - sg.co[sI]);
        const int b1f = sg.br1[sI], b2f = sg.br2[sI];
        const int sn = sg.sn[sI];
        const int r0 = sg.ro[sI] - 2 * f;  // packed index of global row r is r0 + r
        const int qfirst = !b1f && QF && f == 2;
        const int pos = base + k * along;
        if (k < l) {
            if (b1f || qfirst) {
                put_z(pos, x[r0 + 2 * k]);
                tvel[pos] = x[r0 + 2 * k + 1];
                if (k == f) tvel[pos - along] = b1f ? R(0) : bq_first;
            } else if (k == f) {
                const R tv = x[r0 + 2 * f];
                tvel[pos] = tv;
                tvel[pos - along] = (ends[6 * sI + 2] - row_z(pos) - ends[6 * sI + 1] * tv) / ends[6 * sI];
            } else {
                put_z(pos, x[r0 + 2 * k - 1]);
                tvel[pos] = x[r0 + 2 * k];
            }
        } else {
            const R xl = sn >= 0 ? x[r0 + 2 * f + sn] : R(0);
            if (b2f) {
                tvel[pos] = R(0);
                put_z(pos, xl);
            } else if (QL && l == L) {
                tvel[pos] = bq_last;
                put_z(pos, xl);
            } else {
                R tprev;
                if (l > f) tprev = (b1f || qfirst) ? x[r0 + 2 * l - 1] : x[r0 + 2 * l - 2];
                else tprev = R(tvel[pos - along]);
                tvel[pos] = (ends[6 * sI + 5] - ends[6 * sI + 3] * tprev - row_z(pos)) / ends[6 * sI + 4];
            }
        }
    }
}

// The lines a sweep launch covers: lines start .. start + n - 1 of one grid, or the lines of
// every member of a batch in one list (member m's at list positions lstart[m] ..
// lstart[m + 1] - 1, its lines first[m] onwards).
struct OneGridLines {
    DevGrid g;
    DevParams p;
    int start, n;
    __device__ __forceinline__ int count() const { return n; }
    __device__ __forceinline__ void at(int li, int& m, int& line) const {
        m = 0;
        line = start + li;
    }
    __device__ __forceinline__ const DevGrid& grid(int) const { return g; }
    __device__ __forceinline__ const DevParams& params(int) const { return p; }
};

// Which of a group's lines are swept now, and by whom: computed by every warp alike.  Lane l
// of a warp holds the values of shared memory line l's sweep needs.  Of the lines still to do
// (todo), those whose needs added up in order fit `cap` are taken; line l gets warps [start,
// end) of the 16, at least one, the others in proportion to the needs.  (Few instructions and
// few dependent shuffles: this is on every CTA's path, once per 16 lines.)
struct TeamPick {
    unsigned sel;      // lines of this round (0: the first line left does not fit at all)
    int line;          // this warp's line
    int first, warps;  // its team
    int off;           // where the line's region of the shared memory starts
};
__device__ __forceinline__ TeamPick pick_team(unsigned todo, int need, int cap) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool in = (todo >> lane) & 1u;  // todo has no bit beyond the group's kWL lines
    int sum = in ? need : 0;
#pragma unroll
    for (int o = 1; o < kWL; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    TeamPick t;
    t.sel = __ballot_sync(0xffffffffu, in && sum <= cap);
    t.line = t.first = t.warps = t.off = 0;
    if (t.sel == 0) return t;
    const int last = 31 - __clz(t.sel);
    const int total = __shfl_sync(0xffffffffu, sum, last);
    // the spare warps up to this line by the needs up to it; all of them up to the last line
    // (the product is monotone in sum and at most spare, whatever the reciprocal's rounding)
    const int spare = kWL - __popc(t.sel);
    const int share = lane >= last ? spare : min((int)((float)(spare * sum) * __frcp_rn((float)total)), spare);
    int prev = __shfl_up_sync(0xffffffffu, share, 1);
    if (lane == 0) prev = 0;
    const int before = __popc(t.sel & ((1u << lane) - 1u));
    const int start = before + prev, end = before + 1 + share;
    t.line = 31 - __clz(__ballot_sync(0xffffffffu, ((t.sel >> lane) & 1u) && start <= w));
    const int v = __shfl_sync(0xffffffffu, (sum - need) << 10 | end << 5 | start, t.line);
    t.first = v & 31;
    t.warps = ((v >> 5) & 31) - t.first;
    t.off = v >> 10;
    return t;
}

// Fused sweep of one direction.  CTA b takes lines b, b + G, b + 2G, ... (G = gridDim.x)
// in groups of 16; every warp sets a line up, then the group's lines are swept by teams
// (pick_team), in as many rounds as their rows need of the shared memory; when no line has more
// than kRowSlice rows, each by its own warp in a slice of its own (short lines gain nothing
// from more warps, and the picking and the barriers cost them 1 us of 9).  A line of more than
// RB rows, or that does not fit alone, is swept by the whole CTA in its region of global
// scratch.  Adjacent long lines (a wet band) fall on different CTAs.
// Against one warp per short line and then the whole CTA on one long line after another
// (the lines of more than 96 rows of a grid with at most 16 lines per CTA): the 2047 rows of
// about 240 solver rows of a 2048 x 2048 reach 88 -> 29 us (the solve of a line up to 480 rows
// is one warp's, so the other 15 waited), the 99-row lines of a 400 x 60 channel 20 -> 12; one
// long column among short ones, as on a 1048 x 980 reach, 15.1 -> 14.9.
// Warps with nothing to sweep wait at the CTA barriers rather than exit: the
// warp-synchronous steps of a warp whose sibling warps had exited were measured an order of
// magnitude slower on B200.
template <int DIR, int SOLVER, class R, class Lines>
__device__ __forceinline__ void hydro_sweep_loop(const Lines& lines, int cap, int RB, double* gscr_d, int RG) {
    constexpr bool MIX = sizeof(R) == sizeof(float);
    extern __shared__ double dyn_smem_d[];
    R* dyn_smem = reinterpret_cast<R*>(dyn_smem_d);
    __shared__ LineShared sgw[kWL];
    __shared__ int s_mem[kWL], s_line[kWL];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nlines = lines.count();
    const int G = gridDim.x;
    for (int j0 = 0; (int)blockIdx.x + j0 * G < nlines; j0 += kWL) {
        const int li = blockIdx.x + (j0 + w) * G;
        LineShared& sg = sgw[w];
        if (li < nlines) {  // warp-uniform
            int m = 0, line = 0;
            lines.at(li, m, line);
            if (lane == 0) {
                s_mem[w] = m;
                s_line[w] = line;
            }
            hydro_setup<DIR, WarpG, MIX>(lines.grid(m), lines.params(m), line, sg);
        } else if (lane == 0) {
            sg.nseg = sg.R = 0;
        }
        __syncthreads();
        const LineShared& mine = sgw[lane & (kWL - 1)];
        if (!__any_sync(0xffffffffu, mine.R > kRowSlice)) {  // the same in every warp
            if (sg.nseg > 0) {
                R* A = dyn_smem + w * (4 * kRowSlice + kEnds);
                hydro_body<DIR, SOLVER, R>(lines.grid(s_mem[w]), lines.params(s_mem[w]), s_line[w], sg, A, A + kRowSlice,
                                           A + 2 * kRowSlice, A + 3 * kRowSlice, A + 4 * kRowSlice, (R*)nullptr,
                                           SolvePlan{32, chunk_len(sg.R, 32)}, WarpTeam());
            }
            __syncthreads();
            continue;
        }
        const SolvePlan mp = solve_plan(mine.R, SOLVER == 0 ? 256 : 32);
        const int need = 4 * mp.rows() + kEnds + 4 * mp.red() + (mp.rows() > RB ? cap : 0);
        unsigned todo = __ballot_sync(0xffffffffu, lane < kWL && mine.nseg > 0);
        while (todo) {
            TeamPick t = pick_team(todo, need, cap);
            const bool global = t.sel == 0;  // the first line left, by the whole CTA
            if (global) {
                t.line = __ffs(todo) - 1;
                t.sel = 1u << t.line;
                t.warps = kWL;
            }
            const LineShared& sl = sgw[t.line];
            const Team tm(t.first, t.warps);
            const int pv = __shfl_sync(0xffffffffu, mp.m << 10 | mp.t1, t.line);
            const SolvePlan pl{pv & 1023, pv >> 10};
            const int lm = s_mem[t.line], ln = s_line[t.line];
            // two calls, so that the first one's rows are known to be shared memory (through
            // generic addresses the long columns' sweep took 15.6 instead of 14.8 us)
            if (__builtin_expect(!global, 1)) {
                const int P = pl.rows();
                R* A = dyn_smem + t.off;
                R* ends = A + 4 * P;
                hydro_body<DIR, SOLVER, R>(lines.grid(lm), lines.params(lm), ln, sl, A, A + P, A + 2 * P, A + 3 * P, ends,
                                           ends + kEnds, pl, tm);
            } else {
                R* A = reinterpret_cast<R*>(gscr_d) + (size_t)blockIdx.x * (4 * (size_t)RG + kEnds);
                hydro_body<DIR, SOLVER, R>(lines.grid(lm), lines.params(lm), ln, sl, A, A + RG, A + 2 * RG, A + 3 * RG,
                                           A + 4 * RG, dyn_smem, pl, tm);
            }
            todo &= ~t.sel;
            __syncthreads();  // the regions and sgw are reused
        }
    }
}

template <int DIR, int SOLVER, class R>
__global__ void __launch_bounds__(kTL, 1) k_hydro_sweep(DevGrid g, DevParams p, int startidx, int endidx, int cap, int RB,
                                                     double* gscr_d, int RG) {
    hydro_sweep_loop<DIR, SOLVER, R>(OneGridLines{g, p, startidx, endidx - startidx + 1}, cap, RB, gscr_d, RG);
}
template <int DIR, int SOLVER, class R>
__global__ void __launch_bounds__(kTL, 1) k_hydro_sweep_b(BatchLines bl, int cap, int RB, double* gscr_d, int RG) {
    hydro_sweep_loop<DIR, SOLVER, R>(bl, cap, RB, gscr_d, RG);
}

// ---- sediment sweeps --------------------------------------------------------------

// The sediment rows in the arithmetic type R (double: the FP64 form; float: the mixed
// form).  Every operand is read in FP64 and taken to R at its use; the wet/dry tests on
// the depths compare the stored FP64 values, so both forms take the same branches.

// Row of the FSj system for one interior wet cell before the segment-end terms
// (_FSj_calculate__mactrix_coeff, Sediment_Transport.cu:205-302): aa, bb, cc, dd of the row,
// with the source S gated by t < bed_change_start.
template <class R>
__device__ __forceinline__ void fsj_cell_coeffs(const DevGrid& g, const DevParams& p, double t, int pos, R& aa, R& bb,
                                                R& cc, R& dd) {
    const int P = g.P;
    const double* FS = g.FS;
    const double* H = g.H_moi;
    // FSj runs right after the half-step's state update, which left u = t_u and v = t_v
    // on every cell it reads; reading u and v lets it run beside the next half-step's
    // sweeps, which write t_u and t_v
    const double *u = g.u, *v = g.v;
    // every operand first (one memory round trip; the branches below only select)
    const double Hd = H[pos], FSd = FS[pos], VTHd = g.VTH[pos], Fwd = g.Fw[pos];
    const double u0 = u[pos], u1 = u[pos - P], hu0 = g.Htdu[pos], hu1 = g.Htdu[pos - P], kx0 = g.Kx[pos],
                 kx1 = g.Kx[pos - P];
    const double Hm1 = H[pos - 1], Hp2 = H[pos + 2], Hm2 = H[pos - 2], Hp1 = H[pos + 1];
    const double FSp1 = FS[pos + 1], FSm1 = FS[pos - 1];
    const double hv0 = g.Htdv[pos], hv1 = g.Htdv[pos - 1], ky0 = g.Ky[pos], ky1 = g.Ky[pos - 1];
    const double v0 = v[pos], v1 = v[pos - 1];
    const R Hp = R(Hd), FSp = R(FSd), VTHp = R(VTHd);
    const double s_start = p.bed_change_start;
    const R sqrtg = sqrt(R(p.g));
    const R c = 18 * log(12 * Hp / R(p.Ks));
    const R Uf = sqrtg * fabs(VTHp) / c;
    const R fq = 1 - FSp;
    const R wsm = R(p.wss) * ((fq * fq) * (fq * fq));  // wss (1 - FS)^4
    R Zf = 0;
    R S;
    const R gamav = R(0.98) - R(0.198) * Zf + R(0.032) * Zf * Zf;  // evaluated before Zf (Sediment_Transport.cu:236)
    if (FSd > 0.00001) Zf = wsm / (R(0.4) * (Uf + 2 * wsm));
    if (p.ketdinh) S = source_chs<R>(p, wsm, Zf, FSp, R(Fwd), VTHp, Hp);
    else S = source_nchs<R>(p, wsm, Zf, Uf, Hp, FSp);
    if (t < s_start) S = 0;
    aa = -gamav * R(0.5) * (R(u0) + R(u1)) / R(p.dX2) - R(hu1) * R(kx1) / (Hp * (R(p.dXbp)));
    cc = gamav * R(0.5) * (R(u0) + R(u1)) / R(p.dX2) - R(hu0) * R(kx0) / (Hp * (R(p.dXbp)));
    bb = R(p.HaiChiadT) + (R(hu0) * R(kx0) + R(hu1) * R(kx1)) / (Hp * (R(p.dXbp)));
    R pp = 0, qq = 0;
    if ((Hm1 > p.H_TINH) && (Hp2 > p.H_TINH)) pp = R(FSp1 - FSd);
    if ((Hm2 > p.H_TINH) && (Hp1 > p.H_TINH)) qq = R(FSd - FSm1);
    pp = (1 / (Hp * R(p.dYbp))) * (R(hv0) * R(ky0) * pp - R(hv1) * R(ky1) * qq);
    if ((Hm2 > p.H_TINH) && (Hp2 > p.H_TINH)) {
        qq = R(FSp1 - FSm1) / R(p.dY2);
        qq = (R(v0) + R(v1)) * R(0.5) * qq * gamav;
    } else
        qq = 0;
    dd = FSp / (R(p.dT) * R(0.5)) - qq + pp + (S / Hp);
}

// Row of the FSi system for one interior wet cell before the segment-end terms
// (_FSi_calculate__mactrix_coeff, Sediment_Transport.cu:62-165).  The terms that depend on
// the cell alone (gamav and the gated source over the depth, rowC arrays 0 and 1) were
// computed by the state update that precedes the sweep (fsi_cell_terms).
template <class R>
__device__ __forceinline__ void fsi_cell_coeffs(const DevGrid& g, const DevParams& p, int pos, R& aa, R& bb, R& cc,
                                                R& dd) {
    const int P = g.P;
    const double* FS = g.FS;
    const double* H = g.H_moi;
    // every operand first (one memory round trip; the branches below only select)
    const double Hd = H[pos], FSd = FS[pos];
    const R gamav = rowCr<R>(g, 0)[pos], src = rowCr<R>(g, 1)[pos];
    const double tv0 = g.t_v[pos], tv1 = g.t_v[pos - 1], hv0 = g.Htdv[pos], hv1 = g.Htdv[pos - 1], ky0 = g.Ky[pos],
                 ky1 = g.Ky[pos - 1];
    const double Hp2 = H[pos + 2 * P], Hm1 = H[pos - P], Hm2 = H[pos - 2 * P], Hp1 = H[pos + P];
    const double FSp1 = FS[pos + P], FSm1 = FS[pos - P];
    const double hu0 = g.Htdu[pos], hu1 = g.Htdu[pos - P], kx0 = g.Kx[pos], kx1 = g.Kx[pos - P];
    const double tu0 = g.t_u[pos], tu1 = g.t_u[pos - P];
    const R Hp = R(Hd);
    aa = -gamav * R(0.5) * (R(tv1) + R(tv0)) / R(p.dY2) - R(hv1) * R(ky1) / (Hp * R(p.dYbp));
    cc = gamav * R(0.5) * (R(tv1) + R(tv0)) / R(p.dY2) - R(hv0) * R(ky0) / (Hp * R(p.dYbp));
    bb = R(p.HaiChiadT) + (R(hv0) * R(ky0) + R(hv1) * R(ky1)) / (Hp * R(p.dYbp));
    R pp = 0, qq = 0;
    if ((Hp2 > p.H_TINH) && (Hm1 > p.H_TINH)) pp = R(FSp1 - FSd);
    if (Hm2 > p.H_TINH && Hp1 > p.H_TINH) qq = R(FSd - FSm1);
    pp = (1 / (Hp * R(p.dXbp))) * (R(hu0) * R(kx0) * pp - R(hu1) * R(kx1) * qq);
    if (Hp2 > p.H_TINH && Hm2 > p.H_TINH) {
        qq = R(FSp1 - FSm1) / R(p.dX2);
        qq = (R(tu0) + R(tu1)) * R(0.5) * qq * gamav;
    } else
        qq = 0;
    dd = R(FSd) / (R(p.dT) * R(0.5)) - qq + pp + src;
}

// FSj rows of every interior wet cell (columns 3..M-1), wpc warps per row of the grid over
// the row's span (coef_shape), written column-major (colT arrays 0..3 in R: aa bb cc dd), with TILE
// through a tile.
template <int TILE, class R>
__device__ __forceinline__ void coef_fsj_body(const DevGrid& g, const DevParams& p, int half, int wpc, int bx) {
    const double t = g.clock[half];
    if constexpr (!TILE) {
        const RowLane rl(2, wpc, bx);
        const int i = rl.i;
        if (i > g.N) return;
        const int lo = max(g.rlo[i], 3), hi = min(g.rhi[i], g.M - 1);
        for (int j = lo + rl.off; j <= hi; j += rl.stride) {
            const int pos = i * g.P + j;
            if (g.khouot[pos] != 0) continue;
            R aa, bb, cc, dd;
            fsj_cell_coeffs<R>(g, p, t, pos, aa, bb, cc, dd);
            const size_t q = (size_t)j * g.LT + i;
            colTr<R>(g, 0)[q] = aa;
            colTr<R>(g, 1)[q] = bb;
            colTr<R>(g, 2)[q] = cc;
            colTr<R>(g, 3)[q] = dd;
        }
    } else {
        R* const dst[4] = {colTr<R>(g, 0), colTr<R>(g, 1), colTr<R>(g, 2), colTr<R>(g, 3)};
        colmajor_tile<4>(
            g, 2 + kTileRows * bx, g.N, 3, g.M - 1,
            [&](int i, int j, R* v) {
                const int pos = i * g.P + j;
                if (g.khouot[pos] != 0) return false;
                fsj_cell_coeffs<R>(g, p, t, pos, v[0], v[1], v[2], v[3]);
                return true;
            },
            dst);
    }
}

template <int TILE, class R>
__global__ void __launch_bounds__(256) k_coef_fsj(DevGrid g, DevParams p, int half, int wpc) {
    coef_fsj_body<TILE, R>(g, p, half, wpc, blockIdx.x);
}
// Three CTAs per SM, where 89 registers allow two: the batch's 1100 CTAs are one wave less (a
// step of 16 reaches 332 us, now 322; one reach's launch is no faster for it).
template <int TILE, class R>
__global__ void __launch_bounds__(256, 3) k_coef_fsj_b(BatchRef br, int half) {
    const BatchMember bm(br);
    coef_fsj_body<TILE, R>(bm.g, bm.p, half, 1, bm.bx);
}

// Segments of a sediment line and their row offsets (one row per interior cell
// first+1..last-1, the reference's SN+1 rows).
template <int DIR, class G>
__device__ __forceinline__ void fs_setup(const DevGrid& g, const DevParams& p, int line, LineShared& sg) {
    const int tid = G::rank();
    const int nseg = DIR == 0 ? g.mocj[line] : g.moci[line];
    if (tid < nseg) {
        const int f = DIR == 0 ? g.dauj[line * HYD_SEGL + tid] : g.daui[line * HYD_SEGL + tid];
        const int l = DIR == 0 ? g.cuoij[line * HYD_SEGL + tid] : g.cuoii[line * HYD_SEGL + tid];
        int b1, b2;
        if (DIR == 0) seg_flags_u(g, p, line, f, l, b1, b2);
        else seg_flags_v(g, p, line, f, l, b1, b2);
        sg.first[tid] = f;
        sg.last[tid] = l;
        sg.br1[tid] = b1;
        sg.br2[tid] = b2;
    }
    G::sync();
    if (tid == 0) {
        int r = 0;
        for (int s = 0; s < nseg; s++) {
            sg.ro[s] = r;
            const int n = sg.last[s] - sg.first[s] - 1;
            if (n > 0) r += n;
        }
        sg.ro[nseg] = r;
        sg.R = r;
        sg.nseg = nseg;
    }
    G::sync();
}

// Rows, solve and extraction of one sediment line (_FSi/_FSj_calculate__mactrix_coeff
// and _FSi/_FSj_extract_solution, Sediment_Transport.cu:62-340, driven by Scan_FSi/
// Scan_FSj and FSi/FSj_extract_solution 570-618).  DIR 0: FSj (line = column j, cells
// i), DIR 1: FSi (line = row i, cells j).
template <int DIR, int SOLVER, class R, class TM>
__device__ __forceinline__ void fs_body(const DevGrid& g, const DevParams& p, int half, int line,
                                        const LineShared& sg, R* A, R* B, R* Cc, R* D, R* red, SolvePlan pl,
                                        const TM& tm) {
    const int T = tm.size;
    const int tid = tm.rank;
    const int P = g.P;
    const int along = DIR == 0 ? P : 1;
    const int base = DIR == 0 ? line : line * P;
    (void)half;  // both rows are precomputed (k_coef_fsj, the state update's FSi terms)
    const int Rn = sg.R;
    for (int r = Rn + tid; r < pl.rows(); r += T) {  // identity rows up to the solver's rows
        A[r] = R(0);
        B[r] = R(1);
        Cc[r] = R(0);
        D[r] = R(0);
    }
    const double* FS = g.FS;
    for (int rr = tid; rr < Rn; rr += T) {
        const int sI = seg_of_row(sg, rr);
        const int f = sg.first[sI], l = sg.last[sI];
        const int k = f + 1 + (rr - sg.ro[sI]);
        const int b1f = sg.br1[sI], b2f = sg.br2[sI];
        const int pos = base + k * along;
        R aa, bb, cc, dd;
        if (DIR == 0) {  // precomputed by k_coef_fsj
            const size_t q = (size_t)line * g.LT + k;
            aa = colTr<R>(g, 0)[q];
            bb = colTr<R>(g, 1)[q];
            cc = colTr<R>(g, 2)[q];
            dd = colTr<R>(g, 3)[q];
            if (k == f + 1) {
                if (b1f || g.u[base + f * along] == 0) bb += aa;
                else dd -= aa * R(FS[base + f * along]);
            }
            if (k == l - 1) {
                if (b2f && g.u[base + l * along] == 0) bb += cc;
                else dd -= cc * R(FS[base + l * along]);
            }
        } else {
            fsi_cell_coeffs<R>(g, p, pos, aa, bb, cc, dd);
            if (k == f + 1) {
                if (b1f || g.t_v[base + f * along] == 0) bb = bb + aa;
                else dd = dd - aa * R(FS[base + f * along]);
            }
            if (k == l - 1) {
                if (b2f || g.t_v[base + l * along] == 0) bb = bb + cc;
                else dd = dd - cc * R(FS[base + l * along]);
            }
        }
        A[rr] = (k == f + 1) ? R(0) : aa;
        B[rr] = bb;
        Cc[rr] = (k == l - 1) ? R(0) : cc;
        D[rr] = dd;
    }
    tm.sync();
    solve_line<SOLVER, R>(A, B, Cc, D, pl, Rn, red, tm);
    const R* x = B;
    const double* vel = DIR == 0 ? g.u : g.t_v;  // FSj: u = t_u here (see fsj_cell_coeffs)
    for (int c = tid; c < Rn; c += T) {
        const int sI = seg_of_row(sg, c);
        const int f = sg.first[sI], l = sg.last[sI];
        const int k = f + 1 + (c - sg.ro[sI]);
        const int b1f = sg.br1[sI], b2f = sg.br2[sI];
        const int pos = base + k * along;
        double xv = x[c];
        if (xv < 0) xv = p.NDnen;
        g.tFS[pos] = xv;
        if (k == f + 1) {
            // FSj: t_u[pos - width]; FSi: t_v[i*width + first]
            const double vb = DIR == 0 ? vel[pos - P] : vel[base + f * along];
            g.tFS[base + f * along] = (b1f || vb == 0) ? xv : FS[base + f * along];
        }
        if (k == l - 1) {
            const double vb = DIR == 0 ? vel[pos + P] : vel[base + l * along];
            g.tFS[base + l * along] = (b2f || vb == 0) ? xv : FS[base + l * along];
        }
    }
}

// Fused sediment sweep of one direction: as k_hydro_sweep.
template <int DIR, int SOLVER, class R, class Lines>
__device__ __forceinline__ void fs_sweep_loop(const Lines& lines, int half, int cap, int RB, double* gscr_d, int RG) {
    extern __shared__ double dyn_smem_d[];
    R* dyn_smem = reinterpret_cast<R*>(dyn_smem_d);
    __shared__ LineShared sgw[kWL];
    __shared__ int s_mem[kWL], s_line[kWL];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nlines = lines.count();
    const int G = gridDim.x;
    for (int j0 = 0; (int)blockIdx.x + j0 * G < nlines; j0 += kWL) {
        const int li = blockIdx.x + (j0 + w) * G;
        LineShared& sg = sgw[w];
        if (li < nlines) {  // warp-uniform
            int m = 0, line = 0;
            lines.at(li, m, line);
            if (lane == 0) {
                s_mem[w] = m;
                s_line[w] = line;
            }
            fs_setup<DIR, WarpG>(lines.grid(m), lines.params(m), line, sg);
        } else if (lane == 0) {
            sg.nseg = sg.R = 0;
        }
        __syncthreads();
        const LineShared& mine = sgw[lane & (kWL - 1)];
        if (!__any_sync(0xffffffffu, mine.R > kRowSlice)) {  // the same in every warp
            if (sg.R > 0) {
                R* A = dyn_smem + w * 4 * kRowSlice;
                fs_body<DIR, SOLVER, R>(lines.grid(s_mem[w]), lines.params(s_mem[w]), half, s_line[w], sg, A, A + kRowSlice,
                                        A + 2 * kRowSlice, A + 3 * kRowSlice, (R*)nullptr,
                                        SolvePlan{32, chunk_len(sg.R, 32)}, WarpTeam());
            }
            __syncthreads();
            continue;
        }
        const SolvePlan mp = solve_plan(mine.R, SOLVER == 0 ? 256 : 32);
        const int need = 4 * mp.rows() + 4 * mp.red() + (mp.rows() > RB ? cap : 0);
        unsigned todo = __ballot_sync(0xffffffffu, lane < kWL && mine.R > 0);
        while (todo) {
            TeamPick t = pick_team(todo, need, cap);
            const bool global = t.sel == 0;  // the first line left, by the whole CTA
            if (global) {
                t.line = __ffs(todo) - 1;
                t.sel = 1u << t.line;
                t.warps = kWL;
            }
            const LineShared& sl = sgw[t.line];
            const Team tm(t.first, t.warps);
            const int pv = __shfl_sync(0xffffffffu, mp.m << 10 | mp.t1, t.line);
            const SolvePlan pl{pv & 1023, pv >> 10};
            const int lm = s_mem[t.line], ln = s_line[t.line];
            if (__builtin_expect(!global, 1)) {
                const int P = pl.rows();
                R* A = dyn_smem + t.off;
                fs_body<DIR, SOLVER, R>(lines.grid(lm), lines.params(lm), half, ln, sl, A, A + P, A + 2 * P, A + 3 * P,
                                        A + 4 * P, pl, tm);
            } else {
                R* A = reinterpret_cast<R*>(gscr_d) + (size_t)blockIdx.x * 4 * (size_t)RG;
                fs_body<DIR, SOLVER, R>(lines.grid(lm), lines.params(lm), half, ln, sl, A, A + RG, A + 2 * RG, A + 3 * RG,
                                        dyn_smem, pl, tm);
            }
            todo &= ~t.sel;
            __syncthreads();  // the regions and sgw are reused
        }
    }
}

template <int DIR, int SOLVER, class R>
__global__ void __launch_bounds__(kTL, 1) k_fs_sweep(DevGrid g, DevParams p, int half, int startidx, int endidx, int cap,
                                                  int RB, double* gscr_d, int RG) {
    fs_sweep_loop<DIR, SOLVER, R>(OneGridLines{g, p, startidx, endidx - startidx + 1}, half, cap, RB, gscr_d, RG);
}
template <int DIR, int SOLVER, class R>
__global__ void __launch_bounds__(kTL, 1) k_fs_sweep_b(BatchLines bl, int half, int cap, int RB, double* gscr_d, int RG) {
    fs_sweep_loop<DIR, SOLVER, R>(bl, half, cap, RB, gscr_d, RG);
}

// Largest dynamic shared memory the kernel may be given on this device.
int max_dyn_smem(const void* f) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, f) != cudaSuccess) return 48 * 1024;
    return optin - (int)a.sharedSizeBytes;
}

template <class F>
cudaError_t allow_all(F* const* fs, int n, int* limit) {
    int lim = 1 << 30;
    for (int i = 0; i < n; i++) {
        const int mx = max_dyn_smem((const void*)fs[i]);
        const cudaError_t e = cudaFuncSetAttribute((const void*)fs[i], cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
        if (e != cudaSuccess) return e;
        if (mx < lim) lim = mx;
    }
    *limit = lim;
    return cudaSuccess;
}

using HydroSweepFn = void(DevGrid, DevParams, int, int, int, int, double*, int);
using FsSweepFn = void(DevGrid, DevParams, int, int, int, int, int, double*, int);
using HydroSweepBFn = void(BatchLines, int, int, double*, int);
using FsSweepBFn = void(BatchLines, int, int, int, double*, int);

// [precision: 0 FP64, 1 mixed][direction][solver]
HydroSweepFn* const kHydroSweep[2][2][2] = {
    {{k_hydro_sweep<0, 0, double>, k_hydro_sweep<0, 1, double>},
     {k_hydro_sweep<1, 0, double>, k_hydro_sweep<1, 1, double>}},
    {{k_hydro_sweep<0, 0, float>, k_hydro_sweep<0, 1, float>},
     {k_hydro_sweep<1, 0, float>, k_hydro_sweep<1, 1, float>}}};
FsSweepFn* const kFsSweep[2][2][2] = {
    {{k_fs_sweep<0, 0, double>, k_fs_sweep<0, 1, double>}, {k_fs_sweep<1, 0, double>, k_fs_sweep<1, 1, double>}},
    {{k_fs_sweep<0, 0, float>, k_fs_sweep<0, 1, float>}, {k_fs_sweep<1, 0, float>, k_fs_sweep<1, 1, float>}}};

HydroSweepBFn* const kHydroSweepB[2][2][2] = {
    {{k_hydro_sweep_b<0, 0, double>, k_hydro_sweep_b<0, 1, double>},
     {k_hydro_sweep_b<1, 0, double>, k_hydro_sweep_b<1, 1, double>}},
    {{k_hydro_sweep_b<0, 0, float>, k_hydro_sweep_b<0, 1, float>},
     {k_hydro_sweep_b<1, 0, float>, k_hydro_sweep_b<1, 1, float>}}};
FsSweepBFn* const kFsSweepB[2][2][2] = {
    {{k_fs_sweep_b<0, 0, double>, k_fs_sweep_b<0, 1, double>}, {k_fs_sweep_b<1, 0, double>, k_fs_sweep_b<1, 1, double>}},
    {{k_fs_sweep_b<0, 0, float>, k_fs_sweep_b<0, 1, float>}, {k_fs_sweep_b<1, 0, float>, k_fs_sweep_b<1, 1, float>}}};

}  // namespace

// Values of shared memory a launch asks for: the longest line it may hold on chip, or room for
// `n` lines side by side (the lines a CTA takes at once) of up to kRowW rows (wide) or
// kRowSlice, whichever is more; more lines than fit are swept in rounds.
namespace {
int sweep_cap(const SweepPlan& sp, int fs, int n, int wide) {
    const int one = fs ? 4 * sp.RBf + 4 * kRedRows : 4 * sp.RB + kEnds + 4 * kRedRows;
    const int side = n * (4 * (wide ? kRowW : kRowSlice) + (fs ? 0 : kEnds));
    const int lim = fs ? sp.lim_f : sp.lim_h;
    return std::min(std::max(one, side), lim);
}
}  // namespace

// Shared-memory sizes and the long-line grid of a grid of N x M cells on the current
// device; opts the sweep kernels into the shared memory they may need.  max_rows > 0 caps
// the rows a long line may hold in shared memory (longer lines then run in global scratch).
cudaError_t sweep_plan(int N, int M, SweepPlan* sp, int max_rows) {
    cudaError_t e;
    int lim_h, lim_f;
    // the row counts below are planned for FP64 rows; the mixed form's FP32 rows take half
    // the bytes of the same plan
    if ((e = allow_all(&kHydroSweep[0][0][0], 8, &lim_h)) != cudaSuccess) return e;
    if ((e = allow_all(&kFsSweep[0][0][0], 8, &lim_f)) != cudaSuccess) return e;
    // the batched kernels' static shared memory may differ: the plan fits both
    for (int i = 0; i < 8; i++) {
        lim_h = std::min(lim_h, max_dyn_smem((const void*)(&kHydroSweepB[0][0][0])[i]));
        lim_f = std::min(lim_f, max_dyn_smem((const void*)(&kFsSweepB[0][0][0])[i]));
    }
    const int L = N > M ? N : M;
    // a line's region: its rows, a hydrodynamic line's segment ends, the reduced rows of a
    // two-level solve
    const size_t fix_h = kEnds + 4 * (size_t)kRedRows, fix_f = 4 * (size_t)kRedRows;
    if ((long long)(sizeof(double) * (fix_h + 4 * kRowW)) > lim_h || (long long)(sizeof(double) * (fix_f + 4 * kRowW)) > lim_f)
        return cudaErrorInvalidValue;
    sp->lim_h = lim_h / (int)sizeof(double);
    sp->lim_f = lim_f / (int)sizeof(double);
    // every row a line can have: rows <= 2 L + 20 (solved by 32 lanes)
    {
        int rg = 0;
        for (int t1 = 32; t1 <= 256; t1 <<= 1) {  // the padded rows of any solve plan
            const int r = t1 * chunk_len(2 * L + HYD_SEGL, t1);
            if (r > rg) rg = r;
        }
        sp->RG = rg;
    }
    sp->need_global = 0;
    sp->wide = 0;
    if (4 * (size_t)sp->RG + fix_h <= (size_t)sp->lim_h) {
        sp->RB = sp->RG;
    } else {  // as many rows as fit; longer lines use global scratch
        sp->RB = (int)((sp->lim_h - fix_h) / 4);
        sp->need_global = 1;
    }
    if (max_rows > 0 && sp->RB > max_rows) {
        sp->RB = max_rows;
        sp->need_global = 1;
    }
    sp->RGf = 0;
    for (int t1 = 32; t1 <= 256; t1 <<= 1) {
        const int r = t1 * chunk_len(L, t1);
        if (r > sp->RGf) sp->RGf = r;
    }
    if (4 * (size_t)sp->RGf + fix_f <= (size_t)sp->lim_f) {
        sp->RBf = sp->RGf;
    } else {
        sp->RBf = (int)((sp->lim_f - fix_f) / 4);
        sp->need_global = 1;
    }
    if (max_rows > 0 && sp->RBf > max_rows) {
        sp->RBf = max_rows;
        sp->need_global = 1;
    }
    sp->smem_lines = sizeof(double) * (size_t)sweep_cap(*sp, 0, kWL, 0);
    sp->smem_fs_lines = sizeof(double) * (size_t)sweep_cap(*sp, 1, kWL, 0);
    int dev = 0, nsm = 0, occ = 0, occf = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kHydroSweep[0][0][0], kTL, sp->smem_lines)) !=
        cudaSuccess)
        return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occf, kFsSweep[0][0][0], kTL, sp->smem_fs_lines)) !=
        cudaSuccess)
        return e;
    if (occ < 1) occ = 1;
    if (occf < 1) occf = 1;
    sp->long_grid = nsm * (occ < occf ? occ : occf);
    if (sp->long_grid > L + 3) sp->long_grid = L + 3;
    sp->scratch_doubles =
        sp->need_global ? (size_t)sp->long_grid * (4 * (size_t)(sp->RG > sp->RGf ? sp->RG : sp->RGf) + kEnds) : 1;
    return cudaSuccess;
}

void sweep_plan_throughput(const int* dims, SweepPlan* const* plans, int count) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    long long total = 0;  // CTAs that give every line of every member its own warp
    for (int k = 0; k < count; k++) total += (std::max(dims[2 * k], dims[2 * k + 1]) + 3 + kWL - 1) / kWL;
    const long long per = std::min(std::max((total + nsm / 2) / nsm, 1LL), 4LL);
    for (int k = 0; k < count; k++) {
        const int g = (int)((std::max(dims[2 * k], dims[2 * k + 1]) + 3 + kWL * per - 1) / (kWL * per));
        if (plans[k]->long_grid > g) plans[k]->long_grid = g;
        plans[k]->wide = 1;
    }
}

namespace {
// Shared memory of a launch over nlines lines: the wide room where the plan asks for it (batch
// members) and where a CTA takes more than kWL lines, so that few rounds are needed.
int launch_cap(const SweepPlan& sp, int fs, int nlines) {
    const int per = (nlines + sp.long_grid - 1) / sp.long_grid;
    return sweep_cap(sp, fs, std::min(kWL, per), sp.wide || per > kWL);
}

void hydro_sweep(int dir, const DevGrid& g, const DevParams& p, const SweepPlan& sp, int startidx, int endidx,
                 int solver, double* scratch, cudaStream_t s) {
    const int nlines = endidx - startidx + 1;
    if (nlines <= 0) return;
    const int sv = solver ? 1 : 0;
    const int cap = launch_cap(sp, 0, nlines);
    const size_t esz = p.mixed ? sizeof(float) : sizeof(double);
    kHydroSweep[p.mixed ? 1 : 0][dir][sv]<<<sp.long_grid, kTL, esz * cap, s>>>(g, p, startidx, endidx, cap, sp.RB, scratch,
                                                                              sp.RG);
    hyd_kernel_launches_add(1);
}

void fs_sweep(int dir, const DevGrid& g, const DevParams& p, const SweepPlan& sp, int half, int startidx,
              int endidx, int solver, double* scratch, cudaStream_t s) {
    const int nlines = endidx - startidx + 1;
    if (nlines <= 0) return;
    const int sv = solver ? 1 : 0;
    const int cap = launch_cap(sp, 1, nlines);
    const size_t esz = p.mixed ? sizeof(float) : sizeof(double);
    kFsSweep[p.mixed ? 1 : 0][dir][sv]<<<sp.long_grid, kTL, esz * cap, s>>>(g, p, half, startidx, endidx, cap, sp.RBf,
                                                                           scratch, sp.RGf);
    hyd_kernel_launches_add(1);
}
}  // namespace

void launch_coef_fsj(const DevGrid& g, const DevParams& p, int half, int shared, cudaStream_t s) {
    const CoefShape c = g.tile_cols || shared ? CoefShape{256, 1} : coef_shape(g);
    const int nb = ((g.N - 1) * c.wpc * 32 + c.threads - 1) / c.threads;
    void (*const k[2][2])(DevGrid, DevParams, int, int) = {{k_coef_fsj<0, double>, k_coef_fsj<1, double>},
                                                           {k_coef_fsj<0, float>, k_coef_fsj<1, float>}};
    k[p.mixed ? 1 : 0][g.tile_cols ? 1 : 0]<<<nb, c.threads, 0, s>>>(g, p, half, c.wpc);
    hyd_kernel_launches_add(1);
}

void launch_sweep_uz(const DevGrid& g, const DevParams& p, const SweepPlan& sp, int startidx, int endidx,
                     int solver, double* scratch, cudaStream_t s) {
    hydro_sweep(0, g, p, sp, startidx, endidx, solver, scratch, s);
}

void launch_sweep_vz(const DevGrid& g, const DevParams& p, const SweepPlan& sp, int startidx, int endidx,
                     int solver, double* scratch, cudaStream_t s) {
    hydro_sweep(1, g, p, sp, startidx, endidx, solver, scratch, s);
}

// FSj over columns 3..M-1 (Engine.py:224-237), FSi over rows 3..N-1 (Engine.py:345-358).
void launch_fs_sweep_j(const DevGrid& g, const DevParams& p, const SweepPlan& sp, int half, int solver,
                       double* scratch, cudaStream_t s) {
    fs_sweep(0, g, p, sp, half, 3, g.M - 1, solver, scratch, s);
}

void launch_fs_sweep_i(const DevGrid& g, const DevParams& p, const SweepPlan& sp, int half, int solver,
                       double* scratch, cudaStream_t s) {
    fs_sweep(1, g, p, sp, half, 3, g.N - 1, solver, scratch, s);
}

// ---- batched sweeps: every member's lines in one persistent launch (the common plan of
// the batch: the largest member's)
void launch_sweep_batch(int dir, const BatchLines& bl, const SweepPlan& sp, int solver, int mixed, double* scratch,
                        int grid, cudaStream_t s) {
    const int cap = sp.lim_h;
    const size_t esz = mixed ? sizeof(float) : sizeof(double);
    kHydroSweepB[mixed ? 1 : 0][dir][solver ? 1 : 0]<<<grid, kTL, esz * cap, s>>>(bl, cap, sp.RB, scratch, sp.RG);
    hyd_kernel_launches_add(1);
}

void launch_fs_sweep_batch(int dir, const BatchLines& bl, const SweepPlan& sp, int half, int solver, int mixed,
                           double* scratch, int grid, cudaStream_t s) {
    const int cap = sp.lim_f;
    const size_t esz = mixed ? sizeof(float) : sizeof(double);
    kFsSweepB[mixed ? 1 : 0][dir][solver ? 1 : 0]<<<grid, kTL, esz * cap, s>>>(bl, half, cap, sp.RBf, scratch, sp.RGf);
    hyd_kernel_launches_add(1);
}

void launch_coef_fsj_batch(const BatchRef& br, int ctas, int half, int mixed, cudaStream_t s) {
    if (mixed) k_coef_fsj_b<0, float><<<ctas, 256, 0, s>>>(br, half);
    else k_coef_fsj_b<0, double><<<ctas, 256, 0, s>>>(br, half);
    hyd_kernel_launches_add(1);
}

// The batched sweeps may use all the shared memory the device allows (their row plans
// are the largest member's).
cudaError_t batch_sweep_setup() {
    int lim;
    cudaError_t e = allow_all(&kHydroSweepB[0][0][0], 8, &lim);
    if (e == cudaSuccess) e = allow_all(&kFsSweepB[0][0][0], 8, &lim);
    return e;
}
