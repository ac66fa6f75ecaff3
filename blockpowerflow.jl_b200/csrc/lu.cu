// LU refactorization on a fixed fill pattern and its multi-RHS solves: sparse front, dense tail.
//
// Reference: cusolverRfRefactor / cusolverRfSolve behind src/cusolverRF.jl:304-331,451-470.
//
// Bound: the elimination's dependency chain, not its arithmetic.  Minimum degree on a grid's
// Jacobian ends in a nearly dense block (25,000 buses: 48k unknowns, 994 column-step levels, of which
// the last ~740 hold one column each and 92 % of the 102 M update pairs).  Column steps with a grid
// barrier per level took 14.2 ms there, and a push-form solve of 256 columns 10.5 ms (1,573 levels).
//
//  * The last m columns (a multiple of 64 that balances the two parts' estimated times, up to 3,072)
//    are one dense block.  What precedes them has 50-250 short levels.
//  * Front: row-wise elimination as a data flow (factor_df_kernel of prec.cu: a warp per row, values
//    are their own ready marks).  Its long last rows, and the tail's rows, whose Schur complement goes
//    to dense storage, take a CTA each (lu_cta_rows_kernel).  No atomics: the factors are deterministic.
//  * Tail: blocked right-looking LU without pivoting (the pivot order is the analysis's) in one
//    cooperative launch, 64 x 64 tiles on the FP64 tensor pipe.  A step costs one grid barrier: a tile
//    substitutes its own row and column panels with the diagonal factors itself, and CTA 0 factors the
//    next diagonal tile as soon as it is updated.
//  * Solves: up to 24,800 rows one right-hand side per CTA in shared memory (trsv_col.cu, the dense
//    tail between the sweeps); larger systems by a data flow over rows, a warp per row with the
//    right-hand sides over the lanes, the tail on the FP64 tensor pipe eight columns a CTA.
//
// Measured (cold caches, column steps and push solves -> this): 25,000 buses, refactor 14.3 -> 1.45 ms, 256 columns
// 11.2 -> 1.13 ms; 9,000 buses, refactor 3.6 ms -> 666 us, 64 columns 2.6 ms -> 377 us; 300 buses, refactor 273 ->
// 104 us, one column 351 -> 49 us.  Errors: 0.89 of those of the column steps (forward, geometric mean over 70 grids
// of 300 to 9,000 buses against solutions refined in extended precision).
// What bounds it now (25,000 buses): the level chains of the short rows (470 us) and of the rows a CTA
// takes (465 us), and the tail's 12 block steps (363 us, of which the diagonal tiles ~20 us each).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "bpf_internal.cuh"
#include "bulk.cuh"
#include "pending.cuh"
#include "prec.cuh"

namespace bpf {

constexpr int kNB = 64;          // tail tile
constexpr int kCtaRow = 96;      // entries of a row from the diagonal on past which a CTA takes it
constexpr int kTailSolveThreads = 640;   // 1,024 leave the substitution 64 registers (25,000 buses, 256 columns 1,054 / 1,029 us)
constexpr int kTS = kNB + 4;     // tile row stride in shared memory (conflict-free DMMA fragments)

__device__ __forceinline__ void lu_dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// ------------------------------------------------------------------------------------
// long front rows and the Schur complement: a CTA per row
// ------------------------------------------------------------------------------------
// A row's L entries (a tail row's: before column s) in order, l = w_k / u_kk, each updating the row by
// U's row k (destinations listed per pair, sources contiguous).  The row, the pivots and the entries'
// pair ranges are in shared memory; the pairs of the next four entries are under way, up to three a
// thread, and an entry costs one barrier.  Front rows depend on one another as in factor_df_kernel
// (values are their own ready marks; positions in dependency order, all CTAs resident, bounded polls).
struct CtaRowsArgs {
    int count, s, m, mp, nmax, wmax;
    const int *order, *rp, *ci, *diag, *fend, *fsrc, *pp, *pdst;
    const double *vals;
    double *fv, *S;
    SweepStore out;
    DevStatus *ds;
};

__global__ void __launch_bounds__(256) lu_cta_rows_kernel(CtaRowsArgs a) {
    extern __shared__ __align__(16) double row[];
    double *w = row, *piv = row + a.wmax, *lv = piv + a.nmax;
    int *p0 = reinterpret_cast<int *>(lv + a.nmax), *src = p0 + a.nmax + 1;   // pair range, source - pair
    const int tid = threadIdx.x;
    const long long lim = a.ds->wait_limit > 0 ? a.ds->wait_limit : kSpinLimit;
    // the tail's rows past the last are the identity: written every time, since the tail's factorization
    // spreads a NaN or an infinity into them
    for (size_t e = (size_t)a.m * a.mp + blockIdx.x * 256 + tid; e < (size_t)a.mp * a.mp; e += (size_t)gridDim.x * 256)
        a.S[e] = e / a.mp == e % a.mp ? 1.0 : 0.0;
    for (int q = blockIdx.x; q < a.count; q += gridDim.x) {
        const int i = __ldg(a.order + q);
        const bool tail = i >= a.s;
        const int rs = __ldg(a.rp + i), len = __ldg(a.rp + i + 1) - rs, nf = __ldg((tail ? a.fend : a.diag) + i) - rs;
        __syncthreads();   // the previous row's storage is free
        if (tail)
            for (int c = tid; c < a.mp; c += 256) w[nf + c] = 0.0;
        __syncthreads();
        for (int e = tid; e < len; e += 256) {
            const int sv = __ldg(a.fsrc + rs + e);
            const double v = sv < 0 ? 0.0 : __ldg(a.vals + sv);
            w[tail && e >= nf ? nf + __ldg(a.ci + rs + e) - a.s : e] = v;
            if (e < nf) {
                const int d = __ldg(a.diag + __ldg(a.ci + rs + e)), p = __ldg(a.pp + rs + e);
                piv[e] = ld_value(a.fv + d);
                p0[e] = p;
                src[e] = d + 1 - p;
            }
        }
        if (tid == 0) p0[nf] = __ldg(a.pp + rs + nf);
        __syncthreads();
        constexpr int D = 4, C = 3;
        int d[D][C];
        double v[D][C];
        bool ok = true;
        auto fetch = [&](int e, int (&dd)[C], double (&vv)[C]) {
#pragma unroll
            for (int c = 0; c < C; c++) {
                dd[c] = -1;
                vv[c] = 0.0;
                if (e < nf) {
                    const int t = p0[e] + tid + 256 * c;
                    if (t < p0[e + 1]) {
                        dd[c] = __ldg(a.pdst + t) - rs;
                        vv[c] = ld_value(a.fv + (t + src[e]));
                    }
                }
            }
        };
#pragma unroll
        for (int u = 0; u < D; u++) fetch(u, d[u], v[u]);
        for (int eb = 0; eb < nf; eb += D) {
#pragma unroll
            for (int u = 0; u < D; u++) {
                const int e = eb + u;
                if (e < nf) {
                    double pv = piv[e];
                    if (is_pending(pv)) ok = poll_value(a.fv + (src[e] + p0[e] - 1), pv, lim, a.ds) && ok;
                    const double l = w[e] / pv;
                    if (tid == 0) {
                        lv[e] = l;
                        if (pv == 0.0 && atomicCAS(&a.ds->err, 0, (int)DEV_ZERO_PIVOT) == 0) a.ds->aux = __ldg(a.ci + rs + e);
                    }
#pragma unroll
                    for (int c = 0; c < C; c++)
                        if (d[u][c] >= 0) {
                            if (is_pending(v[u][c]))
                                ok = poll_value(a.fv + (p0[e] + tid + 256 * c + src[e]), v[u][c], lim, a.ds) && ok;
                            w[d[u][c]] -= l * v[u][c];
                        }
                    for (int t = p0[e] + tid + 256 * C; t < p0[e + 1]; t += 256) {
                        double x = 0.0;
                        ok = poll_value(a.fv + (t + src[e]), x, lim, a.ds) && ok;
                        w[__ldg(a.pdst + t) - rs] -= l * x;
                    }
                    fetch(e + D, d[u], v[u]);
                }
                if (u + 1 < D) __syncthreads();
            }
            if (__syncthreads_or(!ok)) {
                if (tid == 0) atomicCAS(&a.ds->err, 0, (int)DEV_BARRIER_TIMEOUT);
                return;
            }
        }
        for (int e = tid; e < (tail ? nf : len); e += 256) {
            const double x = not_pending(e < nf ? lv[e] : w[e]);
            __stcg(a.fv + rs + e, x);
            if (!tail && e == nf && x == 0.0) {
                if (atomicCAS(&a.ds->err, 0, (int)DEV_ZERO_PIVOT) == 0) a.ds->aux = i;
            }
            sweep_put(a.out, rs + e, x);
        }
        if (tail)
            for (int c = tid; c < a.mp; c += 256) a.S[(size_t)(i - a.s) * a.mp + c] = w[nf + c];
    }
}
static size_t cta_rows_smem(int nmax, int wmax) { return sizeof(double) * (2 * (size_t)nmax + wmax) + sizeof(int) * (2 * (size_t)nmax + 2); }

// ------------------------------------------------------------------------------------
// dense tail: factorization
// ------------------------------------------------------------------------------------
// 64 x 64 tile from global memory (row stride ld) into shared memory.
__device__ __forceinline__ void tile_in(double *t, const double *g, size_t ld) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const int e = threadIdx.x + 256 * u, r = e >> 6, c = e & 63;
        t[r * kTS + c] = __ldcg(g + r * ld + c);
    }
}

// acc += A B of two shared 64 x 64 tiles; warp w holds rows 16 (w / 2).., columns 32 (w & 1)..
__device__ __forceinline__ void tile_mul(double (&acc)[2][4][2], const double *A, const double *B) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wm = warp >> 1, wn = warp & 1, g = lane >> 2,
              t4 = lane & 3;
#pragma unroll
    for (int ks = 0; ks < 16; ks++) {
        const int k = 4 * ks + t4;
        double a[2], b[4];
#pragma unroll
        for (int mi = 0; mi < 2; mi++) a[mi] = A[(wm * 16 + mi * 8 + g) * kTS + k];
#pragma unroll
        for (int ni = 0; ni < 4; ni++) b[ni] = B[k * kTS + wn * 32 + ni * 8 + g];
#pragma unroll
        for (int mi = 0; mi < 2; mi++)
#pragma unroll
            for (int ni = 0; ni < 4; ni++) lu_dmma(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
    }
}

// f(row, column, value) over a thread's accumulators.
template <typename F>
__device__ __forceinline__ void tile_each(const double (&acc)[2][4][2], F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wm = warp >> 1, wn = warp & 1, g = lane >> 2,
              t4 = lane & 3;
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) f(wm * 16 + mi * 8 + g, wn * 32 + ni * 8 + 2 * t4 + i, acc[mi][ni][i]);
}

__device__ __forceinline__ void tile_zero(double (&acc)[2][4][2]) {
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
}

// LU of the shared tile T (no pivoting): the packed factors row by row into F (row stride ld) and column by column
// into D, the pivots' reciprocals into R.  Thread (ti, tj) of 16 x 16 holds rows ti + 16 r, columns tj + 16 c; a
// pivot row and column go through shared memory, one barrier a step.
__device__ __forceinline__ void tile_lu(double *T, double *bufs, double *F, size_t ld, double *D, double *R, int row0,
                                        DevStatus *ds) {
    double *rowA = bufs, *colA = bufs + 128;
    const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
    double a[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) a[r][c] = T[(ti + 16 * r) * kTS + tj + 16 * c];
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
#pragma unroll 1
        for (int kl = 0; kl < 16; kl++) {
            const int k = 16 * kk + kl, o = 64 * (k & 1);
            if (ti == kl)
#pragma unroll
                for (int c = 0; c < 4; c++) rowA[o + tj + 16 * c] = a[kk][c];
            if (tj == kl)
#pragma unroll
                for (int r = 0; r < 4; r++) colA[o + ti + 16 * r] = a[r][kk];
            __syncthreads();
            const double piv = rowA[o + k], inv = 1.0 / piv;
            if (threadIdx.x == 0) {
                R[k] = inv;
                if (piv == 0.0 && atomicCAS(&ds->err, 0, (int)DEV_ZERO_PIVOT) == 0) ds->aux = row0 + k;
            }
            double l[4], u[4];
#pragma unroll
            for (int r = kk; r < 4; r++) {
                const int i = ti + 16 * r;
                l[r] = i > k ? colA[o + i] * inv : 0.0;
            }
#pragma unroll
            for (int c = kk; c < 4; c++) {
                const int j = tj + 16 * c;
                u[c] = j > k ? rowA[o + j] : 0.0;
            }
#pragma unroll
            for (int r = kk; r < 4; r++)
#pragma unroll
                for (int c = kk; c < 4; c++) a[r][c] -= l[r] * u[c];
            if (tj == kl)
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (ti + 16 * r > k) a[r][kk] = l[r];
        }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int i = ti + 16 * r, j = tj + 16 * c;
            F[i * ld + j] = a[r][c];
            D[j * kNB + i] = a[r][c];
        }
}

// Substitution with a 64 x 64 triangle, 8 Q right-hand sides a warp: x[q][b][i] is unknown 8 b + 2 t4 + i of right-hand
// side 8 q + g (a DMMA's accumulators); m(k, j): what unknown k takes from j, j > k (DESC: j < k); SCALE: unknowns
// times rinv[k].  Eight unknowns at a time by broadcasts within four lanes, the others by the tensor pipe, whose
// operand is the solved block as it lies.  (Products with an inverted triangle are as many, but lose its condition
// where it grows: 1e-7 for a triangle of ones on the diagonal and -0.54 above, 1e-17 so.)
template <bool DESC, bool SCALE, int Q, class M>
__device__ __forceinline__ void tri_substitute(double (&x)[Q][8][2], M m, const double *rinv) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int bi = 0; bi < 8; bi++) {
        const int b = DESC ? 7 - bi : bi;
#pragma unroll
        for (int ci = 0; ci < 8; ci++) {
            const int c = DESC ? 7 - ci : ci, k = 8 * b + c;
            const double a0 = m(k, 8 * b + 2 * t4), a1 = m(k, 8 * b + 2 * t4 + 1);
#pragma unroll
            for (int q = 0; q < Q; q++) {
                double v = x[q][b][c & 1];
                if (SCALE) v *= rinv[k];
                const double xk = __shfl_sync(0xffffffffu, v, (lane & 28) | (c >> 1));
                if (SCALE && t4 == c >> 1) x[q][b][c & 1] = xk;
                if (DESC ? 2 * t4 < c : 2 * t4 > c) x[q][b][0] -= xk * a0;
                if (DESC ? 2 * t4 + 1 < c : 2 * t4 + 1 > c) x[q][b][1] -= xk * a1;
            }
        }
#pragma unroll
        for (int ni = DESC ? 0 : b + 1; ni < (DESC ? b : 8); ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const double v = m(8 * b + 2 * t4 + i, 8 * ni + g);
#pragma unroll
                for (int q = 0; q < Q; q++) lu_dmma(x[q][ni][0], x[q][ni][1], -x[q][b][i], v);
            }
    }
}

// S (mp x mp, nb tiles a side; destroyed) -> F: the tiles of L and U; D: the diagonal ones column by column; R: the
// pivots' reciprocals.  row0: the first row of the tail (diagnostics).
__global__ void __launch_bounds__(256, 1)
lu_tail_factor_kernel(int nb, double *S, double *F, double *D, double *R, int row0, DevStatus *ds) {
    extern __shared__ __align__(16) double tiles[];
    __shared__ unsigned s_gen;
    if (threadIdx.x == 0) s_gen = barrier_gen_start(ds);
    __syncthreads();
    unsigned gen = s_gen;
    double *T0 = tiles, *T1 = T0 + kNB * kTS, *T2 = T1 + kNB * kTS, *T3 = T2 + kNB * kTS, *bufs = T3 + kNB * kTS,
           *rinv = bufs + 256;
    const size_t ld = (size_t)nb * kNB;
    auto at = [&](int i, int j) { return (size_t)i * kNB * ld + (size_t)j * kNB; };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    if (blockIdx.x == 0) {
        tile_in(T0, S, ld);
        __syncthreads();
        tile_lu(T0, bufs, F, ld, D, R, row0, ds);
    }
    if (nb > 1 && !grid_barrier(ds, gen)) return;
    for (int k = 0; k + 1 < nb; k++) {
        const int side = nb - 1 - k, ntile = side * side;
        // the diagonal tile, U's rows in T1 and L's columns in T2
        tile_in(T1, F + at(k, k), ld);
        tile_in(T2, D + (size_t)k * kNB * kNB, kNB);
        if (threadIdx.x < kNB) rinv[threadIdx.x] = __ldcg(R + k * kNB + threadIdx.x);
        // tile 0, the next diagonal one, is CTA 0's alone; the others go round the other CTAs
        for (int t = blockIdx.x; t < ntile; t += (gridDim.x > 1 && t == 0) ? ntile : max(1, (int)gridDim.x - 1)) {
            const int i = k + 1 + t / side, j = k + 1 + t % side;
            __syncthreads();
            tile_in(T0, S + at(i, k), ld);
            tile_in(T3, S + at(k, j), ld);
            __syncthreads();
            // T0 <- T0 U^{-1}, a row per right-hand side, on warps 0 - 3; T3 <- L^{-1} T3, a column each, on 4 - 7
            double x[2][8][2];
            const int v0 = 16 * (warp & 3) + g;
            if (warp < 4) {
#pragma unroll
                for (int q = 0; q < 2; q++)
#pragma unroll
                    for (int ni = 0; ni < 8; ni++)
#pragma unroll
                        for (int e = 0; e < 2; e++) x[q][ni][e] = T0[(v0 + 8 * q) * kTS + 8 * ni + 2 * t4 + e];
                tri_substitute<false, true, 2>(x, [&](int kc, int jc) { return T1[kc * kTS + jc]; }, rinv);
#pragma unroll
                for (int q = 0; q < 2; q++)
#pragma unroll
                    for (int ni = 0; ni < 8; ni++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int r = v0 + 8 * q, c = 8 * ni + 2 * t4 + e;
                            T0[r * kTS + c] = x[q][ni][e];
                            if (j == k + 1) F[at(i, k) + r * ld + c] = x[q][ni][e];
                        }
            } else {
#pragma unroll
                for (int q = 0; q < 2; q++)
#pragma unroll
                    for (int ni = 0; ni < 8; ni++)
#pragma unroll
                        for (int e = 0; e < 2; e++) x[q][ni][e] = T3[(8 * ni + 2 * t4 + e) * kTS + v0 + 8 * q];
                tri_substitute<false, false, 2>(x, [&](int kc, int jc) { return T2[kc * kTS + jc]; }, rinv);
#pragma unroll
                for (int q = 0; q < 2; q++)
#pragma unroll
                    for (int ni = 0; ni < 8; ni++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int r = 8 * ni + 2 * t4 + e, c = v0 + 8 * q;
                            T3[r * kTS + c] = x[q][ni][e];
                            if (i == k + 1) F[at(k, j) + r * ld + c] = x[q][ni][e];
                        }
            }
            __syncthreads();
            double s[2][4][2];
            tile_zero(s);
            tile_mul(s, T0, T3);
            double *gs = S + at(i, j);
            if (t == 0) __syncthreads();
            tile_each(s, [&](int r, int c, double v) {
                const double y = __ldcg(gs + r * ld + c) - v;
                if (t == 0) T0[r * kTS + c] = y;
                else gs[r * ld + c] = y;
            });
            if (t == 0) {
                __syncthreads();
                tile_lu(T0, bufs, F + at(k + 1, k + 1), ld, D + (size_t)(k + 1) * kNB * kNB, R + (k + 1) * kNB,
                        row0 + (k + 1) * kNB, ds);
            }
        }
        if (!grid_barrier(ds, gen)) return;
    }
}
constexpr size_t kTailFactorSmem = sizeof(double) * (4 * kNB * kTS + 256 + kNB);

// ------------------------------------------------------------------------------------
// dense tail: solves of row-major blocks
// ------------------------------------------------------------------------------------
// Rows s.. of the n x p block Z hold the tail's right-hand sides; rows s.. of W receive U^{-1} L^{-1}
// of them.  A CTA takes eight columns, kept in shared memory; a block step solves with the diagonal tile (warp 0, the
// tile in shared memory), then updates the other rows, eight rows a warp on the tensor pipe.
__global__ void __launch_bounds__(kTailSolveThreads)
lu_tail_solve_kernel(int s, int m, int nb, const double *__restrict__ F, const double *__restrict__ D,
                     const double *__restrict__ R, int p, const double *__restrict__ Z, double *W) {
    extern __shared__ __align__(16) double ysm[];   // [mp][8], then the diagonal tile by columns [64][kTS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int c0 = 8 * blockIdx.x, mp = nb * kNB;
    const size_t ld = mp;
    double *tile = ysm + 8 * (size_t)mp;
    for (int e = threadIdx.x; e < 8 * mp; e += blockDim.x) {
        const int r = e >> 3, c = c0 + (e & 7);
        ysm[e] = r < m && c < p ? __ldcg(Z + (size_t)(s + r) * p + c) : 0.0;
    }
    auto fetch = [&](const double *A, size_t lda, double (&a)[16]) {   // eight rows of A, 64 columns
#pragma unroll
        for (int ks = 0; ks < 16; ks++) a[ks] = __ldg(A + g * lda + 4 * ks + t4);
    };
    for (int sweep = 0; sweep < 2; sweep++)
        for (int bi = 0; bi < nb; bi++) {
            const int b = sweep == 0 ? bi : nb - 1 - bi;
            const int r0 = sweep == 0 ? 8 * (b + 1) : 0, r1 = sweep == 0 ? 8 * nb : 8 * b;
            double *yb = ysm + (size_t)b * kNB * 8;
            // U's rows and right-hand sides times the pivots' reciprocals: no product in the substitution's chain
            for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x)
                tile[(e >> 6) * kTS + (e & 63)] =
                    __ldg(D + (size_t)b * kNB * kNB + e) * (sweep == 0 ? 1.0 : __ldg(R + b * kNB + (e & 63)));
            __syncthreads();
            double a[16];
            if (warp == 0) {
                double x[1][8][2];
#pragma unroll
                for (int ni = 0; ni < 8; ni++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int r = 8 * ni + 2 * t4 + e;
                        x[0][ni][e] = yb[r * 8 + g] * (sweep == 0 ? 1.0 : __ldg(R + b * kNB + r));
                    }
                auto by_column = [&](int k, int j) { return tile[k * kTS + j]; };
                if (sweep == 0) tri_substitute<false, false, 1>(x, by_column, nullptr);
                else tri_substitute<true, false, 1>(x, by_column, nullptr);
#pragma unroll
                for (int ni = 0; ni < 8; ni++)
#pragma unroll
                    for (int e = 0; e < 2; e++) yb[(8 * ni + 2 * t4 + e) * 8 + g] = x[0][ni][e];
            } else if (r0 + warp < r1) {   // the other warps' first tiles are under way meanwhile
                fetch(F + (size_t)8 * (r0 + warp) * ld + (size_t)b * kNB, ld, a);
            }
            __syncthreads();
            for (int t = r0 + warp; t < r1; t += nw) {
                if (warp == 0 || t >= r0 + nw) fetch(F + (size_t)8 * t * ld + (size_t)b * kNB, ld, a);
                double d0 = 0.0, d1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll
                for (int ks = 0; ks < 16; ks += 2) {
                    lu_dmma(d0, d1, a[ks], yb[(4 * ks + t4) * 8 + g]);
                    lu_dmma(e0, e1, a[ks + 1], yb[(4 * ks + 4 + t4) * 8 + g]);
                }
                double *y = ysm + (size_t)(8 * t + g) * 8 + 2 * t4;
                y[0] -= d0 + e0;
                y[1] -= d1 + e1;
            }
            __syncthreads();
        }
    for (int e = threadIdx.x; e < 8 * m; e += blockDim.x) {
        const int r = e >> 3, c = c0 + (e & 7);
        if (c < p) W[(size_t)(s + r) * p + c] = ysm[e];
    }
}
static size_t tail_solve_smem(int mp) { return sizeof(double) * (8 * (size_t)mp + kNB * kTS); }

// ------------------------------------------------------------------------------------
// front sweeps of row-major blocks as a data flow
// ------------------------------------------------------------------------------------
// Rows in level order, a warp per row and group of 32 CPL columns (blockIdx.y; groups are
// independent of one another), position q to warp q mod W (all warps resident).  The values of Z start
// pending (pending.cuh); a row reads the rows it needs, eight in flight, those that are there longest
// first; polls what is not there yet (one word, then its own), and writes its result:
// Z_i = (B_{bperm(i)} - sum a Z_c) dinv.  Groups of 64 columns and not whole rows of 256: twice the
// rows in flight for half the registers (25,000 buses, 256 columns, backward: 4.6 ms with two rows in
// flight and the entries in column order).
template <int CPL>
__global__ void __launch_bounds__(512)
lu_sweep_wide_kernel(TriKernelArgs t, int p, const double *__restrict__ B, const int *__restrict__ bperm, double *Z,
                     DevStatus *ds) {
    constexpr int U = 8;   // entries whose rows are in flight at once
    const int lane = threadIdx.x & 31, wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nw = gridDim.x * (blockDim.x >> 5), col = 32 * CPL * blockIdx.y + lane;
    const long long lim = ds->wait_limit > 0 ? ds->wait_limit : kSpinLimit;
    for (int q = wid; q < t.n; q += nw) {
        const int i = __ldg(t.rows + q), rs = __ldg(t.rp + q), re = __ldg(t.rp + q + 1);
        const size_t bi = bperm ? __ldg(bperm + i) : i;
        double acc[CPL];
#pragma unroll
        for (int j = 0; j < CPL; j++) acc[j] = col + 32 * j < p ? __ldcg(B + bi * p + col + 32 * j) : 0.0;
        for (int kb = rs; kb < re; kb += 32) {
            int c = 0;
            double a = 0.0;
            if (kb + lane < re) {
                c = __ldg(t.ci + kb + lane);
                a = __ldg(t.val + kb + lane);
            }
            const int cnt = min(32, re - kb);
            for (int s0 = 0; s0 < cnt; s0 += U) {
                double v[U][CPL];
                unsigned miss = 0;   // entries with a pending value in some lane
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const double *row = Z + (size_t)__shfl_sync(0xffffffffu, c, min(s0 + u, cnt - 1)) * p;
#pragma unroll
                    for (int j = 0; j < CPL; j++) v[u][j] = col + 32 * j < p ? ld_value(row + col + 32 * j) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    bool m = false;
#pragma unroll
                    for (int j = 0; j < CPL; j++) m = m || is_pending(v[u][j]);
                    if (__any_sync(0xffffffffu, m)) miss |= 1u << u;
                }
                for (long long it = 0; miss; it++) {
                    bool ok = it <= lim;
                    if ((it & 31) == 31) ok = ok && ld_relaxed_i32(&ds->err) == 0;
                    if (!__all_sync(0xffffffffu, ok)) {
                        if (lane == 0) atomicCAS(&ds->err, 0, (int)DEV_BARRIER_TIMEOUT);
                        return;
                    }
                    // one word of the first missing row, until it is there; then the lanes' own words
                    const int f = __ffs(miss) - 1;
                    const double *row = Z + (size_t)__shfl_sync(0xffffffffu, c, min(s0 + f, cnt - 1)) * p;
                    if (is_pending(ld_value(row + 32 * CPL * blockIdx.y))) {
                        __nanosleep(20);
                        continue;
                    }
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if ((miss >> u) & 1u) {
                            const double *r = Z + (size_t)__shfl_sync(0xffffffffu, c, min(s0 + u, cnt - 1)) * p;
                            bool m = false;
#pragma unroll
                            for (int j = 0; j < CPL; j++) {
                                if (is_pending(v[u][j])) v[u][j] = ld_value(r + col + 32 * j);
                                m = m || is_pending(v[u][j]);
                            }
                            if (!__any_sync(0xffffffffu, m)) miss &= ~(1u << u);
                        }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const double as = __shfl_sync(0xffffffffu, a, min(s0 + u, cnt - 1));
                    if (s0 + u < cnt) {
#pragma unroll
                        for (int j = 0; j < CPL; j++) acc[j] -= as * v[u][j];
                    }
                }
            }
        }
        const double dv = t.dinv ? __ldg(t.dinv + q) : 1.0;
#pragma unroll
        for (int j = 0; j < CPL; j++)
            if (col + 32 * j < p) __stcg(Z + (size_t)i * p + col + 32 * j, not_pending(acc[j] * dv));
    }
}

// The same for narrow blocks (p <= NP): lanes over a row's entries, a warp sum per column.
template <int NP>
__global__ void __launch_bounds__(512)
lu_sweep_narrow_kernel(TriKernelArgs t, int p, const double *__restrict__ B, const int *__restrict__ bperm, double *Z,
                       DevStatus *ds) {
    const int lane = threadIdx.x & 31, wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nw = gridDim.x * (blockDim.x >> 5);
    const long long lim = ds->wait_limit > 0 ? ds->wait_limit : kSpinLimit;
    for (int q = wid; q < t.n; q += nw) {
        const int i = __ldg(t.rows + q), rs = __ldg(t.rp + q), re = __ldg(t.rp + q + 1);
        const size_t bi = bperm ? __ldg(bperm + i) : i;
        const double dv = t.dinv ? __ldg(t.dinv + q) : 1.0;
        const double b = lane < p ? __ldcg(B + bi * p + lane) : 0.0;
        double acc[NP];
#pragma unroll
        for (int j = 0; j < NP; j++) acc[j] = 0.0;
        bool ok = true;
        for (int k = rs + lane; k < re; k += 32) {
            const double *row = Z + (size_t)__ldg(t.ci + k) * p;
            const double a = __ldg(t.val + k);
            double v[NP];
#pragma unroll
            for (int j = 0; j < NP; j++) v[j] = j < p ? ld_value(row + j) : 0.0;
#pragma unroll
            for (int j = 0; j < NP; j++) {
                if (j < p && is_pending(v[j])) ok = poll_value(row + j, v[j], lim, ds) && ok;
                acc[j] += a * v[j];
            }
        }
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) atomicCAS(&ds->err, 0, (int)DEV_BARRIER_TIMEOUT);
            return;
        }
        double x = 0.0;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const double sum = warp_sum(acc[j]);
            if (lane == j) x = sum;
        }
        if (lane < p) __stcg(Z + (size_t)i * p + lane, not_pending((b - x) * dv));
    }
}

// Column-major -> row-major, and len values of `mark` set pending on the way.
__global__ void lu_in_kernel(int n, int p, const double *__restrict__ src, int ld, double *__restrict__ dst,
                             double *__restrict__ mark, size_t len) {
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (r < n && c < p) tile[j][threadIdx.x] = src[(size_t)c * ld + r];
    }
    const size_t nt = (size_t)gridDim.x * gridDim.y * 256,
                 id = ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 256 + threadIdx.y * 32 + threadIdx.x;
    for (size_t e = id; e < len; e += nt) mark[e] = pending_value();
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        if (r < n && c < p) dst[(size_t)r * p + c] = tile[threadIdx.x][j];
    }
}

// Row-major rows rowof(r) -> column-major rows r.
__global__ void lu_out_kernel(int n, int p, const double *__restrict__ src, const int *__restrict__ rowof,
                              double *__restrict__ dst, int ld) {
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        if (r < n && c < p) tile[j][threadIdx.x] = src[(size_t)__ldg(rowof + r) * p + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (r < n && c < p) dst[(size_t)c * ld + r] = tile[threadIdx.x][j];
    }
}

// ------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------
bpf_status lu_factor(bpf_ctx *ctx, bpf_prec *P, const double *vals) {
    bool taken = false;
    if (P->n == 0) return BPF_SUCCESS;
    BPF_TRY(factor_df(ctx, P, P->forder, P->nshort, vals, &taken));
    if (!taken) return set_error(ctx, BPF_ERR_NOT_SUPPORTED, "LU refactorization: a row of %d entries", P->max_row);
    const int nb = P->tail_mp / kNB, count = P->nlong + P->tail_m;
    if (count > 0) {
        CtaRowsArgs a{count, P->tail_s, P->tail_m, P->tail_mp, P->cta_nmax, P->cta_wmax, P->forder + P->nshort, P->rp, P->ci, P->diag,
                      P->fend, P->fsrc, P->pp, P->pdst, vals, P->fv, P->tail_S, sweep_store(P), ctx->dstat};
        const size_t smem = cta_rows_smem(P->cta_nmax, P->cta_wmax);
        BPF_CUDA(ctx, cudaFuncSetAttribute(lu_cta_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        BPF_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lu_cta_rows_kernel, 256, smem));
        if (per_sm < 1) return set_error(ctx, BPF_ERR_CUDA, "LU rows do not fit on an SM");
        void *args[] = {&a};
        KScope ks(ctx, BPF_KC_FACTOR, 12.0 * P->cta_pairs + 8.0 * P->tail_m * (double)P->tail_mp, 2.0 * P->cta_pairs);
        BPF_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)lu_cta_rows_kernel, dim3(std::min(per_sm * ctx->num_sms, count)),
                                                  dim3(256), args, smem, ctx->stream));
        BPF_LAUNCHED(ctx);
    }
    if (nb == 0) return BPF_SUCCESS;
    BPF_CUDA(ctx, cudaFuncSetAttribute(lu_tail_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTailFactorSmem));
    // at most a tile each in the first step; one CTA fills an SM's shared memory
    const int grid = std::min(ctx->num_sms, std::max(1, (nb - 1) * (nb - 1)));
    double *S = P->tail_S, *F = P->tail_F, *D = P->tail_D, *R = D + (size_t)nb * kNB * kNB;
    int row0 = P->tail_s, nbv = nb;
    DevStatus *ds = ctx->dstat;
    void *args[] = {&nbv, &S, &F, &D, &R, &row0, &ds};
    const double m = P->tail_mp;
    KScope ks(ctx, BPF_KC_FACTOR, 16.0 * m * m, 2.0 / 3.0 * m * m * m);
    BPF_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)lu_tail_factor_kernel, dim3(grid), dim3(256), args,
                                              kTailFactorSmem, ctx->stream));
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

static bpf_status lu_sweep(bpf_ctx *ctx, const TriDev &t, int p, const double *B, const int *bperm, double *Z) {
    if (t.n == 0) return BPF_SUCCESS;
    TriKernelArgs a = t.args();
    DevStatus *ds = ctx->dstat;
    void *args[] = {&a, &p, (void *)&B, (void *)&bperm, &Z, &ds};
    const void *kern = p <= 1    ? (const void *)lu_sweep_narrow_kernel<1>
                       : p <= 4  ? (const void *)lu_sweep_narrow_kernel<4>
                       : p <= 8  ? (const void *)lu_sweep_narrow_kernel<8>
                       : p <= 32 ? (const void *)lu_sweep_wide_kernel<1>
                                 : (const void *)lu_sweep_wide_kernel<2>;
    int per_sm = 0;
    BPF_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 512, 0));
    if (per_sm < 1) return set_error(ctx, BPF_ERR_CUDA, "LU sweep does not fit on an SM");
    const int groups = p <= 32 ? 1 : ceil_div(p, 64);
    const dim3 grid(std::max(1, std::min(per_sm * ctx->num_sms / groups, ceil_div(t.n, 16))), groups);
    KScope ks(ctx, BPF_KC_TRSV, 12.0 * t.nnz + 16.0 * t.n + 16.0 * (double)t.n * p, 2.0 * ((double)t.nnz + t.n) * p);
    BPF_CUDA(ctx, cudaLaunchCooperativeKernel(kern, grid, dim3(512), args, 0, ctx->stream));
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

bpf_status lu_solve(bpf_ctx *ctx, const bpf_prec *P, int nrhs, double *X, int ldx) {
    const int n = P->n;
    if (n == 0 || nrhs == 0) return BPF_SUCCESS;
    if (P->col) return trsv_col(ctx, P, nrhs, X, ldx, X, ldx);
    const int chunk = 256, nb = P->tail_mp / kNB, s = P->tail_s;
    bpf_status st;
    double *buf = (double *)ws_get(ctx, WS_A, sizeof(double) * 3 * (size_t)n * std::min(nrhs, chunk), &st);
    if (!buf) return st;
    const size_t tail_smem = tail_solve_smem(P->tail_mp);
    BPF_CUDA(ctx, cudaFuncSetAttribute(lu_tail_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tail_smem));
    for (int c0 = 0; c0 < nrhs; c0 += chunk) {
        const int p = std::min(chunk, nrhs - c0);
        double *B = buf, *Z = buf + (size_t)n * p, *W = Z + (size_t)n * p, *Xc = X + (size_t)c0 * ldx;
        const dim3 grid(ceil_div(n, 32), ceil_div(p, 32)), block(32, 8);
        lu_in_kernel<<<grid, block, 0, ctx->stream>>>(n, p, Xc, ldx, B, Z, 2 * (size_t)n * p);
        BPF_LAUNCHED(ctx);
        BPF_TRY(lu_sweep(ctx, P->lower, p, B, P->pos0, Z));
        if (nb > 0) {
            KScope ks(ctx, BPF_KC_TRSV, 8.0 * P->tail_mp * P->tail_mp + 16.0 * P->tail_m * (double)p,
                      2.0 * P->tail_mp * (double)P->tail_mp * p);
            lu_tail_solve_kernel<<<ceil_div(p, 8), kTailSolveThreads, tail_smem, ctx->stream>>>(
                s, P->tail_m, nb, P->tail_F, P->tail_D, P->tail_D + (size_t)nb * kNB * kNB, p, Z, W);
            BPF_LAUNCHED(ctx);
        }
        BPF_TRY(lu_sweep(ctx, P->upper, p, Z, nullptr, W));
        lu_out_kernel<<<grid, block, 0, ctx->stream>>>(n, p, W, P->pos1, Xc, ldx);
        BPF_LAUNCHED(ctx);
    }
    return BPF_SUCCESS;
}

// Update pairs of the rows a CTA takes (`cta`; of a tail row, the L entries before column s), of a
// pattern closed under elimination: every U entry (k, j) of an L entry (i, k) gives a destination from
// row i's storage start rp[i] on (a tail row's columns from s on are dense after its entries before s).
// False if they exceed INT_MAX.
static bool lu_pairs(int n, int s, const std::vector<int> &rp, const std::vector<int> &ci, const std::vector<int> &diag,
                     const std::vector<int> &fend, const std::vector<char> &cta, std::vector<int> &pp, PairVec &pdst) {
    pp.assign(rp[n] + 1, 0);
    long long total = 0;
    for (int i = 0; i < n; i++) {
        const int end = !cta[i] ? rp[i] : i < s ? diag[i] : fend[i];
        for (int e = rp[i]; e < rp[i + 1]; e++) {
            if (e < end) total += rp[ci[e] + 1] - diag[ci[e]] - 1;
            if (total > 2147483647ll) return false;
            pp[e + 1] = (int)total;
        }
    }
    pdst.resize(total);
    std::atomic<int> next(0);
    run_threads(total >= 200000, [&]() {
        std::vector<int> pos(n, -1);
        for (;;) {
            const int b = next.fetch_add(64);
            if (b >= n) break;
            for (int i = b; i < std::min(n, b + 64); i++) {
                if (!cta[i]) continue;
                const int end = i < s ? diag[i] : fend[i];
                for (int k = rp[i]; k < rp[i + 1]; k++) pos[ci[k]] = (i < s || k < end) ? k : end + ci[k] - s;
                for (int e = rp[i]; e < end; e++) {
                    int w = pp[e];
                    for (int j = diag[ci[e]] + 1; j < rp[ci[e] + 1]; j++) pdst[w++] = pos[ci[j]];
                }
            }
        }
    });
    return true;
}

// Set up the front / tail form of the L + U pattern (rp, ci, diag; pivot-step numbering; fsrc: source
// entry of A per pattern entry, -1 for fill; rowP / colQ: original row and column of each step).
// *fits = false, and nothing made, when its update pairs would exceed INT_MAX.
bpf_status lu_setup(bpf_ctx *ctx, int n, const std::vector<int> &rp, const std::vector<int> &ci,
                    const std::vector<int> &diag, const std::vector<int> &fsrc, const std::vector<int> &rowP,
                    const std::vector<int> &colQ, bool *fits, bpf_prec **out) {
    *fits = true;
    *out = nullptr;
    // forward levels of every row (dependencies: its L entries)
    std::vector<int> lev(n, 0), pre(n + 1, 0);   // pre[s]: levels of the rows before s
    for (int i = 0; i < n; i++) {
        for (int k = rp[i]; k < diag[i]; k++) lev[i] = std::max(lev[i], lev[ci[k]] + 1);
        pre[i + 1] = std::max(pre[i], lev[i] + 1);
    }
    auto back = [&](int s, std::vector<int> &bl) {   // backward levels of the rows before s
        bl.assign(n, 0);
        int nl = 0;
        for (int i = s - 1; i >= 0; i--) {
            for (int k = diag[i] + 1; k < rp[i + 1]; k++)
                if (ci[k] < s) bl[i] = std::max(bl[i], bl[ci[k]] + 1);
            nl = std::max(nl, bl[i] + 1);
        }
        return nl;
    };
    // Tail size: estimated microseconds of the levels (1.5 a level in the factorization, and in each
    // sweep 0.4 in shared memory or 1.5 through L2) against the dense block (28 a 64-column step of
    // factorization and solve, and its tiles 7 each over the SMs).
    bool col = n > 0 && trsv_col_fits(ctx, n, BPF_F64);
    std::vector<int> bl;
    int best = 0;
    double best_us = -1.0;
    for (int m : {0, 64, 128, 192, 256, 384, 512, 640, 768, 1024, 1280, 1536, 2048, 2560, 3072}) {
        if (m > 0 && m - 63 > n) break;
        const int s = std::max(0, n - m), nb = m / kNB;
        const double us = 1.5 * pre[s] + (col ? 0.4 : 1.5) * (pre[s] + back(s, bl)) + 28.0 * nb +
                          7.0 * nb * (double)nb * nb / (3.0 * ctx->num_sms);
        if (best_us < 0.0 || us < best_us) {
            best_us = us;
            best = m;
        }
    }
    const int mp = best, s = std::max(0, n - mp), m = n - s;
    std::vector<int> fend(n, 0);   // end of a row's entries before column s
    for (int i = 0; i < n; i++)
        fend[i] = (int)(std::lower_bound(ci.begin() + rp[i], ci.begin() + rp[i + 1], s) - ci.begin());
    // rows a CTA takes: the tail's, front rows with a long U part or too many entries for gather lists,
    // and the rows that depend on those
    std::vector<char> cta(n, 0);
    long long warp_pairs = 0;   // update pairs of the other rows
    for (int i = 0; i < n; i++) {
        cta[i] = i >= s || rp[i + 1] - diag[i] > kCtaRow || rp[i + 1] - rp[i] > kGatherRow;
        for (int k = rp[i]; k < diag[i] && !cta[i]; k++) cta[i] = cta[ci[k]];
        for (int k = rp[i]; k < diag[i] && !cta[i]; k++) warp_pairs += rp[ci[k] + 1] - diag[ci[k]] - 1;
    }
    if (!gather_fits(gather_ints(s, rp, diag, cta), warp_pairs)) cta.assign(n, 1);
    int nmax = 0, wmax = 0;
    for (int i = 0; i < n; i++) {
        const int len = rp[i + 1] - rp[i];
        if (!cta[i]) continue;
        nmax = std::max(nmax, i < s ? diag[i] - rp[i] : fend[i] - rp[i]);
        wmax = std::max(wmax, i < s ? len : fend[i] - rp[i] + mp);
    }
    std::vector<int> pp;
    std::vector<long long> goff;
    PairVec pdst, gsrc;
    if (cta_rows_smem(nmax, wmax) + 1024 > (size_t)ctx->max_smem_optin || !lu_pairs(n, s, rp, ci, diag, fend, cta, pp, pdst)) {
        *fits = false;
        return BPF_SUCCESS;
    }
    const long long gathered = build_gather(s, rp, ci, diag, cta, goff, gsrc);
    // sweep schedules: forward the front's levels then the tail's rows as one more, over columns
    // before s; backward the front's rows only
    TriHost lo, up;
    const int nbl = back(s, bl);
    auto build = [&](TriHost &t, int rows, int nlev, const std::vector<int> &lv, bool lower) {
        t.n = rows;
        t.nlev = nlev;
        t.unit = lower;
        t.keep_last = lower && m > 0;
        t.lev_ptr.assign(nlev + 1, 0);
        auto level = [&](int i) { return i < s ? lv[i] : nlev - 1; };
        for (int i = 0; i < rows; i++) t.lev_ptr[level(i) + 1]++;
        for (int l = 0; l < nlev; l++) {
            t.max_level_rows = std::max(t.max_level_rows, t.lev_ptr[l + 1]);
            t.lev_ptr[l + 1] += t.lev_ptr[l];
        }
        t.rows.resize(rows);
        std::vector<int> fill(t.lev_ptr.begin(), t.lev_ptr.end() - 1);
        for (int i = 0; i < rows; i++) t.rows[fill[level(i)]++] = i;
        t.rp.assign(rows + 1, 0);
        for (int q = 0; q < rows; q++) {
            const int i = t.rows[q], b = lower ? rp[i] : diag[i] + 1, e = lower ? (i < s ? diag[i] : fend[i]) : rp[i + 1];
            for (int u = b; u < e; u++) {   // what is there longest first: backward, the last column
                const int k = lower ? u : e - 1 - (u - b);
                t.ci.push_back(ci[k]);
                t.map.push_back(k);
            }
            t.rp[q + 1] = (int)t.ci.size();
            if (!lower) t.dmap.push_back(diag[i]);
        }
    };
    build(lo, n, pre[s] + (m > 0 ? 1 : 0), lev, true);
    build(up, s, nbl, bl, false);

    bpf_prec *P = new bpf_prec();
    P->ctx = ctx;
    P->kind = PREC_LU;
    P->n = n;
    P->nnz = n > 0 ? rp[n] : 0;
    P->npairs = gathered;
    P->cta_pairs = (long long)pdst.size();
    P->cta_nmax = nmax;
    P->cta_wmax = wmax;
    P->tail_s = s;
    P->tail_m = m;
    P->tail_mp = mp;
    std::vector<int> forder, flong;   // dependencies first: short rows by level, long ones by level, the tail
    for (int i : lo.rows) {
        if (cta[i]) {
            flong.push_back(i);
            if (i < s) P->nlong++;
        } else {
            forder.push_back(i);
            P->max_row = std::max(P->max_row, rp[i + 1] - rp[i]);
        }
    }
    P->nshort = (int)forder.size();
    forder.insert(forder.end(), flong.begin(), flong.end());
    auto fail = [&](bpf_status e) {
        cudaStreamSynchronize(ctx->stream);
        bpf_prec_destroy(P);
        return e;
    };
    std::vector<int> pos0, pos1, pos01(n), tpos[2];
    TriStream cs[2];
    tpos[0].assign(P->nnz, -1);
    tpos[1].assign(P->nnz, -1);
    if (col) {
        const int nring = trsv_col_ring(ctx, n, BPF_F64);
        col = tri_to_stream(lo, BPF_F64, nring, 0, n, true, pos0, cs[0], tpos[0]) &&
              tri_to_stream(up, BPF_F64, nring, (int)cs[0].coff.size() - 1, n, true, pos1, cs[1], tpos[1]);
    }
    P->col = col;
    P->lev = !col;
    if (col) {
        for (int q = 0; q < n; q++) pos01[q] = q < s ? pos0[up.rows[q]] : q;
        std::vector<int> b0(n), b1(n);   // positions of the block's rows
        for (int i = 0; i < n; i++) {
            b0[rowP[i]] = pos0[i];
            b1[colQ[i]] = pos1[i];
        }
        pos0.swap(b0);
        pos1.swap(b1);
    } else {
        for (int w = 0; w < 2; w++) {
            const TriHost &t = w == 0 ? lo : up;
            std::fill(tpos[w].begin(), tpos[w].end(), -1);
            for (size_t k = 0; k < t.map.size(); k++) tpos[w][t.map[k]] = (int)k;
            for (size_t q = 0; q < t.dmap.size(); q++) tpos[w][t.dmap[q]] = -2 - (int)q;
        }
        pos0 = rowP;   // rows of the right-hand sides, and steps of the solution's rows
        pos1.resize(n);
        for (int i = 0; i < n; i++) pos1[colQ[i]] = i;
    }
    bpf_status st;
    if ((st = tri_upload(ctx, lo, P->lower, !col)) != BPF_SUCCESS) return fail(st);
    if ((st = tri_upload(ctx, up, P->upper, !col)) != BPF_SUCCESS) return fail(st);
    cudaError_t e = cudaSuccess;
    auto up_v = [&](auto **d, const auto &h) {
        if (e != cudaSuccess || h.empty()) return;
        e = cudaMalloc((void **)d, sizeof(h[0]) * h.size());
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(*d, h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice, ctx->stream);
    };
    up_v(&P->rp, rp);
    up_v(&P->ci, ci);
    up_v(&P->diag, diag);
    up_v(&P->fend, fend);
    up_v(&P->fsrc, fsrc);
    up_v(&P->pp, pp);
    up_v(&P->pdst, pdst);
    up_v(&P->forder, forder);
    up_v(&P->goff, goff);
    up_v(&P->gsrc, gsrc);
    up_v(&P->pos0, pos0);
    up_v(&P->pos1, pos1);
    if (col) up_v(&P->pos01, pos01);
    up_v(&P->tpos[0], tpos[0]);
    up_v(&P->tpos[1], tpos[1]);
    if (col)
        for (int w = 0; w < 2; w++) {
            P->cs[w].nchunk = (int)cs[w].coff.size() - 1;
            P->cs[w].nslab = cs[w].cslab.back();
            P->cs[w].nstage = cs[w].nstage;
            P->cs[w].diag = cs[w].diag;
            P->cs[w].len = cs[w].bytes.size();
            up_v(&P->cs[w].coff, cs[w].coff);
            up_v(&P->cs[w].cslab, cs[w].cslab);
            up_v(&P->cs[w].head, cs[w].head);
            up_v(&P->cs[w].bytes, cs[w].bytes);
        }
    if (mp > 0) {
        const size_t tail_bytes = sizeof(double) * (size_t)mp * mp;
        if (e == cudaSuccess) e = cudaMalloc((void **)&P->tail_S, tail_bytes);
        if (e == cudaSuccess) e = cudaMalloc((void **)&P->tail_F, tail_bytes);
        if (e == cudaSuccess) e = cudaMemsetAsync(P->tail_F, 0, tail_bytes, ctx->stream);
        if (e == cudaSuccess) e = cudaMalloc((void **)&P->tail_D, sizeof(double) * (size_t)mp * (kNB + 1));
    }
    if (e == cudaSuccess && P->nnz > 0) e = cudaMalloc((void **)&P->fv, sizeof(double) * P->nnz);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // host vectors die on return
    if (e != cudaSuccess) return fail(cuda_error(ctx, e, "LU setup", __FILE__, __LINE__));
    *out = P;
    return BPF_SUCCESS;
}

}  // namespace bpf
