// One block-Arnoldi orthogonalization in one launch (blocks of up to 32 columns).
//
// Reference: src/block_gmres.jl:301-316 (block Gram-Schmidt against the basis, QR of the new block).
//
// Bound: with narrow blocks, launches.  An iteration's two Gram-Schmidt passes, Cholesky-QR2, its
// third pass and the re-orthogonalization of an ill-conditioned block were 38 kernels, 25 of them
// gated off nearly always, 3-13 us each: 300 us an iteration of a 300-bus solve with 16 columns,
// whose arithmetic is worth a few.  Here they are one cooperative launch: a CTA keeps its rows of the
// new block W in shared memory from the first product to the finished basis block, and what CTAs
// exchange are p x p partial sums through global memory, one grid barrier each (seven an iteration).
//
//  * Products V_j^T W: a warp per basis block over the CTA's rows, FP64 tensor pipe (m8n8k4).  A pass'
//    partial sums are added over the CTAs element by element by all threads, in a fixed order.
//  * Update W -= sum_j V_j Psi_j: 16 rows a warp, or the blocks j split over warps where rows are few.
//  * Cholesky-QR: every CTA sums the partial Gram matrices and factors them itself, identically, so the
//    rare decisions (shift, third pass, re-orthogonalization, breakdown) need no further exchange.
//
// Same algorithm and decisions as gram / tsmm / cholqr / reorth_fold (dense.cu, small.cu); the sums are
// grouped differently, so results agree to rounding.
//
// Measured, a whole solve per iteration, kernel by kernel -> one launch: 300 buses 8 columns 418 -> 119 us,
// 24 columns 560 -> 189; 1500 buses 16 columns 599 -> 173; 9000 buses 8 columns 1981 -> 410 (long basis), 32
// columns 1436 -> 742; 70000 buses 8 columns 2258 -> 1057.  With few columns now bound by the latency of a
// product's 100 to 200 basis blocks a warp at a time, with 32 by HBM and the tensor pipe in turn (13 TFLOP/s).
// Loads one step ahead and as pairs of columns, coefficients in shared memory, the update's order reversed and
// four lanes an element of a sum took 9000 buses 8 columns from 547 to 410 us, 32 columns from 926 to 742.
#include <algorithm>

#include "arnoldi.cuh"
#include "bpf_internal.cuh"
#include "dense.cuh"

namespace bpf {

struct ArnoldiArgs {
    int n, p, k, rows;   // rows: of a CTA
    const double *V;     // k blocks of n x p
    size_t strideV;
    const double *Q;     // the new block (row-major)
    double *Vn;          // the finished basis block
    double *Psi, *Psi2;  // k blocks p x p: coefficients, and those of a second pass
    double *C;           // p x p: R of the new block
    double *part;        // gridDim.x blocks of group p^2 partial sums
    int group;           // basis blocks whose products are in flight at a time
    double *gsum;        // p^2
    SolveState *st;
    int *snap;           // the grid's decision to skip, by epoch
    int epoch;
    DevStatus *ds;
};

constexpr int kArnoldiWarps = 8;

__device__ __forceinline__ void arn_dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Blocks of coefficients that one step of the update takes.
__host__ __device__ constexpr int arn_step(int nt) { return nt == 1 ? 4 : nt == 2 ? 3 : nt == 3 ? 2 : 1; }
__host__ __device__ constexpr int arn_buf(int nt) {
    const int pt = 8 * nt, warps = kArnoldiWarps * pt * pt, coef = 2 * arn_step(nt) * pt * (pt + 2);
    return warps > coef ? warps : coef;
}

// The shared-memory pieces of a CTA.
template <int NT>
struct ArnoldiSmem {
    static constexpr int PT = 8 * NT, LW = PT + 4, LG = PT + 1;
    double *w;      // rows x LW: the CTA's rows of the block
    double *buf;    // arn_buf(NT): partial results of warps (kArnoldiWarps x PT^2 or 8 PT), or two steps' coefficients
    double *g, *x, *r, *t;   // PT x LG: Gram matrix / R^{-T}, inverse, accumulated R, scratch
    double *dref, *rs;
};

// Two adjacent values of a row at column c (zero beyond p): one 16-byte load where rows are 16-byte aligned.
template <bool EVEN>
__device__ __forceinline__ double2 arn_load2(const double *row, int c, int p, bool ok) {
    double2 v = make_double2(0.0, 0.0);
    if (EVEN) {
        if (ok && c < p) v = __ldcg(reinterpret_cast<const double2 *>(row + c));
    } else {
        if (ok && c < p) v.x = __ldcg(row + c);
        if (ok && c + 1 < p) v.y = __ldcg(row + c + 1);
    }
    return v;
}

// Partial sums of V_j^T W over the CTA's rows, j < nb: part[j].  A warp per j; the next 4 U rows of V (of
// this j or the warp's next) are on their way while these are multiplied.  Lane (g, t4) takes columns 16 mp
// + 2 g + {0, 1} of row t4 as one load: the two are the same row of two tiles' A fragments.
template <int NT, bool EVEN>
__device__ __forceinline__ void arn_gram(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, const double *A, int nb,
                                         double *part) {
    constexpr int LW = ArnoldiSmem<NT>::LW, U = NT == 1 ? 10 : NT == 2 ? 8 : 4, MP = (NT + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p;
    const size_t pp = (size_t)p * p;
    if (warp >= nb) return;
    double acc[2 * MP][NT][2];
#pragma unroll
    for (int mi = 0; mi < 2 * MP; mi++)
#pragma unroll
        for (int ni = 0; ni < NT; ni++) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
    double2 cur[U][MP], nxt[U][MP];
    auto load = [&](double2 (&v)[U][MP], int j, int k0) {
        const double *Aj = A + (size_t)j * a.strideV;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int lr = k0 + 4 * u, r = r0 + lr + t4;
            const bool ok = lr < a.rows && r < a.n;
#pragma unroll
            for (int mp = 0; mp < MP; mp++) v[u][mp] = arn_load2<EVEN>(Aj + (size_t)r * p, 16 * mp + 2 * g, p, ok);
        }
    };
    load(cur, warp, 0);
    for (int j = warp, k0 = 0; j < nb;) {
        int jn = j, kn = k0 + 4 * U;
        if (kn >= a.rows) {
            kn = 0;
            jn += kArnoldiWarps;
        }
        if (jn < nb) load(nxt, jn, kn);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (k0 + 4 * u >= a.rows) break;
            double bv[NT];
#pragma unroll
            for (int ni = 0; ni < NT; ni++) bv[ni] = s.w[(k0 + 4 * u + t4) * LW + 8 * ni + g];
#pragma unroll
            for (int mp = 0; mp < MP; mp++)
#pragma unroll
                for (int ni = 0; ni < NT; ni++) {
                    arn_dmma(acc[2 * mp][ni][0], acc[2 * mp][ni][1], cur[u][mp].x, bv[ni]);
                    arn_dmma(acc[2 * mp + 1][ni][0], acc[2 * mp + 1][ni][1], cur[u][mp].y, bv[ni]);
                }
        }
        if (jn != j) {
#pragma unroll
            for (int mi = 0; mi < 2 * MP; mi++)
#pragma unroll
                for (int ni = 0; ni < NT; ni++)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int row = 16 * (mi / 2) + 2 * g + (mi & 1), col = 8 * ni + 2 * t4 + i;
                        if (row < p && col < p) part[j * pp + (size_t)row * p + col] = acc[mi][ni][i];
                        acc[mi][ni][i] = 0.0;
                    }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int mp = 0; mp < MP; mp++) cur[u][mp] = nxt[u][mp];
        j = jn;
        k0 = kn;
    }
}

// W -= sum_j V_j S_j on the CTA's rows (ends with a barrier).  Eight row tiles or more: a warp takes two of
// them at a time, the coefficients of JB blocks a step come through shared memory (every warp reading them
// from L2 was four times the basis' bytes), V's next blocks are on their way while these are multiplied.  From
// the last block to the first: the products before went the other way, so L2 holds the last ones, and this
// leaves the first ones for the next products.  Lane (g, t4) takes columns 8 kk + 2 t4 + {0, 1} of row g as one
// load: the two are two k-steps' A fragments.
template <int NT, bool EVEN>
__device__ __forceinline__ void arn_update(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, const double *S) {
    constexpr int PT = ArnoldiSmem<NT>::PT, LW = ArnoldiSmem<NT>::LW, LS = PT + 2, JB = arn_step(NT);
    constexpr int ES = (JB * PT * PT + 255) / 256;   // coefficients a thread brings
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p;
    const size_t pp = (size_t)p * p;
    const int tiles = a.rows / 8;
    if (tiles >= kArnoldiWarps) {
        double *sb = s.buf;   // two steps of JB blocks of PT x LS
        for (int e = threadIdx.x; e < 2 * JB * PT * LS; e += 256) sb[e] = 0.0;   // the padding stays zero
        for (int t0 = warp; t0 - warp < tiles; t0 += 2 * kArnoldiWarps) {
            double acc[2][NT][2];
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int ni = 0; ni < NT; ni++) acc[q][ni][0] = acc[q][ni][1] = 0.0;
            double2 cur[JB][2][NT], nxt[JB][2][NT];
            double sv[ES];
            auto load = [&](double2 (&v)[JB][2][NT], int j0) {   // blocks j0 .. j0 + JB - 1, those below 0 as zeros
#pragma unroll
                for (int jb = 0; jb < JB; jb++)
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int t = t0 + q * kArnoldiWarps, r = r0 + 8 * t + g;
                        const bool ok = j0 + jb >= 0 && t < tiles && r < a.n;
                        const double *row = a.V + (size_t)(ok ? j0 + jb : 0) * a.strideV + (size_t)(ok ? r : 0) * p;
#pragma unroll
                        for (int kk = 0; kk < NT; kk++) v[jb][q][kk] = arn_load2<EVEN>(row, 8 * kk + 2 * t4, p, ok);
                    }
            };
            auto load_s = [&](int j0) {
#pragma unroll
                for (int u = 0; u < ES; u++) {
                    const int e = threadIdx.x + 256 * u, jb = e / (int)pp;
                    sv[u] = jb < JB && j0 + jb >= 0 ? __ldcg(S + j0 * (long long)pp + e) : 0.0;
                }
            };
            load(cur, a.k - JB);
            load_s(a.k - JB);
            for (int j0 = a.k - JB, step = 0; j0 > -JB; j0 -= JB, step ^= 1) {
                double *b = sb + step * JB * PT * LS;
                __syncthreads();   // the readers of the step before last are done (and, first, the zeros are there)
#pragma unroll
                for (int u = 0; u < ES; u++) {
                    const int e = threadIdx.x + 256 * u, jb = e / (int)pp, x = e - jb * (int)pp;
                    if (jb < JB) b[jb * PT * LS + (x / p) * LS + x % p] = sv[u];
                }
                if (j0 > 0) {
                    load(nxt, j0 - JB);
                    load_s(j0 - JB);
                }
                __syncthreads();
#pragma unroll
                for (int jb = 0; jb < JB; jb++)
#pragma unroll
                    for (int kk = 0; kk < NT; kk++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            double bv[NT];
#pragma unroll
                            for (int ni = 0; ni < NT; ni++) bv[ni] = b[jb * PT * LS + (8 * kk + 2 * t4 + h) * LS + 8 * ni + g];
#pragma unroll
                            for (int q = 0; q < 2; q++)
#pragma unroll
                                for (int ni = 0; ni < NT; ni++)
                                    arn_dmma(acc[q][ni][0], acc[q][ni][1], h ? cur[jb][q][kk].y : cur[jb][q][kk].x, bv[ni]);
                        }
#pragma unroll
                for (int jb = 0; jb < JB; jb++)
#pragma unroll
                    for (int q = 0; q < 2; q++)
#pragma unroll
                        for (int kk = 0; kk < NT; kk++) cur[jb][q][kk] = nxt[jb][q][kk];
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int t = t0 + q * kArnoldiWarps;
                if (t < tiles)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++)
#pragma unroll
                        for (int i = 0; i < 2; i++) s.w[(8 * t + g) * LW + 8 * ni + 2 * t4 + i] -= acc[q][ni][i];
            }
            __syncthreads();
        }
        return;
    }
    // few rows: the blocks j split over the warps of a tile
    const int split = kArnoldiWarps / tiles, share = warp / tiles;
    if (warp < tiles * split) {
        const int t = warp % tiles, r = r0 + 8 * t + g;
        double acc[NT][2];
#pragma unroll
        for (int ni = 0; ni < NT; ni++) acc[ni][0] = acc[ni][1] = 0.0;
        for (int j = share; j < a.k; j += split) {
            const double *row = a.V + (size_t)j * a.strideV + (size_t)r * p, *Sj = S + j * pp;
            double2 av[NT];
            double bv[2 * NT][NT];
#pragma unroll
            for (int kk = 0; kk < NT; kk++) {
                av[kk] = arn_load2<EVEN>(row, 8 * kk + 2 * t4, p, r < a.n);
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++) {
                        const int c = 8 * kk + 2 * t4 + h;
                        bv[2 * kk + h][ni] = c < p && 8 * ni + g < p ? __ldcg(Sj + (size_t)c * p + 8 * ni + g) : 0.0;
                    }
            }
#pragma unroll
            for (int kk = 0; kk < NT; kk++)
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++) arn_dmma(acc[ni][0], acc[ni][1], h ? av[kk].y : av[kk].x, bv[2 * kk + h][ni]);
        }
#pragma unroll
        for (int ni = 0; ni < NT; ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int c = 8 * ni + 2 * t4 + i;
                if (split == 1) s.w[(8 * t + g) * LW + c] -= acc[ni][i];
                else s.buf[(size_t)warp * 8 * PT + g * PT + c] = acc[ni][i];
            }
    }
    __syncthreads();
    if (split > 1) {
        for (int e = threadIdx.x; e < a.rows * PT; e += 32 * kArnoldiWarps) {
            const int row = e / PT, c = e % PT;
            double v = 0.0;
            for (int q = 0; q < split; q++) v += s.buf[(size_t)(q * tiles + row / 8) * 8 * PT + (row % 8) * PT + c];
            s.w[row * LW + c] -= v;
        }
        __syncthreads();
    }
}

// Sum over the CTAs of element e of their partial sums; four lanes (8 apart) share an element's CTAs.
__device__ __forceinline__ double arn_total(const ArnoldiArgs &a, size_t len, size_t e) {
    double s = 0.0;
    if (e < len) {
        const double *q = a.part + e;
#pragma unroll 8
        for (unsigned c = (threadIdx.x >> 3) & 3; c < gridDim.x; c += 4) s += __ldcg(q + c * len);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    return s + __shfl_xor_sync(0xffffffffu, s, 16);
}

// f(e, total of e) for this CTA's share of the elements (all: every element).
template <class F>
__device__ __forceinline__ void arn_totals(const ArnoldiArgs &a, size_t len, bool all, F f) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (size_t e0 = ((all ? 0 : (size_t)blockIdx.x) * kArnoldiWarps + w) * 8; e0 < len;
         e0 += (size_t)(all ? 1 : gridDim.x) * kArnoldiWarps * 8) {
        const size_t e = e0 + (l & 7);
        const double v = arn_total(a, len, e);
        if (l < 8 && e < len) f(e, v);
    }
}

// One Gram-Schmidt pass: coefficients into out (and added to acc), W updated.  False: a barrier gave up.
template <int NT, bool EVEN>
__device__ __forceinline__ bool arn_project(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, double *out, double *acc,
                                            unsigned &gen, bool skip, bool check) {
    const size_t pp = (size_t)a.p * a.p;
    for (int j0 = 0; j0 < a.k; j0 += a.group) {
        const int nb = min(a.group, a.k - j0);
        const size_t len = nb * pp;
        if (!skip) arn_gram<NT, EVEN>(a, s, r0, a.V + (size_t)j0 * a.strideV, nb, a.part + blockIdx.x * len);
        if (!grid_barrier(a.ds, gen)) return false;
        if (check && *(volatile int *)a.snap == a.epoch) return false;   // some CTA saw the solve stopped
        arn_totals(a, len, false, [&](size_t e, double v) {
            out[j0 * pp + e] = v;
            if (acc) acc[j0 * pp + e] += v;
        });
        if (!grid_barrier(a.ds, gen)) return false;
    }
    arn_update<NT, EVEN>(a, s, r0, out);
    return true;
}

// One pass of Cholesky-QR on the CTAs' rows: s.r <- R s.r (first: R).  0: done; 1: a barrier gave up; 2:
// breakdown.  shift / ill: set when the pass needed the shift / lost more than eight digits.
template <int NT>
__device__ __forceinline__ int arn_cholqr(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, bool first, unsigned &gen,
                                          bool &shifted, bool *ill) {
    constexpr int PT = ArnoldiSmem<NT>::PT, LW = ArnoldiSmem<NT>::LW, LG = ArnoldiSmem<NT>::LG;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p, tid = threadIdx.x;
    const size_t pp = (size_t)p * p;
    // W^T W of the CTA's rows: the rows over the warps, their results added in order
    {
        double acc[NT][NT][2];
#pragma unroll
        for (int mi = 0; mi < NT; mi++)
#pragma unroll
            for (int ni = 0; ni < NT; ni++) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
        for (int k0 = 4 * warp; k0 < a.rows; k0 += 4 * kArnoldiWarps) {
            double v[NT];
#pragma unroll
            for (int ni = 0; ni < NT; ni++) v[ni] = s.w[(k0 + t4) * LW + 8 * ni + g];
#pragma unroll
            for (int mi = 0; mi < NT; mi++)
#pragma unroll
                for (int ni = 0; ni < NT; ni++) arn_dmma(acc[mi][ni][0], acc[mi][ni][1], v[mi], v[ni]);
        }
#pragma unroll
        for (int mi = 0; mi < NT; mi++)
#pragma unroll
            for (int ni = 0; ni < NT; ni++)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    s.buf[(size_t)warp * PT * PT + (8 * mi + g) * PT + 8 * ni + 2 * t4 + i] = acc[mi][ni][i];
        __syncthreads();
        for (int e = tid; e < p * p; e += 256) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < kArnoldiWarps; q++) v += s.buf[(size_t)q * PT * PT + (e / p) * PT + e % p];
            a.part[blockIdx.x * pp + e] = v;
        }
    }
    if (!grid_barrier(a.ds, gen)) return 1;
    // the sum over the CTAs: each its own, or, where that is much to read, shared out first
    const bool shared_out = pp * gridDim.x > 16384;
    if (shared_out) {
        arn_totals(a, pp, false, [&](size_t e, double v) { a.gsum[e] = v; });
        if (!grid_barrier(a.ds, gen)) return 1;
    }
    double trace = 0.0;
    if (shared_out)
        for (int e = tid; e < p * p; e += 256) s.t[(e / p) * LG + e % p] = __ldcg(a.gsum + e);
    else
        arn_totals(a, pp, true, [&](size_t e, double v) { s.t[((int)e / p) * LG + (int)e % p] = v; });
    __syncthreads();
    for (int i = 0; i < p; i++) trace += s.t[i * LG + i];
    int fail = 0;
    bool illcond = false;
    for (int attempt = 0; attempt < 2; attempt++) {
        const double shift = attempt == 0 ? 0.0
                                          : 11.0 * ((double)a.n * p + (double)p * (p + 1)) * 1.1102230246251565e-16 * trace;
        for (int e = tid; e < p * p; e += 256) {
            const int i = e / p, j = e % p;
            s.g[i * LG + j] = s.t[i * LG + j] + (i == j ? shift : 0.0);
            s.x[i * LG + j] = i == j ? 1.0 : 0.0;
        }
        __syncthreads();
        fail = 0;
        // elimination on [G | I] with unscaled pivot rows: G = Lt D Lt^T, X = Lt^{-1}
        for (int j = 0; j < p; j++) {
            const double d = s.g[j * LG + j], ref = s.t[j * LG + j] + shift;
            if (attempt == 0 && !(d >= 1e-8 * ref)) illcond = true;
            if (!(d > 1e-13 * ref) || !(d > 0.0)) {
                fail = 1;
                break;
            }
            const double dinv = 1.0 / d;
            for (int e = tid; e < (p - j - 1) * p; e += 256) {
                const int i = j + 1 + e / p, c = e % p;
                const double f = s.g[j * LG + i] * dinv;
                if (c >= i) s.g[i * LG + c] -= f * s.g[j * LG + c];
                else if (c <= j) s.x[i * LG + c] -= f * s.x[j * LG + c];
            }
            __syncthreads();
        }
        if (!fail) break;
        shifted = true;
        __syncthreads();
    }
    if (ill) *ill = fail != 0 || illcond || shifted;
    if (fail) return 2;
    for (int i = tid; i < p; i += 256) s.rs[i] = 1.0 / sqrt(s.g[i * LG + i]);
    __syncthreads();
    // t = R, g = R^{-1}; then r = R r
    for (int e = tid; e < p * p; e += 256) {
        const int i = e / p, j = e % p;
        s.t[i * LG + j] = j >= i ? s.g[i * LG + j] * s.rs[i] : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < p * p; e += 256) {
        const int i = e / p, j = e % p;
        s.g[i * LG + j] = i <= j ? s.x[j * LG + i] * s.rs[j] : 0.0;
    }
    if (first) {
        for (int e = tid; e < p * p; e += 256) s.r[(e / p) * LG + e % p] = s.t[(e / p) * LG + e % p];
    } else {
        double v[4];   // p^2 <= 1024
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int e = tid + 256 * u, i = e / p, j = e % p;
            v[u] = 0.0;
            if (e < p * p)
                for (int c = i; c <= j; c++) v[u] += s.t[i * LG + c] * s.r[c * LG + j];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int e = tid + 256 * u;
            if (e < p * p) s.r[(e / p) * LG + e % p] = v[u];
        }
    }
    __syncthreads();
    // W <- W R^{-1}, 256 / p rows at a time
    const int per = 256 / p;
    for (int b = 0; b < a.rows; b += per) {
        const int row = b + tid / p, c = tid % p;
        const bool ok = tid < per * p && row < a.rows;
        double v = 0.0;
        if (ok)
            for (int i = 0; i <= c; i++) v += s.w[row * LW + i] * s.g[i * LG + c];
        __syncthreads();
        if (ok) s.w[row * LW + c] = v;
    }
    __syncthreads();
    return 0;
}

// Cholesky-QR2, with the third pass where one needed the shift.  Results as arn_cholqr.
template <int NT>
__device__ __forceinline__ int arn_qr(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, unsigned &gen, bool &shifted,
                                      bool *ill) {
    shifted = false;
    int f = arn_cholqr<NT>(a, s, r0, true, gen, shifted, ill);
    if (f == 0) f = arn_cholqr<NT>(a, s, r0, false, gen, shifted, nullptr);
    if (f == 0 && shifted) {
        bool again = false;
        f = arn_cholqr<NT>(a, s, r0, false, gen, again, nullptr);
    }
    return f;
}

template <int NT, bool EVEN>
__global__ void __launch_bounds__(256, 1) arnoldi_kernel(ArnoldiArgs a) {
    constexpr int PT = ArnoldiSmem<NT>::PT, LW = ArnoldiSmem<NT>::LW, LG = ArnoldiSmem<NT>::LG;
    extern __shared__ __align__(16) double sm[];
    __shared__ unsigned s_gen;
    __shared__ int s_off;
    if (threadIdx.x == 0) {
        s_gen = barrier_gen_start(a.ds);
        s_off = a.st->active == 0;
        // the Hessenberg update on the other stream may clear `active` while CTAs start: the first barrier
        // spreads what any of them saw
        if (s_off) *(volatile int *)a.snap = a.epoch;
    }
    __syncthreads();
    unsigned gen = s_gen;
    ArnoldiSmem<NT> s;
    s.w = sm;
    s.buf = s.w + a.rows * LW;
    s.g = s.buf + arn_buf(NT);
    s.x = s.g + PT * LG;
    s.r = s.x + PT * LG;
    s.t = s.r + PT * LG;
    s.rs = s.t + PT * LG;
    const int r0 = blockIdx.x * a.rows, p = a.p;
    for (int e = threadIdx.x; e < a.rows * PT; e += 256) {
        const int row = e / PT, c = e % PT;
        s.w[row * LW + c] = r0 + row < a.n && c < p ? a.Q[(size_t)(r0 + row) * p + c] : 0.0;
    }
    __syncthreads();
    if (!arn_project<NT, EVEN>(a, s, r0, a.Psi, nullptr, gen, s_off != 0, true)) return;
    if (!arn_project<NT, EVEN>(a, s, r0, a.Psi2, a.Psi, gen, false, false)) return;
    bool shifted = false, ill = false;
    int f = arn_qr<NT>(a, s, r0, gen, shifted, &ill);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->qr_shift = shifted;
        a.st->qr_reorth = ill;
    }
    if (f == 0 && ill) {
        // W = V Psi + Q1 R1, Q1 = V Phi + Q2 C2:  Psi += Phi R1, C = C2 R1
        double *R1 = s.buf;   // kept beside the second factorization: buf is free between products
        double keep[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int e = threadIdx.x + 256 * u;
            keep[u] = e < p * p ? s.r[(e / p) * LG + e % p] : 0.0;
        }
        if (!arn_project<NT, EVEN>(a, s, r0, a.Psi2, nullptr, gen, false, false)) return;
        bool shift2 = false;
        f = arn_qr<NT>(a, s, r0, gen, shift2, nullptr);
        if (f == 0) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = threadIdx.x + 256 * u;
                if (e < p * p) R1[e] = keep[u];
            }
            __syncthreads();
            const size_t len = (size_t)a.k * p * p;
            for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < len; e += (size_t)gridDim.x * 256) {
                const int b = (int)(e % p);
                const double *ph = a.Psi2 + e - b;
                double v = 0.0;
                for (int c = 0; c <= b; c++) v += __ldcg(ph + c) * R1[c * p + b];
                a.Psi[e] += v;
            }
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = threadIdx.x + 256 * u, i = e / p, j = e % p;
                v[u] = 0.0;
                if (e < p * p)
                    for (int c = i; c <= j; c++) v[u] += s.r[i * LG + c] * R1[c * p + j];
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = threadIdx.x + 256 * u;
                if (e < p * p) s.r[(e / p) * LG + e % p] = v[u];
            }
            __syncthreads();
        }
    }
    if (f == 1) return;
    if (f == 2) {   // the host decides whether this iteration counted
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.st->qr_fail = 1;
            atomicMin(&a.st->qr_fail_iter, a.k);
        }
        return;
    }
    for (int e = threadIdx.x; e < a.rows * p; e += 256) {
        const int row = e / p, c = e % p;
        if (r0 + row < a.n) a.Vn[(size_t)(r0 + row) * p + c] = s.w[row * LW + c];
    }
    if (blockIdx.x == 0)
        for (int e = threadIdx.x; e < p * p; e += 256) a.C[e] = s.r[(e / p) * LG + e % p];
}

// Rows of a CTA: all SMs where there are 16 rows for each, fewer CTAs (and shorter sums) otherwise.
static int arnoldi_rows(const bpf_ctx *ctx, int n) { return std::max(16, ceil_div(ceil_div(n, ctx->num_sms), 8) * 8); }

static size_t arnoldi_smem(int rows, int p) {
    const int nt = (p + 7) / 8, pt = 8 * nt;
    return sizeof(double) * ((size_t)rows * (pt + 4) + (size_t)arn_buf(nt) +
                             4 * (size_t)pt * (pt + 1) + pt);
}

// Up to 32 columns a warp holds a whole p x p product in registers, and a slab fits beside the Cholesky.
bool arnoldi_ok(const bpf_ctx *ctx, int n, int p) {
    return ctx->fp64_mma && p <= 32 && arnoldi_smem(arnoldi_rows(ctx, n), p) + 1024 <= (size_t)ctx->max_smem_optin;
}

// Products of 65536 sums (64 blocks of 32 columns) at a time: the partial sums of all CTAs stay within
// 78 MB, at two barriers for each further group.
static int arnoldi_group(int p, int k) { return std::min(k, 65536 / (p * p)); }

size_t arnoldi_partials(const bpf_ctx *ctx, int n, int p, int k) {
    return ((size_t)ceil_div(n, arnoldi_rows(ctx, n)) * arnoldi_group(p, k) + 1) * p * p;
}

bpf_status arnoldi_step(bpf_ctx *ctx, int n, int p, int k, const double *V, size_t strideV, const double *Q, double *Vn,
                        double *Psi, double *Psi2, double *C, SolveState *st) {
    bpf_status s;
    double *part = (double *)ws_get(ctx, WS_PARTIAL, sizeof(double) * arnoldi_partials(ctx, n, p, k), &s);
    if (!part) return s;
    ArnoldiArgs a;
    a.n = n;
    a.p = p;
    a.k = k;
    a.rows = arnoldi_rows(ctx, n);
    a.group = arnoldi_group(p, k);
    a.V = V;
    a.strideV = strideV;
    a.Q = Q;
    a.Vn = Vn;
    a.Psi = Psi;
    a.Psi2 = Psi2;
    a.C = C;
    const int grid = ceil_div(n, a.rows);
    a.gsum = part;
    a.part = part + (size_t)p * p;
    a.st = st;
    a.snap = &ctx->dstat->pad[1];
    a.epoch = ++ctx->arnoldi_epoch;
    a.ds = ctx->dstat;
    const size_t smem = arnoldi_smem(a.rows, p);
    const bool even = p % 2 == 0 && ((uintptr_t)V & 15) == 0 && strideV % 2 == 0;
    const void *kern = p <= 8    ? (even ? (const void *)arnoldi_kernel<1, true> : (const void *)arnoldi_kernel<1, false>)
                       : p <= 16 ? (even ? (const void *)arnoldi_kernel<2, true> : (const void *)arnoldi_kernel<2, false>)
                       : p <= 24 ? (even ? (const void *)arnoldi_kernel<3, true> : (const void *)arnoldi_kernel<3, false>)
                                 : (even ? (const void *)arnoldi_kernel<4, true> : (const void *)arnoldi_kernel<4, false>);
    BPF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void *args[] = {&a};
    // the basis read four times (two passes), the block in and out; products and updates of both passes
    KScope ks(ctx, BPF_KC_GRAM, 8.0 * n * p * (4.0 * k + 2.0), 8.0 * n * p * (double)p * k);
    BPF_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(256), args, smem, ctx->stream));
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

}  // namespace bpf
