// One block-Arnoldi orthogonalization in one launch (blocks of up to 64 columns).
//
// Reference: src/block_gmres.jl:301-316 (block Gram-Schmidt against the basis, QR of the new block).
//
// Bound: with narrow blocks, launches.  An iteration's two Gram-Schmidt passes, Cholesky-QR2, its
// third pass and the re-orthogonalization of an ill-conditioned block were 38 kernels, 25 of them
// gated off nearly always, 3-13 us each: 300 us an iteration of a 300-bus solve with 16 columns,
// whose arithmetic is worth a few.  Here they are one cooperative launch: a CTA keeps its rows of the
// new block W in shared memory from the first product to the finished basis block, and what CTAs
// exchange are p x p partial sums through global memory: two grid barriers a Gram-Schmidt pass (each group of
// basis blocks), one a Cholesky pass whose sums every CTA takes itself, two where they are shared out.  Six
// or eight an ordinary iteration.
//
//  * Products V_j^T W: a warp per basis block over the CTA's rows, FP64 tensor pipe (m8n8k4).  A pass'
//    partial sums are added over the CTAs element by element by all threads, in a fixed order.
//  * Update W -= sum_j V_j Psi_j: 16 rows a warp, or the blocks j split over warps where rows are few.
//  * Cholesky-QR: every CTA sums the partial Gram matrices and factors them itself, identically, so the
//    rare decisions (shift, third pass, re-orthogonalization, breakdown) need no further exchange.  A pass
//    that each CTA sums for itself has no barrier after its reads, so passes alternate between two sets
//    of partial sums: a set is written again only behind the barrier of the pass between.
//
// Same algorithm and decisions as gram / tsmm / cholqr / reorth_fold (dense.cu, small.cu); the sums are
// grouped differently, so results agree to rounding.
//
// Measured, a whole solve per iteration, kernel by kernel -> one launch: 300 buses 8 columns 418 -> 114 us,
// 24 columns 560 -> 174; 1500 buses 16 columns 599 -> 162; 3000 buses 64 columns 671 -> 514; 9000 buses 8 columns
// 1981 -> 408 (long basis), 32 columns 1436 -> 687, 48 columns 1411 -> 963, 64 columns 1393 -> 1233 (the
// projections there are gram and tsmm, qr_only); 70000 buses 8 columns 2258 -> 1030.  With few columns now bound by
// the latency of a product's 100 to 200 basis blocks, with 32 by HBM and the tensor pipe in turn (14 TFLOP/s).
// What counted, 9000 buses: loads one step ahead as pairs of columns, coefficients in shared memory, the update's
// order reversed and four lanes an element of a sum, 8 columns 547 -> 410 us and 32 columns 926 -> 742; the
// factorization in registers and R^{-1} applied on the tensor pipe, 32 columns 742 -> 687.
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
    double *part2;       // gridDim.x blocks of p^2: those of every other Cholesky pass
    int group;           // basis blocks whose products are in flight at a time
    double *gsum;        // p^2
    SolveState *st;
    int *snap;           // the grid's decision to skip, by epoch
    int epoch;
    int qr_only;
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
// Warps that share a row of tiles of W^T W.
__host__ __device__ constexpr int arn_parts(int nt) { return kArnoldiWarps / nt; }
// Doubles for partial results of warps (arn_parts x PT^2, or kArnoldiWarps x 8 PT) and two steps' coefficients.
__host__ __device__ constexpr int arn_buf(int nt) {
    const int pt = 8 * nt, coef = 2 * arn_step(nt) * pt * (pt + 2);
    const int warps = arn_parts(nt) * pt * pt > kArnoldiWarps * 8 * pt ? arn_parts(nt) * pt * pt : kArnoldiWarps * 8 * pt;
    return warps > coef ? warps : coef;
}
// The Cholesky's matrix g and buf are not needed at the same time: they share memory.
__host__ __device__ constexpr int arn_area(int nt) {
    const int g = 8 * nt * (8 * nt + 1), bf = arn_buf(nt);
    return ((g > bf ? g : bf) + 1) & ~1;
}

// The shared-memory pieces of a CTA.
template <int NT>
struct ArnoldiSmem {
    static constexpr int PT = 8 * NT, LW = PT + 4, LG = PT + 1;
    double *w;        // rows x LW: the CTA's rows of the block
    double *buf;      // arn_buf(NT)
    double *g;        // PT x LG: pivot rows, then R^{-1} (in buf's memory)
    double *r, *t;    // PT x LG: accumulated R, scratch
    double *rs;
};

__device__ __forceinline__ void cp_async16(double *dst, const double *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

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

// Partial sums of V_j^T W over the CTA's rows, j < nb: part[j].  A warp per j (from 33 columns two, each half
// of the product's rows); the next 4 U rows of V (of this j or the warp's next) are on their way while these are
// multiplied.  Lane (g, t4) takes columns 16 mp + 2 g + {0, 1} of row t4 as one load: the two are the same row
// of two tiles' A fragments.
template <int NT, bool EVEN>
__device__ __forceinline__ void arn_gram(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, const double *A, int nb,
                                         double *part) {
    constexpr int LW = ArnoldiSmem<NT>::LW, U = NT == 1 ? 10 : NT == 2 ? 8 : NT <= 4 ? 4 : 2;
    constexpr int MH = NT > 4 ? 2 : 1, MP = (NT + 2 * MH - 1) / (2 * MH);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p;
    const size_t pp = (size_t)p * p;
    nb *= MH;   // j MH + half
    if (warp >= nb) return;
    double acc[2 * MP][NT][2];
#pragma unroll
    for (int mi = 0; mi < 2 * MP; mi++)
#pragma unroll
        for (int ni = 0; ni < NT; ni++) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
    double2 cur[U][MP], nxt[U][MP];
    const int c0 = 16 * MP * (warp % MH);   // kArnoldiWarps is a multiple of MH: a warp keeps its half
    auto load = [&](double2 (&v)[U][MP], int j, int k0) {
        const double *Aj = A + (size_t)(j / MH) * a.strideV;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int lr = k0 + 4 * u, r = r0 + lr + t4;
            const bool ok = lr < a.rows && r < a.n;
#pragma unroll
            for (int mp = 0; mp < MP; mp++) v[u][mp] = arn_load2<EVEN>(Aj + (size_t)r * p, c0 + 16 * mp + 2 * g, p, ok);
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
                        const int row = c0 + 16 * (mi / 2) + 2 * g + (mi & 1), col = 8 * ni + 2 * t4 + i;
                        if (row < p && col < p) part[(j / MH) * pp + (size_t)row * p + col] = acc[mi][ni][i];
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
            double sv[NT > 4 ? 1 : ES];
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
            auto load_s = [&](int j0, double *b) {
                if constexpr (NT > 4 && !EVEN) {
                    for (int e = threadIdx.x; e < (int)pp; e += 256)
                        b[(e / p) * LS + e % p] = __ldcg(S + j0 * (long long)pp + e);
                } else if constexpr (NT > 4) {   // one block a step: straight to shared memory, not by L1
                    for (int e = 2 * threadIdx.x; e < (int)pp; e += 512)
                        cp_async16(b + (e / p) * LS + e % p, S + j0 * (long long)pp + e);
                    asm volatile("cp.async.commit_group;" ::: "memory");
                } else {
#pragma unroll
                    for (int u = 0; u < ES; u++) {
                        const int e = threadIdx.x + 256 * u, jb = e / (int)pp;
                        sv[u] = jb < JB && j0 + jb >= 0 ? __ldcg(S + j0 * (long long)pp + e) : 0.0;
                    }
                }
            };
            if (NT > 4) __syncthreads();   // the zeros are there
            load(cur, a.k - JB);
            load_s(a.k - JB, sb);
            for (int j0 = a.k - JB, step = 0; j0 > -JB; j0 -= JB, step ^= 1) {
                double *b = sb + step * JB * PT * LS;
                if constexpr (NT > 4) {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncthreads();   // this step's coefficients; the other buffer's readers are done
                } else {
                    __syncthreads();   // the readers of the step before last are done (and, first, the zeros are there)
#pragma unroll
                    for (int u = 0; u < ES; u++) {
                        const int e = threadIdx.x + 256 * u, jb = e / (int)pp, x = e - jb * (int)pp;
                        if (jb < JB) b[jb * PT * LS + (x / p) * LS + x % p] = sv[u];
                    }
                }
                if (j0 > 0) {
                    load(nxt, j0 - JB);
                    load_s(j0 - JB, sb + (step ^ 1) * JB * PT * LS);
                }
                if (NT <= 4) __syncthreads();
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
#pragma unroll
            for (int kk = 0; kk < NT; kk++) av[kk] = arn_load2<EVEN>(row, 8 * kk + 2 * t4, p, r < a.n);
            constexpr int HB = NT <= 4 ? 2 * NT : 2;   // k-steps whose coefficients are in flight
#pragma unroll
            for (int k0 = 0; k0 < 2 * NT; k0 += HB) {
                double bv[HB][NT];
#pragma unroll
                for (int h = 0; h < HB; h++)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++) {
                        const int c = 8 * ((k0 + h) / 2) + 2 * t4 + (h & 1);
                        bv[h][ni] = c < p && 8 * ni + g < p ? __ldcg(Sj + (size_t)c * p + 8 * ni + g) : 0.0;
                    }
#pragma unroll
                for (int h = 0; h < HB; h++)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++)
                        arn_dmma(acc[ni][0], acc[ni][1], h & 1 ? av[(k0 + h) / 2].y : av[(k0 + h) / 2].x, bv[h][ni]);
            }
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
__device__ __forceinline__ double arn_total(const double *part, size_t len, size_t e) {
    double s = 0.0;
    if (e < len) {
        const double *q = part + e;
#pragma unroll 8
        for (unsigned c = (threadIdx.x >> 3) & 3; c < gridDim.x; c += 4) s += __ldcg(q + c * len);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    return s + __shfl_xor_sync(0xffffffffu, s, 16);
}

// f(e, total of e) for this CTA's share of the elements (all: every element).
template <class F>
__device__ __forceinline__ void arn_totals(const double *part, size_t len, bool all, F f) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (size_t e0 = ((all ? 0 : (size_t)blockIdx.x) * kArnoldiWarps + w) * 8; e0 < len;
         e0 += (size_t)(all ? 1 : gridDim.x) * kArnoldiWarps * 8) {
        const size_t e = e0 + (l & 7);
        const double v = arn_total(part, len, e);
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
        arn_totals(a.part, len, false, [&](size_t e, double v) {
            out[j0 * pp + e] = v;
            if (acc) acc[j0 * pp + e] += v;
        });
        if (!grid_barrier(a.ds, gen)) return false;
    }
    arn_update<NT, EVEN>(a, s, r0, out);
    return true;
}

// r <- t r, both PT x PT upper triangular (no barrier at the end): a row of tiles a warp.
template <int NT>
__device__ __forceinline__ void arn_mul_r(const double *t, double *r) {
    constexpr int LG = 8 * NT + 1;
    const int lane = threadIdx.x & 31, mi = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    double acc[NT][2];
#pragma unroll
    for (int ni = 0; ni < NT; ni++) acc[ni][0] = acc[ni][1] = 0.0;
    if (mi < NT) {
        for (int ks = 2 * mi; ks < 2 * NT; ks++) {
            const double v = t[(8 * mi + g) * LG + 4 * ks + t4];
#pragma unroll
            for (int ni = 0; ni < NT; ni++) arn_dmma(acc[ni][0], acc[ni][1], v, r[(4 * ks + t4) * LG + 8 * ni + g]);
        }
    }
    __syncthreads();
    if (mi < NT)
#pragma unroll
        for (int ni = 0; ni < NT; ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) r[(8 * mi + g) * LG + 8 * ni + 2 * t4 + i] = acc[ni][i];
}

// One pass of Cholesky-QR on the CTAs' rows: s.r <- R s.r (first: R).  0: done; 1: a barrier gave up; 2:
// breakdown.  shift / ill: set when the pass needed the shift / lost more than eight digits.  part: a.part and
// a.part2 in turn (other CTAs may still be reading those of the pass before).
template <int NT>
__device__ __forceinline__ int arn_cholqr(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, double *part, bool first,
                                          unsigned &gen, bool &shifted, bool *ill) {
    constexpr int PT = ArnoldiSmem<NT>::PT, LW = ArnoldiSmem<NT>::LW, LG = ArnoldiSmem<NT>::LG;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p, tid = threadIdx.x;
    const size_t pp = (size_t)p * p;
    // W^T W of the CTA's rows: a row of tiles a warp, the rows of W in arn_parts, whose sums are added in order
    {
        constexpr int PARTS = arn_parts(NT);
        const int mi = warp % NT, q = warp / NT;
        if (q < PARTS) {
            double acc[NT][2];
#pragma unroll
            for (int ni = 0; ni < NT; ni++) acc[ni][0] = acc[ni][1] = 0.0;
#pragma unroll 2
            for (int k0 = 4 * q; k0 < a.rows; k0 += 4 * PARTS) {
                double v[NT];
#pragma unroll
                for (int ni = 0; ni < NT; ni++) v[ni] = s.w[(k0 + t4) * LW + 8 * ni + g];
                const double m = s.w[(k0 + t4) * LW + 8 * mi + g];
#pragma unroll
                for (int ni = 0; ni < NT; ni++) arn_dmma(acc[ni][0], acc[ni][1], m, v[ni]);
            }
#pragma unroll
            for (int ni = 0; ni < NT; ni++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int row = 8 * mi + g, col = 8 * ni + 2 * t4 + i;
                    if (PARTS > 1) s.buf[q * PT * PT + row * PT + col] = acc[ni][i];
                    else if (row < p && col < p) part[blockIdx.x * pp + (size_t)row * p + col] = acc[ni][i];
                }
        }
        if (PARTS > 1) {
            __syncthreads();
            for (int e = tid; e < p * p; e += 256) {
                double v = 0.0;
#pragma unroll
                for (int u = 0; u < PARTS; u++) v += s.buf[u * PT * PT + (e / p) * PT + e % p];
                part[blockIdx.x * pp + e] = v;
            }
        }
    }
    if (!grid_barrier(a.ds, gen)) return 1;
    // the sum over the CTAs: each its own, or, where that is much to read, shared out first
    const bool shared_out = pp * gridDim.x > 16384;
    if (shared_out) {
        arn_totals(part, pp, false, [&](size_t e, double v) { a.gsum[e] = v; });
        if (!grid_barrier(a.ds, gen)) return 1;
    }
    double trace = 0.0;
    if (shared_out)
        for (int e = tid; e < p * p; e += 256) s.t[(e / p) * LG + e % p] = __ldcg(a.gsum + e);
    else
        arn_totals(part, pp, true, [&](size_t e, double v) { s.t[((int)e / p) * LG + (int)e % p] = v; });
    __syncthreads();
    for (int i = 0; i < p; i++) trace += s.t[i * LG + i];
    int fail = 0;
    bool illcond = false;
    // Elimination on [G | I] with unscaled pivot rows, G = Lt D Lt^T, X = Lt^{-1}: G's upper triangle and X's lower
    // one share a matrix of which a thread keeps rows a16 + 16 u and columns b16 + 16 v in registers; a step needs
    // the pivot row only (its G part divided by the pivot are the factors), which its owners pass on: one barrier a
    // step (some 200 cycles; with the matrices in shared memory a step of 64 columns took about 1 us).
    constexpr int TT = (PT + 15) / 16;
    const int a16 = tid >> 4, b16 = tid & 15;
    double M[TT][TT];
    double *prow = s.g;   // two pivot rows of PT
    for (int attempt = 0; attempt < 2; attempt++) {
        const double shift = attempt == 0 ? 0.0
                                          : 11.0 * ((double)a.n * p + (double)p * (p + 1)) * 1.1102230246251565e-16 * trace;
#pragma unroll
        for (int u = 0; u < TT; u++)
#pragma unroll
            for (int v = 0; v < TT; v++) {
                const int i = a16 + 16 * u, c = b16 + 16 * v;
                M[u][v] = i < p && c < p && c >= i ? s.t[i * LG + c] + (i == c ? shift : 0.0) : 0.0;
                if (i == 0 && c < PT) prow[c] = M[u][v];
            }
        __syncthreads();
        fail = 0;
        for (int j = 0; j < p; j++) {
            const double *row = prow + (j & 1) * PT;
            const double d = row[j], ref = s.t[j * LG + j] + shift;
            if (attempt == 0 && !(d >= 1e-8 * ref)) illcond = true;
            if (!(d > 1e-13 * ref) || !(d > 0.0)) {
                fail = 1;
                break;
            }
            const double dinv = 1.0 / d;
            double rv[TT];
#pragma unroll
            for (int v = 0; v < TT; v++) {
                const int c = b16 + 16 * v;
                rv[v] = c == j ? 1.0 : c < p ? row[c] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < TT; u++) {
                const int i = a16 + 16 * u;
                if (i <= j || i >= p) continue;
                const double f = row[i] * dinv;
#pragma unroll
                for (int v = 0; v < TT; v++) {
                    const int c = b16 + 16 * v;
                    if (c >= i || c <= j) M[u][v] -= f * rv[v];
                    if (i == j + 1 && c < PT) prow[((j + 1) & 1) * PT + c] = M[u][v];
                }
            }
            __syncthreads();
        }
        if (!fail) break;
        shifted = true;
        __syncthreads();
    }
    if (ill) *ill = fail != 0 || illcond || shifted;
    if (fail) return 2;
#pragma unroll
    for (int u = 0; u < TT; u++)
        if (a16 == b16 && a16 + 16 * u < p) s.rs[a16 + 16 * u] = 1.0 / sqrt(M[u][u]);
    __syncthreads();
    // t = R, g = R^{-1} (zero below the diagonal and beyond p); then r = R r
#pragma unroll
    for (int u = 0; u < TT; u++)
#pragma unroll
        for (int v = 0; v < TT; v++) {
            const int i = a16 + 16 * u, c = b16 + 16 * v;
            if (i >= PT || c >= PT) continue;
            const bool in = i < p && c < p;
            const double rs = in ? s.rs[i] : 0.0;
            s.t[i * LG + c] = in && c >= i ? M[u][v] * rs : 0.0;
            s.g[c * LG + i] = in && c <= i ? (c == i ? 1.0 : M[u][v]) * rs : 0.0;
        }
    __syncthreads();
    if (first) {
        for (int e = tid; e < PT * PT; e += 256) s.r[(e / PT) * LG + e % PT] = s.t[(e / PT) * LG + e % PT];
    } else {
        arn_mul_r<NT>(s.t, s.r);
    }
    __syncthreads();
    // W <- W R^{-1}, a warp's row tiles in place
    for (int t = warp; t < a.rows / 8; t += kArnoldiWarps) {
        double acc[NT][2];
#pragma unroll
        for (int ni = 0; ni < NT; ni++) acc[ni][0] = acc[ni][1] = 0.0;
#pragma unroll
        for (int ks = 0; ks < 2 * NT; ks++) {
            const double v = s.w[(8 * t + g) * LW + 4 * ks + t4];
#pragma unroll
            for (int ni = 0; ni < NT; ni++)
                if (ks < 2 * (ni + 1)) arn_dmma(acc[ni][0], acc[ni][1], v, s.g[(4 * ks + t4) * LG + 8 * ni + g]);
        }
        __syncwarp();
#pragma unroll
        for (int ni = 0; ni < NT; ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) s.w[(8 * t + g) * LW + 8 * ni + 2 * t4 + i] = acc[ni][i];
    }
    __syncthreads();
    return 0;
}

// Cholesky-QR2, with the third pass where one needed the shift.  Results as arn_cholqr.
template <int NT>
__device__ __forceinline__ int arn_qr(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, unsigned &gen, bool &shifted,
                                      bool *ill) {
    shifted = false;
    int f = arn_cholqr<NT>(a, s, r0, a.part, true, gen, shifted, ill);
    if (f == 0) f = arn_cholqr<NT>(a, s, r0, a.part2, false, gen, shifted, nullptr);
    if (f == 0 && shifted) {
        bool again = false;
        f = arn_cholqr<NT>(a, s, r0, a.part, false, gen, again, nullptr);
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
    s.buf = s.g = s.w + a.rows * LW;
    s.r = s.g + arn_area(NT);
    s.t = s.r + PT * LG;
    s.rs = s.t + PT * LG;
    const int r0 = blockIdx.x * a.rows, p = a.p;
    for (int e = threadIdx.x; e < a.rows * PT; e += 256) {
        const int row = e / PT, c = e % PT;
        s.w[row * LW + c] = r0 + row < a.n && c < p ? a.Q[(size_t)(r0 + row) * p + c] : 0.0;
    }
    __syncthreads();
    if (a.qr_only) {   // the projections were done: only spread the decision to skip
        if (!grid_barrier(a.ds, gen)) return;
        if (*(volatile int *)a.snap == a.epoch) return;
    } else {
        if (!arn_project<NT, EVEN>(a, s, r0, a.Psi, nullptr, gen, s_off != 0, true)) return;
        if (!arn_project<NT, EVEN>(a, s, r0, a.Psi2, a.Psi, gen, false, false)) return;
    }
    bool shifted = false, ill = false;
    int f = arn_qr<NT>(a, s, r0, gen, shifted, &ill);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->qr_shift = shifted;
        a.st->qr_reorth = ill;
    }
    if (f == 0 && ill) {
        if (!grid_barrier(a.ds, gen)) return;   // the last pass' sums have been read: the products reuse their place
        // W = V Psi + Q1 R1, Q1 = V Phi + Q2 C2:  Psi += Phi R1, C = C2 R1; R1 stays in C meanwhile
        if (blockIdx.x == 0)
            for (int e = threadIdx.x; e < p * p; e += 256) a.C[e] = s.r[(e / p) * LG + e % p];
        if (!arn_project<NT, EVEN>(a, s, r0, a.Psi2, nullptr, gen, false, false)) return;
        bool shift2 = false;
        f = arn_qr<NT>(a, s, r0, gen, shift2, nullptr);
        if (f == 0) {
            double *R1 = s.g;
            for (int e = threadIdx.x; e < PT * PT; e += 256) {
                const int i = e / PT, j = e % PT;
                R1[i * LG + j] = i < p && j < p ? __ldcg(a.C + i * p + j) : 0.0;
            }
            __syncthreads();
            const size_t len = (size_t)a.k * p * p;
            for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < len; e += (size_t)gridDim.x * 256) {
                const int b = (int)(e % p);
                const double *ph = a.Psi2 + e - b;
                double v = 0.0;
                for (int c = 0; c <= b; c++) v += __ldcg(ph + c) * R1[c * LG + b];
                a.Psi[e] += v;
            }
            // r = C2 R1 in R1's place
            arn_mul_r<NT>(s.r, R1);
            __syncthreads();
            for (int e = threadIdx.x; e < PT * PT; e += 256) s.r[(e / PT) * LG + e % PT] = R1[(e / PT) * LG + e % PT];
            __syncthreads();
        }
        if (f != 1 && !grid_barrier(a.ds, gen)) return;   // all have read C
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

// Rows of a CTA: all SMs but eight (the Hessenberg update on the other stream takes a CTA per eight columns)
// where there are 16 rows for each, fewer CTAs (and shorter sums) otherwise.
static int arnoldi_rows(const bpf_ctx *ctx, int n) {
    return std::max(16, ceil_div(ceil_div(n, std::max(1, ctx->num_sms - 8)), 8) * 8);
}

static int arnoldi_nt(int p) { return p <= 32 ? (p + 7) / 8 : p <= 48 ? 6 : 8; }

static size_t arnoldi_smem(int rows, int p) {
    const int nt = arnoldi_nt(p), pt = 8 * nt;
    return sizeof(double) * ((size_t)rows * (pt + 4) + (size_t)arn_area(nt) + 2 * (size_t)pt * (pt + 1) + pt);
}

// Up to 64 columns a warp or two hold a whole p x p product in registers, and a slab fits beside the Cholesky.
bool arnoldi_ok(const bpf_ctx *ctx, int n, int p) {
    return ctx->fp64_mma && p <= 64 &&
           arnoldi_smem(arnoldi_rows(ctx, n), p) + 1024 <= (size_t)ctx->max_smem_optin;
}

// Products of 65536 sums (64 blocks of 32 columns) at a time: the partial sums of all CTAs stay within
// 78 MB, at two barriers for each further group.
static int arnoldi_group(int p, int k) { return std::min(k, 65536 / (p * p)); }

size_t arnoldi_partials(const bpf_ctx *ctx, int n, int p, int k) {
    return ((size_t)ceil_div(n, arnoldi_rows(ctx, n)) * (arnoldi_group(p, k) + 1) + 1) * p * p;
}

bpf_status arnoldi_step(bpf_ctx *ctx, int n, int p, int k, const double *V, size_t strideV, const double *Q, double *Vn,
                        double *Psi, double *Psi2, double *C, SolveState *st, bool qr_only) {
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
    a.part2 = a.part + (size_t)grid * a.group * p * p;
    a.st = st;
    a.snap = &ctx->dstat->pad[1];
    a.epoch = ++ctx->arnoldi_epoch;
    a.qr_only = qr_only ? 1 : 0;
    a.ds = ctx->dstat;
    const size_t smem = arnoldi_smem(a.rows, p);
    const bool even = p % 2 == 0;   // every block is 16-byte aligned then (workspaces and multiples of p doubles)
    const void *kern = p <= 8    ? (even ? (const void *)arnoldi_kernel<1, true> : (const void *)arnoldi_kernel<1, false>)
                       : p <= 16 ? (even ? (const void *)arnoldi_kernel<2, true> : (const void *)arnoldi_kernel<2, false>)
                       : p <= 24 ? (even ? (const void *)arnoldi_kernel<3, true> : (const void *)arnoldi_kernel<3, false>)
                       : p <= 32 ? (even ? (const void *)arnoldi_kernel<4, true> : (const void *)arnoldi_kernel<4, false>)
                       : p <= 48 ? (even ? (const void *)arnoldi_kernel<6, true> : (const void *)arnoldi_kernel<6, false>)
                                 : (even ? (const void *)arnoldi_kernel<8, true> : (const void *)arnoldi_kernel<8, false>);
    BPF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void *args[] = {&a};
    // the basis read four times (two passes), the block in and out; products and updates of both passes
    KScope ks(ctx, BPF_KC_GRAM, 8.0 * n * p * (qr_only ? 2.0 : 4.0 * k + 2.0), 8.0 * n * p * (double)p * (qr_only ? 1 : k));
    BPF_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(256), args, smem, ctx->stream));
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

}  // namespace bpf
