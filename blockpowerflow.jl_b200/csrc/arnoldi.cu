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
//  * Update W -= sum_j V_j Psi_j: eight rows a warp, the blocks j split over warps where rows are few.
//  * Cholesky-QR: every CTA sums the partial Gram matrices and factors them itself, identically, so the
//    rare decisions (shift, third pass, re-orthogonalization, breakdown) need no further exchange.
//
// Same algorithm and decisions as gram / tsmm / cholqr / reorth_fold (dense.cu, small.cu); the sums are
// grouped differently, so results agree to rounding.
//
// Measured, a whole solve per iteration, kernel by kernel -> one launch: 300 buses 8 columns 418 -> 120 us,
// 24 columns 560 -> 198; 1500 buses 16 columns 599 -> 188; 9000 buses 8 columns 1981 -> 547 (long basis), 32
// columns 1436 -> 926; 70000 buses 8 columns 2258 -> 1312.
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

// The shared-memory pieces of a CTA.
template <int NT>
struct ArnoldiSmem {
    static constexpr int PT = 8 * NT, LW = PT + 4, LG = PT + 1;
    double *w;      // rows x LW: the CTA's rows of the block
    double *buf;    // kArnoldiWarps x max(8 PT, PT^2): partial results of warps
    double *g, *x, *r, *t;   // PT x LG: Gram matrix / R^{-T}, inverse, accumulated R, scratch
    double *dref, *rs;
};

// Partial sums of A_j^T W over the CTA's rows, j < nb (A = nullptr: W^T W, one block): part[j].
template <int NT>
__device__ __forceinline__ void arn_gram(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, const double *A, int nb,
                                         double *part) {
    constexpr int LW = ArnoldiSmem<NT>::LW, U = NT <= 2 ? 8 : 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p;
    const size_t pp = (size_t)p * p;
    for (int j = warp; j < nb; j += kArnoldiWarps) {
        const double *Aj = A + (size_t)j * a.strideV;
        double acc[NT][NT][2];
#pragma unroll
        for (int mi = 0; mi < NT; mi++)
#pragma unroll
            for (int ni = 0; ni < NT; ni++) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
        for (int k0 = 0; k0 < a.rows; k0 += 4 * U) {
            double av[U][NT];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int r = r0 + k0 + 4 * u + t4;
                const bool ok = k0 + 4 * u < a.rows && r < a.n;
#pragma unroll
                for (int mi = 0; mi < NT; mi++)
                    av[u][mi] = ok && 8 * mi + g < p ? __ldcg(Aj + (size_t)r * p + 8 * mi + g) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (k0 + 4 * u >= a.rows) break;
                double bv[NT];
#pragma unroll
                for (int ni = 0; ni < NT; ni++) bv[ni] = s.w[(k0 + 4 * u + t4) * LW + 8 * ni + g];
#pragma unroll
                for (int mi = 0; mi < NT; mi++)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++) arn_dmma(acc[mi][ni][0], acc[mi][ni][1], av[u][mi], bv[ni]);
            }
        }
#pragma unroll
        for (int mi = 0; mi < NT; mi++)
#pragma unroll
            for (int ni = 0; ni < NT; ni++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int row = 8 * mi + g, col = 8 * ni + 2 * t4 + i;
                    if (row < p && col < p) part[j * pp + (size_t)row * p + col] = acc[mi][ni][i];
                }
    }
}

// W -= sum_j V_j S_j on the CTA's rows (ends with a barrier).
template <int NT>
__device__ __forceinline__ void arn_update(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, const double *S) {
    constexpr int PT = ArnoldiSmem<NT>::PT, LW = ArnoldiSmem<NT>::LW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, p = a.p;
    const size_t pp = (size_t)p * p;
    const int tiles = a.rows / 8, split = tiles >= kArnoldiWarps ? 1 : kArnoldiWarps / tiles;
    const int part = split == 1 ? 0 : warp / tiles, ksteps = (p + 3) / 4;
    const bool busy = split == 1 || warp < tiles * split;
    for (int t = split == 1 ? warp : warp % tiles; busy && t < tiles; t += split == 1 ? kArnoldiWarps : tiles) {
        double acc[NT][2];
#pragma unroll
        for (int ni = 0; ni < NT; ni++) acc[ni][0] = acc[ni][1] = 0.0;
        const int r = r0 + 8 * t + g;
        for (int j = part; j < a.k; j += split) {
            const double *Vj = a.V + (size_t)j * a.strideV + (size_t)r * p, *Sj = S + j * pp;
            double av[2 * NT], bv[2 * NT][NT];   // ksteps <= 2 NT
#pragma unroll
            for (int ks = 0; ks < 2 * NT; ks++) {
                const int c = 4 * ks + t4;
                av[ks] = r < a.n && c < p ? __ldcg(Vj + c) : 0.0;
#pragma unroll
                for (int ni = 0; ni < NT; ni++)
                    bv[ks][ni] = c < p && 8 * ni + g < p ? __ldcg(Sj + (size_t)c * p + 8 * ni + g) : 0.0;
            }
#pragma unroll
            for (int ks = 0; ks < 2 * NT; ks++)
                if (ks < ksteps)
#pragma unroll
                    for (int ni = 0; ni < NT; ni++) arn_dmma(acc[ni][0], acc[ni][1], av[ks], bv[ks][ni]);
        }
#pragma unroll
        for (int ni = 0; ni < NT; ni++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int c = 8 * ni + 2 * t4 + i;
                if (split == 1) s.w[(8 * t + g) * LW + c] -= acc[ni][i];
                else s.buf[(size_t)warp * 8 * PT + g * PT + c] = acc[ni][i];
            }
        if (split > 1) break;
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

// Sum over the CTAs of element e of their partial sums.
__device__ __forceinline__ double arn_total(const ArnoldiArgs &a, size_t len, size_t e) {
    double s = 0.0;
    const double *q = a.part + e;
#pragma unroll 8
    for (unsigned c = 0; c < gridDim.x; c++) s += __ldcg(q + c * len);
    return s;
}

// One Gram-Schmidt pass: coefficients into out (and added to acc), W updated.  False: a barrier gave up.
template <int NT>
__device__ __forceinline__ bool arn_project(const ArnoldiArgs &a, const ArnoldiSmem<NT> &s, int r0, double *out, double *acc,
                                            unsigned &gen, bool skip, bool check) {
    const size_t pp = (size_t)a.p * a.p;
    for (int j0 = 0; j0 < a.k; j0 += a.group) {
        const int nb = min(a.group, a.k - j0);
        const size_t len = nb * pp;
        if (!skip) arn_gram<NT>(a, s, r0, a.V + (size_t)j0 * a.strideV, nb, a.part + blockIdx.x * len);
        if (!grid_barrier(a.ds, gen)) return false;
        if (check && *(volatile int *)a.snap == a.epoch) return false;   // some CTA saw the solve stopped
        for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < len; e += (size_t)gridDim.x * 256) {
            const double v = arn_total(a, len, e);
            out[j0 * pp + e] = v;
            if (acc) acc[j0 * pp + e] += v;
        }
        if (!grid_barrier(a.ds, gen)) return false;
    }
    arn_update<NT>(a, s, r0, out);
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
        for (size_t e = (size_t)blockIdx.x * 256 + tid; e < pp; e += (size_t)gridDim.x * 256) a.gsum[e] = arn_total(a, pp, e);
        if (!grid_barrier(a.ds, gen)) return 1;
    }
    double trace = 0.0;
    for (int e = tid; e < p * p; e += 256) {
        const double v = shared_out ? __ldcg(a.gsum + e) : arn_total(a, pp, e);
        s.t[(e / p) * LG + e % p] = v;
    }
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

template <int NT>
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
    s.g = s.buf + kArnoldiWarps * PT * (NT > 1 ? PT : 8);
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
    if (!arn_project<NT>(a, s, r0, a.Psi, nullptr, gen, s_off != 0, true)) return;
    if (!arn_project<NT>(a, s, r0, a.Psi2, a.Psi, gen, false, false)) return;
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
        if (!arn_project<NT>(a, s, r0, a.Psi2, nullptr, gen, false, false)) return;
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
    return sizeof(double) * ((size_t)rows * (pt + 4) + (size_t)kArnoldiWarps * pt * (nt > 1 ? pt : 8) +
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
    const void *kern = p <= 8    ? (const void *)arnoldi_kernel<1>
                       : p <= 16 ? (const void *)arnoldi_kernel<2>
                       : p <= 24 ? (const void *)arnoldi_kernel<3>
                                 : (const void *)arnoldi_kernel<4>;
    BPF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void *args[] = {&a};
    // the basis read four times (two passes), the block in and out; products and updates of both passes
    KScope ks(ctx, BPF_KC_GRAM, 8.0 * n * p * (4.0 * k + 2.0), 8.0 * n * p * (double)p * k);
    BPF_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(256), args, smem, ctx->stream));
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

}  // namespace bpf
