// CSR SpMM on row-major (RHS-interleaved) blocks, and the column-major <-> row-major
// conversions at the API boundary.
//
// Replaces mul!(W, A, P) (src/block_gmres.jl:299, :220,268; src/block_bicgstab.jl:135,145,
// 252,264), which CUDA.jl maps to cusparseSpMM on column-major blocks.  Here the block is
// stored row-major (the p values of one unknown are contiguous), so every nonzero a_ij
// gathers one contiguous p-vector of X: a group of G lanes per row reads it with coalesced
// loads while the row's (col, val) pairs are loaded once per group and broadcast by shuffles.
//
// Algorithmic bytes per launch: 12*nnz + 4*(n+1) + 8*n*p (X) + 8*n*p (Y written)
// [+ 8*n*p when beta != 0 or the residual form reads B].
#include <cstdint>
#include <type_traits>

#include "bpf_internal.cuh"

namespace bpf {

template <int G, int CPL, typename TX>
__global__ void __launch_bounds__(256)
spmm_rm_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci,
               const double *__restrict__ av, int base, int p, double alpha,
               const TX *__restrict__ X, double beta, double *__restrict__ Y,
               const double *__restrict__ Bres, const int *gate) {
    // one decision per CTA: the gate (st->active) may be cleared by the other stream mid-launch
    __shared__ int s_off;
    if (threadIdx.x == 0) s_off = (gate && *gate == 0) ? 1 : 0;
    __syncthreads();
    if (s_off) return;
    const int lane = threadIdx.x & 31;
    const int glane = lane % G;                    // lane within the row group
    const int groups_per_block = blockDim.x / G;
    const int grp = blockIdx.x * groups_per_block + threadIdx.x / G;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane / G * G));
    for (int row = grp; row < n; row += gridDim.x * groups_per_block) {
        double acc[CPL];
#pragma unroll
        for (int j = 0; j < CPL; j++) acc[j] = 0.0;
        const int rs = __ldg(rp + row) - base, re = __ldg(rp + row + 1) - base;
        for (int kb = rs; kb < re; kb += G) {
            int k = kb + glane;
            int c = 0;
            double a = 0.0;
            if (k < re) {
                c = __ldg(ci + k) - base;
                a = __ldg(av + k);
            }
            const int cnt = min(G, re - kb);
            #pragma unroll 4   // several entries' loads in flight; same summation order
            for (int t = 0; t < cnt; t++) {
                const int ct = __shfl_sync(gmask, c, t, G);
                const double at = __shfl_sync(gmask, a, t, G);
                const TX *xr = X + (size_t)ct * p;
#pragma unroll
                for (int j = 0; j < CPL; j++) {
                    const int col = glane + j * G;
                    if (col < p) acc[j] += at * (double)__ldg(xr + col);
                }
            }
        }
        double *yr = Y + (size_t)row * p;
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const int col = glane + j * G;
            if (col < p) {
                double v;
                if (Bres) {
                    v = Bres[(size_t)row * p + col] - acc[j];
                } else {
                    v = alpha * acc[j];
                    if (beta != 0.0) v += beta * yr[col];
                }
                yr[col] = v;
            }
        }
    }
}

// Blocks of 64, 128, ... columns: a warp per row, lane l holding columns 2l, 2l + 1 (+ 64 j) as
// one 16-byte load per gathered row segment, half the load instructions of the 8-byte form and
// twice the bytes each one brings; eight entries' loads in flight.  Same products and summation
// order per output as spmm_rm_kernel.
template <int C2>
__global__ void __launch_bounds__(256)
spmm_rm2_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                const double *__restrict__ av, int base, int p, double alpha,
                const double *__restrict__ X, double beta, double *__restrict__ Y,
                const double *__restrict__ Bres, const int *gate) {
    __shared__ int s_off;
    if (threadIdx.x == 0) s_off = (gate && *gate == 0) ? 1 : 0;
    __syncthreads();
    if (s_off) return;
    const int lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < n; row += gridDim.x * warps) {
        double2 acc[C2];
#pragma unroll
        for (int j = 0; j < C2; j++) acc[j] = make_double2(0.0, 0.0);
        const int rs = __ldg(rp + row) - base, re = __ldg(rp + row + 1) - base;
        for (int kb = rs; kb < re; kb += 32) {
            const int k = kb + lane;
            int c = 0;
            double a = 0.0;
            if (k < re) {
                c = __ldg(ci + k) - base;
                a = __ldg(av + k);
            }
            const int cnt = min(32, re - kb);
#pragma unroll 8
            for (int t = 0; t < cnt; t++) {
                const int ct = __shfl_sync(0xffffffffu, c, t);
                const double at = __shfl_sync(0xffffffffu, a, t);
                const double2 *xr = reinterpret_cast<const double2 *>(X + (size_t)ct * p);
#pragma unroll
                for (int j = 0; j < C2; j++) {
                    const double2 v = __ldg(xr + lane + 32 * j);
                    acc[j].x += at * v.x;
                    acc[j].y += at * v.y;
                }
            }
        }
        double2 *yr = reinterpret_cast<double2 *>(Y + (size_t)row * p);
#pragma unroll
        for (int j = 0; j < C2; j++) {
            double2 v;
            if (Bres) {
                const double2 b = reinterpret_cast<const double2 *>(Bres + (size_t)row * p)[lane + 32 * j];
                v = make_double2(b.x - acc[j].x, b.y - acc[j].y);
            } else {
                v = make_double2(alpha * acc[j].x, alpha * acc[j].y);
                if (beta != 0.0) {
                    const double2 y0 = yr[lane + 32 * j];
                    v.x += beta * y0.x;
                    v.y += beta * y0.y;
                }
            }
            yr[lane + 32 * j] = v;
        }
    }
}

template <int C2>
static bpf_status launch_spmm2(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci,
                               const double *av, int base, int p, double alpha, const double *X,
                               double beta, double *Y, const double *B, const int *gate) {
    const int threads = 256, rows_per_block = threads / 32;
    int blocks = (int)std::min<long long>(ceil_div(n, rows_per_block), (long long)ctx->num_sms * 16);
    if (blocks < 1) blocks = 1;
    const double np = (double)n * p;
    const double bytes = 12.0 * nnz + 4.0 * (n + 1) + 8.0 * np + 8.0 * np + ((B || beta != 0.0) ? 8.0 * np : 0.0);
    KScope ks(ctx, BPF_KC_SPMM, bytes, 2.0 * nnz * p);
    spmm_rm2_kernel<C2><<<blocks, threads, 0, ctx->stream>>>(n, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

template <int G, int CPL, typename TX>
static bpf_status launch_spmm(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci,
                              const double *av, int base, int p, double alpha, const TX *X,
                              double beta, double *Y, const double *B, const int *gate) {
    const int threads = 256;
    const int groups = threads / G;
    long long blocks_needed = ceil_div(n, groups);
    int blocks = (int)std::min<long long>(blocks_needed, (long long)ctx->num_sms * 16);
    if (blocks < 1) blocks = 1;
    const double np = (double)n * p;
    const double bytes = 12.0 * nnz + 4.0 * (n + 1) + sizeof(TX) * np + 8.0 * np +
                         ((B || beta != 0.0) ? 8.0 * np : 0.0);
    KScope ks(ctx, BPF_KC_SPMM, bytes, 2.0 * nnz * p);
    spmm_rm_kernel<G, CPL, TX><<<blocks, threads, 0, ctx->stream>>>(n, rp, ci, av, base, p, alpha,
                                                                    X, beta, Y, B, gate);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

template <typename TX>
static bpf_status spmm_dispatch(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci,
                                const double *av, int base, int p, double alpha, const TX *X,
                                double beta, double *Y, const double *B, const int *gate) {
    if (n == 0 || p == 0) return BPF_SUCCESS;
    if constexpr (std::is_same<TX, double>::value) {
        // 16-byte rows: p a multiple of 64 and every block 16-byte aligned
        const bool aligned = ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y) |
                               reinterpret_cast<uintptr_t>(B)) & 15) == 0;
        if (aligned && p % 64 == 0 && p <= 256) {
            if (p == 64) return launch_spmm2<1>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
            if (p == 128) return launch_spmm2<2>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
            if (p == 192) return launch_spmm2<3>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
            return launch_spmm2<4>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
        }
    }
    if (p <= 4) return launch_spmm<4, 1>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 8) return launch_spmm<8, 1>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 16) return launch_spmm<16, 1>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 32) return launch_spmm<32, 1>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 64) return launch_spmm<32, 2>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 128) return launch_spmm<32, 4>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    if (p <= 256) return launch_spmm<32, 8>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
    return launch_spmm<32, 16>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
}

bpf_status spmm_rowmajor(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci,
                         const double *av, int base, int p, double alpha, const double *X,
                         double beta, double *Y, const double *B, const int *gate) {
    if (p > 512) {
        return set_error(ctx, BPF_ERR_NOT_SUPPORTED, "spmm: p=%d > 512 right-hand sides", p);
    }
    return spmm_dispatch<double>(ctx, n, nnz, rp, ci, av, base, p, alpha, X, beta, Y, B, gate);
}

bpf_status spmm_rowmajor_f32x(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci,
                              const double *av, int base, int p, const float *X, double *Y,
                              const int *gate) {
    if (p > 512) {
        return set_error(ctx, BPF_ERR_NOT_SUPPORTED, "spmm: p=%d > 512 right-hand sides", p);
    }
    return spmm_dispatch<float>(ctx, n, nnz, rp, ci, av, base, p, 1.0, X, 0.0, Y, nullptr, gate);
}

// ------------------------------------------------------------------------------------
// The product on column-major blocks (bpf_spmm)
// ------------------------------------------------------------------------------------
// Few columns, or a small product: straight from the columns, a thread per row holding CPT of them.
// A gathered value costs a 32-byte sector, but there is one launch and no copy of X.  Eight entries'
// loads in flight a thread; products and summation order as spmm_rm_kernel.
template <int CPT>
__global__ void __launch_bounds__(128)
spmm_cm_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci, const double *__restrict__ av, int base,
               int p, double alpha, const double *__restrict__ X, int ldx, double beta, double *__restrict__ Y, int ldy) {
    const int row = blockIdx.x * 128 + threadIdx.x;
    if (row >= n) return;
    const int rs = __ldg(rp + row) - base, re = __ldg(rp + row + 1) - base;
    for (int c0 = blockIdx.y * CPT; c0 < p; c0 += gridDim.y * CPT) {
        const double *Xc = X + (size_t)c0 * ldx;
        const int pc = min(CPT, p - c0);
        double acc[CPT];
#pragma unroll
        for (int j = 0; j < CPT; j++) acc[j] = 0.0;
        for (int k = rs; k < re; k += 8) {
            int c[8];
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                c[u] = k + u < re ? __ldg(ci + k + u) - base : 0;
                v[u] = k + u < re ? __ldg(av + k + u) : 0.0;
            }
            double x[8][CPT];
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int j = 0; j < CPT; j++) x[u][j] = k + u < re && j < pc ? __ldg(Xc + (size_t)j * ldx + c[u]) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int j = 0; j < CPT; j++)
                    if (k + u < re) acc[j] += v[u] * x[u][j];
        }
#pragma unroll
        for (int j = 0; j < CPT; j++)
            if (j < pc) {
                double *y = Y + (size_t)(c0 + j) * ldy + row;
                double v = alpha * acc[j];
                if (beta != 0.0) v += beta * *y;
                *y = v;
            }
    }
}

// X (column-major) into panels of W columns: panel q holds n rows of w doubles (the last panel's rows may be
// narrower; w even, a pad column is zero).  64 rows of one panel a CTA.
template <int W>
__global__ void __launch_bounds__(256)
cm_to_panels_kernel(int n, int p, const double *__restrict__ src, int ld, double *__restrict__ dst) {
    constexpr int R = 64;
    __shared__ double tile[W][R + 1];
    const int r0 = blockIdx.x * R, c0 = blockIdx.y * W;
    const int pc = min(W, p - c0), w = (pc + 1) & ~1, nr = min(R, n - r0);
    const int x = threadIdx.x % R;
#pragma unroll
    for (int q = 0; q < W * R / 256; q++) {
        const int c = threadIdx.x / R + 256 / R * q;
        if (c < w) tile[c][x] = c < pc && x < nr ? src[(size_t)(c0 + c) * ld + r0 + x] : 0.0;
    }
    __syncthreads();
    double *d = dst + (size_t)c0 * n + (size_t)r0 * w;
    if (w == W)
        for (int e = threadIdx.x; e < nr * W; e += 256) d[e] = tile[e % W][e / W];
    else
        for (int e = threadIdx.x; e < nr * w; e += 256) d[e] = tile[e % w][e / w];
}

// Y = alpha A X + beta Y from panels of X, Y column-major: G lanes a row, two columns a lane, so an entry
// gathers one contiguous row of the panel; the CTA's tile of Y turns in shared memory.  Summation order as
// spmm_rm_kernel.  Bound: the gathers from L2 (1 GB at 70000 buses x 128 columns, 6-7 TB/s); many warps with
// few loads each carry them best: 32 registers and 64 warps an SM 165 us, eight loads in flight a lane at 48-64
// registers 190-230 us, entries staged in shared memory 230 us.
template <int G>
__global__ void __launch_bounds__(256)
spmm_panel_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci, const double *__restrict__ av, int base,
                  int p, double alpha, const double *__restrict__ XP, double beta, double *__restrict__ Y, int ldy) {
    constexpr int NG = 256 / G, ROWS = NG > 32 ? NG : 32, W = 2 * G;
    __shared__ double tile[W][ROWS + 1];
    const int lane = threadIdx.x & 31, gl = lane % G, grp = threadIdx.x / G;
    const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (lane / G * G);
    const int r0 = blockIdx.x * ROWS, c0 = blockIdx.y * W;
    const int pc = min(W, p - c0), w2 = (pc + 1) / 2;
    const double2 *Xp = reinterpret_cast<const double2 *>(XP + (size_t)c0 * n) + min(gl, w2 - 1);
#pragma unroll 1
    for (int lr = grp; lr < ROWS; lr += NG) {
        const int row = r0 + lr;
        double2 acc = make_double2(0.0, 0.0);
        if (row < n) {
            const int rs = __ldg(rp + row) - base, re = __ldg(rp + row + 1) - base;
            for (int kb = rs; kb < re; kb += G) {
                const int k = kb + gl;
                int c = 0;
                double a = 0.0;
                if (k < re) {
                    c = __ldg(ci + k) - base;
                    a = __ldg(av + k);
                }
                const int cnt = min(G, re - kb);
#pragma unroll 8
                for (int t = 0; t < cnt; t++) {
                    const int ct = __shfl_sync(gmask, c, t, G);
                    const double at = __shfl_sync(gmask, a, t, G);
                    const double2 v = __ldg(Xp + (size_t)ct * w2);
                    acc.x += at * v.x;
                    acc.y += at * v.y;
                }
            }
        }
        tile[2 * gl][lr] = acc.x;
        tile[2 * gl + 1][lr] = acc.y;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < pc * ROWS; e += 256) {
        const int c = e / ROWS, lr = e % ROWS;
        if (r0 + lr < n) {
            double *y = Y + (size_t)(c0 + c) * ldy + r0 + lr;
            double v = alpha * tile[c][lr];
            if (beta != 0.0) v += beta * *y;
            *y = v;
        }
    }
}

// X into panels, then the product.
template <int G>
static bpf_status launch_spmm_panel(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci, const double *av,
                                    int base, int p, double alpha, const double *X, int ldx, double *xp, double beta,
                                    double *Y, int ldy) {
    constexpr int W = 2 * G, ROWS = 256 / G > 32 ? 256 / G : 32;
    cm_to_panels_kernel<W><<<dim3(ceil_div(n, 64), ceil_div(p, W)), 256, 0, ctx->stream>>>(n, p, X, ldx, xp);
    BPF_LAUNCHED(ctx);
    const double np = (double)n * p;
    KScope ks(ctx, BPF_KC_SPMM, 12.0 * nnz + 4.0 * (n + 1) + 16.0 * np + (beta != 0.0 ? 8.0 * np : 0.0), 2.0 * nnz * p);
    spmm_panel_kernel<G><<<dim3(ceil_div(n, ROWS), ceil_div(p, W)), 256, 0, ctx->stream>>>(n, rp, ci, av, base, p, alpha,
                                                                                         xp, beta, Y, ldy);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

bpf_status spmm_colmajor(bpf_ctx *ctx, int n, long long nnz, const int *rp, const int *ci, const double *av, int base,
                         int p, double alpha, const double *X, int ldx, double beta, double *Y, int ldy, BlockOverlap ov) {
    if (n == 0 || p == 0) return BPF_SUCCESS;
    // Straight from the columns while its 32 bytes a gathered value cost less than the panels' copy and
    // second launch.  Direct / panels, cold caches: 300 buses x 16 8.3 / 17.6 us, 9000 x 16 (1.9 M products)
    // 16.4 / 17.4, 30000 x 5 (2.0 M) 20.4 / 19.5, 9000 x 33 (4.0 M) 24.6 / 25, 9000 x 64 38.9 / 27; one to four
    // columns fill only a quarter of a panel row's sectors: 70000 x 3 22.6, x 8 43 / 32.
    if (ov == BlockOverlap::kNone && (p <= 4 || (double)nnz * p <= 2e6)) {
        const double np = (double)n * p;
        KScope ks(ctx, BPF_KC_SPMM, 12.0 * nnz + 4.0 * (n + 1) + 16.0 * np + (beta != 0.0 ? 8.0 * np : 0.0), 2.0 * nnz * p);
        // more columns a thread share its row's entries; fewer where threads are few
        const int cpt = p == 1 ? 1 : p <= 2 || np < 32768 ? 2 : 4;
        const auto kern = cpt == 1 ? spmm_cm_kernel<1> : cpt == 2 ? spmm_cm_kernel<2> : spmm_cm_kernel<4>;
        kern<<<dim3(ceil_div(n, 128), std::min(ceil_div(p, cpt), 65535)), 128, 0, ctx->stream>>>(n, rp, ci, av, base, p, alpha,
                                                                                                X, ldx, beta, Y, ldy);
        BPF_LAUNCHED(ctx);
        return BPF_SUCCESS;
    }
    const int chunk = 256;
    bpf_status st;
    double *xp = (double *)ws_get(ctx, WS_A, sizeof(double) * (size_t)n * ((std::min(p, chunk) + 1) & ~1), &st);
    if (!xp) return st;
    for (int c0 = 0; c0 < p; c0 += chunk) {
        const int pc = std::min(chunk, p - c0);
        // Panels of 64 columns (a warp a row) move the most bytes an instruction: 70000 buses x 128 columns 211
        // us against 222 in panels of 32, 30000 x 128 90 against 97; less than a wave of such CTAs (9000 x 64)
        // 31.7 against 27.3.  Narrower blocks take as many lanes a row as they fill.
        const bool wave = (long long)ceil_div(n, 32) * ceil_div(pc, 64) >= 8LL * ctx->num_sms;
        const auto launch = pc <= 8             ? launch_spmm_panel<4>
                            : pc <= 16          ? launch_spmm_panel<8>
                            : pc <= 32 || !wave ? launch_spmm_panel<16>
                                                : launch_spmm_panel<32>;
        BPF_TRY(launch(ctx, n, nnz, rp, ci, av, base, pc, alpha, X + (size_t)c0 * ldx, ldx, xp, beta, Y + (size_t)c0 * ldy, ldy));
    }
    return BPF_SUCCESS;
}

// ------------------------------------------------------------------------------------
// layout conversions (32x32 tiles through shared memory)
// ------------------------------------------------------------------------------------
// *gate may be cleared by another stream meanwhile: a CTA decides once.
__device__ __forceinline__ bool gated_off(const int *gate) {
    if (!gate) return false;
    __shared__ int off;
    if (threadIdx.x == 0 && threadIdx.y == 0) off = *gate == 0;
    __syncthreads();
    return off != 0;
}

__global__ void cm_to_rm_kernel(int n, int p, const double *__restrict__ src, int ld,
                                double *__restrict__ dst, const int *gate) {
    if (gated_off(gate)) return;
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        int c = c0 + j, r = r0 + threadIdx.x;
        if (r < n && c < p) tile[j][threadIdx.x] = src[(size_t)c * ld + r];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        int r = r0 + j, c = c0 + threadIdx.x;
        if (r < n && c < p) dst[(size_t)r * p + c] = tile[threadIdx.x][j];
    }
}

__global__ void rm_to_cm_kernel(int n, int p, const double *__restrict__ src,
                                double *__restrict__ dst, int ld, const int *gate) {
    if (gated_off(gate)) return;
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        int r = r0 + j, c = c0 + threadIdx.x;
        if (r < n && c < p) tile[j][threadIdx.x] = src[(size_t)r * p + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        int c = c0 + j, r = r0 + threadIdx.x;
        if (r < n && c < p) dst[(size_t)c * ld + r] = tile[threadIdx.x][j];
    }
}

bpf_status colmajor_to_rowmajor(bpf_ctx *ctx, int n, int p, const double *src, int ld,
                                double *dst, const int *gate) {
    if (n == 0 || p == 0) return BPF_SUCCESS;
    dim3 grid(ceil_div(n, 32), ceil_div(p, 32)), block(32, 8);
    cm_to_rm_kernel<<<grid, block, 0, ctx->stream>>>(n, p, src, ld, dst, gate);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

bpf_status rowmajor_to_colmajor(bpf_ctx *ctx, int n, int p, const double *src, double *dst,
                                int ld, const int *gate) {
    if (n == 0 || p == 0) return BPF_SUCCESS;
    dim3 grid(ceil_div(n, 32), ceil_div(p, 32)), block(32, 8);
    rm_to_cm_kernel<<<grid, block, 0, ctx->stream>>>(n, p, src, dst, ld, gate);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

}  // namespace bpf
