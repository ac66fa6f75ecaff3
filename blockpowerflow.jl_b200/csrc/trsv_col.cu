// Triangular solves with one right-hand side per CTA, the whole column in shared memory
// (ILU(0) / IC(0) factors of up to 24,767 rows in FP64, about 49,600 in FP32, where that is the faster way:
// prec_by_columns in prec.cu has the line and both sides' times).
//
// Reference: ldiv! of src/preconditioners_nvidia.jl:13-35,49-71 (two cusparseSpSM / SpSV).
//
// What bounds a sparse triangular solve here is the chain of dependency levels, so the design
// makes a level as short as the machine allows.  Passing a row from one CTA to the next goes
// through L2 (a store, a release, a poll and a gather: ~2.5 us a level, measured on the 9,000-bus
// minimum-degree factors), while the right-hand sides are independent of one another: a CTA that
// keeps one column (17k rows: 136 KB) in shared memory never leaves its SM for anything but the
// factor's entries, which no row's result delays, and a level ends with a __syncthreads.
//
//  * With that, the entries' way into the SM is what remains: a level of a long chain lasts
//    ~250 cycles, an L2 round trip ~800.  So the factors are one byte stream in the order in which
//    they are used, cut into chunks of up to 16 KB that a producer warp brings to a ring in shared
//    memory ahead of use by bulk asynchronous copies.
//  * A slab is up to 32 rows of one level, a row per lane; unknowns are numbered by level
//    position within a sweep, so a slab's results are contiguous over the lanes.  Its entries come
//    in groups of four a row (a level's rows are sorted by length, so little is padding), a lane's
//    four 16-bit columns in one 8-byte load and its values in 16-byte loads, and a padding entry
//    is a zero times the unknown after the last, which is zero: no branch or predicate between the
//    barrier and the result (with them a slab took ~1,000 cycles).
//  * An LU's long rows (more than kWideRow entries) are slabs of their own, a row's entries over the
//    32 lanes and a warp sum at the end; an ILU(0)'s too, past kWideIlu entries, where the level's slab would be
//    mostly padding (a slab of one row takes 1,280 bytes per four entries: 3,000 levels of one row of 200
//    entries made 186 MB and 18.0 ms, 2.2 ms so).
//  * Slab g goes to warp g mod nw, levels notwithstanding: a warp fetches its next slab's
//    entries, if they have arrived, then passes the level barriers that separate it from the last,
//    so in a long chain of narrow levels the fetches of the coming levels overlap the current one.
//    A warp waits for entries only when no barrier is left to pass, so the slabs that hold their
//    slot can be finished by their warps: no deadlock, and all waits are bounded.
//  * Between the sweeps the column passes through Y, renumbered; blocks are column-major as in
//    the API, so no layout conversion is needed there, and may be solved in place.
//
// Measured (ldiv_ calls, start of this design -> now): 530 rows, 16 columns 121 -> 20 us; 17k rows, one
// column 196 -> 77 us; 17k rows, 64 columns 143 -> 94 us in minimum-degree order (26 + 26 levels),
// 2,210 -> 575 us in reverse Cuthill-McKee order (456 + 456).  What remains is the instruction
// latency of a slab (~500 cycles from barrier to barrier) and four passes over the column.
// Tried on the way, 17k rows, 64 columns, minimum degree / reverse Cuthill-McKee: entries by plain
// loads one slab ahead (103 / 966 us); rows that poll the values they read in shared memory instead
// of level barriers (113 / 868 us: nearly every warp waits, and the polls take the issue slots from
// the others).
//
// Same products and summation order per row as the level-scheduled kernel, but for the rows over all lanes:
// identical results.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "bpf_internal.cuh"
#include "bulk.cuh"
#include "prec.cuh"

namespace bpf {

constexpr int kChunk = 16384;      // bytes of a chunk, at most
constexpr int kWideRow = 16;       // entries past which an LU's row takes a whole warp
constexpr int kWideIlu = 32;       // and an ILU(0)'s or IC(0)'s, where its level has too few of them for its lanes
constexpr int kColWarps = 23;      // computing warps, at most
constexpr int kChunkRing = 6;      // chunks in flight, at most (as many as fit beside the column)
// Bytes of a sweep's stream, at most (offsets are int): 25 million entries of long rows, or every row with a level
// of its own.  Grids' factors take 1 to 20 MB.
constexpr size_t kStreamMax = size_t(1) << 28;

// A group of four entries of 32 rows: [lane][4] 16-bit columns, then the values as [2][lane][2]
// doubles or [lane][4] floats.
template <typename TF>
struct ColGroup;
template <>
struct ColGroup<double> {
    static constexpr int bytes = 256 + 1024;
    unsigned c[4];
    double a[4];
    __device__ __forceinline__ void load(unsigned p, int lane) {
        unsigned x, y;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(p + 8 * lane));
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a[0]), "=d"(a[1]) : "r"(p + 256 + 16 * lane));
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a[2]), "=d"(a[3]) : "r"(p + 768 + 16 * lane));
        c[0] = x & 0xFFFFu;
        c[1] = x >> 16;
        c[2] = y & 0xFFFFu;
        c[3] = y >> 16;
    }
};
template <>
struct ColGroup<float> {
    static constexpr int bytes = 256 + 512;
    unsigned c[4];
    float a[4];
    __device__ __forceinline__ void load(unsigned p, int lane) {
        unsigned x, y;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(p + 8 * lane));
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3])
                     : "r"(p + 256 + 16 * lane));
        c[0] = x & 0xFFFFu;
        c[1] = x >> 16;
        c[2] = y & 0xFFFFu;
        c[3] = y >> 16;
    }
};
__device__ __forceinline__ double warp_total(double v) { return warp_sum(v); }
__device__ __forceinline__ float warp_total(float v) { return warp_sumf(v); }
// Unknown i of the column at shared address y.
__device__ __forceinline__ void col_get(unsigned y, unsigned i, double &v) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(y + 8 * i));
}
__device__ __forceinline__ void col_get(unsigned y, unsigned i, float &v) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(y + 4 * i));
}
__device__ __forceinline__ void col_put(unsigned y, unsigned i, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(y + 8 * i), "d"(v) : "memory");
}
__device__ __forceinline__ void col_put(unsigned y, unsigned i, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(y + 4 * i), "f"(v) : "memory");
}

struct ColArgs {
    int n, nring;
    const unsigned char *stream[2];
    const int *coff[2], *cslab[2];   // per chunk: byte offset, first slab
    // per slab: first position | rows << 16 | groups of entries << 22 | last part << 27 | one row over
    // all lanes << 28; offset of
    // its entries in the ring | slot << 20 | parity of the slot's phase << 24; stage; chunk (of both
    // sweeps)
    const int4 *head[2];
    int nchunk[2], nslab[2], nstage[2], diag[2];
    const int *pos0, *pos01, *pos1;
    // the LU's dense tail: unknowns s.. of both sweeps, nb tiles of 64 (0: none)
    int s, nb;
    const double *F, *D, *R;   // its tiles, the diagonal ones by columns, the pivots' reciprocals
};

// Counters of the ring, relaxed: `ready` only tells that a slot's mbarrier phase is over (its own wait
// then orders the reads of the slot), and a slab is counted as finished when the entries it read are
// already part of a result.  (Release operations here wait for the global loads in flight: twice
// the time of a level.)
__device__ __forceinline__ unsigned ld_relaxed_cta(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_cta(unsigned *p, unsigned v) {
    asm volatile("st.relaxed.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void red_relaxed_cta(unsigned *p, unsigned v) {
    asm volatile("red.relaxed.cta.shared.add.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
// The barrier of the computing warps (the producer warp takes no part).
__device__ __forceinline__ void col_barrier(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// The ring's shared state: chunks that have arrived, slabs finished per slot.
struct RingState {
    uint64_t full[kChunkRing];
    unsigned done[kChunkRing];
    unsigned ready;
};

// The producer: brings the chunks of both sweeps in order, a chunk into its slot once every slab of
// the slot's previous chunk is finished, and counts the arrived ones in r.ready.  Gives up after lim polls
// without a change (the computing warps' own waits report it), its copies landed.
__device__ __forceinline__ void col_produce(const ColArgs &a, unsigned char *ring, RingState &r, long long lim) {
    const int total = a.nchunk[0] + a.nchunk[1];
    int issued = 0, arrived = 0, islot = 0, aslot = 0;
    unsigned aparity = 0;
    long long idle = 0;
    auto slabs = [&](int c) {
        const int w = c >= a.nchunk[0] ? 1 : 0, k = w ? c - a.nchunk[0] : c;
        return (unsigned)(__ldg(a.cslab[w] + k + 1) - __ldg(a.cslab[w] + k));
    };
    unsigned need = 0;   // slabs of the chunk that the next one to issue replaces
    while (arrived < total) {
        bool moved = false;
        if (issued < total && (issued < a.nring || ld_relaxed_cta(r.done + islot) == need)) {
            const int w = issued >= a.nchunk[0] ? 1 : 0, k = w ? issued - a.nchunk[0] : issued;
            const int o = __ldg(a.coff[w] + k);
            const unsigned bytes = (unsigned)(__ldg(a.coff[w] + k + 1) - o);
            st_relaxed_cta(r.done + islot, 0u);
            mbar_expect_tx(r.full + islot, bytes);
            if (bytes > 0) bulk_g2s(ring + (size_t)islot * kChunk, a.stream[w] + o, bytes, r.full + islot);
            if (++islot == a.nring) islot = 0;
            if (++issued >= a.nring && issued < total) need = slabs(issued - a.nring);
            moved = true;
        }
        if (arrived < issued && mbar_try_wait(r.full + aslot, aparity)) {
            st_relaxed_cta(&r.ready, (unsigned)++arrived);
            if (++aslot == a.nring) {
                aslot = 0;
                aparity ^= 1u;
            }
            moved = true;
        }
        if (moved) idle = 0;
        else if (++idle > lim) break;
    }
    for (; arrived < issued; arrived++) {
        mbar_wait_bounded(r.full + aslot, aparity);
        if (++aslot == a.nring) {
            aslot = 0;
            aparity ^= 1u;
        }
    }
}

// One sweep over the column y (y[n] = 0 for the padding).  A slab's entries: its groups and, with a
// diagonal, 32 inverse diagonals.  A stage's slabs read what earlier stages wrote (a level, or a
// further part of its long rows).
template <typename TF>
__device__ __forceinline__ bool col_sweep(const int4 *head, int nslab, int nstage, bool diag, unsigned y,
                                          unsigned ring, RingState &r, int nw, long long lim, bool ok) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int passed = 0, seen = -1;
    // Headers of the warp's next 32 slabs, one a lane: a global load in flight would be waited for at
    // every level barrier (an L2 round trip a level), so one load serves 32 slabs.
    int4 heads = make_int4(0, 0, 0, 0);
    for (int g = warp, i = 0; ok && g < nslab; g += nw, i = (i + 1) & 31) {
        if (i == 0) heads = __ldg(head + min(g + lane * nw, nslab - 1));
        int4 h;
        h.x = __shfl_sync(0xffffffffu, heads.x, i);
        h.y = __shfl_sync(0xffffffffu, heads.y, i);
        h.z = __shfl_sync(0xffffffffu, heads.z, i);
        h.w = __shfl_sync(0xffffffffu, heads.w, i);
        const int q = h.x & 0xFFFF, rows = (h.x >> 16) & 0x3F, ng = (h.x >> 22) & 0x1F, slot = (h.y >> 20) & 0xF;
        const unsigned parity = (unsigned)(h.y >> 24) & 1u, ch = ring + (unsigned)(h.y & 0xFFFFF);
        ColGroup<TF> e, en;
        // the chunk's arrival is checked once per warp and chunk
        bool early = h.w == seen;
        const unsigned want = (unsigned)h.w + 1u;
        if (!early) early = __all_sync(0xffffffffu, ld_relaxed_cta(&r.ready) >= want && mbar_try_wait(r.full + slot, parity));
        if (early && ng > 0) e.load(ch, lane);
        for (; passed < h.z; passed++) col_barrier(32 * nw);
        if (!early) {
            long long it = 0;
            while (!(ld_relaxed_cta(&r.ready) >= want && mbar_try_wait(r.full + slot, parity)) && ++it < lim) {
            }
            ok = __all_sync(0xffffffffu, it < lim);
            if (!ok) break;
            if (ng > 0) e.load(ch, lane);
        }
        seen = h.w;
        const bool wide = (h.x >> 28) & 1;
        if (wide || lane < rows) {
            TF acc = (TF)0;
            if (!wide || lane == 0) col_get(y, q + lane, acc);
            for (int j = 0; j < ng; j++) {
                TF v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) col_get(y, e.c[u], v[u]);
                if (j + 1 < ng) en.load(ch + (j + 1) * ColGroup<TF>::bytes, lane);
#pragma unroll
                for (int u = 0; u < 4; u++) acc -= e.a[u] * v[u];
                e = en;
            }
            if (wide) acc = warp_total(acc);
            if (diag && ((h.x >> 27) & 1)) {
                TF dv;
                col_get(ch + ng * ColGroup<TF>::bytes, lane, dv);
                acc *= dv;
            }
            if (!wide || lane == 0) col_put(y, q + lane, acc);
        }
        __syncwarp();
        if (lane == 0) red_relaxed_cta(r.done + slot, 1u);
    }
    // every warp passes every barrier, whatever its waits brought
    for (; passed < nstage; passed++) col_barrier(32 * nw);
    return ok;
}

// A warp's four columns of diagonal tile b of the dense tail, rows lane and lane + 32; of U each row times its
// pivot's reciprocal (r), which takes the product out of the substitution's chain.
template <bool UP>
__device__ __forceinline__ void col_tail_load(const ColArgs &a, int b, double (&d)[4][2], double (&r)[2]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (b < 0 || b >= a.nb || warp >= 16) return;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const double *col = a.D + (size_t)b * 4096 + 64 * (UP ? 63 - 4 * warp - c : 4 * warp + c) + lane;
        d[c][0] = __ldg(col);
        d[c][1] = __ldg(col + 32);
    }
    if (UP) {
        r[0] = __ldg(a.R + 64 * b + lane);
        r[1] = __ldg(a.R + 64 * b + 32 + lane);
    }
}

// One sweep over a dense tail in shared memory, at address y, by 64-wide block steps.  The diagonal tile's
// substitution passes through warps 0 - 15, four unknowns each, whose columns of the tile were fetched during the
// step before; then a warp updates four rows at a time, two columns a lane.
template <bool UP>
__device__ __forceinline__ void col_tail(const ColArgs &a, unsigned y, int nw) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t ld = (size_t)a.nb * 64;
    double d[4][2], r[2];
    col_tail_load<UP>(a, UP ? a.nb - 1 : 0, d, r);
#pragma unroll 1
    for (int bi = 0; bi < a.nb; bi++) {
        const int b = UP ? a.nb - 1 - bi : bi;
        const unsigned yb = y + 512 * b;
        const int k0 = UP ? 63 - 4 * warp : 4 * warp;   // the first of the warp's unknowns, downwards in U
        const bool high = (k0 & 32) != 0;
        if (UP) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                d[c][0] *= r[0];
                d[c][1] *= r[1];
            }
        }
#pragma unroll 1
        for (int w = 0; w < 16; w++) {
            if (warp == w) {
                double v0, v1;
                col_get(yb, lane, v0);
                col_get(yb, lane + 32, v1);
                if (UP && w == 0) {
                    v0 *= r[0];
                    v1 *= r[1];
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int k = UP ? k0 - c : k0 + c;
                    const double xk = __shfl_sync(0xffffffffu, high ? v1 : v0, k & 31);
                    if (UP ? lane < k : lane > k) v0 -= d[c][0] * xk;
                    if (UP ? lane + 32 < k : lane + 32 > k) v1 -= d[c][1] * xk;
                }
                col_put(yb, lane, v0);
                col_put(yb, lane + 32, v1);
            }
            col_barrier(32 * nw);
        }
        col_tail_load<UP>(a, UP ? b - 1 : b + 1, d, r);
        double x0, x1;
        col_get(yb, 2 * lane, x0);
        col_get(yb, 2 * lane + 1, x1);
        const double *A = a.F + (size_t)b * 64;
        const int r1 = UP ? 64 * b : 64 * a.nb;
        for (int q = (UP ? 0 : 64 * (b + 1)) + 4 * warp; q < r1; q += 4 * nw) {
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = __ldg(reinterpret_cast<const double2 *>(A + (size_t)(q + u) * ld) + lane);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const double s = warp_sum(v[u].x * x0 + v[u].y * x1);
                if (lane == 0) {
                    double o;
                    col_get(y, q + u, o);
                    col_put(y, q + u, o - s);
                }
            }
        }
        col_barrier(32 * nw);
    }
}

template <typename TF>
__global__ void __launch_bounds__(32 * (kColWarps + 1), 1)
trsv_col_kernel(ColArgs a, const double *X, size_t ldx, double *Y, size_t ldy, size_t step, const int *gate, DevStatus *ds) {
    extern __shared__ __align__(128) unsigned char col_smem[];
    __shared__ RingState r;
    __shared__ int s_off;
    const int nw = (blockDim.x >> 5) - 1;   // computing warps; the last warp is the producer
    if (threadIdx.x == 0) {
        s_off = (gate && *gate == 0) ? 1 : 0;
        for (int b = 0; b < a.nring; b++) {
            mbar_init(r.full + b, 1);
            r.done[b] = 0;
        }
        r.ready = 0;
        mbar_init_fence();
    }
    __syncthreads();
    if (s_off) return;
    unsigned char *ring = col_smem;
    const long long lim = ds->wait_limit > 0 ? ds->wait_limit : kSpinLimit;   // polls of the computing warps' waits
    if ((int)(threadIdx.x >> 5) == nw) {
        if ((threadIdx.x & 31) == 0) col_produce(a, ring, r, 4 * lim);
        return;
    }
    const int n = a.n, tid = threadIdx.x, nt = 32 * nw;
    const unsigned rbase = smem_u32(ring), y = rbase + a.nring * kChunk;
    X += blockIdx.x * ldx;
    Y += blockIdx.x * ldy;
    for (int i = n + tid; i <= max(n, a.s + 64 * a.nb); i += nt) col_put(y, i, (TF)0);
    for (int i0 = tid; i0 < n; i0 += 8 * nt) {   // eight loads in flight
        int at[8];
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = min(i0 + u * nt, n - 1);
            at[u] = __ldg(a.pos0 + i);
            v[u] = X[i * step];
        }
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i0 + u * nt < n) col_put(y, at[u], (TF)v[u]);
    }
    col_barrier(nt);
    bool ok = col_sweep<TF>(a.head[0], a.nslab[0], a.nstage[0], a.diag[0] != 0, y, rbase, r, nw, lim, true);
    if constexpr (std::is_same<TF, double>::value)
        if (a.nb > 0) {
            col_tail<false>(a, y + 8 * a.s, nw);
            col_tail<true>(a, y + 8 * a.s, nw);
        }
    for (int i0 = tid; i0 < n; i0 += 8 * nt) {   // forward results in backward positions, through Y
        int at[8];
#pragma unroll
        for (int u = 0; u < 8; u++) at[u] = __ldg(a.pos01 + min(i0 + u * nt, n - 1));
#pragma unroll
        for (int u = 0; u < 8; u++) {
            TF v;
            col_get(y, at[u], v);
            if (i0 + u * nt < n) Y[(i0 + u * nt) * step] = (double)v;
        }
    }
    col_barrier(nt);
    for (int i0 = tid; i0 < n; i0 += 8 * nt) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = Y[min(i0 + u * nt, n - 1) * step];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i0 + u * nt < n) col_put(y, i0 + u * nt, (TF)v[u]);
    }
    for (int i = n + tid; i <= a.s + 64 * a.nb; i += nt) col_put(y, i, (TF)0);   // (the tail's padding)
    col_barrier(nt);
    ok = col_sweep<TF>(a.head[1], a.nslab[1], a.nstage[1], a.diag[1] != 0, y, rbase, r, nw, lim, ok);
    if (!ok) atomicCAS(&ds->err, 0, (int)DEV_BARRIER_TIMEOUT);
    for (int i0 = tid; i0 < n; i0 += 8 * nt) {
        int at[8];
#pragma unroll
        for (int u = 0; u < 8; u++) at[u] = __ldg(a.pos1 + min(i0 + u * nt, n - 1));
#pragma unroll
        for (int u = 0; u < 8; u++) {
            TF v;
            col_get(y, at[u], v);
            if (i0 + u * nt < n) Y[(i0 + u * nt) * step] = (double)v;
        }
    }
}

// Chunks that fit in shared memory beside the column (1 KB left for the kernel's own variables).
int trsv_col_ring(const bpf_ctx *ctx, int n, int fdtype) {
    const long long left = (long long)ctx->max_smem_optin - 1024 - 512 - (n + 1ll) * (fdtype == BPF_F32 ? 4 : 8);
    return left <= 0 ? 0 : (int)std::min<long long>(kChunkRing, left / kChunk);
}
// Whether a factor of n rows is kept for the column solves: the column and two chunks fit.
bool trsv_col_fits(const bpf_ctx *ctx, int n, int fdtype) { return n < 0xFFFF && trsv_col_ring(ctx, n, fdtype) >= 2; }

bpf_status trsv_col(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, size_t ldx, double *Y, size_t ldy,
                    const int *gate, size_t step) {
    if (P->n == 0 || p == 0) return BPF_SUCCESS;
    const bool f32 = P->fdtype == BPF_F32;
    const size_t es = f32 ? sizeof(float) : sizeof(double);
    ColArgs a;
    a.n = P->n;
    a.nring = trsv_col_ring(ctx, P->n, P->fdtype);
    a.s = P->tail_s;
    a.nb = P->tail_mp / 64;
    a.F = P->tail_F;
    a.D = P->tail_D;
    a.R = P->tail_D + (size_t)P->tail_mp * 64;
    const size_t smem = (size_t)a.nring * kChunk + (std::max(P->n, a.s + P->tail_mp) + 1) * es;
    double fb = 0.0;
    for (int w = 0; w < 2; w++) {
        a.stream[w] = P->cs[w].bytes;
        a.coff[w] = P->cs[w].coff;
        a.nchunk[w] = P->cs[w].nchunk;
        a.cslab[w] = P->cs[w].cslab;
        a.head[w] = reinterpret_cast<const int4 *>(P->cs[w].head);
        a.nslab[w] = P->cs[w].nslab;
        a.nstage[w] = P->cs[w].nstage;
        a.diag[w] = P->cs[w].diag;
        fb += (double)P->cs[w].len;
    }
    a.pos0 = P->pos0;
    a.pos01 = P->pos01;
    a.pos1 = P->pos1;
    // Computing warps for about two average levels, up to kColWarps: more of them only make the barriers of
    // a long chain of narrow levels wider.  One more warp brings the chunks.
    const int per_level = P->n / std::max(1, std::min(P->lower.nlev, P->upper.nlev));
    // (the dense tail of an LU takes 16 at least).
    const int threads = 32 * (1 + std::min(kColWarps, std::max(a.nb > 0 ? 16 : 4, ceil_div(2 * per_level, 32))));
    KScope ks(ctx, BPF_KC_TRSV, fb + 12.0 * P->n + 16.0 * (double)P->n * p,
              2.0 * ((double)P->lower.nnz + P->upper.nnz + P->n) * p);
    auto kern = f32 ? trsv_col_kernel<float> : trsv_col_kernel<double>;
    BPF_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<p, threads, smem, ctx->stream>>>(a, X, ldx, Y, ldy, step, gate, ctx->dstat);
    BPF_LAUNCHED(ctx);
    return BPF_SUCCESS;
}

// The same for row-major blocks: in place, or through a column-major copy in the context's workspace.
bpf_status trsv_col_rowmajor(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, double *Y, const int *gate) {
    if (P->n == 0 || p == 0) return BPF_SUCCESS;
    if (p == 1) return trsv_col(ctx, P, 1, X, P->n, Y, P->n, gate);
    // Small blocks stay in place: a strided value costs a 32-byte sector, four times a column, where the copies
    // cost two launches.  A GMRES iteration with and without the copies: 530 unknowns 16 columns 142 / 134 us, 2,800
    // unknowns 8 columns 139 / 134, 4,700 unknowns 16 columns 208 / 212, 17,000 unknowns 8 columns 410 / 434.
    if (P->n <= 3072) return trsv_col(ctx, P, p, X, 1, Y, 1, gate, p);
    bpf_status s;
    double *buf = (double *)ws_get(ctx, WS_COL, sizeof(double) * (size_t)P->n * p, &s);
    if (!buf) return s;
    BPF_TRY(rowmajor_to_colmajor(ctx, P->n, p, X, buf, P->n, gate));
    BPF_TRY(trsv_col(ctx, P, p, buf, P->n, buf, P->n, gate));
    return colmajor_to_rowmajor(ctx, P->n, p, buf, P->n, Y, gate);
}

// The byte stream of a level-sorted factor.  Rows of a level are re-sorted by length (t.rows, t.rp,
// ... follow); pos[i] = position of row i; tpos[k] = value index (in units of the factor type) of
// pattern entry k in the stream (-2 - index: its reciprocal's).  nring: slots of the ring; chunk0:
// chunks of the sweep before.
// False, with out and tpos in part filled, when the stream would pass kStreamMax.
bool tri_to_stream(TriHost &t, int fdtype, int nring, int chunk0, int ntot, bool lu, std::vector<int> &pos,
                   TriStream &out, std::vector<int> &tpos) {
    const size_t es = fdtype == BPF_F32 ? sizeof(float) : sizeof(double);
    const int n = t.n;
    std::vector<int> ord(n);
    for (int q = 0; q < n; q++) ord[q] = q;
    for (int l = 0; l < t.nlev - (t.keep_last ? 1 : 0); l++)
        std::stable_sort(ord.begin() + t.lev_ptr[l], ord.begin() + t.lev_ptr[l + 1],
                         [&](int x, int y) { return t.rp[x + 1] - t.rp[x] > t.rp[y + 1] - t.rp[y]; });
    TriHost s = t;
    s.rp.assign(n + 1, 0);
    for (int q = 0; q < n; q++) {
        const int o = ord[q], len = t.rp[o + 1] - t.rp[o];
        s.rows[q] = t.rows[o];
        s.rp[q + 1] = s.rp[q] + len;
        std::copy(t.ci.begin() + t.rp[o], t.ci.begin() + t.rp[o + 1], s.ci.begin() + s.rp[q]);
        std::copy(t.map.begin() + t.rp[o], t.map.begin() + t.rp[o + 1], s.map.begin() + s.rp[q]);
        if (!t.unit) s.dmap[q] = t.dmap[o];
    }
    t = std::move(s);
    pos.resize(ntot);
    for (int i = n; i < ntot; i++) pos[i] = i;
    for (int q = 0; q < n; q++) pos[t.rows[q]] = q;

    // a slab part: positions q0.. (rows of them), its entries j0.. in ng groups, whether it is the
    // rows' last part, its stage, whether one row takes all lanes
    struct Part {
        int q0, rows, j0, ng, last, stage, wide;
    };
    const size_t gb = 256 + 128 * es;
    auto part_bytes = [&](int ng) { return ng * gb + (t.unit ? 0 : 32 * es); };
    const int gmax = (int)((kChunk - 32 * es) / gb);   // groups of one part
    std::vector<Part> cur;
    int nslab = 0, stage = 0;
    size_t body = 0, total = 0;
    out.coff.assign(1, 0);
    out.cslab.assign(1, 0);
    auto close = [&]() {
        if (cur.empty()) return;
        const int ns = (int)cur.size();
        size_t off = 0;
        const size_t at = out.bytes.size();
        out.bytes.resize(at + body, 0);
        unsigned char *ch = out.bytes.data() + at;
        for (int k = 0; k < ns; k++) {
            const Part &d = cur[k];
            const int c = chunk0 + (int)out.coff.size() - 1, slot = c % nring;
            for (int v : {d.q0 | (d.rows << 16) | (d.ng << 22) | (d.last << 27) | (d.wide << 28),
                          (slot * kChunk + (int)off) | (slot << 20) | (((c / nring) & 1) << 24), d.stage, c})
                out.head.push_back(v);
            for (int g = 0; g < d.ng; g++) {
                unsigned short *c16 = reinterpret_cast<unsigned short *>(ch + off + g * gb);
                std::fill(c16, c16 + 128, (unsigned short)ntot);   // padding: the zero after the last unknown
                const size_t vbase = (at + off + g * gb + 256) / es;
                for (int r = 0; r < (d.wide ? 32 : d.rows); r++)
                    for (int u = 0; u < 4; u++) {
                        const int row = d.wide ? d.q0 : d.q0 + r;
                        const int e = t.rp[row] + d.j0 + (d.wide ? 128 * g + 4 * r + u : 4 * g + u);
                        if (e >= t.rp[row + 1]) break;
                        c16[4 * r + u] = (unsigned short)pos[t.ci[e]];
                        tpos[t.map[e]] = (int)(vbase + (fdtype == BPF_F32 ? 4 * r + u : 64 * (u / 2) + 2 * r + u % 2));
                    }
            }
            if (!t.unit && d.last)
                for (int r = 0; r < d.rows; r++) tpos[t.dmap[d.q0 + r]] = -2 - (int)((at + off + d.ng * gb) / es + r);
            off += part_bytes(d.ng);
        }
        out.coff.push_back((int)out.bytes.size());
        out.cslab.push_back(nslab);
        cur.clear();
        body = 0;
    };
    auto add = [&](const Part &d) {
        if (!cur.empty() && body + part_bytes(d.ng) > (size_t)kChunk) close();
        cur.push_back(d);
        body += part_bytes(d.ng);
        nslab++;
    };
    for (int l = 0; l < t.nlev; l++) {
        int rest = 0;   // further parts the widest slab needs (each a stage of its own)
        for (int pass = 0; pass <= rest; pass++, stage++) {
            int longest = 0;
            for (int q0 = t.lev_ptr[l], rows; q0 < t.lev_ptr[l + 1]; q0 += rows) {
                const int first = t.rp[q0 + 1] - t.rp[q0];
                int wide = lu ? first > kWideRow : 0;
                if (!lu && first > kWideIlu) {   // the rows of this slab are no longer than its first one
                    int cnt = 1;
                    while (cnt < 32 && q0 + cnt < t.lev_ptr[l + 1] && t.rp[q0 + cnt + 1] - t.rp[q0 + cnt] > kWideIlu) cnt++;
                    wide = cnt * ((first + 127) / 128) < (first + 3) / 4;
                }
                int w = 0;
                for (rows = 0; rows < (wide ? 1 : 32) && q0 + rows < t.lev_ptr[l + 1]; rows++) {
                    const int len = t.rp[q0 + rows + 1] - t.rp[q0 + rows];
                    if (lu && !wide && len > kWideRow) break;
                    w = std::max(w, len);
                }
                const int ng = wide ? (w + 127) / 128 : (w + 3) / 4;
                const int parts = std::max(1, (ng + gmax - 1) / gmax);
                rest = std::max(rest, parts - 1);
                if (pass >= parts) continue;
                const int g0 = pass * gmax;
                const int groups = std::min(gmax, ng - g0);
                total += part_bytes(groups);
                if (total > kStreamMax) return false;
                out.groups += groups;
                longest = std::max(longest, groups);
                add(Part{q0, rows, (wide ? 128 : 4) * g0, groups, pass == parts - 1 ? 1 : 0, stage, wide});
            }
            out.chain += longest;
        }
    }
    close();
    out.diag = t.unit ? 0 : 1;
    out.nstage = stage;
    return true;
}

}  // namespace bpf
