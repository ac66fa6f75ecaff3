// Internal types of the preconditioner / triangular-factor machinery.
#pragma once

#include <algorithm>
#include <memory>
#include <system_error>
#include <thread>
#include <type_traits>
#include <utility>
#include <vector>

#include "bpf_internal.cuh"

namespace bpf {

// A triangular factor analysed on the host: rows stored level by level.
struct TriHost {
    int n = 0;
    int nlev = 0;
    int max_level_rows = 0;
    bool unit = true;
    bool keep_last = false;    // the last level's rows stay in their order (the LU's dense tail)
    std::vector<int> lev_ptr;  // nlev+1, positions into rows
    std::vector<int> rows;     // n, row id at each level-sorted position
    std::vector<int> rp;       // n+1, per level-sorted position
    std::vector<int> ci;       // off-diagonal column ids
    std::vector<int> map;      // position of each off-diagonal entry in the source pattern
    std::vector<int> dmap;     // position of the diagonal in the source pattern (non-unit)
};

// Plain-pointer view passed to kernels.
struct TriKernelArgs {
    int n, nlev, nnz;
    const int *lev_ptr, *rows, *rp, *ci, *map, *dmap;
    double *val;
    float *valf;
    double *dinv;
    float *dinvf;
};

struct TriDev {
    int n = 0, nlev = 0, nnz = 0, max_level_rows = 0;
    bool unit = true;
    std::vector<int> lev_ptr_h;
    int *lev_ptr = nullptr, *rows = nullptr, *rp = nullptr, *ci = nullptr, *map = nullptr,
        *dmap = nullptr;
    double *val = nullptr;
    float *valf = nullptr;
    double *dinv = nullptr;
    float *dinvf = nullptr;
    TriKernelArgs args() const {
        TriKernelArgs a;
        a.n = n;
        a.nlev = nlev;
        a.nnz = nnz;
        a.lev_ptr = lev_ptr;
        a.rows = rows;
        a.rp = rp;
        a.ci = ci;
        a.map = map;
        a.dmap = dmap;
        a.val = val;
        a.valf = valf;
        a.dinv = dinv;
        a.dinvf = dinvf;
        return a;
    }
};

enum PrecKind { PREC_ILU0 = 1, PREC_IC0 = 2, PREC_LU = 3, PREC_BJ = 4 };

TriHost build_tri(int n, const int *rp, const int *ci, const int *diag, int part, bool unit);
// An allocator whose value-less construct leaves the element uninitialised, so resize() of a
// buffer that is written in full right after (tens of millions of update pairs) neither zero-fills
// it nor takes its first-touch page faults on one thread.
template <typename T>
struct NoInitAlloc : std::allocator<T> {
    template <typename U>
    struct rebind {
        using other = NoInitAlloc<U>;
    };
    NoInitAlloc() = default;
    template <typename U>
    NoInitAlloc(const NoInitAlloc<U> &) noexcept {}
    template <typename U>
    void construct(U *p) noexcept(std::is_nothrow_default_constructible<U>::value) {
        ::new (static_cast<void *>(p)) U;
    }
    template <typename U, typename... Args>
    void construct(U *p, Args &&...args) {
        ::new (static_cast<void *>(p)) U(std::forward<Args>(args)...);
    }
};
using PairVec = std::vector<int, NoInitAlloc<int>>;

// f() on up to 16 host threads (this one alone when small); f takes its work from a shared counter, so
// fewer threads than asked do as well.
template <typename F>
void run_threads(bool large, const F &f) {
    const unsigned hw = std::thread::hardware_concurrency();
    const int nthreads = large ? (int)std::min(16u, std::max(1u, hw)) : 1;
    std::vector<std::thread> pool;
    try {
        for (int t = 1; t < nthreads; t++) pool.emplace_back(f);
    } catch (const std::system_error &) {
        // a thread limit: the calling thread takes what the helpers do not
    }
    f();
    for (auto &th : pool) th.join();
}
// Gather lists (bpf_prec::goff, gsrc) of the first `rows` rows of up to kGatherRow entries but those `skip` marks
// (if not empty); returns the number of updates.
constexpr int kGatherRow = 256;
// A list has an int per L entry and entry of its row, updated or not, where an update is two ints as a pair: lists
// are made while they take 256 MB or no more than the pairs would beyond that (grids: 25 ints a row), and never
// past 2^32 ints.
constexpr long long kGatherFree = 1LL << 26;
inline bool gather_fits(long long ints, long long pairs) {
    return ints <= kGatherFree || (ints <= (1LL << 32) && ints <= kGatherFree + 2 * pairs);
}
long long gather_ints(int rows, const std::vector<int> &rp, const std::vector<int> &diag, const std::vector<char> &skip);
long long build_gather(int rows, const std::vector<int> &rp, const std::vector<int> &ci, const std::vector<int> &diag,
                       const std::vector<char> &skip, std::vector<long long> &goff, PairVec &gsrc);
// false (and empty outputs) when the pair count exceeds INT_MAX; count_only: pp alone
bool build_pairs(int n, const int *rp, const int *ci, const int *diag, bool ic,
                 std::vector<int> &pp, PairVec &pdst, PairVec &psrc, bool count_only = false);
// A sweep's factor as the byte stream of the column solves (trsv_col.cu).
struct TriStream {
    std::vector<unsigned char> bytes;
    std::vector<int> coff, cslab, head;   // per chunk: byte offset, first slab; slab headers
    int diag = 0, nstage = 0;
    long long groups = 0, chain = 0;   // groups of entries; their sum over the stages' longest slabs
};
// ntot: unknowns (rows from t.n on keep their positions); lu: long rows over a whole warp
bool tri_to_stream(TriHost &t, int fdtype, int nring, int chunk0, int ntot, bool lu, std::vector<int> &pos,
                   TriStream &out, std::vector<int> &tpos);
// values = false: the schedule only (the values are kept elsewhere)
bpf_status tri_upload(bpf_ctx *ctx, const TriHost &h, TriDev &d, bool values = true);
void tri_free(TriDev &d);
bpf_status tri_scatter(bpf_ctx *ctx, const TriDev &d, const double *fv);

}  // namespace bpf

// The preconditioner object behind the C ABI (NVIDIA_ILU0 / NVIDIA_IC0).
struct bpf_prec {
    bpf_ctx *ctx = nullptr;
    int kind = 0;
    int n = 0, nnz = 0, nrhs = 0;
    int fdtype = BPF_F64;
    // pattern (0-based device copies) and factor values in pattern order
    int *rp = nullptr, *ci = nullptr, *diag = nullptr;
    double *fv = nullptr;
    // Data-flow factorization: the longest row, the longest that goes by pairs (0: none), and the source entry of A per pattern entry (null: the
    // same position; -1: fill, zero)
    int max_row = 0, pair_row = 0;
    int *fsrc = nullptr;
    // Rows of up to kGatherRow entries: per L entry and entry of the row, the position of U's entry that
    // updates it (-1: none), from goff[i] on (-1: a longer row, or lists past their limit: by its update pairs).
    long long *goff = nullptr;
    int *gsrc = nullptr;
    int *pp = nullptr, *pdst = nullptr, *psrc = nullptr;
    long long npairs = 0;
    bpf::TriDev lower;   // forward solve (L unit for ILU0; L for IC0)
    bpf::TriDev upper;   // backward solve (U for ILU0; L' for IC0)
    // LU on a fill pattern (the RF refactorization, lu.cu): rows and columns from tail_s on, tail_m of
    // them padded to tail_mp, are a dense block: tail_S receives the Schur complement, tail_F holds
    // the 64 x 64 tiles of its factors, tail_D the diagonal ones by columns and then the pivots' reciprocals.
    // fend[i]: end of row i's entries before column tail_s.
    // forder: the rows in the order of the factorization, nshort rows a warp takes, then nlong front
    // rows a CTA takes (long rows, and what depends on them), then the tail;
    // cta_nmax / cta_wmax: most entries to eliminate, longest storage of a CTA's row.
    int tail_s = 0, tail_m = 0, tail_mp = 0, nshort = 0, nlong = 0, cta_nmax = 0, cta_wmax = 0;
    long long cta_pairs = 0;
    // (ILU(0) kept for column solves: the stream's order, long rows of a level first.)
    int *forder = nullptr;
    int *fend = nullptr;
    double *tail_S = nullptr, *tail_F = nullptr, *tail_D = nullptr;
    // LU whose front still has more than 2^31 - 1 update pairs (or BPF_LU_PAIRLESS=1): right-looking
    // column steps that find an entry's updates by a search in its row.  Step k (scale column k of L by
    // 1 / u_kk, then apply its updates) waits for the steps that update row k or column k;
    // cl_lev_ptr / cl_ent / cl_row: the L entries of each level's steps and their rows.
    bool pairless = false;
    int cl_nlev = 0, cl_max_level = 0;
    int *cl_lev_ptr = nullptr, *cl_ent = nullptr, *cl_row = nullptr;
    // and its solves in push form (right-looking): per level of each sweep, the factor entries whose
    // source row became final at that level, as (source row, target row, position in fv).
    int ps_nlev[2] = {0, 0}, ps_max_level = 0;
    int *ps_ptr[2] = {nullptr, nullptr}, *ps_src[2] = {nullptr, nullptr},
        *ps_dst[2] = {nullptr, nullptr}, *ps_pos[2] = {nullptr, nullptr};
    // Symmetric reordering (bpf_ilu0_create_ordered): the factors are those of A_hat =
    // A(perm, perm); perm[i] = original row of factor row i; amap[k] = position of A's entry
    // k in A_hat's pattern; zbuf = n x zcols factor-ordered scratch of the solves.
    int ordering = BPF_ORDER_NATURAL;
    int *perm = nullptr, *amap = nullptr;
    std::vector<int> perm_host;
    double *zbuf = nullptr;
    int zcols = 0;
    // Where a factor entry goes in each sweep's storage, per pattern entry: its value's index (the
    // level-sorted val, or the stream in units of the factor type), -1 nowhere, -2 - index its
    // reciprocal (the level-sorted dinv, or the stream).
    int *tpos[2] = {nullptr, nullptr};
    // Column solves (trsv_col.cu): each sweep's factor as a byte stream; lev: the level-sorted storage is kept too,
    // at lpos (as tpos), because some number of columns goes faster that way (prec_by_columns);
    // sums and longest rows of both sweeps that tell which.  pos0[r] / pos1[r] = forward / backward position of the block's row r, pos01[q] =
    // forward position of the row at backward position q.
    bool col = false, lev = true;
    int *lpos[2] = {nullptr, nullptr};
    double col_groups = 0.0, col_chain = 0.0, col_stages = 0.0, long_rows = 0.0;
    struct ColStream {
        unsigned char *bytes = nullptr;
        int *coff = nullptr, *cslab = nullptr, *head = nullptr;
        int nchunk = 0, nslab = 0, nstage = 0, diag = 0;
        size_t len = 0;
    } cs[2];
    int *pos0 = nullptr, *pos01 = nullptr, *pos1 = nullptr;
    // Sync-free triangular solves: one ready word per factor row, 2e when the forward sweep of
    // launch e has produced the row and 2e + 1 after the backward sweep (monotone across
    // launches, so nothing is reset between them).
    unsigned *sf_flags = nullptr;
    mutable unsigned sf_epoch = 0;
    // Block-Jacobi (bpf_block_jacobi_create): rows of each block (nblk x 32, -1 padded), block and
    // local index of every row, dense inverses (nblk x 32 x 32); fv holds A's values.
    int bj_nblk = 0, bj_bs = 0;
    int *bj_rows = nullptr, *bj_blk = nullptr, *bj_loc = nullptr;
    double *bj_inv = nullptr;
};

namespace bpf {
bpf_status prec_setup(bpf_ctx *ctx, int kind, int n, const std::vector<int> &rp,
                      const std::vector<int> &ci, const std::vector<int> &diag, int fdtype,
                      const std::vector<int> &perm, bpf_prec **out);
bpf_status csr_pattern_to_host(bpf_ctx *ctx, const bpf_csr_desc *A, std::vector<int> &rp,
                               std::vector<int> &ci, bool need_diag, std::vector<int> *diag);
bpf_status factor_numeric(bpf_ctx *ctx, bpf_prec *P);
// The whole numeric step from A's values (device, A's entry order): values in, factors in fv and
// in the level-sorted storage of both sweeps.
bpf_status prec_factor(bpf_ctx *ctx, bpf_prec *P, const double *vals);
// Data-flow factorization of the listed rows (order: device, dependencies first) from A's values;
// *taken = false when a row does not fit in shared memory.
bpf_status factor_df(bpf_ctx *ctx, bpf_prec *P, const int *order, int rows, const double *vals, bool *taken);
// LU with a dense tail (lu.cu).
bpf_status lu_setup(bpf_ctx *ctx, int n, const std::vector<int> &rp, const std::vector<int> &ci,
                    const std::vector<int> &diag, const std::vector<int> &fsrc, const std::vector<int> &rowP,
                    const std::vector<int> &colQ, bool *fits, bpf_prec **out);
bpf_status lu_factor(bpf_ctx *ctx, bpf_prec *P, const double *vals);
bpf_status lu_solve(bpf_ctx *ctx, const bpf_prec *P, int nrhs, double *X, int ldx);   // in place
// Column-per-CTA triangular solves (trsv_col.cu) of a preconditioner kept for them (P->col):
// column-major blocks (Y may be X with the same leading dimension; step: doubles between a column's
// elements), or row-major ones.
bool trsv_col_fits(const bpf_ctx *ctx, int n, int fdtype);
int trsv_col_ring(const bpf_ctx *ctx, int n, int fdtype);
bpf_status trsv_col(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, size_t ldx, double *Y, size_t ldy,
                    const int *gate = nullptr, size_t step = 1);
bpf_status trsv_col_rowmajor(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, double *Y,
                             const int *gate = nullptr);
// Whether a solve of p columns goes by the column solves or by the level-sorted kernels.
bool prec_by_columns(const bpf_ctx *ctx, const bpf_prec *P, int p, bool rowmajor);
// Row-major blocks by the level-sorted kernels (no allocation).
bpf_status prec_apply_levels(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, double *Y, const int *gate = nullptr);
bpf_status prec_apply_rowmajor(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X,
                               double *Y, const int *gate = nullptr);
// Reordered preconditioners: make the factor-ordered scratch hold p columns (allocates when it
// grows; prec_apply_rowmajor itself never allocates and rejects p > zcols).
bpf_status prec_reserve_z(bpf_ctx *ctx, bpf_prec *P, int p);
// A's values into the factor storage (a copy, or the scatter through amap when reordered).
bpf_status prec_load_values(bpf_ctx *ctx, bpf_prec *P, const double *vals);
// Block-Jacobi: inverses of the diagonal blocks from fv; Y = P X (row-major, Y may be X).
bpf_status bj_setup(bpf_ctx *ctx, bpf_prec *P);
bpf_status bj_apply_rowmajor(bpf_ctx *ctx, const bpf_prec *P, int p, const double *X, double *Y);
// Y = U^{-1} L^{-1} Y in place (row-major n x p, p <= 256) for an LU factor with push lists.
bpf_status lu_solve_push_rowmajor(bpf_ctx *ctx, const bpf_prec *P, int p, double *Y);
}  // namespace bpf

namespace bpf {
// The storage of the two sweeps that a factor entry goes to: CSR or stream (bpf_prec::tpos), and CSR besides the
// stream (lpos).
struct SweepStore {
    const int *tpos[2], *lpos[2];
    double *val[2], *dinv[2];      // level-sorted storage, FP64 and FP32
    float *valf[2], *dinvf[2];
    unsigned char *stream[2];      // or the streams (column solves), of FP32 values if f32
    int col, f32;
};

__device__ __forceinline__ void sweep_put_level(const SweepStore &s, int w, int t, double v) {
    const int k = t >= 0 ? t : -2 - t;
    if (t >= 0) {
        s.val[w][k] = v;
        s.valf[w][k] = (float)v;
    } else {
        s.dinv[w][k] = v;
        s.dinvf[w][k] = (float)v;
    }
}

__device__ __forceinline__ void sweep_put(const SweepStore &s, int e, double x) {
#pragma unroll
    for (int w = 0; w < 2; w++) {
        const int t = s.tpos[w] ? __ldg(s.tpos[w] + e) : -1;
        if (t == -1) continue;
        const double v = t >= 0 ? x : 1.0 / x;
        const int k = t >= 0 ? t : -2 - t;
        if (!s.col) sweep_put_level(s, w, t, v);
        else if (s.f32) reinterpret_cast<float *>(s.stream[w])[k] = (float)v;
        else reinterpret_cast<double *>(s.stream[w])[k] = v;
        if (s.lpos[w]) sweep_put_level(s, w, __ldg(s.lpos[w] + e), v);
    }
}

SweepStore sweep_store(const bpf_prec *P);
}  // namespace bpf
