// One block-Arnoldi orthogonalization in one launch (arnoldi.cu).
#pragma once

#include "bpf_internal.cuh"
#include "dense.cuh"

namespace bpf {

// Whether blocks of p columns and n rows go by arnoldi_step.
bool arnoldi_ok(const bpf_ctx *ctx, int n, int p);
// Doubles of WS_PARTIAL that arnoldi_step needs at iteration k.
size_t arnoldi_partials(const bpf_ctx *ctx, int n, int p, int k);
// Iteration k (1-based) of block-GMRES from Q (n x p row-major, the preconditioned product): the
// coefficients Psi (k blocks p x p) of two Gram-Schmidt passes against V_0..V_{k-1}, the orthonormal
// block Vn and its R factor C; re-orthogonalization of an ill-conditioned block folded into Psi and C.
// Psi2: k blocks of scratch.  qr_only: Q is projected already, with its coefficients in Psi.  A breakdown records k in st->qr_fail_iter.  Skipped when !st->active.
bpf_status arnoldi_step(bpf_ctx *ctx, int n, int p, int k, const double *V, size_t strideV, const double *Q, double *Vn,
                        double *Psi, double *Psi2, double *C, SolveState *st, bool qr_only = false);

}  // namespace bpf
