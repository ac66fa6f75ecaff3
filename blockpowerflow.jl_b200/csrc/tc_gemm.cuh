// BF16 tensor-core GEMM (tcgen05, TMEM accumulator) used by the learned warm-start network.
#pragma once

#include "bpf_internal.cuh"

namespace bpf {

// D (M x N, FP32, row stride ldd) = [D +] A (M x K) B (N x K)^T; A and B K-major BF16 (row
// strides lda, ldb, multiples of 8; 16-byte aligned bases); K a multiple of 64.  splits = K
// slices over the grid (0: chosen to fill the SMs); with splits > 1 the slices add into D
// atomically (D is cleared first unless accumulate).  *err_dev is raised if a bounded wait
// gave up.
bpf_status tc_gemm_bf16_tn(bpf_ctx *ctx, int M, int N, int K, const void *A, int lda, const void *B,
                           int ldb, float *D, int ldd, bool accumulate, int *err_dev, int splits = 0);

// One product of a launch.  kTcStore: D = A B^T (one K slice).  kTcPartial: K slice z writes its product at
// D + z * slice; the reader sums the `splits` of them in order.  kTcAdd: slices add to D atomically.
enum TcMode { kTcStore, kTcPartial, kTcAdd };
struct TcProduct {
    int M, N, K, lda, ldb, ldd;
    const void *A, *B;
    float *D;
    int mode;
    int mt, nt, splits, kps;   // tiles; K slices and their length
    size_t slice;              // floats between the slices' partial products (M * ldd)
};
struct TcGroup {
    TcProduct q[2];
    int second;   // first CTA of the second product
};

// The product's tiles and K slices (splits = 0: chosen as tc_gemm_bf16_tn does); mode kTcStore.
TcProduct tc_product(const bpf_ctx *ctx, int M, int N, int K, const void *A, int lda, const void *B, int ldb, float *D,
                     int ldd, int splits = 0);
// One launch for a product, or two that do not depend on each other.
bpf_status tc_gemm_group(bpf_ctx *ctx, const TcProduct &a, const TcProduct *b, int *err_dev);

}  // namespace bpf
