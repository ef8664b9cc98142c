// tc_gemm.h - the tensor-core products of tc_gemm.cu as mlp.cu launches them.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cumf {

// C[M x N] = act(A[M x K] B[N x K]^T + bias): bf16 operands, fp32 or bf16 output.
cudaError_t launch_tc_gemm(const void *A, const void *B, int M, int N, int K, const float *bias, int act,
                           void *out, int out_f32, int ldo, float *pre_out, int *status, cudaStream_t s);

// The products of a training step whose outputs feed later products both as they are and
// transposed (the weight gradients take both operands K-major, K = the batch rows).  With acc =
// A[M x K] B[N x K]^T, M a multiple of 128 and N of 32:
//   kTrainForward  x = acc + bias;  slope = gelu'(x);  D = gelu(x)
//   kTrainLoss     d = acc + bias - T;                 D = scale d
//   kTrainBack                                         D = acc * slope
// D (bf16) goes to `out` (M x N) and `out_t` (N x M).  kTrainLoss and kTrainBack set D's rows from
// `valid` on to zero and leave D's column sums over each 32 rows in colsum[M / 32][N].
enum TrainMode { kTrainForward, kTrainLoss, kTrainBack };
struct TrainEpilogue {
    const float *bias;
    float *slope;  // M x N: written by kTrainForward, read by kTrainBack
    __nv_bfloat16 *out, *out_t;
    float *colsum;
    int valid;
    const float *T;  // kTrainLoss: `valid` x N; the sums of d^2 over 32 x 32 blocks go to loss[M / 32][N / 32]
    float scale;
    double *loss;
};
cudaError_t launch_train_gemm(TrainMode mode, const void *A, const void *B, int M, int N, int K,
                              const TrainEpilogue &ep, int *status, cudaStream_t s);

// Three products C_j[M_j x N_j] = A_j[M_j x K] B_j[N_j x K]^T over the same K in one launch, K in
// `splits` parts each: out[splits][M][N] (fp32) are the parts' sums.
struct WgradJob {
    const void *A, *B;
    int M, N, splits;
    float *out;
};
constexpr int kWgradJobs = 3;
// The parts that launch_tc_gemm would add for a plain fp32 product, and the most that it would for
// any K up to this one.
int product_splits(int M, int N, int64_t K);
int product_splits_limit(int M, int N, int64_t K);
cudaError_t launch_wgrad(const WgradJob *job, int K, int *status, cudaStream_t s);

}  // namespace cumf
