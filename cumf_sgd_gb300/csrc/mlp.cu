// mlp.cu - the learned warm start: user features and a small MLP that maps them to an
// initial user-factor row, trained and run on the tensor cores (tc_gemm.cu).
//
// Features of user u (k + 3 values), from the user's ratings and the item factors Q:
//   x[0:k] = sum_i (r_ui - mean_u) q_i / deg_u      (rating-centred mean of the rated items)
//   x[k]   = log(1 + deg_u) / 4,  x[k+1] = (mean_u - 3) / 2,  x[k+2] = var_u / 2
// The centred mean is zero for a user with one rating, so users with few ratings stay inside
// the range the network was trained on (an uncentred mean of one item's factors does not).
// MLP: d_in -> H (GELU) -> H (GELU) -> d_out, bf16 weights and activations, fp32
// accumulation (tcgen05), fp32 master weights updated with Adam.  Every matrix product of the
// forward and backward passes is a TN product C = A B^T on the tcgen05 GEMM:
//   forward   H1 = gelu(X W1^T + b1), H2 = gelu(H1 W2^T + b2), Y = H2 W3^T + b3
//   backward  dW = dZ^T A  ->  (dZ^T)(A^T)^T on transposed copies; dA = dZ W -> dZ (W^T)^T
// Loss: mean over rows of the squared error summed over the output dimension.
#include <cub/cub.cuh>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <string>
#include <vector>

#include "cumf_sgd.h"
#include "index_walk.h"
#include "internal.h"
#include "rng.h"
#include "tc_gemm.h"
#include "train_common.h"

namespace cumf {

namespace {

constexpr int kT = 256;

int grid_of(int64_t n) {
    int64_t g = (n + kT - 1) / kT;
    if (g > 152 * 64) g = 152 * 64;
    return (int)(g < 1 ? 1 : g);
}

// ---- feature gather --------------------------------------------------------------------

__global__ void user_stats_kernel(const cumf_node *R, int64_t nnz, int32_t m, int32_t n, float *deg, float *sum,
                                  float *sum2) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const cumf_node x = R[i];
        if ((uint32_t)x.u >= (uint32_t)m || (uint32_t)x.v >= (uint32_t)n) continue;
        atomicAdd(deg + x.u, 1.f);
        atomicAdd(sum + x.u, x.r);
        atomicAdd(sum2 + x.u, x.r * x.r);
    }
}

// One warp per rating: acc[u][0:k] += (r - mean_u) q_v / deg_u.
__global__ void user_qsum_kernel(const cumf_node *R, int64_t nnz, int32_t m, int32_t n, const float *Q, int k,
                                 const float *deg, const float *sum, float *X, int ldx) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = w0; i < nnz; i += nw) {
        const cumf_node x = R[i];
        if ((uint32_t)x.u >= (uint32_t)m || (uint32_t)x.v >= (uint32_t)n) continue;
        const float d = deg[x.u];
        const float c = (x.r - sum[x.u] / d) / d;
        const float *q = Q + (int64_t)x.v * k;
        float *dst = X + (int64_t)x.u * ldx;
        if ((k & 3) == 0 && (ldx & 3) == 0) {  // 16-byte vector atomics (sm_90+)
            const float4 *q4 = reinterpret_cast<const float4 *>(q);
            float4 *d4 = reinterpret_cast<float4 *>(dst);
            for (int j = lane; j < (k >> 2); j += 32) {
                const float4 a = q4[j];
                atomicAdd(d4 + j, make_float4(c * a.x, c * a.y, c * a.z, c * a.w));
            }
        } else {
            for (int j = lane; j < k; j += 32) atomicAdd(dst + j, c * q[j]);
        }
    }
}

// Sort keys of the ratings: the user, or m for a rating outside [0, m) x [0, n) (sorted last
// and left out); values: the rating and its item's bits, which travel with the key (the sort of
// 5.2 M pairs took 141 us with 8-byte values as with 4-byte indices), so that what follows reads
// them in order instead of gathering the records.
__global__ void user_keys_kernel(const cumf_node *R, uint32_t nnz, int32_t m, int32_t n, uint32_t *key,
                                 float2 *val) {
    index_walk(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, nnz, [&](uint32_t i) {
        const cumf_node x = R[i];
        const bool ok = (uint32_t)x.u < (uint32_t)m && (uint32_t)x.v < (uint32_t)n;
        key[i] = ok ? (uint32_t)x.u : (uint32_t)m;
        val[i] = make_float2(x.r, __int_as_float(x.v));
    });
}

// seg[u] = the first sorted position whose key is >= u, u = 0..m (binary search).
__global__ void user_segments_kernel(const uint32_t *key, uint32_t nnz, int32_t m, int64_t *seg) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u <= m; u += (int64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nnz;
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (key[mid] < (uint32_t)u) lo = mid + 1;
            else hi = mid;
        }
        seg[u] = lo;
    }
}

// V consecutive floats in one load (the caller checks the alignment).
template <int V>
__device__ __forceinline__ void load_cols(float (&dst)[V], const float *src) {
    if constexpr (V == 4) {
        const float4 x = __ldg(reinterpret_cast<const float4 *>(src));
        dst[0] = x.x, dst[1] = x.y, dst[2] = x.z, dst[3] = x.w;
    } else if constexpr (V == 2) {
        const float2 x = __ldg(reinterpret_cast<const float2 *>(src));
        dst[0] = x.x, dst[1] = x.y;
    } else {
        dst[0] = __ldg(src);
    }
}

// One warp per user over the user's ratings in their original order (a stable sort by user):
// the rating sum and sum of squares by a fixed-order warp reduction, then
// sum (r - mean) q / deg accumulated rating by rating in registers; X[u] = (that sum,
// log(1 + deg)/4, (mean - 3)/2, var/2).  A lane owns V consecutive columns (one load of V
// floats per rating) in each of G groups, 32 V G columns per pass.  The ratings are fetched 32
// at a time (one per lane, then broadcast), the next 32 while these are used; the item rows of
// four ratings are loaded before they are added, in rating order.  No atomics: the features
// are the same bits on every run and for every V and G.
//
// Bound by the item rows out of L2 (512 bytes per rating at 128 columns).  5.2 M ratings, 50,000
// users, 128 columns: 360 us with the records gathered through a sorted index and four
// loads of one float per rating, 150 us so; eight rows in flight are no faster.
template <int V, int G>
__global__ void __launch_bounds__(kT) user_rows_kernel(const float2 *val, const int64_t *seg, int32_t m,
                                                       const float *Q, int k, float *X, int ldx) {
    constexpr int F = 4;
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t u = w0; u < m; u += nw) {
        const int64_t a = seg[u];
        const uint32_t cnt = (uint32_t)(seg[u + 1] - a);
        const float2 *row = val + a;
        float s = 0.f, s2 = 0.f;
        index_walk<4>(lane, 32, cnt, [&](uint32_t t) {
            const float r = row[t].x;
            s += r;
            s2 += r * r;
        });
        for (int o = 16; o >= 1; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        const float d = (float)cnt;
        const float mean = cnt > 0 ? s / d : 0.f;
        float *xu = X + u * ldx;
        for (int c0 = 0; c0 < k; c0 += 32 * V * G) {
            const int cl = c0 + lane * V;  // this lane's first column; a group is 32 V further
            float acc[G][V];
            const float *q0[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                q0[g] = Q + (cl + g * 32 * V < k ? cl + g * 32 * V : 0);  // a lane past k loads column 0, unused
#pragma unroll
                for (int j = 0; j < V; ++j) acc[g][j] = 0.f;
            }
            float2 next = make_float2(0.f, 0.f);
            if ((uint32_t)lane < cnt) next = row[lane];
            index_walk(0, 32, cnt, [&](uint32_t t0) {
                const float c = (next.x - s / d) / d;
                const int item = __float_as_int(next.y);
                if (cnt - t0 > 32 + (uint32_t)lane) next = row[t0 + 32 + lane];
                const int some = (int)(cnt - t0 < 32 ? cnt - t0 : 32);
                float c4[F], q[F][G][V];
                int j0 = 0;
                for (; j0 + F <= some; j0 += F) {
#pragma unroll
                    for (int h = 0; h < F; ++h) {
                        c4[h] = __shfl_sync(0xffffffffu, c, j0 + h);
                        const int64_t at = (int64_t)__shfl_sync(0xffffffffu, item, j0 + h) * k;
#pragma unroll
                        for (int g = 0; g < G; ++g) load_cols<V>(q[h][g], q0[g] + at);
                    }
#pragma unroll
                    for (int h = 0; h < F; ++h)
#pragma unroll
                        for (int g = 0; g < G; ++g)
#pragma unroll
                            for (int j = 0; j < V; ++j) acc[g][j] += c4[h] * q[h][g][j];
                }
                for (; j0 < some; ++j0) {
                    c4[0] = __shfl_sync(0xffffffffu, c, j0);
                    const int64_t at = (int64_t)__shfl_sync(0xffffffffu, item, j0) * k;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        load_cols<V>(q[0][g], q0[g] + at);
#pragma unroll
                        for (int j = 0; j < V; ++j) acc[g][j] += c4[0] * q[0][g][j];
                    }
                }
            });
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (cl + g * 32 * V < k) {
#pragma unroll
                    for (int j = 0; j < V; ++j) xu[cl + g * 32 * V + j] = acc[g][j];
                }
        }
        if (lane == 0) {
            xu[k] = logf(1.f + d) * 0.25f;
            xu[k + 1] = cnt > 0 ? (mean - 3.f) * 0.5f : 0.f;
            xu[k + 2] = (cnt > 0 ? fmaxf(s2 / d - mean * mean, 0.f) : 0.f) * 0.5f;
        }
    }
}

// The widest load that every row of Q allows (k and the base a multiple of it) and that still
// gives most lanes a column: 4 floats from 65 columns on, 2 from 33 on.
void launch_user_rows(int grid, const float2 *val, const int64_t *seg, int32_t m, const float *Q, int k, float *X,
                      cudaStream_t s) {
    auto can = [&](int v) { return k % v == 0 && reinterpret_cast<uintptr_t>(Q) % (4 * v) == 0; };
    if (k > 128 && can(4)) user_rows_kernel<4, 2><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
    else if (k > 64 && can(4)) user_rows_kernel<4, 1><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
    else if (k > 32 && k <= 64 && can(2)) user_rows_kernel<2, 1><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
    else if (k <= 32) user_rows_kernel<1, 1><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
    else if (k <= 64) user_rows_kernel<1, 2><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
    else user_rows_kernel<1, 4><<<grid, kT, 0, s>>>(val, seg, m, Q, k, X, k + 3);
}

// x[u] = (acc[u][0:k], log(1 + deg)/4, (mean - 3)/2, var/2) for the m users (ldx = k + 3).
__global__ void user_finish_kernel(int32_t m, int k, const float *acc, const float *deg, const float *sum,
                                   const float *sum2, float *X, int ldx) {
    const int64_t total = (int64_t)m * ldx;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t u = i / ldx;
        const int c = (int)(i - u * ldx);
        if (c < k) {
            X[i] = acc[u * k + c];
            continue;
        }
        const float d = deg[u];
        const float mean = d > 0 ? sum[u] / d : 0.f;
        if (c == k)
            X[i] = logf(1.f + d) * 0.25f;
        else if (c == k + 1)
            X[i] = d > 0 ? (mean - 3.f) * 0.5f : 0.f;
        else
            X[i] = (d > 0 ? fmaxf(sum2[u] / d - mean * mean, 0.f) : 0.f) * 0.5f;
    }
}

// ---- 32 x 32 tile kernels: an elementwise result written row-major and transposed --------
//
// The weight-gradient products dW = dZ^T A take both operands K-major (K = the batch rows), and
// the products dA = dZ W take W transposed, so the batch's features and the bf16 weights are
// needed row-major and transposed (activations and their gradients get both copies from the
// products' epilogues).  A block computes a 32 x 32 tile, writes it row-major, stages it in shared
// memory (fp32, conflict-free) and writes the transpose.
constexpr int kTile = 32;
constexpr int kTileRows = 8;  // threads per column of a tile (blockDim = 32 x 8)

// Dt[c][r] = tile[r - r0][c - c0] for the tile's valid rows r < nr and columns c < nc.
__device__ __forceinline__ void store_tile_t(const float (*tile)[kTile + 1], __nv_bfloat16 *Dt, int64_t ldt, int r0,
                                             int c0, int nr, int nc) {
    for (int j = threadIdx.y; j < kTile; j += kTileRows) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (c < nc && r < nr) Dt[(int64_t)c * ldt + r] = __float2bfloat16_rn(tile[threadIdx.x][j]);
    }
}

// D (rp x ldd bf16) and, when Dt != NULL, Dt (ldd x rp) from the fp32 rows of S (cols wide):
// row r < valid is S[perm[*batch_idx * batch + r]] (perm NULL: S[r]); other rows and the
// columns cols..ldd are zero.  With F instead of D, the valid rows as fp32 (ldd wide).
struct ConvertJob {
    const float *S;
    int cols;
    const int32_t *perm;
    const int *batch_idx;
    int64_t batch;
    int valid, rp, ldd;
    __nv_bfloat16 *D, *Dt;
    float *F;
};
struct ConvertJobs {
    ConvertJob job[3];  // blockIdx.z picks one; tiles outside its rp x ldd return
    int64_t *step;      // not NULL: Adam's step count, which this launch advances
};

__global__ void __launch_bounds__(kTile * kTileRows) convert_t_kernel(const __grid_constant__ ConvertJobs jobs) {
    if (jobs.step && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0) ++*jobs.step;
    const ConvertJob &jb = jobs.job[blockIdx.z];
    const float *S = jb.S;
    const int cols = jb.cols, valid = jb.valid, rp = jb.rp, ldd = jb.ldd;
    __nv_bfloat16 *D = jb.D, *Dt = jb.Dt;
    __shared__ float tile[kTile][kTile + 1];
    const int r0 = blockIdx.x * kTile, c0 = blockIdx.y * kTile;
    if (r0 >= rp || c0 >= ldd) return;
    const int32_t *idx = jb.perm ? jb.perm + (int64_t)*jb.batch_idx * jb.batch : nullptr;
    for (int j = threadIdx.y; j < kTile; j += kTileRows) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        float v = 0.f;
        if (r < valid && c < cols) v = S[(int64_t)(idx ? idx[r] : r) * cols + c];
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        if (jb.F) {
            if (r < valid && c < cols) jb.F[(int64_t)r * ldd + c] = v;
            continue;
        }
        if (r < rp && c < ldd) D[(int64_t)r * ldd + c] = b;
        tile[j][threadIdx.x] = __bfloat162float(b);
    }
    if (!Dt) return;
    __syncthreads();
    store_tile_t(tile, Dt, rp, r0, c0, rp, ldd);
}

struct Adam {
    float *w, *m1, *m2;
    float lr, b1, b2, eps;
    const int64_t *step;  // t, the number of this step; NULL: gradients only
};

// Adam's update of element i (value w, moments m1 and m2) with gradient g; returns the new
// value.  c1, c2: 1 - b1^t, 1 - b2^t.  The moments' roundings are spelled out: left to the
// compiler's choice of fma they change with the code around them, and a last bit here travels
// through the bf16 weights.
__device__ __forceinline__ float adam_element(const Adam &ad, int64_t i, float g, float w, float m1, float m2,
                                              float c1, float c2) {
    const float a = __fmaf_rn(1.f - ad.b1, g, __fmul_rn(ad.b1, m1));
    const float b = __fmaf_rn(__fmul_rn(1.f - ad.b2, g), g, __fmul_rn(ad.b2, m2));
    ad.m1[i] = a;
    ad.m2[i] = b;
    w -= ad.lr * (a / c1) / (sqrtf(b / c2) + ad.eps);
    ad.w[i] = w;
    return w;
}

// What follows a step's products: the weight gradients' K parts and the bias gradients' tile
// sums added (in order), the gradients stored, Adam's update, the bf16 copies and transposes of
// the new weights, and the loss.  Blocks first[l].. take the 32 x 32 tiles of weight l, blocks
// first[3 + l].. 32 columns of bias l, the last block the loss and the device state.
struct FinishWeight {
    const float *part;  // [splits][rows][ld]
    int64_t off;
    int rows, cols, ld;  // ld >= cols: the padded columns of W1 are left out
    int splits;
    __nv_bfloat16 *b, *bt;
};
struct FinishBias {
    const float *part;  // [tiles][cols]
    int64_t off;
    int cols;
};
struct FinishArgs {
    FinishWeight w[3];
    FinishBias bias[3];
    int first[7];
    int tiles;  // parts of a bias gradient
    float *grads;
    Adam adam;
    const double *loss_part;
    int loss_parts;
    double *loss, *loss_sum;
    int *batch_idx;  // advanced, and loss added to loss_sum, where not NULL
};

__global__ void __launch_bounds__(kTile * kTileRows) finish_step_kernel(const __grid_constant__ FinishArgs args) {
    __shared__ float tile[kTile][kTile + 1];
    __shared__ float corr[2];
    __shared__ double sums[kTileRows];
    const int bx = (int)blockIdx.x, tx = threadIdx.x, ty = threadIdx.y;
    const bool adam = args.adam.step != nullptr;
    if (adam && tx == 0 && ty == 0) {
        const float t = (float)*args.adam.step;
        corr[0] = 1.f - powf(args.adam.b1, t);
        corr[1] = 1.f - powf(args.adam.b2, t);
    }
    __syncthreads();
    const float c1 = corr[0], c2 = corr[1];
    if (bx >= args.first[6]) {  // loss
        double acc = 0;
        for (int i = ty * kTile + tx; i < args.loss_parts; i += kTile * kTileRows) acc += args.loss_part[i];
        for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (tx == 0) sums[ty] = acc;
        __syncthreads();
        if (tx == 0 && ty == 0) {
            double total = 0;
            for (int y = 0; y < kTileRows; ++y) total += sums[y];
            *args.loss = total;
            if (args.batch_idx) {
                ++*args.batch_idx;
                *args.loss_sum += total;
            }
        }
        return;
    }
    int l = 0;
    while (bx >= args.first[l + 1]) ++l;
    const int at = bx - args.first[l];
    if (l >= 3) {  // bias: lane y adds tiles y, y + 8, .. in order, then the 8 lane sums are added in order
        const FinishBias &fb = args.bias[l - 3];
        const int c = at * kTile + tx;
        float sum = 0.f;
        if (c < fb.cols)
            for (int t = ty; t < args.tiles; t += kTileRows) sum += fb.part[(int64_t)t * fb.cols + c];
        tile[ty][tx] = sum;
        __syncthreads();
        if (ty == 0 && c < fb.cols) {
            float g = 0.f;
            for (int y = 0; y < kTileRows; ++y) g += tile[y][tx];
            args.grads[fb.off + c] = g;
            const int64_t i = fb.off + c;
            if (adam) adam_element(args.adam, i, g, args.adam.w[i], args.adam.m1[i], args.adam.m2[i], c1, c2);
        }
        return;
    }
    const FinishWeight &fw = args.w[l];
    const int tiles_c = (fw.cols + kTile - 1) / kTile;
    const int r0 = at / tiles_c * kTile, c0 = at % tiles_c * kTile;
    const int c = c0 + tx;
    const int64_t part = (int64_t)fw.rows * fw.ld;
    constexpr int kRows = kTile / kTileRows;  // this thread's rows of the tile, loaded together
    const bool in = c < fw.cols;
    float g[kRows], w[kRows], m1[kRows], m2[kRows];
    const float *p = fw.part + (int64_t)(r0 + ty) * fw.ld + c;
    const int64_t i0 = fw.off + (int64_t)(r0 + ty) * fw.cols + c;
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
        const int64_t i = i0 + (int64_t)q * kTileRows * fw.cols;
        g[q] = in ? p[(int64_t)q * kTileRows * fw.ld] : 0.f;
        const bool load = in && adam;
        w[q] = load ? args.adam.w[i] : 0.f;
        m1[q] = load ? args.adam.m1[i] : 0.f;
        m2[q] = load ? args.adam.m2[i] : 0.f;
    }
    if (in)
#pragma unroll 4
        for (int z = 1; z < fw.splits; ++z)
#pragma unroll
            for (int q = 0; q < kRows; ++q) g[q] += p[z * part + (int64_t)q * kTileRows * fw.ld];
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
        float v = 0.f;
        if (in) {
            const int64_t i = i0 + (int64_t)q * kTileRows * fw.cols;
            args.grads[i] = g[q];
            if (adam) {
                const __nv_bfloat16 b = __float2bfloat16_rn(adam_element(args.adam, i, g[q], w[q], m1[q], m2[q], c1, c2));
                fw.b[(int64_t)(r0 + ty + q * kTileRows) * fw.ld + c] = b;
                v = __bfloat162float(b);
            }
        }
        tile[ty + q * kTileRows][tx] = v;
    }
    if (!adam || !fw.bt) return;
    __syncthreads();
    store_tile_t(tile, fw.bt, fw.rows, r0, c0, fw.rows, fw.cols);
}

__global__ void init_weights_kernel(float *w, int64_t n, float scale, uint64_t key) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        // uniform(-scale, scale) from the counter hash
        const float u = init_uniform(key, (uint64_t)i);  // (0, 1]
        w[i] = (2.f * u - 1.f) * scale;
    }
}

}  // namespace

struct Mlp {
    int d_in, dp, h, d_out;  // dp = d_in padded to a multiple of 64
    // fp32 parameters (flattened: W1[h][d_in], b1[h], W2[h][h], b2[h], W3[d_out][h], b3[d_out])
    DevBuf params, grads, m1, m2;
    int64_t count = 0;
    int64_t off_w1, off_b1, off_w2, off_b2, off_w3, off_b3;
    // bf16 operand copies: W1p[h][dp], W2[h][h], W3[d_out][h] and transposes W2T[h][h], W3T[h][d_out]
    DevBuf w1b, w2b, w3b, w2t, w3t;
    DevBuf status;
    int64_t step = 0;
    // workspace for batches of up to cap_fwd rows (forward) / cap rows (backward)
    int64_t cap = 0;      // rows of the backward buffers
    int64_t cap_fwd = 0;  // rows of the forward buffers
    DevBuf xb, tb, h1, h2, slope1, slope2, dy, dyt, h2t, h1t, xbt, dp2, dp2t, dp1, dp1t, loss;
    DevBuf wpart;  // the weight gradients' K parts (W1 padded to [h][dp])
    DevBuf colws;  // (cap / 32) x (h + h + d_out) column sums over 32 rows
    DevBuf lossp;  // (cap / 32) x (d_out / 32) sums of squared errors
};

namespace {

// dW1 = dZ1^T X (padded input columns give columns that are left out), dW2 = dZ2^T H1,
// dW3 = dY^T H2 over rp rows, their K parts in mp->wpart.
void wgrad_jobs(Mlp *mp, int64_t rp, WgradJob *job) {
    const int h = mp->h, dout = mp->d_out, dp = mp->dp;
    job[0] = {mp->dp1t.p, mp->xbt.p, h, dp, 0, nullptr};
    job[1] = {mp->dp2t.p, mp->h1t.p, h, h, 0, nullptr};
    job[2] = {mp->dyt.p, mp->h2t.p, dout, h, 0, nullptr};
    float *out = mp->wpart.as<float>();
    for (int j = 0; j < kWgradJobs; ++j) {
        job[j].splits = product_splits(job[j].M, job[j].N, rp);
        job[j].out = out;
        out += (int64_t)job[j].splits * job[j].M * job[j].N;
    }
}

// Workspace for batches of up to `rows` rows: the forward buffers, and with `train` also
// those of the backward pass (the batch's targets, the activations' transposes and slopes, gradients).
// A capacity is 0 while its buffers are replaced: where one cannot be had, the others have gone.
int mlp_ensure(Mlp *mp, int64_t rows, bool train) {
    const int64_t r = (rows + 127) / 128 * 128;
    const size_t b2 = 2;
    const int h = mp->h, dp = mp->dp, dout = mp->d_out;
    if (rows > mp->cap_fwd) {
        mp->cap_fwd = 0;
        CUMF_CUDA(mp->xb.alloc(r * dp * b2));
        CUMF_CUDA(mp->h1.alloc(r * h * b2));
        CUMF_CUDA(mp->h2.alloc(r * h * b2));
        mp->cap_fwd = r;
    }
    if (!train || rows <= mp->cap) return CUMF_OK;
    mp->cap = 0;
    CUMF_CUDA(mp->tb.alloc(r * dout * 4));
    CUMF_CUDA(mp->slope1.alloc(r * h * 4));
    CUMF_CUDA(mp->slope2.alloc(r * h * 4));
    CUMF_CUDA(mp->dy.alloc(r * dout * b2));
    CUMF_CUDA(mp->dyt.alloc(r * dout * b2));
    CUMF_CUDA(mp->h2t.alloc(r * h * b2));
    CUMF_CUDA(mp->h1t.alloc(r * h * b2));
    CUMF_CUDA(mp->xbt.alloc(r * dp * b2));
    CUMF_CUDA(mp->dp2.alloc(r * h * b2));
    CUMF_CUDA(mp->dp2t.alloc(r * h * b2));
    CUMF_CUDA(mp->dp1.alloc(r * h * b2));
    CUMF_CUDA(mp->dp1t.alloc(r * h * b2));
    CUMF_CUDA(mp->colws.alloc((r / kTile) * (2 * h + dout) * 4));
    CUMF_CUDA(mp->lossp.alloc((r / kTile) * (dout / kTile) * sizeof(double)));
    const int wm[kWgradJobs] = {h, h, dout}, wn[kWgradJobs] = {dp, h, h};
    size_t parts = 0;
    for (int j = 0; j < kWgradJobs; ++j) parts += (size_t)product_splits_limit(wm[j], wn[j], r) * wm[j] * wn[j];
    CUMF_CUDA(mp->wpart.alloc(parts * 4));
    mp->cap = r;
    return CUMF_OK;
}

const dim3 kTileBlock(kTile, kTileRows);

dim3 tiles_of(int64_t rows, int cols) { return dim3((unsigned)((rows + kTile - 1) / kTile), (unsigned)((cols + kTile - 1) / kTile)); }

ConvertJob convert_job(const float *S, int cols, const int32_t *perm, const int *batch_idx, int64_t batch, int valid,
                       int rp, int ldd, void *D, void *Dt) {
    return ConvertJob{S, cols, perm, batch_idx, batch, valid, rp, ldd, static_cast<__nv_bfloat16 *>(D),
                      static_cast<__nv_bfloat16 *>(Dt), nullptr};
}

// n (1..3) conversions in one launch.
cudaError_t convert(const ConvertJob *job, int n, cudaStream_t s, int64_t *step = nullptr) {
    ConvertJobs jobs{};
    jobs.step = step;
    unsigned gx = 1, gy = 1;
    for (int i = 0; i < n; ++i) {
        jobs.job[i] = job[i];
        const dim3 g = tiles_of(job[i].rp, job[i].ldd);
        gx = g.x > gx ? g.x : gx;
        gy = g.y > gy ? g.y : gy;
    }
    convert_t_kernel<<<dim3(gx, gy, n), kTileBlock, 0, s>>>(jobs);
    return cudaGetLastError();
}

// bf16 operand copies of the fp32 master weights.
int mlp_refresh(Mlp *mp, cudaStream_t s) {
    const float *P = mp->params.as<float>();
    const int h = mp->h, dout = mp->d_out;
    const ConvertJob jobs[3] = {
        convert_job(P + mp->off_w1, mp->d_in, nullptr, nullptr, 0, h, h, mp->dp, mp->w1b.p, nullptr),
        convert_job(P + mp->off_w2, h, nullptr, nullptr, 0, h, h, h, mp->w2b.p, mp->w2t.p),
        convert_job(P + mp->off_w3, h, nullptr, nullptr, 0, dout, dout, h, mp->w3b.p, mp->w3t.p)};
    CUMF_CUDA(convert(jobs, 3, s));
    return CUMF_OK;
}

// Y (fp32 rows x d_out) of rows [0, rows) of X (fp32 rows x d_in).
int mlp_forward_ws(Mlp *mp, const float *X, int64_t rows, float *Y, cudaStream_t s) {
    if (int rc = mlp_ensure(mp, rows, false)) return rc;
    const float *P = mp->params.as<float>();
    const int h = mp->h;
    const int64_t rp = (rows + 127) / 128 * 128;  // padding rows are zero
    const ConvertJob job = convert_job(X, mp->d_in, nullptr, nullptr, 0, (int)rows, (int)rp, mp->dp, mp->xb.p, nullptr);
    CUMF_CUDA(convert(&job, 1, s));
    int *st = mp->status.as<int>();
    CUMF_CUDA(launch_tc_gemm(mp->xb.p, mp->w1b.p, (int)rp, h, mp->dp, P + mp->off_b1, 1, mp->h1.p, 0, h, nullptr, st, s));
    CUMF_CUDA(launch_tc_gemm(mp->h1.p, mp->w2b.p, (int)rp, h, h, P + mp->off_b2, 1, mp->h2.p, 0, h, nullptr, st, s));
    CUMF_CUDA(launch_tc_gemm(mp->h2.p, mp->w3b.p, (int)rows, mp->d_out, h, P + mp->off_b3, 0, Y, 1, mp->d_out, nullptr,
                             st, s));
    return CUMF_OK;
}

// The batch of a step: row r is X[perm[*batch_idx * batch + r]] (perm NULL: X[r]), T likewise.
struct Batch {
    const float *X, *T;
    int64_t rows;
    const int32_t *perm;
    int *batch_idx;
    int64_t batch;
};

// Loss (mp->loss) and gradients (mp->grads) of a batch; with `adam` (its step count advanced
// first), also the update, the next batch's index and the loss added to *loss_sum.
int mlp_step_ws(Mlp *mp, const Batch &bt, cudaStream_t s, const Adam &adam = Adam{}, int64_t *step = nullptr,
                double *loss_sum = nullptr) {
    if (int rc = mlp_ensure(mp, bt.rows, true)) return rc;
    const float *P = mp->params.as<float>();
    const int h = mp->h, dout = mp->d_out, dp = mp->dp;
    const int rows = (int)bt.rows, rp = (int)((bt.rows + 127) / 128 * 128);  // padding rows are zero
    const int tiles = rp / kTile;
    float *col1 = mp->colws.as<float>(), *col2 = col1 + (int64_t)tiles * h, *col3 = col2 + (int64_t)tiles * h;
    int *st = mp->status.as<int>();
    // X's two copies; the targets' rows too where they are gathered (with the many blocks of this
    // launch, not behind two dependent loads in each block of the loss)
    ConvertJob job[2] = {
        convert_job(bt.X, mp->d_in, bt.perm, bt.batch_idx, bt.batch, rows, rp, dp, mp->xb.p, mp->xbt.p),
        convert_job(bt.T, dout, bt.perm, bt.batch_idx, bt.batch, rows, rp, dout, nullptr, nullptr)};
    job[1].F = mp->tb.as<float>();
    CUMF_CUDA(convert(job, bt.perm ? 2 : 1, s, step));
    auto ep = [&](DevBuf &out, DevBuf &out_t) {
        TrainEpilogue e{};
        e.out = out.as<__nv_bfloat16>();
        e.out_t = out_t.as<__nv_bfloat16>();
        e.valid = rows;
        return e;
    };
    TrainEpilogue e1 = ep(mp->h1, mp->h1t), e2 = ep(mp->h2, mp->h2t), e3 = ep(mp->dy, mp->dyt);
    TrainEpilogue g2 = ep(mp->dp2, mp->dp2t), g1 = ep(mp->dp1, mp->dp1t);
    e1.bias = P + mp->off_b1, e1.slope = mp->slope1.as<float>();
    e2.bias = P + mp->off_b2, e2.slope = mp->slope2.as<float>();
    e3.bias = P + mp->off_b3, e3.T = bt.perm ? mp->tb.as<float>() : bt.T;
    e3.scale = 1.f / (float)rows, e3.colsum = col3, e3.loss = mp->lossp.as<double>();
    g2.slope = e2.slope, g2.colsum = col2;
    g1.slope = e1.slope, g1.colsum = col1;
    // H1, H2, dY, then dZ2 = dY W3 * slope2, dZ1 = dZ2 W2 * slope1, then the weight gradients
    CUMF_CUDA(launch_train_gemm(kTrainForward, mp->xb.p, mp->w1b.p, rp, h, dp, e1, st, s));
    CUMF_CUDA(launch_train_gemm(kTrainForward, mp->h1.p, mp->w2b.p, rp, h, h, e2, st, s));
    CUMF_CUDA(launch_train_gemm(kTrainLoss, mp->h2.p, mp->w3b.p, rp, dout, h, e3, st, s));
    CUMF_CUDA(launch_train_gemm(kTrainBack, mp->dy.p, mp->w3t.p, rp, h, dout, g2, st, s));
    CUMF_CUDA(launch_train_gemm(kTrainBack, mp->dp2.p, mp->w2t.p, rp, h, h, g1, st, s));
    WgradJob jobs[kWgradJobs];
    wgrad_jobs(mp, rp, jobs);
    CUMF_CUDA(launch_wgrad(jobs, rp, st, s));

    FinishArgs f{};
    auto bf = [](DevBuf &b) { return b.as<__nv_bfloat16>(); };
    f.w[0] = {jobs[0].out, mp->off_w1, h, mp->d_in, dp, jobs[0].splits, bf(mp->w1b), nullptr};
    f.w[1] = {jobs[1].out, mp->off_w2, h, h, h, jobs[1].splits, bf(mp->w2b), bf(mp->w2t)};
    f.w[2] = {jobs[2].out, mp->off_w3, dout, h, h, jobs[2].splits, bf(mp->w3b), bf(mp->w3t)};
    f.bias[0] = {col1, mp->off_b1, h};
    f.bias[1] = {col2, mp->off_b2, h};
    f.bias[2] = {col3, mp->off_b3, dout};
    for (int l = 0; l < 3; ++l) {
        f.first[l + 1] = f.first[l] + f.w[l].rows / kTile * ((f.w[l].cols + kTile - 1) / kTile);
    }
    for (int l = 0; l < 3; ++l) f.first[l + 4] = f.first[l + 3] + f.bias[l].cols / kTile;
    f.tiles = tiles;
    f.grads = mp->grads.as<float>();
    f.adam = adam;
    f.loss_part = mp->lossp.as<double>();
    f.loss_parts = tiles * (dout / kTile);
    f.loss = mp->loss.as<double>();
    f.loss_sum = loss_sum;
    f.batch_idx = loss_sum ? bt.batch_idx : nullptr;
    finish_step_kernel<<<f.first[6] + 1, kTileBlock, 0, s>>>(f);
    CUMF_CUDA(cudaGetLastError());
    return CUMF_OK;
}

int mlp_check_status(Mlp *mp, cudaStream_t s) {
    int st = 0;
    CUMF_CUDA(cudaMemcpyAsync(&st, mp->status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    CUMF_CUDA(cudaStreamSynchronize(s));
    if (st) return fail(CUMF_ERR_TIMEOUT, "a tensor-core GEMM gave up waiting");
    return CUMF_OK;
}

}  // namespace

}  // namespace cumf

using namespace cumf;

extern "C" {

int cumf_mlp_create(int d_in, int hidden, int d_out, uint64_t seed, void **out) {
    if (!out || d_in <= 0 || hidden <= 0 || d_out <= 0 || hidden % 64 || d_out % 64)
        return fail(CUMF_ERR_ARG, "mlp_create: hidden and d_out must be positive multiples of 64");
    Mlp *mp = new Mlp();
    mp->d_in = d_in;
    mp->dp = (d_in + 63) / 64 * 64;
    mp->h = hidden;
    mp->d_out = d_out;
    int64_t o = 0;
    mp->off_w1 = o; o += (int64_t)hidden * d_in;
    mp->off_b1 = o; o += hidden;
    mp->off_w2 = o; o += (int64_t)hidden * hidden;
    mp->off_b2 = o; o += hidden;
    mp->off_w3 = o; o += (int64_t)d_out * hidden;
    mp->off_b3 = o; o += d_out;
    mp->count = o;
    auto cleanup = [&](int rc) { delete mp; return rc; };
    if (cudaError_t e = mp->params.alloc(o * 4)) return cleanup(cuda_fail(e, "mlp params"));
    if (cudaError_t e = mp->grads.alloc(o * 4)) return cleanup(cuda_fail(e, "mlp grads"));
    if (cudaError_t e = mp->m1.alloc(o * 4)) return cleanup(cuda_fail(e, "mlp adam"));
    if (cudaError_t e = mp->m2.alloc(o * 4)) return cleanup(cuda_fail(e, "mlp adam"));
    if (cudaError_t e = mp->w1b.alloc((size_t)hidden * mp->dp * 2)) return cleanup(cuda_fail(e, "mlp w1"));
    if (cudaError_t e = mp->w2b.alloc((size_t)hidden * hidden * 2)) return cleanup(cuda_fail(e, "mlp w2"));
    if (cudaError_t e = mp->w3b.alloc((size_t)d_out * hidden * 2)) return cleanup(cuda_fail(e, "mlp w3"));
    if (cudaError_t e = mp->w2t.alloc((size_t)hidden * hidden * 2)) return cleanup(cuda_fail(e, "mlp w2t"));
    if (cudaError_t e = mp->w3t.alloc((size_t)d_out * hidden * 2)) return cleanup(cuda_fail(e, "mlp w3t"));
    if (cudaError_t e = mp->status.alloc(sizeof(int))) return cleanup(cuda_fail(e, "mlp status"));
    if (cudaError_t e = mp->loss.alloc(sizeof(double))) return cleanup(cuda_fail(e, "mlp loss"));
    cudaMemset(mp->status.p, 0, sizeof(int));
    cudaMemset(mp->m1.p, 0, o * 4);
    cudaMemset(mp->m2.p, 0, o * 4);
    cudaMemset(mp->params.p, 0, o * 4);  // biases start at zero
    // Weights U(-a, a) with a = sqrt(6 / (fan_in + fan_out)) (Glorot uniform).
    float *P = mp->params.as<float>();
    const struct { int64_t off, n; int fi, fo; } layers[3] = {
        {mp->off_w1, (int64_t)hidden * d_in, d_in, hidden},
        {mp->off_w2, (int64_t)hidden * hidden, hidden, hidden},
        {mp->off_w3, (int64_t)d_out * hidden, hidden, d_out}};
    for (int l = 0; l < 3; ++l)
        init_weights_kernel<<<grid_of(layers[l].n), kT>>>(P + layers[l].off, layers[l].n,
                                                           sqrtf(6.f / (layers[l].fi + layers[l].fo)),
                                                           init_key(seed, 10 + l));
    if (int rc = mlp_refresh(mp, 0)) return cleanup(rc);
    if (cudaError_t e = cudaDeviceSynchronize()) return cleanup(cuda_fail(e, "mlp init"));
    *out = mp;
    return CUMF_OK;
}

int cumf_mlp_destroy(void *mlp) {
    delete static_cast<Mlp *>(mlp);
    return CUMF_OK;
}

int64_t cumf_mlp_param_count(void *mlp) { return mlp ? static_cast<Mlp *>(mlp)->count : 0; }

int cumf_mlp_get_params(void *mlp, float *host, int64_t count, int which) {
    Mlp *mp = static_cast<Mlp *>(mlp);
    if (!mp || !host || count != mp->count || which < 0 || which > 1) return fail(CUMF_ERR_ARG, "mlp_get_params");
    CUMF_CUDA(cudaMemcpy(host, which ? mp->grads.p : mp->params.p, count * 4, cudaMemcpyDeviceToHost));
    return CUMF_OK;
}

int cumf_mlp_set_params(void *mlp, const float *host, int64_t count) {
    Mlp *mp = static_cast<Mlp *>(mlp);
    if (!mp || !host || count != mp->count) return fail(CUMF_ERR_ARG, "mlp_set_params");
    CUMF_CUDA(cudaMemcpy(mp->params.p, host, count * 4, cudaMemcpyHostToDevice));
    if (int rc = mlp_refresh(mp, 0)) return rc;
    CUMF_CUDA(cudaDeviceSynchronize());
    return CUMF_OK;
}

int cumf_mlp_forward(void *mlp, const float *d_X, int64_t rows, float *d_Y, void *stream) {
    TraceRange trace("warm start: MLP inference");
    Mlp *mp = static_cast<Mlp *>(mlp);
    if (!mp || !d_X || !d_Y || rows < 0) return fail(CUMF_ERR_ARG, "mlp_forward: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t chunk = 1 << 16;
    for (int64_t r0 = 0; r0 < rows; r0 += chunk) {
        const int64_t r = std::min(chunk, rows - r0);
        if (int rc = mlp_forward_ws(mp, d_X + r0 * mp->d_in, r, d_Y + r0 * mp->d_out, s)) return rc;
    }
    return mlp_check_status(mp, s);
}

int cumf_mlp_loss_grad(void *mlp, const float *d_X, const float *d_T, int64_t rows, double *loss, void *stream) {
    Mlp *mp = static_cast<Mlp *>(mlp);
    if (!mp || !d_X || !d_T || rows <= 0) return fail(CUMF_ERR_ARG, "mlp_loss_grad: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (int rc = mlp_step_ws(mp, Batch{d_X, d_T, rows, nullptr, nullptr, 0}, s)) return rc;
    double l = 0;
    CUMF_CUDA(cudaMemcpyAsync(&l, mp->loss.p, sizeof(double), cudaMemcpyDeviceToHost, s));
    if (int rc = mlp_check_status(mp, s)) return rc;
    if (loss) *loss = l / (double)rows;
    return CUMF_OK;
}

int cumf_mlp_train(void *mlp, const float *d_X, const float *d_T, int64_t rows, int epochs, int batch, float lr,
                   uint64_t seed, double *final_loss, void *stream) {
    TraceRange trace("warm start: MLP training");
    Mlp *mp = static_cast<Mlp *>(mlp);
    if (!mp || !d_X || !d_T || rows <= 0 || epochs < 0 || batch <= 0)
        return fail(CUMF_ERR_ARG, "mlp_train: bad arguments");
    if (rows > 0x7fffffffll) return fail(CUMF_ERR_ARG, "mlp_train: more than 2^31 - 1 rows");
    if (final_loss) *final_loss = 0;
    if (epochs == 0) return CUMF_OK;
    if (batch > rows) batch = (int)rows;
    const int64_t full = rows / batch, tail = rows % batch;
    if (int rc = mlp_ensure(mp, batch, true)) return rc;  // the workspace, before any capture

    // Device state of the replayed step: Adam's step count and corrections, the batch index
    // into the epoch's permutation, the epoch's loss.
    struct State {
        int64_t step;
        int batch_idx;
        int pad;
        double loss_sum;
    };
    DevBuf perm_d, state;
    CUMF_CUDA(perm_d.alloc((size_t)rows * 4));
    CUMF_CUDA(state.alloc(sizeof(State)));
    State *st = state.as<State>();
    struct Host {
        void *p[2] = {nullptr, nullptr};
        ~Host() {
            for (void *x : p)
                if (x) cudaFreeHost(x);
        }
    } perm_h;
    for (int k = 0; k < 2; ++k) CUMF_CUDA(cudaMallocHost(&perm_h.p[k], (size_t)rows * 4));
    // A private stream (capture is not possible on the legacy default stream), ordered after
    // the caller's stream and before its later work.
    struct Res {
        cudaStream_t ws = nullptr;
        cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
        cudaGraphExec_t exec[2] = {nullptr, nullptr};
        ~Res() {
            for (cudaGraphExec_t x : exec)
                if (x) cudaGraphExecDestroy(x);
            for (cudaEvent_t x : ev)
                if (x) cudaEventDestroy(x);
            if (ws) cudaStreamDestroy(ws);
        }
    } res;
    CUMF_CUDA(cudaStreamCreateWithFlags(&res.ws, cudaStreamNonBlocking));
    for (cudaEvent_t &x : res.ev) CUMF_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
    cudaStream_t user = (cudaStream_t)stream, ws = res.ws;
    CUMF_CUDA(cudaEventRecord(res.ev[0], user));
    CUMF_CUDA(cudaStreamWaitEvent(ws, res.ev[0], 0));
    const State init = {mp->step, 0, 0, 0.0};
    CUMF_CUDA(cudaMemcpyAsync(st, &init, sizeof(State), cudaMemcpyHostToDevice, ws));
    CUMF_CUDA(cudaStreamSynchronize(ws));  // `init` is a host local

    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    // One training step of r rows at the batch the device index names.
    auto enqueue_step = [&](int64_t r) -> int {
        const Adam adam = {mp->params.as<float>(), mp->m1.as<float>(), mp->m2.as<float>(), lr, b1, b2, eps, &st->step};
        return mlp_step_ws(mp, Batch{d_X, d_T, r, perm_d.as<int32_t>(), &st->batch_idx, batch}, ws, adam, &st->step,
                           &st->loss_sum);
    };
    // Capture the full-batch step and the last, shorter one; replay them every epoch.
    auto capture = [&](int64_t r, cudaGraphExec_t *exec) -> int {
        CUMF_CUDA(cudaStreamBeginCapture(ws, cudaStreamCaptureModeRelaxed));
        const int rc = enqueue_step(r);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(ws, &g);
        if (rc != CUMF_OK || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return rc != CUMF_OK ? rc : cuda_fail(e, "mlp_train: capture");
        }
        const cudaError_t ei = cudaGraphInstantiate(exec, g, 0);
        cudaGraphDestroy(g);
        CUMF_CUDA(ei);
        return CUMF_OK;
    };
    if (full > 0)
        if (int rc = capture(batch, &res.exec[0])) return rc;
    if (tail > 0)
        if (int rc = capture(tail, &res.exec[1])) return rc;

    // Permutations from one glibc rand() stream, epoch by epoch; the next epoch's is drawn on
    // the host while the device runs the current one (two pinned buffers).
    GlibcRand rng((uint32_t)seed);
    auto draw = [&](int32_t *perm) {
        for (int64_t i = 0; i < rows; ++i) perm[i] = (int32_t)i;
        glibc_random_shuffle(perm, rows, rng);
    };
    draw(static_cast<int32_t *>(perm_h.p[0]));
    for (int e = 0; e < epochs; ++e) {
        const int k = e & 1;
        CUMF_CUDA(cudaMemsetAsync(&st->batch_idx, 0, sizeof(int), ws));
        CUMF_CUDA(cudaMemsetAsync(&st->loss_sum, 0, sizeof(double), ws));
        CUMF_CUDA(cudaMemcpyAsync(perm_d.p, perm_h.p[k], (size_t)rows * 4, cudaMemcpyHostToDevice, ws));
        CUMF_CUDA(cudaEventRecord(res.ev[1 + k], ws));  // perm_h[k] may be redrawn after this
        for (int64_t i = 0; i < full; ++i) CUMF_CUDA(cudaGraphLaunch(res.exec[0], ws));
        if (tail > 0) CUMF_CUDA(cudaGraphLaunch(res.exec[1], ws));
        if (e + 1 < epochs) {
            CUMF_CUDA(cudaEventSynchronize(res.ev[1 + (k ^ 1)]));
            draw(static_cast<int32_t *>(perm_h.p[k ^ 1]));
        }
    }
    mp->step += (int64_t)epochs * (full + (tail > 0 ? 1 : 0));
    double sum = 0;
    CUMF_CUDA(cudaMemcpyAsync(&sum, &st->loss_sum, sizeof(double), cudaMemcpyDeviceToHost, ws));
    if (int rc = mlp_check_status(mp, ws)) return rc;  // synchronizes ws
    CUMF_CUDA(cudaEventRecord(res.ev[3], ws));
    CUMF_CUDA(cudaStreamWaitEvent(user, res.ev[3], 0));
    if (final_loss) *final_loss = sum / (double)rows;
    return CUMF_OK;
}

int cumf_user_features(const cumf_node *d_R, int64_t nnz, const float *d_Q, int32_t n, int k, int32_t m,
                       float *d_X, void *stream) {
    TraceRange trace("warm start: user features");
    if (!d_Q || !d_X || m <= 0 || n <= 0 || k <= 0 || nnz < 0 || (nnz > 0 && !d_R))
        return fail(CUMF_ERR_ARG, "user_features: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (nnz < 0xffffffffll && m < 0x7fffffff) {
        // The ratings stably sorted by user (32-bit keys), then one warp per user.
        const uint32_t N = (uint32_t)nnz;
        int end_bit = 1;
        while (end_bit < 32 && ((uint32_t)m >> end_bit) != 0) ++end_bit;
        auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
        const size_t kb = up((size_t)N * 4 + 4), vb = up((size_t)N * 8 + 8), sb = up(((size_t)m + 1) * 8);
        cub::DoubleBuffer<uint32_t> key(nullptr, nullptr);
        cub::DoubleBuffer<float2> val(nullptr, nullptr);
        size_t tmp_bytes = 0;
        CUMF_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, key, val, N, 0, end_bit, s));
        void *buf = nullptr;
        CUMF_CUDA(scratch_alloc(&buf, 2 * kb + 2 * vb + sb + up(tmp_bytes), s));
        char *p = static_cast<char *>(buf);
        key.d_buffers[0] = reinterpret_cast<uint32_t *>(p);
        key.d_buffers[1] = reinterpret_cast<uint32_t *>(p + kb);
        val.d_buffers[0] = reinterpret_cast<float2 *>(p + 2 * kb);
        val.d_buffers[1] = reinterpret_cast<float2 *>(p + 2 * kb + vb);
        int64_t *seg = reinterpret_cast<int64_t *>(p + 2 * kb + 2 * vb);
        void *tmp = p + 2 * kb + 2 * vb + sb;
        cudaError_t e = cudaSuccess;
        if (N > 0) {
            user_keys_kernel<<<grid_of(N), kT, 0, s>>>(d_R, N, m, n, key.Current(), val.Current());
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, val, N, 0, end_bit, s);
        }
        if (e == cudaSuccess) {
            user_segments_kernel<<<grid_of((int64_t)m + 1), kT, 0, s>>>(key.Current(), N, m, seg);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            launch_user_rows(grid_of((int64_t)m * 32), val.Current(), seg, m, d_Q, k, d_X, s);
            e = cudaGetLastError();
        }
        const cudaError_t ef = cudaFreeAsync(buf, s);
        CUMF_CUDA(e);
        CUMF_CUDA(ef);
        CUMF_CUDA(cudaStreamSynchronize(s));
        return CUMF_OK;
    }
    // 2^32 ratings or more: vector atomics into per-user rows.  One stream-ordered scratch: the
    // centred mean accumulates in k-wide rows (16-byte aligned for the vector atomics), then
    // degree, rating sum and sum of squares per user.
    const size_t acc_bytes = (size_t)m * k * 4, scratch = acc_bytes + 3 * (size_t)m * 4;
    void *buf = nullptr;
    CUMF_CUDA(scratch_alloc(&buf, scratch, s));
    float *acc = static_cast<float *>(buf);
    float *deg = acc + (size_t)m * k, *sum = deg + m, *sum2 = sum + m;
    cudaError_t e = cudaMemsetAsync(buf, 0, scratch, s);
    if (e == cudaSuccess && nnz > 0) {
        user_stats_kernel<<<grid_of(nnz), kT, 0, s>>>(d_R, nnz, m, n, deg, sum, sum2);
        user_qsum_kernel<<<grid_of(nnz * 32), kT, 0, s>>>(d_R, nnz, m, n, d_Q, k, deg, sum, acc, k);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        user_finish_kernel<<<grid_of((int64_t)m * (k + 3)), kT, 0, s>>>(m, k, acc, deg, sum, sum2, d_X, k + 3);
        e = cudaGetLastError();
    }
    const cudaError_t ef = cudaFreeAsync(buf, s);
    CUMF_CUDA(e);
    CUMF_CUDA(ef);
    CUMF_CUDA(cudaStreamSynchronize(s));
    return CUMF_OK;
}

}  // extern "C"
