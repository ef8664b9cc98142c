// strata.cu - deterministic training: a stratified schedule of the same per-rating update.
//
// Batch-Hogwild (sgd_update.cu) lets thousands of workers update shared rows without locks,
// so results vary from run to run.  With `deterministic` set, the shuffled ratings are
// bucketed into a G x G grid of blocks (user group u mod G, item group v mod G) and an epoch
// runs the G strata in a seeded random order: stratum s holds the blocks (a, (a + s) mod G)
// for a = 0 .. G-1, which share no user and no item, so G workers update them in parallel
// without any row in common and the result is the same on every run and equal to the serial
// restatement.  Within a block every row sees its ratings in input order (a stable sort).  The per-rating arithmetic is the update of
// singleGPU/sgd_k128_kernel_hogwild_warp32.h:85-99 exactly as the batch-Hogwild kernel does it
// (lane-partial fused multiply-adds, group butterfly, storage rounding, stochastic rounding
// keyed by the rating's position in the stratified array).
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "cumf_sgd.h"
#include "device_common.cuh"
#include "internal.h"
#include "train_common.h"

namespace cumf {

namespace {

constexpr int kMaxChunk = 32;  // ratings of a block whose rows are in shared memory together

__global__ void block_key_kernel(const cumf_node *__restrict__ R, int64_t nnz, int G, uint32_t *keys,
                                 int64_t *idx, unsigned long long *counts) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const cumf_node x = R[i];
        const uint32_t key = ((uint32_t)x.u % (uint32_t)G) * (uint32_t)G + (uint32_t)x.v % (uint32_t)G;
        keys[i] = key;
        idx[i] = i;
        atomicAdd(&counts[key], 1ull);
    }
}

__global__ void gather_records_kernel(const cumf_node *__restrict__ R, const int64_t *__restrict__ idx, int64_t nnz,
                                      cumf_node *out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = R[idx[i]];
}

// x without its r lowest set bits, r <= N.
template <int N>
__device__ __forceinline__ uint32_t drop_lowest(uint32_t x, int r) {
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (r > i) x &= x - 1;
    return x;
}

// One warp per block of the stratum; the block's ratings `chunk` at a time.
//
// A stratum takes as long as its longest block, so what counts is one block's time per rating.
// Rows fetched rating by rating were a chain of L2 latencies: a block's ratings share most of
// their rows, so that a fetch ahead has to be checked against every update since.  Here the
// distinct rows of a chunk come to shared memory together, are updated there and written back
// before the next chunk; a stratum's blocks share no row, so nobody else reads them meanwhile.
// Ratings without a row in common commute, so each step takes the first 32 / L ratings that wait
// for no earlier one, L lanes each: every row still sees its ratings in order.
// One block of threads per worker, so that they spread over all SMs.
//
// Bound by the chain of a popular item's updates: about 190 ns each (shared memory, dot product,
// butterfly, update; 450 before), 130 ns per rating where half of them pair up.  Per stratum,
// 10,000 x 2,000, 0.9M ratings, k = 128, fp16 (longest block 80 ratings): 34 us with the rows
// loaded one rating ahead, 12.9 so, 10.2 with the next stratum's start overlapped.  Per epoch,
// 480,189 x 17,770, 99M ratings: fp16 153 -> 65 ms, fp32 (one rating at a time) 130 -> 89.
template <int K, int KIND, int L, bool SR>
__global__ void __launch_bounds__(32) stratum_kernel(const cumf_node *__restrict__ R,
                                                     const unsigned long long *__restrict__ block_off, int G,
                                                     int stratum, int chunk, void *Pv, void *Qv, uint32_t m,
                                                     uint32_t n, float lr, float lp, float lq, uint32_t round_key,
                                                     int *status) {
    constexpr int ROW_WORDS = K * store_bytes(KIND) / 16;
    constexpr int NV = ROW_WORDS / L;
    static_assert(NV >= 1 && NV * L == ROW_WORDS, "lane split must cover the row");
    constexpr int W = 32 / L;                                     // ratings per step
    constexpr int TW = ROW_WORDS < 32 ? ROW_WORDS : 32;           // lanes that copy a row
    constexpr int T = 32 / TW, E = ROW_WORDS / TW;                // rows per instruction, words per lane and row
    constexpr int B = 8;                                          // instructions in flight per matrix
    constexpr uint32_t kAll = 0xffffffffu, kNoRow = 0xffffffffu;  // no rating's row (m, n < 2^31)
    extern __shared__ uint4 rows[];                               // chunk user rows, then chunk item rows
    uint4 *const items = rows + chunk * ROW_WORDS;
    const int lane = threadIdx.x, a = blockIdx.x;
    const int blk = a * G + (a + stratum) % G;
    const uint64_t pol = l2_policy(true, true);
    const unsigned long long i0 = block_off[blk], i1 = block_off[blk + 1];
    cumf_node next = {-1, -1, 0.f};
    if (lane < chunk && i0 + lane < i1) next = R[i0 + lane];
    // Up to here the kernel may run beside the stratum before it (programmatic dependent launch: R
    // and block_off are inputs, unchanged by either); the rows are read once that one is complete.
    // Every block waits, with ratings or without, so that the strata complete in their order; and
    // the next stratum's blocks come only now, so that at most two kernels share the GPU.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    bool bad = false;
    for (unsigned long long base = i0; base < i1; base += chunk) {
        const int cnt = (int)(i1 - base < (unsigned long long)chunk ? i1 - base : (unsigned long long)chunk);
        const cumf_node x = next;
        next = {-1, -1, 0.f};
        if (lane < chunk && base + chunk + lane < i1) next = R[base + chunk + lane];
        const bool ok = lane < cnt && ((uint32_t)x.u < m) & ((uint32_t)x.v < n);
        bad |= lane < cnt && !ok;
        // Lane t has rating t.  A row's place is that of the first rating of the chunk that has it.
        const uint32_t u = ok ? (uint32_t)x.u : kNoRow, v = ok ? (uint32_t)x.v : kNoRow;
        const uint32_t same_u = __match_any_sync(kAll, u), same_v = __match_any_sync(kAll, v);
        const int place_u = ok ? __ffs(same_u) - 1 : 0, place_v = ok ? __ffs(same_v) - 1 : 0;
        const uint32_t first_u = __ballot_sync(kAll, ok && place_u == lane);
        const uint32_t first_v = __ballot_sync(kAll, ok && place_v == lane);
        const uint32_t before = (same_u | same_v) & ((1u << lane) - 1u);  // the ratings that this one waits for
        // Each row that is the first of its kind, between its place and global memory.
        const int sub = lane / TW, word = lane % TW;
        auto row_of = [&](int t, const uint32_t rows_of, uint32_t first, void *F, uint4 *&at) {
            const uint32_t row = __shfl_sync(kAll, rows_of, t & 31);
            at = reinterpret_cast<uint4 *>(F) + (uint64_t)row * ROW_WORDS + word;
            return t < cnt && (first >> (t & 31) & 1u);
        };
#pragma unroll 1
        for (int e = 0; e < E; ++e)
#pragma unroll 1
            for (int t0 = 0; t0 < cnt; t0 += T * B) {
                uint4 p[B], q[B];
                bool hp[B], hq[B];
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    uint4 *ap, *aq;
                    hp[b] = row_of(t0 + b * T + sub, u, first_u, Pv, ap);
                    hq[b] = row_of(t0 + b * T + sub, v, first_v, Qv, aq);
                    if (hp[b]) p[b] = ld_row_hint(ap + e * TW, pol);
                    if (hq[b]) q[b] = ld_row_hint(aq + e * TW, pol);
                }
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const int at = (t0 + b * T + sub) * ROW_WORDS + e * TW + word;
                    if (hp[b]) rows[at] = p[b];
                    if (hq[b]) items[at] = q[b];
                }
            }
        __syncwarp();

        const int g = lane / L;
        uint4 *const my_rows = rows + (lane % L) * NV, *const my_items = items + (lane % L) * NV;
        uint32_t pending = __ballot_sync(kAll, ok);
        // The step's rating of this group of lanes, or none (-1): whether there is any.
        auto pick = [&](int &mine) {
            const uint32_t ready = __ballot_sync(kAll, (pending >> lane & 1u) && (before & pending) == 0);
            mine = __ffs(drop_lowest<W - 1>(ready, g)) - 1;
            pending &= drop_lowest<W>(ready, W) | ~ready;
            return ready != 0;
        };
        int mine;
        bool more = pick(mine);
        int at_u = __shfl_sync(kAll, place_u, mine & 31) * ROW_WORDS;
        int at_v = __shfl_sync(kAll, place_v, mine & 31) * ROW_WORDS;
        float r = __shfl_sync(kAll, x.r, mine & 31);
        while (more) {
            uint4 p[NV], q[NV], wp[NV], wq[NV];
#pragma unroll
            for (int w = 0; w < NV; ++w) p[w] = my_rows[at_u + w], q[w] = my_items[at_v + w];
            // the next step's, while this one is computed
            int mine2;
            more = pick(mine2);
            const int at_u2 = __shfl_sync(kAll, place_u, mine2 & 31) * ROW_WORDS;
            const int at_v2 = __shfl_sync(kAll, place_v, mine2 & 31) * ROW_WORDS;
            const float r2 = __shfl_sync(kAll, x.r, mine2 & 31);
            float sdot = 0.f;
#pragma unroll
            for (int w = 0; w < NV; ++w) sdot = dot_word<KIND>(p[w], q[w], sdot);
#pragma unroll
            for (int o = L / 2; o >= 1; o >>= 1) sdot += __shfl_xor_sync(kAll, sdot, o);
            const uint32_t key = SR ? (round_key ^ lowbias32((uint32_t)(base + (mine & 31)))) : 0u;
#pragma unroll
            for (int w = 0; w < NV; ++w)
                update_word<KIND, SR>(p[w], q[w], wp[w], wq[w], lr, r - sdot, -lp, -lq, key, (lane % L) * NV + w);
            if (mine >= 0) {
#pragma unroll
                for (int w = 0; w < NV; ++w) my_rows[at_u + w] = wp[w], my_items[at_v + w] = wq[w];
            }
            __syncwarp();
            mine = mine2, at_u = at_u2, at_v = at_v2, r = r2;
        }
#pragma unroll 1
        for (int e = 0; e < E; ++e)
#pragma unroll 4
            for (int t0 = 0; t0 < cnt; t0 += T) {
                uint4 *ap, *aq;
                const int t = t0 + sub, at = t * ROW_WORDS + e * TW + word;
                const bool hp = row_of(t, u, first_u, Pv, ap), hq = row_of(t, v, first_v, Qv, aq);
                if (hp) st_row_hint(ap + e * TW, rows[at], pol);
                if (hq) st_row_hint(aq + e * TW, items[at], pol);
            }
        __syncwarp();  // the next chunk reads what any lane stored
    }
    if (bad && status != nullptr) atomicExch(status, (int)CUMF_ERR_RANGE);
}

using StratumFn = void (*)(const cumf_node *, const unsigned long long *, int, int, int, void *, void *, uint32_t,
                           uint32_t, float, float, float, uint32_t, int *);

// One 16-byte word per lane (the update kernel's default layout).
template <int K>
StratumFn pick(int precision) {
    switch (precision) {
        case CUMF_FP16: return &stratum_kernel<K, kHalf, K * 2 / 16, false>;
        case CUMF_FP16_SR: return &stratum_kernel<K, kHalf, K * 2 / 16, true>;
        case CUMF_BF16: return &stratum_kernel<K, kBf16, K * 2 / 16, false>;
        case CUMF_BF16_SR: return &stratum_kernel<K, kBf16, K * 2 / 16, true>;
        default: return &stratum_kernel<K, kFloat, (K * 4 / 16 > 32 ? 32 : K * 4 / 16), false>;
    }
}

}  // namespace

// The strata of epoch ep in a seeded random order: Fisher-Yates over 0 .. G-1 drawing
// splitmix64(seed ^ tag, epoch, step) mod (step + 1).
void strata_order(uint64_t seed, int ep, int G, int *order) {
    for (int i = 0; i < G; ++i) order[i] = i;
    uint64_t h = splitmix64(seed ^ (0x5354ull << 48)) + (uint64_t)ep * 0x9E3779B97F4A7C15ull;
    for (int i = G - 1; i > 0; --i) {
        h = splitmix64(h);
        const int j = (int)(h % (uint64_t)(i + 1));
        const int t = order[i];
        order[i] = order[j];
        order[j] = t;
    }
}

int strata_groups(int64_t nnz, int requested) {
    if (requested > 1) return requested;
    // About 24 ratings per block: G^2 blocks, G workers per stratum.
    const double g = sqrt((double)std::max<int64_t>(1, nnz) / 24.0);
    return (int)std::max(1.0, std::min(2048.0, std::floor(g)));
}

int strata_layout(const cumf_node *d_R, int64_t nnz, int G, cumf_node *d_out, unsigned long long *d_block_off,
                  cudaStream_t s) {
    if (G < 1 || (int64_t)G * G > (1ll << 26)) return fail(CUMF_ERR_ARG, "strata: group count out of range");
    const int64_t blocks = (int64_t)G * G;
    DevBuf keys, keys2, idx, idx2, counts, tmp;
    const size_t n = (size_t)std::max<int64_t>(1, nnz);
    CUMF_CUDA(keys.alloc(n * 4, s));
    CUMF_CUDA(keys2.alloc(n * 4, s));
    CUMF_CUDA(idx.alloc(n * 8, s));
    CUMF_CUDA(idx2.alloc(n * 8, s));
    CUMF_CUDA(counts.alloc((size_t)(blocks + 1) * 8, s));
    unsigned long long *cnt = static_cast<unsigned long long *>(counts.p);
    CUMF_CUDA(cudaMemsetAsync(cnt, 0, (size_t)(blocks + 1) * 8, s));
    const int grid = (int)std::min<int64_t>(65535, (nnz + 255) / 256 + 1);
    block_key_kernel<<<grid, 256, 0, s>>>(d_R, nnz, G, static_cast<uint32_t *>(keys.p),
                                          static_cast<int64_t *>(idx.p), cnt);
    CUMF_CUDA(cudaGetLastError());
    // Stable sort by block (keeps the input order inside a block), then block offsets.
    int end_bit = 1;
    while (end_bit < 32 && ((uint64_t)1 << end_bit) < (uint64_t)blocks) ++end_bit;
    size_t tb = 0;
    CUMF_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, static_cast<uint32_t *>(keys.p),
                                              static_cast<uint32_t *>(keys2.p), static_cast<int64_t *>(idx.p),
                                              static_cast<int64_t *>(idx2.p), nnz, 0, end_bit, s));
    size_t tb2 = 0;
    CUMF_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb2, cnt, d_block_off, blocks + 1, s));
    CUMF_CUDA(tmp.alloc(std::max(tb, tb2) + 16, s));
    CUMF_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, static_cast<uint32_t *>(keys.p),
                                              static_cast<uint32_t *>(keys2.p), static_cast<int64_t *>(idx.p),
                                              static_cast<int64_t *>(idx2.p), nnz, 0, end_bit, s));
    CUMF_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb2, cnt, d_block_off, blocks + 1, s));
    gather_records_kernel<<<grid, 256, 0, s>>>(d_R, static_cast<const int64_t *>(idx2.p), nnz, d_out);
    CUMF_CUDA(cudaGetLastError());
    CUMF_CUDA(cudaStreamSynchronize(s));
    return CUMF_OK;
}

int strata_epochs(const cumf_node *d_S, const unsigned long long *d_block_off, int G, void *d_P, int32_t m,
                  void *d_Q, int32_t n, int k, int precision, const float *h_lr, int first_epoch, int n_epochs,
                  float lambda_p, float lambda_q, uint64_t seed, int *d_status, cudaStream_t s) {
    StratumFn fn = nullptr;
    switch (k) {
        case 32: fn = pick<32>(precision); break;
        case 64: fn = pick<64>(precision); break;
        case 128: fn = pick<128>(precision); break;
        case 256: fn = pick<256>(precision); break;
        default: return fail(CUMF_ERR_ARG, "strata: k must be 32, 64, 128 or 256");
    }
    // 32 ratings where all G workers are resident with them (at most 32 workers per SM), else 16:
    // the blocks are of unequal length, so that those that start late end with the long ones.
    // 480,189 x 17,770, 99M ratings, G = 2031, k = 128, fp32: 89 ms per epoch with 16, 93 with 8.
    const int row = k * (precision == CUMF_FP32 ? 4 : 2);
    auto bytes = [&](int c) { return (size_t)c * 2 * row; };
    int dev = 0, sms = 0, per_sm = 0;
    CUMF_CUDA(cudaGetDevice(&dev));
    CUMF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CUMF_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    int chunk = kMaxChunk;
    if (std::min<int64_t>(32, per_sm / (int64_t)(bytes(chunk) + 1024)) * sms < G) chunk /= 2;
    CUMF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(kMaxChunk)));
    // Each stratum's blocks start while the one before still runs.
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(32);
    cfg.dynamicSmemBytes = bytes(chunk);
    cfg.stream = s;
    cfg.attrs = &overlap;
    std::vector<int> order(G);
    for (int ep = first_epoch; ep < first_epoch + n_epochs; ++ep) {
        const uint32_t round_key = (uint32_t)(splitmix64(seed ^ (kTagRound << 48)) + (uint64_t)ep);
        strata_order(seed, ep, G, order.data());
        for (int j = 0; j < G; ++j) {
            // The first one is ordered after all that the caller has put on the stream.
            cfg.numAttrs = ep == first_epoch && j == 0 ? 0 : 1;
            CUMF_CUDA(cudaLaunchKernelEx(&cfg, fn, d_S, d_block_off, G, order[j], chunk, d_P, d_Q, (uint32_t)m,
                                         (uint32_t)n, h_lr[ep], lambda_p, lambda_q, round_key, d_status));
        }
    }
    return CUMF_OK;
}

}  // namespace cumf

using namespace cumf;

extern "C" int cumf_dev_strata_layout(const cumf_node *d_R, int64_t nnz, int groups, cumf_node *d_out,
                                      unsigned long long *d_block_off, void *stream) {
    if (nnz < 0 || (nnz > 0 && (!d_R || !d_out)) || !d_block_off) return fail(CUMF_ERR_ARG, "strata_layout: bad arguments");
    return strata_layout(d_R, nnz, groups, d_out, d_block_off, static_cast<cudaStream_t>(stream));
}

extern "C" int cumf_dev_strata_epochs(const cumf_node *d_S, const unsigned long long *d_block_off, int groups,
                                      void *d_P, int32_t m, void *d_Q, int32_t n, int k, int precision,
                                      const float *h_lr, int first_epoch, int n_epochs, float lambda_p,
                                      float lambda_q, uint64_t seed, int *d_status, void *stream) {
    if (groups < 1 || !d_block_off || !d_P || !d_Q || !h_lr || first_epoch < 0 || n_epochs < 0 || m < 1 || n < 1)
        return fail(CUMF_ERR_ARG, "strata_epochs: bad arguments");
    if (precision < CUMF_FP16 || precision > CUMF_FP16_SR) return fail(CUMF_ERR_ARG, "unknown precision");
    return strata_epochs(d_S, d_block_off, groups, d_P, m, d_Q, n, k, precision, h_lr, first_epoch, n_epochs,
                         lambda_p, lambda_q, seed, d_status, static_cast<cudaStream_t>(stream));
}
