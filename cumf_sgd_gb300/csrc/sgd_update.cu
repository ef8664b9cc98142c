// sgd_update.cu - the batch-Hogwild SGD update kernel.
//
// Semantics follow sgd_k128_kernel_hogwild_warp32_lrate
// (singleGPU/sgd_k128_kernel_hogwild_warp32.h:3-104) launched by sgd_update_k128
// (singleGPU/sgd_kernel.cu:198-248):
//   - W workers; each does ceil(nnz/(W*128)) batches per epoch (sgd_kernel.cu:203);
//   - a batch is 128 consecutive records (start+i) % nnz from a uniform start (warp32.h:42-52);
//   - per record: e = r - <p_u, q_v>;  p <- p + lr (e q - lp p);  q <- q + lr (e p_old - lq q)
//     in fp32, stored back rounded to the storage type (warp32.h:85-99);
//   - lr = table[epoch] (warp32.h:32); no locks or atomics (Hogwild).
//
// GB300 layout: a worker is a group of G lanes (G = 4..32, a power of two) rather than a
// whole warp.  Each lane owns E = k/G consecutive elements of a row and moves them with
// 16-byte ld.global.cg / st.global.cg, so a k=128 fp16 row (256 B) is one vector per lane
// of a 16-lane group and two workers share a warp.  The dot product is a butterfly of
// shfl.xor within the group (every lane ends with the same bits).  Two kernels:
//   sgd_hogwild_kernel  one record at a time, the next one's rows in flight;
//   sgd_pair_kernel     two records at a time, where a lane holds one 16-byte word of a row (every
//                       default width but fp32 k = 256) and no row is much contended.
// Either way a worker applies its records strictly in order: a row that an earlier record has
// just written is forwarded to a record whose loads were issued before the store.  Records
// are staged 32 (narrow groups: 16) at a time through shared memory (4-byte cp.async copies of
// the 12-byte records).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "device_common.cuh"
#include "internal.h"

namespace cumf {

namespace {

constexpr int kBlock = 256;   // threads per block
constexpr int kMinBlocks = 4; // >= 1024 resident threads per SM (<= 64 registers)
// Threads per block and blocks per SM of sgd_pair_kernel: 1024 threads per SM (64 registers), or
// 640 (96 registers) in smaller blocks with stochastic rounding.
constexpr int pair_block(bool sr) { return sr ? 64 : 128; }
constexpr int pair_min_blocks(bool sr) { return sr ? 10 : 8; }
// Threads per SM that a wave of workers stands for (cumf_default_workers): part of the sample
// schedule through the automatic worker count, so it stays whatever a kernel's occupancy is.
constexpr int kWaveThreads = 1024;
constexpr int kDefaultPrefetch = 2;
constexpr int kDefaultHints = 1;
constexpr int kDefaultRing = 0;
constexpr int kBatch = 128;   // records per batch (update_vector_size, sgd_kernel.cu:198)
// Records staged in shared memory at a time: 32, or 16 for narrow groups (keeps the
// staging buffer of a 256-thread block under 27 KB).
__host__ __device__ constexpr int chunk_of(int lanes) { return lanes >= 8 ? 32 : 16; }

struct UpdateArgs {
    const cumf_node *R;
    uint64_t nnz;
    void *P;
    void *Q;
    uint32_t m, n;
    const float *lr;
    int first_epoch, n_epochs;
    int num_workers;
    int batches;
    float lambda_p, lambda_q;
    uint64_t seed;
    int *status;
    int prefetch;   // rows of record j+prefetch are pulled into L2 while record j runs (0 = off)
    int hints;      // 1 = L2 eviction hints (ratings evict_first, factor rows evict_last)
    int freeze_q;   // 1 = item rows are read but never written (user-side fold-in)
    const uint2 *contended;  // users' and items' flags of sample_rows_kernel, or NULL: run
    int run_contended;       // run if either flag is set (1) or if neither is (0)
};

// Of the two launches that follow sample_rows_kernel, the other one runs.
__device__ __forceinline__ bool skip_launch(const UpdateArgs &a) {
    if (a.contended == nullptr) return false;
    const uint2 f = __ldg(a.contended);
    return ((f.x | f.y) != 0) != (a.run_contended != 0);
}

// Copy of a word the compiler cannot see through: the update phase re-widens the packed
// rows instead of keeping the dot phase's fp32 copies alive across the group reduction.
__device__ __forceinline__ uint4 opaque(uint4 w) {
    asm volatile("" : "+r"(w.x), "+r"(w.y), "+r"(w.z), "+r"(w.w));
    return w;
}

// The new rows of one record: p + lr*(e*q - lp*p) and q + lr*(e*p_old - lq*q)
// (warp32.h:89-99), in fp32, stored rounded to the storage type (stochastically when SR; the
// random bits of element pair h of word i of this lane are lowbias32(key + 2*pair) for p and
// lowbias32(key + 2*pair + 1) for q).  kUpdateQ = false (item rows frozen): wq is fq and none
// of q's arithmetic or random bits is computed.
template <class C, int NV, bool SR, bool kUpdateQ>
__device__ __forceinline__ void update_rows(const uint4 (&fp)[NV], const uint4 (&fq)[NV], uint4 (&wp)[NV],
                                            uint4 (&wq)[NV], float lr, float err, float lp, float lq, uint32_t key,
                                            int lane) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint4 fpi = opaque(fp[i]), fqi = opaque(fq[i]);
#pragma unroll
        for (int h = 0; h < C::kPairs; ++h) {
            const float2 pp = C::get(fpi, h), qq = C::get(fqi, h);
            const float px = __fmaf_rn(lr, __fmaf_rn(err, qq.x, -__fmul_rn(lp, pp.x)), pp.x);
            const float py = __fmaf_rn(lr, __fmaf_rn(err, qq.y, -__fmul_rn(lp, pp.y)), pp.y);
            if (kUpdateQ) {
                const float qx = __fmaf_rn(lr, __fmaf_rn(err, pp.x, -__fmul_rn(lq, qq.x)), qq.x);
                const float qy = __fmaf_rn(lr, __fmaf_rn(err, pp.y, -__fmul_rn(lq, qq.y)), qq.y);
                if (SR) {
                    const uint32_t pair = (uint32_t)(((lane * NV + i) * C::kPairs + h) * 2);
                    C::put_sr(wp[i], h, px, py, lowbias32(key + pair));
                    C::put_sr(wq[i], h, qx, qy, lowbias32(key + pair + 1u));
                } else {
                    C::put(wp[i], h, px, py);
                    C::put(wq[i], h, qx, qy);
                }
            } else if (SR) {
                const uint32_t pair = (uint32_t)(((lane * NV + i) * C::kPairs + h) * 2);
                C::put_sr(wp[i], h, px, py, lowbias32(key + pair));
            } else {
                C::put(wp[i], h, px, py);
            }
        }
        if (!kUpdateQ) wq[i] = fq[i];
    }
}

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem, uint64_t pol) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 4, %2;\n" ::"r"(sa), "l"(gmem), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int K, int KIND, int G, bool SR>
__global__ void __launch_bounds__(kBlock, kMinBlocks)
sgd_hogwild_kernel(const UpdateArgs a) {
    if (skip_launch(a)) return;
    using C = Conv<KIND>;
    constexpr int SB = store_bytes(KIND);
    constexpr int ROW_WORDS = K * SB / 16;          // uint4 words per row
    constexpr int NV = ROW_WORDS / G;               // uint4 words per lane
    constexpr int GPB = kBlock / G;                 // groups (workers) per block
    constexpr int kChunk = chunk_of(G);
    constexpr int CPB = kBatch / kChunk;            // chunks per batch
    constexpr int WPL = kChunk * 3 / G;             // staged record words per lane
    static_assert(NV >= 1 && NV * G == ROW_WORDS, "lane split must cover the row");
    static_assert((kChunk * 3) % G == 0 && kBatch % kChunk == 0, "chunk must split evenly");

    // [group][buffer][field][record], padded so groups of one warp hit different banks.
    __shared__ uint32_t s_rec[GPB][2][3][kChunk + 1];

    const int lane = threadIdx.x % G;
    const int gib = threadIdx.x / G;
    const int worker = blockIdx.x * GPB + gib;
    if (worker >= a.num_workers) return;
    const unsigned gmask =
        (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));

    uint4 *const P = reinterpret_cast<uint4 *>(a.P) + lane * NV;
    uint4 *const Q = reinterpret_cast<uint4 *>(a.Q) + lane * NV;
    const uint32_t *const Rw = reinterpret_cast<const uint32_t *>(a.R);
    const uint64_t nnz = a.nnz;
    const float lp = a.lambda_p, lq = a.lambda_q;
    const int chunks = a.batches * CPB;
    const int pd = a.prefetch;
    const uint64_t pol_rec = l2_policy(a.hints != 0, false);
    const uint64_t pol_row = l2_policy(a.hints != 0, true);
    // Lanes whose 16-byte slice starts a 128-byte line issue the L2 prefetches.
    const bool pf_lane = ((lane * NV * 16) & 127) == 0;
    int bad = 0;

    for (int ep = a.first_epoch; ep < a.first_epoch + a.n_epochs; ++ep) {
        const float lr = __ldg(a.lr + ep);
        const uint32_t round_key = (uint32_t)(splitmix64(a.seed ^ (kTagRound << 48)) + (uint64_t)ep);

        // Asynchronous copy of the records of chunk t into buffer buf.
        auto fetch = [&](int t, int buf) {
            const uint64_t start = batch_start(a.seed, ep, worker, t / CPB, nnz);
            uint64_t base = start + (uint64_t)((t % CPB) * kChunk);
            while (base >= nnz) base -= nnz;  // start < nnz: wraps only when nnz < 128
#pragma unroll
            for (int i = 0; i < WPL; ++i) {
                const int word = lane + i * G;
                uint64_t rec = base + (uint64_t)(word / 3);
                while (rec >= nnz) rec -= nnz;
                cp_async4(&s_rec[gib][buf][word % 3][word / 3], Rw + rec * 3 + (word % 3), pol_rec);
            }
            cp_async_commit();
        };

        fetch(0, 0);
        cp_async_wait_all();
        __syncwarp(gmask);

        // Prologue: rows of the first record.
        uint32_t u = s_rec[gib][0][0][0], v = s_rec[gib][0][1][0];
        bool ok = (u < a.m) & (v < a.n);
        uint4 fp[NV], fq[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            fp[i] = ok ? ld_row_hint(P + (uint64_t)u * ROW_WORDS + i, pol_row) : make_uint4(0, 0, 0, 0);
            fq[i] = ok ? ld_row_hint(Q + (uint64_t)v * ROW_WORDS + i, pol_row) : make_uint4(0, 0, 0, 0);
        }

        for (int t = 0; t < chunks; ++t) {
            const int buf = t & 1;
            const bool has_next_chunk = (t + 1 < chunks);
            if (has_next_chunk) fetch(t + 1, buf ^ 1);

#pragma unroll 1
            for (int j = 0; j < kChunk; ++j) {
                // L2 prefetch of the rows of record j + pd (same or next chunk).
                if (pd > 0) {
                    const int jj = j + pd;
                    uint32_t pu = 0xffffffffu, pv = 0xffffffffu;
                    if (jj < kChunk) {
                        pu = s_rec[gib][buf][0][jj];
                        pv = s_rec[gib][buf][1][jj];
                    } else if (has_next_chunk && jj - kChunk < kChunk) {
                        if (jj == kChunk) {  // first look into the next chunk: wait for its copy
                            cp_async_wait_all();
                            __syncwarp(gmask);
                        }
                        pu = s_rec[gib][buf ^ 1][0][jj - kChunk];
                        pv = s_rec[gib][buf ^ 1][1][jj - kChunk];
                    }
                    if (pf_lane && pu < a.m && pv < a.n) {
                        prefetch_l2(P + (uint64_t)pu * ROW_WORDS);
                        prefetch_l2(Q + (uint64_t)pv * ROW_WORDS);
                    }
                }
                // Next record: same chunk, or the first record of the next chunk.
                uint32_t un = 0xffffffffu, vn = 0xffffffffu;
                if (j + 1 < kChunk) {
                    un = s_rec[gib][buf][0][j + 1];
                    vn = s_rec[gib][buf][1][j + 1];
                } else if (has_next_chunk) {
                    cp_async_wait_all();
                    __syncwarp(gmask);
                    un = s_rec[gib][buf ^ 1][0][0];
                    vn = s_rec[gib][buf ^ 1][1][0];
                }
                const bool okn = (un < a.m) & (vn < a.n);
                uint4 np[NV], nq[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    np[i] = okn ? ld_row_hint(P + (uint64_t)un * ROW_WORDS + i, pol_row) : make_uint4(0, 0, 0, 0);
                    nq[i] = okn ? ld_row_hint(Q + (uint64_t)vn * ROW_WORDS + i, pol_row) : make_uint4(0, 0, 0, 0);
                }

                if (ok) {
                    const float r = __uint_as_float(s_rec[gib][buf][2][j]);
                    // Lane partial dot in element order, then the group butterfly.
                    float s = 0.f;
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
#pragma unroll
                        for (int h = 0; h < C::kPairs; ++h) {
                            const float2 pp = C::get(fp[i], h), qq = C::get(fq[i], h);
                            s = __fmaf_rn(pp.x, qq.x, s);
                            s = __fmaf_rn(pp.y, qq.y, s);
                        }
                    }
#pragma unroll
                    for (int o = G / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(gmask, s, o);
                    const float err = r - s;
                    uint32_t key = 0;
                    if (SR) {
                        const uint32_t sample = (uint32_t)worker * (uint32_t)(chunks * kChunk) +
                                                (uint32_t)(t * kChunk + j);
                        key = round_key ^ lowbias32(sample);
                    }
                    uint4 wp[NV], wq[NV];
                    // Frozen item rows: the stochastic-rounding kernels skip q's arithmetic and
                    // random bits; the others compute q and keep the old row (fewer registers).
                    if (SR && a.freeze_q) {
                        update_rows<C, NV, SR, false>(fp, fq, wp, wq, lr, err, lp, lq, key, lane);
                    } else {
                        update_rows<C, NV, SR, true>(fp, fq, wp, wq, lr, err, lp, lq, key, lane);
                        if (a.freeze_q) {
#pragma unroll
                            for (int i = 0; i < NV; ++i) wq[i] = fq[i];
                        }
                    }
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        st_row_hint(P + (uint64_t)u * ROW_WORDS + i, wp[i], pol_row);
                        if (!a.freeze_q) st_row_hint(Q + (uint64_t)v * ROW_WORDS + i, wq[i], pol_row);
                    }
                    // Forward the fresh rows when the next record reuses them (its loads
                    // were issued before these stores).
                    if (un == u) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) np[i] = wp[i];
                    }
                    if (vn == v) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) nq[i] = wq[i];
                    }
                } else {
                    bad = 1;
                }
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    fp[i] = np[i];
                    fq[i] = nq[i];
                }
                u = un;
                v = vn;
                ok = okn;
            }
            __syncwarp(gmask);  // buffer `buf` is refilled by the next iteration's fetch
        }
    }
    if (bad && a.status != nullptr && lane == 0) atomicExch(a.status, (int)CUMF_ERR_RANGE);
}


// ---- two records at a time ----------------------------------------------------------------
//
// What bounds an epoch depends on the worker count.  With a few workers (small matrices, fold-in
// epochs) it is the chain of one record: load, dot, butterfly, update.  Records j and j+1 that
// share no row are independent, so both chains run interleaved here; a pair that shares a row
// takes the serial branch, with the same bits either way.  The rows are loaded at the start of
// their own pair, not a pair ahead: a worker then has two records between load and store, as
// many as with one record at a time and the next one's rows in flight.  Loading a pair ahead
// (four records) is faster still (3,000 x 1,200: 0.25 ms) but loses twice the updates on popular
// rows: 10,000 x 2,000, 0.9M ratings, Zipf 1.0, 20 epochs, test RMSE 0.8069 at 878 workers and
// 0.905 at 7,904, against 0.8038 and 0.842 so (0.8030 and 0.841 one record at a time).
// With the GPU full the epoch is bound by L2: what pays there is fewer instructions per record (no
// zero fill, no register moves, no forwarding; fp16 and bf16 products accumulate by
// mixed-precision fma, exact as the widened ones; f32x2 pairs in the update).  1024 threads per
// SM: with 80 registers and 768 threads an epoch with row copies takes 8.36 ms, 8.25 here.  The
// random bits of stochastic rounding want 96 registers (0.93 ms with 64, and 0.98 in blocks of 128).
// Measured per epoch on GB300 against one record at a time: 300 x 120, 20,000 ratings, fp32
// 0.41 -> 0.23 ms; 3,000 x 1,200, 200,000, fp16 0.56 -> 0.35; 120,047 x 62,501, 12.4M, k = 64,
// bf16-SR 2.59 -> 0.85 (to 1.12 by cvt.rs); 480,189 x 17,770, 99M, fp16 with row copies
// 8.63 -> 8.25.

// ---- contended rows -----------------------------------------------------------------------
//
// A row that many workers hold at once is bound by its cache lines, and of the updates that meet
// on it some are lost: which ones depends on how long a record is between load and store, so the
// two kernels leave such rows at other values.  How far two records at a time are from one, as a
// multiple of how far two runs of one are apart (medians over 36 pairs of runs of the largest
// entry difference of P or Q; 10,000 x 2,000, 0.9M ratings, 878 workers, 15 epochs from a trained
// model, T records in flight on the most popular row):
//      T     fp16, k = 32 / 64 / 128 / 256     fp32, k = 32 / 64 / 128
//      2     1.1  1.1  1.1  1.2                1.3  1.3  1.2
//      5     1.1  1.2  1.2  1.4                1.2  1.4  1.5
//      17    1.1  1.1  1.4  1.4                1.2  2.4  1.7
//      28    1.1  1.0  2.1  1.7                1.2  1.4  2.4
//      73    1.0  1.1  2.5  3.1                1.3  3.2  2.1
// (stochastic rounding, k = 128 and 256: at most 1.3 up to 28, 2.3 at 73).  Nor are two records at a
// time faster on wide rows there: fp16, k = 128, 7.2 ms for 9.6 at T = 17, 9.9 for 9.8 at 28, 19.9
// for 20.7 at 73.  So a launch takes one record at a time when a row is named by more than
// contended_limit records in flight.  Whether one is, is sampled on the device before the launch
// (some thousand ratings counted by hashed id, about 10 us), and of the two launches that follow
// one returns at once.
// A 16-byte atomic exchange instead of the store spares a popular row the turns of its lines
// (480,189 x 17,770, 99M ratings, fp16, 14.2 -> 10.4 ms), but loses other updates again: 10 epochs
// there leave Q 1.8 times as far off, 20 epochs at T = 160 P 3.3 times.
constexpr int kIdBits = 14;  // hashed ids per side: 16,384 (unpopular ids share few hits)
constexpr int kSampleThreads = 1024;
constexpr int kLimitHits = 16;      // samples that a limit stands for
constexpr int kMinHits = 12;        // with fewer, chance would decide
constexpr int kMaxSamples = 32768;  // < 2^16: 16-bit counters, two to a word

// Rows of one cache line stand more (up to 73 as above, and there two records at a time are still
// faster: fp16, k = 64, 10.7 ms for 12.7), and so do rows that random rounding moves as far anyway.
constexpr int contended_limit(int row_bytes, bool sr) { return row_bytes <= 128 ? 64 : sr ? 16 : 4; }

__device__ __forceinline__ uint32_t id_hash(uint32_t id) { return (id * 0x9E3779B1u) >> (32 - kIdBits); }

// Block 0: users, block 1: items (n = 0: item rows are not written).  flags[block] = an id was
// drawn `limit` times or more.
__global__ void __launch_bounds__(kSampleThreads) sample_rows_kernel(const cumf_node *R, uint64_t nnz, uint32_t m,
                                                                     uint32_t n, int samples, uint32_t limit,
                                                                     uint64_t key, uint32_t *flags) {
    __shared__ uint32_t cnt[(1 << kIdBits) / 2];
    for (int i = threadIdx.x; i < (1 << kIdBits) / 2; i += kSampleThreads) cnt[i] = 0;
    __syncthreads();
    const uint32_t rows = blockIdx.x == 0 ? m : n;
    const uint32_t *const ids = reinterpret_cast<const uint32_t *>(R) + blockIdx.x;
#pragma unroll 8
    for (int i = threadIdx.x; i < samples; i += kSampleThreads) {
        const uint32_t id = __ldg(ids + 3 * mulhi64(splitmix64(key + (uint64_t)i), nnz));
        if (id < rows) {
            const uint32_t h = id_hash(id);
            atomicAdd(&cnt[h >> 1], 1u << ((h & 1) * 16));
        }
    }
    __syncthreads();
    int over = 0;
    for (int i = threadIdx.x; i < (1 << kIdBits) / 2; i += kSampleThreads)
        over |= (cnt[i] & 0xffffu) >= limit || (cnt[i] >> 16) >= limit;
    over = __syncthreads_or(over);
    if (threadIdx.x == 0) flags[blockIdx.x] = over != 0;
}

// FROZEN: a.freeze_q is set, and neither q's arithmetic nor its random bits are computed (a kernel of
// its own: the choice within the kernel cost the others a sixth of their time, 5,000 x 2,000,
// 400,000 ratings, fp16-SR, k = 64 0.70 -> 0.82 ms).  5.2M ratings, 50,000 users, k = 128, bf16-SR:
// 0.76 ms with q computed, 0.57 so; without stochastic rounding q's arithmetic hides.
template <int K, int KIND, int G, bool SR, bool FROZEN>
__global__ void __launch_bounds__(pair_block(SR), pair_min_blocks(SR)) sgd_pair_kernel(const UpdateArgs a) {
    if (skip_launch(a)) return;
    constexpr int ROW_WORDS = K * store_bytes(KIND) / 16;
    static_assert(ROW_WORDS == G, "one word per lane");
    constexpr int kChunk = chunk_of(G);
    constexpr int CPB = kBatch / kChunk;
    constexpr int CW = kChunk * 3;  // words of a staged chunk
    constexpr int WPL = CW / G;
    static_assert(CW % G == 0 && kBatch % kChunk == 0 && kChunk % 2 == 0, "chunk must split evenly");
    // Two chunks per group, records as they are in memory; the odd stride keeps the groups of a
    // warp on different banks.
    __shared__ uint32_t s_rec[pair_block(SR) / G][2 * CW + 1];
    const int lane = threadIdx.x % G;
    const int worker = blockIdx.x * (pair_block(SR) / G) + threadIdx.x / G;
    if (worker >= a.num_workers) return;
    const unsigned gmask =
        (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    uint4 *const P = reinterpret_cast<uint4 *>(a.P) + lane;
    uint4 *const Q = reinterpret_cast<uint4 *>(a.Q) + lane;
    const uint32_t *const Rw = reinterpret_cast<const uint32_t *>(a.R);
    uint32_t *const rec = s_rec[threadIdx.x / G];
    const uint64_t nnz = a.nnz;
    const uint32_t m1 = a.m - 1, n1 = a.n - 1;
    const float nlp = -a.lambda_p, nlq = -a.lambda_q;
    const int chunks = a.batches * CPB;
    const uint32_t x0 = (uint32_t)worker * (uint32_t)(chunks * kChunk);  // sample index of the first record
    const uint64_t pol_rec = l2_policy(a.hints != 0, false);
    const uint64_t pol_row = l2_policy(a.hints != 0, true);
    const bool pf_lane = a.prefetch > 0 && (lane & 7) == 0;  // lanes that start a 128-byte line
    int bad = 0;

    for (int ep = a.first_epoch; ep < a.first_epoch + a.n_epochs; ++ep) {
        const float lr = __ldg(a.lr + ep);
        const uint32_t round_key = (uint32_t)(splitmix64(a.seed ^ (kTagRound << 48)) + (uint64_t)ep);
        const uint64_t stream = sample_stream(a.seed, ep, worker);

        // Asynchronous copy of the records of chunk t into half t & 1 of the ring.
        auto fetch = [&](int t) {
            uint64_t base = batch_start_of(stream, t / CPB, nnz) + (uint64_t)((t % CPB) * kChunk);
            while (base >= nnz) base -= nnz;  // start < nnz: wraps more than once only when nnz < 128
            uint32_t *dst = rec + (t & 1) * CW + lane;
            if (base + kChunk <= nnz) {
                const uint32_t *src = Rw + base * 3 + lane;
#pragma unroll
                for (int i = 0; i < WPL; ++i) cp_async4(dst + i * G, src + i * G, pol_rec);
            } else {
                for (int i = 0; i < WPL; ++i) {
                    const int word = lane + i * G;
                    uint64_t r = base + (uint64_t)(word / 3);
                    while (r >= nnz) r -= nnz;
                    cp_async4(dst + i * G, Rw + r * 3 + (word % 3), pol_rec);
                }
            }
            cp_async_commit();
        };
        __syncwarp(gmask);  // the last epoch's records are no longer read
        fetch(0);
        cp_async_wait_all();
        __syncwarp(gmask);

        // One record on its own: rows p and q become the updated ones, and are stored.
        auto apply = [&](uint4 &p, uint4 &q, uint32_t uu, uint32_t vv, float r, uint32_t x) {
            float s = dot_word<KIND>(p, q, 0.f);
#pragma unroll
            for (int o = G / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(gmask, s, o);
            uint4 wp, wq;
            update_word<KIND, SR, !FROZEN>(p, q, wp, wq, lr, r - s, nlp, nlq, SR ? round_key ^ lowbias32(x) : 0u, lane);
            p = wp;
            st_row_hint(P + (uint64_t)uu * ROW_WORDS, p, pol_row);
            if (!FROZEN && !a.freeze_q) {
                q = wq;
                st_row_hint(Q + (uint64_t)vv * ROW_WORDS, q, pol_row);
            }
        };
        uint32_t nu[2], nv[2];  // ids of the next pair
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            nu[e] = rec[3 * e];
            nv[e] = rec[3 * e + 1];
        }

        for (int t = 0; t < chunks; ++t) {
            __syncwarp(gmask);  // the half refilled next is no longer read
            if (t + 1 < chunks) fetch(t + 1);
            const uint32_t *cur = rec + (t & 1) * CW;
            const int next_half = (t & 1) ? -2 * CW : 0;  // added to an index past this chunk's end

#pragma unroll 1
            for (int j = 0; j < kChunk; j += 2) {
                const uint32_t ua = nu[0], ub = nu[1], va = nv[0], vb = nv[1];
                // Ids outside the matrices load the last row instead; such records are not applied.
                uint4 *const pa = P + (uint64_t)min(ua, m1) * ROW_WORDS, *const qa = Q + (uint64_t)min(va, n1) * ROW_WORDS;
                uint4 *const pb = P + (uint64_t)min(ub, m1) * ROW_WORDS, *const qb = Q + (uint64_t)min(vb, n1) * ROW_WORDS;
                uint4 fpa = ld_row_hint(pa, pol_row), fqa = ld_row_hint(qa, pol_row);
                uint4 fpb = ld_row_hint(pb, pol_row), fqb = ld_row_hint(qb, pol_row);
                if (j == kChunk - 2) {  // the look-ahead enters the next chunk
                    cp_async_wait_all();
                    __syncwarp(gmask);
                }
                // (Past the last chunk this reads old records' ids, which are not used.)
                const uint32_t *ahead = cur + 3 * (j + 2) + (j + 2 >= kChunk ? next_half : 0);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    nu[e] = ahead[3 * e];
                    nv[e] = ahead[3 * e + 1];
                }
                if (pf_lane) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        prefetch_l2(P + (uint64_t)min(nu[e], m1) * ROW_WORDS);
                        prefetch_l2(Q + (uint64_t)min(nv[e], n1) * ROW_WORDS);
                    }
                }
                const bool oka = (ua <= m1) & (va <= n1), okb = (ub <= m1) & (vb <= n1);
                const float ra = __uint_as_float(cur[3 * j + 2]), rb = __uint_as_float(cur[3 * j + 5]);
                const uint32_t x = x0 + (uint32_t)(t * kChunk + j);
                if (__builtin_expect(oka & okb & (ua != ub) & (va != vb), 1)) {
                    float sa = dot_word<KIND>(fpa, fqa, 0.f), sb = dot_word<KIND>(fpb, fqb, 0.f);
#pragma unroll
                    for (int o = G / 2; o >= 1; o >>= 1) {
                        sa += __shfl_xor_sync(gmask, sa, o);
                        sb += __shfl_xor_sync(gmask, sb, o);
                    }
                    uint4 wpa, wqa, wpb, wqb;
                    update_word<KIND, SR, !FROZEN>(fpa, fqa, wpa, wqa, lr, ra - sa, nlp, nlq,
                                                   SR ? round_key ^ lowbias32(x) : 0u, lane);
                    st_row_hint(pa, wpa, pol_row);
                    if (!FROZEN && !a.freeze_q) st_row_hint(qa, wqa, pol_row);
                    update_word<KIND, SR, !FROZEN>(fpb, fqb, wpb, wqb, lr, rb - sb, nlp, nlq,
                                                   SR ? round_key ^ lowbias32(x + 1u) : 0u, lane);
                    st_row_hint(pb, wpb, pol_row);
                    if (!FROZEN && !a.freeze_q) st_row_hint(qb, wqb, pol_row);
                } else {
                    if (oka) {
                        apply(fpa, fqa, ua, va, ra, x);
                        if (ub == ua) fpb = fpa;
                        if (vb == va) fqb = fqa;
                    }
                    if (okb) apply(fpb, fqb, ub, vb, rb, x + 1u);
                    if (!(oka & okb)) bad = 1;
                }
            }
        }
    }
    if (bad && a.status != nullptr && lane == 0) atomicExch(a.status, (int)CUMF_ERR_RANGE);
}


// ---- deeper pipeline: rows staged asynchronously through a shared-memory ring ----------
//
// Same semantics as sgd_hogwild_kernel, with D records' rows in flight per worker instead
// of one and no registers held for them: the rows of record x+D-1 are copied (cp.async,
// 16 bytes per lane, L2 only) into ring slot (x+D-1) % D while record x is computed.  Each
// lane only ever reads back its own slices, so the copy needs no cross-lane handoff.
// In-order semantics per worker: a record whose row was written by one of the D-1 records
// processed after its copy was issued takes the row from the previous record's registers
// (distance 1) or re-reads it from global memory (distance 2..D-1).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, uint64_t pol) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "l"(pol)
                 : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr int kRingDepth = 4;
constexpr int kRingMinBlocks = 4;

template <int K, int KIND, int G, int D>
struct RingLayout {
    static constexpr int SB = store_bytes(KIND);
    static constexpr int ROW_WORDS = K * SB / 16;
    static constexpr int GPB = kBlock / G;
    static constexpr int kChunk = chunk_of(G);
    static constexpr size_t rec_bytes = (size_t)GPB * 2 * 3 * (kChunk + 1) * 4;
    static constexpr size_t rec_bytes_aligned = (rec_bytes + 15) / 16 * 16;
    static constexpr size_t ring_bytes = (size_t)GPB * D * 2 * ROW_WORDS * 16;
    static constexpr size_t smem = rec_bytes_aligned + ring_bytes;
};

template <int K, int KIND, int G, bool SR, int D>
__global__ void __launch_bounds__(kBlock, kRingMinBlocks)
sgd_ring_kernel(const UpdateArgs a) {
    using C = Conv<KIND>;
    using L = RingLayout<K, KIND, G, D>;
    constexpr int ROW_WORDS = L::ROW_WORDS;
    constexpr int NV = ROW_WORDS / G;
    constexpr int GPB = L::GPB;
    constexpr int kChunk = L::kChunk;
    constexpr int CPB = kBatch / kChunk;
    constexpr int WPL = kChunk * 3 / G;
    static_assert(NV >= 1 && NV * G == ROW_WORDS, "lane split must cover the row");
    static_assert(kChunk >= 2 * D - 1, "a staged chunk must land before its first use");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    typedef uint32_t RecBuf[2][3][kChunk + 1];
    RecBuf *s_rec = reinterpret_cast<RecBuf *>(smem_raw);

    const int lane = threadIdx.x % G;
    const int gib = threadIdx.x / G;
    const int worker = blockIdx.x * GPB + gib;
    if (worker >= a.num_workers) return;
    const unsigned gmask =
        (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    uint4 *const ring = reinterpret_cast<uint4 *>(smem_raw + L::rec_bytes_aligned) +
                        (size_t)gib * D * 2 * ROW_WORDS + lane * NV;

    uint4 *const P = reinterpret_cast<uint4 *>(a.P) + lane * NV;
    uint4 *const Q = reinterpret_cast<uint4 *>(a.Q) + lane * NV;
    const uint32_t *const Rw = reinterpret_cast<const uint32_t *>(a.R);
    const uint64_t nnz = a.nnz;
    const float lp = a.lambda_p, lq = a.lambda_q;
    const int chunks = a.batches * CPB;
    const int total = chunks * kChunk;
    const uint64_t pol_rec = l2_policy(a.hints != 0, false);
    const uint64_t pol_row = l2_policy(a.hints != 0, true);
    int bad = 0;

    for (int ep = a.first_epoch; ep < a.first_epoch + a.n_epochs; ++ep) {
        const float lr = __ldg(a.lr + ep);
        const uint32_t round_key = (uint32_t)(splitmix64(a.seed ^ (kTagRound << 48)) + (uint64_t)ep);

        auto fetch = [&](int t) {  // records of chunk t into buffer t & 1 (copies join the next group)
            const uint64_t start = batch_start(a.seed, ep, worker, t / CPB, nnz);
            uint64_t base = start + (uint64_t)((t % CPB) * kChunk);
            while (base >= nnz) base -= nnz;
#pragma unroll
            for (int i = 0; i < WPL; ++i) {
                const int word = lane + i * G;
                uint64_t rec = base + (uint64_t)(word / 3);
                while (rec >= nnz) rec -= nnz;
                cp_async4(&s_rec[gib][t & 1][word % 3][word / 3], Rw + rec * 3 + (word % 3), pol_rec);
            }
        };
        auto rec_field = [&](int x, int f) -> uint32_t { return s_rec[gib][(x / kChunk) & 1][f][x % kChunk]; };
        auto issue = [&](int y) {  // rows of record y into slot y % D; always commits one group
            if (y < total) {
                const uint32_t uy = rec_field(y, 0), vy = rec_field(y, 1);
                if ((uy < a.m) & (vy < a.n)) {
                    uint4 *slot = ring + (size_t)(y % D) * 2 * ROW_WORDS;
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        cp_async16(slot + i, P + (uint64_t)uy * ROW_WORDS + i, pol_row);
                        cp_async16(slot + ROW_WORDS + i, Q + (uint64_t)vy * ROW_WORDS + i, pol_row);
                    }
                }
            }
            cp_async_commit();
        };

        fetch(0);
        cp_async_commit();
        cp_async_wait_all();
        __syncwarp(gmask);
        if (chunks > 1) fetch(1);  // joins the first row group below
#pragma unroll 1
        for (int y = 0; y < D - 1; ++y) issue(y);

        uint32_t pu[D - 1], pv[D - 1];
#pragma unroll
        for (int i = 0; i < D - 1; ++i) pu[i] = pv[i] = 0xffffffffu;
        uint4 wp[NV], wq[NV];  // rows written by the previous record
#pragma unroll
        for (int i = 0; i < NV; ++i) wp[i] = wq[i] = make_uint4(0, 0, 0, 0);

#pragma unroll 1
        for (int x = 0; x < total; ++x) {
            const int t = x / kChunk, j = x % kChunk;
            if (j == 0 && t >= 1) {
                __syncwarp(gmask);  // everyone is done with chunk t-1's buffer
                if (t + 1 < chunks) fetch(t + 1);
            }
            if (j == kChunk - D + 1 && t + 1 < chunks) __syncwarp(gmask);  // chunk t+1 visible to all lanes
            issue(x + D - 1);
            cp_async_wait_group<D - 1>();  // this lane's slices of record x have landed

            const uint32_t u = rec_field(x, 0), v = rec_field(x, 1);
            const bool ok = (u < a.m) & (v < a.n);
            if (ok) {
                const float r = __uint_as_float(rec_field(x, 2));
                const uint4 *slot = ring + (size_t)(x % D) * 2 * ROW_WORDS;
                bool p_reload = false, q_reload = false;
#pragma unroll
                for (int i = 1; i < D - 1; ++i) {
                    p_reload |= (u == pu[i]);
                    q_reload |= (v == pv[i]);
                }
                uint4 fp[NV], fq[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    fp[i] = (u == pu[0]) ? wp[i] : p_reload ? ld_row(P + (uint64_t)u * ROW_WORDS + i) : slot[i];
                    fq[i] = (v == pv[0]) ? wq[i] : q_reload ? ld_row(Q + (uint64_t)v * ROW_WORDS + i) : slot[ROW_WORDS + i];
                }
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < NV; ++i) {
#pragma unroll
                    for (int h = 0; h < C::kPairs; ++h) {
                        const float2 pp = C::get(fp[i], h), qq = C::get(fq[i], h);
                        s = __fmaf_rn(pp.x, qq.x, s);
                        s = __fmaf_rn(pp.y, qq.y, s);
                    }
                }
#pragma unroll
                for (int o = G / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(gmask, s, o);
                const float err = r - s;
                uint32_t key = 0;
                if (SR) key = round_key ^ lowbias32((uint32_t)worker * (uint32_t)total + (uint32_t)x);
                if (SR && a.freeze_q) {
                    update_rows<C, NV, SR, false>(fp, fq, wp, wq, lr, err, lp, lq, key, lane);
                } else {
                    update_rows<C, NV, SR, true>(fp, fq, wp, wq, lr, err, lp, lq, key, lane);
                    if (a.freeze_q) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) wq[i] = fq[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    st_row_hint(P + (uint64_t)u * ROW_WORDS + i, wp[i], pol_row);
                    if (!a.freeze_q) st_row_hint(Q + (uint64_t)v * ROW_WORDS + i, wq[i], pol_row);
                }
            } else {
                bad = 1;
            }
#pragma unroll
            for (int i = D - 2; i >= 1; --i) {
                pu[i] = pu[i - 1];
                pv[i] = pv[i - 1];
            }
            pu[0] = ok ? u : 0xffffffffu;
            pv[0] = ok ? v : 0xffffffffu;
        }
        cp_async_wait_all();
        __syncwarp(gmask);
    }
    if (bad && a.status != nullptr && lane == 0) atomicExch(a.status, (int)CUMF_ERR_RANGE);
}

using KernelFn = void (*)(const UpdateArgs);

struct KernelEntry {
    int k, kind, lanes;
    bool sr;
    KernelFn fn;          // sgd_hogwild_kernel
    KernelFn pair;        // sgd_pair_kernel (nullptr where a lane holds several words)
    KernelFn frozen;      // the same with item rows frozen
    KernelFn ring;        // deeper-pipeline variant (nullptr where not built)
    size_t ring_smem;     // its dynamic shared memory per block
};

template <int K, int KIND, int G, bool SR, bool FROZEN>
constexpr KernelFn pair_kernel() {
    if constexpr (K * store_bytes(KIND) / 16 == G) return &sgd_pair_kernel<K, KIND, G, SR, FROZEN>;
    else return nullptr;
}

#define CUMF_K(K, KIND, G, SR) {K, KIND, G, SR, &sgd_hogwild_kernel<K, KIND, G, SR>, pair_kernel<K, KIND, G, SR, false>(), \
    pair_kernel<K, KIND, G, SR, SR>(), &sgd_ring_kernel<K, KIND, G, SR, kRingDepth>, RingLayout<K, KIND, G, kRingDepth>::smem}
#define CUMF_K_ALL_G(K, KIND, SR, G1, G2) CUMF_K(K, KIND, G1, SR), CUMF_K(K, KIND, G2, SR)

// For each (k, storage) two lane widths: one 16-byte word per lane, or two.
const KernelEntry kKernels[] = {
    // fp16 (rows of 2k bytes)
    CUMF_K(32, kHalf, 4, false),
    CUMF_K_ALL_G(64, kHalf, false, 8, 4),
    CUMF_K_ALL_G(128, kHalf, false, 16, 8),
    CUMF_K_ALL_G(256, kHalf, false, 32, 16),
    CUMF_K(32, kHalf, 4, true),
    CUMF_K_ALL_G(64, kHalf, true, 8, 4),
    CUMF_K_ALL_G(128, kHalf, true, 16, 8),
    CUMF_K_ALL_G(256, kHalf, true, 32, 16),
    // bf16
    CUMF_K(32, kBf16, 4, false),
    CUMF_K_ALL_G(64, kBf16, false, 8, 4),
    CUMF_K_ALL_G(128, kBf16, false, 16, 8),
    CUMF_K_ALL_G(256, kBf16, false, 32, 16),
    CUMF_K(32, kBf16, 4, true),
    CUMF_K_ALL_G(64, kBf16, true, 8, 4),
    CUMF_K_ALL_G(128, kBf16, true, 16, 8),
    CUMF_K_ALL_G(256, kBf16, true, 32, 16),
    // fp32 (rows of 4k bytes)
    CUMF_K_ALL_G(32, kFloat, false, 8, 4),
    CUMF_K_ALL_G(64, kFloat, false, 16, 8),
    CUMF_K_ALL_G(128, kFloat, false, 32, 16),
    CUMF_K_ALL_G(256, kFloat, false, 32, 16),
};

#undef CUMF_K_ALL_G
#undef CUMF_K

const KernelEntry *find_kernel(int k, int precision, int lanes) {
    const int kind = store_of_precision(precision);
    const bool sr = (precision == CUMF_BF16_SR || precision == CUMF_FP16_SR);
    const KernelEntry *first = nullptr;
    for (const KernelEntry &e : kKernels) {
        if (e.k != k || e.kind != kind || e.sr != sr) continue;
        if (lanes == 0) return &e;  // first listed = tuned default
        if (e.lanes == lanes) return &e;
        if (!first) first = &e;
    }
    return lanes == 0 ? first : nullptr;
}

}  // namespace

int default_lanes(int k, int precision) {
    const KernelEntry *e = find_kernel(k, precision, 0);
    return e ? e->lanes : 0;
}

bool lanes_supported(int k, int precision, int lanes) {
    return find_kernel(k, precision, lanes) != nullptr;
}

// The ring kernels need more than the default 48 KB of dynamic shared memory.
static cudaError_t prepare_ring(const KernelEntry *e) {
    return cudaFuncSetAttribute(e->ring, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e->ring_smem);
}

int resident_workers(int k, int precision, int lanes, int sm_count) {
    const KernelEntry *e = find_kernel(k, precision, lanes);
    if (!e) return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, e->fn, kBlock, 0) != cudaSuccess) return 0;
    int threads = blocks * kBlock;
    if (e->pair) {  // either kernel may run (launch_sgd_update)
        const int t = pair_block(e->sr);
        for (KernelFn fn : {e->pair, e->frozen}) {
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, t, 0) != cudaSuccess) return 0;
            threads = std::min(threads, blocks * t);
        }
    }
    return threads / e->lanes * sm_count;
}

int wave_workers(int k, int precision, int lanes, int sm_count) {
    const KernelEntry *e = find_kernel(k, precision, lanes);
    int devices = 0;
    if (!e || cudaGetDeviceCount(&devices) != cudaSuccess || devices <= 0) return 0;
    return kWaveThreads / e->lanes * sm_count;
}

// With the hot rows split into copies, or with the item rows frozen (fold-in epochs), no
// worker queues on a hot row's lines: the kernel is issue-bound while P and Q stay mostly in
// L2, and the prefetch instructions cost more than they save (c2, 480,189 x 17,770, per
// epoch: fp16 9.03 against 9.69 ms, fp32 18.2 against 19.9, bf16-SR 20.0 against 20.8; a
// 5.2M-rating fold-in epoch: fp16 0.76 against 0.85 ms, bf16-SR 1.31 against 1.37); with
// factors far beyond L2 the row loads go to DRAM and the prefetch pays again (c3, 1,000,990 x
// 624,961, 416 MB of fp16 factors: 28.2 ms with it against 31.4 without).
static int copies_prefetch(int32_t m, int32_t n, int k, int precision, int l2) {
    const double bytes = ((double)m + (double)n) * k * elem_bytes(precision);
    return bytes > 2.0 * l2 ? kDefaultPrefetch : 0;
}

Tuning resolve_tuning(int k, int precision, Tuning t) {
    if (t.lanes == 0) t.lanes = default_lanes(k, precision);
    if (t.prefetch < 0) t.prefetch = kDefaultPrefetch;
    if (t.prefetch > 15) t.prefetch = 15;
    if (t.hints < 0) t.hints = kDefaultHints;
    if (t.ring < 0) t.ring = kDefaultRing;
    return t;
}

cudaError_t launch_sgd_update(const cumf_node *d_R, int64_t nnz, void *d_P, int32_t m,
                              void *d_Q, int32_t n, int k, int precision, int num_workers,
                              const Tuning &tuning, const float *d_lr, int first_epoch,
                              int n_epochs, float lambda_p, float lambda_q, uint64_t seed,
                              int *d_status, cudaStream_t stream, int *lanes_used, void *d_flags) {
    Tuning t = resolve_tuning(k, precision, tuning);
    int dev = 0, l2 = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        l2 = 126 << 20;
        sms = 152;
    }
    const KernelEntry *e = find_kernel(k, precision, t.lanes);
    if (!e) return cudaErrorInvalidValue;
    if (tuning.prefetch < 0 && (tuning.copies || tuning.freeze_q)) t.prefetch = copies_prefetch(m, n, k, precision, l2);
    if (lanes_used) *lanes_used = e->lanes;
    if (nnz <= 0 || n_epochs <= 0 || num_workers <= 0) return cudaSuccess;
    UpdateArgs a;
    a.R = d_R;
    a.nnz = (uint64_t)nnz;
    a.P = d_P;
    a.Q = d_Q;
    a.m = (uint32_t)m;
    a.n = (uint32_t)n;
    a.lr = d_lr;
    a.first_epoch = first_epoch;
    a.n_epochs = n_epochs;
    a.num_workers = num_workers;
    a.batches = (int)batches_per_worker(nnz, num_workers);
    a.lambda_p = lambda_p;
    a.lambda_q = lambda_q;
    a.seed = seed;
    a.status = d_status;
    a.prefetch = t.prefetch;
    a.hints = t.hints;
    a.freeze_q = t.freeze_q;
    a.contended = nullptr;
    a.run_contended = 0;
    // Every worker has to run an epoch before any runs the next one's learning rate: with more
    // workers than fit, one launch per epoch.
    if (n_epochs > 1 && !t.ring && num_workers > resident_workers(k, precision, e->lanes, sms)) {
        for (int ep = first_epoch; ep < first_epoch + n_epochs; ++ep) {
            const cudaError_t ce = launch_sgd_update(d_R, nnz, d_P, m, d_Q, n, k, precision, num_workers, tuning, d_lr, ep,
                                                     1, lambda_p, lambda_q, seed, d_status, stream, nullptr, d_flags);
            if (ce != cudaSuccess) return ce;
        }
        return cudaSuccess;
    }
    if (t.ring) {
        cudaError_t ce = prepare_ring(e);
        if (ce != cudaSuccess) return ce;
        const int gpb = kBlock / e->lanes;
        e->ring<<<(num_workers + gpb - 1) / gpb, kBlock, e->ring_smem, stream>>>(a);
        return cudaGetLastError();
    }
    auto launch = [&](bool pair, const uint2 *contended) {
        const int threads = pair ? pair_block(e->sr) : kBlock, gpb = threads / e->lanes;
        a.contended = contended;
        a.run_contended = pair ? 0 : 1;
        (!pair ? e->fn : t.freeze_q ? e->frozen : e->pair)<<<(num_workers + gpb - 1) / gpb, threads, 0, stream>>>(a);
        return cudaGetLastError();
    };
    if (!e->pair) return launch(false, nullptr);
    // A copied row has few workers by its plan; and no row is named by more records than there are.
    const int wave = pair_block(e->sr) * pair_min_blocks(e->sr) / e->lanes * sms;
    const int64_t in_flight = 2ll * std::min(num_workers, wave);
    const int limit = contended_limit(k * elem_bytes(precision), e->sr);
    if (tuning.copies || in_flight <= limit) return launch(true, nullptr);
    // One record at a time also where that cannot be sampled: too few hits, no scratch, or a
    // stream capture (its replays may meet other ratings).
    const int samples = (int)std::min<int64_t>((kLimitHits * in_flight + limit - 1) / limit, kMaxSamples);
    const int64_t hits = (int64_t)samples * limit / in_flight;
    void *flags = d_flags;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (hits < kMinHits || cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
        (flags == nullptr && scratch_alloc(&flags, sizeof(uint2), stream) != cudaSuccess)) {
        cudaGetLastError();
        return launch(false, nullptr);
    }
    sample_rows_kernel<<<2, kSampleThreads, 0, stream>>>(d_R, a.nnz, a.m, t.freeze_q ? 0 : a.n, samples,
                                                         (uint32_t)(hits + 1), splitmix64(seed), static_cast<uint32_t *>(flags));
    cudaError_t ce = cudaGetLastError();
    if (ce == cudaSuccess) ce = launch(false, static_cast<const uint2 *>(flags));
    if (ce == cudaSuccess) ce = launch(true, static_cast<const uint2 *>(flags));
    const cudaError_t ef = flags == d_flags ? cudaSuccess : cudaFreeAsync(flags, stream);
    return ce == cudaSuccess ? ef : ce;
}

}  // namespace cumf
