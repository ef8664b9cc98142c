// batch.cu - many independent factorizations in one persistent launch.
//
// Problems of uneven size (m, n, nnz) and factor length k in {32, 64, 128}, fp16 factors,
// share one launch: a grid of resident blocks whose G-lane worker groups (G = 8, 16 or 32,
// chosen by the autotuner) take tasks from a global counter.  A task is one Hogwild worker of one problem: it runs that worker's
// epochs of the launch in order, each its ceil(nnz/(W*128)) batches of 128 records exactly as
// in sgd_update.cu, so a problem never has more than W workers in flight and there is no
// barrier between epochs (as in the reference's persistent kernel).  The task table order is
// chosen by the autotuner.  Each lane owns k/G consecutive halves of a row (4 to 32 B).
// The launch (counter reset + kernel) can be captured in a CUDA graph and replayed.
// Problems may carry copies of their most-rated rows (hot_rows.cu); the batch then runs one
// launch per epoch and merges the copies between epochs, all inside the same graph.
// Autotuning times candidate schedules (lanes per worker, blocks per SM, workers per
// problem, task order) with an all-zero learning-rate table: the kernel then does the same loads and stores but
// writes back the values it read (p + 0 = p, exactly representable), so the factors are
// left bit for bit unchanged.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <numeric>
#include <string>
#include <vector>

#include "cumf_sgd.h"
#include "device_common.cuh"
#include "internal.h"
#include "train_common.h"

namespace cumf {

namespace {

constexpr int kBT = 256;       // threads per block
constexpr int kBChunk = 32;    // records staged in shared memory at a time

struct BatchProblemDev {
    const cumf_node *R;
    uint64_t nnz;
    void *P;
    void *Q;
    uint32_t m, n;
    int k;
    int workers;
    int batches;
    float lp, lq;
    uint64_t seed;
    const float *lr;
};

struct BatchTask {
    int problem;
    int worker;
};

__device__ __forceinline__ void bcp_async4(void *smem, const void *gmem) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// ---- two records at a time ----------------------------------------------------------------
//
// A worker is a group of G lanes and a row is G slices of SB bytes (k / G halves); a dot product
// adds the slices' partial sums in a butterfly over G (the order that the oracle replays with
// lanes = G).  Records j and j+1 that share no row are independent: the low half of the lanes
// takes record j, the high half record j+1, each lane two slices of its record, hl and hl + G/2,
// so the butterfly's first step is an addition within the lane.  With rows of 64 to 256 bytes the
// kernel was bound by instructions per record, and this nearly halves those for ids, addresses
// and shuffles.  A pair that shares a row or names one outside the matrices goes one record after
// the other, with the same bits.  The lanes of a worker see each other's stores through the
// __syncwarp that begins every pair.
template <int SB>
struct Slice {
    uint32_t w[SB / 4];
};

template <int SB>
__device__ __forceinline__ void load_slice(Slice<SB> &s, const char *p) {
    if constexpr (SB == 4) {
        s.w[0] = __ldcg(reinterpret_cast<const uint32_t *>(p));
    } else if constexpr (SB == 8) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2 *>(p));
        s.w[0] = v.x;
        s.w[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < SB / 16; ++i) {
            const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(p) + i);
            s.w[4 * i] = v.x;
            s.w[4 * i + 1] = v.y;
            s.w[4 * i + 2] = v.z;
            s.w[4 * i + 3] = v.w;
        }
    }
}

template <int SB>
__device__ __forceinline__ void store_slice(char *p, const Slice<SB> &s) {
    if constexpr (SB == 4) {
        __stcg(reinterpret_cast<uint32_t *>(p), s.w[0]);
    } else if constexpr (SB == 8) {
        __stcg(reinterpret_cast<uint2 *>(p), make_uint2(s.w[0], s.w[1]));
    } else {
#pragma unroll
        for (int i = 0; i < SB / 16; ++i)
            __stcg(reinterpret_cast<uint4 *>(p) + i,
                   make_uint4(s.w[4 * i], s.w[4 * i + 1], s.w[4 * i + 2], s.w[4 * i + 3]));
    }
}

__device__ __forceinline__ float2 widen(uint32_t w) { return __half22float2(*reinterpret_cast<__half2 *>(&w)); }

// <p, q> over one slice, in element order.  A product of two fp16 values is exact in fp32, so the
// mixed-precision fma rounds as the fma of the widened values does.
template <int SB>
__device__ __forceinline__ float dot_slice(const Slice<SB> &p, const Slice<SB> &q) {
    float s = 0.f;
#pragma unroll
    for (int h = 0; h < SB / 4; ++h)
        asm("{.reg .f16 x, y, z, w; mov.b32 {x, y}, %1; mov.b32 {z, w}, %2;\n"
            " fma.rn.f32.f16 %0, x, z, %0; fma.rn.f32.f16 %0, y, w, %0;}\n"
            : "+f"(s)
            : "r"(p.w[h]), "r"(q.w[h]));
    return s;
}

// p + lr*(e*q - lp*p) and q + lr*(e*p_old - lq*q) (warp32.h:89-99), two elements per instruction;
// nlp = -lambda_p, nlq = -lambda_q (-(l*x) and (-l)*x are the same bits).
template <int SB>
__device__ __forceinline__ void update_slice(Slice<SB> &p, Slice<SB> &q, float lr, float err, float nlp, float nlq) {
#pragma unroll
    for (int h = 0; h < SB / 4; ++h) {
        const float2 pp = widen(p.w[h]), qq = widen(q.w[h]);
        const float2 a = __ffma2_rn(both(lr), __ffma2_rn(both(err), qq, __fmul2_rn(both(nlp), pp)), pp);
        const float2 b = __ffma2_rn(both(lr), __ffma2_rn(both(err), pp, __fmul2_rn(both(nlq), qq)), qq);
        const __half2 ha = __floats2half2_rn(a.x, a.y), hb = __floats2half2_rn(b.x, b.y);
        p.w[h] = *reinterpret_cast<const uint32_t *>(&ha);
        q.w[h] = *reinterpret_cast<const uint32_t *>(&hb);
    }
}

// What a lane keeps through a task.
struct PairLane {
    char *P, *Q;  // factor matrices at the lane's first slice
    float lr, nlp, nlq;
    int hl;       // lane within its half of the group
};

// One record on the G/2 lanes of `mask` (one half of the group, or both with a record each).
template <int G, int SB>
__device__ __forceinline__ void pair_record(const PairLane &c, unsigned mask, uint32_t u, uint32_t v, float r) {
    constexpr int H = G / 2;
    char *const p = c.P + (uint64_t)u * (G * SB), *const q = c.Q + (uint64_t)v * (G * SB);
    Slice<SB> p0, p1, q0, q1;
    load_slice(p0, p);
    load_slice(q0, q);
    load_slice(p1, p + H * SB);
    load_slice(q1, q + H * SB);
    float s = dot_slice(p0, q0) + dot_slice(p1, q1);
#pragma unroll
    for (int o = H / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(mask, s, o);
    const float err = r - s;
    update_slice(p0, q0, c.lr, err, c.nlp, c.nlq);
    update_slice(p1, q1, c.lr, err, c.nlp, c.nlq);
    store_slice(p, p0);
    store_slice(p + H * SB, p1);
    store_slice(q, q0);
    store_slice(q + H * SB, q1);
}

// One worker's epoch on one problem.
template <int G, int SB>
__device__ void run_task(const BatchProblemDev &pr, int worker, int ep, int lane, unsigned gmask, uint32_t *rec,
                         int *bad) {
    constexpr int H = G / 2;
    constexpr int CW = kBChunk * 3;       // words of a staged chunk
    constexpr int WPL = CW / G;
    constexpr int CPB = 128 / kBChunk;    // chunks per batch
    static_assert(CW % G == 0, "record staging must split over the lanes");
    const int half = lane / H;
    const int shift = threadIdx.x & 31 & ~(G - 1);
    const uint32_t group = (G == 32) ? 0xffffffffu : (1u << G) - 1u;
    PairLane c;
    c.hl = lane % H;
    c.P = static_cast<char *>(pr.P) + c.hl * SB;
    c.Q = static_cast<char *>(pr.Q) + c.hl * SB;
    c.lr = __ldg(pr.lr + ep);
    c.nlp = -pr.lp;
    c.nlq = -pr.lq;
    const uint32_t *const Rw = reinterpret_cast<const uint32_t *>(pr.R);
    const uint64_t nnz = pr.nnz;
    const uint32_t m1 = pr.m - 1, n1 = pr.n - 1;
    const int chunks = pr.batches * CPB;
    const uint64_t stream = sample_stream(pr.seed, ep, worker);
    // Asynchronous copy of the records of chunk t into half t & 1 of the ring.
    auto fetch = [&](int t) {
        uint64_t base = batch_start_of(stream, t / CPB, nnz) + (uint64_t)((t % CPB) * kBChunk);
        while (base >= nnz) base -= nnz;  // start < nnz: wraps more than once only when nnz < 128
        uint32_t *dst = rec + (t & 1) * CW + lane;
        if (base + kBChunk <= nnz) {
            const uint32_t *src = Rw + base * 3 + lane;
#pragma unroll
            for (int i = 0; i < WPL; ++i) bcp_async4(dst + i * G, src + i * G);
        } else {
            for (int i = 0; i < WPL; ++i) {
                const int word = lane + i * G;
                uint64_t r = base + (uint64_t)(word / 3);
                while (r >= nnz) r -= nnz;
                bcp_async4(dst + i * G, Rw + r * 3 + (word % 3));
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // Bit j (even): records j and j + 1 of chunk t have to go one after the other.
    auto scan = [&](int t) {
        uint32_t slow = 0;
#pragma unroll
        for (int i = 0; i < kBChunk / G; ++i) {
            const int j = lane + i * G;
            const uint32_t *w = rec + (t & 1) * CW + 3 * j, *w2 = rec + (t & 1) * CW + 3 * (j ^ 1);
            const uint32_t u = w[0], v = w[1], u2 = w2[0], v2 = w2[1];
            const bool s = (u > m1) | (v > n1) | (u2 > m1) | (v2 > n1) | (u == u2) | (v == v2);
            slow |= ((__ballot_sync(gmask, s) >> shift) & group) << (i * G);
        }
        return slow;
    };
    __syncwarp(gmask);  // the last epoch's or task's records are no longer read
    fetch(0);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp(gmask);
    uint32_t slow = scan(0);
    uint32_t nu = rec[3 * half], nv = rec[3 * half + 1];  // ids of this half's next record
    for (int t = 0; t < chunks; ++t) {
        __syncwarp(gmask);  // the half refilled next is no longer read
        if (t + 1 < chunks) fetch(t + 1);
        const uint32_t *cur = rec + (t & 1) * CW + 3 * half;
        const int next_half = (t & 1) ? -2 * CW : 0;  // added to an index past this chunk's end
#pragma unroll 1
        for (int j = 0; j < kBChunk; j += 2, slow >>= 2) {
            const uint32_t u = nu, v = nv;
            if (j == kBChunk - 2) asm volatile("cp.async.wait_all;\n" ::: "memory");  // the look-ahead enters the next chunk
            __syncwarp(gmask);  // the last pair's stores, and the next chunk's records
            // (Past the last chunk this reads old records' ids, which are not used.)
            const uint32_t *ahead = cur + 3 * (j + 2) + (j + 2 >= kBChunk ? next_half : 0);
            nu = ahead[0];
            nv = ahead[1];
            const float r = __uint_as_float(cur[3 * j + 2]);
            if (__builtin_expect((slow & 1u) == 0, 1)) {
                pair_record<G, SB>(c, gmask, u, v, r);
            } else {
                const bool ok = (u <= m1) & (v <= n1);
                if (!ok) *bad = 1;
                for (int e = 0; e < 2; ++e) {
                    if (half == e && ok) pair_record<G, SB>(c, ((1u << H) - 1u) << (shift + e * H), u, v, r);
                    __syncwarp(gmask);
                }
            }
        }
        slow = scan(t + 1);  // (past the last chunk: old records, not used)
    }
}

// Persistent grid; each G-lane group takes tasks from the global counter.  G is the lanes
// per worker (8, 16 or 32; 32 needs every k >= 64).
template <int G>
__global__ void __launch_bounds__(kBT, 4)
batch_kernel(const BatchProblemDev *probs, const BatchTask *tasks, int tasks_per_epoch, int first_epoch, int n_epochs,
             int *counter, int *status) {
    constexpr int GPB = kBT / G;
    __shared__ uint32_t s_rec[GPB][2 * kBChunk * 3 + 1];  // two chunks per group, records as in memory
    const int lane = threadIdx.x % G;
    const int gib = threadIdx.x / G;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    const int leader = (threadIdx.x & 31) & ~(G - 1);
    int bad = 0;
    while (true) {
        int g = 0;
        if (lane == 0) g = atomicAdd(counter, 1);
        g = __shfl_sync(gmask, g, leader);
        if (g >= tasks_per_epoch) break;
        const BatchTask t = tasks[g];
        const BatchProblemDev pr = probs[t.problem];
        if (pr.nnz == 0 || pr.batches == 0) continue;
        for (int ep = first_epoch; ep < first_epoch + n_epochs; ++ep) {
            if (pr.k == 128 && G == 8) run_task<G, 32>(pr, t.worker, ep, lane, gmask, s_rec[gib], &bad);
            else if ((pr.k == 128 && G == 16) || (pr.k == 64 && G == 8))
                run_task<G, 16>(pr, t.worker, ep, lane, gmask, s_rec[gib], &bad);
            else if ((pr.k == 128 && G == 32) || (pr.k == 64 && G == 16) || (pr.k == 32 && G == 8))
                run_task<G, 8>(pr, t.worker, ep, lane, gmask, s_rec[gib], &bad);
            else if ((pr.k == 64 && G == 32) || (pr.k == 32 && G == 16))
                run_task<G, 4>(pr, t.worker, ep, lane, gmask, s_rec[gib], &bad);
            else
                bad = 1;
        }
    }
    // (Only the half of the lanes whose record it was has seen a bad one.)
    if (__any_sync(gmask, bad) && status && lane == 0) atomicExch(status, (int)CUMF_ERR_RANGE);
}

}  // namespace

struct Batch {
    std::vector<cumf_batch_problem> probs;
    std::vector<BatchProblemDev> dev_probs;
    cumf_batch_tuning tuning;
    DevBuf d_probs, d_probs_zero_lr, d_tasks, d_counter, d_status, d_zero_lr;
    int tasks_per_epoch = 0;
    int sm_count = 0;
    int64_t samples_per_epoch = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_first = -1, graph_n = -1;
    bool any_hot = false;  // a problem has row copies: one launch per epoch, merges between
    ~Batch() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

namespace {

int64_t work_of(const cumf_batch_problem &p) { return p.nnz * (int64_t)p.k; }

// Rebuilds worker counts, the device problem table and the task table for b->tuning.
int batch_plan(Batch *b) {
    const cumf_batch_tuning &t = b->tuning;
    const int nprob = (int)b->probs.size();
    b->dev_probs.resize(nprob);
    b->samples_per_epoch = 0;
    std::vector<int> workers(nprob);
    for (int i = 0; i < nprob; ++i) {
        const cumf_batch_problem &p = b->probs[i];
        int w = p.num_workers;
        if (w <= 0) {  // enough workers for ~batches_target batches each
            const int64_t target = std::max(1, t.batches_target);
            w = (int)std::max<int64_t>(1, (p.nnz + 128 * target - 1) / (128 * target));
        }
        workers[i] = w;
        BatchProblemDev &d = b->dev_probs[i];
        d.R = p.d_R;
        d.nnz = (uint64_t)p.nnz;
        d.P = p.d_P;
        d.Q = p.d_Q;
        d.m = (uint32_t)p.m;
        d.n = (uint32_t)p.n;
        if (p.hot) {  // ratings may name the copies' extra rows
            int32_t hm, hn, mr, nr;
            hot_rows_dims(p.hot, &hm, &hn, &mr, &nr);
            d.m = (uint32_t)mr;
            d.n = (uint32_t)nr;
        }
        d.k = p.k;
        d.workers = w;
        d.batches = (int)batches_per_worker(p.nnz, w);
        d.lp = p.lambda_p;
        d.lq = p.lambda_q;
        d.seed = p.seed;
        d.lr = p.d_lr;
        b->samples_per_epoch += (int64_t)w * d.batches * 128;
    }
    std::vector<int> order(nprob);
    std::iota(order.begin(), order.end(), 0);
    if (t.order == 2)  // largest problems first
        std::stable_sort(order.begin(), order.end(),
                         [&](int a, int c) { return work_of(b->probs[a]) > work_of(b->probs[c]); });
    std::vector<BatchTask> tasks;
    if (t.order == 1) {  // round robin across problems
        int maxw = 0;
        for (int i : order) maxw = std::max(maxw, workers[i]);
        for (int w = 0; w < maxw; ++w)
            for (int i : order)
                if (w < workers[i]) tasks.push_back({i, w});
    } else {
        for (int i : order)
            for (int w = 0; w < workers[i]; ++w) tasks.push_back({i, w});
    }
    b->tasks_per_epoch = (int)tasks.size();
    CUMF_CUDA(b->d_probs.alloc(std::max<size_t>(1, nprob) * sizeof(BatchProblemDev)));
    CUMF_CUDA(cudaMemcpy(b->d_probs.p, b->dev_probs.data(), nprob * sizeof(BatchProblemDev), cudaMemcpyHostToDevice));
    std::vector<BatchProblemDev> zl = b->dev_probs;
    for (BatchProblemDev &d : zl) d.lr = b->d_zero_lr.as<float>();
    CUMF_CUDA(b->d_probs_zero_lr.alloc(std::max<size_t>(1, nprob) * sizeof(BatchProblemDev)));
    CUMF_CUDA(cudaMemcpy(b->d_probs_zero_lr.p, zl.data(), nprob * sizeof(BatchProblemDev), cudaMemcpyHostToDevice));
    CUMF_CUDA(b->d_tasks.alloc(std::max<size_t>(1, tasks.size()) * sizeof(BatchTask)));
    CUMF_CUDA(cudaMemcpy(b->d_tasks.p, tasks.data(), tasks.size() * sizeof(BatchTask), cudaMemcpyHostToDevice));
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    b->graph_first = b->graph_n = -1;
    return CUMF_OK;
}

// Lanes per worker that every problem of the batch supports (k / lanes halves per lane, 2..16).
bool lanes_fit(const Batch *b, int lanes) {
    if (lanes != 8 && lanes != 16 && lanes != 32) return false;
    for (const cumf_batch_problem &p : b->probs)
        if (p.k / lanes < 2) return false;
    return true;
}

cudaError_t kernel_launch(Batch *b, bool zero_lr, int first_epoch, int n_epochs, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(b->d_counter.p, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    const int bps = std::max(1, std::min(4, b->tuning.blocks_per_sm));
    const BatchProblemDev *probs = zero_lr ? b->d_probs_zero_lr.as<BatchProblemDev>() : b->d_probs.as<BatchProblemDev>();
    const int grid = bps * b->sm_count;
    switch (b->tuning.lanes) {
        case 8:
            batch_kernel<8><<<grid, kBT, 0, s>>>(probs, b->d_tasks.as<BatchTask>(), b->tasks_per_epoch, first_epoch,
                                                  n_epochs, b->d_counter.as<int>(), b->d_status.as<int>());
            break;
        case 32:
            batch_kernel<32><<<grid, kBT, 0, s>>>(probs, b->d_tasks.as<BatchTask>(), b->tasks_per_epoch, first_epoch,
                                                   n_epochs, b->d_counter.as<int>(), b->d_status.as<int>());
            break;
        default:
            batch_kernel<16><<<grid, kBT, 0, s>>>(probs, b->d_tasks.as<BatchTask>(), b->tasks_per_epoch, first_epoch,
                                                   n_epochs, b->d_counter.as<int>(), b->d_status.as<int>());
            break;
    }
    return cudaGetLastError();
}

// The epochs of one run: one persistent launch, or with row copies one launch per epoch,
// each followed by the merge of every problem's copies (zero-learning-rate trials leave the
// copies equal, so they need no merge).
int batch_launch(Batch *b, bool zero_lr, int first_epoch, int n_epochs, cudaStream_t s) {
    if (zero_lr || !b->any_hot) {
        CUMF_CUDA(kernel_launch(b, zero_lr, first_epoch, n_epochs, s));
        return CUMF_OK;
    }
    for (int ep = first_epoch; ep < first_epoch + n_epochs; ++ep) {
        CUMF_CUDA(kernel_launch(b, false, ep, 1, s));
        for (const cumf_batch_problem &p : b->probs)
            if (p.hot)
                if (int rc = cumf_hot_rows_merge(p.hot, p.d_P, p.d_Q, p.k, CUMF_FP16, s)) return rc;
    }
    return CUMF_OK;
}

}  // namespace

}  // namespace cumf

using namespace cumf;

extern "C" {

int cumf_batch_create(const cumf_batch_problem *probs, int count, void **handle) {
    if (!probs || count <= 0 || !handle) return fail(CUMF_ERR_ARG, "batch_create: bad arguments");
    int max_epoch_index = 0;
    for (int i = 0; i < count; ++i) {
        const cumf_batch_problem &p = probs[i];
        if (p.k != 32 && p.k != 64 && p.k != 128)
            return fail(CUMF_ERR_ARG, "batch_create: k must be 32, 64 or 128 (problem " + std::to_string(i) + ")");
        if (p.nnz < 0 || p.m < 1 || p.n < 1 || (p.nnz > 0 && (!p.d_R || !p.d_P || !p.d_Q || !p.d_lr)))
            return fail(CUMF_ERR_ARG, "batch_create: malformed problem " + std::to_string(i));
        if (p.num_workers > 0 && batches_per_worker(p.nnz, p.num_workers) * 4 > 0x7fffffffll)
            return fail(CUMF_ERR_ARG, "batch_create: too many batches per worker");
        if (p.hot) {
            int32_t hm, hn, mr, nr;
            hot_rows_dims(p.hot, &hm, &hn, &mr, &nr);
            if (hm != p.m || hn != p.n)
                return fail(CUMF_ERR_ARG, "batch_create: row copies planned for another shape (problem " +
                                              std::to_string(i) + ")");
        }
        max_epoch_index = std::max(max_epoch_index, p.lr_len);
    }
    Batch *b = new Batch();
    b->probs.assign(probs, probs + count);
    for (const cumf_batch_problem &p : b->probs) b->any_hot = b->any_hot || p.hot != nullptr;
    b->tuning.batches_target = 16;
    b->tuning.order = 2;
    b->tuning.blocks_per_sm = 4;
    b->tuning.lanes = 16;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, dev);
    auto bail = [&](int rc) {
        delete b;
        return rc;
    };
    if (cudaError_t e = b->d_counter.alloc(sizeof(int))) return bail(cuda_fail(e, "batch counter"));
    if (cudaError_t e = b->d_status.alloc(sizeof(int))) return bail(cuda_fail(e, "batch status"));
    if (cudaError_t e = b->d_zero_lr.alloc(std::max(1, max_epoch_index) * sizeof(float)))
        return bail(cuda_fail(e, "batch zero lr"));
    cudaMemset(b->d_status.p, 0, sizeof(int));
    cudaMemset(b->d_zero_lr.p, 0, std::max(1, max_epoch_index) * sizeof(float));
    if (int rc = batch_plan(b)) return bail(rc);
    *handle = b;
    return CUMF_OK;
}

int cumf_batch_destroy(void *handle) {
    delete static_cast<Batch *>(handle);
    return CUMF_OK;
}

int cumf_batch_set_tuning(void *handle, const cumf_batch_tuning *t) {
    Batch *b = static_cast<Batch *>(handle);
    if (!b || !t || t->order < 0 || t->order > 2 || t->batches_target < 1 || t->blocks_per_sm < 1 ||
        t->blocks_per_sm > 4)
        return fail(CUMF_ERR_ARG, "batch_set_tuning: bad tuning");
    cumf_batch_tuning c = *t;
    if (c.lanes == 0) c.lanes = 16;
    if (!lanes_fit(b, c.lanes))
        return fail(CUMF_ERR_ARG, "batch_set_tuning: lanes must be 8, 16 or 32 (32 needs every k >= 64)");
    b->tuning = c;
    return batch_plan(b);
}

int cumf_batch_get_info(void *handle, cumf_batch_tuning *t, int *tasks_per_epoch, int64_t *samples_per_epoch) {
    Batch *b = static_cast<Batch *>(handle);
    if (!b) return fail(CUMF_ERR_ARG, "batch_get_info: NULL handle");
    if (t) *t = b->tuning;
    if (tasks_per_epoch) *tasks_per_epoch = b->tasks_per_epoch;
    if (samples_per_epoch) *samples_per_epoch = b->samples_per_epoch;
    return CUMF_OK;
}

int cumf_batch_run(void *handle, int first_epoch, int n_epochs, int use_graph, void *stream) {
    Batch *b = static_cast<Batch *>(handle);
    if (!b || first_epoch < 0 || n_epochs < 0) return fail(CUMF_ERR_ARG, "batch_run: bad arguments");
    for (const cumf_batch_problem &p : b->probs)
        if (first_epoch + n_epochs > p.lr_len) return fail(CUMF_ERR_ARG, "batch_run: epochs beyond a problem's lr table");
    if (n_epochs == 0) return CUMF_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (!use_graph) return batch_launch(b, false, first_epoch, n_epochs, s);
    if (!b->exec || b->graph_first != first_epoch || b->graph_n != n_epochs) {
        if (b->exec) cudaGraphExecDestroy(b->exec);
        if (b->graph) cudaGraphDestroy(b->graph);
        b->exec = nullptr;
        b->graph = nullptr;
        cudaStream_t cap;
        CUMF_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        int rc = e == cudaSuccess ? batch_launch(b, false, first_epoch, n_epochs, cap) : CUMF_OK;
        cudaError_t e2 = cudaStreamEndCapture(cap, &b->graph);
        cudaStreamDestroy(cap);
        if (e != cudaSuccess) return cuda_fail(e, "batch graph capture");
        if (rc != CUMF_OK) return rc;
        if (e2 != cudaSuccess) return cuda_fail(e2, "batch graph end capture");
        CUMF_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
        b->graph_first = first_epoch;
        b->graph_n = n_epochs;
    }
    CUMF_CUDA(cudaGraphLaunch(b->exec, s));
    return CUMF_OK;
}

int cumf_batch_status(void *handle, int *status) {
    Batch *b = static_cast<Batch *>(handle);
    if (!b || !status) return fail(CUMF_ERR_ARG, "batch_status: bad arguments");
    CUMF_CUDA(cudaMemcpy(status, b->d_status.p, sizeof(int), cudaMemcpyDeviceToHost));
    return CUMF_OK;
}

int cumf_batch_autotune(void *handle, void *stream, cumf_batch_tuning *best, double *best_ms) {
    Batch *b = static_cast<Batch *>(handle);
    if (!b) return fail(CUMF_ERR_ARG, "batch_autotune: NULL handle");
    cudaStream_t s = (cudaStream_t)stream;
    Event e0, e1;
    CUMF_CUDA(e0.create());
    CUMF_CUDA(e1.create());
    cumf_batch_tuning top = b->tuning;
    double top_ms = 1e30;
    // Time per sample of one epoch with a zero learning rate (factors unchanged), so schedules
    // with different budgets compare fairly.
    auto trial = [&](const cumf_batch_tuning &cand) -> int {
        b->tuning = cand;
        if (int rc = batch_plan(b)) return rc;
        if (int rc = batch_launch(b, true, 0, 1, s)) return rc;  // warm-up
        CUMF_CUDA(cudaEventRecord(e0.e, s));
        if (int rc = batch_launch(b, true, 0, 1, s)) return rc;
        CUMF_CUDA(cudaEventRecord(e1.e, s));
        CUMF_CUDA(cudaEventSynchronize(e1.e));
        float ms = 0;
        CUMF_CUDA(cudaEventElapsedTime(&ms, e0.e, e1.e));
        const double per = ms / (double)std::max<int64_t>(1, b->samples_per_epoch);
        if (per < top_ms) {
            top_ms = per;
            top = cand;
        }
        return CUMF_OK;
    };
    // Stage 1: lanes per worker x blocks per SM at the default budget and order; stage 2:
    // budget x task order at the chosen lanes and blocks.
    const int lanes_c[] = {8, 16, 32};
    const int occ[] = {3, 4};
    const int targets[] = {4, 8, 16, 32};
    const int orders[] = {0, 1, 2};
    cumf_batch_tuning cand = top;
    for (int g : lanes_c) {
        if (!lanes_fit(b, g)) continue;
        for (int bps : occ) {
            cand.lanes = g;
            cand.blocks_per_sm = bps;
            if (int rc = trial(cand)) return rc;
        }
    }
    const cumf_batch_tuning stage1 = top;
    for (int bt : targets)
        for (int o : orders) {
            cand = stage1;
            cand.batches_target = bt;
            cand.order = o;
            if (int rc = trial(cand)) return rc;
        }
    b->tuning = top;
    if (int rc = batch_plan(b)) return rc;
    if (best) *best = top;
    if (best_ms) *best_ms = top_ms * (double)b->samples_per_epoch;
    return CUMF_OK;
}

}  // extern "C"
