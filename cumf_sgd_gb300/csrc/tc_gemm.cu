// tc_gemm.cu - BF16 tensor-core GEMM for sm_103a on the 5th-generation tensor cores.
//
//   C[M x N] = act(A[M x K] * B[N x K]^T + bias[N])       (A, B bf16 row-major; fp32 accumulate)
//
// Used by the warm-start MLP (forward: activations x W^T; backward: dX = dY W and
// dW = dY^T X, given as TN products on transposed copies; a training step's products have their
// own epilogues, tc_train_kernel and tc_wgrad_kernel below).  One CTA of 256 threads computes a
// 128 x BN tile (BN = 128 or 256):
//   - thread 0 is the TMA producer: operand tiles of 64 K-elements (128-byte rows) arrive by
//     cp.async.bulk.tensor.2d with the 128-byte swizzle into a ring of shared memory (2 stages
//     for K <= 1024, so two CTAs share an SM; 4 stages for longer K),
//     each stage guarded by a `full` mbarrier (armed with the expected byte count) and an
//     `empty` mbarrier;
//   - thread 32 issues tcgen05.mma.cta_group::1.kind::f16 (M=128, N=BN, K=16) four times per
//     stage, accumulating in tensor memory (BN fp32 columns from tcgen05.alloc), and
//     tcgen05.commit releases the stage to the producer through `empty`;
//   - after the last stage a commit to `done` releases the epilogue: eight warps read the
//     accumulator with tcgen05.ld (warp w: lanes 32 (w % 4).., half w / 4 of the columns, 32
//     columns at a time), add the bias, apply the activation, and pass each 32 x 32 block
//     through shared memory (the idle operand ring) so that the global stores are whole
//     128-byte lines;
//   - when the output has too few tiles to fill the GPU and K is long, K is split over grid.z
//     and the partial tiles are added into a zeroed fp32 output with vector atomics.
// Every mbarrier wait is bounded; on timeout the kernel records CUMF_ERR_TIMEOUT, stops
// issuing work, waits (bounded) for what it issued and releases its tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "cumf_sgd.h"
#include "internal.h"
#include "tc_gemm.h"

namespace cumf {

namespace {

constexpr int kTcThreads = 256;  // 8 warps: all read the accumulator in the epilogue
constexpr int kStgStride = 36;    // floats per staged row (144 bytes: 16-byte aligned, conflict-free)
constexpr int kTcBM = 128;
constexpr int kTcBK = 64;
constexpr unsigned long long kWaitNs = 2000000000ull;  // an mbarrier wait gives up after 2 s
constexpr long long kSpinLimit = 1ll << 28;            // and after this many polls in any case

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Instruction descriptor for kind::f16: D fp32 (bits 4-5 = 1), A and B bf16 (7-9, 10-12 = 1),
// both K-major (15, 16 = 0), N >> 3 at 17-22, M >> 4 at 24-28.
template <int BN>
__device__ __forceinline__ uint32_t instr_desc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kTcBM >> 4) << 24);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the phase of parity `parity` of an mbarrier; false after kWaitNs of global time.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    const unsigned long long t0 = global_ns();
    for (long long i = 0; i < kSpinLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 63) == 63 && global_ns() - t0 > kWaitNs) return false;
    }
    return false;
}

__device__ __forceinline__ float gelu(float x) {
    // tanh form (Hendrycks & Gimpel 2016): 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3)))
    const float c = 0.7978845608028654f;
    return 0.5f * x * (1.0f + tanhf(c * (x + 0.044715f * x * x * x)));
}


__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;              // leading byte offset: unused for swizzled K-major
    d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset: one 8-row atom
    d |= (uint64_t)1 << 46;              // descriptor version (sm_100 family)
    d |= (uint64_t)2 << 61;              // 128-byte swizzle
    return d;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}

// Epilogue of one warp's 32 rows x 32 columns (rows r0.., columns col0..; lane = row in r[]):
// the values pass through shared memory (stg, 32 x kStgStride floats) so that the global
// stores are whole 128-byte lines per 8 lanes (fp32) or 64-byte segments per 4 lanes (bf16).
// partial: fp32 partial sums added with vector atomics (split K), no bias or activation.
__device__ __forceinline__ void stage_f32(float *stg, const float (&v)[32], int lane) {
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4 *>(stg + lane * kStgStride + 4 * q) =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    __syncwarp();
}

__device__ __forceinline__ void write_f32(const float *stg, float *dst, int r0, int col0, int M, int N, int ldo,
                                          bool vec_ok, bool atomic, int lane) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        const int row = it * 4 + (lane >> 3), c = (lane & 7) * 4;
        const int gr = r0 + row, col = col0 + c;
        if (gr >= M || col >= N) continue;
        const float4 x = *reinterpret_cast<const float4 *>(stg + row * kStgStride + c);
        float *o = dst + (size_t)gr * ldo + col;
        if (vec_ok && col + 3 < N) {
            if (atomic)
                atomicAdd(reinterpret_cast<float4 *>(o), x);
            else
                *reinterpret_cast<float4 *>(o) = x;
        } else {
            const float xs[4] = {x.x, x.y, x.z, x.w};
            for (int e = 0; e < 4 && col + e < N; ++e) {
                if (atomic)
                    atomicAdd(o + e, xs[e]);
                else
                    o[e] = xs[e];
            }
        }
    }
}

__device__ __forceinline__ void write_bf16(float *stg, const float (&v)[32], __nv_bfloat16 *dst, int r0, int col0,
                                           int M, int N, int ldo, bool vec_ok, int lane) {
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint4 w;
        __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&w);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
        *reinterpret_cast<uint4 *>(stg + lane * kStgStride + 4 * q) = w;
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int row = it * 8 + (lane >> 2), c = (lane & 3) * 8;
        const int gr = r0 + row, col = col0 + c;
        if (gr >= M || col >= N) continue;
        const uint4 x = *reinterpret_cast<const uint4 *>(stg + row * kStgStride + (lane & 3) * 4);
        __nv_bfloat16 *o = dst + (size_t)gr * ldo + col;
        if (vec_ok && col + 7 < N) {
            *reinterpret_cast<uint4 *>(o) = x;
        } else {
            const __nv_bfloat16 *xs = reinterpret_cast<const __nv_bfloat16 *>(&x);
            for (int e = 0; e < 8 && col + e < N; ++e) o[e] = xs[e];
        }
    }
}

__device__ __forceinline__ void epilogue_chunk(float *stg, const uint32_t (&r)[32], int r0, int col0, int M, int N,
                                               const float *__restrict__ bias, int act, void *out, int out_f32,
                                               int ldo, float *pre_out, bool partial, int lane) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
    const bool al16 = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    if (partial) {
        stage_f32(stg, v, lane);
        write_f32(stg, reinterpret_cast<float *>(out), r0, col0, M, N, ldo, al16 && (ldo & 3) == 0, true, lane);
        return;
    }
    if (bias) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (col0 + j < N) v[j] += __ldg(bias + col0 + j);
    }
    if (pre_out) {
        stage_f32(stg, v, lane);
        write_f32(stg, pre_out, r0, col0, M, N, ldo,
                  (reinterpret_cast<uintptr_t>(pre_out) & 15u) == 0 && (ldo & 3) == 0, false, lane);
    }
    if (act == 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = gelu(v[j]);
    }
    if (out_f32) {
        stage_f32(stg, v, lane);
        write_f32(stg, reinterpret_cast<float *>(out), r0, col0, M, N, ldo, al16 && (ldo & 3) == 0, false, lane);
    } else {
        write_bf16(stg, v, reinterpret_cast<__nv_bfloat16 *>(out), r0, col0, M, N, ldo, al16 && (ldo & 7) == 0,
                   lane);
    }
}

template <int BN, int kStages>
struct TmaSmem {
    static constexpr int A_BYTES = kTcBM * 128;  // 128 rows x 64 bf16
    static constexpr int B_BYTES = BN * 128;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int TOTAL = 1024 + kStages * STAGE + 256;  // alignment slack + barriers
};

// One CTA's 128 x BN accumulator: the operand ring and barriers in shared memory, and the tensor
// memory.  Every thread of the CTA calls setup_tile, tile_product and, after the epilogue,
// release_tile.
template <int BN, int kStages>
struct Tile {
    unsigned char *ring;
    uint64_t *full, *empty, *done;
    int *abort_flag, *issued_slot;
    uint32_t tmem;
};

template <int BN, int kStages>
__device__ __forceinline__ Tile<BN, kStages> setup_tile(unsigned char *smem_raw, const CUtensorMap &map_a,
                                                        const CUtensorMap &map_b) {
    Tile<BN, kStages> t;
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    t.ring = smem_raw + (base - raw);
    t.full = reinterpret_cast<uint64_t *>(t.ring + kStages * TmaSmem<BN, kStages>::STAGE);
    t.empty = t.full + kStages;
    t.done = t.empty + kStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(t.done + 1);
    t.abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    t.issued_slot = t.abort_flag + 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&t.full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&t.empty[i])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(t.done)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        *t.abort_flag = 0;
        *t.issued_slot = 0;
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    t.tmem = *tmem_slot;
    return t;
}

// The product over the K stages kt0 .. kt0 + KT: thread 0 streaming, thread 32 issuing, every
// thread waiting.  Returns whether the accumulator is valid; the operand ring is idle then.
template <int BN, int kStages>
__device__ __forceinline__ bool tile_product(const Tile<BN, kStages> &t, const CUtensorMap &map_a,
                                             const CUtensorMap &map_b, int m0, int n0, int kt0, int KT, int *status,
                                             int no_copies) {
    using S = TmaSmem<BN, kStages>;
    uint64_t *full = t.full, *empty = t.empty, *done = t.done;
    int *abort_flag = t.abort_flag, *issued_slot = t.issued_slot;
    const uint32_t base = smem_u32(t.ring), tmem = t.tmem;

    if (threadIdx.x == 0 && KT > 0 && !no_copies) {  // TMA producer (no_copies: the wait self-test)
        for (int i = 0; i < KT; ++i) {
            const int st = i % kStages;
            if (i >= kStages && !mbar_wait(smem_u32(&empty[st]), ((i / kStages) - 1) & 1)) {
                atomicExch(abort_flag, 1);
                break;
            }
            const uint32_t fb = smem_u32(&full[st]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb), "r"(S::STAGE)
                         : "memory");
            const uint32_t a_dst = base + st * S::STAGE;
            tma_load_2d(a_dst, &map_a, (kt0 + i) * kTcBK, m0, fb);
            tma_load_2d(a_dst + S::A_BYTES, &map_b, (kt0 + i) * kTcBK, n0, fb);
            *issued_slot = i + 1;
        }
    } else if (threadIdx.x == 32 && KT > 0) {  // MMA issuer
        for (int i = 0; i < KT; ++i) {
            const int st = i % kStages;
            if (!mbar_wait(smem_u32(&full[st]), (i / kStages) & 1)) {
                atomicExch(abort_flag, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t a0 = base + st * S::STAGE, b0 = a0 + S::A_BYTES;
#pragma unroll
            for (int s = 0; s < kTcBK / 16; ++s) {
                const uint32_t acc = (i > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(sw128_desc(a0 + s * 32)), "l"(sw128_desc(b0 + s * 32)), "r"(instr_desc<BN>()), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(&empty[st]))
                         : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                         smem_u32(done))
                     : "memory");
    }
    // Everyone waits for the accumulator (bounded), then agrees on whether it is valid.
    int ok = 1;
    if (KT > 0) ok = mbar_wait(smem_u32(done), 0) ? 1 : 0;
    __syncwarp();
    ok = __syncthreads_and(ok && (*abort_flag == 0));
    if (!ok) {
        if (threadIdx.x == 0) {
            if (status) atomicExch(status, (int)CUMF_ERR_TIMEOUT);
            // Bounded drain: the last copy issued into each stage, then every MMA.
            const int issued = *issued_slot;
            for (int st = 0; st < kStages && st < issued; ++st) {
                const int last = st + ((issued - 1 - st) / kStages) * kStages;
                mbar_wait(smem_u32(&full[st]), (last / kStages) & 1);
            }
            mbar_wait(smem_u32(done), 0);
        }
        return false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    return KT > 0;
}

template <int BN>
__device__ __forceinline__ void release_tile(uint32_t tmem) {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(BN));
    }
}

// The accumulator's 32 columns c0.. of this warp's 32 tensor-memory lanes (32 (warp % 4)..).
__device__ __forceinline__ void load_acc(uint32_t (&r)[32], uint32_t tmem, int c0) {
    const uint32_t taddr = tmem + ((uint32_t)((threadIdx.x >> 5 & 3) * 32) << 16) + (uint32_t)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
        "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
        "[%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

template <int BN, int kStages>
__global__ void __launch_bounds__(kTcThreads, kStages == 2 ? 2 : 1)
tc_gemm_tma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M,
                   int N, int K, const float *__restrict__ bias, int act, void *out, int out_f32, int ldo,
                   float *pre_out, int *status, int splits, int no_copies) {
    extern __shared__ unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kTcBM, n0 = blockIdx.y * BN;
    const int KT_all = (K + kTcBK - 1) / kTcBK;
    const int kt0 = (int)((long long)KT_all * blockIdx.z / splits);
    const int kt1 = (int)((long long)KT_all * (blockIdx.z + 1) / splits);
    const Tile<BN, kStages> t = setup_tile<BN, kStages>(smem_raw, map_a, map_b);
    if (tile_product(t, map_a, map_b, m0, n0, kt0, kt1 - kt0, status, no_copies)) {
        // Warp w: half w / 4 of the columns; the idle ring holds each warp's staging block.
        float *stg = reinterpret_cast<float *>(t.ring) + warp * (32 * kStgStride);
        const int half = warp >> 2, r0 = m0 + (warp & 3) * 32;
        for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2) && n0 + c0 < N; c0 += 32) {
            uint32_t r[32];
            load_acc(r, t.tmem, c0);
            epilogue_chunk(stg, r, r0, n0 + c0, M, N, bias, act, out, out_f32, ldo, pre_out, splits > 1, lane);
        }
    }
    release_tile<BN>(t.tmem);
}

// ---- products of a training step ----------------------------------------------------------

// gelu(x) as above, and its derivative: they share the tanh, which is most of either.
__device__ __forceinline__ float gelu_slope(float x, float &slope) {
    const float c = 0.7978845608028654f;
    const float t = tanhf(c * (x + 0.044715f * x * x * x));
    slope = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * x * x);
    return 0.5f * x * (1.0f + t);
}

// a + b = s + err exactly (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float a, float b, float &err) {
    const float s = __fadd_rn(a, b), z = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
    return s;
}

// The sum of d[j]^2 as a double.  FP64 arithmetic is some sixty times slower than FP32 here, so
// the exact squares (product and its fma remainder) are added in three floats whose roundings are
// kept (72 bits); values whose squares or remainders would leave FP32's range go through double.
__device__ __forceinline__ double sum_squares(const float (&d)[32]) {
    float top = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) top = fmaxf(top, fabsf(d[j]));
    if (top < 1.152921504606847e18f && (top > 9.313225746154785e-10f || top == 0.f)) {  // 2^60, 2^-30
        float hi = 0.f, mid = 0.f, lo = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float p = __fmul_rn(d[j], d[j]), e = __fmaf_rn(d[j], d[j], -p);
            float a, b, c;
            hi = two_sum(hi, p, a);
            mid = two_sum(mid, a, b);
            mid = two_sum(mid, e, c);
            lo = __fadd_rn(lo, __fadd_rn(b, c));
        }
        return (double)hi + ((double)mid + (double)lo);
    }
    double sum = 0;
    for (int j = 0; j < 32; ++j) sum += (double)d[j] * d[j];
    return sum;
}

// Two bf16 values of exactly representable floats.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// A warp's 32 x 32 block (lane = row) of bf16 values, to out (ldo columns) and out_t (ldt rows);
// with colsum, the block's column sums: rows y, y + 8, y + 16, y + 24 for each y < 8, then these
// eight sums, in order.
__device__ __forceinline__ void write_both(float *stg, const float (&v)[32], int r0, int col0, __nv_bfloat16 *out,
                                           int ldo, __nv_bfloat16 *out_t, int ldt, float *colsum, int lane) {
    stage_f32(stg, v, lane);
#pragma unroll
    for (int it = 0; it < 4; ++it) {  // four lanes per row, 16 bytes each
        const int row = it * 8 + (lane >> 2), c = (lane & 3) * 8;
        const float4 a = *reinterpret_cast<const float4 *>(stg + row * kStgStride + c);
        const float4 b = *reinterpret_cast<const float4 *>(stg + row * kStgStride + c + 4);
        *reinterpret_cast<uint4 *>(out + (size_t)(r0 + row) * ldo + col0 + c) =
            make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
    }
    float x[32];  // lane = column
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = stg[i * kStgStride + lane];
    uint4 *t = reinterpret_cast<uint4 *>(out_t + (size_t)(col0 + lane) * ldt + r0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        t[q] = make_uint4(pack_bf16(x[8 * q], x[8 * q + 1]), pack_bf16(x[8 * q + 2], x[8 * q + 3]),
                          pack_bf16(x[8 * q + 4], x[8 * q + 5]), pack_bf16(x[8 * q + 6], x[8 * q + 7]));
    if (colsum) {
        float total = 0.f;
#pragma unroll
        for (int y = 0; y < 8; ++y) total += ((x[y] + x[y + 8]) + x[y + 16]) + x[y + 24];
        colsum[(size_t)(r0 >> 5) * ldo + col0 + lane] = total;
    }
}

// A 128 x BN tile by 4 BN threads, so that each warp's epilogue is one 32 x 32 block: the
// activation's arithmetic and the stores' latency, not the product (K of a few stages), are what
// these kernels take.  Fused, because every pass over a 4096 x 512 batch between the products
// (transposes, gelu', column sums, loss) was a launch of 2 to 8 us: a training step of 4096 rows
// (131 -> 512 -> 512 -> 128) took 127 us of device time in 25 launches, 70 in 8.
// What the epilogue reads (slopes, targets) is fetched before the product's waits.
template <int BN, int kStages, int MODE>
__global__ void __launch_bounds__(4 * BN, BN == 128 ? 1 : 2)
tc_train_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M, int N,
                int K, const __grid_constant__ TrainEpilogue ep, int *status) {
    static_assert(4 * BN / 32 * 32 * kStgStride * 4 <= kStages * TmaSmem<BN, kStages>::STAGE, "staging fits the ring");
    extern __shared__ unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * BN, c0 = (warp >> 2) * 32;
    const int r0 = blockIdx.x * kTcBM + (warp & 3) * 32, col0 = n0 + c0;
    const bool mine = col0 < N;
    const Tile<BN, kStages> t = setup_tile<BN, kStages>(smem_raw, map_a, map_b);
    float4 in[8];  // the 32 x 32 block of slope or T: lane's rows 4 it + lane / 8, columns 4 (lane % 8)
    if (MODE != kTrainForward) {
        const float *src = MODE == kTrainLoss ? ep.T : ep.slope;
        const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;  // N is a multiple of 32
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const int r = r0 + it * 4 + (lane >> 3);
            in[it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (mine && r < ep.valid) {
                const float *p = src + (int64_t)r * N + col0 + (lane & 7) * 4;
                in[it] = vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
            }
        }
    }
    const bool ok = tile_product(t, map_a, map_b, blockIdx.x * kTcBM, n0, 0, (K + kTcBK - 1) / kTcBK, status, 0);
    if (ok && mine) {
        float *stg = reinterpret_cast<float *>(t.ring) + warp * (32 * kStgStride);
        uint32_t r[32];
        float v[32];
        load_acc(r, t.tmem, c0);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        if (MODE != kTrainBack) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(ep.bias + col0) + q);
                v[4 * q] += b.x, v[4 * q + 1] += b.y, v[4 * q + 2] += b.z, v[4 * q + 3] += b.w;
            }
        }
        if (MODE == kTrainForward) {
            float slope[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = gelu_slope(v[j], slope[j]);
            stage_f32(stg, slope, lane);
            write_f32(stg, ep.slope, r0, col0, M, N, N, true, false, lane);
        } else {
            float w[32];  // the staged block's row `lane`
#pragma unroll
            for (int it = 0; it < 8; ++it)
                *reinterpret_cast<float4 *>(stg + (it * 4 + (lane >> 3)) * kStgStride + (lane & 7) * 4) = in[it];
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 x = *reinterpret_cast<const float4 *>(stg + lane * kStgStride + 4 * q);
                w[4 * q] = x.x, w[4 * q + 1] = x.y, w[4 * q + 2] = x.z, w[4 * q + 3] = x.w;
            }
            const bool valid = r0 + lane < ep.valid;
            if (MODE == kTrainLoss) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = valid ? v[j] - w[j] : 0.f;
                double sum = sum_squares(v);
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane == 0) ep.loss[(size_t)(r0 >> 5) * (N >> 5) + (col0 >> 5)] = sum;
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 2.f * v[j] * ep.scale;
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = valid ? v[j] * w[j] : 0.f;
            }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __bfloat162float(__float2bfloat16_rn(v[j]));
        write_both(stg, v, r0, col0, ep.out, N, ep.out_t, M, MODE == kTrainForward ? nullptr : ep.colsum, lane);
    }
    release_tile<BN>(t.tmem);
}

// The three weight gradients of a step: 128 x 128 tiles of all of them, K in the parts that each
// product alone would have, each part stored by itself.  One launch, since each alone leaves most
// SMs idle or waits for its own first loads; the parts are added by the kernel that applies them,
// in order, so that neither a zeroed output nor atomics are needed and a step gives the same bits
// every run (with one part or two, those of the product alone).
struct WgradArgs {
    CUtensorMap a[kWgradJobs], b[kWgradJobs];
    int M[kWgradJobs], N[kWgradJobs], splits[kWgradJobs];
    int first[kWgradJobs];  // a job's first block; its tiles follow one another, all of a part together
    float *out[kWgradJobs];
};

constexpr int kWgradStages = 3;  // two CTAs per SM
constexpr int kWgradThreads = 512;

__global__ void __launch_bounds__(kWgradThreads, 2)
tc_wgrad_kernel(const __grid_constant__ WgradArgs args, int K, int *status) {
    extern __shared__ unsigned char smem_raw[];
    int j = 0;
    while (j + 1 < kWgradJobs && (int)blockIdx.x >= args.first[j + 1]) ++j;
    const int M = args.M[j], N = args.N[j];
    const int tiles_n = (N + 127) / 128, tiles = (M + kTcBM - 1) / kTcBM * tiles_n;
    const int at = ((int)blockIdx.x - args.first[j]) % tiles, z = ((int)blockIdx.x - args.first[j]) / tiles;
    const int m0 = at / tiles_n * kTcBM, n0 = at % tiles_n * 128;
    const int KT_all = (K + kTcBK - 1) / kTcBK;
    const int kt0 = (int)((long long)KT_all * z / args.splits[j]);
    const int kt1 = (int)((long long)KT_all * (z + 1) / args.splits[j]);
    const Tile<128, kWgradStages> t = setup_tile<128, kWgradStages>(smem_raw, args.a[j], args.b[j]);
    if (tile_product(t, args.a[j], args.b[j], m0, n0, kt0, kt1 - kt0, status, 0)) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int r0 = m0 + (warp & 3) * 32, col0 = n0 + (warp >> 2) * 32;
        if (r0 < M && col0 < N) {
            float *stg = reinterpret_cast<float *>(t.ring) + warp * (32 * kStgStride);
            uint32_t r[32];
            float v[32];
            load_acc(r, t.tmem, (warp >> 2) * 32);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
            stage_f32(stg, v, lane);
            write_f32(stg, args.out[j] + (size_t)z * M * N, r0, col0, M, N, N, true, false, lane);
        }
    }
    release_tile<128>(t.tmem);
}

// ---- persistent variant (many output tiles, no split K) ----------------------------------
//
// One CTA per SM walks tiles t = blockIdx.x, blockIdx.x + gridDim.x, ... (the two n-tiles of an
// m-block are adjacent, so their A rows are read once from DRAM).  Warp 0 (one lane) streams
// operand stages through the ring across tile boundaries; warp 1 (one lane) issues the MMAs
// into one of two tensor-memory accumulators (tile j uses accumulator j % 2) and commits
// `tfull`; kWarps more drain an accumulator (tcgen05.ld, bias, activation, staged coalesced
// stores), kWarps / 4 to a tensor-memory lane quarter, and release it through `tempty` while the
// next tile's MMAs fill the other one.
//
// Up to some 26 stages of K the epilogue is what bounds it (an activation is some fifty
// instructions per output): sixteen warps; at 50,000 x 512 outputs with gelu, K = 512, four
// epilogue warps took 85 us per product, eight 53, sixteen 46.  Their staging blocks take one
// stage of the 256-wide ring and two of the 128-wide one, which a longer product misses: four
// warps and the longer ring from there on.  65,536 x 512 outputs, bf16, sixteen / four: K = 1536
// 88 / 95 us, K = 2048 112 / 101; 16,384 x 4096: K = 2048 191 / 203, K = 3072 277 / 235.
template <int BN, int kStages, int kWarps>
struct PersSmem {
    static constexpr int A_BYTES = kTcBM * 128;
    static constexpr int B_BYTES = BN * 128;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int STG = kWarps * 32 * kStgStride * 4;  // the epilogue warps' staging blocks
    static constexpr int TOTAL = 1024 + kStages * STAGE + STG + 256;
    static_assert(TOTAL <= 232448, "shared memory of one CTA");
};

__device__ __forceinline__ bool aborted(const int *flag) { return *reinterpret_cast<const volatile int *>(flag) != 0; }

template <int BN, int kStages, int kWarps>
__global__ void __launch_bounds__(64 + 32 * kWarps, 1)
tc_gemm_persistent_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M,
                          int N, int K, const float *__restrict__ bias, int act, void *out, int out_f32, int ldo,
                          float *pre_out, int *status) {
    using S = PersSmem<BN, kStages, kWarps>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    unsigned char *aligned = smem_raw + (base - raw);
    float *stg_all = reinterpret_cast<float *>(aligned + kStages * S::STAGE);
    uint64_t *full = reinterpret_cast<uint64_t *>(aligned + kStages * S::STAGE + S::STG);
    uint64_t *empty = full + kStages;
    uint64_t *tfull = empty + kStages;
    uint64_t *tempty = tfull + 2;
    uint64_t *mma_done = tempty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    int *issued_slot = abort_flag + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (N + BN - 1) / BN;
    const int tiles = ((M + kTcBM - 1) / kTcBM) * tiles_n;
    const int my_tiles = (int)blockIdx.x < tiles ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int KT = (K + kTcBK - 1) / kTcBK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[i])));
        }
        for (int i = 0; i < 2; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tfull[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&tempty[i])),
                         "n"(kWarps));  // one arrival per epilogue warp
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(mma_done)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        *abort_flag = 0;
        *issued_slot = 0;
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {  // TMA producer
            int it = 0;
            for (int j = 0; j < my_tiles && !aborted(abort_flag); ++j) {
                const int t = (int)blockIdx.x + j * (int)gridDim.x;
                const int tm = t / tiles_n, tn = t % tiles_n;
                for (int kk = 0; kk < KT; ++kk, ++it) {
                    const int st = it % kStages;
                    if (it >= kStages && !mbar_wait(smem_u32(&empty[st]), ((it / kStages) - 1) & 1)) {
                        atomicExch(abort_flag, 1);
                        break;
                    }
                    const uint32_t fb = smem_u32(&full[st]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb), "r"(S::STAGE)
                                 : "memory");
                    const uint32_t a_dst = base + st * S::STAGE;
                    tma_load_2d(a_dst, &map_a, kk * kTcBK, tm * kTcBM, fb);
                    tma_load_2d(a_dst + S::A_BYTES, &map_b, kk * kTcBK, tn * BN, fb);
                    *issued_slot = it + 1;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            int it = 0;
            bool ok = true;
            for (int j = 0; j < my_tiles && ok; ++j) {
                const int acc = j & 1;
                if (j >= 2 && !mbar_wait(smem_u32(&tempty[acc]), ((j >> 1) - 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(acc * BN);
                for (int kk = 0; kk < KT; ++kk, ++it) {
                    const int st = it % kStages;
                    if (!mbar_wait(smem_u32(&full[st]), (it / kStages) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a0 = base + st * S::STAGE, b0 = a0 + S::A_BYTES;
#pragma unroll
                    for (int sub = 0; sub < kTcBK / 16; ++sub) {
                        const uint32_t accum = (kk > 0 || sub > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
                            "l"(sw128_desc(a0 + sub * 32)), "l"(sw128_desc(b0 + sub * 32)), "r"(instr_desc<BN>()),
                            "r"(accum));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                                     smem_u32(&empty[st]))
                                 : "memory");
                }
                if (!ok) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                                 smem_u32(&tfull[acc]))
                             : "memory");
            }
            if (!ok) atomicExch(abort_flag, 1);
            // Tracks every MMA issued above: the accumulators may be freed once it completes.
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(mma_done))
                         : "memory");
        }
    } else {  // epilogue warps: tensor-memory lanes 32 (warp % 4).., kCols columns each
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        constexpr int kCols = BN / (kWarps / 4);
        float *stg = stg_all + (warp - 2) * (32 * kStgStride);
        for (int j = 0; j < my_tiles; ++j) {
            const int acc = j & 1;
            const int t = (int)blockIdx.x + j * (int)gridDim.x;
            const int tm = t / tiles_n, tn = t % tiles_n;
            int ok = mbar_wait(smem_u32(&tfull[acc]), (j >> 1) & 1) ? 1 : 0;
            ok = __all_sync(0xffffffffu, ok) && !aborted(abort_flag);
            if (!ok) {
                if (lane == 0) atomicExch(abort_flag, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int r0 = tm * kTcBM + quarter * 32, n0 = tn * BN;
            for (int c0 = part * kCols; c0 < (part + 1) * kCols && n0 + c0 < N; c0 += 32) {
                uint32_t r[32];
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                    "[%32];\n"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                      "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                      "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                epilogue_chunk(stg, r, r0, n0 + c0, M, N, bias, act, out, out_f32, ldo, pre_out, false, lane);
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tempty[acc])) : "memory");
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // Bounded drain: every MMA, then (after an abort) the last copy issued into each stage.
        mbar_wait(smem_u32(mma_done), 0);
        if (aborted(abort_flag)) {
            if (status) atomicExch(status, (int)CUMF_ERR_TIMEOUT);
            const int issued = *issued_slot;
            for (int st = 0; st < kStages && st < issued; ++st) {
                const int last = st + ((issued - 1 - st) / kStages) * kStages;
                mbar_wait(smem_u32(&full[st]), (last / kStages) & 1);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(2 * BN));
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        cudaGetLastError();
    }
    return fn;
}

// rows x K bf16 row-major operand, tiles of box_rows x 64 with 128-byte swizzle.
bool make_map(CUtensorMap *map, const void *ptr, int rows, int K, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

template <int BN, int ST>
cudaError_t launch_variant(dim3 grid, const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K,
                           const float *bias, int act, void *out, int out_f32, int ldo, float *pre_out, int *status,
                           int splits, cudaStream_t s, int no_copies = 0) {
    const int sm = TmaSmem<BN, ST>::TOTAL;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_tma_kernel<BN, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    tc_gemm_tma_kernel<BN, ST><<<grid, kTcThreads, sm, s>>>(ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out,
                                                            status, splits, no_copies);
    return cudaGetLastError();
}

template <int BN, int ST, int EW>
cudaError_t launch_persistent(int grid, const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K,
                              const float *bias, int act, void *out, int out_f32, int ldo, float *pre_out, int *status,
                              cudaStream_t s) {
    const int sm = PersSmem<BN, ST, EW>::TOTAL;
    cudaError_t e =
        cudaFuncSetAttribute(tc_gemm_persistent_kernel<BN, ST, EW>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    tc_gemm_persistent_kernel<BN, ST, EW><<<grid, 64 + 32 * EW, sm, s>>>(ma, mb, M, N, K, bias, act, out, out_f32, ldo,
                                                                     pre_out, status);
    return cudaGetLastError();
}

int sm_count_of_current_device() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return sms;
}

namespace {

constexpr int kShortStages = 16;
constexpr int kEpilogueBoundStages = 26;
constexpr int kWideTrainK = 1024;

struct TilePlan {
    bool wide;
    int splits;
};

TilePlan plan_tiles(int M, int N, int64_t K, bool plain, int nsm) {
    const long long tiles_m = (M + kTcBM - 1) / kTcBM;
    const int64_t kt = (K + kTcBK - 1) / kTcBK;
    // Split K when the output has too few tiles to fill the GPU and K is long (weight
    // gradients): about one wave of CTAs, each with at least 8 stages.
    auto splits_for = [&](long long tiles) -> int {
        if (!plain || kt <= kShortStages || tiles >= nsm) return 1;
        return (int)std::max(1ll, std::min<long long>(kt / 8, nsm / tiles));
    };
    // 128 x 256 tiles (one A tile feeds twice the columns) unless they leave most of a wave
    // idle: 128 x 128 tiles when those give at least 1.5 times the CTAs and the wide ones do not
    // fill the SMs (a batch of 4096 rows has 64 wide tiles; a split is capped by K).
    const long long tw = tiles_m * ((N + 255) / 256), tn = tiles_m * ((N + 127) / 128);
    const long long cw = tw * splits_for(tw), cn = tn * splits_for(tn);
    const bool wide = N > 128 && (cw >= nsm || 2 * cn < 3 * cw);
    return {wide, splits_for(wide ? tw : tn)};
}

}  // namespace

cudaError_t launch_tc_gemm(const void *A, const void *B, int M, int N, int K, const float *bias, int act,
                           void *out, int out_f32, int ldo, float *pre_out, int *status, cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % 8) != 0) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return cudaErrorInvalidValue;
    const int sms = sm_count_of_current_device();
    const int tiles_m = (M + kTcBM - 1) / kTcBM;
    const int kt = (K + kTcBK - 1) / kTcBK;
    // Short K (at most 16 stages of 64): a 2-stage ring, so two CTAs share an SM and
    // one CTA's epilogue overlaps another's loads.  Long K: a 4-stage ring, one CTA per SM.
    const bool short_k = kt <= kShortStages;
    const bool plain = out_f32 && !bias && act == 0 && !pre_out;
    const TilePlan plan = plan_tiles(M, N, K, plain, sms > 0 ? sms : 152);
    const bool wide = plan.wide;
    const int BN = wide ? 256 : 128;
    CUtensorMap ma, mb;
    if (!make_map(&ma, A, M, K, kTcBM) || !make_map(&mb, B, N, K, BN)) return cudaErrorInvalidValue;
    const int tiles_n = (N + BN - 1) / BN;
    const int splits = plan.splits;
    if (splits > 1) {
        cudaError_t e = cudaMemset2DAsync(out, (size_t)ldo * 4, 0, (size_t)N * 4, M, s);
        if (e != cudaSuccess) return e;
    }
    // Enough output tiles for two per SM: the persistent kernel, whose epilogues overlap the
    // next tiles' loads and MMAs.
    if (splits == 1 && sms > 0 && (long long)tiles_m * tiles_n >= 2ll * sms) {
        const int g = std::min(tiles_m * tiles_n, sms);
        // (see the kernel: what a tile's epilogue takes, its product has to cover)
        if (kt <= kEpilogueBoundStages)
            return wide ? launch_persistent<256, 3, 16>(g, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status, s)
                        : launch_persistent<128, 4, 16>(g, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status, s);
        return wide ? launch_persistent<256, 4, 4>(g, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status, s)
                    : launch_persistent<128, 6, 4>(g, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status, s);
    }
    const dim3 grid(tiles_m, tiles_n, splits);
    if (wide)
        return short_k ? launch_variant<256, 2>(grid, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status,
                                                splits, s)
                       : launch_variant<256, 4>(grid, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status,
                                                splits, s);
    return short_k ? launch_variant<128, 2>(grid, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status,
                                            splits, s)
                   : launch_variant<128, 4>(grid, ma, mb, M, N, K, bias, act, out, out_f32, ldo, pre_out, status,
                                            splits, s);
}

namespace {

template <int BN, int ST, int MODE>
cudaError_t launch_train(const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K, const TrainEpilogue &ep,
                         int *status, cudaStream_t s) {
    const int sm = TmaSmem<BN, ST>::TOTAL;
    cudaError_t e = cudaFuncSetAttribute(tc_train_kernel<BN, ST, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    tc_train_kernel<BN, ST, MODE><<<dim3(M / kTcBM, (N + BN - 1) / BN), 4 * BN, sm, s>>>(ma, mb, M, N, K, ep, status);
    return cudaGetLastError();
}

template <int BN, int ST>
cudaError_t launch_train_mode(TrainMode mode, const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K,
                              const TrainEpilogue &ep, int *status, cudaStream_t s) {
    switch (mode) {
        case kTrainForward: return launch_train<BN, ST, kTrainForward>(ma, mb, M, N, K, ep, status, s);
        case kTrainLoss: return launch_train<BN, ST, kTrainLoss>(ma, mb, M, N, K, ep, status, s);
        default: return launch_train<BN, ST, kTrainBack>(ma, mb, M, N, K, ep, status, s);
    }
}

}  // namespace

cudaError_t launch_train_gemm(TrainMode mode, const void *A, const void *B, int M, int N, int K,
                              const TrainEpilogue &ep, int *status, cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0 || M % kTcBM || N % 32 || K % 8) return cudaErrorInvalidValue;
    const int sms = sm_count_of_current_device();
    const int nsm = sms > 0 ? sms : 152;
    // One wave of 128-wide tiles that fill at least half of the SMs: one CTA of 16 warps per SM.
    // Otherwise narrower tiles, two CTAs per SM: for a large batch a CTA's epilogue overlaps the
    // other's product; for a small one, or a narrow layer, they are on more SMs.  From K = 1024 on
    // a large batch is bound by its operands, which wide tiles read half as often: layers of 2048,
    // 65,536 rows, loss and gradients 4.33 -> 3.35 ms (K = 512, layers of 512: no difference).
    const long long tm = M / kTcBM, t128 = tm * ((N + 127) / 128), t64 = tm * ((N + 63) / 64);
    const bool one_wave = t128 <= nsm && 2 * t128 >= nsm, long_k = t128 > nsm && K >= kWideTrainK;
    const int BN = N > 64 && (one_wave || long_k) ? 128 : 2 * t64 >= nsm ? 64 : 32;
    CUtensorMap ma, mb;
    if (!make_map(&ma, A, M, K, kTcBM) || !make_map(&mb, B, N, K, BN)) return cudaErrorInvalidValue;
    return BN == 128  ? launch_train_mode<128, 6>(mode, ma, mb, M, N, K, ep, status, s)
           : BN == 64 ? launch_train_mode<64, 4>(mode, ma, mb, M, N, K, ep, status, s)
                      : launch_train_mode<32, 4>(mode, ma, mb, M, N, K, ep, status, s);
}

int product_splits(int M, int N, int64_t K) {
    const int sms = sm_count_of_current_device();
    return plan_tiles(M, N, K, true, sms > 0 ? sms : 152).splits;
}

int product_splits_limit(int M, int N, int64_t K) {
    const int sms = sm_count_of_current_device();
    const long long fewest = (long long)((M + kTcBM - 1) / kTcBM) * ((N + 255) / 256);
    return (int)std::max<long long>(1, std::min<long long>(K / kTcBK / 8, (sms > 0 ? sms : 152) / fewest));
}

cudaError_t launch_wgrad(const WgradJob *job, int K, int *status, cudaStream_t s) {
    WgradArgs args;
    int blocks = 0;
    for (int j = 0; j < kWgradJobs; ++j) {
        if (!make_map(&args.a[j], job[j].A, job[j].M, K, kTcBM) || !make_map(&args.b[j], job[j].B, job[j].N, K, 128))
            return cudaErrorInvalidValue;
        args.M[j] = job[j].M;
        args.N[j] = job[j].N;
        args.splits[j] = job[j].splits;
        args.out[j] = job[j].out;
        args.first[j] = blocks;
        blocks += (job[j].M + 127) / 128 * ((job[j].N + 127) / 128) * job[j].splits;
    }
    const int sm = TmaSmem<128, kWgradStages>::TOTAL;
    cudaError_t e = cudaFuncSetAttribute(tc_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    tc_wgrad_kernel<<<blocks, kWgradThreads, sm, s>>>(args, K, status);
    return cudaGetLastError();
}

}  // namespace cumf

using namespace cumf;

extern "C" int cumf_tc_gemm(const void *d_A, const void *d_B, int M, int N, int K, const float *d_bias, int act,
                            void *d_out, int out_f32, int ldo, float *d_pre, int *d_status, void *stream) {
    if (!d_A || !d_B || !d_out || M <= 0 || N <= 0 || K <= 0 || (K % 8) != 0 || ldo < N)
        return fail(CUMF_ERR_ARG, "tc_gemm: bad arguments (K must be a multiple of 8, ldo >= N)");
    if (act != 0 && act != 1) return fail(CUMF_ERR_ARG, "tc_gemm: act must be 0 (identity) or 1 (gelu)");
    CUMF_CUDA(launch_tc_gemm(d_A, d_B, M, N, K, d_bias, act, d_out, out_f32, ldo, d_pre, d_status,
                             (cudaStream_t)stream));
    return CUMF_OK;
}

extern "C" int cumf_selftest_wait_timeout(int *status_out, double *seconds) {
    if (!status_out) return fail(CUMF_ERR_ARG, "selftest: status_out is NULL");
    *status_out = 0;
    // One 128 x 128 x 64 tile whose producer issues no copies: the MMA thread's wait on the
    // stage barrier runs out, the kernel records CUMF_ERR_TIMEOUT, drains and frees its tensor
    // memory; then an ordinary product on the same context must still be right.
    const int M = 128, N = 128, K = 64;
    void *buf = nullptr;
    const size_t ab = (size_t)M * K * 2, bb = (size_t)N * K * 2, ob = (size_t)M * N * 4;
    CUMF_CUDA(cudaMalloc(&buf, ab + bb + ob + 16));
    char *A = static_cast<char *>(buf);
    char *B = A + ab;
    float *O = reinterpret_cast<float *>(B + bb);
    int *st = reinterpret_cast<int *>(reinterpret_cast<char *>(O) + ob);
    int rc = CUMF_OK;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    do {
        cudaError_t e = cudaMemset(buf, 0, ab + bb + ob + 16);
        if (e == cudaSuccess) {  // A = B = bf16 1.0: every output element is K
            std::vector<uint16_t> ones((M > N ? M : N) * K, 0x3f80);
            e = cudaMemcpy(A, ones.data(), ab, cudaMemcpyHostToDevice);
            if (e == cudaSuccess) e = cudaMemcpy(B, ones.data(), bb, cudaMemcpyHostToDevice);
        }
        CUtensorMap ma, mb;
        if (e == cudaSuccess && (!make_map(&ma, A, M, K, kTcBM) || !make_map(&mb, B, N, K, 128))) {
            rc = fail(CUMF_ERR_CUDA, "selftest: tensor maps");
            break;
        }
        if (e == cudaSuccess) e = cudaEventCreate(&e0);
        if (e == cudaSuccess) e = cudaEventCreate(&e1);
        if (e == cudaSuccess) e = cudaEventRecord(e0, 0);
        if (e == cudaSuccess)
            e = launch_variant<128, 2>(dim3(1, 1, 1), ma, mb, M, N, K, nullptr, 0, O, 1, N, nullptr, st, 1, 0, 1);
        if (e == cudaSuccess) e = cudaEventRecord(e1, 0);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        float ms = 0;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
        if (e == cudaSuccess) e = cudaMemcpy(status_out, st, sizeof(int), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            rc = cuda_fail(e, "selftest: timed-out launch");
            break;
        }
        if (seconds) *seconds = ms * 1e-3;
        // The context is usable: an ordinary product gives K everywhere.
        e = launch_tc_gemm(A, B, M, N, K, nullptr, 0, O, 1, N, nullptr, nullptr, 0);
        std::vector<float> host((size_t)M * N, 0.f);
        if (e == cudaSuccess) e = cudaMemcpy(host.data(), O, ob, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            rc = cuda_fail(e, "selftest: product after the timeout");
            break;
        }
        for (float v : host)
            if (v != (float)K) {
                rc = fail(CUMF_ERR_CUDA, "selftest: product after the timeout is wrong");
                break;
            }
    } while (0);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(buf);
    return rc;
}
