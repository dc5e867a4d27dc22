// Kernels of the noise-surrogate MLP ensemble (no reference counterpart).
//
// The network maps noise parameters to a fixed circuit's outcome
// distribution.  Its matrix products run on the tensor cores: a CTA computes a
// 128 x 32 or 128 x 64 tile of C = A B^T with BF16 operands (kind::f16, FP32
// accumulation in TMEM).  K is streamed in 64-wide chunks by TMA into 2 to 4
// shared-memory stages (128-byte rows, 128-byte swizzle, K-major): one thread
// keeps the loads going, another issues the four K = 16 MMAs of a chunk as it
// lands and commits them to the barrier that frees the stage.  The epilogue
// runs on 8 or 16 warps (32 rows of a quadrant each, tcgen05.ld), applies bias and
// GELU, or the GELU derivative of the backward pass, and goes through shared
// memory so that global accesses are whole rows; it writes the row-major result
// plus, where the next product needs it, its transpose, so that every later
// product is again of the A B^T form with K contiguous.  Several independent
// products of one epilogue can share a launch.  A training step's products are
// small, 2.7 GFLOP at most (a prediction's output layer has 27), and bound by
// latencies: of a chunk's load, multiply and wait, and of the epilogue's chains.
// With 4 warps per CTA (64 columns and 64 tanhf a thread), 16-byte cp.async
// loads and a wait per chunk the ten products of a training step of 5 x 1,024
// rows, 1,024 outcomes took 260 us; with TMA, stages and the work spread over
// more warps the eight launches take 97 us (11 us for 1,024 x 256 x 256, 13 us
// for 1,024 x 1,024 x 256).  The whole step went from 405 to 132 us, the
// prediction of 10,233 points with the ensemble's spread from 1,640 to 283 us.
// Waits on an mbarrier are bounded and record an error in *status.
//
// The other kernels are memory-light helpers: softmax with the KL loss and
// its gradient, bias gradients, Adam with the BF16 weight copies, the
// minibatch gather and the ensemble statistics.
#include <cuda.h>
#include <cuda_bf16.h>

#include <mutex>

#include "dm_common.cuh"
#include "dm_tcgen05.cuh"

namespace dmg {
namespace mlp {

constexpr int kBM = 128, kBK = 64;
constexpr uint32_t kABytes = kBM * kBK * 2;        // 16 KB
// Tile width, threads, stages and CTAs per SM of a launch.  Tiles beyond two per SM: four CTAs per SM, one's
// loads and MMAs beside the others' epilogues (3,456 x 1,024 x 256 for 5 members: 35 us with two of 512
// threads per SM, 27 us).  Fewer: half the tile's columns, twice the CTAs (1,024 x 256 x 256: 13.3 us with 64
// columns, 11.0 us; the GELU derivative's 1,024 x 256 x 1,024: 17.1 and 15.7 us), unless K is long and the
// epilogue only stores (the weight gradients, K = 1,024: 17.7 us with 32 columns, 11.0 us with 64).
template <int BN, int T, int S, int P>
struct Shape {
    static constexpr int kBN = BN, kThreads = T, kStages = S, kPerSm = P;
    static constexpr uint32_t kStage = kABytes + BN * kBK * 2;
    static constexpr uint32_t kSmemBytes = S * kStage + 1024;        // with alignment slack
    // kind::f16: D = F32 (bits 4-5 = 1), A = B = BF16 (bits 7-9 and 10-12 = 1), K-major, N = BN, M = 128.
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t(BN) >> 3) << 17) |
                                       ((uint32_t(kBM) >> 4) << 24);
};
using Small = Shape<32, 256, 3, 3>;      // 61 KB
using Wide = Shape<64, 256, 2, 4>;       // 49 KB
using Deep = Shape<64, 512, 4, 2>;       // 97 KB
constexpr int kLongK = 512;
constexpr int kMaxGroup = 4;                       // products per launch

constexpr float kGeluC = 0.7978845608028654f;   // sqrt(2 / pi)
constexpr float kGeluA = 0.044715f;

__device__ __forceinline__ float gelu(float u) {
    return 0.5f * u * (1.0f + tanhf(kGeluC * fmaf(kGeluA * u * u, u, u)));
}

__device__ __forceinline__ float gelu_grad(float u) {
    const float t = tanhf(kGeluC * fmaf(kGeluA * u * u, u, u));
    return 0.5f * (1.0f + t) + 0.5f * u * (1.0f - t * t) * kGeluC * fmaf(3.0f * kGeluA, u * u, 1.0f);
}

__device__ __forceinline__ uint16_t to_bf16(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float from_bf16(uint16_t b) { return __uint_as_float(uint32_t(b) << 16); }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    return uint32_t(to_bf16(a)) | (uint32_t(to_bf16(b)) << 16);
}

struct GemmGroup {
    int count;
    int first[kMaxGroup + 1];                      // tiles before product i
    dm_mlp_gemm g[kMaxGroup];
    CUtensorMap a[kMaxGroup], b[kMaxGroup];        // K x rows x members, boxes of 64 x 128 (A) and 64 x kBN (B)
};

// K-major operand of 128-byte rows with the 128-byte swizzle: 8 rows are 1024 bytes (the stride
// offset), layout type 2; a K step of 16 values is 32 bytes further in the start address.
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t saddr) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}

__device__ __forceinline__ void tma_load(const CUtensorMap *map, int k, int row, int member, uint32_t dst, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
                 "[%5];" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(k), "r"(row), "r"(member), "r"(bar)
                 : "memory");
}

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

template <int EPI, typename Sh>
__global__ void __launch_bounds__(Sh::kThreads, Sh::kPerSm) gemm_kernel(const __grid_constant__ GemmGroup G, int *status) {
    constexpr int kThreads = Sh::kThreads, kStages = Sh::kStages, kBN = Sh::kBN;
    constexpr uint32_t kStage = Sh::kStage, kTmemCols = kBN;
    constexpr int kCols = kBM * kBN / kThreads;       // columns of a thread in the epilogue
    constexpr int kF32Row = kBN + 4;                  // epilogue rows in shared memory: FP32 values,
    constexpr int kBf16Row = kBN + 8;                 // BF16 values (16-byte accesses of 8 rows hit all banks)
    constexpr int kF4 = kBN / 4, kH8 = kBN / 8;       // 16-byte pieces of such a row
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;
    __shared__ float bias_s[kBN];
    unsigned char *smem = smem_raw + ((1024 - (tcg::smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int gi = 0;
    while (gi + 1 < G.count && int(blockIdx.x) >= G.first[gi + 1]) ++gi;
    const dm_mlp_gemm &g = G.g[gi];
    const int tile = int(blockIdx.x) - G.first[gi], mtiles = g.M / kBM;
    const int m0 = tile % mtiles * kBM, n0 = tile / mtiles * kBN;
    const int64_t z = blockIdx.y;
    const int nch = g.K / kBK;

    if (tid == 0) {
        abort_s = 0;
        for (int i = 0; i < kStages; ++i) {
            tcg::mbar_init(tcg::smem_u32(&full[i]), 1);
            tcg::mbar_init(tcg::smem_u32(&empty[i]), 1);
        }
        tcg::mbar_init(tcg::smem_u32(&done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         tcg::smem_u32(&tmem_base_s)),
                     "n"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    grid_wait();
    if constexpr (EPI == DM_MLP_EPI_GELU_FWD || EPI == DM_MLP_EPI_BIAS_F32)
        if (tid >= 64 && tid < 64 + kBN) bias_s[tid - 64] = waited(g.bias)[z * g.bias_ms + n0 + tid - 64];

    // A thread whose wait gives up flags the abort and stops; the others' waits then run out in turn.
    auto wait_for = [&](uint64_t &bar, uint32_t parity) {
        if (tcg::mbar_wait(tcg::smem_u32(&bar), parity)) return true;
        atomicExch(status, 1);
        *static_cast<volatile int *>(&abort_s) = 1;
        return false;
    };
    int issued = 0;
    if (tid == 0) {                    // the loads
        int c = 0;
        for (; c < nch; ++c) {
            const int st = c % kStages;
            if (c >= kStages && !wait_for(empty[st], uint32_t(c / kStages - 1) & 1)) break;
            const uint32_t bar = tcg::smem_u32(&full[st]), dst = tcg::smem_u32(smem + st * kStage);
            tcg::mbar_expect_tx(bar, kStage);
            tma_load(&G.a[gi], c * kBK, m0, g.a_ms ? int(z) : 0, dst, bar);
            tma_load(&G.b[gi], c * kBK, n0, g.b_ms ? int(z) : 0, dst + kABytes, bar);
        }
        issued = c;
    } else if (tid == 32) {            // the MMAs
        int c = 0;
        for (; c < nch; ++c) {
            const int st = c % kStages;
            if (!wait_for(full[st], uint32_t(c / kStages) & 1)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = tcg::smem_u32(smem + st * kStage);
            const uint64_t da = swizzled_desc(a), db = swizzled_desc(a + kABytes);
#pragma unroll
            for (int ks = 0; ks < kBK / 16; ++ks) {
                const uint32_t acc = (c | ks) ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(da + uint64_t(2 * ks)), "l"(db + uint64_t(2 * ks)), "r"(Sh::kIdesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                tcg::smem_u32(&empty[st])));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            tcg::smem_u32(&done)));
    }
    __syncwarp();
    // the backward pass's pre-activations arrive while the products run (where registers hold them)
    constexpr int kPre = kBM * kF4 / kThreads;
    constexpr bool early = EPI == DM_MLP_EPI_GELU_BWD && kPre <= 4;
    auto load_pre = [&](int q) {
        const int i = tid + q * kThreads;
        return *reinterpret_cast<const float4 *>(g.pre + z * g.pre_ms + int64_t(m0 + i / kF4) * g.ld_pre + n0 +
                                                 4 * (i % kF4));
    };
    float4 pre[early ? kPre : 1];
    if constexpr (early) {
#pragma unroll
        for (int q = 0; q < kPre; ++q) pre[q] = load_pre(q);
    }
    wait_for(done, 0);
    if (tid == 0 && *static_cast<volatile int *>(&abort_s))   // loads in flight are drained before the CTA ends
        for (int i = issued > kStages ? issued - kStages : 0; i < issued; ++i)
            tcg::mbar_wait(tcg::smem_u32(&full[i % kStages]), uint32_t(i / kStages) & 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();

    if (!*static_cast<volatile int *>(&abort_s)) {
        // the thread's row and columns
        const int row = 32 * (warp & 3) + lane, c0 = kCols * (warp >> 2);
        float v[kCols];
#pragma unroll
        for (int j = 0; j < kCols; j += 16) {
            float part[16];
            tmem_ld16(tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(c0 + j), part);
#pragma unroll
            for (int e = 0; e < 16; ++e) v[j + e] = part[e];
        }
        float *st = reinterpret_cast<float *>(smem);             // the tile in FP32 rows, then in BF16 rows
        if constexpr (EPI == DM_MLP_EPI_GELU_FWD || EPI == DM_MLP_EPI_BIAS_F32) {
#pragma unroll
            for (int j = 0; j < kCols; ++j) v[j] += bias_s[c0 + j];
        }
        if constexpr (EPI == DM_MLP_EPI_GELU_FWD || EPI == DM_MLP_EPI_BIAS_F32 || EPI == DM_MLP_EPI_F32) {
            if (g.out_f32) {
#pragma unroll
                for (int j = 0; j < kCols; j += 4)
                    *reinterpret_cast<float4 *>(st + row * kF32Row + c0 + j) =
                        make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                __syncthreads();
                float *o = g.out_f32 + z * g.f32_ms + int64_t(m0) * g.ld_f32 + n0;
#pragma unroll
                for (int i = tid; i < kBM * kF4; i += kThreads)
                    *reinterpret_cast<float4 *>(o + int64_t(i / kF4) * g.ld_f32 + 4 * (i % kF4)) =
                        *reinterpret_cast<const float4 *>(st + (i / kF4) * kF32Row + 4 * (i % kF4));
            }
        }
        if constexpr (EPI == DM_MLP_EPI_GELU_FWD) {
#pragma unroll
            for (int j = 0; j < kCols; ++j) v[j] = gelu(v[j]);
        }
        if constexpr (EPI == DM_MLP_EPI_GELU_BWD) {
#pragma unroll
            for (int q = 0; q < kPre; ++q) {
                const int i = tid + q * kThreads;
                *reinterpret_cast<float4 *>(st + (i / kF4) * kF32Row + 4 * (i % kF4)) =
                    early ? pre[early ? q : 0] : load_pre(q);
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kCols; j += 4) {
                const float4 u = *reinterpret_cast<const float4 *>(st + row * kF32Row + c0 + j);
                v[j] *= gelu_grad(u.x);
                v[j + 1] *= gelu_grad(u.y);
                v[j + 2] *= gelu_grad(u.z);
                v[j + 3] *= gelu_grad(u.w);
            }
        }
        if constexpr (EPI == DM_MLP_EPI_GELU_FWD || EPI == DM_MLP_EPI_GELU_BWD) {
            // behind the FP32 rows, or in their place
            constexpr bool apart = kStages * kStage >= kBM * (kF32Row * 4 + kBf16Row * 2);
            uint16_t *sb = reinterpret_cast<uint16_t *>(smem + (apart ? kBM * kF32Row * 4 : 0));
            if (!apart && (EPI == DM_MLP_EPI_GELU_BWD || g.out_f32)) __syncthreads();
#pragma unroll
            for (int j = 0; j < kCols; j += 8)
                *reinterpret_cast<uint4 *>(sb + row * kBf16Row + c0 + j) =
                    make_uint4(pack2(v[j], v[j + 1]), pack2(v[j + 2], v[j + 3]), pack2(v[j + 4], v[j + 5]),
                               pack2(v[j + 6], v[j + 7]));
            __syncthreads();
            if (g.out_bf16) {
                uint16_t *o = g.out_bf16 + z * g.bf16_ms + int64_t(m0) * g.ld_bf16 + n0;
#pragma unroll
                for (int i = tid; i < kBM * kH8; i += kThreads)
                    *reinterpret_cast<uint4 *>(o + int64_t(i / kH8) * g.ld_bf16 + 8 * (i % kH8)) =
                        *reinterpret_cast<const uint4 *>(sb + (i / kH8) * kBf16Row + 8 * (i % kH8));
            }
            if (g.out_t) {       // column j of the tile: 256 contiguous bytes of 128 rows
                uint16_t *o = g.out_t + z * g.t_ms + int64_t(n0) * g.ld_t + m0;
                if ((reinterpret_cast<uintptr_t>(o) & 15) == 0 && (g.ld_t & 7) == 0) {
#pragma unroll
                    for (int i = tid; i < kBN * 16; i += kThreads) {
                        const int j = i >> 4, r = 8 * (i & 15);
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = uint32_t(sb[(r + 2 * e) * kBf16Row + j]) |
                                   (uint32_t(sb[(r + 2 * e + 1) * kBf16Row + j]) << 16);
                        *reinterpret_cast<uint4 *>(o + int64_t(j) * g.ld_t + r) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                } else {         // a warp writes 32 consecutive rows
                    for (int j = 0; j < kCols; ++j)
                        o[int64_t(c0 + j) * g.ld_t + row] = sb[row * kBf16Row + c0 + j];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols));
}

// ---------------------------------------------------------------------------
// softmax, KL loss and its gradient: one warp per row, 16 rows per CTA, so that
// the transposed gradient leaves in whole sectors (two-byte stores of one row
// per CTA cost a sector each): 52 -> 26 us for 5 x 1,024 rows of 1,024 columns,
// 79 MB.  Up to 1,024 columns a lane holds its 32 logits,
// all loads in flight together; wider rows are read again.  The sums run in the
// order of 256 threads with one value of every 256 each: per lane and 32-column
// slice w first, then over the lanes, then over the slices.
// ---------------------------------------------------------------------------

constexpr int kRowThreads = 256;
constexpr int kSoftRows = 16, kSoftSlices = kRowThreads / 32;
constexpr int kSoftStride = kSoftRows + 2;        // halves per column of the transpose tile

__device__ __forceinline__ float slice_sum(const float (&part)[kSoftSlices]) {
    float r = 0.f;
#pragma unroll
    for (int w = 0; w < kSoftSlices; ++w) {
        float x = part[w];
        for (int o = 16; o > 0; o >>= 1) x = x + __shfl_xor_sync(0xffffffffu, x, o);
        r = w == 0 ? x : r + x;
    }
    return r;
}

// Per: nout / 256 where the row is held in registers, 0 otherwise.
template <int Per>
__global__ void __launch_bounds__(32 * kSoftRows, 2)
    softmax_kernel(const float *__restrict__ logits, const float *__restrict__ targets,
                   const int32_t *__restrict__ index, int64_t samples, int rows, int nout, int64_t row_ms,
                   int64_t out_ms, int64_t ld_t, float grad_scale, float *__restrict__ probs, uint16_t *__restrict__ dz,
                   uint16_t *__restrict__ dzt, float *__restrict__ loss_rows) {
    __shared__ __align__(4) uint16_t tr[kRowThreads * kSoftStride];
    const int lane = threadIdx.x & 31, rl = threadIdx.x >> 5;
    const int64_t r0 = int64_t(blockIdx.x) * kSoftRows, r = r0 + rl, z = blockIdx.y;
    const bool live = r < rows;
    const int per = Per ? Per : nout / kRowThreads;
    const int64_t base = (z * row_ms + (live ? r : r0)) * nout;
    grid_wait();
    const float *row = waited(logits) + base;
    targets = waited(targets);
    // the row's targets: its own, or sample index[z * row_ms + r] of a data set (0 outside it)
    int64_t tbase = base;
    if (index) {
        const int64_t smp = waited(index)[z * row_ms + (live ? r : r0)];
        tbase = (smp < 0 || smp >= samples ? 0 : smp) * nout;
    }
    float held[Per ? Per * kSoftSlices : 1] = {};
    if constexpr (Per > 0) {
#pragma unroll
        for (int k = 0; k < Per * kSoftSlices; ++k) held[k] = row[32 * k + lane];
    }
    auto x = [&](int i, int w) { return Per ? held[Per ? i * kSoftSlices + w : 0] : row[i * kRowThreads + 32 * w + lane]; };
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < per; ++i)
#pragma unroll
        for (int w = 0; w < kSoftSlices; ++w) mx = fmaxf(mx, x(i, w));
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float part[kSoftSlices];
#pragma unroll
    for (int w = 0; w < kSoftSlices; ++w) part[w] = 0.f;
#pragma unroll
    for (int i = 0; i < per; ++i)
#pragma unroll
        for (int w = 0; w < kSoftSlices; ++w) part[w] += expf(x(i, w) - mx);
    const float lse = logf(slice_sum(part));
#pragma unroll
    for (int w = 0; w < kSoftSlices; ++w) part[w] = 0.f;
    float *pr = probs ? probs + (z * out_ms + (live ? r : r0)) * nout : nullptr;
    const bool vec = (ld_t & 7) == 0 && r0 + kSoftRows <= rows && (reinterpret_cast<uintptr_t>(dzt) & 15) == 0;
#pragma unroll
    for (int i = 0; i < per; ++i) {
        float t[kSoftSlices];
#pragma unroll
        for (int w = 0; w < kSoftSlices; ++w) t[w] = targets ? targets[tbase + i * kRowThreads + 32 * w + lane] : 0.f;
#pragma unroll
        for (int w = 0; w < kSoftSlices; ++w) {
            const int c = 32 * w + lane, j = i * kRowThreads + c;
            const float lq = x(i, w) - mx - lse;
            const float q = expf(lq);
            if (pr && live) pr[j] = q;
            if (targets) {
                if (t[w] > 0.f) part[w] += t[w] * (logf(t[w]) - lq);
                const uint16_t d = to_bf16((q - t[w]) * grad_scale);
                if (live) dz[base + j] = d;
                tr[c * kSoftStride + rl] = d;
            }
        }
        if (targets) {           // columns 256 i .. 256 i + 255 of the transpose, 8 rows per thread
            __syncthreads();
            const int c = threadIdx.x >> 1, rr = 8 * (threadIdx.x & 1);
            uint16_t *o = dzt + (z * nout + int64_t(i) * kRowThreads + c) * ld_t + r0 + rr;
            const uint16_t *src = tr + c * kSoftStride + rr;
            if (vec) {
                const uint32_t *s32 = reinterpret_cast<const uint32_t *>(src);
                *reinterpret_cast<uint4 *>(o) = make_uint4(s32[0], s32[1], s32[2], s32[3]);
            } else {
                for (int e = 0; e < 8; ++e)
                    if (r0 + rr + e < rows) o[e] = src[e];
            }
            __syncthreads();
        }
    }
    if (targets && loss_rows) {
        const float loss = slice_sum(part);
        if (live && lane == 0) loss_rows[z * row_ms + r] = loss;
    }
}

static int launch_softmax(const float *logits, const float *targets, const int32_t *index, int64_t samples, int rows,
                          int members, int nout, int64_t row_ms, int64_t out_ms, int64_t ld_t, float grad_scale,
                          float *probs, uint16_t *dz, uint16_t *dzt, float *loss_rows, cudaStream_t s) {
    const dim3 grid((rows + kSoftRows - 1) / kSoftRows, members), block(32 * kSoftRows);
    auto kernel = nout == 256 ? softmax_kernel<1>
                : nout == 512 ? softmax_kernel<2>
                : nout == 768 ? softmax_kernel<3>
                : nout == 1024 ? softmax_kernel<4> : softmax_kernel<0>;
    return launch_early(kernel, grid, block, 0, s, logits, targets, index, samples, rows, nout, row_ms, out_ms, ld_t,
                        grad_scale, probs, dz, dzt, loss_rows);
}

// db[n] = sum_b d_t[n][b] for up to four layers: one warp per (layer, n, member)
struct BiasGrads {
    int count, rows;
    int64_t ld, db_ms;
    int first[kMaxGroup + 1];                      // rows n before layer i
    const uint16_t *dt[kMaxGroup];
    int64_t d_ms[kMaxGroup];
    float *db[kMaxGroup];
};

__global__ void bias_grad_kernel(const __grid_constant__ BiasGrads B) {
    const int lane = threadIdx.x & 31;
    int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    grid_wait();
    if (n >= B.first[B.count]) return;
    int i = 0;
    while (n >= B.first[i + 1]) ++i;
    n -= B.first[i];
    const int64_t z = blockIdx.y;
    const uint16_t *src = B.dt[i] + z * B.d_ms[i] + int64_t(n) * B.ld;
    float s = 0.f;
#pragma unroll 8
    for (int b = lane; b < B.rows; b += 32) s += from_bf16(src[b]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) B.db[i][z * B.db_ms + n] = s;
}

static int launch_bias_grads(const BiasGrads &B, int members, cudaStream_t s) {
    const int warps = 8;
    return launch_early(bias_grad_kernel, dim3((B.first[B.count] + warps - 1) / warps, members), dim3(32 * warps), 0, s, B);
}

struct Layers {
    int n;
    int64_t w_off[8], b_off[8];
    int out[8], in[8];
    int tiles[9];                     // 32 x 32 weight tiles before layer l; then all of them
    int bias_blocks[9];               // blocks of 256 biases before layer l
};

// One block per 32 x 32 tile of a weight matrix, so that the transposed BF16 copy leaves in rows too
// (element by element it cost a sector per value), then blocks of biases.  Vec: four
// weights per thread at once, where every row of every matrix is 16-byte aligned (2 M parameters, 66 MB: 25 -> 12.6 us).
template <bool Vec>
__global__ void __launch_bounds__(256) adam_kernel(float *__restrict__ params, const float *__restrict__ grads,
                                                   float *__restrict__ m, float *__restrict__ v, int64_t P,
                                                   const __grid_constant__ Layers L, float lr, float b1, float b2,
                                                   float eps, float c1, float c2, int step, int members,
                                                   uint16_t *__restrict__ wb, uint16_t *__restrict__ wtb) {
    __shared__ uint16_t tr[32][33];
    grid_wait();
    params = waited(params);      // restrict alone allows loads above the wait: an earlier step's are in it
    grads = waited(grads);
    m = waited(m);
    v = waited(v);
    auto rule = [&](float p, float gr, float &mm, float &vv) {
        mm = b1 * mm + (1.f - b1) * gr;
        vv = b2 * vv + (1.f - b2) * gr * gr;
        return p - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    };
    auto update = [&](int64_t i) {
        float p = params[i];
        if (step > 0) {
            float mm = m[i], vv = v[i];
            p = rule(p, grads[i], mm, vv);
            m[i] = mm;
            v[i] = vv;
            params[i] = p;
        }
        return p;
    };
    int b = blockIdx.x, l = 0;
    if (b >= L.tiles[L.n]) {          // biases (no BF16 copies)
        b -= L.tiles[L.n];
        while (b >= L.bias_blocks[l + 1]) ++l;
        const int i = (b - L.bias_blocks[l]) * 256 + threadIdx.x;
        for (int64_t z = blockIdx.y; z < members; z += gridDim.y)
            if (i < L.out[l]) update(z * P + L.b_off[l] + i);
        return;
    }
    while (b >= L.tiles[l + 1]) ++l;
    const int out = L.out[l], in = L.in[l], across = (in + 31) / 32;
    const int t = b - L.tiles[l], r0 = t / across * 32, c0 = t % across * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int64_t z = blockIdx.y; z < members; z += gridDim.y) {
        const int64_t w0 = z * P + L.w_off[l];
        if constexpr (Vec) {
            const int rr = threadIdx.x >> 3, cc = 4 * (threadIdx.x & 7);
            if (r0 + rr < out && c0 + cc < in) {
                const int64_t i = w0 + int64_t(r0 + rr) * in + c0 + cc;
                float4 p = *reinterpret_cast<const float4 *>(params + i);
                if (step > 0) {
                    const float4 gr = *reinterpret_cast<const float4 *>(grads + i);
                    float4 mm = *reinterpret_cast<const float4 *>(m + i), vv = *reinterpret_cast<const float4 *>(v + i);
                    p.x = rule(p.x, gr.x, mm.x, vv.x);
                    p.y = rule(p.y, gr.y, mm.y, vv.y);
                    p.z = rule(p.z, gr.z, mm.z, vv.z);
                    p.w = rule(p.w, gr.w, mm.w, vv.w);
                    *reinterpret_cast<float4 *>(m + i) = mm;
                    *reinterpret_cast<float4 *>(v + i) = vv;
                    *reinterpret_cast<float4 *>(params + i) = p;
                }
                const uint32_t lo = pack2(p.x, p.y), hi = pack2(p.z, p.w);
                *reinterpret_cast<uint2 *>(wb + i) = make_uint2(lo, hi);
                tr[rr][cc] = uint16_t(lo);
                tr[rr][cc + 1] = uint16_t(lo >> 16);
                tr[rr][cc + 2] = uint16_t(hi);
                tr[rr][cc + 3] = uint16_t(hi >> 16);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = r0 + ty + 8 * k, c = c0 + tx;
                if (r < out && c < in) {
                    const int64_t i = w0 + int64_t(r) * in + c;
                    const uint16_t h = to_bf16(update(i));
                    wb[i] = h;
                    tr[ty + 8 * k][tx] = h;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = c0 + ty + 8 * k, r = r0 + tx;
            if (r < out && c < in) wtb[w0 + int64_t(c) * out + r] = tr[tx][ty + 8 * k];
        }
        __syncthreads();
    }
}

// Row r of member z from sample index[z * rows + r] (sample 0 for an index outside the data set): 32 rows
// per block, the features through shared memory so that the transpose leaves in rows of 32 too.
constexpr int kGatherRows = 32;
__global__ void __launch_bounds__(256) gather_kernel(const float *__restrict__ features, int nfeat,
                                                     const float *__restrict__ targets, int nout, int64_t samples,
                                                     const int32_t *__restrict__ index, int rows, int width,
                                                     uint16_t *__restrict__ x, uint16_t *__restrict__ xt,
                                                     float *__restrict__ t) {
    __shared__ int64_t sample[kGatherRows];
    __shared__ uint16_t tile[kGatherRows][33];
    const int64_t z = blockIdx.y;
    const int r0 = blockIdx.x * kGatherRows, n = min(kGatherRows, rows - r0), tid = threadIdx.x;
    grid_wait();
    features = waited(features);
    targets = waited(targets);
    if (tid < n) {
        const int64_t s = waited(index)[z * rows + r0 + tid];
        sample[tid] = s < 0 || s >= samples ? 0 : s;
    }
    __syncthreads();
    for (int f0 = 0; f0 < width; f0 += 32) {
        for (int i = tid; i < n * 32; i += 256) {
            const int r = i >> 5, f = f0 + (i & 31);
            if (f >= width) continue;
            const uint16_t b = to_bf16(f < nfeat ? features[sample[r] * nfeat + f] : 0.f);
            x[(z * rows + r0 + r) * width + f] = b;
            tile[r][i & 31] = b;
        }
        __syncthreads();
        for (int i = tid; i < 32 * 32; i += 256) {
            const int r = i & 31, f = f0 + (i >> 5);
            if (r < n && f < width) xt[(z * width + f) * rows + r0 + r] = tile[r][i >> 5];
        }
        __syncthreads();
    }
    if (targets)
        for (int r = 0; r < n; ++r) {
            const float4 *src = reinterpret_cast<const float4 *>(targets + sample[r] * nout);
            float4 *dst = reinterpret_cast<float4 *>(t + (z * rows + r0 + r) * nout);
            for (int j = tid; j < nout / 4; j += 256) dst[j] = src[j];
        }
}

// Rows of samples first, first + 1, ... (the last one beyond the data set) for every member alike, kPackCols
// BF16 values per thread.
constexpr int kPackCols = 8, kPackWidth = 64;
__global__ void pack_kernel(const float *__restrict__ features, int nfeat, int64_t samples, int64_t first, int rows,
                            uint16_t *__restrict__ x) {
    grid_wait();
    features = waited(features);
    const int i = blockIdx.x * blockDim.x + threadIdx.x, r = i / (kPackWidth / kPackCols);
    if (r >= rows) return;
    const int f0 = i % (kPackWidth / kPackCols) * kPackCols;
    const int64_t s = first + r < samples ? first + r : samples - 1;
    float v[kPackCols];
#pragma unroll
    for (int e = 0; e < kPackCols; ++e) v[e] = f0 + e < nfeat ? features[s * nfeat + f0 + e] : 0.f;
    *reinterpret_cast<uint4 *>(x + int64_t(i) * kPackCols) =
        make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// One CTA per row: every member's deviation is reduced within the warps, the CTA meets once, and one lane
// per member adds its warps' sums (thread 0 alone over all of them was a chain of 48 shared-memory reads).
// Four columns per load where the rows are 16-byte aligned.  5 members x 10,233 rows x 1,024 columns, 252 MB:
// 139 -> 75 us, with four columns per load 49 us.
template <int Members, bool Vec>
__global__ void __launch_bounds__(kRowThreads) ensemble_kernel(const float *__restrict__ probs, int rows, int nout,
                                                               const float *__restrict__ ref, float *__restrict__ mean,
                                                               float *__restrict__ spread, float *__restrict__ tv_ref) {
    constexpr int V = Vec ? 4 : 1;
    __shared__ float red[kRowThreads / 32][Members + 1];
    const int64_t r = blockIdx.x;
    float dev[Members + 1] = {};                          // the members', then the reference's
    grid_wait();
    probs = waited(probs);
    ref = waited(ref);
    auto load = [](const float *p, float (&v)[V]) {
        if constexpr (Vec) {
            const float4 f = *reinterpret_cast<const float4 *>(p);
            v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
        } else {
            v[0] = *p;
        }
    };
#pragma unroll 2
    for (int j = V * threadIdx.x; j < nout; j += V * kRowThreads) {
        float q[Members][V], mu[V], rv[V];
#pragma unroll
        for (int zz = 0; zz < Members; ++zz) load(probs + (int64_t(zz) * rows + r) * nout + j, q[zz]);
        if (ref) load(ref + r * nout + j, rv);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            mu[e] = q[0][e];
#pragma unroll
            for (int zz = 1; zz < Members; ++zz) mu[e] += q[zz][e];
            mu[e] /= float(Members);
#pragma unroll
            for (int zz = 0; zz < Members; ++zz) dev[zz] += fabsf(q[zz][e] - mu[e]);
            if (ref) dev[Members] += fabsf(mu[e] - rv[e]);
        }
        if constexpr (Vec)
            *reinterpret_cast<float4 *>(mean + r * nout + j) = make_float4(mu[0], mu[1], mu[2], mu[3]);
        else
            mean[r * nout + j] = mu[0];
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int zz = 0; zz <= Members; ++zz) {
        float x = dev[zz];
        for (int o = 16; o > 0; o >>= 1) x = x + __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[w][zz] = x;
    }
    __syncthreads();
    if (w == 0) {
        float x = 0.f;
        if (lane <= Members) {
            x = red[0][lane];
#pragma unroll
            for (int i = 1; i < kRowThreads / 32; ++i) x = x + red[i][lane];
        }
        float sp = 0.f;
#pragma unroll
        for (int zz = 0; zz < Members; ++zz) sp += __shfl_sync(0xffffffffu, x, zz);
        if (lane == 0) spread[r] = 0.5f * sp / float(Members);
        if (ref && lane == Members) tv_ref[r] = 0.5f * x;
    }
}

static int launch_ensemble(const float *probs, int rows, int members, int nout, const float *ref, float *mean,
                           float *spread, float *tv_ref, cudaStream_t s) {
    using Kernel = void (*)(const float *, int, int, const float *, float *, float *, float *);
    static constexpr Kernel kernels[2][8] = {
        {ensemble_kernel<1, false>, ensemble_kernel<2, false>, ensemble_kernel<3, false>, ensemble_kernel<4, false>,
         ensemble_kernel<5, false>, ensemble_kernel<6, false>, ensemble_kernel<7, false>, ensemble_kernel<8, false>},
        {ensemble_kernel<1, true>, ensemble_kernel<2, true>, ensemble_kernel<3, true>, ensemble_kernel<4, true>,
         ensemble_kernel<5, true>, ensemble_kernel<6, true>, ensemble_kernel<7, true>, ensemble_kernel<8, true>}};
    const bool vec = nout % 4 == 0 && aligned16(probs) && aligned16(mean) && (!ref || aligned16(ref));
    return launch_early(kernels[vec][members - 1], dim3(rows), dim3(kRowThreads), 0, s, probs, rows, nout, ref, mean,
                        spread, tv_ref);
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiled encode_fn() {
    static std::once_flag once;
    static EncodeTiled fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
        (void)cudaGetLastError();
    });
    return fn;
}

// Operand map: K values x rows x members (one member where they share the operand).
static bool operand_map(CUtensorMap *map, const uint16_t *base, int K, int rows, int members, int64_t ld, int64_t ms,
                        int box_rows) {
    EncodeTiled enc = encode_fn();
    if (!enc) return false;
    const cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(rows), cuuint64_t(ms ? members : 1)};
    const cuuint64_t strides[2] = {cuuint64_t(ld) * 2, cuuint64_t(ms ? ms : ld) * 2};
    const cuuint32_t box[3] = {kBK, cuuint32_t(box_rows), 1}, unit[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<uint16_t *>(base), dims, strides, box, unit,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// count products of one epilogue and member count in one launch
template <int EPI, typename Sh>
static int launch_shape(const dm_mlp_gemm *g, int count, int *status, cudaStream_t s) {
    GemmGroup G;
    G.count = count;
    G.first[0] = 0;
    for (int i = 0; i < count; ++i) {
        G.g[i] = g[i];
        G.first[i + 1] = G.first[i] + (g[i].M / kBM) * (g[i].N / Sh::kBN);
        if (!operand_map(&G.a[i], g[i].A, g[i].K, g[i].M, g[i].members, g[i].lda, g[i].a_ms, kBM) ||
            !operand_map(&G.b[i], g[i].B, g[i].K, g[i].N, g[i].members, g[i].ldb, g[i].b_ms, Sh::kBN))
            return DM_ERR_CUDA;
    }
    auto kernel = gemm_kernel<EPI, Sh>;
    if (ensure_max_dynamic_smem(reinterpret_cast<const void *>(kernel), int(Sh::kSmemBytes)) != cudaSuccess)
        return DM_ERR_CUDA;
    return launch_early(kernel, dim3(G.first[count], g[0].members), dim3(Sh::kThreads), Sh::kSmemBytes, s, G, status);
}

template <int EPI>
static int launch_gemms(const dm_mlp_gemm *g, int count, int *status, cudaStream_t s) {
    int64_t tiles = 0;
    int longest = 0;
    for (int i = 0; i < count; ++i) {
        tiles += int64_t(g[i].M / kBM) * (g[i].N / Wide::kBN) * g[i].members;
        longest = g[i].K > longest ? g[i].K : longest;
    }
    if (tiles > 2 * sm_count()) return launch_shape<EPI, Wide>(g, count, status, s);
    if constexpr (EPI == DM_MLP_EPI_F32 || EPI == DM_MLP_EPI_BIAS_F32)
        if (longest > kLongK) return launch_shape<EPI, Deep>(g, count, status, s);
    return launch_shape<EPI, Small>(g, count, status, s);
}

static bool mult8(int64_t x) { return x >= 0 && (x & 7) == 0; }

}  // namespace mlp
}  // namespace dmg

using namespace dmg;

extern "C" int dm_mlp_gemm_run(const dm_mlp_gemm *g, int *status_dev, void *stream) {
    using namespace mlp;
    DM_CHECK_ARG(g && status_dev);
    DM_CHECK_ARG(g->M > 0 && g->N > 0 && g->K > 0 && g->members >= 1 && g->members <= 65535);
    DM_CHECK_ARG(g->M % kBM == 0 && g->N % Wide::kBN == 0 && g->K % kBK == 0 && g->M / kBM <= 65535);
    DM_CHECK_ARG(g->A && g->B && aligned16(g->A) && aligned16(g->B));
    DM_CHECK_ARG(mult8(g->lda) && mult8(g->ldb) && g->lda >= g->K && g->ldb >= g->K && mult8(g->a_ms) &&
                 mult8(g->b_ms));
    const bool bias = g->epi == DM_MLP_EPI_GELU_FWD || g->epi == DM_MLP_EPI_BIAS_F32;
    if (bias) DM_CHECK_ARG(g->bias != nullptr && g->bias_ms >= 0);
    if (g->out_f32) DM_CHECK_ARG(aligned16(g->out_f32) && g->ld_f32 >= g->N && (g->ld_f32 & 3) == 0 && (g->f32_ms & 3) == 0);
    if (g->out_bf16) DM_CHECK_ARG(aligned16(g->out_bf16) && g->ld_bf16 >= g->N && mult8(g->ld_bf16) && mult8(g->bf16_ms));
    if (g->out_t) DM_CHECK_ARG(g->ld_t >= g->M && g->t_ms >= 0);
    cudaStream_t s = as_stream(stream);
    switch (g->epi) {
        case DM_MLP_EPI_GELU_FWD:
            DM_CHECK_ARG(g->out_bf16 || g->out_t);
            return launch_gemms<DM_MLP_EPI_GELU_FWD>(g, 1, status_dev, s);
        case DM_MLP_EPI_BIAS_F32:
            DM_CHECK_ARG(g->out_f32);
            return launch_gemms<DM_MLP_EPI_BIAS_F32>(g, 1, status_dev, s);
        case DM_MLP_EPI_GELU_BWD:
            DM_CHECK_ARG(g->pre && aligned16(g->pre) && g->ld_pre >= g->N && (g->ld_pre & 3) == 0 &&
                         (g->pre_ms & 3) == 0 && (g->out_bf16 || g->out_t));
            return launch_gemms<DM_MLP_EPI_GELU_BWD>(g, 1, status_dev, s);
        case DM_MLP_EPI_F32:
            DM_CHECK_ARG(g->out_f32);
            return launch_gemms<DM_MLP_EPI_F32>(g, 1, status_dev, s);
        default:
            return DM_ERR_ARG;
    }
}

extern "C" int dm_mlp_softmax_xent(const float *logits, const float *targets, int rows, int members, int nout,
                                   float grad_scale, float *probs, uint16_t *dz, uint16_t *dzt, float *loss_rows,
                                   void *stream) {
    using namespace mlp;
    DM_CHECK_ARG(logits && rows > 0 && members >= 1 && members <= 65535 && nout > 0);
    DM_CHECK_ARG(nout % kRowThreads == 0 && nout <= 16 * kRowThreads);
    DM_CHECK_ARG(targets ? (dz && dzt) : (probs != nullptr));
    return launch_softmax(logits, targets, nullptr, 0, rows, members, nout, rows, rows, rows, grad_scale, probs, dz, dzt,
                          loss_rows, as_stream(stream));
}

extern "C" int dm_mlp_bias_grad(const uint16_t *d_t, int64_t ld, int64_t d_ms, int N, int rows, int members,
                                float *db, int64_t db_ms, void *stream) {
    DM_CHECK_ARG(d_t && db && N > 0 && rows > 0 && ld >= rows && members >= 1 && members <= 65535);
    mlp::BiasGrads B;
    B.count = 1;
    B.rows = rows;
    B.ld = ld;
    B.db_ms = db_ms;
    B.first[0] = 0;
    B.first[1] = N;
    B.dt[0] = d_t;
    B.d_ms[0] = d_ms;
    B.db[0] = db;
    return mlp::launch_bias_grads(B, members, as_stream(stream));
}

extern "C" int dm_mlp_adam(float *params, const float *grads, float *m, float *v, int64_t count_per_member,
                           int members, const int32_t *shapes, int nlayers, float lr, float beta1, float beta2,
                           float eps, int step, uint16_t *w_bf16, uint16_t *wt_bf16, void *stream) {
    DM_CHECK_ARG(params && shapes && w_bf16 && wt_bf16 && members >= 1 && nlayers >= 1 && nlayers <= 8);
    DM_CHECK_ARG(step <= 0 || (grads && m && v));
    mlp::Layers L;
    L.n = nlayers;
    L.tiles[0] = L.bias_blocks[0] = 0;
    int64_t off = 0;
    for (int l = 0; l < nlayers; ++l) {
        DM_CHECK_ARG(shapes[2 * l] > 0 && shapes[2 * l + 1] > 0);
        L.out[l] = shapes[2 * l];
        L.in[l] = shapes[2 * l + 1];
        L.w_off[l] = off;
        off += int64_t(L.out[l]) * L.in[l];
        L.b_off[l] = off;
        off += L.out[l];
        const int64_t tiles = int64_t((L.out[l] + 31) / 32) * ((L.in[l] + 31) / 32);
        DM_CHECK_ARG(L.tiles[l] + tiles < (int64_t(1) << 30));
        L.tiles[l + 1] = L.tiles[l] + int(tiles);
        L.bias_blocks[l + 1] = L.bias_blocks[l] + (L.out[l] + 255) / 256;
    }
    DM_CHECK_ARG(off == count_per_member);
    const double c1 = step > 0 ? 1.0 - pow(double(beta1), step) : 1.0;
    const double c2 = step > 0 ? 1.0 - pow(double(beta2), step) : 1.0;
    const dim3 grid(L.tiles[nlayers] + L.bias_blocks[nlayers], members < 65535 ? members : 65535);
    bool vec = count_per_member % 4 == 0 && mlp::aligned16(params) && mlp::aligned16(grads) && mlp::aligned16(m) &&
               mlp::aligned16(v) && (reinterpret_cast<uintptr_t>(w_bf16) & 7) == 0;
    for (int l = 0; l < nlayers; ++l) vec = vec && L.w_off[l] % 4 == 0 && L.in[l] % 4 == 0;
    return launch_early(vec ? mlp::adam_kernel<true> : mlp::adam_kernel<false>, grid, dim3(256), 0, as_stream(stream),
                        params, grads, m, v, count_per_member, L, lr, beta1, beta2, eps, float(c1), float(c2), step,
                        members, w_bf16, wt_bf16);
}

extern "C" int dm_mlp_gather(const float *features, int nfeat, const float *targets, int nout, int64_t samples,
                             const int32_t *index, int rows, int members, int width, uint16_t *x, uint16_t *xt,
                             float *t, void *stream) {
    DM_CHECK_ARG(features && index && x && xt && nfeat > 0 && nfeat <= width && samples > 0);
    DM_CHECK_ARG(rows > 0 && members >= 1 && members <= 65535 && width % 8 == 0 && nout > 0 && nout % 4 == 0);
    DM_CHECK_ARG(!targets || (t && mlp::aligned16(targets) && mlp::aligned16(t)));
    return launch_early(mlp::gather_kernel, dim3((rows + mlp::kGatherRows - 1) / mlp::kGatherRows, members), dim3(256), 0,
                        as_stream(stream), features, nfeat, targets, nout, samples, index, rows, width, x, xt, t);
}

extern "C" int dm_mlp_ensemble(const float *probs, int rows, int members, int nout, const float *ref, float *mean,
                               float *spread, float *tv_ref, void *stream) {
    DM_CHECK_ARG(probs && mean && spread && rows > 0 && members >= 1 && members <= 8 && nout > 0);
    DM_CHECK_ARG(!ref || tv_ref);
    return mlp::launch_ensemble(probs, rows, members, nout, ref, mean, spread, tv_ref, as_stream(stream));
}

// ---------------------------------------------------------------------------
// the network as a whole: a forward pass, a gradient, a training step and a
// prediction each in one call, so that a step costs the host one call instead
// of one per kernel and launches what does not depend on one another together
// (the four weight gradients, the four bias gradients)
// ---------------------------------------------------------------------------

namespace dmg {
namespace mlp {

constexpr int kHidden = 256, kInput = 64, kLayers = 4;

struct NetLayer {
    int out, in;
    int64_t w, b;                     // offsets of the weights and biases in a member's parameters
};

static int net_layers(const dm_mlp_net &n, NetLayer (&L)[kLayers]) {
    int64_t off = 0;
    for (int i = 0; i < kLayers; ++i) {
        L[i].out = i == kLayers - 1 ? n.nout : kHidden;
        L[i].in = i == 0 ? kInput : kHidden;
        L[i].w = off;
        off += int64_t(L[i].out) * L[i].in;
        L[i].b = off;
        off += L[i].out;
    }
    return off == n.count ? DM_OK : DM_ERR_ARG;
}

static int check_net(const dm_mlp_net *n, int rows, bool train) {
    if (!n || n->members < 1 || n->members > 65535 || n->batch < kBM || n->batch % kBM) return DM_ERR_ARG;
    if (n->nout < kRowThreads || n->nout % kRowThreads || n->nout > 16 * kRowThreads) return DM_ERR_ARG;
    if (rows < 1 || rows > n->batch || rows % (train ? kBK : 1)) return DM_ERR_ARG;
    const void *need[] = {n->params, n->wb, n->x, n->h[0], n->h[1], n->h[2], n->logits, n->status};
    for (const void *p : need)
        if (!p || !aligned16(p)) return DM_ERR_ARG;
    if (train) {
        const void *more[] = {n->grads, n->wtb,    n->xt,     n->pre[0],  n->pre[1], n->pre[2], n->ht[0],
                              n->ht[1], n->ht[2],  n->t,      n->dz,      n->dzt,    n->du[0],  n->du[1],
                              n->du[2], n->dut[0], n->dut[1], n->dut[2], n->loss_rows};
        for (const void *p : more)
            if (!p || !aligned16(p)) return DM_ERR_ARG;
    }
    return DM_OK;
}

// C[M x N] of a product of the network: A and B with their leading dimensions and member strides
static dm_mlp_gemm product(const dm_mlp_net &n, int epi, int M, int N, int K, const uint16_t *A, int64_t lda,
                           int64_t a_ms, const uint16_t *B, int64_t ldb, int64_t b_ms) {
    dm_mlp_gemm g = {};
    g.epi = epi;
    g.M = M;
    g.N = N;
    g.K = K;
    g.members = n.members;
    g.A = A;
    g.lda = lda;
    g.a_ms = a_ms;
    g.B = B;
    g.ldb = ldb;
    g.b_ms = b_ms;
    return g;
}

// x_ms: the members' stride in x (0: the same rows for all)
static int forward(const dm_mlp_net &n, int rows, bool train, int64_t x_ms, cudaStream_t s) {
    NetLayer L[kLayers];
    int rc = net_layers(n, L);
    const int64_t B = n.batch;
    const int padded = (rows + kBM - 1) / kBM * kBM;
    const uint16_t *A = n.x;
    for (int i = 0; !rc && i < kLayers; ++i) {
        const bool out = i == kLayers - 1;
        dm_mlp_gemm g = product(n, out ? DM_MLP_EPI_BIAS_F32 : DM_MLP_EPI_GELU_FWD, padded, L[i].out, L[i].in, A, L[i].in,
                                i == 0 ? x_ms : B * L[i].in, n.wb + L[i].w, L[i].in, n.count);
        g.bias = n.params + L[i].b;
        g.bias_ms = n.count;
        g.ld_f32 = L[i].out;
        g.f32_ms = B * L[i].out;
        if (out) {
            g.out_f32 = n.logits;
            rc = dm_mlp_gemm_run(&g, n.status, s);
            break;
        }
        g.out_f32 = train ? n.pre[i] : nullptr;
        g.out_bf16 = n.h[i];
        g.ld_bf16 = kHidden;
        g.bf16_ms = B * kHidden;
        if (train) {
            g.out_t = n.ht[i];
            g.ld_t = B;
            g.t_ms = B * kHidden;
        }
        rc = dm_mlp_gemm_run(&g, n.status, s);
        A = n.h[i];
    }
    return rc;
}

// Gradients of the mean KL loss from dz / dzt.
static int backward(const dm_mlp_net &n, int rows, cudaStream_t s) {
    NetLayer L[kLayers];
    int rc = net_layers(n, L);
    if (rc) return rc;
    const int64_t B = n.batch;
    const int padded = (rows + kBM - 1) / kBM * kBM;
    // d of layer i's pre-activations: du[i] = (d of layer i + 1 x W) * gelu'(pre[i]), from the top
    for (int i = kLayers - 2; i >= 0; --i) {
        const bool top = i == kLayers - 2;
        const int K = L[i + 1].out;
        dm_mlp_gemm g = product(n, DM_MLP_EPI_GELU_BWD, padded, kHidden, K, top ? n.dz : n.du[i + 1], K, B * K,
                                n.wtb + L[i + 1].w, K, n.count);
        g.pre = n.pre[i];
        g.ld_pre = kHidden;
        g.pre_ms = B * kHidden;
        g.out_bf16 = n.du[i];
        g.ld_bf16 = kHidden;
        g.bf16_ms = B * kHidden;
        g.out_t = n.dut[i];
        g.ld_t = B;
        g.t_ms = B * kHidden;
        if ((rc = dm_mlp_gemm_run(&g, n.status, s))) return rc;
    }
    // weight gradients: d^T x the layer's input, every layer in one launch; then the bias gradients
    dm_mlp_gemm g[kLayers];
    BiasGrads bg;
    bg.count = kLayers;
    bg.rows = rows;
    bg.ld = B;
    bg.db_ms = n.count;
    bg.first[0] = 0;
    int count = 0;
    for (int i = kLayers - 1; i >= 0; --i, ++count) {
        const bool top = i == kLayers - 1;
        const uint16_t *dt = top ? n.dzt : n.dut[i];
        const int64_t d_ms = B * L[i].out;
        g[count] = product(n, DM_MLP_EPI_F32, L[i].out, L[i].in, rows, dt, B, d_ms, i == 0 ? n.xt : n.ht[i - 1], B,
                           B * L[i].in);
        g[count].out_f32 = n.grads + L[i].w;
        g[count].ld_f32 = L[i].in;
        g[count].f32_ms = n.count;
        bg.dt[count] = dt;
        bg.d_ms[count] = d_ms;
        bg.db[count] = n.grads + L[i].b;
        bg.first[count + 1] = bg.first[count] + L[i].out;
    }
    if ((rc = launch_gemms<DM_MLP_EPI_F32>(g, kLayers, n.status, s))) return rc;
    return launch_bias_grads(bg, n.members, s);
}

// targets: the batch's own (n.t), or rows index[] of a data set of `samples`
static int loss_and_grads(const dm_mlp_net &n, int rows, const float *targets, const int32_t *index, int64_t samples,
                          cudaStream_t s) {
    int rc = forward(n, rows, true, int64_t(n.batch) * kInput, s);
    if (rc) return rc;
    if ((rc = launch_softmax(n.logits, targets, index, samples, rows, n.members, n.nout, n.batch, n.batch, n.batch,
                             float(1.0 / rows), n.probs, n.dz, n.dzt, n.loss_rows, s)))
        return rc;
    return backward(n, rows, s);
}

}  // namespace mlp
}  // namespace dmg

extern "C" int dm_mlp_forward(const dm_mlp_net *net, int rows, int train, void *stream) {
    const int rc = mlp::check_net(net, rows, train != 0);
    return rc ? rc : mlp::forward(*net, rows, train != 0, int64_t(net->batch) * mlp::kInput, as_stream(stream));
}

extern "C" int dm_mlp_backward(const dm_mlp_net *net, int rows, void *stream) {
    const int rc = mlp::check_net(net, rows, true);
    return rc ? rc : mlp::backward(*net, rows, as_stream(stream));
}

extern "C" int dm_mlp_loss_and_grads(const dm_mlp_net *net, int rows, void *stream) {
    const int rc = mlp::check_net(net, rows, true);
    return rc ? rc : mlp::loss_and_grads(*net, rows, net->t, nullptr, 0, as_stream(stream));
}

extern "C" int dm_mlp_train_step(const dm_mlp_net *net, const float *features, int nfeat, const float *targets,
                                 int64_t samples, const int32_t *index, float lr, float beta1, float beta2, float eps,
                                 int step, void *stream) {
    int rc = mlp::check_net(net, net ? net->batch : 0, true);
    if (rc) return rc;
    const dm_mlp_net &n = *net;
    DM_CHECK_ARG(features && targets && index && n.m && n.v && step >= 1 && mlp::aligned16(targets));
    if ((rc = dm_mlp_gather(features, nfeat, nullptr, n.nout, samples, index, n.batch, n.members, mlp::kInput, n.x, n.xt,
                            nullptr, stream)))
        return rc;
    // the softmax reads its targets from the data set (gathering them took 12 us of a 150 us step)
    if ((rc = mlp::loss_and_grads(n, n.batch, targets, index, samples, as_stream(stream)))) return rc;
    const int32_t shapes[2 * mlp::kLayers] = {mlp::kHidden, mlp::kInput,  mlp::kHidden, mlp::kHidden,
                                              mlp::kHidden, mlp::kHidden, n.nout,       mlp::kHidden};
    return dm_mlp_adam(n.params, n.grads, n.m, n.v, n.count, n.members, shapes, mlp::kLayers, lr, beta1, beta2, eps, step,
                       n.wb, n.wtb, stream);
}

extern "C" int dm_mlp_predict(const dm_mlp_net *net, const float *features, int nfeat, int64_t samples, float *out,
                              void *stream) {
    int rc = mlp::check_net(net, net ? net->batch : 0, false);
    if (rc) return rc;
    const dm_mlp_net &n = *net;
    DM_CHECK_ARG(nfeat > 0 && nfeat <= mlp::kInput && samples >= 0);
    DM_CHECK_ARG(samples == 0 || (features && out));      // an empty tensor has no address
    cudaStream_t s = as_stream(stream);
    for (int64_t s0 = 0; s0 < samples; s0 += n.batch) {
        const int rows = int(samples - s0 < n.batch ? samples - s0 : n.batch);
        const int padded = (rows + mlp::kBM - 1) / mlp::kBM * mlp::kBM;
        rc = launch_early(mlp::pack_kernel, dim3((padded * mlp::kPackWidth / mlp::kPackCols + 255) / 256), dim3(256), 0, s,
                          features, nfeat, samples, s0, padded, n.x);
        if (rc) return rc;
        if ((rc = mlp::forward(n, rows, false, 0, s))) return rc;
        if ((rc = mlp::launch_softmax(n.logits, nullptr, nullptr, 0, rows, n.members, n.nout, n.batch, samples, 0, 1.f,
                                      out + s0 * n.nout, nullptr, nullptr, nullptr, s)))
            return rc;
    }
    return DM_OK;
}
