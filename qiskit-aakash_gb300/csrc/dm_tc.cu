// Tensor-core fused pass (FP32 state, 3-way FP16 split on tcgen05).
//
// A pass holds 7 resident qubit axes: every tile of 4**7 = 16,384
// coefficients is streamed into shared memory (cp.async, 16-byte chunks),
// then the pass's register rounds run as matrix products on the tensor
// cores.  A round names 3 of the tile's axes; the round's operations,
// composed in FP64 on the device (compose_passes_kernel before a group of
// passes, or per instance inside the batched sweeps), form one 64x64 real
// transfer matrix U acting on the 64 coefficients that differ only in those
// axes.  With the tile
// viewed as 256 groups x 64 (one row per group), the round is
//     D[g][j'] = sum_j X[g][j] * U[j'][j]           (M = 256, N = 64, K = 64)
// issued as two M = 128 tcgen05.mma.kind::f16 chains into TMEM.  FP32
// accuracy comes from a 3-way FP16 split: inside the pass the tile is held
// in units of 2**-n (x = 2**n a, |x| <= 1), x = h + 2**-11 l with
// h = fp16(x), l = fp16(2**11 (x - h)), and U = Uh + 2**-11 Ul likewise;
//     D = h (2**11 Uh)^T + [h Ul^T + l Uh^T] = 2**11 x U^T + O(2**-22 |x|)
// (the l Ul term is below FP32), the large term and the bracketed
// corrections in separate FP32 accumulators, and the epilogue adds them and
// scales by 2**-11.
// FP16 runs at twice the TF32 rate and halves the operand bytes.  The
// epilogue reads D from TMEM (tcgen05.ld, one group per thread) and writes
// the h / l split directly in the operand layout of the next round.  The
// last round either stores each thread's row straight to global memory (a
// "direct" last round: its rows 0-3 are tile bits 0-3, so lanes 0-15 write
// 16 contiguous coefficients) while the next tile's cp.async load, issued as
// soon as the round's MMAs have read the operands, lands in the freed
// operand region; or, when it acts on local axes 0 and 1, it writes the tile
// back in its natural FP32 layout for 128-bit stores.  Every wait on an
// mbarrier is bounded: a wait that gives up records an error in *status and
// the kernel drains and returns.
//
// Two CTAs of 256 threads share an SM, so one CTA's tile load, barriers
// and MMA waits overlap the other's work.  Shared memory per CTA (dynamic,
// 88 KB): AH / AL 32 KB each (round operand h / l, swizzled K-major FP16
// layout, 256 rows x 64; together they also hold the natural FP32 tile that
// cp.async streams in and the last round writes out), B 24 KB (2**11 Uh and
// Ul stacked as one 128-row operand, then Uh).  The h operand is read once
// per round for both of its terms (N = 128 into two 64-column accumulators
// that the epilogue adds); warps 0-3 own the rows of M block 0 and warps 4-7
// those of M block 1, one row per thread (TMEM lane quadrant = warp % 4).
#include <cuda_fp16.h>
#include <math.h>

#include <mutex>

#include "dm_batch.cuh"
#include "dm_common.cuh"
#include "dm_rounds.cuh"
#include "dm_tc_tile.cuh"
#include "dm_tcgen05.cuh"

namespace dmg {

namespace tc {

constexpr int kThreads = 256;                  // two CTAs per SM
constexpr int kCtasPerSm = 2;
constexpr int kBlocksPerThread = 256 / kThreads;   // M = 128 blocks in one thread's epilogue
constexpr uint32_t kBBytes = 3 * kBImage;      // 24 KB
constexpr uint32_t kSmemBytes = 2 * kABytes + kBBytes;   // 88 KB: two CTAs per SM
constexpr int kUHalves = 3 * 64 * 64;          // FP16 values per round image
constexpr uint32_t kTmemCols = 256;            // two M = 128 blocks x N = 128 (D1 | D2)

// Natural-layout swizzle of the tile (16-byte chunks intact), as in dm_pass.cu.
__device__ __forceinline__ int nat_swz(int e) { return e ^ ((((e >> 5) ^ (e >> 8)) & 7) << 2); }

struct Pass {
    int n, m, low, nrounds;
    int vec0;
    int direct;                      // the last round stores straight to global memory (offsets lastg)
    float up, down;                  // 2**n, 2**-n
    int64_t res_stride[kAxes];
    int64_t nonres_stride[DM_MAX_QUBITS];
    alignas(16) uint32_t natrow[8];
    alignas(16) uint32_t natk[8];
    // direct: global element offsets of the last round's row bits 0-7, K bits 0-5
    alignas(16) int64_t lastg[14];
    Round rounds[DM_MAX_ROUNDS];
};

// Global offsets of a direct last round's 14 bits: its tables hold the linear natural offset
// 2**b of tile bit b, i.e. bit b % 2 of local axis b / 2.
__host__ __device__ inline void direct_offsets(Pass &p, const uint32_t *rowc, const uint32_t *kc) {
    for (int i = 0; i < 14; ++i) {
        const uint32_t c = i < 8 ? rowc[i] : kc[i - 8];
        int b = 0;
        while (b < 2 * kAxes - 1 && (1u << b) != c) ++b;
        p.lastg[i] = p.res_stride[b >> 1] << (b & 1);
    }
}

__device__ __forceinline__ int64_t tile_offset(const Pass &p, int e) {
    int64_t off = e & ((1 << (2 * p.low)) - 1);
    for (int r = p.low; r < kAxes; ++r) off += int64_t((e >> (2 * r)) & 3) * p.res_stride[r];
    return off;
}

// The dynamic shared memory from its first 1024-byte boundary (the swizzle's).
__device__ __forceinline__ unsigned char *aligned_smem() {
    extern __shared__ __align__(1024) unsigned char raw[];
    return raw + ((1024 - (smem_u32(raw) & 1023)) & 1023);
}
constexpr uint32_t kAlignSlack = 1024;

// Per-CTA tensor-core state shared by the single-state and the batched kernels.
struct TcCta {
    unsigned char *AH, *AL, *B;   // operand images h / l (the natural tile before and after the rounds), U
    uint64_t *mbar;               // MMA completion barrier
    int64_t *hi_off;              // kTile / 4 / kThreads chunk offsets of the current pass
    int *abort_s;                 // set when a bounded wait gave up
    uint32_t tmem;                // accumulator columns
    uint32_t phase;               // mbarrier phase to wait for next
    bool pending;                 // an MMA batch committed but not yet waited for
};

// mbarrier init and accumulator allocation (all threads).
__device__ __forceinline__ void tc_setup(TcCta &c, uint32_t *tmem_base_s) {
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        *c.abort_s = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(c.mbar)));
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)),
                     "n"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    c.tmem = *tmem_base_s;
    c.phase = 0;
    c.pending = false;
}

// Drain what is in flight and release the accumulator (all threads).
__device__ __forceinline__ void tc_teardown(TcCta &c) {
    if (c.pending) mbar_wait(smem_u32(c.mbar), c.phase);   // drain before the accumulator is released
    cp_async_wait_all();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "n"(kTmemCols));
}

// Streams tiles t0, t0 + dt, ... of one pass through the rounds (all threads
// of the CTA); round r's images are at umats + p.rounds[r].umoff.  Returns
// false when a bounded wait gave up (*status is then set).
__device__ __forceinline__ bool tc_pass_tiles(float *__restrict__ st, const Pass &p,
                                              const uint16_t *__restrict__ umats, int t0, int dt, TcCta &c,
                                              int *status) {
    unsigned char *AH = c.AH, *AL = c.AL, *B = c.B;
    uint64_t &mbar = *c.mbar;
    int64_t *hi_off = c.hi_off;
    volatile int &abort_s = *c.abort_s;
    const uint32_t tmem = c.tmem;
    uint32_t phase = c.phase;
    bool pending = c.pending;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int ntiles = 1 << (2 * p.m);   // at most 4**10
    const int64_t off_tid = tile_offset(p, 4 * tid);
    __syncthreads();   // earlier readers of hi_off are done
    for (int i = tid; i < kTile / 4 / kThreads; i += kThreads) hi_off[i] = tile_offset(p, 4 * kThreads * i);
    __syncthreads();

    auto tile_base = [&](int t) {
        int64_t base = 0;
        for (int u = 0; u < p.m; ++u) {
            base += int64_t(t & 3) * p.nonres_stride[u];
            t >>= 2;
        }
        return base;
    };
    auto load_tile = [&](int t) {   // natural layout into AH / AL (64 KB)
        const float *src = st + tile_base(t) + off_tid;
#pragma unroll 8
        for (int i = 0; i < kTile / 4 / kThreads; ++i)
            cp_async16(AH + 4 * nat_swz(4 * (tid + kThreads * i)), src + hi_off[i]);
        cp_async_commit();
    };
    auto load_u = [&](int r) {          // round r's three U images into B (contiguous)
        const uint16_t *src = umats + p.rounds[r].umoff;
#pragma unroll
        for (int i = 0; i < int(kBBytes) / 16 / kThreads; ++i) {
            const int c = tid + kThreads * i;
            cp_async16(B + 16 * c, src + 8 * c);
        }
        cp_async_commit();
    };

    load_u(0);
    bool loaded = false;   // the tile's load went out during the previous tile's last round
    for (int t = t0; t < ntiles; t += dt) {
        if (!loaded) load_tile(t);
        loaded = false;
        cp_async_wait_all();
        __syncthreads();
        // ---- natural tile -> round 0's operand (h / l), in place ----
        // Work items are (row, 8-value K chunk) pairs with the row's low three bits on the lane
        // bits, so each 16-byte chunk store of an 8-lane phase covers the 8 rows of one core
        // matrix: all 32 banks.  Every thread reads all of its values before any is written.
        {
            constexpr int kItems = kGroups * 8 / kThreads;   // 8
            const float *nat = reinterpret_cast<const float *>(AH);
            const float up = p.up;      // 2**n: the tile in units of 2**-n
            struct alignas(16) { uint32_t row[8], k[8]; } nt;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 w = reinterpret_cast<const uint4 *>(i < 2 ? p.natrow : p.natk)[i & 1];
                uint32_t *o = i < 2 ? nt.row + 4 * i : nt.k + 4 * (i - 2);
                o[0] = w.x, o[1] = w.y, o[2] = w.z, o[3] = w.w;
            }
            float x[kItems][8];
#pragma unroll
            for (int q = 0; q < kItems; ++q) {
                const int i = tid + kThreads * q;
                const int crow = ((i >> 6) << 3) | (i & 7), c = (i >> 3) & 7;
                // chunk c holds K = 8c .. 8c + 7: K bits 3-5 come from c, bits 0-2 from the element
                const uint32_t nb = xor_bits<8>(uint32_t(crow), nt.row) ^ ((c & 1) ? nt.k[3] : 0u) ^
                                    ((c & 2) ? nt.k[4] : 0u) ^ ((c & 4) ? nt.k[5] : 0u);
                if (p.vec0 == 0) {   // digit 0 is local axis 0: four adjacent natural elements
                    const float4 a4 = *reinterpret_cast<const float4 *>(nat + nb);
                    const float4 b4 = *reinterpret_cast<const float4 *>(nat + (nb ^ nt.k[2]));
                    x[q][0] = a4.x; x[q][1] = a4.y; x[q][2] = a4.z; x[q][3] = a4.w;
                    x[q][4] = b4.x; x[q][5] = b4.y; x[q][6] = b4.z; x[q][7] = b4.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        x[q][e] = nat[nb ^ ((e & 1) ? nt.k[0] : 0u) ^ ((e & 2) ? nt.k[1] : 0u) ^
                                      ((e & 4) ? nt.k[2] : 0u)];
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kItems; ++q) {
                const int i = tid + kThreads * q;
                const int crow = ((i >> 6) << 3) | (i & 7), c = (i >> 3) & 7;
                uint32_t hw[4], lw[4];
#pragma unroll
                for (int e = 0; e < 8; e += 2) split2(x[q][e] * up, x[q][e + 1] * up, hw[e >> 1], lw[e >> 1]);
                const uint32_t o = operand_chunk(crow, c);
                *reinterpret_cast<uint4 *>(AH + o) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                *reinterpret_cast<uint4 *>(AL + o) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            }
        }
        for (int r = 0; r < p.nrounds; ++r) {
            // round 0's U was waited for with the tile; later rounds wait for their U
            if (r > 0) cp_async_wait_all();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (tid == 0) {
                // D[:, 0:64] = h (2**11 Uh)^T and D[:, 64:128] = h Ul^T + l Uh^T: the h operand is
                // read once for both of its terms (N = 128 over the stacked images 2**11 Uh | Ul); the
                // large term's accumulator takes only its own four K steps, the two correction terms
                // (2**-11 smaller) share the other, and the epilogue adds the two in FP32
                const uint32_t ah = smem_u32(AH), al = smem_u32(AL), b0 = smem_u32(B);
#pragma unroll
                for (int mb = 0; mb < 2; ++mb) {
                    const uint32_t aoff = mb * (kABytes / 2);
#pragma unroll
                    for (int term = 0; term < 2; ++term) {
                        const uint32_t d = tmem + mb * 128 + (term == 0 ? 0u : 64u);
                        const uint32_t a = (term == 0 ? ah : al) + aoff;
                        const uint32_t b = b0 + term * 2 * kBImage;
                        const uint32_t idesc = term == 0 ? kIdesc128 : kIdesc64;
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {      // K = 16 per MMA: two core matrices
                            const uint64_t da = operand_desc(a + ks * kOperandStep);
                            const uint64_t db = smem_desc(b + ks * 2 * kLBO);
                            const uint32_t acc = (term | ks) ? 1u : 0u;
                            asm volatile(
                                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
                                "l"(da), "l"(db), "r"(idesc), "r"(acc));
                        }
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                    smem_u32(&mbar)));
            }
            pending = true;
            const bool ok = mbar_wait(smem_u32(&mbar), phase);
            if (ok) {
                phase ^= 1;
                pending = false;
            }
            if (!__all_sync(0xffffffffu, ok)) {
                if ((tid & 31) == 0) {
                    atomicExch(status, 1);
                    abort_s = 1;
                }
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            __syncthreads();
            if (abort_s) break;
            // B is free: fetch the next round's U (or round 0's, for the next tile)
            load_u(r + 1 < p.nrounds ? r + 1 : 0);
            // ---- epilogue: D -> next operand (h / l), or the natural tile after the last round ----
            // the thread holds row tid % 128 of M block tid / 128 (TMEM columns 0-127 / 128-255)
            const Round R = p.rounds[r];
            uint32_t tk[3][4];
            digit_tables(R.kc, tk);
            const bool last = r + 1 == p.nrounds;
            if (last && p.direct && t + dt < ntiles) {
                // the operands are consumed and this round writes straight to global memory: the next
                // tile's load overlaps the epilogue
                load_tile(t + dt);
                loaded = true;
            }
#pragma unroll 1
            for (int i = 0; i < kBlocksPerThread; ++i) {
                const int mb = kBlocksPerThread == 1 ? (warp >> 2) : i;
                float v[64];
                const uint32_t ta = tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(mb * 128);
                // D[:, 0:64] + D[:, 64:128], 32 columns of each at a time (one wait per half)
                tcg::tmem_ld32_pair_add(ta, ta + 64, v);
                tcg::tmem_ld32_pair_add(ta + 32, ta + 96, v + 32);
                const uint32_t base = xor_bits<8>(uint32_t((tid & 127) + 128 * mb), R.rowc);
                if (!last) {
                    store_all<true>(v, R.vec, base, tk, AH, AL);   // split from the accumulator scale
                } else if (p.direct) {
                    // the row straight to global memory: rows 0-3 are tile bits 0-3 (16 contiguous
                    // coefficients on lanes 0-15)
                    const float down = p.down * kLoUnscale;
                    const int row = (tid & 127) + 128 * mb;
                    int64_t rowg = tile_base(t);
#pragma unroll
                    for (int b = 0; b < 8; ++b)
                        if ((row >> b) & 1) rowg += p.lastg[b];
                    float *row_ptr = st + rowg;
                    const int64_t k0 = p.lastg[8], k1 = p.lastg[9];
#pragma unroll
                    for (int d2 = 0; d2 < 4; ++d2) {
                        const int64_t o2 = (d2 & 1 ? p.lastg[12] : 0) + (d2 & 2 ? p.lastg[13] : 0);
#pragma unroll
                        for (int d1 = 0; d1 < 4; ++d1) {
                            float *q = row_ptr + o2 + (d1 & 1 ? p.lastg[10] : 0) + (d1 & 2 ? p.lastg[11] : 0);
                            const int j = 4 * d1 + 16 * d2;
                            q[0] = v[j] * down;
                            q[k0] = v[j + 1] * down;
                            q[k1] = v[j + 2] * down;
                            q[k0 + k1] = v[j + 3] * down;
                        }
                    }
                } else {
                    const float down = p.down * kLoUnscale;   // back to coefficients
#pragma unroll
                    for (int j = 0; j < 64; ++j) v[j] *= down;
                    store_all<false>(v, R.vec, base, tk, AH, AL);   // natural FP32 layout into AH / AL
                }
            }
            if (!last) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        if (abort_s) break;
        if (p.direct) continue;   // written by the last round
        __syncthreads();
        // ---- write the tile back with 128-bit stores, each chunk's slot refilled with the next
        // tile's chunk as soon as it is read: a chunk is read and reloaded by the same thread ----
        {
            float *dst = st + tile_base(t) + off_tid;
            const float *out = reinterpret_cast<const float *>(AH);
            const bool next = t + dt < ntiles;
            const float *src = st + (next ? tile_base(t + dt) : 0) + off_tid;
#pragma unroll 8
            for (int i = 0; i < kTile / 4 / kThreads; ++i) {
                const int e = 4 * (tid + kThreads * i);
                const float4 v = *reinterpret_cast<const float4 *>(out + nat_swz(e));
                *reinterpret_cast<float4 *>(dst + hi_off[i]) = v;
                if (next) cp_async16(AH + 4 * nat_swz(e), src + hi_off[i]);
            }
            if (next) {
                cp_async_commit();
                loaded = true;
            }
        }
    }
    cp_async_wait_all();   // round 0's images prefetched for a tile that does not come
    __syncthreads();
    c.phase = phase;
    c.pending = pending;
    return !abort_s;
}

__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    pass_tc_kernel(float *__restrict__ st, const __grid_constant__ Pass p, const uint16_t *__restrict__ umats,
                   int *status) {
    unsigned char *smem = aligned_smem();
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int64_t hi_off[kTile / 4 / kThreads];
    __shared__ int abort_s;
    TcCta c{smem, smem + kABytes, smem + 2 * kABytes, &mbar, hi_off, &abort_s, 0, 0, false};
    tc_setup(c, &tmem_base_s);
    grid_wait();
    tc_pass_tiles(st, p, waited(umats), blockIdx.x, gridDim.x, c, status);
    tc_teardown(c);
}

// ---------------------------------------------------------------------------
// batched sweeps on the tensor cores
// ---------------------------------------------------------------------------

constexpr int64_t kScratchHalves = int64_t(DM_MAX_ROUNDS) * kUHalves;   // a pass's round images

// Kernel parameters of one batched pass, each field by a thread of its own (the pass table is in
// global memory: one thread reading it field by field takes microseconds).
static_assert(sizeof(Round) == sizeof(dm_tc_round), "a round's table is copied as words");
static_assert(offsetof(dm_tc_round, rowc) == 8 && offsetof(dm_tc_round, kc) == 40, "its order");
__device__ void batch_tc_setup(Pass &ps, const dm_batch_tc_pass &bp, int n) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int nr = bp.ops.nrounds;
    // the digit positions of the resident axes (local axis r = the r-th lowest)
    unsigned resident = 0;
#pragma unroll
    for (int r = 0; r < kAxes; ++r) resident |= 1u << (n - 1 - bp.ops.axes[r]);
    if (tid == 0) {
        ps.n = n;
        ps.m = n - kAxes;
        ps.low = __ffs(~resident) - 1;
        ps.nrounds = nr;
        ps.vec0 = bp.tables.vec0 == 0 ? 0 : -1;
        ps.direct = bp.tables.direct_last ? 1 : 0;
        ps.up = ldexpf(1.0f, n);
        ps.down = ldexpf(1.0f, -n);
    } else if (tid >= 32 && tid < 64) {
        if (lane < kAxes) ps.res_stride[lane] = int64_t(1) << (2 * (n - 1 - bp.ops.axes[lane]));
        // the lane-th lowest position that is not resident
        if (lane < n && !((resident >> lane) & 1))
            ps.nonres_stride[lane - __popc(resident & ((1u << lane) - 1))] = int64_t(1) << (2 * lane);
    } else if (tid >= 64 && tid < 96) {
        if (lane < 8) ps.natrow[lane] = bp.tables.natrow[lane];
        else if (lane < 14) ps.natk[lane - 8] = bp.tables.natk[lane - 8];
    } else if (tid >= 96 && tid < 128) {
        if (lane < 14 && bp.tables.direct_last) {
            // direct last round: the offset 2**b of tile bit b, bit b % 2 of local axis b / 2
            const dm_tc_round &L = bp.tables.rounds[nr - 1];
            const int bit = __ffs(lane < 8 ? L.rowc[lane] : L.kc[lane - 8]) - 1;
            ps.lastg[lane] = (int64_t(1) << (2 * (n - 1 - bp.ops.axes[bit >> 1]))) << (bit & 1);
        }
    }
    const uint32_t *in = reinterpret_cast<const uint32_t *>(bp.tables.rounds);
    uint32_t *out = reinterpret_cast<uint32_t *>(ps.rounds);
    constexpr int kWords = sizeof(Round) / 4;
    for (int i = tid; i < nr * kWords; i += kThreads)
        out[i] = i % kWords == kWords - 1 ? uint32_t(i / kWords * kUHalves)               // umoff
               : i % kWords == kWords - 2 ? uint32_t(int32_t(in[i - kWords + 2]) >> 24)   // vec, the fourth byte
               : i / kWords < nr - 1      ? operand_offset(in[i + 2]) : in[i + 2];
}

// Round r's matrix U (64 x 64 in its K-digit order), composed in FP64 from the
// round's operations and written as the FP16 images that the MMAs read, K-major
// (value (n%8)*8 + k%8 + (k/8)*64 + (n/8)*512 for output n, input k), with
// Uh = fp16(U) and Ul = fp16(2**11 (U - Uh)): three images 2**11 Uh | Ul | Uh
// for the cp.async-fed kernels, two images Uh | Ul for the TMA-fed one.
//
// What bounds it is the FP64 pipe: two FMAs per clock and SM, one warp
// instruction per 64 cycles on each of its four quarters.  So the operations are
// not applied to the 64 columns of U one by one (40-70 FP64 instructions per
// entry of a two-CX round with noise and rotations).  They act on pairs of the
// round's three digits: those up to the first operation that needs the third
// pair form two 16 x 16 blocks, T1 on the digits (y, x) and T2 on (c, x), and
//     U[(y',x',c'), (y,x,c)] = sum_m T2[(c',x'), (c,m)] T1[(y',m), (y,x)],
// four FMAs per entry (a single pair with maps on the third digit: one product).
// A one-axis map counts to the block that its neighbours on its digit belong to.
// The few operations beyond (a third CX) are applied to the columns.  The split
// into FP16 parts works on the bits of the doubles, without FP64 instructions
// (its conversions and subtractions were five of them per entry).
// 1,024 points of a 10-qubit template: 78.0 -> 72.8 ms.
constexpr int kColStride = 65;   // doubles per column: a warp's lanes spread over the banks
constexpr int kBlkStride = 17;   // doubles per column of a block
constexpr int kBlkDoubles = 16 * kBlkStride;

// A 4x4 map on four values S apart.
__device__ __forceinline__ void map1_at(double *x, int S, const double (&m)[16], bool row0, bool xy) {
    double x0 = x[0], x1 = x[S], x2 = x[2 * S], x3 = x[3 * S];
    if (xy) {
        map4_tp_xy(m, x0, x1, x2, x3);
    } else if (row0) {
        map4<true>(m, x0, x1, x2, x3);
    } else {
        map4<false>(m, x0, x1, x2, x3);
        x[0] = x0;
    }
    x[S] = x1;
    x[2 * S] = x2;
    x[3 * S] = x3;
}

// A pair operation on the 16 values at col, the operation's axes SA and SB apart.
// Map2: 16x16 general maps too (the single-state passes; the batched plans hold none).
template <bool Map2>
__device__ __forceinline__ void pair_at(double *col, int SA, int SB, const dm_op &op, const double *__restrict__ mg) {
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = col[(i >> 2) * SA + (i & 3) * SB];
    if (Map2 && op.kind == DM_OP_MAP2) {   // y[4 pa + pb] = sum_s mg[16 (4 pa + pb) + s] x[s]
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < 16; ++j) acc = fma(mg[16 * i + j], x[j], acc);
            col[(i >> 2) * SA + (i & 3) * SB] = acc;
        }
        return;
    }
    if (op.kind == DM_OP_CX) {
        CxCoef<double> cx{1.0, 0.0, 1.0, 0.0, 0.0};
        const bool ideal = (op.flags & DM_CX_IDEAL) != 0;
        if (!ideal) cx = CxCoef<double>{mg[0], mg[1], mg[2], mg[3], mg[4]};
        cx16(x, cx, ideal);
    } else {   // DM_OP_DIAG2: entry (pa, pb) scaled by mg[4 pa + pb]
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] *= mg[i];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) col[(i >> 2) * SA + (i & 3) * SB] = x[i];
}

__device__ __forceinline__ void load_map(double (&m)[16], const double *__restrict__ mg, bool &row0, bool &xy) {
#pragma unroll
    for (int i = 0; i < 16; ++i) m[i] = mg[i];
    row0 = m[0] == 1.0 && m[1] == 0.0 && m[2] == 0.0 && m[3] == 0.0;
    xy = row0 && m[4] == 0.0 && m[8] == 0.0;
}

// u (a map's entry) -> FP16 parts h = fp16(u), l = fp16(2**11 (u - h)), both rounded to nearest as from
// the FP64 values.  |u| = f + g, f its leading 24 bits, g the 29 below; f and f - h + g are rounded to odd
// where bits are dropped, which a later rounding to 11 bits does not notice.
__device__ __forceinline__ void split_bits(double u, uint16_t &h16, uint16_t &l16) {
    const uint32_t hi = uint32_t(__double2hiint(u)), lo = uint32_t(__double2loint(u));
    const int e = int((hi >> 20) & 0x7FF) - 1023;
    const uint32_t sign = (hi >> 16) & 0x8000u;
    if (e > 14) {                          // beyond FP16 (or not a number): the conversions' own results
        const __half h = __double2half(u);
        h16 = __half_as_ushort(h);
        l16 = __half_as_ushort(__double2half((u - double(__half2float(h))) * double(kLoScale)));
        return;
    }
    if (e < -60) {                         // both parts round to zero
        h16 = l16 = uint16_t(sign);
        return;
    }
    const uint32_t tail = lo & 0x1FFFFFFFu;
    const uint32_t fb = uint32_t(e + 127) << 23 | (hi & 0xFFFFFu) << 3 | lo >> 29;
    const __half h = __float2half_rn(__uint_as_float(fb | (tail != 0 ? 1u : 0u)));
    const float a = __uint_as_float(fb) - __half2float(h);        // exact
    const float t = __uint2float_rz(tail);
    const float g = __uint_as_float(__float_as_uint(t) | (uint32_t(t) != tail ? 1u : 0u)) *
                    __uint_as_float(uint32_t(e - 52 + 127) << 23);
    const float s = __fadd_rz(a, g);
    const uint32_t odd = g - (s - a) != 0.0f ? 1u : 0u;
    const __half l = __float2half_rn(__uint_as_float(__float_as_uint(s) | odd) * kLoScale);
    h16 = uint16_t(__half_as_ushort(h) | sign);
    l16 = uint16_t(__half_as_ushort(l) ^ sign);
}

// How a round's operations [begin, end) are composed: up to `stop` as the two blocks, T2's pair
// operations from p2 on.  Without a second pair T2 holds maps on c alone (single).
struct RoundPlan {
    int16_t begin, p2, stop, end;
    int8_t y, x, c, single;
};

__device__ __forceinline__ RoundPlan plan_round(const dm_op *ops, int begin, int end) {
    RoundPlan P;
    int m1 = 0, m2 = 0, p2 = end, stop = end;
    for (int i = begin; i < end; ++i) {
        const dm_op &op = ops[i];
        if (op.kind == DM_OP_MAP1) continue;
        const int m = (1 << ((op.flags >> 8) & 3)) | (1 << ((op.flags >> 12) & 3));
        if (m1 == 0) {
            m1 = m;
        } else if (m2 == 0) {
            if (m != m1) {
                m2 = m;
                p2 = i;
            }
        } else if (m != m2) {
            stop = i;
            break;
        }
    }
    if (m1 == 0) m1 = 3;
    const int c = 31 - __clz(7 ^ m1), x = __ffs(m2 ? m1 & m2 : m1) - 1;
    P.begin = int16_t(begin);
    P.p2 = int16_t(p2);
    P.stop = int16_t(stop);
    P.end = int16_t(end);
    P.c = int8_t(c);
    P.x = int8_t(x);
    P.y = int8_t(3 - c - x);
    P.single = m2 == 0;
    return P;
}

// A pass's operations in shared memory (an operation's own read from global memory would cost every warp
// a round trip per operation), 16 coefficients each; 16x16 maps keep theirs at mats + moff.
struct ComposeShared {
    double coefs[DM_MAX_PASS_OPS * kCoefStride];
    dm_op ops[DM_MAX_PASS_OPS];
    RoundPlan plan[DM_MAX_ROUNDS];
};
static_assert(sizeof(dm_op) == 16, "operations are copied as words");

// The operations of rounds [r0, r1) of a pass and their plans (all threads of the block).
__device__ __forceinline__ void compose_load(ComposeShared &cs, const dm_batch_pass &bp, const double *__restrict__ mats,
                                             int r0, int r1) {
    const int o0 = r0 > 0 ? bp.round_end[r0 - 1] : 0, o1 = bp.round_end[r1 - 1];
    for (int i = o0 * kCoefStride + int(threadIdx.x); i < o1 * kCoefStride; i += blockDim.x) {
        const dm_op &op = bp.ops[i / kCoefStride];
        if (op.kind != DM_OP_MAP2 && (op.kind != DM_OP_CX || i % kCoefStride < 5))
            cs.coefs[i] = mats[op.moff + i % kCoefStride];
    }
    for (int i = o0 * 4 + int(threadIdx.x); i < o1 * 4; i += blockDim.x)
        reinterpret_cast<uint32_t *>(cs.ops)[i] = reinterpret_cast<const uint32_t *>(bp.ops)[i];
    __syncthreads();
    for (int r = r0 + int(threadIdx.x); r < r1; r += blockDim.x)
        cs.plan[r] = plan_round(cs.ops, r > 0 ? bp.round_end[r - 1] : 0, bp.round_end[r]);
    __syncthreads();
}

template <bool Map2>
__device__ __forceinline__ const double *op_coefs(const ComposeShared &cs, const double *mats, int i) {
    return Map2 && cs.ops[i].kind == DM_OP_MAP2 ? mats + cs.ops[i].moff : cs.coefs + kCoefStride * i;
}

// Columns c0 .. c0 + nc - 1 of block T1 (second = false) or T2 of a round by one warp.
template <bool Map2>
__device__ void compose_block(const ComposeShared &cs, const RoundPlan &P, const double *mats, bool second, int c0, int nc,
                              double *blk, int lane) {
    const int high = second ? P.c : P.y;
    double *w = blk + c0 * kBlkStride;
    for (int i = lane; i < nc * 16; i += 32) w[(i >> 4) * kBlkStride + (i & 15)] = (i & 15) == c0 + (i >> 4) ? 1.0 : 0.0;
    __syncwarp();
    for (int i = P.begin; i < P.stop; ++i) {
        const dm_op &op = cs.ops[i];
        const int da = (op.flags >> 8) & 3;
        if (op.kind == DM_OP_MAP1) {
            if ((da == P.x ? i >= P.p2 : da == P.c) != second) continue;
            double m[16];
            bool row0, xy;
            load_map(m, op_coefs<Map2>(cs, mats, i), row0, xy);
            const int S = da == high ? 4 : 1;
            for (int g = lane; g < nc * 4; g += 32)
                map1_at(w + (g >> 2) * kBlkStride + (g & 3) * (5 - S), S, m, row0, xy);
        } else {
            if ((i >= P.p2) != second) continue;
            const int SA = da == high ? 4 : 1;
            if (lane < nc) pair_at<Map2>(w + lane * kBlkStride, SA, 5 - SA, op, op_coefs<Map2>(cs, mats, i));
        }
        __syncwarp();
    }
}

// Columns k0 .. k0 + C - 1 (k0 a multiple of C) of a round from its blocks by one warp, into the images at
// img (three or two of them); w: the warp's scratch of C columns.
template <bool Map2, int C>
__device__ void compose_cols(const ComposeShared &cs, const RoundPlan &P, const double *mats, const double *t1,
                             const double *t2, int k0, double *w, uint16_t *__restrict__ img, bool three, int lane) {
    const bool more = P.stop < P.end;
    const int uh = three ? 8192 : 0;   // three: 2**11 Uh at 0, Ul at 4096, Uh at 8192; two: Uh at 0, Ul at 4096
    struct alignas(2 * C) Chunk {      // row j of the C columns: one chunk of C halves per image
        uint32_t v[C / 2];
    };
    double u[C];
    auto entries = [&](int j) {
        const int jy = (j >> (2 * P.y)) & 3, jx = (j >> (2 * P.x)) & 3, jc = (j >> (2 * P.c)) & 3;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int k = k0 + c, ky = (k >> (2 * P.y)) & 3, kx = (k >> (2 * P.x)) & 3, kc = (k >> (2 * P.c)) & 3;
            const double *a = t1 + (4 * ky + kx) * kBlkStride + 4 * jy;
            const double *b = t2 + 4 * kc * kBlkStride + 4 * jc;
            if (P.single) {
                u[c] = b[0] * a[jx];
            } else {
                u[c] = b[jx] * a[0];
#pragma unroll
                for (int m = 1; m < 4; ++m) u[c] = fma(b[m * kBlkStride + jx], a[m], u[c]);
            }
        }
    };
    auto images = [&](int j) {
        const uint32_t pos = uint32_t(k0 >> 3) * 64 + uint32_t(k0 & 7) + uint32_t(j & 7) * 8 + uint32_t(j >> 3) * 512;
        Chunk h2, l2, s2;
#pragma unroll
        for (int c = 0; c < C; c += 2) {
            uint16_t h0, h1, l0, l1;
            split_bits(u[c], h0, l0);
            split_bits(u[c + 1], h1, l1);
            h2.v[c >> 1] = uint32_t(h0) | (uint32_t(h1) << 16);
            l2.v[c >> 1] = uint32_t(l0) | (uint32_t(l1) << 16);
            const __half2 s = __floats2half2_rn(__half2float(__ushort_as_half(h0)) * kLoScale,
                                                __half2float(__ushort_as_half(h1)) * kLoScale);
            s2.v[c >> 1] = *reinterpret_cast<const uint32_t *>(&s);
        }
        if (three) *reinterpret_cast<Chunk *>(img + pos) = s2;
        *reinterpret_cast<Chunk *>(img + 4096 + pos) = l2;
        *reinterpret_cast<Chunk *>(img + uh + pos) = h2;
    };
    if (!more) {
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            entries(lane + 32 * half);
            images(lane + 32 * half);
        }
        return;
    }
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        entries(lane + 32 * half);
#pragma unroll
        for (int c = 0; c < C; ++c) w[c * kColStride + lane + 32 * half] = u[c];
    }
    __syncwarp();
    for (int i = P.stop; i < P.end; ++i) {
        const dm_op &op = cs.ops[i];
        const int da = (op.flags >> 8) & 3, db = (op.flags >> 12) & 3;
        if (op.kind == DM_OP_MAP1) {
            double m[16];
            bool row0, xy;
            load_map(m, op_coefs<Map2>(cs, mats, i), row0, xy);
            const int S = 1 << (2 * da), g = lane & 15;
            double *col = w + (lane >> 4) * kColStride + (((g >> (2 * da)) << (2 * da + 2)) | (g & (S - 1)));
#pragma unroll
            for (int it = 0; it < C / 2; ++it) map1_at(col + 2 * it * kColStride, S, m, row0, xy);
        } else if (lane < 4 * C) {     // lane = (column, value of the third digit)
            pair_at<Map2>(w + (lane >> 2) * kColStride + (lane & 3) * (1 << (2 * (3 - da - db))), 1 << (2 * da),
                          1 << (2 * db), op, op_coefs<Map2>(cs, mats, i));
        }
        __syncwarp();
    }
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int c = 0; c < C; ++c) u[c] = w[c * kColStride + lane + 32 * half];
        images(lane + 32 * half);
    }
    __syncwarp();   // the columns are read before the next item's are written
}

// A batched pass's composition works in the operand region, which is free between passes: the blocks of
// up to kBlockRounds rounds, the warps' columns, the operations.
constexpr int kBlockRounds = 8;
struct ComposeWork {
    double blocks[kBlockRounds * 2 * kBlkDoubles];
    double cols[kThreads / 32 * 8 * kColStride];
    ComposeShared cs;
};
static_assert(sizeof(ComposeWork) <= kSmemBytes, "blocks, columns and operations fit the pass's shared memory");

// This CTA's share of a batched pass's round images (three per round): the group's ranks take equal runs
// of (round, columns) items and compose the blocks of their own rounds; alone a CTA takes 8 columns per
// warp and whole blocks, in a group 2 and half blocks, for the work is then spread thinner than the warps.
template <int C>
__device__ void compose_items(ComposeWork &cw, int nrounds, uint16_t *__restrict__ umats, int rank, int G) {
    constexpr int kPer = 64 / C, nc = C == 8 ? 16 : 8;       // items of a round, columns of a block unit
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = kThreads / 32;
    const int total = nrounds * kPer, first = total * rank / G, last = total * (rank + 1) / G;
    for (int rb = first / kPer; rb * kPer < last; rb += kBlockRounds) {
        const int re = min(rb + kBlockRounds, (last + kPer - 1) / kPer);
        for (int i = warp; i < (re - rb) * 2 * (16 / nc); i += warps) {
            const int b = i / (16 / nc);
            compose_block<false>(cw.cs, cw.cs.plan[rb + (b >> 1)], nullptr, b & 1, i % (16 / nc) * nc, nc,
                                 cw.blocks + b * kBlkDoubles, lane);
        }
        __syncthreads();
        for (int i = max(first, rb * kPer) + warp; i < min(last, re * kPer); i += warps) {
            const int r = i / kPer, b = 2 * (r - rb);
            compose_cols<false, C>(cw.cs, cw.cs.plan[r], nullptr, cw.blocks + b * kBlkDoubles,
                                   cw.blocks + (b + 1) * kBlkDoubles, i % kPer * C, cw.cols + warp * C * kColStride,
                                   umats + int64_t(r) * kUHalves, true, lane);
        }
        __syncthreads();
    }
}

__device__ __noinline__ void compose_share(const dm_batch_pass &bp, const double *mats, uint16_t *umats,
                                           unsigned char *smem, int rank, int G) {
    ComposeWork &cw = *reinterpret_cast<ComposeWork *>(smem);
    const int nr = bp.nrounds;
    compose_load(cw.cs, bp, mats, 0, nr);
    if (G < 8)
        compose_items<8>(cw, nr, umats, rank, G);
    else
        compose_items<2>(cw, nr, umats, rank, G);
}

// ---------------------------------------------------------------------------
// groups of CTAs
//
// G CTAs (a group) run one instance together: each takes every G-th tile of a
// pass and its share of the round-matrix composition, with one barrier among
// the group per pass.  One CTA per instance leaves a sweep waiting for its
// largest instance (a 12-qubit, 47-layer one takes a CTA 0.4 s) and keeps 304
// states in flight, far more than L2 holds; with groups the tail is a G-th of
// that and up to 10 qubits the states in flight stay in L2 (19 groups of 16
// CTAs x 4 MB).  Measured: a batch of 576 instances of 6-12 qubits whose
// largest ones are the longest, 511 -> 362 ms; 1,024 points of a 10-qubit
// template, 3.4 waves of CTAs, 79.5 -> 78.0 ms.  A pass costs a group about
// 20 us beside its tiles (16 us each where two CTAs share an SM), so work that
// fills the chip evenly stays at one CTA per instance.
//
// A cooperative launch does not take two CTAs per SM of a kernel that
// allocates tensor memory, so groups form among CTAs that run already: a CTA
// joins the group of its ticket, and the first member closes the group when it
// is full or, with the chip shared and CTAs still to come, after kJoinNs with
// the members it has (later ones leave).  A group therefore only ever waits
// for running CTAs.  Every wait is bounded and ends in *status = 1.
// ---------------------------------------------------------------------------

struct GroupSync {
    unsigned joined;                  // members so far, kClosed once the first member closed the group
    unsigned size;                    // members of the closed group
    unsigned arrived;                 // barrier arrivals since the launch began
    int inst;                         // instance the group runs next
    unsigned pad[28];                 // one 128-byte line per group
};
constexpr unsigned kClosed = 0x80000000u;
constexpr uint64_t kJoinNs = 1000000;

constexpr int kSegSlots = 512;        // template coefficients composed at a time (>= DM_MAX_PASS_OPS)
constexpr int kMaxGroup = 32;
constexpr int kBigQubits = 11, kBigGroup = 8;   // instances that several CTAs share in an uneven batch

// The scratch buffer: round images (two sets per group, or one when a CTA is its own group),
// template coefficients, group counters, the CTA tickets and the launch's abort flag.
struct GroupScratch {
    uint16_t *images;
    double *coefs;
    GroupSync *sync;
    unsigned *tickets;
    int *abort;
};
__host__ __device__ inline size_t scratch_images_bytes(int ctas) { return size_t(ctas) * size_t(kScratchHalves) * 2; }
__host__ __device__ inline size_t scratch_coefs_bytes(int ctas) { return size_t(ctas) * kSegSlots * kCoefStride * 8; }
__host__ __device__ inline size_t scratch_sync_bytes(int ctas) { return (size_t(ctas) + 1) * sizeof(GroupSync); }
__host__ __device__ inline GroupScratch group_scratch(unsigned char *p, int ctas) {
    GroupScratch g;
    g.images = reinterpret_cast<uint16_t *>(p);
    g.coefs = reinterpret_cast<double *>(p + scratch_images_bytes(ctas));
    g.sync = reinterpret_cast<GroupSync *>(p + scratch_images_bytes(ctas) + scratch_coefs_bytes(ctas));
    g.tickets = &(g.sync + ctas)->joined;
    g.abort = &(g.sync + ctas)->inst;
    return g;
}

// One CTA's place in its group (rank < 0: the group was closed without it).
struct Group {
    int id, G, rank;
    GroupSync *sync;
    int *abort;                       // set by any CTA whose wait gave up
    unsigned epoch;                   // barriers passed
};

// Bounded wait of one thread for *word, read with acquire, to satisfy pred.
template <typename Pred>
__device__ __forceinline__ bool group_wait(const unsigned *word, const int *abort, uint64_t limit_ns, Pred pred) {
    const uint64_t t0 = tcg::global_ns();
    for (uint32_t it = 1;; ++it) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if (pred(v)) return true;
        if ((it & 15) == 0) {
            if (*static_cast<const volatile int *>(abort) != 0 || tcg::global_ns() - t0 > limit_ns ||
                it >= tcg::kWaitPollCap)
                return false;
            __nanosleep(32);
        }
    }
}

// Joins a group of up to G CTAs (all threads; g in shared memory), or stays alone.
template <bool Grouped>
__device__ __forceinline__ void group_join(const GroupScratch &gs, int G, Group &g) {
    if (threadIdx.x == 0 && !Grouped) {
        g = Group{int(blockIdx.x), 1, 0, gs.sync + blockIdx.x, gs.abort, 0};
    } else if (threadIdx.x == 0) {
        const int id = int(atomicAdd(gs.tickets, 1u)) / G;
        GroupSync *sync = gs.sync + id;
        const unsigned old = atomicAdd(&sync->joined, 1u);
        int rank = old & kClosed ? -1 : int(old), size = 0;
        if (rank == 0) {
            const bool full = group_wait(&sync->joined, gs.abort, kJoinNs, [&](unsigned v) { return v >= unsigned(G); });
            const unsigned members = full ? unsigned(G) : atomicOr(&sync->joined, kClosed);
            size = int(members < unsigned(G) ? members : unsigned(G));
            __threadfence();
            atomicExch(&sync->size, unsigned(size));
        } else if (rank > 0) {
            if (group_wait(&sync->size, gs.abort, tcg::kWaitLimitNs, [](unsigned v) { return v != 0; }))
                size = int(*static_cast<volatile unsigned *>(&sync->size));
            else
                rank = -2;
        }
        g = Group{id, size, rank, sync, gs.abort, 0};
    }
    __syncthreads();
}

// Barrier of the group (all threads): what its CTAs wrote before is visible after.  False when a wait
// gave up here or in another CTA of the launch.
template <bool Grouped>
__device__ __forceinline__ bool group_barrier(Group &g, int *ok_s) {
    __syncthreads();
    if (!Grouped) return true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&g.sync->arrived, 1u);
        const unsigned want = (g.epoch += 1) * unsigned(g.G);
        const bool ok = group_wait(&g.sync->arrived, g.abort, tcg::kWaitLimitNs,
                                   [=](unsigned v) { return int(v - want) >= 0; });
        __threadfence();
        *ok_s = ok ? 1 : 0;
    }
    __syncthreads();
    return *ok_s != 0;
}

// The group's next instance (all threads), or -1 when none is left, -2 when a wait gave up.
template <bool Grouped>
__device__ __forceinline__ int group_next(Group &g, int *counter, int ninst, int *inst_s, int *ok_s) {
    if (threadIdx.x == 0 && (!Grouped || g.rank == 0)) {
        const int i = atomicAdd(counter, 1);
        if (Grouped) *static_cast<volatile int *>(&g.sync->inst) = i;
        *inst_s = i;
    }
    if (!group_barrier<Grouped>(g, ok_s)) return -2;
    if (Grouped) {
        if (threadIdx.x == 0) *inst_s = *static_cast<volatile int *>(&g.sync->inst);
        __syncthreads();
    }
    const int i = *inst_s;
    return i < ninst ? i : -1;
}

// This CTA's part of |0...0>: 2**-n where every digit is I or Z.
__device__ __forceinline__ void group_init_zero(float *st, int n, int rank, int G) {
    const int64_t total = int64_t(1) << (2 * n);
    const float amp = ldexpf(1.0f, -n);
    for (int64_t e = (int64_t(rank) * kThreads + threadIdx.x) * 4; e < total; e += int64_t(G) * kThreads * 4) {
        const uint64_t x = uint64_t(e) ^ (uint64_t(e) >> 1);
        const float v = (x & 0x5555555555555554ull) == 0 ? amp : 0.0f;   // digit 0 of the four values: I, X, Y, Z
        *reinterpret_cast<float4 *>(st + e) = make_float4(v, 0.0f, 0.0f, v);
    }
}

// The single-state launches: CTA (r, c) takes the columns 8c .. 8c + 7 of a round, 2 per warp, after a
// quarter of its blocks per warp.
constexpr int kComposeWarps = 4, kComposeCols = 2, kComposeGrid = 64 / (kComposeWarps * kComposeCols);

__device__ __forceinline__ void compose_round(const dm_batch_pass &bp, int r, const double *__restrict__ mats,
                                              uint16_t *__restrict__ img, bool three) {
    __shared__ ComposeShared cs;
    __shared__ double blocks[2 * kBlkDoubles], cols[kComposeWarps * kComposeCols * kColStride];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    compose_load(cs, bp, mats, r, r + 1);
    compose_block<true>(cs, cs.plan[r], mats, warp >> 1, (warp & 1) * 8, 8, blocks + (warp >> 1) * kBlkDoubles, lane);
    __syncthreads();
    compose_cols<true, kComposeCols>(cs, cs.plan[r], mats, blocks, blocks + kBlkDoubles,
                                     (int(blockIdx.y) * kComposeWarps + warp) * kComposeCols,
                                     cols + warp * kComposeCols * kColStride, img, three, lane);
}

// One pass's round images (CTA x = round of the pass).
__global__ void __launch_bounds__(32 * kComposeWarps)
    compose_pass_kernel(const __grid_constant__ dm_batch_pass bp, const double *__restrict__ mats,
                        uint16_t *__restrict__ images, int image_halves) {
    compose_round(bp, blockIdx.x, mats, images + int64_t(blockIdx.x) * image_halves, image_halves == kUHalves);
}

// The round images of several passes (CTA x = entry of the round table).  A pass's composition alone
// is a launch of a few microseconds on a few dozen warps; one launch for many passes fills the chip
// (20 passes of 10 qubits: 18-25 us each alone, 52 us together; 24 passes of the 14-qubit QFT: 20 us
// per launch of up to 16).
__global__ void __launch_bounds__(32 * kComposeWarps)
    compose_passes_kernel(const dm_batch_pass *__restrict__ passes, const dm_compose_round *__restrict__ rounds,
                          const double *__restrict__ mats, uint16_t *__restrict__ images) {
    const dm_compose_round e = rounds[blockIdx.x];
    compose_round(passes[e.pass], e.round, mats + e.mats_off, images + e.image_off, e.format == DM_IMAGE_TC);
}

// Shared memory of the batched kernels beside the operand and matrix regions.  In a group the tile
// routine is a call of its own (one per pass): inlined into the group's loops it has too few registers
// and spills in the tile loop (10 % of a sweep); with the constants of a lone CTA it has enough.
struct BatchShared {
    Pass ps;
    alignas(16) int64_t hi_off[kTile / 4 / kThreads];
    uint64_t mbar;
    uint32_t tmem, phase;
    int pending, abort_s;
};
constexpr uint32_t kBatchSmemBytes = kSmemBytes + (sizeof(BatchShared) + 15) / 16 * 16 + kAlignSlack;

__device__ __forceinline__ bool batch_tiles_inline(float *st, const uint16_t *umats, int t0, int dt, int *status) {
    unsigned char *smem = aligned_smem();
    BatchShared &b = *reinterpret_cast<BatchShared *>(smem + kSmemBytes);
    TcCta c{smem, smem + kABytes, smem + 2 * kABytes, &b.mbar, b.hi_off, &b.abort_s, b.tmem, b.phase, b.pending != 0};
    const bool ok = tc_pass_tiles(st, b.ps, umats, t0, dt, c, status);
    __syncthreads();      // every thread has read phase and pending
    if (threadIdx.x == 0) {
        b.phase = c.phase;
        b.pending = c.pending ? 1 : 0;
    }
    __syncthreads();
    return ok;
}

__device__ __noinline__ bool batch_tiles_call(float *st, const uint16_t *umats, int t0, int dt, int *status) {
    return batch_tiles_inline(st, umats, t0, dt, status);
}

template <bool Grouped>
__device__ __forceinline__ bool batch_tiles(float *st, const uint16_t *umats, const Group &g, int *status) {
    if constexpr (Grouped)
        return batch_tiles_call(st, umats, g.rank, g.G, status);
    else
        return batch_tiles_inline(st, umats, 0, 1, status);
}

__device__ __forceinline__ BatchShared &batch_setup(unsigned char *smem) {
    BatchShared &b = *reinterpret_cast<BatchShared *>(smem + kSmemBytes);
    TcCta c{smem, smem + kABytes, smem + 2 * kABytes, &b.mbar, b.hi_off, &b.abort_s, 0, 0, false};
    tc_setup(c, &b.tmem);
    if (threadIdx.x == 0) b.phase = b.pending = 0;
    __syncthreads();
    return b;
}

__device__ __forceinline__ void batch_teardown(unsigned char *smem) {
    BatchShared &b = *reinterpret_cast<BatchShared *>(smem + kSmemBytes);
    __syncthreads();
    TcCta c{smem, smem + kABytes, smem + 2 * kABytes, &b.mbar, b.hi_off, &b.abort_s, b.tmem, b.phase, b.pending != 0};
    tc_teardown(c);
}

// Grouped: groups of up to G CTAs per instance; otherwise one CTA per instance (G = 1).
template <bool Grouped>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    batch_tc_kernel(float *__restrict__ states, double *__restrict__ probs, const double *__restrict__ mats,
                    const dm_batch_instance *__restrict__ insts, int ninst, const dm_batch_tc_pass *__restrict__ passes,
                    int *counter, unsigned char *__restrict__ scratch, int ctas, int G, int *status) {
    unsigned char *smem = aligned_smem();
    __shared__ int inst_s, ok_s;
    __shared__ Group g;
    __shared__ dm_batch_instance I;
    __shared__ unsigned npass_s;
    BatchShared &b = batch_setup(smem);
    group_join<Grouped>(group_scratch(scratch, ctas), G, g);
    if (threadIdx.x == 0) npass_s = 0;
    bool ok = g.rank != -2;
    while (g.rank >= 0) {
        const int ii = group_next<Grouped>(g, counter, ninst, &inst_s, &ok_s);
        if (ii < 0) {
            ok = ii == -1;
            break;
        }
        if (threadIdx.x == 0) I = insts[ii];
        __syncthreads();
        const int rank = Grouped ? g.rank : 0, members = Grouped ? g.G : 1;
        float *st = states + I.state_off;
        group_init_zero(st, I.n, rank, members);
        for (int pi = 0; pi < I.npasses && ok; ++pi) {
            const dm_batch_tc_pass &bp = passes[I.pass_begin + pi];
            // in a group the next pass's images are composed while this one's are read: two sets
            uint16_t *umats = group_scratch(scratch, ctas).images +
                              int64_t(Grouped ? g.id * G + int(npass_s & 1) : g.id) * kScratchHalves;
            batch_tc_setup(b.ps, bp, I.n);
            compose_share(bp.ops, mats + I.mats_off, umats, smem, rank, members);
            ok = group_barrier<Grouped>(g, &ok_s);
            if (Grouped && threadIdx.x == 0) npass_s += 1;
            if (ok) ok = batch_tiles<Grouped>(st, umats, g, status);
        }
        if (ok) ok = group_barrier<Grouped>(g, &ok_s);
        if (!ok) break;
        if (rank == 0)
            batch_z_readout<float, kThreads>(st, I.n, I.meas_err, probs + I.prob_off, reinterpret_cast<double *>(smem));
    }
    if (!ok && threadIdx.x == 0) {
        atomicExch(g.abort, 1);
        atomicExch(status, 1);
    }
    batch_teardown(smem);
}

// Template sweeps on the tensor cores: per instance the slots' recipe chains
// are composed in FP64, up to kSegSlots of them at a time and shared among the
// group's threads, the round matrices from those coefficients, then the tiles
// streamed.  Slot s of the program is op s of the concatenated tensor-core
// passes; op o of a pass reads 16 coefficients at 16 o.
template <bool Grouped>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    batch_param_tc_kernel(float *__restrict__ states, double *__restrict__ probs, const dm_param_program P,
                          const dm_batch_tc_pass *__restrict__ passes, const double *__restrict__ params,
                          int params_stride, int ninst, int *counter, unsigned char *__restrict__ scratch, int ctas,
                          int G, int *status) {
    unsigned char *smem = aligned_smem();
    __shared__ int inst_s, ok_s;
    __shared__ double prm[DM_PARAMS_MIN_STRIDE];
    __shared__ Group g;
    __shared__ int slot, seg_begin, seg_end;          // the pass's first slot; slots in coefs
    __shared__ unsigned npass_s;
    BatchShared &b = batch_setup(smem);
    group_join<Grouped>(group_scratch(scratch, ctas), G, g);
    const int tid = threadIdx.x;
    if (tid == 0) npass_s = 0;
    bool ok = g.rank != -2;
    while (g.rank >= 0) {
        const int ii = group_next<Grouped>(g, counter, ninst, &inst_s, &ok_s);
        if (ii < 0) {
            ok = ii == -1;
            break;
        }
        if (tid < DM_PARAMS_MIN_STRIDE) prm[tid] = params[int64_t(ii) * params_stride + tid];
        if (tid == 0) slot = seg_begin = seg_end = 0;
        __syncthreads();
        const int rank = Grouped ? g.rank : 0, members = Grouped ? g.G : 1;
        float *st = states + (int64_t(ii) << (2 * P.n));
        group_init_zero(st, P.n, rank, members);
        for (int pi = 0; pi < P.npasses && ok; ++pi) {
            const dm_batch_tc_pass &bp = passes[pi];
            double *coefs = group_scratch(scratch, ctas).coefs + int64_t(g.id) * kSegSlots * kCoefStride;
            if (slot + bp.ops.nops > seg_end) {
                // the next passes' slots; the last barrier lies after every read of the previous ones
                __syncthreads();
                if (tid == 0) {
                    int end = slot;
                    for (int q = pi; q < P.npasses && end + passes[q].ops.nops - slot <= kSegSlots; ++q)
                        end += passes[q].ops.nops;
                    seg_begin = slot;
                    seg_end = end;
                }
                __syncthreads();
                for (int i = seg_begin + rank * kThreads + tid; i < seg_end; i += members * kThreads)
                    compose_slot(P, i, prm, coefs + (i - seg_begin) * kCoefStride);
                if (!(ok = group_barrier<Grouped>(g, &ok_s))) break;
            }
            uint16_t *umats = group_scratch(scratch, ctas).images +
                              int64_t(Grouped ? g.id * G + int(npass_s & 1) : g.id) * kScratchHalves;
            batch_tc_setup(b.ps, bp, P.n);
            compose_share(bp.ops, coefs + (slot - seg_begin) * kCoefStride, umats, smem, rank, members);
            ok = group_barrier<Grouped>(g, &ok_s);
            if (tid == 0) {
                npass_s += 1;
                slot += bp.ops.nops;
            }
            if (ok) ok = batch_tiles<Grouped>(st, umats, g, status);
        }
        if (ok) ok = group_barrier<Grouped>(g, &ok_s);
        if (!ok) break;
        if (rank == 0)
            batch_z_readout<float, kThreads>(st, P.n, prm[11], probs + (int64_t(ii) << P.n),
                                             reinterpret_cast<double *>(smem));
    }
    if (!ok && tid == 0) {
        atomicExch(g.abort, 1);
        atomicExch(status, 1);
    }
    batch_teardown(smem);
}

// The largest power of two of CTAs per instance, up to kMaxGroup, that ninst instances keep busy.
static int spread_group(int ctas, int ninst) {
    int G = 1;
    while (2 * G <= kMaxGroup && 2 * G * ninst <= ctas) G *= 2;
    return G;
}

}  // namespace tc

}  // namespace dmg

using namespace dmg;

constexpr int kBatchTcMaxQubits = 12;   // the Z read-out's 2**n doubles fit the operand region

// Offsets must be distinct powers of two (operand) so that their XOR stays inside
// a 32 KB operand image, or natural-tile element offsets below 4**7.
static bool valid_tables(const uint32_t *rowc, const uint32_t *kc, int vec, bool natural) {
    uint32_t seen = 0;
    for (int i = 0; i < 14; ++i) {
        const uint32_t c = i < 8 ? rowc[i] : kc[i - 8];
        if (natural) {
            if (c == 0 || c >= uint32_t(tc::kTile)) return false;
        } else {
            if (c == 0 || (c & (c - 1)) || c >= tc::kABytes || (seen & c)) return false;
            seen |= c;
        }
    }
    if (vec >= 0) {
        if (vec > 2) return false;
        // natural: four FP32 elements (16 bytes); operand: four FP16 values (8 bytes)
        const uint32_t lo = natural ? 1 : 2, hi = natural ? 2 : 4, align = natural ? 4 : 8;
        if (kc[2 * vec] != lo || kc[2 * vec + 1] != hi) return false;
        for (int i = 0; i < 14; ++i) {   // the other bits keep 16-byte alignment
            if (i >= 8 && (i - 8) / 2 == vec) continue;
            const uint32_t c = i < 8 ? rowc[i] : kc[i - 8];
            if (c % align) return false;
        }
    }
    return true;
}

// A direct last round's tables: the linear natural offsets 2**b of 14 distinct tile bits, rows 0-3
// on tile bits 0-3 (lanes 0-15 of a warp store 16 contiguous coefficients).
static bool direct_tables(const uint32_t *rowc, const uint32_t *kc) {
    uint32_t seen = 0;
    for (int i = 0; i < 14; ++i) {
        const uint32_t c = i < 8 ? rowc[i] : kc[i - 8];
        if (c == 0 || (c & (c - 1)) || c >= uint32_t(tc::kTile) || (seen & c)) return false;
        seen |= c;
    }
    return (rowc[0] | rowc[1] | rowc[2] | rowc[3]) == 15u;
}

extern "C" int dm_apply_pass_tc(void *state_dev, int n, const dm_tc_pass *pass, const uint16_t *umats_dev,
                                size_t umats_count, int *status_dev, void *stream) {
    DM_CHECK_ARG(state_dev && pass && umats_dev && status_dev && valid_n(n));
    if (reinterpret_cast<uintptr_t>(state_dev) & 15 || reinterpret_cast<uintptr_t>(umats_dev) & 15) return DM_ERR_ARG;
    if (n < tc::kAxes) return DM_ERR_PROGRAM;
    const int nr = pass->nrounds;
    if (nr < 1 || nr > DM_MAX_ROUNDS) return DM_ERR_PROGRAM;
    static thread_local tc::Pass p;   // ~3.5 KB: keep it off the host stack
    bool resident[DM_MAX_QUBITS] = {false};
    for (int r = 0; r < tc::kAxes; ++r) {
        const int q = pass->axes[r];
        if (q < 0 || q >= n || (r > 0 && q >= pass->axes[r - 1])) return DM_ERR_PROGRAM;
        resident[q] = true;
        p.res_stride[r] = axis_stride(n, q);
    }
    int low = 0;
    while (low < tc::kAxes && pass->axes[low] == n - 1 - low) ++low;
    if (low < 1) return DM_ERR_PROGRAM;   // 16-byte chunks need the lowest axis resident
    p.low = low;
    p.n = n;
    p.m = n - tc::kAxes;
    p.up = float(ldexp(1.0, n));
    p.down = float(ldexp(1.0, -n));
    int m = 0;
    for (int q = n - 1; q >= 0; --q)
        if (!resident[q]) p.nonres_stride[m++] = axis_stride(n, q);
    for (int u = m; u < DM_MAX_QUBITS; ++u) p.nonres_stride[u] = 0;
    p.nrounds = nr;
    p.vec0 = pass->vec0 == 0 ? 0 : -1;
    p.direct = pass->direct_last ? 1 : 0;
    if (pass->direct_last != 0 && pass->direct_last != 1) return DM_ERR_PROGRAM;
    // round 0 conversion reads: natural offsets of round 0's bits
    if (!valid_tables(pass->natrow, pass->natk, p.vec0, true)) return DM_ERR_PROGRAM;
    for (int i = 0; i < 8; ++i) p.natrow[i] = pass->natrow[i];
    for (int i = 0; i < 6; ++i) p.natk[i] = pass->natk[i];
    for (int r = 0; r < nr; ++r) {
        const dm_tc_round &in = pass->rounds[r];
        tc::Round &o = p.rounds[r];
        for (int i = 0; i < 3; ++i) {
            if (in.digits[i] < 0 || in.digits[i] >= tc::kAxes) return DM_ERR_PROGRAM;
        }
        o.vec = in.vec;
        const bool direct_round = p.direct && r + 1 == nr;
        if (!(direct_round ? direct_tables(in.rowc, in.kc) : valid_tables(in.rowc, in.kc, in.vec, r + 1 == nr)))
            return DM_ERR_PROGRAM;
        const bool operand = r + 1 < nr;
        for (int i = 0; i < 8; ++i) o.rowc[i] = operand ? tc::operand_offset(in.rowc[i]) : in.rowc[i];
        for (int i = 0; i < 6; ++i) o.kc[i] = operand ? tc::operand_offset(in.kc[i]) : in.kc[i];
        if (direct_round) tc::direct_offsets(p, in.rowc, in.kc);
        if (in.umoff < 0 || (in.umoff & 7) || size_t(in.umoff) + tc::kUHalves > umats_count) return DM_ERR_PROGRAM;
        o.umoff = in.umoff;
    }
    constexpr uint32_t smem = tc::kSmemBytes + tc::kAlignSlack;
    if (ensure_max_dynamic_smem(reinterpret_cast<const void *>(tc::pass_tc_kernel), int(smem)) != cudaSuccess)
        return DM_ERR_CUDA;
    const int64_t ntiles = int64_t(1) << (2 * p.m);
    // 88 KB of shared memory, <= 128 registers per thread and 256 TMEM columns per CTA: two CTAs per SM
    int64_t grid = int64_t(sm_count()) * tc::kCtasPerSm;
    if (grid > ntiles) grid = ntiles;
    // An early start at every size: circuits of 6 layers with every pass on this kernel take 63.6 us on 9 qubits
    // (69.7 without), 72.8 (80.0) on 10, 118 (132) on 11, 370 (349, the one loss) on 12, 1.46 ms both ways on 13,
    // 6.07 (6.20) on 14, 25.9 (26.3) on 15 and 108.2 (109.0) on 16.  The TMA-fed passes are another matter.
    return launch_early(tc::pass_tc_kernel, dim3(unsigned(grid)), dim3(tc::kThreads), smem, as_stream(stream),
                        static_cast<float *>(state_dev), p, umats_dev, status_dev);
}

extern "C" size_t dm_batch_tc_scratch_bytes(void) {
    const int ctas = sm_count() * tc::kCtasPerSm;
    return tc::scratch_images_bytes(ctas) + tc::scratch_coefs_bytes(ctas) + tc::scratch_sync_bytes(ctas);
}

// Clears the work counter and the group counters and launches a batched kernel on whole groups of CTAs.
template <typename Kernel, typename... Args>
static int launch_groups(Kernel kernel, int G, int ctas, int *counter_dev, void *scratch_dev, cudaStream_t s,
                         Args... args) {
    if (ensure_max_dynamic_smem(reinterpret_cast<const void *>(kernel), int(tc::kBatchSmemBytes)) != cudaSuccess)
        return DM_ERR_CUDA;
    DM_CUDA_TRY(cudaMemsetAsync(counter_dev, 0, sizeof(int), s));
    DM_CUDA_TRY(cudaMemsetAsync(tc::group_scratch(static_cast<unsigned char *>(scratch_dev), ctas).sync, 0,
                                tc::scratch_sync_bytes(ctas), s));
    kernel<<<ctas / G * G, tc::kThreads, tc::kBatchSmemBytes, s>>>(args...);
    count_launch();
    return launch_status();
}

// The rounds and operations of a tensor-core pass (round_axes[r][0..2] the
// round's local axes in K-digit order, each op on axes of its round, digit
// positions in its flags, coefficients inside mats_len values); 16x16
// general maps only where the caller composes them.
static int validate_round_ops(const dm_batch_pass &o, int64_t mats_len, bool map2) {
    if (o.nrounds < 1 || o.nrounds > DM_MAX_ROUNDS) return DM_ERR_PROGRAM;
    if (o.nops < 0 || o.nops > DM_MAX_PASS_OPS) return DM_ERR_PROGRAM;
    int prev_end = 0;
    for (int r = 0; r < o.nrounds; ++r) {
        for (int i = 0; i < 3; ++i) {
            const int a = o.round_axes[r][i];
            if (a < 0 || a >= tc::kAxes) return DM_ERR_PROGRAM;
            for (int j = 0; j < i; ++j)
                if (o.round_axes[r][j] == a) return DM_ERR_PROGRAM;
        }
        const int end = o.round_end[r];
        if (end < prev_end || end > o.nops) return DM_ERR_PROGRAM;
        for (int i = prev_end; i < end; ++i) {
            const dm_op &op = o.ops[i];
            int64_t need = 0;
            switch (op.kind) {
                case DM_OP_MAP1: need = 16; break;
                case DM_OP_DIAG2: need = 16; break;
                case DM_OP_CX: need = 5; break;
                case DM_OP_MAP2:
                    if (!map2) return DM_ERR_PROGRAM;
                    need = 256;
                    break;
                default: return DM_ERR_PROGRAM;
            }
            if (op.moff < 0 || op.moff + need > mats_len) return DM_ERR_PROGRAM;
            const int da = (op.flags >> 8) & 3, db = (op.flags >> 12) & 3;
            if (op.a < 0 || op.a >= tc::kAxes || da >= 3 || o.round_axes[r][da] != op.a) return DM_ERR_PROGRAM;
            if (op.kind != DM_OP_MAP1 &&
                (op.b < 0 || op.b >= tc::kAxes || op.b == op.a || db >= 3 || db == da || o.round_axes[r][db] != op.b))
                return DM_ERR_PROGRAM;
        }
        prev_end = end;
    }
    return prev_end == o.nops ? DM_OK : DM_ERR_PROGRAM;
}

// One tensor-core batched pass against an instance of n qubits with a coefficient block of mats_len values.
static int validate_batch_tc_pass(const dm_batch_tc_pass &bp, int n, int64_t mats_len) {
    const dm_batch_pass &o = bp.ops;
    if (o.k != tc::kAxes || o.nrounds < 1 || o.nrounds > DM_MAX_ROUNDS) return DM_ERR_PROGRAM;
    if (o.axes[0] != n - 1) return DM_ERR_PROGRAM;   // 16-byte chunks need the lowest axis resident
    for (int r = 0; r < tc::kAxes; ++r)
        if (o.axes[r] < 0 || o.axes[r] >= n || (r > 0 && o.axes[r] >= o.axes[r - 1])) return DM_ERR_PROGRAM;
    const int vec0 = bp.tables.vec0 == 0 ? 0 : -1;
    if (!valid_tables(bp.tables.natrow, bp.tables.natk, vec0, true)) return DM_ERR_PROGRAM;
    if (bp.tables.direct_last != 0 && bp.tables.direct_last != 1) return DM_ERR_PROGRAM;
    for (int r = 0; r < o.nrounds; ++r) {
        const dm_tc_round &tr = bp.tables.rounds[r];
        for (int i = 0; i < 3; ++i)
            if (tr.digits[i] != o.round_axes[r][i]) return DM_ERR_PROGRAM;
        const bool direct_round = bp.tables.direct_last && r + 1 == o.nrounds;
        if (!(direct_round ? direct_tables(tr.rowc, tr.kc) : valid_tables(tr.rowc, tr.kc, tr.vec, r + 1 == o.nrounds)))
            return DM_ERR_PROGRAM;
    }
    return validate_round_ops(o, mats_len, false);
}

extern "C" int dm_compose_rounds(int format, const dm_batch_pass *pass, const double *mats_dev, size_t mats_count,
                                 uint16_t *images_dev, size_t images_count, void *stream) {
    DM_CHECK_ARG(pass && mats_dev && images_dev && (format == DM_IMAGE_TC || format == DM_IMAGE_TMA));
    if (reinterpret_cast<uintptr_t>(images_dev) & 15 || reinterpret_cast<uintptr_t>(mats_dev) & 7) return DM_ERR_ARG;
    if (mats_count > size_t(INT32_MAX)) return DM_ERR_RANGE;
    const int rc = validate_round_ops(*pass, int64_t(mats_count), true);
    if (rc) return rc;
    const int halves = format == DM_IMAGE_TC ? tc::kUHalves : 2 * 4096;
    if (images_count < size_t(pass->nrounds) * size_t(halves)) return DM_ERR_ARG;
    tc::compose_pass_kernel<<<dim3(pass->nrounds, tc::kComposeGrid), 32 * tc::kComposeWarps, 0, as_stream(stream)>>>(
        *pass, mats_dev, images_dev, halves);
    count_launch();
    return launch_status();
}

extern "C" int dm_compose_passes(const dm_batch_pass *passes_host, const dm_batch_pass *passes_dev, int npasses,
                                 const dm_compose_round *rounds_host, const dm_compose_round *rounds_dev, int nrounds,
                                 const double *mats_dev, size_t mats_count, uint16_t *images_dev, size_t images_count,
                                 void *stream) {
    DM_CHECK_ARG(passes_host && passes_dev && rounds_host && rounds_dev && mats_dev && images_dev && npasses >= 1 &&
                 nrounds >= 1);
    if (reinterpret_cast<uintptr_t>(images_dev) & 15 || reinterpret_cast<uintptr_t>(mats_dev) & 7) return DM_ERR_ARG;
    if (mats_count > size_t(INT32_MAX)) return DM_ERR_RANGE;
    for (int i = 0; i < nrounds; ++i) {
        const dm_compose_round &e = rounds_host[i];
        if (e.pass < 0 || e.pass >= npasses) return DM_ERR_ARG;
        if (e.format != DM_IMAGE_TC && e.format != DM_IMAGE_TMA) return DM_ERR_ARG;
        if (e.mats_off < 0 || size_t(e.mats_off) > mats_count) return DM_ERR_ARG;
        // the rounds of a pass follow one another with one coefficient offset: the pass is checked once
        if (i == 0 || e.pass != rounds_host[i - 1].pass || e.mats_off != rounds_host[i - 1].mats_off) {
            const int rc = validate_round_ops(passes_host[e.pass], int64_t(mats_count) - e.mats_off, true);
            if (rc) return rc;
        }
        if (e.round < 0 || e.round >= passes_host[e.pass].nrounds) return DM_ERR_PROGRAM;
        const int64_t halves = e.format == DM_IMAGE_TC ? tc::kUHalves : 2 * 4096;
        if (e.image_off < 0 || (e.image_off & 7) || size_t(e.image_off + halves) > images_count) return DM_ERR_ARG;
    }
    tc::compose_passes_kernel<<<dim3(nrounds, tc::kComposeGrid), 32 * tc::kComposeWarps, 0, as_stream(stream)>>>(
        passes_dev, rounds_dev, mats_dev, images_dev);
    count_launch();
    return launch_status();
}

extern "C" int dm_batch_run_tc(float *states_dev, size_t states_count, double *probs_dev, size_t probs_count,
                               const double *mats_dev, size_t mats_count, const dm_batch_instance *insts_host,
                               const dm_batch_instance *insts_dev, int ninst, const dm_batch_tc_pass *passes_host,
                               const dm_batch_tc_pass *passes_dev, int npasses, int *counter_dev, void *scratch_dev,
                               size_t scratch_bytes, int *status_dev, void *stream) {
    DM_CHECK_ARG(states_dev && probs_dev && mats_dev && insts_host && insts_dev && passes_host && passes_dev &&
                 counter_dev && scratch_dev && status_dev && ninst >= 1 && npasses >= 1);
    if (reinterpret_cast<uintptr_t>(states_dev) & 15 || reinterpret_cast<uintptr_t>(scratch_dev) & 15) return DM_ERR_ARG;
    for (int i = 0; i < ninst; ++i) {
        const dm_batch_instance &I = insts_host[i];
        if (I.n < tc::kAxes || I.n > kBatchTcMaxQubits) return DM_ERR_RANGE;
        const int64_t total = int64_t(1) << (2 * I.n);
        if (I.state_off < 0 || (I.state_off & 3) || size_t(I.state_off + total) > states_count) return DM_ERR_ARG;
        if (I.prob_off < 0 || size_t(I.prob_off + (int64_t(1) << I.n)) > probs_count) return DM_ERR_ARG;
        if (I.mats_off < 0 || I.mats_len < 0 || size_t(I.mats_off + I.mats_len) > mats_count) return DM_ERR_ARG;
        if (I.npasses < 0 || I.pass_begin < 0 || I.pass_begin + I.npasses > npasses) return DM_ERR_PROGRAM;
        for (int p = 0; p < I.npasses; ++p) {
            const int rc = validate_batch_tc_pass(passes_host[I.pass_begin + p], I.n, I.mats_len);
            if (rc) return rc;
        }
    }
    if (scratch_bytes < dm_batch_tc_scratch_bytes()) return DM_ERR_ARG;
    // One CTA per instance is the faster form while the work is even: a batch then takes its total over
    // the CTAs.  It cannot take less than its largest instance, so where that is the longer of the two
    // (4096 mixed instances: 0.65 of the total's share; 576: 1.8) the leading large ones (the caller
    // orders them largest first) run on groups of kBigGroup; and what does not fill the chip, on
    // groups that do.
    const int ctas = sm_count() * tc::kCtasPerSm;
    double total = 0, largest = 0;
    int big = 0;
    for (int i = 0; i < ninst; ++i) {
        const double w = ldexp(double(insts_host[i].npasses), 2 * insts_host[i].n);
        total += w;
        largest = w > largest ? w : largest;
        if (big == i && insts_host[i].n >= tc::kBigQubits) ++big;
    }
    if (largest * ctas <= total) big = 0;
    for (int part = 0; part < 2; ++part) {
        const int begin = part ? big : 0, count = part ? ninst - big : big;
        if (count == 0) continue;
        int G = tc::spread_group(ctas, count);
        if (!part && G < tc::kBigGroup) G = tc::kBigGroup;
        const int e = launch_groups(G > 1 ? tc::batch_tc_kernel<true> : tc::batch_tc_kernel<false>, G, ctas, counter_dev,
                                    scratch_dev, as_stream(stream), states_dev, probs_dev, mats_dev, insts_dev + begin,
                                    count, passes_dev, counter_dev, static_cast<unsigned char *>(scratch_dev), ctas, G,
                                    status_dev);
        if (e) return e;
    }
    return DM_OK;
}

extern "C" int dm_batch_run_params_tc(const dm_param_program *host, const dm_param_program *dev,
                                      const dm_batch_tc_pass *passes_host, const dm_batch_tc_pass *passes_dev,
                                      const double *params_dev, int params_stride, int ninst, float *states_dev,
                                      size_t states_count, double *probs_dev, size_t probs_count, int *counter_dev,
                                      void *scratch_dev, size_t scratch_bytes, int *status_dev, void *stream) {
    DM_CHECK_ARG(host && dev && passes_host && passes_dev && params_dev && states_dev && probs_dev && counter_dev &&
                 scratch_dev && status_dev);
    DM_CHECK_ARG(ninst >= 1 && params_stride >= DM_PARAMS_MIN_STRIDE);
    if (reinterpret_cast<uintptr_t>(states_dev) & 15 || reinterpret_cast<uintptr_t>(scratch_dev) & 15) return DM_ERR_ARG;
    const dm_param_program &P = *host;
    if (P.n < tc::kAxes || P.n > kBatchTcMaxQubits) return DM_ERR_RANGE;
    if (P.npasses < 1) return DM_ERR_PROGRAM;
    for (int p = 0; p < P.npasses; ++p) {
        // op o of a pass reads the o-th 16-value slot of the shared-memory coefficients
        const dm_batch_pass &o = passes_host[p].ops;
        if (o.nops < 0 || o.nops > DM_MAX_PASS_OPS) return DM_ERR_PROGRAM;
        for (int i = 0; i < o.nops; ++i)
            if (o.ops[i].moff != i * kCoefStride) return DM_ERR_PROGRAM;
        const int rc = validate_batch_tc_pass(passes_host[p], P.n, int64_t(o.nops) * kCoefStride);
        if (rc) return rc;
    }
    const int rc = validate_param_slots(
        P, P.npasses, [&](int p) { return int(passes_host[p].ops.nops); },
        [&](int p, int o) { return passes_host[p].ops.ops[o].kind; });
    if (rc) return rc;
    if (host->n != dev->n || host->npasses != dev->npasses || host->nslots != dev->nslots) return DM_ERR_ARG;
    if (size_t(ninst) * (size_t(1) << (2 * P.n)) > states_count) return DM_ERR_ARG;
    if (size_t(ninst) * (size_t(1) << P.n) > probs_count) return DM_ERR_ARG;
    if (scratch_bytes < dm_batch_tc_scratch_bytes()) return DM_ERR_ARG;
    // whole waves of one instance per CTA, then what is left on groups that fill the chip
    const int ctas = sm_count() * tc::kCtasPerSm;
    const int whole = tc::spread_group(ctas, ninst % ctas) > 1 ? ninst / ctas * ctas : ninst;
    for (int part = 0; part < 2; ++part) {
        const int begin = part ? whole : 0, count = part ? ninst - whole : whole;
        if (count == 0) continue;
        const int G = part ? tc::spread_group(ctas, count) : 1;
        const int e = launch_groups(
            G > 1 ? tc::batch_param_tc_kernel<true> : tc::batch_param_tc_kernel<false>, G, ctas, counter_dev, scratch_dev,
            as_stream(stream), states_dev + (int64_t(begin) << (2 * P.n)), probs_dev + (int64_t(begin) << P.n), *dev, passes_dev,
            params_dev + int64_t(begin) * params_stride, params_stride, count, counter_dev,
            static_cast<unsigned char *>(scratch_dev), ctas, G, status_dev);
        if (e) return e;
    }
    return DM_OK;
}
