// Memory noise of one clock cycle on every qubit (dm_simulator.py:397-425):
// on each Pauli axis X, Y <- sqrt(g) f (X, Y) and Z <- g Z + (1-g)(2p-1) I.
//
// The reference sweeps the state once per qubit.  Here a sweep holds several
// axes: a CTA loads a tile of 4**K coefficients (times a 64-byte contiguous
// run, unless the axes are the lowest ones) into shared memory, runs two axes
// at a time in registers (16 coefficients per thread) and writes the tile
// back, so n qubits take one sweep up to kMaxLow axes and two to four above.
// FP32 is bound by HBM, FP64 by the FP64 pipe (two FMAs per clock and SM), so
// the scale factors are taken out of the axes where g allows (Defer): with
// k = sqrt(g) f and c = (1-g)(2p-1)/g an axis is (I, X, Y, Z) -> (I, X, Y,
// Z + c I), one FMA per four coefficients, followed by a factor 1, k, k, g;
// the factors of all axes are one product k**#XY g**#Z per coefficient, taken
// from a table as the last sweep writes back.  That is n/4 + 1 FP64
// operations per coefficient instead of n.  Defer needs c to stay small (the
// unscaled Z grows like g**-n), so it is used for g >= 1/2, which every
// physical decay factor per cycle is; below that, and on a few qubits, each
// axis is scaled at once.
// Measured for all qubits: n = 13 FP64 672 us in three sweeps (6.8 ms as 13),
// n = 14 FP32 1.32 ms in three (4.5 ms as 14, each at the HBM roof).
#include <math.h>

#include "dm_common.cuh"

namespace dmg {

namespace noise {

constexpr int kThreads = 256;
constexpr int kMaxLow = 6;         // axes of a sweep over the lowest axes: 16 / 32 KB tiles
constexpr int kMaxHigh = 4;        // axes of a sweep above them: 256 rows of 16 contiguous elements and more
constexpr int kMaxTile = 1 << (2 * kMaxLow);
// Up to this many qubits each axis is scaled at once: the call is host time, and the table of factors (324
// values, 2.6 KB of kernel parameters in FP64) is more of it than the few FP64 operations it saves.  One
// qubit: 9.8 us a call with the table from 648 calls of pow, 4.1 with it from 2 n + 2, 3.3 without it.
constexpr int kFewQubits = 4;

template <typename T, bool Defer>
struct Args {
    T k, g, d;
};
template <typename T>
struct Args<T, true> {
    T c;
    T scale[DM_MAX_QUBITS + 1][DM_MAX_QUBITS + 1];   // k**a g**b for a X/Y and b Z digits
};

// Position of tile element e in shared memory: 16-byte chunks stay whole, the chunk index inside
// a 128-byte row is XORed with the next rows' bits so that strided groups spread over the banks.
template <typename T>
__device__ __forceinline__ int swz(int e) {
    constexpr int C = sizeof(T) == 4 ? 2 : 1;
    return e ^ ((((e >> (C + 3)) ^ (e >> (C + 6))) & 7) << C);
}

// X/Y and Z digits of a coefficient index (digits I 00, X 01, Y 10, Z 11)
__device__ __forceinline__ void count_digits(uint64_t i, int &xy, int &z) {
    const uint64_t even = 0x5555555555555555ull, lo = i & even, hi = (i >> 1) & even;
    xy = __popcll(lo ^ hi);
    z = __popcll(lo & hi);
}

// One axis of four coefficients
template <typename T, bool Defer>
__device__ __forceinline__ void axis(const Args<T, Defer> &a, T &x0, T &x1, T &x2, T &x3) {
    if constexpr (Defer) {
        x3 = fma(a.c, x0, x3);
    } else {
        x1 *= a.k;
        x2 *= a.k;
        x3 = fma(a.g, x3, a.d * x0);
    }
}

// One sweep over axes lo .. lo + K - 1 (digit positions) of a tile of 4**K rows of 2**rlog
// contiguous elements (rlog = 0 when lo = 0: the tile itself is contiguous).  The top axis is applied
// as the tile loads and the one below it as it leaves, each thread holding the four rows of a group,
// so that shared memory carries only the axes between them; in FP32 over the lowest axes a
// 16-byte access holds axis 0 whole, applied on load too.  Vec: 16-byte global accesses.
template <typename T, bool Defer, bool Vec>
__global__ void __launch_bounds__(kThreads) sweep_kernel(T *__restrict__ st, int K, int lo, int rlog, int last,
                                                         const __grid_constant__ Args<T, Defer> a) {
    __shared__ __align__(16) T tile[kMaxTile];
    __shared__ T scale[DM_MAX_QUBITS + 1][DM_MAX_QUBITS + 1];
    constexpr int V = Vec ? 16 / int(sizeof(T)) : 1;
    struct alignas(Vec ? 16 : alignof(T)) Pack {
        T v[V];
    };
    const int tsize = 1 << (2 * K + rlog);
    const int tid = threadIdx.x;
    // tile b: outer digits above the axes, then the run inside the 4**lo contiguous block
    const int runs_log = 2 * lo - rlog;
    const int64_t b = blockIdx.x;
    const int64_t base = ((b >> runs_log) << (2 * (lo + K))) + ((b & ((int64_t(1) << runs_log) - 1)) << rlog);
    auto offset = [&](int e) { return base + (int64_t(e >> rlog) << (2 * lo)) + (e & ((1 << rlog) - 1)); };
    if constexpr (Defer)
        if (last)
            for (int i = tid; i < (DM_MAX_QUBITS + 1) * (DM_MAX_QUBITS + 1); i += kThreads)
                scale[i / (DM_MAX_QUBITS + 1)][i % (DM_MAX_QUBITS + 1)] =
                    a.scale[i / (DM_MAX_QUBITS + 1)][i % (DM_MAX_QUBITS + 1)];
    // over the lowest axes a pack lies along axis 0: all of it in FP32, half of it in FP64
    const bool along = V > 1 && rlog == 0;
    const bool low_pack = V == 4 && along;
    const int top = 2 * (K - 1) + rlog;            // log2 of the top axis's element stride
    const bool fill_axis = K > 1 || !along;
    if (fill_axis) {
        for (int g = tid * V; g < tsize / 4; g += kThreads * V) {
            Pack x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = *reinterpret_cast<const Pack *>(st + offset(g + (j << top)));
#pragma unroll
            for (int i = 0; i < V; ++i) axis<T, Defer>(a, x[0].v[i], x[1].v[i], x[2].v[i], x[3].v[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (V == 4)
                    if (low_pack) axis<T, Defer>(a, x[j].v[0], x[j].v[1], x[j].v[2], x[j].v[3]);
                *reinterpret_cast<Pack *>(tile + swz<T>(g + (j << top))) = x[j];
            }
        }
    } else {
        for (int e = tid * V; e < tsize; e += kThreads * V) {
            Pack x = *reinterpret_cast<const Pack *>(st + offset(e));
            if constexpr (V == 4) axis<T, Defer>(a, x.v[0], x.v[1], x.v[2], x.v[3]);
            *reinterpret_cast<Pack *>(tile + swz<T>(e)) = x;
        }
    }
    __syncthreads();
    // the axes left, the highest of them on the way out
    const int first = low_pack ? 1 : 0;
    const bool out_axis = K - 2 >= (along ? 1 : 0);
    const int end = out_axis ? K - 2 : fill_axis ? K - 1 : K;   // shared-memory rounds: axes first .. end - 1
    for (int r = first; r < end; r += 2) {
        const int s0 = 2 * r + rlog;
        if (r + 1 < end) {
            for (int g = tid; g < tsize / 16; g += kThreads) {
                const int p = swz<T>(((g >> s0) << (s0 + 4)) | (g & ((1 << s0) - 1)));
                T v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = tile[p ^ swz<T>(j << s0)];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    axis<T, Defer>(a, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) axis<T, Defer>(a, v[j], v[j + 4], v[j + 8], v[j + 12]);
#pragma unroll
                for (int j = 0; j < 16; ++j)   // Defer leaves every entry without a Z digit alone
                    if (!Defer || (j & 3) == 3 || j >= 12) tile[p ^ swz<T>(j << s0)] = v[j];
            }
        } else {
            for (int g = tid; g < tsize / 4; g += kThreads) {
                const int p = swz<T>(((g >> s0) << (s0 + 2)) | (g & ((1 << s0) - 1)));
                T v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = tile[p ^ swz<T>(j << s0)];
                axis<T, Defer>(a, v[0], v[1], v[2], v[3]);
#pragma unroll
                for (int j = Defer ? 3 : 1; j < 4; ++j) tile[p ^ swz<T>(j << s0)] = v[j];
            }
        }
        __syncthreads();
    }
    // way out: groups of four rows along axis K - 2 (or single packs), the deferred factors, the store
    const int so = 2 * (K - 2) + rlog;
    auto finish = [&](int64_t o, Pack &x) {
        if (Defer && last) {
            // digits of the pack's first element; its V elements differ in the lowest digit only
            int xy, z;
            count_digits(uint64_t(o) & ~uint64_t(3), xy, z);
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const int d = V == 4 ? i : (int(o) & 3) + i;
                x.v[i] *= d == 0 ? scale[xy][z] : d == 3 ? scale[xy][z + 1] : scale[xy + 1][z];
            }
        }
        *reinterpret_cast<Pack *>(st + o) = x;
    };
    if (out_axis) {
        for (int g = tid * V; g < tsize / 4; g += kThreads * V) {
            const int e = ((g >> so) << (so + 2)) | (g & ((1 << so) - 1));
            Pack x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = *reinterpret_cast<const Pack *>(tile + swz<T>(e + (j << so)));
#pragma unroll
            for (int i = 0; i < V; ++i) axis<T, Defer>(a, x[0].v[i], x[1].v[i], x[2].v[i], x[3].v[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) finish(offset(e + (j << so)), x[j]);
        }
    } else {
        for (int e = tid * V; e < tsize; e += kThreads * V) {
            Pack x = *reinterpret_cast<const Pack *>(tile + swz<T>(e));
            finish(offset(e), x);
        }
    }
}

template <typename T, bool Defer>
static int run(T *st, int n, const Args<T, Defer> &a, cudaStream_t s) {
    const bool vec = (reinterpret_cast<uintptr_t>(st) & 15) == 0;
    // the fewest sweeps (kMaxLow axes in the first, kMaxHigh in each further one), the axes spread evenly over
    // them.  No other split was timed; where the first sweep is left with 4 axes its CTAs hold 256 coefficients
    // only (n = 7, 8, 11, 12, 15, 16): n = 16 FP32 44.8 ms for four sweeps of 5.05 ms by bytes, 85.6 ms by axis.
    const int sweeps = n <= kMaxLow ? 1 : 1 + (n - kMaxLow + kMaxHigh - 1) / kMaxHigh;
    int lo = 0;
    for (int i = 0; i < sweeps; ++i) {
        const int left = n - lo, after = (sweeps - 1 - i) * kMaxHigh;
        int K = (left + sweeps - 1 - i) / (sweeps - i);
        if (i == 0 && K < left - after) K = left - after;
        if (i > 0 && K > kMaxHigh) K = kMaxHigh;
        // above the lowest axes a tile's rows fill it: 16 elements and more, as far as the 4**lo block goes
        int rlog = lo == 0 ? 0 : 2 * (kMaxLow - K);
        if (rlog > 2 * lo) rlog = 2 * lo;
        const int64_t tiles = pow4(n - K) >> rlog;
        const int last = i == sweeps - 1 ? 1 : 0;
        if (vec)
            sweep_kernel<T, Defer, true><<<unsigned(tiles), kThreads, 0, s>>>(st, K, lo, rlog, last, a);
        else
            sweep_kernel<T, Defer, false><<<unsigned(tiles), kThreads, 0, s>>>(st, K, lo, rlog, last, a);
        count_launch();
        const int rc = launch_status();
        if (rc) return rc;
        lo += K;
    }
    return DM_OK;
}

template <typename T>
static int apply(T *st, int n, double f, double p, double g, cudaStream_t s) {
    const double k = sqrt(g) * f, d = (1 - g) * (2 * p - 1);
    if (n <= kFewQubits || !(g >= 0.5 && fabs(d) <= g)) return run<T, false>(st, n, {T(k), T(g), T(d)}, s);
    Args<T, true> a{};
    a.c = T(d / g);
    double gp[DM_MAX_QUBITS + 1];
    for (int j = 0; j <= n; ++j) gp[j] = pow(g, j);
    for (int i = 0; i <= n; ++i) {
        const double kp = pow(k, i);
        for (int j = 0; i + j <= n; ++j) a.scale[i][j] = T(kp * gp[j]);
    }
    return run<T, true>(st, n, a, s);
}

}  // namespace noise

}  // namespace dmg

using namespace dmg;

extern "C" int dm_apply_memory_noise(void *state_dev, int n, int dtype, double f, double p, double g, void *stream) {
    DM_CHECK_ARG(state_dev && valid_n(n) && valid_dtype(dtype));
    return dtype == DM_F64 ? noise::apply(static_cast<double *>(state_dev), n, f, p, g, as_stream(stream))
                           : noise::apply(static_cast<float *>(state_dev), n, f, p, g, as_stream(stream));
}
