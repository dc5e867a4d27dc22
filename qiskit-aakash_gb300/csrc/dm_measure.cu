// Measurement probabilities (dm_simulator.py:427-538).
//
// For measurement axis col_q (1=X, 2=Y, 3=Z) on qubit q with polarisation
// err, the probability of outcome b is
//     P(b) = sum_{s in {0, col}^n} a_s prod_q w(s_q, b_q),
//     w(0, b) = 1,  w(col, 0) = err,  w(col, 1) = -err,
// the row-times-vector product the reference forms with a 2**n x 2**n
// Kronecker matrix (dm_simulator.py:444-468).  Here: gather the 2**m
// coefficients of the sub-lattice (unmeasured qubits pinned to I, which is
// what summing P over their outcomes leaves, times 2 each), scale by
// err**popcount and apply an in-place Walsh-Hadamard transform.
#include <math.h>

#include <cuda.h>

#include <mutex>

#include "dm_common.cuh"

namespace dmg {

struct SubLattice {
    int m;
    int64_t stride[DM_MAX_QUBITS];   // flat-index step of measured bit j (bit m-1-j of the outcome)
    double errpow[DM_MAX_QUBITS + 1];
    double scale;                    // 2**(n-m)
};

// Walsh-Hadamard butterflies over bits [lo, lo + nb) of the 2**m vector, the
// first sweep (lo = 0) gathering and scaling the sub-lattice as it loads.
// FP64 additions bound a CTA (two per clock and SM: a CTA of 2,048 elements
// and 11 bits took 13.6 us at n = 12), so a CTA takes 1,024 elements: all bits
// of a vector up to 2**10, else at most 7 of them, as 2**nb rows of
// 2**(10 - nb) contiguous elements (lo > 0) or 2**(10 - nb) whole blocks of
// 2**nb (lo = 0).  Measured at n = 12: 16 us for the whole read-out, gather
// included, 23 us before.
constexpr int kWhtBits = 7, kWhtTileLog = 10;

template <typename T, bool Gather>
__global__ void __launch_bounds__(256) wht_kernel(const T *__restrict__ st, const __grid_constant__ SubLattice L,
                                                  double *__restrict__ v, int lo, int nb, int tlog) {
    __shared__ double tile[1 << kWhtTileLog];
    const int tsize = 1 << tlog;
    const int rlog = tlog - nb;              // lo > 0: log2 of the contiguous run of a row
    const int64_t b = blockIdx.x;
    const int runs_log = lo - rlog;
    const int64_t base = Gather ? b << tlog
                                : ((b >> runs_log) << (lo + nb)) | ((b & ((int64_t(1) << runs_log) - 1)) << rlog);
    auto at = [&](int e) { return Gather ? base + e : base + (int64_t(e >> rlog) << lo) + (e & ((1 << rlog) - 1)); };
    for (int e = threadIdx.x; e < tsize; e += blockDim.x) {
        if constexpr (Gather) {
            const int64_t i = base + e;
            int64_t idx = 0;
            int pop = 0;
            for (int j = 0; j < L.m; ++j)
                if ((i >> (L.m - 1 - j)) & 1) {
                    idx += L.stride[j];
                    ++pop;
                }
            tile[e] = double(st[idx]) * L.errpow[pop] * L.scale;
        } else {
            tile[e] = v[at(e)];
        }
    }
    __syncthreads();
    const int s0 = Gather ? 0 : rlog;        // log2 of the first bit's element stride
    for (int k = 0; k < nb; ++k) {
        const int sb = s0 + k;
        for (int p = threadIdx.x; p < tsize / 2; p += blockDim.x) {
            const int i0 = ((p >> sb) << (sb + 1)) | (p & ((1 << sb) - 1));
            const int i1 = i0 | (1 << sb);
            const double x = tile[i0], y = tile[i1];
            tile[i0] = x + y;
            tile[i1] = x - y;
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < tsize; e += blockDim.x) v[at(e)] = tile[e];
}

template <typename T>
static int axis_probs(const T *st, const SubLattice &L, double *v, cudaStream_t s) {
    // the bits of a sweep; above the first one a row's run is 2**(kWhtTileLog - nb) elements
    const int sweeps = L.m <= kWhtTileLog ? 1 : (L.m + kWhtBits - 1) / kWhtBits;
    int lo = 0;
    for (int i = 0; i < sweeps; ++i) {
        const int nb = (L.m - lo + sweeps - 1 - i) / (sweeps - i);
        const int tlog = L.m < kWhtTileLog ? L.m : kWhtTileLog;
        const unsigned grid = unsigned(int64_t(1) << (L.m - tlog));
        if (i == 0)
            wht_kernel<T, true><<<grid, 256, 0, s>>>(st, L, v, lo, nb, tlog);
        else
            wht_kernel<T, false><<<grid, 256, 0, s>>>(st, L, v, lo, nb, tlog);
        count_launch();
        const int rc = launch_status();
        if (rc) return rc;
        lo += nb;
    }
    return DM_OK;
}

// --- basis N: contraction of every axis with the rows [1, +-err n] ----------
//
// One axis: d = err (nx X + ny Y + nz Z), then I + d and I - d: 5 FP64
// operations per four values (the FP64 pipe is the bound, 67 us at n = 12).
// The lowest 6 axes of a 4**6 tile are contracted in shared memory, the rest
// three axes at a time in registers over contiguous runs.  Measured at n = 12
// in FP64: 83 + 19 us, where three axes per thread through local memory and
// one launch per further axis took 182 + 50 us.

struct NRows {
    double w[3];
};

__device__ __forceinline__ void contract(const NRows &R, double i, double x, double y, double z, double &p, double &q) {
    const double d = fma(R.w[2], z, fma(R.w[1], y, R.w[0] * x));
    p = i + d;
    q = i - d;
}

constexpr int kNLow = 6, kNHigh = 3;

// (tiles, 4**t) -> (tiles, 2**t), one tile per CTA.
template <typename T>
__global__ void __launch_bounds__(256) contract_low(const T *__restrict__ st, int t, const __grid_constant__ NRows R,
                                                    double *__restrict__ out) {
    constexpr int kHalf = 1 << (2 * kNLow - 1);
    __shared__ double buf[kHalf + kHalf / 2];
    // the fastest axis as the tile loads; then buf holds rows of 2**j values per remaining index
    const T *src = st + (int64_t(blockIdx.x) << (2 * t));
    for (int g = threadIdx.x; g < 1 << (2 * (t - 1)); g += blockDim.x) {
        double p, q;
        contract(R, double(src[4 * g]), double(src[4 * g + 1]), double(src[4 * g + 2]), double(src[4 * g + 3]), p, q);
        buf[2 * g] = p;
        buf[2 * g + 1] = q;
    }
    __syncthreads();
    double *in = buf, *to = buf + kHalf;
    for (int j = 1; j < t; ++j) {            // (h, 4, 2**j) -> (h, 2, 2**j)
        const int count = 1 << (2 * (t - 1 - j) + j);
        for (int g = threadIdx.x; g < count; g += blockDim.x) {
            const int i = g & ((1 << j) - 1), h = g >> j;
            const double *x = in + ((h << 2) << j) + i;
            double p, q;
            contract(R, x[0], x[1 << j], x[2 << j], x[3 << j], p, q);
            to[((h << 1) << j) + i] = p;
            to[((h << 1 | 1) << j) + i] = q;
        }
        __syncthreads();
        double *tmp = in;
        in = to;
        to = tmp;
    }
    for (int e = threadIdx.x; e < 1 << t; e += blockDim.x) out[(int64_t(blockIdx.x) << t) + e] = in[e];
}

// (outer, 4**K, inner) -> (outer, 2**K, inner), inner = 2**inner_log: one thread per (outer, inner).
template <int K>
__global__ void __launch_bounds__(128) contract_high(const double *__restrict__ in, int64_t count, int inner_log,
                                                     const __grid_constant__ NRows R, double *__restrict__ out) {
    const int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (g >= count) return;
    const int64_t o = g >> inner_log, i = g & ((int64_t(1) << inner_log) - 1);
    double v[1 << (2 * K)];
    const double *src = in + ((o << (2 * K)) << inner_log) + i;
#pragma unroll
    for (int e = 0; e < 1 << (2 * K); ++e) v[e] = src[int64_t(e) << inner_log];
#pragma unroll
    for (int j = 0; j < K; ++j)              // (h, 4, 2**j) -> (h, 2, 2**j), in place front to back
#pragma unroll
        for (int e = 0; e < 1 << (2 * (K - 1 - j) + j); ++e) {
            const int r = e & ((1 << j) - 1), h = e >> j;
            double p, q;
            contract(R, v[(4 * h << j) + r], v[((4 * h + 1) << j) + r], v[((4 * h + 2) << j) + r],
                     v[((4 * h + 3) << j) + r], p, q);
            v[(2 * h << j) + r] = p;
            v[((2 * h + 1) << j) + r] = q;
        }
    double *dst = out + ((o << K) << inner_log) + i;
#pragma unroll
    for (int e = 0; e < 1 << K; ++e) dst[int64_t(e) << inner_log] = v[e];
}

}  // namespace dmg

using namespace dmg;

extern "C" int dm_axis_probs(const void *state_dev, int n, int dtype, const int *mode, double err, double *out_dev,
                             void *stream) {
    DM_CHECK_ARG(state_dev && mode && out_dev && valid_n(n) && valid_dtype(dtype));
    SubLattice L;
    L.m = 0;
    for (int q = 0; q < n; ++q) {
        DM_CHECK_ARG(mode[q] >= 0 && mode[q] <= 3);
        if (mode[q]) L.stride[L.m++] = int64_t(mode[q]) * axis_stride(n, q);
    }
    L.errpow[0] = 1.0;
    for (int j = 1; j <= DM_MAX_QUBITS; ++j) L.errpow[j] = L.errpow[j - 1] * err;
    L.scale = ldexp(1.0, n - L.m);
    cudaStream_t s = as_stream(stream);
    return dtype == DM_F64 ? axis_probs(static_cast<const double *>(state_dev), L, out_dev, s)
                           : axis_probs(static_cast<const float *>(state_dev), L, out_dev, s);
}

static int low_axes(int n) { return n < 3 ? n : 3; }

extern "C" size_t dm_nbasis_probs_scratch_bytes(int n) {
    if (!valid_n(n)) return 0;
    const int t = low_axes(n);
    if (t == n) return 0;
    const size_t first = size_t(pow4(n - t)) << t;   // after contracting the low t axes
    return (first + first / 2) * sizeof(double);
}

// The contractions of dm_nbasis_probs and dm_nbasis_probs_noalloc.  scratch: the two buffers of
// dm_nbasis_probs_scratch_bytes (sized for a three-axis first step; this one contracts up to six).
static int nbasis(const void *state_dev, int n, int dtype, const double *nvec3, double err, double *out_dev,
                  double *scratch, cudaStream_t s) {
    NRows R;
    for (int c = 0; c < 3; ++c) R.w[c] = err * nvec3[c];
    const int t = n < kNLow ? n : kNLow;
    double *bufA = scratch;
    double *bufB = scratch ? scratch + (size_t(pow4(n - low_axes(n))) << low_axes(n)) : nullptr;
    double *dst = t == n ? out_dev : bufA;
    const unsigned tiles = unsigned(pow4(n - t));
    if (dtype == DM_F64)
        contract_low<double><<<tiles, 256, 0, s>>>(static_cast<const double *>(state_dev), t, R, dst);
    else
        contract_low<float><<<tiles, 256, 0, s>>>(static_cast<const float *>(state_dev), t, R, dst);
    count_launch();
    int rc = launch_status();
    const double *src = dst;
    for (int done = t; !rc && done < n;) {
        const int K = n - done < kNHigh ? n - done : kNHigh;
        const int64_t count = pow4(n - done - K) << done;
        double *d = done + K == n ? out_dev : (src == bufA ? bufB : bufA);
        const unsigned grid = unsigned((count + 127) / 128);
        if (K == 3)
            contract_high<3><<<grid, 128, 0, s>>>(src, count, done, R, d);
        else if (K == 2)
            contract_high<2><<<grid, 128, 0, s>>>(src, count, done, R, d);
        else
            contract_high<1><<<grid, 128, 0, s>>>(src, count, done, R, d);
        count_launch();
        rc = launch_status();
        src = d;
        done += K;
    }
    return rc;
}

extern "C" int dm_nbasis_probs(const void *state_dev, int n, int dtype, const double *nvec3, double err,
                               double *out_dev, void *scratch_dev, void *stream) {
    DM_CHECK_ARG(state_dev && nvec3 && out_dev && valid_n(n) && valid_dtype(dtype));
    DM_CHECK_ARG(low_axes(n) == n || scratch_dev);
    return nbasis(state_dev, n, dtype, nvec3, err, out_dev, static_cast<double *>(scratch_dev), as_stream(stream));
}

// ---------------------------------------------------------------------------
// dm_nbasis_probs_noalloc: the basis-N probabilities with the scratch held in
// a file-scope device array instead of a caller buffer.
// ---------------------------------------------------------------------------

namespace dmg {

constexpr int kNoallocMaxQubits = 10;
// Contraction buffers for n <= kNoallocMaxQubits: 4**7 * 2**3 doubles after
// the first (three-axis) step plus half that for the ping-pong partner.
constexpr size_t kNoallocScratchDoubles = (size_t(1) << 14) * 8 * 3 / 2;   // 196,608 doubles = 1.5 MiB

// Every GPU that loads this library holds this array until the process exits.
static __device__ __align__(256) double g_nbasis_scratch[kNoallocScratchDoubles];

constexpr int kMaxDevices = 64;

// The unique ID of the current CUDA context (driver entry points resolved at
// run time), or 0 when it cannot be read.  A device's primary context gets a
// new ID when it is destroyed and created again (cudaDeviceReset), and the
// module holding g_nbasis_scratch is then loaded again, possibly elsewhere.
static unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static std::once_flag once;
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(p);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(p);
        (void)cudaGetLastError();
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr ||
        get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// Device address of g_nbasis_scratch, resolved with the device current, once
// per device and context: it is looked up again when the device's context
// has changed since (or when its ID cannot be read).  Host code must not pass
// the symbol itself to a kernel: on the host it names a shadow variable, not
// device memory.
static int noalloc_scratch(double **out) {
    static std::mutex mu;
    static double *addr[kMaxDevices] = {nullptr};
    static unsigned long long ctx_of[kMaxDevices] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return DM_ERR_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) return DM_ERR_RANGE;
    // 0 (no context current on this thread yet, or no ID): look the address up, which also makes
    // the runtime's context current; a later call then records that context's ID
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr || ctx == 0 || ctx != ctx_of[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_nbasis_scratch) != cudaSuccess) {
            (void)cudaGetLastError();
            return DM_ERR_CUDA;
        }
        addr[dev] = static_cast<double *>(p);
        ctx_of[dev] = ctx;
    }
    *out = addr[dev];
    return DM_OK;
}

}  // namespace dmg

extern "C" int dm_nbasis_probs_noalloc(const void *state_dev, int n, int dtype, const double *nvec3, double err,
                                       double *out_dev, void *stream) {
    DM_CHECK_ARG(state_dev && nvec3 && out_dev && valid_n(n) && valid_dtype(dtype));
    if (n > kNoallocMaxQubits) return DM_ERR_RANGE;
    const int t = low_axes(n);
    double *scratch = nullptr;
    if (t < n) {
        int rc = noalloc_scratch(&scratch);
        if (rc) return rc;
    }
    // Every buffer element read is written earlier in the same call, so the array's contents from a
    // previous call never leak into a result.
    return nbasis(state_dev, n, dtype, nvec3, err, out_dev, scratch, as_stream(stream));
}
