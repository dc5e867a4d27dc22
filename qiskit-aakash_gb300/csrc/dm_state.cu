// State set-up, read-out and conversion kernels.
#include <math.h>
#include <string.h>

#include <vector>

#include "dm_common.cuh"

namespace dmg {

// ---------------------------------------------------------------------------
// product states (dm_simulator.py:284-349)
// ---------------------------------------------------------------------------

struct ProductSupport {
    int n;
    int nnz[DM_MAX_QUBITS];
    int8_t digit[DM_MAX_QUBITS][4];
    double val[DM_MAX_QUBITS][4];
    double scale;
};

// Writes the non-zero entries of a Kronecker product of per-qubit
// 4-vectors; the rest of the state was cleared with cudaMemsetAsync.
template <typename T>
__global__ void __launch_bounds__(256) product_kernel(T *__restrict__ st, const __grid_constant__ ProductSupport p,
                                                      int64_t support) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < support;
         i += int64_t(gridDim.x) * blockDim.x) {
        int64_t rem = i, idx = 0, stride = 1;
        double v = p.scale;
        for (int q = p.n - 1; q >= 0; --q) {
            const int k = p.nnz[q];
            const int c = int(rem % k);
            rem /= k;
            idx += int64_t(p.digit[q][c]) * stride;
            v *= p.val[q][c];
            stride <<= 2;
        }
        st[idx] = T(v);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) chop_kernel(const T *__restrict__ st, int64_t total, double thr,
                                                   double *__restrict__ out) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < total;
         i += int64_t(gridDim.x) * blockDim.x) {
        const double v = double(st[i]);
        out[i] = fabs(v) < thr ? 0.0 : v;
    }
}

// The same over pairs: 16-byte stores (out may be mapped host memory, written over the
// CPU-GPU link), total even, both pointers 16-byte aligned.
template <typename T>
__global__ void __launch_bounds__(256) chop_pairs_kernel(const T *__restrict__ st, int64_t pairs, double thr,
                                                         double2 *__restrict__ out) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < pairs;
         i += int64_t(gridDim.x) * blockDim.x) {
        const double a = double(st[2 * i]), b = double(st[2 * i + 1]);
        out[i] = make_double2(fabs(a) < thr ? 0.0 : a, fabs(b) < thr ? 0.0 : b);
    }
}

struct GatherIdx {
    int64_t idx[64];
};

template <typename T>
__global__ void gather_kernel(const T *__restrict__ st, const __grid_constant__ GatherIdx g, int count,
                              double *__restrict__ out) {
    const int i = threadIdx.x;
    if (i < count) out[i] = double(st[g.idx[i]]);
}

// ---------------------------------------------------------------------------
// overlap (dm_simulator.py:1277-1282)
// ---------------------------------------------------------------------------

constexpr int kOverlapMaxBlocks = 4096;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ double block_sum(double v) {
    __shared__ double part[32];
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) part[w] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    v = threadIdx.x < nw ? part[threadIdx.x] : 0.0;
    if (w == 0) v = warp_sum(v);
    __syncthreads();
    return v;
}

template <typename T>
__global__ void __launch_bounds__(256) dot_partial_kernel(const T *__restrict__ a, const T *__restrict__ b,
                                                          int64_t total, double *__restrict__ partial) {
    double acc = 0.0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < total;
         i += int64_t(gridDim.x) * blockDim.x)
        acc = fma(double(a[i]), double(b[i]), acc);
    acc = block_sum(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

__global__ void __launch_bounds__(256) sum_partials_kernel(const double *__restrict__ partial, int count,
                                                           double scale, double *__restrict__ out) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < count; i += blockDim.x) acc += partial[i];
    acc = block_sum(acc);
    if (threadIdx.x == 0) out[0] = acc * scale;
}

// max |a - b| over two states (any dtypes), in FP64: one atomicMax per block on
// the bit pattern, which orders non-negative doubles like their values.
template <typename TA, typename TB>
__global__ void __launch_bounds__(256) max_abs_diff_kernel(const TA *__restrict__ a, const TB *__restrict__ b,
                                                           int64_t total, unsigned long long *__restrict__ out) {
    double m = 0.0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < total;
         i += int64_t(gridDim.x) * blockDim.x)
        m = fmax(m, fabs(double(a[i]) - double(b[i])));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double part[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) part[w] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < int(blockDim.x >> 5); ++i) m = fmax(m, part[i]);
        atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(m)));
    }
}

// ---------------------------------------------------------------------------
// Pauli basis -> matrix basis (dm_simulator.py:1198-1255)
//
// One axis takes (I,X,Y,Z) to the entries (row, column) 00: I+Z, 01: X-iY,
// 10: X+iY, 11: I-Z.  With the sign of (-i)**#Y folded into the real
// coefficients (- where #Y mod 4 is 1 or 2), the real butterflies
// 00: I+Z, 11: I-Z, 01: X+Y, 10: X-Y on every axis give a real matrix M, its
// row and column bits interleaved in the digits, and
//     rho = (M + M^T) / 2 + i (M - M^T) / 2.
// That is one FP64 addition per coefficient and axis and two at the end, half
// of what complex butterflies take; the FP64 pipe (two operations per clock
// and SM) bounds this conversion, 0.37 ms of additions at n = 12 against
// 0.14 ms of traffic.  The axes run in shared memory: the lowest 6 in one
// sweep, then up to 4 per sweep, the top 3 in the sweep that writes rho, each
// of whose CTAs holds a tile of M and the tile of M^T (512-byte runs in,
// 128-byte runs out).  Measured at n = 12 in FP64: 525 us (sweeps of 238, 108
// and 179 us, the FP64 pipe 80 % busy), where one complex sweep per axis and a
// de-interleaving gather took 1,157 us.
//
// An infinity or NaN in M would reach both parts of rho, and as inf - inf.  Tiles
// that hold one are computed again by mat_exact, even and odd #Y apart.
// ---------------------------------------------------------------------------

constexpr int kMatLow = 6;        // axes of the first sweep
constexpr int kMatMid = 4;        // axes of a middle sweep (rows of 2**(12 - 2K) contiguous doubles)
constexpr int kMatTop = 3;        // axes of the last sweep
constexpr int kMatRun = 3;        // lowest axes held whole by a tile of the last sweep
constexpr int kMatTile = 1 << (2 * kMatLow);

// Bank swizzle of a tile of doubles: index bits 4-7 permuted onto bits 0-3, so that groups strided
// over two axes, and rows or columns of the interleaved matrix, spread over the 16 double banks.
__device__ __forceinline__ int mat_swz(int e) {
    return e ^ ((e >> 3) & 10) ^ ((e >> 5) & 5);
}

// v / 2, negated if neg: on the exponent and sign bits of a normal number, which keeps the FP64
// pipe free for the butterflies.
__device__ __forceinline__ double mat_half(double v, bool neg) {
    const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
    if (e < 2 || e == 0x7ff) return v * (neg ? -0.5 : 0.5);
    return __hiloint2double((hi - (1 << 20)) ^ (neg ? int(0x80000000u) : 0), __double2loint(v));
}

__device__ __forceinline__ void mat_axis(double &i, double &x, double &y, double &z) {
    const double a = i + z, b = x + y, c = x - y, d = i - z;
    i = a;
    x = b;
    y = c;
    z = d;
}

// Butterflies on K axes of a tile, the first at element stride 2**s0 (all threads of the CTA).
__device__ __forceinline__ void mat_axes(double *tile, int tsize, int K, int s0) {
    for (int r = 0; r < K; r += 2, s0 += 4) {
        if (r + 1 < K) {
            for (int g = threadIdx.x; g < tsize / 16; g += blockDim.x) {
                const int p = mat_swz(((g >> s0) << (s0 + 4)) | (g & ((1 << s0) - 1)));
                double v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = tile[p ^ mat_swz(j << s0)];
#pragma unroll
                for (int j = 0; j < 4; ++j) mat_axis(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) mat_axis(v[j], v[j + 4], v[j + 8], v[j + 12]);
#pragma unroll
                for (int j = 0; j < 16; ++j) tile[p ^ mat_swz(j << s0)] = v[j];
            }
        } else {
            for (int g = threadIdx.x; g < tsize / 4; g += blockDim.x) {
                const int p = mat_swz(((g >> s0) << (s0 + 2)) | (g & ((1 << s0) - 1)));
                double v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = tile[p ^ mat_swz(j << s0)];
                mat_axis(v[0], v[1], v[2], v[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) tile[p ^ mat_swz(j << s0)] = v[j];
            }
        }
        __syncthreads();
    }
}

// bits 0, 1, 2, ... of x to bits 0, 2, 4, ... (x < 64)
__device__ __forceinline__ int spread6(int x) {
    x = (x | (x << 4)) & 0x30f;
    x = (x | (x << 2)) & 0x333;
    return (x | (x << 1)) & 0x555;
}

// even bits of x gathered
__device__ __forceinline__ uint32_t compact(uint32_t x) {
    x &= 0x55555555u;
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0f0f0f0fu;
    x = (x | (x >> 4)) & 0x00ff00ffu;
    return (x | (x >> 8)) & 0x0000ffffu;
}

// Where entry i (row-major) of tile t's part lies in rho; sr, sc: its tile row and column, bits spread apart.
__device__ __forceinline__ int64_t mat_entry(int i, int n, int lowbits, int topbits, uint32_t t, int &sr, int &sc) {
    const int bits = lowbits + topbits, c = i & ((1 << bits) - 1), r = i >> bits;
    const uint32_t ro = compact(t >> 1) << lowbits, co = compact(t) << lowbits;
    sc = spread6(c);
    sr = spread6(r);
    const uint32_t row = ro | uint32_t(r & ((1 << lowbits) - 1)) | (uint32_t(r >> lowbits) << (n - topbits));
    const uint32_t col = co | uint32_t(c & ((1 << lowbits) - 1)) | (uint32_t(c >> lowbits) << (n - topbits));
    return (int64_t(row) << n) | col;
}

__device__ __forceinline__ bool mat_nonfinite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// Tile t's part of rho, from the tile of M (a) and the tile of M holding the transposed entries (b).
// lowbits: the matrix bits of the run axes; topbits: those of the top axes, at bit n - topbits.
// True where this thread met an infinity or a NaN.
__device__ __forceinline__ bool mat_write(const double *a, const double *b, int n, int lowbits, int topbits,
                                          uint32_t t, double2 *__restrict__ out) {
    bool bad = false;
    for (int i = threadIdx.x; i < 1 << (2 * (lowbits + topbits)); i += blockDim.x) {
        int sr, sc;
        const int64_t at = mat_entry(i, n, lowbits, topbits, t, sr, sc);
        const double u = a[mat_swz(sc | (sr << 1))], w = b[mat_swz(sr | (sc << 1))];
        bad = bad || mat_nonfinite(u) || mat_nonfinite(w);
        out[at] = make_double2(u + w, u - w);
    }
    return bad;
}

// Tile t's part of rho again, straight from the state: the real part from the coefficients of even #Y,
// the imaginary part from those of odd #Y, so that neither sees the other's infinities.  The digits
// between the run and the top axes are summed (I and Z, or X and Y, as the tile's digit says), the
// others run as butterflies in the tile.  2**(n - 6) loads per entry: for infinities and NaN only.
template <typename T>
__device__ __noinline__ void mat_exact(const T *__restrict__ st, double *tile, int n, int lowbits, int topbits,
                                       uint32_t t, double2 *__restrict__ out) {
    const int K = lowbits + topbits, tsize = 1 << (2 * K), mid = n - K;
    for (int part = 0; part < 2; ++part) {
        __syncthreads();
        for (int e = threadIdx.x; e < tsize; e += blockDim.x) {
            const uint64_t at =
                uint64_t(e & ((1 << (2 * lowbits)) - 1)) | (uint64_t(e >> (2 * lowbits)) << (2 * (n - topbits)));
            double sum = 0.0;
            for (uint32_t m = 0; m < 1u << mid; ++m) {
                uint64_t i = at;
                uint32_t neg = 0;
                for (int j = 0; j < mid; ++j) {
                    const uint32_t d = (t >> (2 * j)) & 3, b = (m >> j) & 1;
                    i |= uint64_t(d == 0 || d == 3 ? 3 * b : 1 + b) << (2 * (lowbits + j));
                    neg ^= b & (d >> 1);
                }
                const int ys = __popcll((i >> 1) & ~i & 0x5555555555555555ull);
                if ((ys & 1) != part) continue;
                neg ^= uint32_t(ys + 1) >> 1 & 1;
                const double v = double(st[i]);
                sum += neg ? -v : v;
            }
            tile[mat_swz(e)] = sum;
        }
        __syncthreads();
        mat_axes(tile, tsize, K, 0);
        for (int i = threadIdx.x; i < tsize; i += blockDim.x) {
            int sr, sc;
            const int64_t o = mat_entry(i, n, lowbits, topbits, t, sr, sc);
            const double v = tile[mat_swz(sc | (sr << 1))];
            if (part == 0)
                out[o].x = v;
            else
                out[o].y = v;
        }
    }
}

// The lowest L axes of one contiguous tile per CTA, with the signs; all of rho when L = n.
template <typename T>
__global__ void __launch_bounds__(256) mat_low_kernel(const T *__restrict__ st, int n, int L, double *__restrict__ w,
                                                      double2 *__restrict__ out) {
    __shared__ double tile[kMatTile];
    const int tsize = 1 << (2 * L);
    const int64_t base = int64_t(blockIdx.x) << (2 * L);
    for (int e = threadIdx.x; e < tsize; e += blockDim.x) {
        const uint64_t i = uint64_t(base + e);
        const int ys = __popcll((i >> 1) & ~i & 0x5555555555555555ull);
        const double v = double(st[i]);
        tile[mat_swz(e)] = mat_half(v, (ys + 1) & 2);   // the 1/2 of the last step
    }
    __syncthreads();
    mat_axes(tile, tsize, L, 0);
    if (L == n) {
        if (__syncthreads_or(mat_write(tile, tile, n, n, 0, 0, out))) mat_exact(st, tile, n, n, 0, 0, out);
        return;
    }
    for (int e = threadIdx.x; e < tsize; e += blockDim.x) w[base + e] = tile[mat_swz(e)];
}

// Axes lo .. lo + K - 1 in place: a full tile of 4**K rows (16 coefficients for every thread).
__global__ void __launch_bounds__(256) mat_mid_kernel(double *__restrict__ w, int K, int lo) {
    __shared__ double tile[kMatTile];
    const int rlog = 2 * (kMatLow - K), run = (1 << rlog) - 1;
    const int runs_log = 2 * lo - rlog;
    const int64_t b = blockIdx.x;
    const int64_t base = ((b >> runs_log) << (2 * (lo + K))) + ((b & ((int64_t(1) << runs_log) - 1)) << rlog);
    for (int e = threadIdx.x; e < kMatTile; e += blockDim.x)
        tile[mat_swz(e)] = w[base + (int64_t(e >> rlog) << (2 * lo)) + (e & run)];
    __syncthreads();
    mat_axes(tile, kMatTile, K, rlog);
    for (int e = threadIdx.x; e < kMatTile; e += blockDim.x)
        w[base + (int64_t(e >> rlog) << (2 * lo)) + (e & run)] = tile[mat_swz(e)];
}

// The top K axes and rho: CTA t holds tile t (the digits between the run and the top axes) and the
// tile t' of the transposed entries (row and column bits exchanged), and writes both.
template <typename T>
__global__ void __launch_bounds__(256) mat_top_kernel(const T *__restrict__ st, const double *__restrict__ w, int n,
                                                      int K, double2 *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char mat_smem[];
    double *a = reinterpret_cast<double *>(mat_smem);
    const uint32_t t = blockIdx.x;
    const uint32_t tt = ((t & 0x55555555u) << 1) | ((t >> 1) & 0x55555555u);
    if (tt < t) return;
    const int tsize = 1 << (2 * (K + kMatRun));
    double *b = tt == t ? a : a + tsize;
    for (int e = threadIdx.x; e < tsize; e += blockDim.x) {
        const int64_t in = (e & 63) | (int64_t(e >> 6) << (2 * (n - K)));
        a[mat_swz(e)] = w[in | (int64_t(t) << 6)];
        if (tt != t) b[mat_swz(e)] = w[in | (int64_t(tt) << 6)];
    }
    __syncthreads();
    mat_axes(a, tsize, K, 2 * kMatRun);
    if (tt != t) mat_axes(b, tsize, K, 2 * kMatRun);
    bool bad = mat_write(a, b, n, kMatRun, K, t, out);
    if (tt != t) bad = mat_write(b, a, n, kMatRun, K, tt, out) || bad;
    if (__syncthreads_or(bad)) {
        mat_exact(st, a, n, kMatRun, K, t, out);
        if (tt != t) mat_exact(st, b, n, kMatRun, K, tt, out);
    }
}

}  // namespace dmg

using namespace dmg;

extern "C" int dm_init_product(void *state_dev, int n, int dtype, const double *v, double scale, void *stream) {
    DM_CHECK_ARG(state_dev && v && valid_n(n) && valid_dtype(dtype));
    ProductSupport p;
    memset(&p, 0, sizeof(p));
    p.n = n;
    p.scale = scale;
    int64_t support = 1;
    for (int q = 0; q < n; ++q) {
        int k = 0;
        for (int d = 0; d < 4; ++d)
            if (v[4 * q + d] != 0.0) {
                p.digit[q][k] = int8_t(d);
                p.val[q][k] = v[4 * q + d];
                ++k;
            }
        if (k == 0) {  // an all-zero factor: the whole state is zero
            p.nnz[q] = 1;
            p.digit[q][0] = 0;
            p.val[q][0] = 0.0;
            k = 1;
        }
        p.nnz[q] = k;
        support *= k;
    }
    cudaStream_t s = as_stream(stream);
    DM_CUDA_TRY(cudaMemsetAsync(state_dev, 0, size_t(pow4(n)) * dtype_size(dtype), s));
    if (dtype == DM_F64)
        product_kernel<double><<<grid_for(support, 256), 256, 0, s>>>(static_cast<double *>(state_dev), p, support);
    else
        product_kernel<float><<<grid_for(support, 256), 256, 0, s>>>(static_cast<float *>(state_dev), p, support);
    count_launch();
    return launch_status();
}

extern "C" int dm_load_state(void *state_dev, int n, int dtype, const double *host_coeffs, void *stream) {
    DM_CHECK_ARG(state_dev && host_coeffs && valid_n(n) && valid_dtype(dtype));
    const size_t total = size_t(pow4(n));
    cudaStream_t s = as_stream(stream);
    if (dtype == DM_F64) {
        DM_CUDA_TRY(cudaMemcpyAsync(state_dev, host_coeffs, total * 8, cudaMemcpyHostToDevice, s));
        DM_CUDA_TRY(cudaStreamSynchronize(s));
        return DM_OK;
    }
    std::vector<float> tmp(total);
    for (size_t i = 0; i < total; ++i) tmp[i] = float(host_coeffs[i]);
    DM_CUDA_TRY(cudaMemcpyAsync(state_dev, tmp.data(), total * 4, cudaMemcpyHostToDevice, s));
    DM_CUDA_TRY(cudaStreamSynchronize(s));
    return DM_OK;
}

extern "C" int dm_chop_copy(const void *state_dev, int n, int dtype, double threshold, double *out_dev,
                            void *stream) {
    DM_CHECK_ARG(valid_n(n));
    return dm_chop_copy_range(state_dev, n, dtype, 0, pow4(n), threshold, out_dev, stream);
}

extern "C" int dm_chop_copy_range(const void *state_dev, int n, int dtype, int64_t offset, int64_t count,
                                  double threshold, double *out_dev, void *stream) {
    DM_CHECK_ARG(state_dev && out_dev && valid_n(n) && valid_dtype(dtype));
    DM_CHECK_ARG(offset >= 0 && count > 0 && offset + count <= pow4(n));
    const int64_t total = count;
    if (dtype == DM_F64)
        state_dev = static_cast<const double *>(state_dev) + offset;
    else
        state_dev = static_cast<const float *>(state_dev) + offset;
    cudaStream_t s = as_stream(stream);
    if (total % 2 == 0 && (reinterpret_cast<uintptr_t>(out_dev) & 15) == 0) {
        const int64_t pairs = total / 2;
        auto *out2 = reinterpret_cast<double2 *>(out_dev);
        if (dtype == DM_F64)
            chop_pairs_kernel<double><<<grid_for(pairs, 256), 256, 0, s>>>(static_cast<const double *>(state_dev),
                                                                          pairs, threshold, out2);
        else
            chop_pairs_kernel<float><<<grid_for(pairs, 256), 256, 0, s>>>(static_cast<const float *>(state_dev),
                                                                         pairs, threshold, out2);
    } else if (dtype == DM_F64) {
        chop_kernel<double><<<grid_for(total, 256), 256, 0, s>>>(static_cast<const double *>(state_dev), total,
                                                                 threshold, out_dev);
    } else {
        chop_kernel<float><<<grid_for(total, 256), 256, 0, s>>>(static_cast<const float *>(state_dev), total,
                                                                threshold, out_dev);
    }
    count_launch();
    return launch_status();
}

extern "C" void *dm_host_alloc(size_t bytes) {
    if (bytes == 0) return nullptr;
    void *p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return p;
}

extern "C" void *dm_host_device_pointer(void *host) {
    void *d = nullptr;
    if (!host || cudaHostGetDevicePointer(&d, host, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return d;
}

extern "C" int dm_host_free(void *host) {
    if (!host) return DM_ERR_ARG;
    DM_CUDA_TRY(cudaFreeHost(host));
    return DM_OK;
}

extern "C" int dm_gather(const void *state_dev, int n, int dtype, const int64_t *idx, int count, double *out_dev,
                         void *stream) {
    DM_CHECK_ARG(state_dev && idx && out_dev && valid_n(n) && valid_dtype(dtype));
    DM_CHECK_ARG(count >= 1 && count <= 64);
    GatherIdx g;
    const int64_t total = pow4(n);
    for (int i = 0; i < count; ++i) {
        DM_CHECK_ARG(idx[i] >= 0 && idx[i] < total);
        g.idx[i] = idx[i];
    }
    cudaStream_t s = as_stream(stream);
    if (dtype == DM_F64)
        gather_kernel<double><<<1, 64, 0, s>>>(static_cast<const double *>(state_dev), g, count, out_dev);
    else
        gather_kernel<float><<<1, 64, 0, s>>>(static_cast<const float *>(state_dev), g, count, out_dev);
    count_launch();
    return launch_status();
}

extern "C" size_t dm_overlap_scratch_bytes(int n) {
    (void)n;
    return sizeof(double) * kOverlapMaxBlocks;
}

extern "C" int dm_overlap(const void *a_dev, const void *b_dev, int n, int dtype, double *out_dev, void *scratch_dev,
                          void *stream) {
    DM_CHECK_ARG(a_dev && b_dev && out_dev && scratch_dev && valid_n(n) && valid_dtype(dtype));
    const int64_t total = pow4(n);
    int blocks = grid_for(total, 256, 4);
    if (blocks > kOverlapMaxBlocks) blocks = kOverlapMaxBlocks;
    cudaStream_t s = as_stream(stream);
    double *partial = static_cast<double *>(scratch_dev);
    if (dtype == DM_F64)
        dot_partial_kernel<double><<<blocks, 256, 0, s>>>(static_cast<const double *>(a_dev),
                                                          static_cast<const double *>(b_dev), total, partial);
    else
        dot_partial_kernel<float><<<blocks, 256, 0, s>>>(static_cast<const float *>(a_dev),
                                                         static_cast<const float *>(b_dev), total, partial);
    count_launch();
    int rc = launch_status();
    if (rc) return rc;
    sum_partials_kernel<<<1, 256, 0, s>>>(partial, blocks, ldexp(1.0, n), out_dev);
    count_launch();
    return launch_status();
}

extern "C" size_t dm_pauli_to_matrix_scratch_bytes(int n) {
    if (!valid_n(n)) return 0;
    return size_t(pow4(n)) * sizeof(double2);
}

template <typename T>
static int launch_mat_top(const T *st, const double *w, int n, int top, double2 *out, cudaStream_t s) {
    const int smem = 2 * (1 << (2 * (top + kMatRun))) * int(sizeof(double));
    if (ensure_max_dynamic_smem(reinterpret_cast<const void *>(mat_top_kernel<T>),
                                2 * (1 << (2 * (kMatTop + kMatRun))) * int(sizeof(double))) != cudaSuccess)
        return DM_ERR_CUDA;
    mat_top_kernel<T><<<unsigned(pow4(n - top - kMatRun)), 256, smem, s>>>(st, w, n, top, out);
    count_launch();
    return launch_status();
}

extern "C" int dm_pauli_to_matrix(const void *state_dev, int n, int dtype, double *out_dev, void *scratch_dev,
                                  void *stream) {
    DM_CHECK_ARG(state_dev && out_dev && scratch_dev && valid_n(n) && valid_dtype(dtype));
    if (n > 15) return DM_ERR_RANGE;  // 2**n x 2**n complex128 output beyond 16 GB
    cudaStream_t s = as_stream(stream);
    double *w = static_cast<double *>(scratch_dev);
    auto *out = reinterpret_cast<double2 *>(out_dev);
    const int L = n < kMatLow ? n : kMatLow;
    const unsigned tiles = unsigned(pow4(n - L));
    if (dtype == DM_F64)
        mat_low_kernel<double><<<tiles, 256, 0, s>>>(static_cast<const double *>(state_dev), n, L, w, out);
    else
        mat_low_kernel<float><<<tiles, 256, 0, s>>>(static_cast<const float *>(state_dev), n, L, w, out);
    count_launch();
    int rc = launch_status();
    if (rc || L == n) return rc;
    const int top = n - L < kMatTop ? n - L : kMatTop;
    int lo = L;
    while (lo < n - top) {
        const int left = n - top - lo, sweeps = (left + kMatMid - 1) / kMatMid;
        const int K = (left + sweeps - 1) / sweeps;
        mat_mid_kernel<<<unsigned(pow4(n - kMatLow)), 256, 0, s>>>(w, K, lo);
        count_launch();
        if ((rc = launch_status())) return rc;
        lo += K;
    }
    return dtype == DM_F64 ? launch_mat_top(static_cast<const double *>(state_dev), w, n, top, out, s)
                           : launch_mat_top(static_cast<const float *>(state_dev), w, n, top, out, s);
}

extern "C" int dm_max_abs_diff(const void *a_dev, int dtype_a, const void *b_dev, int dtype_b, int n, double *out_dev,
                               void *stream) {
    DM_CHECK_ARG(a_dev && b_dev && out_dev && valid_n(n) && valid_dtype(dtype_a) && valid_dtype(dtype_b));
    const int64_t total = pow4(n);
    cudaStream_t s = as_stream(stream);
    DM_CUDA_TRY(cudaMemsetAsync(out_dev, 0, sizeof(double), s));
    const int blocks = grid_for(total, 256, 4);
    auto *out = reinterpret_cast<unsigned long long *>(out_dev);
    if (dtype_a == DM_F32 && dtype_b == DM_F64)
        max_abs_diff_kernel<<<blocks, 256, 0, s>>>(static_cast<const float *>(a_dev), static_cast<const double *>(b_dev),
                                                   total, out);
    else if (dtype_a == DM_F64 && dtype_b == DM_F64)
        max_abs_diff_kernel<<<blocks, 256, 0, s>>>(static_cast<const double *>(a_dev),
                                                   static_cast<const double *>(b_dev), total, out);
    else if (dtype_a == DM_F32 && dtype_b == DM_F32)
        max_abs_diff_kernel<<<blocks, 256, 0, s>>>(static_cast<const float *>(a_dev), static_cast<const float *>(b_dev),
                                                   total, out);
    else
        max_abs_diff_kernel<<<blocks, 256, 0, s>>>(static_cast<const double *>(a_dev),
                                                   static_cast<const float *>(b_dev), total, out);
    count_launch();
    return launch_status();
}
