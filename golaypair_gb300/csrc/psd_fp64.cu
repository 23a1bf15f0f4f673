// psd_fp64.cu -- plain FP64 CUDA-core PSD kernels.
//
// Restates src/utils/fourier.cpp:25-52 in double precision as a direct DFT
// whose twiddle for (j, k) is exp(-2 pi i ((j k) mod L) / L), read from a
// table kept in shared memory.  Two uses:
//   * psd_fp64_filter: the plain FP64 filter (the comparator of the
//     tensor-core path): bins k = 1..L/2, a few at a time for the rows that
//     no bin has ruled out yet, those that cost least first;
//   * psd_fp64_values: every bin of a batch (tests).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "gp_device.cuh"
#include "rows.cuh"

namespace gp {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ void load_tw(double2* stw, const double* tw, int L) {
    for (int m = threadIdx.x; m < L; m += blockDim.x) stw[m] = make_double2(tw[2 * m], tw[2 * m + 1]);
}

__device__ __forceinline__ double bin_power(const int8_t* x, int L, int k, const double2* tw) {
    double re = 0.0, im = 0.0;
    int m = 0;
    for (int j = 0; j < L; ++j) {
        const double v = (double)x[j];
        const double2 w = tw[m];
        re = fma(v, w.x, re);
        im = fma(-v, w.y, im);
        m += k;
        if (m >= L) m -= L;
    }
    return re * re + im * im;
}

// The plain FP64 filter.  It is bound by the FP64 pipe (two DFMA per cycle and
// SM on GB300), so everything else serves to issue fewer of them:
//  * x is real, so a bin needs the folded sums e_j = x_j + x_{L-j} (cosines)
//    and o_j = x_j - x_{L-j} (sines), j = 1 .. (L-1)/2: half the DFMAs of the
//    direct sum, and fewer roundings (the folds are exact integers);
//  * a bin k with g = gcd(k, L) > 1 is a bin of the length L / g sequence
//    y_j = x_j + x_{j + L/g} + .. (exact integers), 1/g of the DFMAs.  Those
//    bins go first, the largest g first: ten of length 45's 22 cost as much as
//    two of the others and rule out three rows of four;
//  * a block keeps a list of the rows still alive and computes one round of
//    bins of each at a time, so a warp's lanes leave together (one row per
//    thread to the end runs to the last bin of its slowest row).  A round is
//    one group of up to kBins bins of the same g, or several that hold fewer
//    (with all of length 45's ten cheap bins in one round: 0.55 ms against 0.31,
//    too many lanes idle at its end);
//  * the integers' doubles come from a table, or from their floats' bits: a
//    conversion takes the same pipe.
// 2^20 rows of length 45: 0.224 ms, 0.674 with the bins in order, 3.600 with a
// row per thread and direct sums; of the prime length 37 0.445, 0.474 before.
constexpr int kBins = 4;
constexpr int kFoldMax = 256;  // range of the table (x_j +- x_{L-j} of int8 rows)

// rows per block: up to four per thread (full warps until the last rounds),
// fewer where shared memory or the number of rows asks for it
struct F64Layout {
    int rows;
    size_t lut, bins, x, list, words, total;
};

// The bins in the order they are computed: by falling g = gcd(k, L).  Groups
// of up to kBins bins of one g, rounds of groups.
struct F64Bins {
    uint16_t k[kMaxLen / 2];
    uint16_t g[kMaxLen / 2];
    uint16_t group[kMaxLen / 2 + 1];  // a group's first bin
    uint16_t round[kMaxLen / 2 + 1];  // a round's first group
    int rounds;
};
F64Layout f64_layout(int L, int64_t n, int num_sms) {
    F64Layout s{};
    s.lut = sizeof(double2) * (size_t)L;
    s.bins = s.lut + sizeof(double) * (2 * kFoldMax + 1);
    s.x = (s.bins + sizeof(F64Bins) + 15) & ~size_t(15);
    int r = 4 * kBlock;
    while (r > kBlock / 2 && (n < (int64_t)r * num_sms * 2 || (size_t)r * L > 48 * 1024)) r /= 2;
    s.rows = r;
    s.list = (s.x + (size_t)r * L + 15) & ~size_t(15);
    s.words = s.list + 2 * sizeof(uint16_t) * (size_t)r;
    s.total = s.words + sizeof(uint32_t) * (size_t)(r / 32);
    return s;
}

__device__ __forceinline__ void order_bins(F64Bins& o, int L) {
    const int H = L / 2;
    for (int t = threadIdx.x; t < H; t += blockDim.x) {
        int u = L, v = t + 1;
        while (v) {
            const int r = u % v;
            u = v;
            v = r;
        }
        o.round[t] = (uint16_t)u;  // for now, bin t + 1's g
    }
    __syncthreads();
    for (int t = threadIdx.x; t < H; t += blockDim.x) {
        const int g = o.round[t];
        int at = 0;
        for (int q = 0; q < H; ++q) at += o.round[q] > g || (o.round[q] == g && q < t);
        o.k[at] = (uint16_t)(t + 1);
        o.g[at] = (uint16_t)g;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int groups = 0, rounds = 0, in_round = kBins;
        for (int t = 0; t < H; ++groups) {
            int n = 1;
            while (n < kBins && t + n < H && o.g[t + n] == o.g[t]) ++n;
            if (in_round >= kBins) {
                o.round[rounds++] = (uint16_t)groups;
                in_round = 0;
            }
            in_round += n;
            o.group[groups] = (uint16_t)t;
            t += n;
        }
        o.group[groups] = (uint16_t)H;
        o.round[rounds] = (uint16_t)groups;
        o.rounds = rounds;
    }
    __syncthreads();
}

// An integer below 2^24 as a double, without the FP64 pipe: its float's bits,
// with the exponent's bias of a double.
__device__ __forceinline__ double small_double(int v) {
    const uint32_t f = __float_as_uint((float)v);
    const uint32_t hi = (f & 0x80000000u) | (((f & 0x7FFFFFFFu) >> 3) + 0x38000000u);
    return __hiloint2double(v ? (int)hi : 0, (int)(f << 29));
}

// True if NB bins k[0..NB), all with gcd(k, L) = g, are within thr.  ONE: g = 1.
template <int NB, bool ONE>
__device__ __forceinline__ bool bins_pass(const int8_t* x, int L, int g, const uint16_t* k, const double2* tw,
                                          const double* lut, double thr) {
    const int M = ONE ? L : L / g, J = (M - 1) / 2;
    auto fold = [&](int j) {
        int y = x[j];
        if constexpr (!ONE)
            for (int i = j + M; i < L; i += M) y += x[i];
        return y;
    };
    auto dbl = [&](int v) {
        if constexpr (ONE)
            return lut[v];
        else
            return small_double(v);
    };
    double re[NB], im[NB];
    int m[NB];
    const int y0 = fold(0), yh = M % 2 == 0 ? fold(M / 2) : 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        m[b] = k[b];
        re[b] = dbl((ONE ? k[b] : k[b] / g) % 2 ? y0 - yh : y0 + yh);
        im[b] = 0.0;
    }
    for (int j = 1; j <= J; ++j) {
        const int p = fold(j), q = fold(M - j);
        const double e = dbl(p + q), o = dbl(p - q);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const double2 w = tw[m[b]];
            re[b] = fma(e, w.x, re[b]);
            im[b] = fma(o, w.y, im[b]);
            m[b] += k[b];
            if (m[b] >= L) m[b] -= L;
        }
    }
    bool pass = true;
#pragma unroll
    for (int b = 0; b < NB; ++b) pass = pass && re[b] * re[b] + im[b] * im[b] <= thr;
    return pass;
}

__global__ void __launch_bounds__(kBlock) psd_fp64_filter_kernel(PsdF64Args a, F64Layout lay) {
    extern __shared__ double2 sh_tw[];
    __shared__ int s_alive[2];
    uint8_t* smem = reinterpret_cast<uint8_t*>(sh_tw);
    double* lut = reinterpret_cast<double*>(smem + lay.lut) + kFoldMax;
    int8_t* srows = reinterpret_cast<int8_t*>(smem + lay.x);
    uint16_t* list[2] = {reinterpret_cast<uint16_t*>(smem + lay.list),
                         reinterpret_cast<uint16_t*>(smem + lay.list) + lay.rows};
    uint32_t* words = reinterpret_cast<uint32_t*>(smem + lay.words);
    F64Bins& bins = *reinterpret_cast<F64Bins*>(smem + lay.bins);
    const int L = a.src.L, H = L / 2;
    const int lane = threadIdx.x & 31;
    load_tw(sh_tw, a.tw, L);
    order_bins(bins, L);
    for (int v = threadIdx.x; v <= 2 * kFoldMax; v += blockDim.x) lut[v - kFoldMax] = (double)(v - kFoldMax);
    const int64_t row0 = (int64_t)blockIdx.x * lay.rows;
    const int rows = (int)(a.n - row0 < lay.rows ? a.n - row0 : lay.rows);
    // stage this block's rows (coalesced)
    if (a.src.seqs) {
        const int8_t* src = a.src.seqs + row0 * L;
        const int bytes = rows * L;
        int i = threadIdx.x;
        if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {  // by 16 bytes, then the rest
            for (int v = threadIdx.x; v < bytes / 16; v += blockDim.x)
                reinterpret_cast<uint4*>(srows)[v] = reinterpret_cast<const uint4*>(src)[v];
            i += bytes / 16 * 16;
        }
        for (; i < bytes; i += blockDim.x) srows[i] = src[i];
    } else {
        for (int r = threadIdx.x; r < rows; r += blockDim.x) decode_row(a.src, row0 + r, srows + (size_t)r * L);
    }
    for (int w = threadIdx.x; w < lay.rows / 32; w += blockDim.x) words[w] = 0u;
    if (threadIdx.x < 2) s_alive[threadIdx.x] = 0;
    __syncthreads();
    int alive = rows, cur = 0;
    for (int r = 0; r < bins.rounds && alive > 0; ++r, cur ^= 1) {
        for (int i = threadIdx.x; i - lane < alive; i += blockDim.x) {
            bool pass = i < alive;
            const int row = pass ? (r == 0 ? i : (int)list[cur][i]) : 0;
            const int8_t* x = srows + (size_t)row * L;
            for (int q = bins.round[r]; q < bins.round[r + 1] && __any_sync(0xFFFFFFFFu, pass); ++q) {
                const int t = bins.group[q], n = bins.group[q + 1] - t, g = bins.g[t];
                const uint16_t* k = bins.k + t;
                auto within = [&](auto one) {
                    constexpr bool ONE = decltype(one)::value;
                    if (n == 4) return bins_pass<4, ONE>(x, L, g, k, sh_tw, lut, a.thr);
                    if (n == 3) return bins_pass<3, ONE>(x, L, g, k, sh_tw, lut, a.thr);
                    if (n == 2) return bins_pass<2, ONE>(x, L, g, k, sh_tw, lut, a.thr);
                    return bins_pass<1, ONE>(x, L, g, k, sh_tw, lut, a.thr);
                };
                if (pass) pass = g == 1 ? within(std::true_type()) : within(std::false_type());
            }
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, pass);
            if (bal) {
                int base = 0;
                if (lane == 0) base = atomicAdd(&s_alive[cur ^ 1], __popc(bal));
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                if (pass) list[cur ^ 1][base + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)row;
            }
        }
        __syncthreads();
        alive = s_alive[cur ^ 1];
        if (threadIdx.x == 0) s_alive[cur] = 0;  // counts the round after next
        __syncthreads();
    }
    for (int i = threadIdx.x; i < alive; i += blockDim.x) {
        const int row = H > 0 ? (int)list[cur][i] : i;
        atomicOr(&words[row >> 5], 1u << (row & 31));
    }
    __syncthreads();
    for (int w = threadIdx.x; w < lay.rows / 32; w += blockDim.x) {
        const int64_t word = (row0 >> 5) + w;
        if (word < a.mask_words) a.mask[word] = words[w];
    }
}

__global__ void __launch_bounds__(kBlock) psd_values_kernel(RowSrc src, const double* tw, int64_t n, double* out) {
    extern __shared__ double2 sh_tw[];
    const int L = src.L;
    int8_t* xs = reinterpret_cast<int8_t*>(sh_tw + L) + (int64_t)threadIdx.x * L;
    load_tw(sh_tw, tw, L);
    __syncthreads();
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n) return;
    decode_row(src, row, xs);
    for (int k = 0; k < L; ++k) out[row * L + k] = bin_power(xs, L, k, sh_tw);
}

}  // namespace

void build_twiddle64(int L, double* out) {
    for (int m = 0; m < L; ++m) {
        const long double ang = 6.283185307179586476925286766559L * (long double)m / (long double)L;
        out[2 * m] = (double)std::cos(ang);
        out[2 * m + 1] = (double)std::sin(ang);
    }
}

cudaError_t launch_psd_fp64(const PsdF64Args& a, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    const F64Layout lay = f64_layout(a.src.L, a.n, a.num_sms);
    const int64_t blocks = (a.n + lay.rows - 1) / lay.rows;
    static const size_t most = [] {
        size_t m = 0;
        for (int L = 1; L <= kMaxLen; ++L) m = std::max(m, f64_layout(L, INT64_MAX, 1).total);
        return m;
    }();
    cudaError_t e = allow_smem(psd_fp64_filter_kernel, most);
    if (e != cudaSuccess) return e;
    psd_fp64_filter_kernel<<<(unsigned)blocks, kBlock, lay.total, st>>>(a, lay);
    return cudaGetLastError();
}

cudaError_t launch_psd_fp64_values(const RowSrc& src, const double* tw, int64_t n, double* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int64_t blocks = (n + kBlock - 1) / kBlock;
    auto bytes = [](int L) { return sizeof(double2) * L + (size_t)kBlock * L + 16; };
    const size_t smem = bytes(src.L);
    cudaError_t e = allow_smem(psd_values_kernel, bytes(kMaxLen));
    if (e != cudaSuccess) return e;
    psd_values_kernel<<<(unsigned)blocks, kBlock, smem, st>>>(src, tw, n, out);
    return cudaGetLastError();
}

}  // namespace gp
