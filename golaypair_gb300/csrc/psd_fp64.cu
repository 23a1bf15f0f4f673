// psd_fp64.cu -- plain FP64 CUDA-core PSD kernels.
//
// Restates src/utils/fourier.cpp:25-52 in double precision as a direct DFT
// whose twiddle for (j, k) is exp(-2 pi i ((j k) mod L) / L), read from a
// table kept in shared memory.  Two uses:
//   * psd_fp64_filter: the plain FP64 filter (the comparator of the
//     tensor-core path): bins k = 1..L/2 in order, a few at a time for the
//     rows that no bin has ruled out yet;
//   * psd_fp64_values: every bin of a batch (tests).
#include <cmath>

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
//  * a block keeps a list of the rows still alive and computes kBins bins of
//    each per round, so a warp's lanes leave together (one row per thread to
//    the end runs to the last bin of its slowest row: 22 bins at length 45
//    where a row needs 7.4 on average; four a round come to 9);
//  * the integers' doubles come from a table: a conversion takes the same pipe.
// 2^20 rows of length 45: 0.674 ms, 3.600 ms before (one row per thread, direct
// sum); about 400 DFMA a row, the pipe's rate.
constexpr int kBins = 4;
constexpr int kFoldMax = 256;  // |x_j +- x_{L-j}| for int8 rows

// rows per block: up to eight per thread (full warps until the last rounds),
// fewer where shared memory or the number of rows asks for it
struct F64Layout {
    int rows;
    size_t lut, x, list, words, total;
};
F64Layout f64_layout(int L, int64_t n, int num_sms) {
    F64Layout s{};
    s.lut = sizeof(double2) * (size_t)L;
    s.x = s.lut + sizeof(double) * (2 * kFoldMax + 1);
    int r = 4 * kBlock;
    while (r > kBlock / 2 && (n < (int64_t)r * num_sms * 2 || (size_t)r * L > 48 * 1024)) r /= 2;
    s.rows = r;
    s.list = (s.x + (size_t)r * L + 15) & ~size_t(15);
    s.words = s.list + 2 * sizeof(uint16_t) * (size_t)r;
    s.total = s.words + sizeof(uint32_t) * (size_t)(r / 32);
    return s;
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
    const int L = a.src.L, H = L / 2, J = (L - 1) / 2;
    const int lane = threadIdx.x & 31;
    load_tw(sh_tw, a.tw, L);
    for (int v = threadIdx.x; v <= 2 * kFoldMax; v += blockDim.x) lut[v - kFoldMax] = (double)(v - kFoldMax);
    const int64_t row0 = (int64_t)blockIdx.x * lay.rows;
    const int rows = (int)(a.n - row0 < lay.rows ? a.n - row0 : lay.rows);
    // stage this block's rows (coalesced)
    if (a.src.seqs) {
        const int8_t* src = a.src.seqs + row0 * L;
        for (int i = threadIdx.x; i < rows * L; i += blockDim.x) srows[i] = src[i];
    } else {
        for (int r = threadIdx.x; r < rows; r += blockDim.x) decode_row(a.src, row0 + r, srows + (size_t)r * L);
    }
    for (int w = threadIdx.x; w < lay.rows / 32; w += blockDim.x) words[w] = 0u;
    if (threadIdx.x < 2) s_alive[threadIdx.x] = 0;
    __syncthreads();
    int alive = rows, cur = 0;
    for (int k0 = 1; k0 <= H && alive > 0; k0 += kBins, cur ^= 1) {
        for (int i = threadIdx.x; i - lane < alive; i += blockDim.x) {
            bool pass = i < alive;
            const int row = pass ? (k0 == 1 ? i : (int)list[cur][i]) : 0;
            const int8_t* x = srows + (size_t)row * L;
            double re[kBins], im[kBins];
            int m[kBins], step[kBins];
#pragma unroll
            for (int b = 0; b < kBins; ++b) {
                const int k = k0 + b < H ? k0 + b : H;  // past the last bin: the last one again
                step[b] = m[b] = k;
                int c = x[0];
                if (!(L & 1)) c += (k & 1) ? -x[H] : x[H];
                re[b] = lut[c];
                im[b] = 0.0;
            }
            for (int j = 1; j <= J; ++j) {
                const int p = x[j], q = x[L - j];
                const double e = lut[p + q], o = lut[p - q];
#pragma unroll
                for (int b = 0; b < kBins; ++b) {
                    const double2 w = sh_tw[m[b]];
                    re[b] = fma(e, w.x, re[b]);
                    im[b] = fma(o, w.y, im[b]);
                    m[b] += step[b];
                    if (m[b] >= L) m[b] -= L;
                }
            }
#pragma unroll
            for (int b = 0; b < kBins; ++b) pass = pass && re[b] * re[b] + im[b] * im[b] <= a.thr;
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
    cudaError_t e =
        cudaFuncSetAttribute(psd_fp64_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.total);
    if (e != cudaSuccess) return e;
    psd_fp64_filter_kernel<<<(unsigned)blocks, kBlock, lay.total, st>>>(a, lay);
    return cudaGetLastError();
}

cudaError_t launch_psd_fp64_values(const RowSrc& src, const double* tw, int64_t n, double* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int64_t blocks = (n + kBlock - 1) / kBlock;
    const size_t smem = sizeof(double2) * src.L + (size_t)kBlock * src.L + 16;
    cudaError_t e = cudaFuncSetAttribute(psd_values_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    psd_values_kernel<<<(unsigned)blocks, kBlock, smem, st>>>(src, tw, n, out);
    return cudaGetLastError();
}

}  // namespace gp
