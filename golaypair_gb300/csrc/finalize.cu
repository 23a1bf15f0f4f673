// finalize.cu -- exact per-survivor work after the tensor-core filter.
//
// For every candidate whose mask bit survived the guarded filter, a warp:
//   * computes the PSD bins 0..L/2 in FP64 (src/utils/fourier.cpp:25-43) and
//     re-applies the exact filter (fourier.cpp:45-52);
//   * for each role (A / B) of the candidate, optionally checks that the
//     sequence is the lexicographic minimum of its orbit, as isCanonical
//     (src/utils/orderly_equivalence.cpp:53-68) with the generator sets of
//     constructGenerators(0|1, L) (:17-51): for A the affine maps
//     i -> u*i + t (u a unit mod L), for B the dihedral maps i -> +-i + t;
//   * writes a record: the word, the role and the signature
//     rint(psd[k]) (or bound - rint(psd[k]) for inverted roles), k = 1..L-1
//     (src/utils/io.cpp:14-36).
#include <algorithm>

#include "gp_device.cuh"
#include "finalize.h"
#include "rows.cuh"

namespace gp {

namespace {

constexpr int kWarps = 8;
constexpr int kListThreads = 256;

// A block lists the set bits of 256 mask words at a time, with one addition to
// the job's count: atomics on one address take about a nanosecond each (one per
// word that has bits took 31 us for the 17 M candidates of an order-57 iteration,
// now 6.8).
__device__ __forceinline__ void list_bits(const uint32_t* mask, int64_t n, const unsigned long long* n_dev,
                                          uint32_t* out, unsigned long long* count, int64_t cap, int* status) {
    __shared__ uint32_t warp_sum[kListThreads / 32];
    __shared__ unsigned long long first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n_dev && (int64_t)*n_dev < n) n = (int64_t)*n_dev;
    const int64_t nwords = (n + 31) / 32;
    for (int64_t w0 = (int64_t)blockIdx.x * kListThreads; w0 < nwords; w0 += (int64_t)gridDim.x * kListThreads) {
        const int64_t wi = w0 + threadIdx.x;
        uint32_t m = wi < nwords ? mask[wi] : 0u;
        const uint32_t c = (uint32_t)__popc(m);
        uint32_t to = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, to, o);
            if (lane >= o) to += y;
        }
        if (lane == 31) warp_sum[warp] = to;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int q = 0; q < kListThreads / 32; ++q) {
            before += q < warp ? warp_sum[q] : 0u;
            total += warp_sum[q];
        }
        if (threadIdx.x == 0 && total) first = atomicAdd(count, (unsigned long long)total);
        __syncthreads();
        for (unsigned long long pos = first + before + to - c; m; m &= m - 1u, ++pos) {
            if ((int64_t)pos < cap)
                out[pos] = (uint32_t)(wi * 32 + __ffs((int)m) - 1);
            else
                atomicCAS(status, 0, GP_KSTATUS_OVERFLOW);
        }
    }
}

__global__ void mask_to_list_kernel(const uint32_t* mask, int64_t n, const unsigned long long* n_dev, uint32_t* out,
                                    unsigned long long* count, int64_t cap, int* status) {
    list_bits(mask, n, n_dev, out, count, cap, status);
}

// every job's mask in one launch: grid row y serves job y
__global__ void mask_to_list_multi_kernel(ListMultiArgs a) {
    const ListJob& j = a.job[blockIdx.y];
    list_bits(j.mask, j.n, j.n_dev, j.out, j.count, j.cap, a.status);
}

// Rows a warp computes the spectra of at once: 32 lanes over the lanes that a
// row's L/2 + 1 bins take, to the next power of two.  The spectra are bound by
// the FP64 pipe (two DFMA per cycle and SM on GB300), as in psd_fp64.cu: x is
// real, so bins above L/2 repeat those below and a bin needs only the folded
// sums x_j + x_{L-j} and x_j - x_{L-j} (exact integers, made once per row):
// a quarter of the DFMAs of L bins of L terms by 32 lanes.  1.4 M survivors of
// five orders: 7.3 ms, 10.0 with the direct sums (both with the canonical check
// of the general path).
__host__ __device__ __forceinline__ int rows_at_once(int L) {
    int r = 8;
    while (r > 1 && 32 / r < L / 2 + 1) r /= 2;
    return r;
}

// shared memory: the twiddles, then per warp its rows' folded sums, spectra
// and values
struct FinalizeLayout {
    size_t fold, psd, x, per_warp;
};
__host__ __device__ __forceinline__ FinalizeLayout finalize_layout(int L) {
    const size_t R = (size_t)rows_at_once(L), H = (size_t)L / 2;
    FinalizeLayout s;
    s.fold = 0;
    s.psd = R * (H + 1) * sizeof(double2);
    s.x = s.psd + R * (H + 1) * sizeof(double);
    s.per_warp = (s.x + R * L + 15) & ~size_t(15);
    return s;
}

// True if a rotation of x's decimation by u is less than x (L digits of b bits,
// b L <= 63; first digit highest).
__device__ __forceinline__ bool image_less(uint64_t x, int b, int L, int u) {
    const uint64_t digit = (1ull << b) - 1ull, all = (1ull << (b * L)) - 1ull;
    uint64_t y = 0;
    for (int i = 0, at = b * (L - 1); i < L; ++i) {
        y = (y << b) | ((x >> at) & digit);
        at -= b * u;
        at += at < 0 ? b * L : 0;
    }
    bool less = false;
    for (int t = 0; t < L; ++t) {
        less = less || y < x;
        y = ((y << b) & all) | (y >> (b * (L - 1)));
    }
    return less;
}

__device__ __forceinline__ void finalize_rows(const FinalizeArgs& a, double2* sh_tw) {
    const int L = a.src.L, H = L / 2, J = (L - 1) / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = rows_at_once(L), G = 32 / R;  // G lanes to a row
    const FinalizeLayout lay = finalize_layout(L);
    uint8_t* mine = reinterpret_cast<uint8_t*>(sh_tw + L) + (size_t)warp * lay.per_warp;
    double2* fold_all = reinterpret_cast<double2*>(mine + lay.fold);
    double* psd_all = reinterpret_cast<double*>(mine + lay.psd);
    int8_t* xs_all = reinterpret_cast<int8_t*>(mine + lay.x);
    for (int m = threadIdx.x; m < L; m += blockDim.x) sh_tw[m] = make_double2(a.tw[2 * m], a.tw[2 * m + 1]);
    __syncthreads();
    int64_t cnt = (int64_t)*a.n_idx;
    if (cnt > a.idx_cap) cnt = a.idx_cap;
    unsigned passed = 0;  // lane 0: rows that pass
    for (int64_t i0 = ((int64_t)blockIdx.x * kWarps + warp) * R; i0 < cnt; i0 += (int64_t)gridDim.x * kWarps * R) {
        const int n = (int)(cnt - i0 < R ? cnt - i0 : R);
        const int g = lane / G, gl = lane % G;  // this lane's row and place in it
        const bool in = g < n;
        const uint32_t my_row = in ? a.idx[i0 + g] : 0u;
        int8_t* xg = xs_all + g * L;
        double2* fold = fold_all + g * (H + 1);
        double* pg = psd_all + g * (H + 1);
        if (in) {
            if (a.src.seqs) {
                for (int j = gl; j < L; j += G) xg[j] = a.src.seqs[(int64_t)my_row * L + j];
            } else {
                const uint4 w = a.src.words[my_row];
                const uint64_t lo = ((uint64_t)w.y << 32) | w.x, hi = ((uint64_t)w.w << 32) | w.z;
                for (int j = gl; j < L; j += G)
                    xg[j] = (int8_t)(2 * word_digit(lo, hi, a.src.pack_bits, L, j) - a.src.alpha_c);
            }
        }
        __syncwarp();
        if (in)
            for (int j = 1 + gl; j <= J; j += G)
                fold[j] = make_double2((double)(xg[j] + xg[L - j]), (double)(xg[j] - xg[L - j]));
        __syncwarp();
        bool fail = false;
        if (in) {
            const double x0 = (double)xg[0], xh = L % 2 == 0 ? (double)xg[H] : 0.0;
            for (int k = gl; k <= H; k += G) {
                double re = k % 2 ? x0 - xh : x0 + xh, im = 0.0;
                int m = k;
                for (int j = 1; j <= J; ++j) {
                    const double2 w = sh_tw[m], f = fold[j];
                    re = fma(f.x, w.x, re);
                    im = fma(f.y, w.y, im);
                    m += k;
                    if (m >= L) m -= L;
                }
                const double p = re * re + im * im;
                pg[k] = p;
                if (k >= 1 && p > a.thr) fail = true;
            }
        }
        const uint32_t failed = __ballot_sync(0xFFFFFFFFu, fail);
        __syncwarp();
        for (int q = 0; q < n; ++q) {  // its rows one by one, by the whole warp
            if ((failed >> (q * G)) & (G == 32 ? 0xFFFFFFFFu : (1u << G) - 1u)) continue;
            ++passed;
            const uint32_t row = __shfl_sync(0xFFFFFFFFu, my_row, q * G);
            const int8_t* xs = xs_all + q * L;
            const double* psd = psd_all + q * (H + 1);
            if (a.prune_tab) {
                // p(L/2) is the square of the alternating sum and p(L/3) the norm
                // of an Eisenstein integer: both exact integers here
                bool keep = true;
                if (L % 2 == 0) {
                    const int m = a.bound - __double2int_rn(psd[L / 2]);
                    keep = m >= 0 && m <= a.bound && (a.prune_tab[m] & 1);
                }
                if (keep && L % 3 == 0) {
                    const int m = a.bound - __double2int_rn(psd[L / 3]);
                    keep = m >= 0 && m <= a.bound && (a.prune_tab[m] & 2);
                }
                if (!keep) continue;
            }
            const uint8_t roles = a.roles ? a.roles[row] : a.fixed_role;
            for (int r = 0; r < 2; ++r) {
                if (!((roles >> r) & 1)) continue;
                bool canonical = true;
                if (a.check_canonical) {
                    // r = 0: affine maps (constructGenerators(0, L)); r = 1: dihedral
                    const int nmul = r == 0 ? a.n_units : (L > 2 ? 2 : 1);
                    if (a.src.words && a.src.pack_bits * L <= 63) {
                        // a lane per multiplier (comparing every image digit by
                        // digit: 88 us, now 73, for the survivors of 17 M order-57
                        // candidates; five orders 7.3 ms, now 4.6)
                        const uint4 w = a.src.words[row];
                        const uint64_t x = ((uint64_t)w.y << 32) | w.x;
                        for (int m0 = 0; m0 < nmul && canonical; m0 += 32) {
                            const int mi = m0 + lane;
                            const int u = r == 0 ? (mi < nmul ? a.units[mi] : 1) : (mi == 1 ? L - 1 : 1);
                            canonical = !__any_sync(0xFFFFFFFFu, mi < nmul && image_less(x, a.src.pack_bits, L, u));
                        }
                    } else {
                        const int maps = nmul * L;
                        for (int e0 = 0; e0 < maps && canonical; e0 += 32) {
                            const int e = e0 + lane;
                            bool less = false;
                            if (e < maps) {
                                const int mi = e / L;
                                const int u = r == 0 ? a.units[mi] : (mi == 0 ? 1 : L - 1);
                                int idx = e - mi * L;
                                for (int d = 0; d < L; ++d) {
                                    const int v = xs[idx], x = xs[d];
                                    if (v != x) {
                                        less = v < x;
                                        break;
                                    }
                                    idx += u;
                                    if (idx >= L) idx -= L;
                                }
                            }
                            canonical = !__any_sync(0xFFFFFFFFu, less);
                        }
                    }
                }
                if (!canonical) continue;
                unsigned long long pos = 0;
                if (lane == 0) pos = atomicAdd(a.rec_count, 1ull);
                pos = __shfl_sync(0xFFFFFFFFu, pos, 0);
                if ((int64_t)pos >= a.rec_cap) {
                    if (lane == 0) atomicCAS(a.status, 0, GP_KSTATUS_OVERFLOW);
                    continue;
                }
                const bool inv = (a.invert_roles >> r) & 1;
                for (int k = 1 + lane; k < L; k += 32) {
                    const int s = __double2int_rn(psd[k <= H ? k : L - k]);
                    a.rec_sig[pos * (L - 1) + (k - 1)] = (uint16_t)(inv ? a.bound - s : s);
                }
                if (lane == 0) {
                    a.rec_words[pos] = a.src.words ? a.src.words[row] : make_uint4(row, 0, 0, 0);
                    if (a.rec_role) a.rec_role[pos] = (uint8_t)(1 << r);
                    if (a.rec_src) a.rec_src[pos] = row;
                }
            }
        }
        __syncwarp();
    }
    if (lane == 0 && passed) atomicAdd(a.psd_pass, (unsigned long long)passed);
}

__global__ void __launch_bounds__(kWarps * 32) finalize_kernel(FinalizeArgs a) {
    extern __shared__ double2 sh_tw[];
    finalize_rows(a, sh_tw);
}

// every job's survivors in one launch: grid row y serves job y
__global__ void __launch_bounds__(kWarps * 32) finalize_multi_kernel(FinalizeMultiArgs m) {
    extern __shared__ double2 sh_tw[];
    finalize_rows(m.job[blockIdx.y], sh_tw);
}

size_t finalize_smem(int L) { return sizeof(double2) * L + kWarps * finalize_layout(L).per_warp; }

size_t most_smem() {
    static const size_t most = [] {
        size_t m = 0;
        for (int L = 1; L <= kMaxLen; ++L) m = std::max(m, finalize_smem(L));
        return m;
    }();
    return most;
}

}  // namespace

cudaError_t launch_mask_to_list(const uint32_t* mask, int64_t n, uint32_t* out, unsigned long long* count,
                                int64_t cap, int* status, int num_sms, cudaStream_t st,
                                const unsigned long long* n_dev) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks = ((n + 31) / 32 + kListThreads - 1) / kListThreads;
    if (blocks > (int64_t)num_sms * 16) blocks = (int64_t)num_sms * 16;
    mask_to_list_kernel<<<(unsigned)blocks, kListThreads, 0, st>>>(mask, n, n_dev, out, count, cap, status);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const FinalizeArgs& a, int64_t max_rows, int num_sms, cudaStream_t st) {
    if (max_rows <= 0) return cudaSuccess;
    int64_t blocks = (max_rows + kWarps - 1) / kWarps;
    if (blocks > (int64_t)num_sms * 16) blocks = (int64_t)num_sms * 16;
    const size_t smem = finalize_smem(a.src.L);
    cudaError_t e = allow_smem(finalize_kernel, most_smem());
    if (e != cudaSuccess) return e;
    finalize_kernel<<<(unsigned)blocks, kWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_mask_to_list_multi(const ListMultiArgs& a, int num_sms, cudaStream_t st) {
    if (a.njobs <= 0 || a.njobs > kMaxMultiJobs) return a.njobs == 0 ? cudaSuccess : cudaErrorInvalidValue;
    int64_t maxn = 0;
    for (int j = 0; j < a.njobs; ++j) maxn = a.job[j].n > maxn ? a.job[j].n : maxn;
    if (maxn <= 0) return cudaSuccess;
    int64_t blocks = ((maxn + 31) / 32 + kListThreads - 1) / kListThreads;
    // per job as many blocks as its own launch would take: blocks of a job
    // with fewer rows end at once
    if (blocks > (int64_t)num_sms * 16) blocks = (int64_t)num_sms * 16;
    mask_to_list_multi_kernel<<<dim3((unsigned)blocks, (unsigned)a.njobs), kListThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_finalize_multi(const FinalizeMultiArgs& a, const int64_t* max_rows, int num_sms,
                                  cudaStream_t st) {
    if (a.njobs <= 0 || a.njobs > kMaxMultiJobs) return a.njobs == 0 ? cudaSuccess : cudaErrorInvalidValue;
    int64_t rows = 0;
    size_t smem = 0;
    for (int j = 0; j < a.njobs; ++j) {
        rows = max_rows[j] > rows ? max_rows[j] : rows;
        smem = std::max(smem, finalize_smem(a.job[j].src.L));
    }
    if (rows <= 0) return cudaSuccess;
    int64_t blocks = (rows + kWarps - 1) / kWarps;
    // per job as many blocks as its own launch would take: blocks of a job
    // with fewer rows end at once
    if (blocks > (int64_t)num_sms * 16) blocks = (int64_t)num_sms * 16;
    cudaError_t e = allow_smem(finalize_multi_kernel, most_smem());
    if (e != cudaSuccess) return e;
    finalize_multi_kernel<<<dim3((unsigned)blocks, (unsigned)a.njobs), kWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace gp
