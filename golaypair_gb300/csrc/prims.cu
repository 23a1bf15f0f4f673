// prims.cu -- device building blocks of the sort/match stages: exclusive scan,
// stable compaction, and a stable LSD radix sort of fixed-width keys.
//
// Keys are rows of W 32-bit words, word 0 most significant.  The sort
// permutes a uint32 index array (keys stay in place and are gathered per
// pass), 4 or 8 bits per pass (the sort's tuner picks); a pass whose digit
// is the same for every key is skipped.  One kernel counts every digit of every
// key first, so the passes run without waiting for the host in between, and a
// pass is two launches (block histograms, scatter) up to kScatterScanBlocks
// blocks and kTotalWords words: the scatter sums the blocks before its own.
// The passes take the leading digits only, as many as hold twice the entropy
// that n distinct rows need; rows that still agree stand next to each other
// then and are ranked by whole keys, unless more than kRunMax of them do.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>
#include <utility>
#include <vector>

#include "prims.h"

namespace gp {

namespace {

constexpr int kScanBlock = 1024;

__global__ void scan_block_kernel(const uint32_t* in, uint32_t* out, uint32_t* block_sums, int64_t n) {
    __shared__ uint32_t warp_tot[32];
    const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
    uint32_t v = i < n ? in[i] : 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    const uint32_t before = warp ? warp_tot[warp - 1] : 0u;
    if (i < n) out[i] = before + x - v;  // exclusive
    if (threadIdx.x == kScanBlock - 1 && block_sums) block_sums[blockIdx.x] = before + x;
}

__global__ void scan_add_kernel(uint32_t* out, const uint32_t* block_off, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
    if (i < n) out[i] += block_off[blockIdx.x];
}

__global__ void compact_kernel(const uint32_t* flags, const uint32_t* pos, const uint32_t* src, uint32_t* dst,
                               int64_t n, uint32_t* count) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (flags[i]) dst[pos[i]] = src ? src[i] : (uint32_t)i;
        if (i == n - 1) *count = pos[i] + (flags[i] ? 1u : 0u);
    }
}

// ------------------------------------------------------------ radix sort
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int64_t kScatterScanBlocks = 256;  // 2^19 keys
constexpr int kRunMax = 32;
// Words whose digit totals are held at once: 4 MB here and on the host (a line of
// 8 MB held whole took 8 GB of either).  Candidate lines have some 20 words.
constexpr int kTotalWords = 1024;
constexpr int kTailPasses = 4;  // about what the two kernels for runs and the wait cost

template <int RB>
__device__ __forceinline__ uint32_t key_digit(const uint32_t* keys, int W, uint32_t idx, int word, int shift) {
    return (keys[(int64_t)idx * W + word] >> shift) & ((1u << RB) - 1u);
}

// Every digit's counts over the keys of rows [0, n): total[digit * NB + d]
// for digit = 0 (the last word's low bits) .. (32 / RB) W - 1.  One block row
// (blockIdx.y) per word.
template <int RB>
__global__ void __launch_bounds__(kSortThreads) radix_totals_kernel(const uint32_t* keys, int W, int sort_words,
                                                                    int64_t n, uint32_t* total) {
    constexpr int NB = 1 << RB, ND = 32 / RB;
    __shared__ uint32_t h[ND * NB];
    for (int word = blockIdx.y; word < sort_words; word += gridDim.y) {
        for (int i = threadIdx.x; i < ND * NB; i += kSortThreads) h[i] = 0;
        __syncthreads();
        for (int64_t i0 = (int64_t)blockIdx.x * kSortThreads; i0 < n; i0 += (int64_t)gridDim.x * kSortThreads) {
            const int64_t i = i0 + threadIdx.x;
            const bool has = i < n;
            const uint32_t k = has ? keys[i * W + word] : 0u;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                // most keys share a digit: one addition for a warp that agrees
                const uint32_t x = has ? (k >> (RB * d)) & (NB - 1u) : 0x100u;
                int same;
                __match_all_sync(0xFFFFFFFFu, x, &same);
                if (same) {
                    if (has && (threadIdx.x & 31) == 0) atomicAdd(&h[d * NB + x], 32u);
                } else if (has) {
                    atomicAdd(&h[d * NB + x], 1u);
                }
            }
        }
        __syncthreads();
        const int first = (sort_words - 1 - word) * ND;
        for (int i = threadIdx.x; i < ND * NB; i += kSortThreads)
            if (h[i]) atomicAdd(&total[(int64_t)first * NB + i], h[i]);
        __syncthreads();
    }
}

// RB bits per pass: 2^RB buckets (RB <= 8, so one thread per bucket).
// counts: by block, then bucket (ROWS), or by bucket, then block.
template <int RB, bool ROWS>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const uint32_t* keys, int W, const uint32_t* idx,
                                                                   int64_t n, int word, int shift, uint32_t* counts,
                                                                   int64_t nblocks) {
    constexpr int NB = 1 << RB;
    __shared__ uint32_t h[NB];
    if (threadIdx.x < NB) h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + (int64_t)k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[key_digit<RB>(keys, W, idx[i], word, shift)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < NB)
        counts[ROWS ? (int64_t)blockIdx.x * NB + threadIdx.x : (int64_t)threadIdx.x * nblocks + blockIdx.x] =
            h[threadIdx.x];
}

// ROWS: the buckets' first places are the digit's totals before them plus the
// counts of the blocks before this one; otherwise offsets has been scanned.
template <int RB, bool ROWS>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(const uint32_t* keys, int W, const uint32_t* idx_in,
                                                                      uint32_t* idx_out, int64_t n, int word, int shift,
                                                                      const uint32_t* offsets, int64_t nblocks,
                                                                      const uint32_t* total) {
    constexpr int NB = 1 << RB;
    __shared__ uint32_t base[NB];
    __shared__ uint32_t wh[kSortThreads / 32][NB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (ROWS) {
        uint32_t before = 0;
        if (threadIdx.x < NB) {
#pragma unroll 8
            for (int64_t b = 0; b < (int64_t)blockIdx.x; ++b) before += offsets[b * NB + threadIdx.x];
        }
        const uint32_t t = threadIdx.x < NB ? total[threadIdx.x] : 0u;
        uint32_t x = t;  // inclusive scan of the totals over the block
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wh[0][warp] = x;
        __syncthreads();
        uint32_t warps = 0;
        for (int q = 0; q < warp; ++q) warps += wh[0][q];
        __syncthreads();
        if (threadIdx.x < NB) base[threadIdx.x] = warps + x - t + before;
    } else if (threadIdx.x < NB) {
        base[threadIdx.x] = offsets[(int64_t)threadIdx.x * nblocks + blockIdx.x];
    }
    const int64_t tile0 = (int64_t)blockIdx.x * kSortTile;
    for (int k = 0; k < kSortItems; ++k) {
        if (threadIdx.x < NB)
            for (int w = 0; w < kSortThreads / 32; ++w) wh[w][threadIdx.x] = 0;
        __syncthreads();
        const int64_t i = tile0 + (int64_t)k * kSortThreads + threadIdx.x;
        const bool valid = i < n;
        uint32_t my_idx = 0, d = 0x100u + (uint32_t)lane;  // invalid lanes: unique sentinel
        if (valid) {
            my_idx = idx_in[i];
            d = key_digit<RB>(keys, W, my_idx, word, shift);
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) wh[warp][d] = __popc(peers);
        __syncthreads();
        if (threadIdx.x < NB) {
            uint32_t run = base[threadIdx.x];
            for (int w = 0; w < kSortThreads / 32; ++w) {
                const uint32_t c = wh[w][threadIdx.x];
                wh[w][threadIdx.x] = run;
                run += c;
            }
            base[threadIdx.x] = run;
        }
        __syncthreads();
        if (valid) idx_out[wh[warp][d] + rank] = my_idx;
        __syncthreads();
    }
}

// The leading digits of row i and row j agree: words before w, and mask of w.
__device__ __forceinline__ bool same_lead(const uint32_t* keys, int W, uint32_t i, uint32_t j, int w, uint32_t mask) {
    const uint32_t *a = keys + (int64_t)i * W, *b = keys + (int64_t)j * W;
    if ((a[w] ^ b[w]) & mask) return false;
    for (int k = w - 1; k >= 0; --k)
        if (a[k] != b[k]) return false;
    return true;
}

// first[p]: the p-th row in order starts a run of equal leading digits;
// *longer: some run has more than kRunMax rows.
__global__ void run_starts_kernel(const uint32_t* keys, int W, const uint32_t* idx, int64_t n, int w, uint32_t mask,
                                  uint8_t* first, int* longer) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t i = idx[p];
        const bool same = p > 0 && same_lead(keys, W, i, idx[p - 1], w, mask);
        first[p] = same ? 0 : 1;
        if (same && p >= kRunMax && same_lead(keys, W, i, idx[p - kRunMax], w, mask)) *longer = 1;
    }
}

// Each row of a run goes to its place among the run's rows, by the words from
// w on, equal rows in the order they stand in.
__global__ void run_rank_kernel(const uint32_t* keys, int W, int sort_words, const uint32_t* idx, int64_t n, int w,
                                const uint8_t* first, uint32_t* out) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t i = idx[p];
        int64_t at = p;
        const uint32_t* a = keys + (int64_t)i * W;
        for (int64_t q = p; !first[q];) {  // rows before it that are greater
            const uint32_t* b = keys + (int64_t)idx[--q] * W;
            int k = w;
            while (k < sort_words && a[k] == b[k]) ++k;
            if (k < sort_words && a[k] < b[k]) --at;
        }
        for (int64_t q = p + 1; q < n && !first[q]; ++q) {  // rows after it that are less
            const uint32_t* b = keys + (int64_t)idx[q] * W;
            int k = w;
            while (k < sort_words && a[k] == b[k]) ++k;
            if (k < sort_words && b[k] < a[k]) ++at;
        }
        out[at] = i;
    }
}

__global__ void iota_kernel(uint32_t* p, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = (uint32_t)i;
}

__global__ void adjacent_diff_kernel(const uint32_t* keys, int W, const uint32_t* idx, int64_t n, int cmp_words,
                                     uint32_t* flags) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t f = 1;
        if (i > 0) {
            const uint32_t* a = keys + (int64_t)idx[i] * W;
            const uint32_t* b = keys + (int64_t)idx[i - 1] * W;
            f = 0;
            for (int w = 0; w < cmp_words; ++w)
                if (a[w] != b[w]) {
                    f = 1;
                    break;
                }
        }
        flags[i] = f;
    }
}

unsigned grid_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    if (g > 65535 * 16) g = 65535 * 16;
    return (unsigned)(g < 1 ? 1 : g);
}

}  // namespace

size_t scan_tmp_bytes(int64_t n) {
    size_t total = 0;
    while (n > kScanBlock) {
        n = (n + kScanBlock - 1) / kScanBlock;
        total += (size_t)n * 4 * 2;
    }
    return total + 256;
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* tmp, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
    if (nb == 1) {
        scan_block_kernel<<<1, kScanBlock, 0, st>>>(in, out, nullptr, n);
        return cudaGetLastError();
    }
    uint32_t* sums = tmp;
    uint32_t* sums_scan = tmp + nb;
    scan_block_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(in, out, sums, n);
    cudaError_t e = exclusive_scan_u32(sums, sums_scan, nb, tmp + 2 * nb, st);
    if (e != cudaSuccess) return e;
    scan_add_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(out, sums_scan, n);
    return cudaGetLastError();
}

cudaError_t compact_flags(const uint32_t* flags, const uint32_t* src, uint32_t* dst, int64_t n, uint32_t* pos_tmp,
                          uint32_t* scan_tmp, uint32_t* d_count, cudaStream_t st) {
    if (n <= 0) return cudaMemsetAsync(d_count, 0, 4, st);
    cudaError_t e = exclusive_scan_u32(flags, pos_tmp, n, scan_tmp, st);
    if (e != cudaSuccess) return e;
    compact_kernel<<<grid_for(n, 256), 256, 0, st>>>(flags, pos_tmp, src, dst, n, d_count);
    return cudaGetLastError();
}

cudaError_t mark_unique(const uint32_t* keys, int W, const uint32_t* idx, int64_t n, int cmp_words, uint32_t* flags,
                        cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    adjacent_diff_kernel<<<grid_for(n, 256), 256, 0, st>>>(keys, W, idx, n, cmp_words, flags);
    return cudaGetLastError();
}

cudaError_t iota_u32(uint32_t* p, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    iota_kernel<<<grid_for(n, 256), 256, 0, st>>>(p, n);
    return cudaGetLastError();
}

size_t radix_sort_tmp_bytes(int64_t n, int sort_words) {
    const int64_t nb = (n + kSortTile - 1) / kSortTile;
    return (size_t)n * 4                      // ping-pong index
           + (size_t)nb * 256 * 4 * 2         // counts + offsets
           + scan_tmp_bytes(nb * 256) + (size_t)std::min(sort_words, kTotalWords) * 4096 + 1024;
}

// Sorts idx (a permutation of row numbers) by the keys' first `sort_words`
// words (of W).  Stable.  tmp: radix_sort_tmp_bytes(n, sort_words) bytes of device memory.
// radix_bits: 4 or 8 bits per pass.
cudaError_t radix_sort_keys(const uint32_t* keys, int W, int sort_words, uint32_t* idx, int64_t n, void* tmp,
                            cudaStream_t st, int radix_bits) {
    if (n <= 1 || sort_words < 1) return cudaSuccess;
    if (radix_bits != 4 && radix_bits != 8) return cudaErrorInvalidValue;
    const int NB = 1 << radix_bits;
    const int per_word = 32 / radix_bits;
    const int64_t digits = (int64_t)per_word * sort_words;
    const int64_t nb = (n + kSortTile - 1) / kSortTile;
    uint8_t* t = static_cast<uint8_t*>(tmp);
    uint32_t* alt = reinterpret_cast<uint32_t*>(t);
    t += (size_t)n * 4;
    uint32_t* counts = reinterpret_cast<uint32_t*>(t);
    t += (size_t)nb * 256 * 4;
    uint32_t* offs = reinterpret_cast<uint32_t*>(t);
    t += (size_t)nb * 256 * 4;
    t = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(t) + 255) & ~uintptr_t(255));
    uint32_t* stmp = reinterpret_cast<uint32_t*>(t);
    // every digit's totals (at most 4 KB a word), read back for up to
    // kTotalWords words at a time, the leading ones first
    const int slice = std::min(sort_words, kTotalWords);
    int* longer = reinterpret_cast<int*>(stmp);
    uint32_t* total = stmp + 16;
    stmp += 16 + (size_t)slice * 1024;
    // Digits that differ, and the leading ones [lead, digits) that the first
    // passes sort by.  Digits that go together (a candidate's spectrum) hold
    // less than the sum of their entropies, hence twice log2 n; 43 passes of
    // an order-51 file of 380,000 lines become 7 (35 us each there).
    std::vector<char> varies(digits, 0);
    std::vector<uint32_t> htotal((size_t)slice * per_word * NB);
    int64_t lead = 0, below = 0;
    double entropy = 0.0;
    cudaError_t e;
    for (int w0 = 0; w0 < sort_words; w0 += slice) {
        const int words = std::min(slice, sort_words - w0);
        const int64_t last = per_word * (int64_t)(sort_words - w0 - words);  // the slice's last digit
        e = cudaMemsetAsync(longer, 0, 64 + (size_t)words * per_word * NB * 4, st);
        if (e != cudaSuccess) return e;
        const dim3 tg((unsigned)std::min<int64_t>((n + kSortThreads - 1) / kSortThreads, 1216), (unsigned)words);
        if (radix_bits == 8)
            radix_totals_kernel<8><<<tg, kSortThreads, 0, st>>>(keys + w0, W, words, n, total);
        else
            radix_totals_kernel<4><<<tg, kSortThreads, 0, st>>>(keys + w0, W, words, n, total);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(htotal.data(), total, (size_t)words * per_word * NB * 4, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        for (int bi = per_word * words - 1; bi >= 0; --bi) {
            double h = 0.0;
            for (int d = 0; d < NB; ++d) {
                const uint32_t c = htotal[(size_t)bi * NB + d];
                if (c == 0 || c == (uint32_t)n) continue;
                varies[last + bi] = 1;
                h -= (double)c / (double)n * std::log2((double)c / (double)n);
            }
            if (entropy >= 2.0 * std::log2((double)n)) {
                below += varies[last + bi];
            } else {
                entropy += h;
                lead = last + bi;
            }
        }
    }
    if (below <= kTailPasses) lead = below = 0;
    const bool rows = nb <= kScatterScanBlocks && sort_words <= slice;  // the totals of every digit are there
    uint32_t* cur = idx;
    uint32_t* nxt = alt;
    auto sort_by = [&](int64_t from) {
        for (int64_t bi = from; bi < digits; ++bi) {
            if (!varies[bi]) continue;  // every key has the same digit here
            const int word = (int)(sort_words - 1 - bi / per_word);
            const int shift = (int)(radix_bits * (bi % per_word));
            const uint32_t* tot = rows ? total + (size_t)bi * NB : nullptr;
            auto pass = [&](auto rb) {
                constexpr int RB = decltype(rb)::value;
                if (rows) {
                    radix_hist_kernel<RB, true><<<(unsigned)nb, kSortThreads, 0, st>>>(keys, W, cur, n, word, shift, counts, nb);
                    radix_scatter_kernel<RB, true><<<(unsigned)nb, kSortThreads, 0, st>>>(keys, W, cur, nxt, n, word, shift,
                                                                                          counts, nb, tot);
                    return cudaGetLastError();
                }
                radix_hist_kernel<RB, false><<<(unsigned)nb, kSortThreads, 0, st>>>(keys, W, cur, n, word, shift, counts, nb);
                const cudaError_t se = exclusive_scan_u32(counts, offs, nb * NB, stmp, st);
                if (se != cudaSuccess) return se;
                radix_scatter_kernel<RB, false><<<(unsigned)nb, kSortThreads, 0, st>>>(keys, W, cur, nxt, n, word, shift,
                                                                                       offs, nb, tot);
                return cudaGetLastError();
            };
            const cudaError_t pe =
                radix_bits == 8 ? pass(std::integral_constant<int, 8>{}) : pass(std::integral_constant<int, 4>{});
            if (pe != cudaSuccess) return pe;
            std::swap(cur, nxt);
        }
        return cudaSuccess;
    };
    e = sort_by(lead);
    if (e != cudaSuccess) return e;
    if (below) {
        const int w = (int)(sort_words - 1 - lead / per_word);
        const uint32_t mask = ~0u << (radix_bits * (lead % per_word));
        uint8_t* first = reinterpret_cast<uint8_t*>(counts);  // counts and offs: a byte per row at least
        run_starts_kernel<<<grid_for(n, 256), 256, 0, st>>>(keys, W, cur, n, w, mask, first, longer);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        int hlonger = 0;
        e = cudaMemcpyAsync(&hlonger, longer, 4, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        if (hlonger) {
            // rows with equal keys still stand in their first order
            e = sort_by(0);
        } else {
            run_rank_kernel<<<grid_for(n, 256), 256, 0, st>>>(keys, W, sort_words, cur, n, w, first, nxt);
            e = cudaGetLastError();
            std::swap(cur, nxt);
        }
        if (e != cudaSuccess) return e;
    }
    if (cur != idx) return cudaMemcpyAsync(idx, cur, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
    return cudaSuccess;
}

}  // namespace gp
