// gen_text.cu -- candidate files from the generation stage's records.
//
// The records stand on the device, in the order the finalize kernel appended
// them.  They are sorted there by role and word (the reference's FKM order:
// numeric order of the words, see rows.cuh), and their lines
// (src/utils/io.cpp:14-36) are written there too; the host copies the text
// and writes the two files.
//
// What bounds it: the copy and the files.  A generation call over an order-57
// window of 2^32 words with 40 MB of lines: 17.5 ms, 46 with the records
// copied, sorted and formatted by host threads.
#include <algorithm>
#include <new>

#include "ctx.h"
#include "gen_text.h"
#include "pair_text.cuh"
#include "prims.h"
#include "rows.cuh"

namespace gp {

namespace {

enum GtBuf { kGtKeys, kGtIdx, kGtTmp, kGtLen, kGtOff, kGtScan, kGtText, kGtCount };

// Key of a record: its role, then its word's W - 1 significant 32-bit words.
__global__ void record_keys_kernel(GenRecords r, int W, uint32_t* keys, unsigned* n_a) {
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < r.n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        bool a = false;
        if (i < r.n) {
            a = r.role[i] == 1;
            const uint4 w = r.words[i];
            uint32_t* k = keys + i * W;
            k[0] = a ? 0u : 1u;
            if (W == 5) {
                k[1] = w.w;
                k[2] = w.z;
            }
            k[W - 2] = w.y;
            k[W - 1] = w.x;
        }
        const int na = __syncthreads_count(a);
        if (threadIdx.x == 0 && na) atomicAdd(n_a, (unsigned)na);
    }
}

__global__ void record_bytes_kernel(GenRecords r, const uint32_t* idx, uint32_t* len) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < r.n; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t i = idx[k];
        const uint4 w = r.words[i];
        const uint64_t lo = ((uint64_t)w.y << 32) | w.x, hi = ((uint64_t)w.w << 32) | w.z;
        const uint16_t* sig = r.sig + (int64_t)i * (r.L - 1);
        int n = 5;  // "PSD", the blank after the signature, the newline
        for (int j = 0; j < r.L - 1; ++j) n += dec_digits(sig[j]);
        for (int j = 0; j < r.L; ++j) n += value_bytes(r.alpha[word_digit(lo, hi, r.b, r.L, j)]);
        len[k] = (uint32_t)n;
    }
}

__global__ void record_lines_kernel(GenRecords r, const uint32_t* idx, const uint32_t* off, char* text) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < r.n; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t i = idx[k];
        const uint4 w = r.words[i];
        const uint64_t lo = ((uint64_t)w.y << 32) | w.x, hi = ((uint64_t)w.w << 32) | w.z;
        const uint16_t* sig = r.sig + (int64_t)i * (r.L - 1);
        char* o = text + off[k];
        *o++ = 'P';
        *o++ = 'S';
        *o++ = 'D';
        for (int j = 0; j < r.L - 1; ++j) o = put_dec(o, sig[j]);
        *o++ = ' ';
        for (int j = 0; j < r.L; ++j) {
            const int v = r.alpha[word_digit(lo, hi, r.b, r.L, j)];
            if (v < 0) *o++ = '-';
            o = put_dec(o, (unsigned)(v < 0 ? -v : v));
            *o++ = ' ';
        }
        *o = '\n';
    }
}

}  // namespace

int records_to_text(gp_ctx* c, const GenRecords& r, GenText& out, cudaStream_t s) {
    out = GenText();
    if (r.n <= 0) {
        out.p.reset(new char[1]);
        return GP_OK;
    }
    // the longest line: five digits a signature value, "-15 " a value
    const uint64_t longest = 5 + 5ull * (r.L - 1) + 4ull * r.L;
    if ((uint64_t)r.n * longest >= (1ull << 32)) return GP_OK;
    const int W = r.b * r.L <= 64 ? 3 : 5;
    const int64_t n = r.n;
    DevBuf* b = c->gt;
    KeepSmall keep{c->gt};
    if (!b[kGtKeys].ensure((size_t)n * W * 4) || !b[kGtIdx].ensure((size_t)n * 4) ||
        !b[kGtTmp].ensure(radix_sort_tmp_bytes(n, W)) || !b[kGtLen].ensure((size_t)n * 4) ||
        !b[kGtOff].ensure((size_t)n * 4) || !b[kGtScan].ensure(scan_tmp_bytes(n)) || !b[kGtCount].ensure(4))
        return GP_OK;
    const unsigned grid = (unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)c->num_sms * 8);
    uint32_t *keys = b[kGtKeys].as<uint32_t>(), *idx = b[kGtIdx].as<uint32_t>(), *len = b[kGtLen].as<uint32_t>(),
             *off = b[kGtOff].as<uint32_t>();
    unsigned* count = b[kGtCount].as<unsigned>();
    GP_CUDA_TRY(c, cudaMemsetAsync(count, 0, 4, s));
    record_keys_kernel<<<grid, 256, 0, s>>>(r, W, keys, count);
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, iota_u32(idx, n, s));
    GP_CUDA_TRY(c, radix_sort_keys(keys, W, W, idx, n, b[kGtTmp].p, s, 8));
    record_bytes_kernel<<<grid, 256, 0, s>>>(r, idx, len);
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, exclusive_scan_u32(len, off, n, b[kGtScan].as<uint32_t>(), s));
    unsigned n_a = 0;
    uint32_t last[2] = {0, 0};
    GP_CUDA_TRY(c, cudaMemcpyAsync(&n_a, count, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last[0], off + n - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last[1], len + n - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    const size_t bytes = (size_t)last[0] + last[1];
    if (!b[kGtText].ensure(bytes)) return GP_OK;
    record_lines_kernel<<<grid, 256, 0, s>>>(r, idx, off, b[kGtText].as<char>());
    GP_CUDA_TRY(c, cudaGetLastError());
    uint32_t bytes_a = (uint32_t)bytes;
    std::shared_ptr<char[]> text(new (std::nothrow) char[bytes]);
    if (!text) return GP_OK;
    if ((int64_t)n_a < n) GP_CUDA_TRY(c, cudaMemcpyAsync(&bytes_a, off + n_a, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(text.get(), b[kGtText].p, bytes, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    out.p = std::move(text);
    out.bytes_a = bytes_a;
    out.bytes = bytes;
    out.n_a = (int64_t)n_a;
    out.n = n;
    return GP_OK;
}

}  // namespace gp
