// capi_sortmatch.cu -- sort and match stages.
//
// gp_sort replaces GNU_sort (src/core/sort/sort.cpp:7-22), i.e.
// `sort -S 2G -T dir files | uniq > out` in the C locale: every line becomes
// a fixed-width key (4 bits per character for the candidate alphabet
// ' ' '-' '0'-'9' 'D' 'P' 'S', else 8 bits per byte; the pad code sorts
// below every character, so a prefix sorts first as in a byte compare), the
// keys are radix-sorted on the device (stable LSD, prims.cu) and adjacent
// duplicates are dropped.
//
// gp_match replaces match_pairs (src/core/match/match_pairs.cpp:15-121):
// the sorted files are grouped by their first token, equal tokens of A and
// B are joined, and every pair of the cross product is checked on the device
// by exact integer PAF (src/utils/golay.cpp:27-44) using per-line PAF
// vectors.  Pairs are written in the reference's order: token order, then A
// line order, then B line order.
#include <algorithm>
#include <stdexcept>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include <fcntl.h>
#include <sys/stat.h>
#include <unistd.h>

#include "ctx.h"
#include "prims.h"
#include "host_par.h"
#include "pair_text.cuh"
#include "survivors.h"

namespace {

// 4-bit codes preserving byte order; 0 = padding
__host__ __device__ inline int code4(unsigned char ch) {
    switch (ch) {
        case ' ': return 1;
        case '-': return 2;
        case 'D': return 13;
        case 'P': return 14;
        case 'S': return 15;
        default: return (ch >= '0' && ch <= '9') ? 3 + (ch - '0') : -1;
    }
}

template <class Off>
__global__ void build_keys_kernel(const char* text, const Off* start, const uint32_t* len, int64_t n, int W,
                                  int nibble, uint32_t* keys) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const char* s = text + start[i];
        const uint32_t l = len[i];
        uint32_t* k = keys + i * W;
        const int per = nibble ? 8 : 4;
        const int bits = nibble ? 4 : 8;
        for (int w = 0; w < W; ++w) {
            uint32_t v = 0;
            for (int c = 0; c < per; ++c) {
                const uint32_t pos = (uint32_t)(w * per + c);
                uint32_t code = 0;
                if (pos < l) {
                    const unsigned char ch = (unsigned char)s[pos];
                    code = nibble ? (uint32_t)code4(ch) : (uint32_t)ch;
                }
                v = (v << bits) | code;
            }
            k[w] = v;
        }
    }
}

// PAF(s) = sum_i x_i x_{(i+s) mod L}, s = 1..L/2 (src/utils/golay.cpp:27-33)
__global__ void paf_kernel(const int8_t* seqs, int64_t n, int L, int H, int* paf) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int8_t* x = seqs + i * L;
        for (int s = 1; s <= H; ++s) {
            int r = 0;
            int j2 = s;
            for (int j = 0; j < L; ++j) {
                r += (int)x[j] * (int)x[j2];
                if (++j2 == L) j2 = 0;
            }
            paf[i * H + (s - 1)] = r;
        }
    }
}

struct GroupPair {
    uint32_t a0, na, b0, nb;
    uint64_t first;  // index of this group's first pair in the flattened product
};

// one thread per candidate pair of [w0, w0 + n): flags[w - w0] = 1 if pair w is
// complementary
__global__ void pair_check_kernel(const GroupPair* gps, int64_t ng, uint64_t w0, uint64_t n, const int* pafa,
                                  const int* pafb, int H, int target, uint32_t* flags) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t w = w0 + i;
        int64_t lo = 0, hi = ng - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (gps[mid].first <= w)
                lo = mid;
            else
                hi = mid - 1;
        }
        const GroupPair g = gps[lo];
        const uint64_t off = w - g.first;
        const uint32_t ia = g.a0 + (uint32_t)(off / g.nb);
        const uint32_t ib = g.b0 + (uint32_t)(off % g.nb);
        const int* pa = pafa + (int64_t)ia * H;
        const int* pb = pafb + (int64_t)ib * H;
        uint32_t ok = 1;
        for (int s = 0; s < H; ++s)
            if (pa[s] + pb[s] != target) {
                ok = 0;
                break;
            }
        flags[i] = ok;
    }
}

unsigned grid_for(int64_t n) {
    int64_t g = (n + 255) / 256;
    if (g > 65535 * 8) g = 65535 * 8;
    return (unsigned)(g < 1 ? 1 : g);
}

// ------------------------------------------------------------ text on the device
// A file's bytes go to the device as they are; its lines are found, keyed,
// compared and written out there.  Offsets are 32 bits: more text than that
// takes the host's line index (gp_sort_text, gp_match_texts).  Sort and match
// of the 430,000 lines of a whole order 51: 10.6 ms, 43.3 with the lines, the
// parse, the merge and the copies on host threads.
constexpr int kTextThreads = 256;
constexpr int kTextEach = 16;                            // bytes per thread
constexpr int kTextBlock = kTextThreads * kTextEach;
constexpr uint64_t kMaxDeviceText = (uint64_t(1) << 32) - 2 * kTextBlock;

// Newlines of a text padded to whole blocks (by anything but newlines).
// WRITE = false: per block; true: line i + 1 starts after the i-th newline.
// *other: set when a character is none of "0-9", "-", "P", "S", "D", blank, newline.
template <bool WRITE>
__global__ void __launch_bounds__(kTextThreads) line_starts_kernel(const char* text, uint32_t n, uint32_t* counts,
                                                                   const uint32_t* offs, uint32_t* start,
                                                                   int* other) {
    __shared__ uint32_t s_warp[kTextThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t p0 = blockIdx.x * (uint32_t)kTextBlock + threadIdx.x * kTextEach;
    const uint4 w = *reinterpret_cast<const uint4*>(text + p0);
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    uint32_t nl = 0;
    bool odd = false;
#pragma unroll
    for (int k = 0; k < kTextEach; ++k) {
        const int c = (ww[k >> 2] >> (8 * (k & 3))) & 0xFF;
        if (p0 + k >= n) break;
        if (c == '\n')
            nl |= 1u << k;
        else if (code4((unsigned char)c) < 0)
            odd = true;
    }
    const uint32_t mine = (uint32_t)__popc(nl);
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int q = 0; q < kTextThreads / 32; ++q) {
        if (q < warp) before += s_warp[q];
        total += s_warp[q];
    }
    if constexpr (!WRITE) {
        if (threadIdx.x == 0) counts[blockIdx.x] = total;
        if (odd) *other = 1;
    } else {
        uint32_t* out = start + offs[blockIdx.x] + before + incl - mine + 1;
        for (uint32_t m = nl; m; m &= m - 1u) *out++ = p0 + (uint32_t)__ffs((int)m);
        if (blockIdx.x == 0 && threadIdx.x == 0) start[0] = 0;
    }
}

// Lengths without the newline, and the longest.
__global__ void line_lengths_kernel(const uint32_t* start, int64_t n, uint32_t* len, unsigned* longest) {
    unsigned most = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t l = start[i + 1] - start[i] - 1;
        len[i] = l;
        most = l > most ? l : most;
    }
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    if ((threadIdx.x & 31) == 0 && most) atomicMax(longest, most);
}

// Candidate lines: the first token's place, then exactly L integers, read
// as parse_candidates reads them (the text holds none of the characters on
// which the two could differ).  A line of blanks is no candidate (tok_len 0);
// *bad: a line with fewer integers.
__global__ void parse_lines_kernel(const char* text, const uint32_t* start, const uint32_t* len, int64_t n, int L,
                                   uint32_t* tok_off, uint32_t* tok_len, int8_t* seqs, int* bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const char* q = text + start[i];
        const char* const end = q + len[i];
        while (q < end && *q == ' ') ++q;
        const char* const t = q;
        while (q < end && *q != ' ') ++q;
        tok_off[i] = (uint32_t)(t - text);
        tok_len[i] = (uint32_t)(q - t);
        if (q == t) {
            *bad = 1;  // a line of blanks (left to the host)
            continue;
        }
        int got = 0;
        for (; got < L; ++got) {
            while (q < end && *q == ' ') ++q;
            const bool neg = q < end && *q == '-';
            if (neg) ++q;
            if (q >= end || *q < '0' || *q > '9') break;
            unsigned v = 0;
            for (; q < end && *q >= '0' && *q <= '9'; ++q) v = v * 10 + (unsigned)(*q - '0');
            seqs[i * L + got] = (int8_t)(neg ? 0u - v : v);
        }
        if (got != L) *bad = 1;
    }
}

// -1, 0, 1: byte order of two tokens, a prefix first
__device__ __forceinline__ int compare_tokens(const char* a, uint32_t la, const char* b, uint32_t lb) {
    const uint32_t l = la < lb ? la : lb;
    for (uint32_t k = 0; k < l; ++k) {
        const unsigned char x = (unsigned char)a[k], y = (unsigned char)b[k];
        if (x != y) return x < y ? -1 : 1;
    }
    return la == lb ? 0 : la < lb ? -1 : 1;
}

// *bad: a token above the next line's (the merge of unsorted files is the host's)
__global__ void tokens_sorted_kernel(const char* text, const uint32_t* off, const uint32_t* len, int64_t n, int* bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i + 1 < n; i += (int64_t)gridDim.x * blockDim.x)
        if (compare_tokens(text + off[i], len[i], text + off[i + 1], len[i + 1]) > 0) *bad = 1;
}

// For every a line the b lines with its token: [b0, b0 + nb).
__global__ void token_ranges_kernel(const char* ta, const uint32_t* oa, const uint32_t* la, int64_t na,
                                    const char* tb, const uint32_t* ob, const uint32_t* lb, int64_t nb_lines,
                                    uint32_t* b0, uint32_t* nb, unsigned long long* total) {
    unsigned long long sum = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x) {
        const char* t = ta + oa[i];
        const uint32_t l = la[i];
        uint32_t lo = 0, hi = (uint32_t)nb_lines;  // first line not below the token
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (compare_tokens(tb + ob[mid], lb[mid], t, l) < 0)
                lo = mid + 1;
            else
                hi = mid;
        }
        uint32_t e = lo, step = 1;  // first line above it: a few lines on
        while (e < nb_lines && compare_tokens(tb + ob[e], lb[e], t, l) == 0) {
            ++e;
            if (++step > 8) {
                uint32_t top = (uint32_t)nb_lines;
                while (e < top) {
                    const uint32_t mid = e + (top - e) / 2;
                    if (compare_tokens(tb + ob[mid], lb[mid], t, l) <= 0)
                        e = mid + 1;
                    else
                        top = mid;
                }
                break;
            }
        }
        b0[i] = lo;
        nb[i] = e - lo;
        sum += e - lo;
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, sum);
}

// one thread per candidate pair (a line, line of its range): flags[w] = 1 if
// the pair is complementary
__global__ void range_check_kernel(const uint32_t* first, const uint32_t* b0, int64_t na, uint32_t total,
                                   const int* pafa, const int* pafb, int H, int target, uint32_t* flags,
                                   uint32_t* ia, uint32_t* ib) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (uint64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = na - 1;  // the last a line whose first pair is <= w
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (first[mid] <= w)
                lo = mid;
            else
                hi = mid - 1;
        }
        const uint32_t b = b0[lo] + (uint32_t)(w - first[lo]);
        ia[w] = (uint32_t)lo;
        ib[w] = b;
        const int* pa = pafa + lo * H;
        const int* pb = pafb + (int64_t)b * H;
        uint32_t ok = 1;
        for (int s = 0; s < H; ++s)
            if (pa[s] + pb[s] != target) {
                ok = 0;
                break;
            }
        flags[w] = ok;
    }
}

// The kept pairs' lines (src/io.cpp PairWriter).
__global__ void match_line_bytes_kernel(const int8_t* a, const int8_t* b, const uint32_t* ia, const uint32_t* ib,
                                        const uint32_t* keep, int64_t n, int L, uint32_t* bytes) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        bytes[k] = (uint32_t)gp::pair_line_bytes(a + (int64_t)ia[keep[k]] * L, b + (int64_t)ib[keep[k]] * L, L);
}
__global__ void __launch_bounds__(256) match_lines_kernel(const int8_t* a, const int8_t* b, const uint32_t* ia,
                                                          const uint32_t* ib, const uint32_t* keep, int64_t n, int L,
                                                          const uint32_t* at, char* text) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t k = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < n; k += warps)
        gp::put_pair_line(a + (int64_t)ia[keep[k]] * L, b + (int64_t)ib[keep[k]] * L, L, text + at[k]);
}

// A file's bytes, unset until read: pieces read by host threads.  A directory
// is an error, not a file of no bytes.
struct FileText {
    std::unique_ptr<char[]> p;
    size_t n = 0;
};
bool read_file(const char* path, FileText& t) {
    const int fd = open(path, O_RDONLY);
    if (fd < 0) return false;
    struct Closer {
        int fd;
        ~Closer() { close(fd); }
    } closer{fd};
    struct stat sb;
    const bool known = fstat(fd, &sb) == 0;
    if (known && S_ISDIR(sb.st_mode)) throw std::runtime_error(std::string(path) + " is a directory");
    const size_t size = known && S_ISREG(sb.st_mode) && sb.st_size > 0 ? (size_t)sb.st_size : 0;
    t.p.reset(new char[size + 1]);
    constexpr size_t kPiece = size_t(2) << 20;
    const size_t pieces = (size + kPiece - 1) / kPiece;
    std::vector<size_t> got(pieces, 0);
    gp::par_for(pieces, [&](size_t k) {
        const size_t lo = k * kPiece, hi = std::min(size, lo + kPiece);
        size_t at = lo;
        while (at < hi) {
            const ssize_t r = pread(fd, t.p.get() + at, hi - at, (off_t)at);
            if (r <= 0) break;
            at += (size_t)r;
        }
        got[k] = at - lo;
    });
    t.n = 0;
    for (size_t k = 0; k < pieces; ++k) {  // a file cut short meanwhile ends at its first short piece
        t.n += got[k];
        if (got[k] < std::min(kPiece, size - k * kPiece)) break;
    }
    t.p[t.n] = 0;
    return true;
}

// A stage's output file: closed on every way out, and whole only if every
// write and the close say so (a large write goes past the stream's buffer, so
// on a full disk the close alone can succeed).
struct OutFile {
    FILE* f;
    bool whole = true;
    OutFile(const char* path, const char* mode) : f(fopen(path, mode)) {}
    ~OutFile() {
        if (f) fclose(f);
    }
    OutFile(const OutFile&) = delete;
    OutFile& operator=(const OutFile&) = delete;
    void put(const char* p, size_t n) { whole = fwrite(p, 1, n, f) == n && whole; }
    bool close() {
        whole = fclose(f) == 0 && whole;
        f = nullptr;
        return whole;
    }
};

// The sort's output (an input may have the same name: it has been read by now).
int write_file(gp_ctx* c, const char* p, size_t n, const char* path) {
    OutFile f(path, "w");
    if (!f.f) return c->fail(GP_ERR_IO, "sort: cannot write %s", path);
    f.put(p, n);
    return f.close() ? GP_OK : c->fail(GP_ERR_IO, "sort: write failed: %s", path);
}

// The same from device text.
int write_text(gp_ctx* c, const char* d_text, size_t n, const char* path, cudaStream_t s) {
    std::unique_ptr<char[]> h(new char[n + 1]);
    GP_CUDA_TRY(c, cudaMemcpyAsync(h.get(), d_text, n, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    return write_file(c, h.get(), n, path);
}

// The context's sort and match buffers, one use each.
enum TextBuf { kTbText, kTbTextB, kTbCount, kTbOffs, kTbScan, kTbMisc, kTbStart, kTbLen, kTbStartB, kTbLenB, kTbKeys, kTbIdx,
               kTbTmp, kTbFlag, kTbPos, kTbOrder, kTbOutLen, kTbOutOff, kTbOut, kTbTokA, kTbTokLenA, kTbTokB,
               kTbTokLenB, kTbSeqA, kTbSeqB, kTbPafA, kTbPafB, kTbIa, kTbIb };

// A text of n bytes, ending in a newline, at d_text (room for a block past
// it): its lines' starts (lines + 1 entries) and lengths, their number, the
// longest, and whether it holds other characters than candidate lines do.
struct Lines {
    int64_t n = 0;
    unsigned longest = 0;
    int other = 0;
};
int find_lines(gp_ctx* c, const char* d_text, size_t n, DevBuf& start, DevBuf& len, Lines& out, cudaStream_t s) {
    const int64_t blocks = (int64_t)((n + kTextBlock - 1) / kTextBlock);
    DevBuf &cnt = c->st[kTbCount], &off = c->st[kTbOffs], &scan = c->st[kTbScan], &misc = c->st[kTbMisc];
    if (!cnt.ensure((size_t)blocks * 4) || !off.ensure((size_t)blocks * 4) || !scan.ensure(gp::scan_tmp_bytes(blocks)) ||
        !misc.ensure(64))
        return c->fail(GP_ERR_NOMEM, "text: device allocation");
    GP_CUDA_TRY(c, cudaMemsetAsync(misc.p, 0, 64, s));
    int* d_other = misc.as<int>();
    unsigned* d_longest = misc.as<unsigned>() + 1;
    line_starts_kernel<false><<<(unsigned)blocks, kTextThreads, 0, s>>>(d_text, (uint32_t)n, cnt.as<uint32_t>(),
                                                                        nullptr, nullptr, d_other);
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, gp::exclusive_scan_u32(cnt.as<uint32_t>(), off.as<uint32_t>(), blocks, scan.as<uint32_t>(), s));
    uint32_t last[2] = {0, 0};
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last[0], off.as<uint32_t>() + blocks - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last[1], cnt.as<uint32_t>() + blocks - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    out.n = (int64_t)last[0] + last[1];
    if (!start.ensure((size_t)(out.n + 1) * 4) || !len.ensure((size_t)out.n * 4 + 4))
        return c->fail(GP_ERR_NOMEM, "text: device allocation");
    line_starts_kernel<true><<<(unsigned)blocks, kTextThreads, 0, s>>>(d_text, (uint32_t)n, nullptr, off.as<uint32_t>(),
                                                                       start.as<uint32_t>(), nullptr);
    line_lengths_kernel<<<(unsigned)std::min<int64_t>((out.n + 255) / 256 + 1, 4096), 256, 0, s>>>(
        start.as<uint32_t>(), out.n, len.as<uint32_t>(), d_longest);
    GP_CUDA_TRY(c, cudaGetLastError());
    int h[2] = {0, 0};
    GP_CUDA_TRY(c, cudaMemcpyAsync(h, misc.p, 8, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    out.other = h[0];
    out.longest = (unsigned)h[1];
    return GP_OK;
}

struct Cand {
    std::vector<size_t> tok_off, tok_len;  // first token in the text (of any size)
    std::vector<int8_t> seqs;                // L per line
    size_t n = 0;
};

// Parses candidate lines: a first token, then exactly L integers.  Chunks
// of whole lines are parsed by host threads, then joined in order.
bool parse_candidates(const std::string& text, int L, Cand& out, std::string& err) {
    const char* base = text.data();
    const char* tend = base + text.size();
    const std::vector<size_t> cut = gp::line_chunks(base, text.size(), std::min<size_t>(4 * gp::host_threads(), text.size() / (1 << 18) + 1));
    const size_t nc = cut.size() - 1;
    std::vector<Cand> part(nc);
    std::vector<char> bad(nc, 0);
    gp::par_for(nc, [&](size_t k) {
        Cand& o = part[k];
        const char* p = base + cut[k];
        const char* end = base + cut[k + 1];
        while (p < end) {
            const char* nl = (const char*)memchr(p, '\n', (size_t)(end - p));
            if (!nl) nl = end;
            const char* q = p;
            while (q < nl && *q == ' ') ++q;
            if (q < nl) {
                const char* t = q;
                while (q < nl && *q != ' ') ++q;
                o.tok_off.push_back((size_t)(t - base));
                o.tok_len.push_back((size_t)(q - t));
                int got = 0;
                while (got < L) {
                    while (q < nl && *q == ' ') ++q;
                    if (q >= nl) break;
                    const char* e;
                    const long v = gp::read_long(q, tend, &e);
                    if (e == q) break;
                    o.seqs.push_back((int8_t)v);
                    ++got;
                    q = e;
                }
                if (got != L) {
                    bad[k] = 1;
                    return;
                }
                o.n++;
            }
            p = nl + 1;
        }
    });
    for (size_t k = 0; k < nc; ++k)
        if (bad[k]) {
            err = "candidate line with fewer than L values";
            return false;
        }
    size_t n = 0, ns = 0;
    for (const Cand& o : part) {
        n += o.n;
        ns += o.seqs.size();
    }
    out.tok_off.reserve(n);
    out.tok_len.reserve(n);
    out.seqs.reserve(ns);
    for (const Cand& o : part) {
        out.tok_off.insert(out.tok_off.end(), o.tok_off.begin(), o.tok_off.end());
        out.tok_len.insert(out.tok_len.end(), o.tok_len.begin(), o.tok_len.end());
        out.seqs.insert(out.seqs.end(), o.seqs.begin(), o.seqs.end());
        out.n += o.n;
    }
    return true;
}

// src/io.cpp PairWriter line: a entries, one more space, b entries
void put_pair(std::string& s, const int8_t* a, const int8_t* b, int L) {
    for (int i = 0; i < L; ++i) gp::put_int_sp(s, a[i]);
    s.push_back(' ');
    for (int i = 0; i < L; ++i) gp::put_int_sp(s, b[i]);
    s.push_back('\n');
}

}  // namespace

// Candidate pairs checked at once: their indices in a slice are 32 bits, and the
// slice's arrays 12 GB.
constexpr uint64_t kMatchSlice = uint64_t(1) << 30;

// Match two candidate texts and append the pairs to `out`: any size of text and
// any number of candidate pairs, up to 2^32 - 1 lines a side.  Returns
// GP_EMPTY_INPUT if either text is empty.
int gp_match_texts(gp_ctx* c, int L, int compress, int paf, const std::string& ta, const std::string& tb,
                   std::string& out, int64_t* n_pairs) {
    if (ta.empty() || tb.empty()) return GP_EMPTY_INPUT;
    Cand A, B;
    std::string err;
    if (!parse_candidates(ta, L, A, err) || !parse_candidates(tb, L, B, err)) return c->fail(GP_ERR_FORMAT, "match: %s", err.c_str());
    if (std::max(A.n, B.n) > UINT32_MAX)
        return c->fail(GP_ERR_UNSUPPORTED, "match: %zu lines", std::max(A.n, B.n));
    // group boundaries and the merge on the first token (std::string order)
    auto tok = [](const std::string& t, const Cand& x, size_t i) {
        return std::string_view(t.data() + x.tok_off[i], x.tok_len[i]);
    };
    std::vector<GroupPair> gps;
    uint64_t total = 0;
    size_t i = 0, j = 0;
    while (i < A.n && j < B.n) {
        const auto x = tok(ta, A, i), y = tok(tb, B, j);
        const int cmp = x.compare(y);
        if (cmp == 0) {
            size_t i2 = i, j2 = j;
            while (i2 < A.n && tok(ta, A, i2) == x) ++i2;
            while (j2 < B.n && tok(tb, B, j2) == y) ++j2;
            gps.push_back({(uint32_t)i, (uint32_t)(i2 - i), (uint32_t)j, (uint32_t)(j2 - j), total});
            total += (uint64_t)(i2 - i) * (j2 - j);
            i = i2;
            j = j2;
        } else if (cmp < 0) {
            ++i;
        } else {
            ++j;
        }
    }
    if (n_pairs) *n_pairs = 0;
    if (total == 0) return GP_OK;
    cudaStream_t s = c->s_comp;
    const int H = L / 2;
    DevBuf da, db, dpa, dpb, dg, df, dpos, dscan, dlist;
    const int64_t slice = (int64_t)std::min(total, kMatchSlice);
    if (!da.ensure(A.seqs.size() + 16) || !db.ensure(B.seqs.size() + 16) || !dpa.ensure(A.n * (H + 1) * 4) ||
        !dpb.ensure(B.n * (H + 1) * 4) || !dg.ensure(gps.size() * sizeof(GroupPair)) || !df.ensure(slice * 4) ||
        !dpos.ensure(slice * 4) || !dscan.ensure(gp::scan_tmp_bytes(slice)) || !dlist.ensure(slice * 4 + 4))
        return c->fail(GP_ERR_NOMEM, "match: device allocation");
    GP_CUDA_TRY(c, cudaMemcpyAsync(da.p, A.seqs.data(), A.seqs.size(), cudaMemcpyHostToDevice, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(db.p, B.seqs.data(), B.seqs.size(), cudaMemcpyHostToDevice, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(dg.p, gps.data(), gps.size() * sizeof(GroupPair), cudaMemcpyHostToDevice, s));
    if (H > 0) {
        paf_kernel<<<grid_for((int64_t)A.n), 256, 0, s>>>(da.as<int8_t>(), (int64_t)A.n, L, H, dpa.as<int>());
        paf_kernel<<<grid_for((int64_t)B.n), 256, 0, s>>>(db.as<int8_t>(), (int64_t)B.n, L, H, dpb.as<int>());
    }
    std::vector<uint64_t> keep;  // in the flattened product
    std::vector<uint32_t> kept;  // in a slice
    for (uint64_t w0 = 0; w0 < total; w0 += slice) {
        const int64_t n = (int64_t)std::min<uint64_t>(slice, total - w0);
        pair_check_kernel<<<grid_for(n), 256, 0, s>>>(dg.as<GroupPair>(), (int64_t)gps.size(), w0, (uint64_t)n,
                                                      dpa.as<int>(), dpb.as<int>(), H, paf * compress,
                                                      df.as<uint32_t>());
        GP_CUDA_TRY(c, cudaGetLastError());
        uint32_t* d_cnt = dlist.as<uint32_t>() + n;
        GP_CUDA_TRY(c, gp::compact_flags(df.as<uint32_t>(), nullptr, dlist.as<uint32_t>(), n, dpos.as<uint32_t>(),
                                         dscan.as<uint32_t>(), d_cnt, s));
        uint32_t nk = 0;
        GP_CUDA_TRY(c, cudaMemcpyAsync(&nk, d_cnt, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        kept.resize(nk);
        if (nk) GP_CUDA_TRY(c, cudaMemcpy(kept.data(), dlist.p, (size_t)nk * 4, cudaMemcpyDeviceToHost));
        for (uint32_t k : kept) keep.push_back(w0 + k);
    }
    // pair lines in order, formatted in blocks by host threads
    const size_t per = 1 << 14;
    const size_t nblk = (keep.size() + per - 1) / per;
    std::vector<std::string> blk(nblk);
    gp::par_for(nblk, [&](size_t bi) {
        const size_t lo = bi * per, hi = std::min(keep.size(), lo + per);
        std::string& o = blk[bi];
        o.reserve((hi - lo) * (size_t)(6 * L + 2));
        size_t g = (size_t)(std::upper_bound(gps.begin(), gps.end(), keep[lo],
                                             [](uint64_t w, const GroupPair& x) { return w < x.first; }) -
                            gps.begin()) - 1;
        for (size_t k = lo; k < hi; ++k) {
            const uint64_t w = keep[k];
            while (g + 1 < gps.size() && gps[g + 1].first <= w) ++g;
            const uint64_t off = w - gps[g].first;
            const uint32_t ia = gps[g].a0 + (uint32_t)(off / gps[g].nb);
            const uint32_t ib = gps[g].b0 + (uint32_t)(off % gps[g].nb);
            put_pair(o, A.seqs.data() + (size_t)ia * L, B.seqs.data() + (size_t)ib * L, L);
        }
    });
    for (const std::string& o : blk) out += o;
    if (n_pairs) *n_pairs = (int64_t)keep.size();
    return GP_OK;
}

// The sort's tuner: per key width, times whole sorts with 8- and 4-bit
// passes on (up to) the first 2^18 keys, twice each (the first round warms
// up), and keeps the faster; cached in the context.  Leaves di scrambled.
int sort_radix_bits(gp_ctx* c, const uint32_t* dk, int Wk, int64_t n, uint32_t* di, void* tmp, cudaStream_t s,
                    int* bits) {
    const std::string key = "sort:W" + std::to_string(Wk);
    auto it = c->tuned.find(key);
    if (it != c->tuned.end()) {
        *bits = (int)it->second[0];
        return GP_OK;
    }
    *bits = 8;
    if (n < (1 << 14)) return GP_OK;  // too small to time: default, not cached
    const int64_t m = std::min<int64_t>(n, 1 << 18);
    double best = 1e300;
    const int order[4] = {8, 4, 8, 4};
    for (int r = 0; r < 4; ++r) {
        GP_CUDA_TRY(c, gp::iota_u32(di, m, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        const auto t0 = std::chrono::steady_clock::now();
        GP_CUDA_TRY(c, gp::radix_sort_keys(dk, Wk, Wk, di, m, tmp, s, order[r]));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (r >= 2 && el < best) {
            best = el;
            *bits = order[r];
        }
    }
    c->tuned[key] = {*bits, (int64_t)(best * 1e6)};
    return GP_OK;
}

// Sorted, de-duplicated lines of `text` (byte order).
int gp_sort_text(gp_ctx* c, const std::string& text, std::string& out) {
    std::vector<uint64_t> start;
    std::vector<uint32_t> len;
    size_t maxlen = 0;
    bool nibble = true;
    {
        // lines and the character check, by chunks of whole lines on host
        // threads, joined in order
        const char* base = text.data();
        const std::vector<size_t> cut = gp::line_chunks(base, text.size(), std::min<size_t>(4 * gp::host_threads(), text.size() / (1 << 18) + 1));
        const size_t nc = cut.size() - 1;
        std::vector<std::vector<uint64_t>> ps(nc);
        std::vector<std::vector<uint32_t>> pl(nc);
        std::vector<size_t> pmax(nc, 0);
        std::vector<char> pnib(nc, 1);
        gp::par_for(nc, [&](size_t k) {
            const char* p = base + cut[k];
            const char* end = base + cut[k + 1];
            for (const char* q = p; q < end; ++q)
                if (*q != '\n' && code4((unsigned char)*q) < 0) {
                    pnib[k] = 0;
                    break;
                }
            while (p < end) {
                const char* nl = (const char*)memchr(p, '\n', (size_t)(end - p));
                const size_t l = nl ? (size_t)(nl - p) : (size_t)(end - p);
                ps[k].push_back((uint64_t)(p - base));
                pl[k].push_back((uint32_t)l);
                pmax[k] = std::max(pmax[k], l);
                p += l + 1;
            }
        });
        size_t tot = 0;
        for (size_t k = 0; k < nc; ++k) tot += ps[k].size();
        start.reserve(tot);
        len.reserve(tot);
        for (size_t k = 0; k < nc; ++k) {
            start.insert(start.end(), ps[k].begin(), ps[k].end());
            len.insert(len.end(), pl[k].begin(), pl[k].end());
            maxlen = std::max(maxlen, pmax[k]);
            nibble = nibble && pnib[k];
        }
    }
    const int64_t n = (int64_t)start.size();
    out.clear();
    if (n == 0) return GP_OK;
    // line numbers and lengths are 32 bits
    if (n > UINT32_MAX || maxlen > UINT32_MAX)
        return c->fail(GP_ERR_UNSUPPORTED, "sort: %lld lines, the longest of %zu bytes", (long long)n, maxlen);
    const int per = nibble ? 8 : 4;
    const int W = (int)((maxlen + per - 1) / per) + 0;
    const int Wk = W < 1 ? 1 : W;
    cudaStream_t s = c->s_comp;
    DevBuf dt, ds, dl, dk, di, dtmp, dflag, dpos, dscan, dout;
    if (!dt.ensure(text.size() + 16) || !ds.ensure(n * 8) || !dl.ensure(n * 4) || !dk.ensure((size_t)n * Wk * 4) ||
        !di.ensure(n * 4) || !dtmp.ensure(gp::radix_sort_tmp_bytes(n, Wk)) || !dflag.ensure(n * 4) || !dpos.ensure(n * 4) ||
        !dscan.ensure(gp::scan_tmp_bytes(n)) || !dout.ensure(n * 4 + 4))
        return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    GP_CUDA_TRY(c, cudaMemcpyAsync(dt.p, text.data(), text.size(), cudaMemcpyHostToDevice, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(ds.p, start.data(), n * 8, cudaMemcpyHostToDevice, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(dl.p, len.data(), n * 4, cudaMemcpyHostToDevice, s));
    build_keys_kernel<<<grid_for(n), 256, 0, s>>>(dt.as<char>(), ds.as<uint64_t>(), dl.as<uint32_t>(), n, Wk,
                                                  nibble ? 1 : 0, dk.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    int bits = 8;
    int rc = sort_radix_bits(c, dk.as<uint32_t>(), Wk, n, di.as<uint32_t>(), dtmp.p, s, &bits);
    if (rc) return rc;
    GP_CUDA_TRY(c, gp::iota_u32(di.as<uint32_t>(), n, s));
    GP_CUDA_TRY(c, gp::radix_sort_keys(dk.as<uint32_t>(), Wk, Wk, di.as<uint32_t>(), n, dtmp.p, s, bits));
    GP_CUDA_TRY(c, gp::mark_unique(dk.as<uint32_t>(), Wk, di.as<uint32_t>(), n, Wk, dflag.as<uint32_t>(), s));
    uint32_t* d_cnt = dout.as<uint32_t>() + n;
    GP_CUDA_TRY(c, gp::compact_flags(dflag.as<uint32_t>(), di.as<uint32_t>(), dout.as<uint32_t>(), n, dpos.as<uint32_t>(),
                                     dscan.as<uint32_t>(), d_cnt, s));
    uint32_t nu = 0;
    GP_CUDA_TRY(c, cudaMemcpyAsync(&nu, d_cnt, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    std::vector<uint32_t> order(nu);
    if (nu) GP_CUDA_TRY(c, cudaMemcpy(order.data(), dout.p, (size_t)nu * 4, cudaMemcpyDeviceToHost));
    // output: each kept line and its newline at a prefix-sum offset, copied
    // by host threads
    std::vector<size_t> at(nu + 1, 0);
    for (uint32_t k = 0; k < nu; ++k) at[k + 1] = at[k] + len[order[k]] + 1;
    out.resize(at[nu]);
    const size_t lines_per = 1 << 15;
    gp::par_for((nu + lines_per - 1) / lines_per, [&](size_t bi) {
        const size_t lo = bi * lines_per, hi = std::min<size_t>(nu, lo + lines_per);
        for (size_t k = lo; k < hi; ++k) {
            const uint32_t i = order[k];
            std::memcpy(&out[at[k]], text.data() + start[i], len[i]);
            out[at[k] + len[i]] = '\n';
        }
    });
    return GP_OK;
}

// ------------------------------------------------ binary survivor inputs
// Every input a binary survivor file of one job: the records go to the
// device as they are, the device formats their lines (the text the
// generation call would have written, survivors.h), sorts them with the
// same keys as text input and gathers the kept lines in order; the host
// only reads the files and writes the sorted text.

struct SurvGeom {
    int L, bits, k, sig_bytes, word_bytes, rec_bytes;
    int alpha[16];
};

__device__ __forceinline__ void rec_word(const uint8_t* r, int word_bytes, uint64_t& lo, uint64_t& hi) {
    lo = hi = 0;
    for (int i = 0; i < word_bytes; ++i) {
        const uint64_t b = r[i];
        if (i < 8)
            lo |= b << (8 * i);
        else
            hi |= b << (8 * (i - 8));
    }
}

__device__ __forceinline__ int rec_digit(uint64_t lo, uint64_t hi, int bits, int L, int j) {
    const int pos = bits * (L - 1 - j);
    const uint64_t m = (1ull << bits) - 1ull;
    if (pos >= 64) return (int)((hi >> (pos - 64)) & m);
    uint64_t v = lo >> pos;
    if (pos + bits > 64 && pos > 0) v |= hi << (64 - pos);
    return (int)(v & m);
}

__device__ __forceinline__ unsigned rec_sig(const uint8_t* r, const SurvGeom& g, int k) {
    const uint8_t* s = r + g.word_bytes;
    return g.sig_bytes == 1 ? s[k] : (unsigned)(s[2 * k] | (s[2 * k + 1] << 8));
}

// line length (newline included) of every record; a digit past the
// alphabet or bits above the word make the input malformed
__global__ void surv_len_kernel(const uint8_t* recs, int64_t n, SurvGeom g, uint32_t* len, unsigned* maxlen,
                                int* bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t* r = recs + i * g.rec_bytes;
        uint64_t lo, hi;
        rec_word(r, g.word_bytes, lo, hi);
        const int used = g.bits * g.L;
        const bool high = used < 64 ? (lo >> used) != 0 || hi != 0 : (used < 128 && (hi >> (used - 64)) != 0);
        uint32_t l = 3 + 1 + 1;  // "PSD", the space after the signature, the newline
        for (int k = 0; k < g.L - 1; ++k) l += (uint32_t)gp::dec_digits(rec_sig(r, g, k));
        bool ok = !high;
        for (int j = 0; j < g.L; ++j) {
            const int d = rec_digit(lo, hi, g.bits, g.L, j);
            if (d >= g.k) {
                ok = false;
                break;
            }
            const int v = g.alpha[d];
            l += (uint32_t)(gp::dec_digits((unsigned)(v < 0 ? -v : v)) + (v < 0) + 1);
        }
        if (!ok) atomicExch(bad, 1);
        len[i] = l;
        atomicMax(maxlen, l - 1);
    }
}

// each record's line (src/utils/io.cpp:14-36) at its offset
__global__ void surv_format_kernel(const uint8_t* recs, int64_t n, SurvGeom g, const uint32_t* off, char* text,
                                   uint32_t* start, uint32_t* len) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t* r = recs + i * g.rec_bytes;
        uint64_t lo, hi;
        rec_word(r, g.word_bytes, lo, hi);
        char* o = text + off[i];
        char* const o0 = o;
        *o++ = 'P';
        *o++ = 'S';
        *o++ = 'D';
        for (int k = 0; k < g.L - 1; ++k) o = gp::put_dec(o, rec_sig(r, g, k));
        *o++ = ' ';
        for (int j = 0; j < g.L; ++j) {
            const int v = g.alpha[rec_digit(lo, hi, g.bits, g.L, j)];
            if (v < 0) *o++ = '-';
            o = gp::put_dec(o, (unsigned)(v < 0 ? -v : v));
            *o++ = ' ';
        }
        *o = '\n';
        start[i] = off[i];
        len[i] = (uint32_t)(o - o0);  // without the newline, as the text path's line lengths
    }
}

__global__ void gather_len_kernel(const uint32_t* len, const uint32_t* order, int64_t n, uint32_t* out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = len[order[i]] + 1;
}

// one warp per kept line: its bytes and newline at the line's output offset
template <class Off>
__global__ void gather_lines_kernel(const char* text, const Off* start, const uint32_t* len,
                                    const uint32_t* order, const uint32_t* out_off, int64_t n, char* out) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t k = w0; k < n; k += nw) {
        const uint32_t i = order[k];
        const char* src = text + start[i];
        char* dst = out + out_off[k];
        const uint32_t l = len[i] + 1;  // the newline follows the line in the formatted text
        for (uint32_t c = lane; c < l; c += 32) dst[c] = src[c];
    }
}

// n lines on the device (text, starts, lengths without the newline that
// follows each): sorted and de-duplicated by bytes, to a file.  codes: every
// character has a 4-bit code.
int sort_device_lines(gp_ctx* c, const char* d_text, const uint32_t* d_start, const uint32_t* d_len, int64_t n,
                      unsigned longest, bool codes, const char* out_path, cudaStream_t s) {
    const int per = codes ? 8 : 4;
    const int Wk = std::max(1, (int)((longest + per - 1) / per));
    DevBuf &dk = c->st[kTbKeys], &di = c->st[kTbIdx], &dtmp = c->st[kTbTmp], &dflag = c->st[kTbFlag],
           &dpos = c->st[kTbPos], &dord = c->st[kTbOrder], &dlen2 = c->st[kTbOutLen], &dooff = c->st[kTbOutOff],
           &dout = c->st[kTbOut], &dscan = c->st[kTbScan];
    if (!dk.ensure((size_t)n * Wk * 4) || !di.ensure(n * 4) || !dtmp.ensure(gp::radix_sort_tmp_bytes(n, Wk)) ||
        !dflag.ensure(n * 4) || !dpos.ensure(n * 4) || !dord.ensure(n * 4 + 4) || !dlen2.ensure(n * 4) ||
        !dooff.ensure(n * 4) || !dscan.ensure(gp::scan_tmp_bytes(n)))
        return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    build_keys_kernel<<<grid_for(n), 256, 0, s>>>(d_text, d_start, d_len, n, Wk, codes ? 1 : 0, dk.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    int bits = 8;
    int rc = sort_radix_bits(c, dk.as<uint32_t>(), Wk, n, di.as<uint32_t>(), dtmp.p, s, &bits);
    if (rc) return rc;
    GP_CUDA_TRY(c, gp::iota_u32(di.as<uint32_t>(), n, s));
    GP_CUDA_TRY(c, gp::radix_sort_keys(dk.as<uint32_t>(), Wk, Wk, di.as<uint32_t>(), n, dtmp.p, s, bits));
    GP_CUDA_TRY(c, gp::mark_unique(dk.as<uint32_t>(), Wk, di.as<uint32_t>(), n, Wk, dflag.as<uint32_t>(), s));
    uint32_t* d_cnt = dord.as<uint32_t>() + n;
    GP_CUDA_TRY(c, gp::compact_flags(dflag.as<uint32_t>(), di.as<uint32_t>(), dord.as<uint32_t>(), n,
                                     dpos.as<uint32_t>(), dscan.as<uint32_t>(), d_cnt, s));
    uint32_t nu = 0;
    GP_CUDA_TRY(c, cudaMemcpyAsync(&nu, d_cnt, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    gather_len_kernel<<<grid_for(nu), 256, 0, s>>>(d_len, dord.as<uint32_t>(), nu, dlen2.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, gp::exclusive_scan_u32(dlen2.as<uint32_t>(), dooff.as<uint32_t>(), nu, dscan.as<uint32_t>(), s));
    uint32_t o_last = 0, l_last = 0;
    GP_CUDA_TRY(c, cudaMemcpyAsync(&o_last, dooff.as<uint32_t>() + nu - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(&l_last, dlen2.as<uint32_t>() + nu - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    const uint64_t out_bytes = (uint64_t)o_last + l_last;
    if (!dout.ensure(out_bytes + 16)) return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    gather_lines_kernel<<<(unsigned)std::min<int64_t>((nu + 7) / 8, 65535 * 8), 256, 0, s>>>(
        d_text, d_start, d_len, dord.as<uint32_t>(), dooff.as<uint32_t>(), nu, dout.as<char>());
    GP_CUDA_TRY(c, cudaGetLastError());
    return write_text(c, dout.as<char>(), out_bytes, out_path, s);
}

// Sorted, de-duplicated lines of the records (all of one geometry), to a file.
// Returns GP_ERR_FORMAT on a malformed record.
int gp_sort_records(gp_ctx* c, const SurvGeom& g, const std::vector<uint8_t>& recs, int64_t n, const char* out_path) {
    cudaStream_t s = c->s_comp;
    if (n == 0) return write_text(c, nullptr, 0, out_path, s);
    DevBuf dr, dl, doff, dscan, dmisc, dt, ds;
    if (!dr.ensure(recs.size() + 16) || !dl.ensure(n * 4 + 4) || !doff.ensure(n * 4 + 4) ||
        !dscan.ensure(gp::scan_tmp_bytes(n)) || !dmisc.ensure(64) || !ds.ensure(n * 4))
        return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    GP_CUDA_TRY(c, cudaMemcpyAsync(dr.p, recs.data(), recs.size(), cudaMemcpyHostToDevice, s));
    GP_CUDA_TRY(c, cudaMemsetAsync(dmisc.p, 0, 64, s));
    unsigned* d_maxlen = dmisc.as<unsigned>();
    int* d_bad = dmisc.as<int>() + 1;
    surv_len_kernel<<<grid_for(n), 256, 0, s>>>(dr.as<uint8_t>(), n, g, dl.as<uint32_t>(), d_maxlen, d_bad);
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, gp::exclusive_scan_u32(dl.as<uint32_t>(), doff.as<uint32_t>(), n, dscan.as<uint32_t>(), s));
    uint32_t last_off = 0, last_len = 0;
    unsigned hm[2] = {0, 0};
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last_off, doff.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(&last_len, dl.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaMemcpyAsync(hm, dmisc.p, 8, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    if (hm[1]) return c->fail(GP_ERR_FORMAT, "sort: malformed survivor record");
    const uint64_t total = (uint64_t)last_off + last_len;
    if (total >= (uint64_t(1) << 32)) return c->fail(GP_ERR_UNSUPPORTED, "sort: %llu bytes of lines", (unsigned long long)total);
    if (!dt.ensure(total + 16)) return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    surv_format_kernel<<<grid_for(n), 256, 0, s>>>(dr.as<uint8_t>(), n, g, doff.as<uint32_t>(), dt.as<char>(),
                                                   ds.as<uint32_t>(), dl.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    return sort_device_lines(c, dt.as<char>(), ds.as<uint32_t>(), dl.as<uint32_t>(), n, hm[0], true, out_path, s);
}

extern "C" {

int gp_tuned_settings(const gp_ctx* c, char* buf, int cap) {
    if (!c) return GP_ERR_ARG;
    std::string t;
    for (const auto& kv : c->tuned) {
        t += kv.first;
        for (int64_t v : kv.second) t += " " + std::to_string(v);
        t += "\n";
    }
    if (buf && cap > 0) {
        const size_t k = std::min(t.size(), (size_t)cap - 1);
        std::memcpy(buf, t.data(), k);
        buf[k] = 0;
    }
    return (int)t.size() + 1;
}

// Text inputs of the sort, one after another on the device, each ended by a
// newline.
static int sort_files(gp_ctx* c, std::vector<FileText>& files, size_t bytes, const char* out_path) {
    cudaStream_t s = c->s_comp;
    DevBuf& dt = c->st[kTbText];
    if (!dt.ensure(bytes + kTextBlock)) return c->fail(GP_ERR_NOMEM, "sort: device allocation");
    size_t n = 0;
    for (FileText& f : files) {
        if (f.n == 0) continue;
        GP_CUDA_TRY(c, cudaMemcpyAsync(dt.as<char>() + n, f.p.get(), f.n, cudaMemcpyHostToDevice, s));
        n += f.n;
        if (f.p[f.n - 1] != '\n') GP_CUDA_TRY(c, cudaMemsetAsync(dt.as<char>() + n++, '\n', 1, s));
    }
    if (n == 0) return write_text(c, nullptr, 0, out_path, s);
    Lines ln;
    const int rc = find_lines(c, dt.as<char>(), n, c->st[kTbStart], c->st[kTbLen], ln, s);
    if (rc) return rc;
    for (FileText& f : files) f.p.reset();  // find_lines has waited for the copies
    return sort_device_lines(c, dt.as<char>(), c->st[kTbStart].as<uint32_t>(), c->st[kTbLen].as<uint32_t>(), ln.n,
                             ln.longest, !ln.other, out_path, s);
}

static int gp_sort_impl(gp_ctx* c, const char** in_paths, int n_in, const char* out_path) {
    StageRange nvtx_range("gp_sort");
    if (!c || (!in_paths && n_in > 0) || !out_path) return GP_ERR_ARG;
    cudaSetDevice(c->device);
    KeepSmall keep{c->st};
    // every input is read once
    std::vector<FileText> files(n_in);
    size_t bytes = 0;
    bool text_only = true;
    for (int i = 0; i < n_in; ++i) {
        if (!read_file(in_paths[i], files[i])) return c->fail(GP_ERR_IO, "sort: cannot read %s", in_paths[i]);
        bytes += files[i].n + 1;
        text_only = text_only && !(files[i].n >= 8 && std::memcmp(files[i].p.get(), gp::kSurvMagic, 8) == 0);
    }
    if (text_only && bytes < kMaxDeviceText) return sort_files(c, files, bytes, out_path);
    std::vector<std::string> texts(n_in);
    for (int i = 0; i < n_in; ++i) {
        texts[i].assign(files[i].p.get(), files[i].n);
        files[i].p.reset();
    }
    {
        // all inputs binary survivor files of one job: the records are
        // formatted and sorted on the device
        std::vector<uint8_t> recs;
        SurvGeom g{};
        int64_t n = 0;
        bool binary = n_in > 0;
        gp::SurvHeader h0{};
        for (int i = 0; i < n_in && binary; ++i) {
            gp::SurvHeader h;
            const uint8_t* body = nullptr;
            const int kind = gp::surv_parse(texts[i], h, &body);
            if (kind < 0) return c->fail(GP_ERR_FORMAT, "sort: malformed survivor file %s", in_paths[i]);
            if (kind == 0 || (i > 0 && (h.L != h0.L || h.bits != h0.bits || h.k != h0.k || h.sig_bytes != h0.sig_bytes ||
                                        std::memcmp(h.alpha, h0.alpha, 16) != 0))) {
                binary = false;
                break;
            }
            if (i == 0) h0 = h;
            recs.insert(recs.end(), body, body + h.count * gp::surv_record_bytes(h));
            n += (int64_t)h.count;
        }
        if (binary) {
            g.L = h0.L;
            g.bits = h0.bits;
            g.k = h0.k;
            g.sig_bytes = h0.sig_bytes;
            g.word_bytes = h0.word_bytes;
            g.rec_bytes = (int)gp::surv_record_bytes(h0);
            for (int a = 0; a < 16; ++a) g.alpha[a] = h0.alpha[a];
            return gp_sort_records(c, g, recs, n, out_path);
        }
    }
    std::string all;
    for (int i = 0; i < n_in; ++i) {
        std::string& one = texts[i];
        gp::SurvHeader h;
        const uint8_t* body = nullptr;
        const int kind = gp::surv_parse(one, h, &body);
        if (kind < 0 || (kind > 0 && !gp::surv_to_text(h, body, all)))
            return c->fail(GP_ERR_FORMAT, "sort: malformed survivor file %s", in_paths[i]);
        if (kind > 0) continue;
        if (all.empty())
            all.swap(one);  // the first text input: no copy
        else
            all += one;
        if (!all.empty() && all.back() != '\n') all.push_back('\n');
        std::string().swap(one);
    }
    std::string sorted;
    int rc = gp_sort_text(c, all, sorted);
    if (rc) return rc;
    return write_file(c, sorted.data(), sorted.size(), out_path);
}

// No C++ exception (an allocation failure on a huge input) crosses the C ABI.
int gp_sort(gp_ctx* c, const char** in_paths, int n_in, const char* out_path) {
    try {
        return gp_sort_impl(c, in_paths, n_in, out_path);
    } catch (const std::exception& e) {
        return c ? c->fail(GP_ERR_NOMEM, "sort: %s", e.what()) : GP_ERR_NOMEM;
    }
}

// The match on the device: sorted candidate files (every token no greater than
// the next line's), so the merge on the first token is an equality join: each
// a line with the b lines of its token, in file order.  *done = false where
// the host's parser or merge decides: other characters, lines of blanks or
// with too few integers, unsorted tokens, more text or pairs than 32 bits,
// sequences without entries (an order of 0).
static int match_files(gp_ctx* c, int L, int target, const FileText& fa, const FileText& fb, OutFile& f,
                       int64_t* n_pairs, bool* done) {
    *done = false;
    if (L < 1 || fa.n + 2 > kMaxDeviceText || fb.n + 2 > kMaxDeviceText) return GP_OK;
    cudaStream_t s = c->s_comp;
    const FileText* file[2] = {&fa, &fb};
    DevBuf* text[2] = {&c->st[kTbText], &c->st[kTbTextB]};
    DevBuf* start[2] = {&c->st[kTbStart], &c->st[kTbStartB]};
    DevBuf* len[2] = {&c->st[kTbLen], &c->st[kTbLenB]};
    DevBuf* tok[2] = {&c->st[kTbTokA], &c->st[kTbTokB]};
    DevBuf* tlen[2] = {&c->st[kTbTokLenA], &c->st[kTbTokLenB]};
    DevBuf* seqs[2] = {&c->st[kTbSeqA], &c->st[kTbSeqB]};
    DevBuf* paf[2] = {&c->st[kTbPafA], &c->st[kTbPafB]};
    DevBuf& misc = c->st[kTbMisc];
    const int H = L / 2;
    Lines ln[2];
    for (int k = 0; k < 2; ++k) {
        size_t n = file[k]->n;
        if (!text[k]->ensure(n + 1 + kTextBlock)) return c->fail(GP_ERR_NOMEM, "match: device allocation");
        GP_CUDA_TRY(c, cudaMemcpyAsync(text[k]->p, file[k]->p.get(), n, cudaMemcpyHostToDevice, s));
        if (file[k]->p[n - 1] != '\n') GP_CUDA_TRY(c, cudaMemsetAsync(text[k]->as<char>() + n++, '\n', 1, s));
        const int rc = find_lines(c, text[k]->as<char>(), n, *start[k], *len[k], ln[k], s);
        if (rc) return rc;
        if (ln[k].other) return GP_OK;
    }
    int* d_bad = misc.as<int>() + 2;
    unsigned long long* d_total = misc.as<unsigned long long>() + 2;
    GP_CUDA_TRY(c, cudaMemsetAsync(misc.p, 0, 64, s));
    for (int k = 0; k < 2; ++k) {
        const int64_t n = ln[k].n;
        if (!tok[k]->ensure(n * 4) || !tlen[k]->ensure(n * 4) || !seqs[k]->ensure((size_t)n * L + 16) ||
            !paf[k]->ensure((size_t)n * (H + 1) * 4))
            return c->fail(GP_ERR_NOMEM, "match: device allocation");
        parse_lines_kernel<<<grid_for(n), 256, 0, s>>>(text[k]->as<char>(), start[k]->as<uint32_t>(),
                                                       len[k]->as<uint32_t>(), n, L, tok[k]->as<uint32_t>(),
                                                       tlen[k]->as<uint32_t>(), seqs[k]->as<int8_t>(), d_bad);
        tokens_sorted_kernel<<<grid_for(n), 256, 0, s>>>(text[k]->as<char>(), tok[k]->as<uint32_t>(),
                                                         tlen[k]->as<uint32_t>(), n, d_bad);
        GP_CUDA_TRY(c, cudaGetLastError());
    }
    const int64_t na = ln[0].n;
    DevBuf &db0 = c->st[kTbOutLen], &dnb = c->st[kTbFlag], &dfirst = c->st[kTbOutOff], &dscan = c->st[kTbScan];
    if (!db0.ensure(na * 4) || !dnb.ensure(na * 4) || !dfirst.ensure(na * 4) || !dscan.ensure(gp::scan_tmp_bytes(na)))
        return c->fail(GP_ERR_NOMEM, "match: device allocation");
    token_ranges_kernel<<<grid_for(na), 256, 0, s>>>(text[0]->as<char>(), tok[0]->as<uint32_t>(), tlen[0]->as<uint32_t>(),
                                                     na, text[1]->as<char>(), tok[1]->as<uint32_t>(),
                                                     tlen[1]->as<uint32_t>(), ln[1].n, db0.as<uint32_t>(),
                                                     dnb.as<uint32_t>(), d_total);
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, gp::exclusive_scan_u32(dnb.as<uint32_t>(), dfirst.as<uint32_t>(), na, dscan.as<uint32_t>(), s));
    unsigned long long h[8];
    GP_CUDA_TRY(c, cudaMemcpyAsync(h, misc.p, 64, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    if ((int)(uint32_t)h[1] || h[2] >= (1ull << 31)) return GP_OK;
    *done = true;
    const int64_t total = (int64_t)h[2];
    if (n_pairs) *n_pairs = 0;
    if (total == 0) return GP_OK;
    DevBuf &df = c->st[kTbKeys], &dpos = c->st[kTbPos], &dkeep = c->st[kTbOrder], &dia = c->st[kTbIa],
           &dib = c->st[kTbIb];
    if (!df.ensure((size_t)total * 4) || !dpos.ensure((size_t)total * 4) || !dkeep.ensure((size_t)total * 4 + 4) ||
        !dia.ensure((size_t)total * 4) || !dib.ensure((size_t)total * 4) || !dscan.ensure(gp::scan_tmp_bytes(total)))
        return c->fail(GP_ERR_NOMEM, "match: device allocation");
    if (H > 0)
        for (int k = 0; k < 2; ++k)
            paf_kernel<<<grid_for(ln[k].n), 256, 0, s>>>(seqs[k]->as<int8_t>(), ln[k].n, L, H, paf[k]->as<int>());
    range_check_kernel<<<grid_for(total), 256, 0, s>>>(dfirst.as<uint32_t>(), db0.as<uint32_t>(), na, (uint32_t)total,
                                                       paf[0]->as<int>(), paf[1]->as<int>(), H, target,
                                                       df.as<uint32_t>(), dia.as<uint32_t>(), dib.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    uint32_t* d_cnt = dkeep.as<uint32_t>() + total;
    GP_CUDA_TRY(c, gp::compact_flags(df.as<uint32_t>(), nullptr, dkeep.as<uint32_t>(), total, dpos.as<uint32_t>(),
                                     dscan.as<uint32_t>(), d_cnt, s));
    uint32_t nk = 0;
    GP_CUDA_TRY(c, cudaMemcpyAsync(&nk, d_cnt, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    // the kept pairs' lines, blocks of them below 2^31 bytes (five a value at most)
    DevBuf &dbytes = c->st[kTbFlag], &dat = c->st[kTbPos], &dout = c->st[kTbOut];
    const int64_t step = std::min<int64_t>(nk, (int64_t(1) << 31) / (10 * L + 2));
    if (nk && (!dbytes.ensure((size_t)step * 4) || !dat.ensure((size_t)step * 4)))
        return c->fail(GP_ERR_NOMEM, "match: device allocation");
    for (int64_t k0 = 0; k0 < nk; k0 += step) {
        const int64_t n = std::min<int64_t>(step, nk - k0);
        const uint32_t* keep = dkeep.as<uint32_t>() + k0;
        match_line_bytes_kernel<<<grid_for(n), 256, 0, s>>>(seqs[0]->as<int8_t>(), seqs[1]->as<int8_t>(),
                                                            dia.as<uint32_t>(), dib.as<uint32_t>(), keep, n, L,
                                                            dbytes.as<uint32_t>());
        GP_CUDA_TRY(c, cudaGetLastError());
        GP_CUDA_TRY(c, gp::exclusive_scan_u32(dbytes.as<uint32_t>(), dat.as<uint32_t>(), n, dscan.as<uint32_t>(), s));
        uint32_t last[2] = {0, 0};
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[0], dat.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[1], dbytes.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        const size_t bytes = (size_t)last[0] + last[1];
        if (!dout.ensure(bytes + 1)) return c->fail(GP_ERR_NOMEM, "match: device allocation");
        match_lines_kernel<<<(unsigned)std::min<int64_t>((n + 7) / 8, 65535 * 8), 256, 0, s>>>(
            seqs[0]->as<int8_t>(), seqs[1]->as<int8_t>(), dia.as<uint32_t>(), dib.as<uint32_t>(), keep, n, L,
            dat.as<uint32_t>(), dout.as<char>());
        GP_CUDA_TRY(c, cudaGetLastError());
        std::unique_ptr<char[]> out(new char[bytes + 1]);
        GP_CUDA_TRY(c, cudaMemcpyAsync(out.get(), dout.p, bytes, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        f.put(out.get(), bytes);
    }
    if (n_pairs) *n_pairs = nk;
    return GP_OK;
}

static int gp_match_impl(gp_ctx* c, int order, int compress, int paf, const char* path_a, const char* path_b, const char* out_path,
             int append, int64_t* n_pairs) {
    StageRange nvtx_range("gp_match");
    if (!c || !path_a || !path_b || !out_path) return GP_ERR_ARG;
    if (compress < 1 || order % compress) return c->fail(GP_ERR_ARG, "order %d not divisible by %d", order, compress);
    cudaSetDevice(c->device);
    // the reference opens the pair writer (truncating unless appending)
    // before looking at the inputs (src/main.cpp:97-101)
    OutFile f(out_path, append ? "a" : "w");
    if (!f.f) return c->fail(GP_ERR_IO, "match: cannot open %s", out_path);
    KeepSmall keep{c->st};
    FileText fa, fb;
    const bool okA = read_file(path_a, fa), okB = read_file(path_b, fb);
    if (n_pairs) *n_pairs = 0;
    if (!okA || !okB || fa.n == 0 || fb.n == 0) return GP_EMPTY_INPUT;
    bool done = false;
    int rc = match_files(c, order / compress, paf * compress, fa, fb, f, n_pairs, &done);
    if (rc) return rc;
    if (!done) {
        std::string ta(fa.p.get(), fa.n), tb(fb.p.get(), fb.n), out;
        fa.p.reset();
        fb.p.reset();
        rc = gp_match_texts(c, order / compress, compress, paf, ta, tb, out, n_pairs);
        if (rc) return rc;
        f.put(out.data(), out.size());
    }
    return f.close() ? GP_OK : c->fail(GP_ERR_IO, "match: write failed: %s", out_path);
}

// No C++ exception (an allocation failure on a huge input) crosses the C ABI.
int gp_match(gp_ctx* c, int order, int compress, int paf, const char* path_a, const char* path_b, const char* out_path,
             int append, int64_t* n_pairs) {
    try {
        return gp_match_impl(c, order, compress, paf, path_a, path_b, out_path, append, n_pairs);
    } catch (const std::exception& e) {
        return c ? c->fail(GP_ERR_NOMEM, "match: %s", e.what()) : GP_ERR_NOMEM;
    }
}

}  // extern "C"
