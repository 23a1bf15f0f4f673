// capi_equiv.cu -- equivalence filter (kernel (d), second half).
//
// Replaces cache_filter (src/core/filter/filter.cpp:18-163).  The generator
// set is the closure of the index pair ({1..L}, {L+1..2L}) under the
// reference's pair operations (src/utils/equivalence.cpp:46-95,146-277):
// rotate b by 1..L-1, swap a and b, reverse b, decimate both by every unit,
// and (compression 1, even L only) negate the odd positions of both.  It is
// built on the host, as the reference builds it once per run.
//
// Per pair the filter needs its class size and the input pairs in its
// class.  For L >= 3, canon_kernel finds both from canonical forms: every
// group element is an affine map per half (the description below, checked
// against the closure by gp_debug_pair_group_check), so a pair's least image
// over the group takes O(4 phi(L) L^2) work; pairs with equal least images
// are in one class, and the class size is the group order over the number
// of elements that fix the pair (orbit-stabiliser).  For L < 3 class_kernel
// applies every element of the closure with the reference's application
// rule (equivalence.cpp:97-144), hashing the images of several pairs per
// pass over the transposed table and looking them up in a hash set of the
// input pairs.  Text past kHostText is read and written, and its pairs and least
// images sorted, on the device too.  Either way the host then replays the
// reference's in-order erase loop (filter.cpp:117-144) on those class sizes and
// member lists.
#include <algorithm>
#include <chrono>
#include <stdexcept>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "ctx.h"
#include "host_par.h"
#include "pair_text.cuh"
#include "prims.h"

namespace {

constexpr int kMaxW = 256;  // 2L entries per pair

// Entry o of the image of the pair under generator g: the generator table
// is stored transposed (srcT[o * ng + g], signed 1-based source position),
// so that a warp's consecutive generators read consecutive entries.
__device__ __forceinline__ int image_at(const int16_t* srcT, int64_t ng, int64_t g, const int8_t* sx, int o) {
    const int s = srcT[(int64_t)o * ng + g];
    const int v = sx[(s < 0 ? -s : s) - 1];
    return s < 0 ? -v : v;
}

constexpr int kPairsPerCta = 8;  // pairs whose images one pass over the generator table hashes

// FNV-1a over the entries as bytes (value mod 256), folded; the host hashes
// the input pairs with the same steps
__host__ __device__ __forceinline__ uint32_t fnv_step(uint32_t h, int v) { return (h ^ (uint8_t)v) * 16777619u; }
__host__ __device__ __forceinline__ uint32_t fnv_fold(uint32_t h) { return h ^ (h >> 15); }
constexpr uint32_t kFnvBasis = 2166136261u;

// the image of the pair sx under generator g equals target (W entries)
__device__ __forceinline__ bool image_equals(const int16_t* srcT, int64_t ng, int64_t g, const int8_t* sx,
                                             const int8_t* target, int W) {
    for (int o = 0; o < W; ++o)
        if (image_at(srcT, ng, g, sx, o) != target[o]) return false;
    return true;
}

struct ClassArgs {
    const int16_t* srcT;      // generator table, transposed: srcT[o * ng + g]
    int64_t ng;
    int64_t group0;           // first pair group of the launch
    const int8_t* pairs;      // np x W, sorted (the reference's set order)
    int64_t np;
    int W;
    const uint32_t* set_h;    // hash set of the pairs: folded hash, pair index (EMPTY: 0xFFFFFFFF)
    const uint32_t* set_i;
    uint32_t set_mask;
    uint32_t* stab;           // per pair: generators that fix it
    uint32_t* members;        // (pair, member) index pairs
    unsigned long long* nmembers;
    int64_t mcap;
    int* status;
};

// CTA b: pairs of group b / splits (kPairsPerCta consecutive pairs) and the
// generators of share b % splits.
__global__ void __launch_bounds__(256) class_kernel(ClassArgs a, int splits) {
    constexpr int PG = kPairsPerCta;
    __shared__ int8_t sx[PG][kMaxW];
    __shared__ uint32_t self_h[PG];
    const int64_t group = a.group0 + blockIdx.x / splits;
    const int part = blockIdx.x % splits;
    const int64_t x0 = group * PG;
    const int npg = (int)min((int64_t)PG, a.np - x0);
    const int W = a.W;
    for (int k = threadIdx.x; k < PG * W; k += blockDim.x) {
        const int p = k / W, o = k - p * W;
        sx[p][o] = p < npg ? a.pairs[(x0 + p) * W + o] : 0;
    }
    __syncthreads();
    if (threadIdx.x < PG) {
        uint32_t h = kFnvBasis;
        for (int o = 0; o < W; ++o) h = fnv_step(h, sx[threadIdx.x][o]);
        self_h[threadIdx.x] = fnv_fold(h);
    }
    __syncthreads();
    uint32_t stab[PG];
#pragma unroll
    for (int p = 0; p < PG; ++p) stab[p] = 0;
    const int64_t step = (int64_t)splits * blockDim.x;
    for (int64_t g = (int64_t)part * blockDim.x + threadIdx.x; g < a.ng; g += step) {
        uint32_t h[PG];
#pragma unroll
        for (int p = 0; p < PG; ++p) h[p] = kFnvBasis;
        for (int o = 0; o < W; ++o) {  // one read of the generator's entry serves every pair of the group
            const int sgn = a.srcT[(int64_t)o * a.ng + g];
            const int idx = (sgn < 0 ? -sgn : sgn) - 1;
#pragma unroll
            for (int p = 0; p < PG; ++p) {
                const int v = sx[p][idx];
                h[p] = fnv_step(h[p], sgn < 0 ? -v : v);
            }
        }
#pragma unroll
        for (int p = 0; p < PG; ++p) {
            if (p >= npg) continue;
            const uint32_t hp = fnv_fold(h[p]);
            if (hp == self_h[p] && image_equals(a.srcT, a.ng, g, sx[p], sx[p], W)) ++stab[p];
            for (uint32_t slot = hp & a.set_mask;; slot = (slot + 1) & a.set_mask) {
                const uint32_t m = a.set_i[slot];
                if (m == 0xFFFFFFFFu) break;
                if (a.set_h[slot] != hp || !image_equals(a.srcT, a.ng, g, sx[p], a.pairs + (int64_t)m * W, W))
                    continue;
                const unsigned long long pos = atomicAdd(a.nmembers, 1ull);
                if ((int64_t)pos < a.mcap) {
                    a.members[2 * pos] = (uint32_t)(x0 + p);
                    a.members[2 * pos + 1] = m;
                } else {
                    atomicCAS(a.status, 0, GP_KSTATUS_OVERFLOW);
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < PG; ++p) {
        const uint32_t t = __reduce_add_sync(0xFFFFFFFFu, stab[p]);
        if ((threadIdx.x & 31) == 0 && t && p < npg) atomicAdd(&a.stab[x0 + p], t);
    }
}

// ------------------------------------------------------------ canonical forms
// For L >= 3 every element of the pair group is, on each half of the
// result, an affine map of one source half: optionally swap the halves,
// then
//     a'[i] = (-1)^(alpha i + beta_a) * src_a[(u i + s_a) mod L]
//     b'[i] = (-1)^(alpha i + beta_b) * src_b[(e u i + s_b) mod L]
// with u a unit mod L, e = +-1, s_a, s_b any shifts, and the signs only
// where the alternating negation is a generator (alpha, beta_a, beta_b:
// 8 patterns).  These 2 * 2 * phi(L) * L^2 (* 8) maps are all in the group
// (decimation by u, reversal of b, shifts of b and their conjugates by the
// swap, and the negation of one half, which the alternating negation and an
// odd shift give) and as many as its order, so they are the group;
// gp_debug_pair_group_check compares them with the closure.  Two pairs are
// in one class iff they have the same least image (lexicographic, entries as
// signed integers), and the class size is the group order over the number of
// elements that fix the pair.  Per (swap, e, signs, u) the least image takes
// the least shift of each half separately, so a pair costs
// O(4 phi(L) (8) L^2) instead of O(|G| L).
struct CanonArgs {
    const int8_t* pairs;   // np x W
    int64_t np;
    int L;
    const int16_t* units;  // every unit mod L
    int nu;
    int alt;               // 1: the 8 sign patterns
    int8_t* canon;         // np x W: least image
    uint32_t* fixers;      // elements fixing the pair
};

// (-1)^(alpha i + beta) for pattern pat
__device__ __forceinline__ int sign_of(int pat, int i) { return (((pat & 1) & i) ^ (pat >> 1)) ? -1 : 1; }

// One half of an image: H(s)[i] = sign(i) x[h + (m i + s) mod L] for shift s.
struct Half {
    const int8_t* x;
    int L, h, m, pat;
};

// The least shift of a half, and how many shifts give exactly the pair's a
// (fix_a) and b (fix_b).
__device__ __forceinline__ void least_shift(const Half& H, int& s_best, int& fix_a, int& fix_b) {
    const int8_t* x = H.x;
    const int8_t* src = x + H.h;
    const int L = H.L;
    s_best = 0;
    fix_a = fix_b = 0;
    for (int s = 0; s < L; ++s) {
        int cmp = 0;  // sign of H(s) - H(s_best) at the first difference
        bool eqa = true, eqb = true;
        int i1 = s, i2 = s_best;
        for (int i = 0; i < L; ++i) {
            const int sg = sign_of(H.pat, i);
            const int v = sg * src[i1];
            if (cmp == 0) {
                const int w = sg * src[i2];
                if (v != w) cmp = v < w ? -1 : 1;
            }
            eqa = eqa && v == x[i];
            eqb = eqb && v == x[L + i];
            if (!eqa && !eqb && (cmp != 0 || s == s_best)) break;
            i1 += H.m;
            i1 -= i1 >= L ? L : 0;
            i2 += H.m;
            i2 -= i2 >= L ? L : 0;
        }
        if (cmp < 0) s_best = s;
        fix_a += eqa ? 1 : 0;
        fix_b += eqb ? 1 : 0;
    }
}

// -1, 0, 1: half H1 at shift s1 against half H2 at shift s2
__device__ __forceinline__ int compare_halves(const Half& H1, int s1, const Half& H2, int s2) {
    for (int i = 0; i < H1.L; ++i) {
        const int v = sign_of(H1.pat, i) * H1.x[H1.h + s1], w = sign_of(H2.pat, i) * H2.x[H2.h + s2];
        if (v != w) return v < w ? -1 : 1;
        s1 += H1.m;
        s1 -= s1 >= H1.L ? H1.L : 0;
        s2 += H2.m;
        s2 -= s2 >= H2.L ? H2.L : 0;
    }
    return 0;
}

// A pair's least image: a warp per pair.  An image's halves are each one of
// 2 phi(L) (source half, multiplier) maps (x 4 sign patterns with the
// alternating negation), so the lanes first find every such half's least
// shift, and the shifts that fix a and b, and then compare the 4 phi(L) (x 8)
// combinations of two halves.  (Every combination on its own takes each
// half's shifts four times; a CTA of 128 threads per pair left most of them
// idle in its second round at length 57: 7.50 ms for 30,000 pairs, 1.88 by
// halves.)
// Entries +-1 of up to 64 per half are words of one bit each, first entry
// highest: x[m i + s] over all s are the rotations of the decimated word, a
// sign pattern flips fixed bits, and the order of images is the order of the
// numbers (the call goes from 4.24 to 2.72 ms).
constexpr int kCanonWarps = 4;
struct HalfShift {
    uint8_t s, fix_a, fix_b;
};

// A warp's shared memory: the pair, its halves' least words (lengths up to 64),
// their least shifts.
struct CanonLayout {
    size_t words, tab, per_warp;
};
__host__ __device__ __forceinline__ CanonLayout canon_layout(int L, int nhalf) {
    CanonLayout s;
    s.words = (2 * (size_t)L + 7) & ~size_t(7);
    s.tab = s.words + (L <= 64 ? sizeof(uint64_t) * nhalf : 0);
    s.per_warp = (s.tab + sizeof(HalfShift) * nhalf + 7) & ~size_t(7);
    return s;
}

// The least rotation of the word of x's decimation by m, bits flipped by sign,
// and how many rotations equal wa and wb.
__device__ __forceinline__ uint64_t least_rotation(uint64_t x, int L, int m, uint64_t sign, uint64_t wa, uint64_t wb,
                                                   int& fix_a, int& fix_b) {
    uint64_t y = 0;
    for (int i = 0, j = 0; i < L; ++i) {
        y = (y << 1) | ((x >> (L - 1 - j)) & 1ull);
        j += m;
        j -= j >= L ? L : 0;
    }
    const uint64_t all = ~0ull >> (64 - L);
    uint64_t best = ~0ull;
    fix_a = fix_b = 0;
    for (int t = 0; t < L; ++t) {
        const uint64_t v = y ^ sign;
        best = v < best ? v : best;
        fix_a += v == wa;
        fix_b += v == wb;
        y = ((y << 1) & all) | (y >> (L - 1));
    }
    return best;
}

__global__ void __launch_bounds__(32 * kCanonWarps) canon_kernel(CanonArgs a) {
    extern __shared__ __align__(8) uint8_t sh[];
    const int L = a.L, W = 2 * L, npat = a.alt ? 4 : 1, nhalf = 2 * npat * a.nu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // per warp: the pair, then the halves' least shifts
    const CanonLayout lay = canon_layout(L, nhalf);
    uint8_t* mine = sh + (size_t)warp * lay.per_warp;
    int8_t* x = reinterpret_cast<int8_t*>(mine);
    uint64_t* least = reinterpret_cast<uint64_t*>(mine + lay.words);
    HalfShift* tab = reinterpret_cast<HalfShift*>(mine + lay.tab);
    const int ncombo = 4 * a.nu * (a.alt ? 8 : 1);
    // half t: source half t & 1, sign pattern, unit index
    auto half_of = [&](int src, int pat, int ui) { return (ui * npat + pat) * 2 + src; };
    auto half = [&](int t) { return Half{x, L, (t & 1) * L, a.units[(t >> 1) / npat], (t >> 1) % npat}; };
    // combination c: the halves that make a' and b' (u and, reversed, L - u:
    // the units in ascending order mirror each other)
    auto halves = [&](int c, int& ta, int& tb) {
        const int swap = c & 1, e = (c >> 1) & 1;
        c >>= 2;
        int pa = 0, pb = 0;
        if (a.alt) {
            pa = (c & 1) | (c & 2);
            pb = (c & 1) | ((c >> 1) & 2);
            c >>= 3;
        }
        ta = half_of(swap, pa, c);
        tb = half_of(1 - swap, pb, e ? a.nu - 1 - c : c);
    };
    const int64_t warps = (int64_t)gridDim.x * kCanonWarps;
    for (int64_t pr = (int64_t)blockIdx.x * kCanonWarps + warp; pr < a.np; pr += warps) {
        __syncwarp();
        for (int o = lane; o < W; o += 32) x[o] = a.pairs[pr * W + o];
        __syncwarp();
        bool bits = L <= 64;  // the pair's entries are +-1
        uint64_t word[2] = {0, 0};
        if (bits) {
            bool unit = true;
            for (int h = 0; h < 2; ++h) {
                const int v0 = lane < L ? x[h * L + lane] : 1, v1 = lane + 32 < L ? x[h * L + lane + 32] : 1;
                unit = unit && (v0 == 1 || v0 == -1) && (v1 == 1 || v1 == -1);
                const uint64_t w = __ballot_sync(0xFFFFFFFFu, v0 > 0) |
                                   (uint64_t)__ballot_sync(0xFFFFFFFFu, v1 > 0) << 32;
                word[h] = __brevll(w) >> (64 - L);
            }
            bits = __all_sync(0xFFFFFFFFu, unit);
        }
        for (int t = lane; t < nhalf; t += 32) {
            int s = 0, fa, fb;
            if (bits) {
                const int pat = (t >> 1) % npat;
                // negated entries: the odd ones (pattern bit 0), all the others (bit 1)
                uint64_t sign = 0;
                if (pat & 1) sign = (0x5555555555555555ull << (L & 1)) & (~0ull >> (64 - L));
                if (pat & 2) sign ^= ~0ull >> (64 - L);
                least[t] = least_rotation(word[t & 1], L, a.units[(t >> 1) / npat], sign, word[0], word[1], fa, fb);
            } else {
                least_shift(half(t), s, fa, fb);
            }
            tab[t] = HalfShift{(uint8_t)s, (uint8_t)fa, (uint8_t)fb};
        }
        __syncwarp();
        auto compare = [&](int c1, int c2) {  // images of combinations at their least shifts
            int a1, b1, a2, b2;
            halves(c1, a1, b1);
            halves(c2, a2, b2);
            if (bits) {
                if (least[a1] != least[a2]) return least[a1] < least[a2] ? -1 : 1;
                return least[b1] == least[b2] ? 0 : least[b1] < least[b2] ? -1 : 1;
            }
            const int d = a1 == a2 ? 0 : compare_halves(half(a1), tab[a1].s, half(a2), tab[a2].s);
            return d || b1 == b2 ? d : compare_halves(half(b1), tab[b1].s, half(b2), tab[b2].s);
        };
        int best = -1;
        unsigned fix = 0;
        for (int c = lane; c < ncombo; c += 32) {
            int ta, tb;
            halves(c, ta, tb);
            fix += (unsigned)tab[ta].fix_a * tab[tb].fix_b;
            if (best < 0 || compare(c, best) < 0) best = c;
        }
        fix = __reduce_add_sync(0xFFFFFFFFu, fix);
        for (int o = 16; o; o >>= 1) {
            const int other = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            if (other >= 0 && (best < 0 || compare(other, best) < 0)) best = other;
        }
        best = __shfl_sync(0xFFFFFFFFu, best, 0);  // equal images may have left different combinations
        int ta, tb;
        halves(best, ta, tb);
        const Half A = half(ta), B = half(tb);
        for (int o = lane; o < W; o += 32) {
            const Half& H = o < L ? A : B;
            const int i = o < L ? o : o - L;
            if (bits)
                a.canon[pr * W + o] = (least[o < L ? ta : tb] >> (L - 1 - i)) & 1ull ? 1 : -1;
            else
                a.canon[pr * W + o] = (int8_t)(sign_of(H.pat, i) * x[H.h + (H.m * i + tab[o < L ? ta : tb].s) % L]);
        }
        if (lane == 0) a.fixers[pr] = fix;
    }
}

// ------------------------------------------------------------ pair text
// A pair file past kHostText is parsed, its pairs sorted and the kept ones written
// as text on the device: on the host that took 57 of the 73 ms of 30,000 order-57
// pairs (strtol, a vector per pair, std::sort, one digit at a time), here
// about 1 ms beside the file itself.

// What the text holds beside its values.
struct TextInfo {
    uint32_t bad;         // something strtol would read differently: the host parses
    uint32_t present[8];  // bit v + 128: value v occurs
};

constexpr int kParseThreads = 256;
constexpr int kParseEach = 16;                              // bytes per thread
constexpr int kParseBlock = kParseThreads * kParseEach;     // the text is padded with blanks to a multiple

__device__ __forceinline__ bool is_blank(int c) { return c == ' ' || (c >= '\t' && c <= '\r'); }
__device__ __forceinline__ bool is_digit(int c) { return c >= '0' && c <= '9'; }

// Values are runs of an optional '-' and one to three digits, at most 127,
// between blanks.  WRITE = false counts a block's values, true stores them
// from the block's offset.
template <bool WRITE>
__global__ void __launch_bounds__(kParseThreads) pair_values_kernel(const char* text, uint32_t* counts,
                                                                    const uint32_t* offs, int8_t* vals,
                                                                    TextInfo* info) {
    __shared__ uint32_t s_warp[kParseThreads / 32];
    __shared__ uint32_t s_present[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (WRITE && threadIdx.x < 8) s_present[threadIdx.x] = 0;
    const int64_t p0 = (int64_t)blockIdx.x * kParseBlock + threadIdx.x * kParseEach;
    const uint4 w = *reinterpret_cast<const uint4*>(text + p0);
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    int prev = p0 ? text[p0 - 1] : ' ';
    const int after = text[p0 + kParseEach];  // the buffer has a block of blanks past the text
    uint32_t starts = 0;
    bool bad = false;
#pragma unroll
    for (int k = 0; k < kParseEach; ++k) {
        const int c = (ww[k >> 2] >> (8 * (k & 3))) & 0xFF;
        const int next = k + 1 < kParseEach ? (ww[(k + 1) >> 2] >> (8 * ((k + 1) & 3))) & 0xFF : after;
        const bool minus = c == '-';
        if ((is_digit(c) || minus) && is_blank(prev)) starts |= 1u << k;
        if (!is_digit(c) && !minus && !is_blank(c)) bad = true;
        if (minus && (!is_blank(prev) || !is_digit(next))) bad = true;
        prev = c;
    }
    const uint32_t mine = (uint32_t)__popc(starts);
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int q = 0; q < kParseThreads / 32; ++q) {
        if (q < warp) before += s_warp[q];
        total += s_warp[q];
    }
    if constexpr (!WRITE) {
        if (threadIdx.x == 0) counts[blockIdx.x] = total;
        if (bad) info->bad = 1;
    } else {
        int8_t* out = vals + offs[blockIdx.x] + before + incl - mine;
        for (uint32_t m = starts; m; m &= m - 1u) {
            const char* q = text + p0 + __ffs((int)m) - 1;
            const bool neg = *q == '-';
            q += neg ? 1 : 0;
            int v = 0, n = 0;
            for (; is_digit(*q) && n < 4; ++q, ++n) v = v * 10 + (*q - '0');
            if (n > 3 || v > 127) info->bad = 1;
            v = neg ? -v : v;
            *out++ = (int8_t)v;
            atomicOr(&s_present[((v + 128) & 255) >> 5], 1u << (v & 31));
        }
        __syncthreads();
        if (threadIdx.x < 8 && s_present[threadIdx.x]) atomicOr(&info->present[threadIdx.x], s_present[threadIdx.x]);
    }
}

// Sort keys of rows of W values: the values' ranks (code[(uint8_t)v], in the
// order of the values) in b bits each, 32 / b to a word, first value highest.
__global__ void pair_keys_kernel(const int8_t* rows, int64_t n, int W, const uint8_t* code, int b, int Wk,
                                 uint32_t* keys) {
    const int per = 32 / b;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * Wk; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / Wk;
        const int o0 = (int)(e - i * Wk) * per;
        uint32_t k = 0;
        for (int q = 0; q < per; ++q) {
            const int o = o0 + q;
            k = (k << b) | (o < W ? (uint32_t)code[(uint8_t)rows[i * W + o]] : 0u);
        }
        keys[e] = k;
    }
}

__global__ void gather_rows_kernel(const int8_t* rows, const uint32_t* idx, int64_t n, int W, int8_t* out) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * W; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / W;
        out[e] = rows[(int64_t)idx[i] * W + (e - i * W)];
    }
}

// Bytes of each kept pair's line (0: left out).
__global__ void pair_line_bytes_kernel(const int8_t* rows, const uint8_t* alive, int64_t n, int W, uint32_t* bytes) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        bytes[i] = alive[i] ? (uint32_t)gp::pair_line_bytes(rows + i * W, rows + i * W + W / 2, W / 2) : 0u;
}

// The lines, a warp per pair.
__global__ void __launch_bounds__(256) pair_lines_kernel(const int8_t* rows, const uint8_t* alive, int64_t n, int W,
                                                         const uint32_t* at, char* text) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps)
        if (alive[i]) gp::put_pair_line(rows + i * W, rows + i * W + W / 2, W / 2, text + at[i]);
}

// Every unit mod L, ascending.
std::vector<int16_t> all_units(int L) {
    std::vector<int16_t> u;
    for (int v = 1; v < L; ++v)
        if (std::gcd(v, L) == 1) u.push_back((int16_t)v);
    return u;
}

// Units that generate the group of units mod L (greedy: each one added is
// not yet in the subgroup generated by the ones before).
std::vector<int> unit_generators(int L) {
    std::vector<char> in(L, 0);
    std::vector<int> sub = {1 % L}, gens;
    if (L > 1) in[1] = 1;
    for (int u = 2; u < L; ++u) {
        if (std::gcd(u, L) != 1 || in[u]) continue;
        gens.push_back(u);
        for (size_t at = 0; at < sub.size(); ++at)  // closure of sub under multiplication by the generators
            for (int g : gens) {
                const int v = (int)((long long)sub[at] * g % L);
                if (!in[v]) {
                    in[v] = 1;
                    sub.push_back(v);
                }
            }
    }
    return gens;
}

// Closure of the identity pair under the reference's pair operations
// (filter.cpp:70-87: every shift of b, swap, reverse b, every decimation,
// and the alternating negation).  The closure is the group those operations
// generate, so it is built from a generating subset: shift by 1, swap,
// reverse, decimation by generators of the unit group, alternating
// negation.  Same set, about 15x less work at length 57.
// Returns the items flat: count x W entries.
//
// Every generator maps each half affinely (position i takes +-entry
// u*i + s of one half, one u for both halves up to sign, the sign set by the
// parity of i), and so does every product of them.  An element is therefore
// fixed by the entries at positions 0, 1, L and L+1: with by_key the closure
// compares those 64 bits instead of all 2L entries.  The items are built by
// applying generators, never inferred, so when that closure reaches the
// group's known size it is the group; pair_generators checks exactly that
// and otherwise redoes the closure comparing whole items.
uint64_t pair_group_size(int L, int compress);
extern const uint64_t kMaxGroupBytes;

std::vector<int16_t> pair_closure(int L, int compress, bool by_key) {
    const int W = 2 * L;
    const bool use_alt = !(compress > 1 || L % 2 == 1);  // filter.cpp:83-87
    const std::vector<int> units = unit_generators(L);
    std::vector<int16_t> out;            // items, W entries each
    std::vector<uint32_t> slot(1u << 10, UINT32_MAX);  // open addressing: item index per slot
    std::vector<uint64_t> keys;  // by_key: every item's key
    size_t count = 0;
    auto key_of = [&](const int16_t* v) {
        return (uint64_t)(uint16_t)v[0] | (uint64_t)(uint16_t)v[1] << 16 | (uint64_t)(uint16_t)v[L] << 32 |
               (uint64_t)(uint16_t)v[L + 1] << 48;
    };
    auto mix = [](uint64_t h) {  // MurmurHash3's 64-bit finaliser
        h ^= h >> 33;
        h *= 0xff51afd7ed558ccdULL;
        h ^= h >> 33;
        h *= 0xc4ceb9fe1a85ec53ULL;
        return h ^ (h >> 33);
    };
    auto hash = [&](const int16_t* v) {
        uint64_t h = 1469598103934665603ULL;  // FNV-1a over the whole item
        for (int i = 0; i < W; ++i) {
            h ^= (uint16_t)v[i];
            h *= 1099511628211ULL;
        }
        return h ^ (h >> 29);
    };
    auto grow = [&]() {
        std::vector<uint32_t> ns(slot.size() * 2, UINT32_MAX);
        const size_t mask = ns.size() - 1;
        for (size_t i = 0; i < count; ++i) {
            size_t h = (by_key ? mix(keys[i]) : hash(out.data() + i * W)) & mask;
            while (ns[h] != UINT32_MAX) h = (h + 1) & mask;
            ns[h] = (uint32_t)i;
        }
        slot.swap(ns);
    };
    auto add = [&](const int16_t* v) {
        if (2 * (count + 1) > slot.size()) grow();
        const size_t mask = slot.size() - 1;
        const uint64_t k = by_key ? key_of(v) : 0;
        size_t h = (by_key ? mix(k) : hash(v)) & mask;
        while (slot[h] != UINT32_MAX) {
            if (by_key ? keys[slot[h]] == k : std::memcmp(out.data() + (size_t)slot[h] * W, v, (size_t)W * 2) == 0)
                return;
            h = (h + 1) & mask;
        }
        slot[h] = (uint32_t)count++;
        out.insert(out.end(), v, v + W);
        if (by_key) keys.push_back(k);
    };
    auto find_key = [&](uint64_t k) {
        const size_t mask = slot.size() - 1;
        for (size_t h = mix(k) & mask; slot[h] != UINT32_MAX; h = (h + 1) & mask)
            if (keys[slot[h]] == k) return true;
        return false;
    };
    // the generators as maps: output position j takes (neg[j] ? -1 : 1) * input[src[j]]
    struct Gen {
        std::vector<int> src;
        std::vector<char> neg;
    };
    std::vector<Gen> gens;
    auto identity = [&]() {
        Gen g{std::vector<int>(W), std::vector<char>(W, 0)};
        for (int j = 0; j < W; ++j) g.src[j] = j;
        return g;
    };
    if (L > 1) {  // shift_pair by 1: rotate b left by 1
        Gen g = identity();
        for (int i = 0; i < L; ++i) g.src[L + i] = L + (i + 1) % L;
        gens.push_back(g);
    }
    {  // swap_pair
        Gen g = identity();
        for (int i = 0; i < L; ++i) {
            g.src[i] = L + i;
            g.src[L + i] = i;
        }
        gens.push_back(g);
    }
    {  // reverse_pair: reverse b
        Gen g = identity();
        for (int i = 0; i < L; ++i) g.src[L + i] = L + L - 1 - i;
        gens.push_back(g);
    }
    for (int u : units) {  // decimate_pair: both parts, new[i] = old[i*u mod L]
        Gen g = identity();
        for (int i = 0; i < L; ++i) {
            g.src[i] = (int)(((long long)i * u) % L);
            g.src[L + i] = L + g.src[i];
        }
        gens.push_back(g);
    }
    if (use_alt) {  // altnegative_pair: negate odd positions of both
        Gen g = identity();
        for (int i = 1; i < L; i += 2) g.neg[i] = g.neg[L + i] = 1;
        gens.push_back(g);
    }
    const uint64_t expect = pair_group_size(L, compress);
    if (expect * (uint64_t)W * 2 <= kMaxGroupBytes) out.reserve((size_t)expect * W);
    std::vector<int16_t> cur(W), n(W);
    auto at = [&](const Gen& g, int j) { return g.neg[j] ? (int16_t)-cur[g.src[j]] : cur[g.src[j]]; };
    for (int i = 0; i < L; ++i) {
        cur[i] = (int16_t)(i + 1);
        cur[L + i] = (int16_t)(L + i + 1);
    }
    add(cur.data());
    for (size_t item = 0; item < count; ++item) {
        std::memcpy(cur.data(), out.data() + item * W, (size_t)W * 2);
        for (const Gen& g : gens) {
            if (by_key) {  // look the image up by its key; write it out only when new
                const uint64_t k = (uint64_t)(uint16_t)at(g, 0) | (uint64_t)(uint16_t)at(g, 1) << 16 |
                                   (uint64_t)(uint16_t)at(g, L) << 32 | (uint64_t)(uint16_t)at(g, L + 1) << 48;
                if (find_key(k)) continue;
            }
            for (int j = 0; j < W; ++j) n[j] = at(g, j);
            add(n.data());
        }
    }
    return out;
}

std::vector<int16_t> pair_generators(int L, int compress) {
    if (L >= 3) {
        std::vector<int16_t> g = pair_closure(L, compress, true);
        if (g.size() == pair_group_size(L, compress) * (uint64_t)(2 * L)) return g;
    }
    return pair_closure(L, compress, false);
}

// Rewrites a generator item as "output position o takes +-input[src]" over
// the concatenated pair (a then b), following equivalence.cpp:108-136.
std::vector<int16_t> as_sources(const int16_t* item, int L) {
    std::vector<int16_t> out(2 * L);
    const int a0 = item[0];
    const bool swapped = (a0 < 0 && -a0 > L) || (a0 > 0 && a0 > L);
    for (int i = 0; i < L; ++i) {
        const int ia = item[i], ib = item[L + i];
        const int pa = ((ia < 0 ? -ia : ia) - 1) % L, pb = ((ib < 0 ? -ib : ib) - 1) % L;
        if (swapped) {
            // new b[i] = +-a[pa], new a[i] = +-b[pb]
            out[L + i] = (int16_t)((ia < 0 ? -1 : 1) * (pa + 1));
            out[i] = (int16_t)((ib < 0 ? -1 : 1) * (L + pb + 1));
        } else {
            out[i] = (int16_t)((ia < 0 ? -1 : 1) * (pa + 1));
            out[L + i] = (int16_t)((ib < 0 ? -1 : 1) * (L + pb + 1));
        }
    }
    return out;
}

uint64_t pair_group_size(int L, int compress);

unsigned grid_of(int64_t n, int block) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + block - 1) / block, 1 << 16));
}

// The pair file's values as strtol reads them one after the other: whitespace-
// separated integers up to the first token that is not one.
std::vector<int8_t> host_values(const char* text) {
    std::vector<int8_t> vals;
    for (const char* q = text;;) {
        char* e;
        const long v = strtol(q, &e, 10);
        if (e == q) break;
        q = e;
        vals.push_back((int8_t)v);
    }
    return vals;
}

// A pair set on the device: distinct pairs in order, and what sorting rows of
// their values takes.  Buffers eq[..] of the context.
struct PairSet {
    gp_ctx* c;
    int W;
    int64_t np = 0;       // distinct pairs
    int8_t* rows = nullptr;
    int bits = 1, Wk = 1; // key layout
    const uint8_t* code = nullptr;
    bool small = false;   // a small file: parsed, sorted and written by the host
    std::vector<int8_t> host;  // then the rows here too
};

enum EqBuf { kEqText, kEqCount, kEqOffs, kEqScan, kEqVals, kEqInfo, kEqCode, kEqKeys, kEqIdx, kEqTmp, kEqFlag, kEqPos,
             kEqOut, kEqRows, kEqCanon, kEqUnits, kEqFix, kEqAlive, kEqBytes, kEqLine };

// Sorts n rows: idx (device) in the rows' order, equal rows in index order,
// flags[k] = 1 where the k-th row differs from the one before.
int sort_rows(PairSet& ps, const int8_t* rows, int64_t n, uint32_t* idx, uint32_t* flags, cudaStream_t s) {
    gp_ctx* c = ps.c;
    DevBuf &keys = c->eq[kEqKeys], &tmp = c->eq[kEqTmp];
    if (!keys.ensure((size_t)n * ps.Wk * 4) || !tmp.ensure(gp::radix_sort_tmp_bytes(n, ps.Wk)))
        return c->fail(GP_ERR_NOMEM, "equivalence filter: sort buffers");
    pair_keys_kernel<<<grid_of(n * ps.Wk, 256), 256, 0, s>>>(rows, n, ps.W, ps.code, ps.bits, ps.Wk,
                                                             keys.as<uint32_t>());
    GP_CUDA_TRY(c, cudaGetLastError());
    GP_CUDA_TRY(c, gp::iota_u32(idx, n, s));
    GP_CUDA_TRY(c, gp::radix_sort_keys(keys.as<uint32_t>(), ps.Wk, ps.Wk, idx, n, tmp.p, s, 8));
    GP_CUDA_TRY(c, gp::mark_unique(keys.as<uint32_t>(), ps.Wk, idx, n, ps.Wk, flags, s));
    return GP_OK;
}

// Files up to this size are the host's: parsing and sorting on the device is some
// fifty launches and nine waits, as many for two pairs as for twenty thousand.
// The two ways meet between 38 KB (length 6) and 90 KB (length 90).  On the host
// and on the device: 2 pairs of length 6 91 and 330 us, 1,000 (32 KB) 328 and
// 380, 2,000 571 and 417; 100 pairs of length 57 (29 KB) 268 and 485, 200 438 and
// 504, 300 617 and 518.
constexpr size_t kHostText = 40 << 10;

// Numbers of the n rows of W bytes in the rows' order, equal rows in index order.
std::vector<uint32_t> host_order(const uint8_t* rows, int64_t n, int W) {
    std::vector<uint32_t> ord(n);
    for (int64_t i = 0; i < n; ++i) ord[i] = (uint32_t)i;
    std::sort(ord.begin(), ord.end(), [&](uint32_t x, uint32_t y) {
        const int d = std::memcmp(rows + (size_t)x * W, rows + (size_t)y * W, (size_t)W);
        return d != 0 ? d < 0 : x < y;
    });
    return ord;
}

// load_pairs on the host; the rows go to the device for canon_kernel.
int load_pairs_host(PairSet& ps, const char* text, cudaStream_t s) {
    gp_ctx* c = ps.c;
    const int W = ps.W;
    const std::vector<int8_t> vals = host_values(text);
    const int64_t n = (int64_t)vals.size() / W;
    std::vector<uint8_t> bytes((size_t)n * W);  // in the order of the values
    for (size_t i = 0; i < bytes.size(); ++i) bytes[i] = (uint8_t)(vals[i] ^ 0x80);
    const uint8_t* last = nullptr;
    for (uint32_t i : host_order(bytes.data(), n, W)) {
        const uint8_t* row = bytes.data() + (size_t)i * W;
        if (last && std::memcmp(last, row, (size_t)W) == 0) continue;
        last = row;
        ps.host.insert(ps.host.end(), vals.begin() + (size_t)i * W, vals.begin() + (size_t)(i + 1) * W);
    }
    ps.small = true;
    ps.np = (int64_t)ps.host.size() / W;
    if (ps.np == 0) return GP_OK;
    DevBuf& drow = c->eq[kEqRows];
    if (!drow.ensure(ps.host.size())) return c->fail(GP_ERR_NOMEM, "equivalence filter: pairs");
    ps.rows = drow.as<int8_t>();
    GP_CUDA_TRY(c, cudaMemcpyAsync(ps.rows, ps.host.data(), ps.host.size(), cudaMemcpyHostToDevice, s));
    return GP_OK;
}

// filter.cpp:45-62: L values for a, then (if the stream is still good) L for
// b: whitespace-separated integers up to the first token that is not one, W
// per pair, a trailing partial pair dropped; then the set of the pairs.
// `text` holds n bytes and a terminating zero.
int load_pairs(PairSet& ps, const char* text, size_t n, cudaStream_t s) {
    gp_ctx* c = ps.c;
    if (n == 0 || ps.W < 1) return GP_OK;  // no values, or none to a pair
    if (n <= kHostText) return load_pairs_host(ps, text, s);
    const bool huge = n >> 32;  // more text than the device's 32-bit offsets reach
    const int64_t blocks = huge ? 1 : (int64_t)((n + kParseBlock - 1) / kParseBlock);
    DevBuf &dt = c->eq[kEqText], &dcnt = c->eq[kEqCount], &doff = c->eq[kEqOffs], &dscan = c->eq[kEqScan],
           &dv = c->eq[kEqVals], &dinfo = c->eq[kEqInfo], &dcode = c->eq[kEqCode];
    // a value takes two bytes of text at least (one blank), but for the last
    const size_t padded = (size_t)(blocks + 1) * kParseBlock;
    if (!dt.ensure(padded) || !dcnt.ensure((size_t)blocks * 4) || !doff.ensure((size_t)blocks * 4) ||
        !dscan.ensure(gp::scan_tmp_bytes(blocks)) || !dv.ensure(padded / 2 + 1) || !dinfo.ensure(sizeof(TextInfo)) ||
        !dcode.ensure(256))
        return c->fail(GP_ERR_NOMEM, "equivalence filter: text buffers");
    TextInfo info{};
    uint32_t last[2] = {0, 0};
    if (!huge) {
        GP_CUDA_TRY(c, cudaMemsetAsync(static_cast<char*>(dt.p) + n, ' ', padded - n, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(dt.p, text, n, cudaMemcpyHostToDevice, s));
        GP_CUDA_TRY(c, cudaMemsetAsync(dinfo.p, 0, sizeof(TextInfo), s));
        pair_values_kernel<false><<<(unsigned)blocks, kParseThreads, 0, s>>>(dt.as<char>(), dcnt.as<uint32_t>(), nullptr,
                                                                             nullptr, dinfo.as<TextInfo>());
        GP_CUDA_TRY(c, cudaGetLastError());
        GP_CUDA_TRY(c, gp::exclusive_scan_u32(dcnt.as<uint32_t>(), doff.as<uint32_t>(), blocks, dscan.as<uint32_t>(), s));
        pair_values_kernel<true><<<(unsigned)blocks, kParseThreads, 0, s>>>(dt.as<char>(), dcnt.as<uint32_t>(),
                                                                            doff.as<uint32_t>(), dv.as<int8_t>(),
                                                                            dinfo.as<TextInfo>());
        GP_CUDA_TRY(c, cudaGetLastError());
        GP_CUDA_TRY(c, cudaMemcpyAsync(&info, dinfo.p, sizeof info, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[0], doff.as<uint32_t>() + blocks - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[1], dcnt.as<uint32_t>() + blocks - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    }
    int64_t nvals = (int64_t)last[0] + last[1];
    if (huge || info.bad) {  // signs, other characters or large values: as strtol takes them
        const std::vector<int8_t> vals = host_values(text);
        nvals = (int64_t)vals.size();
        info = TextInfo{};
        for (int8_t v : vals) info.present[(v + 128) >> 5] |= 1u << (v & 31);
        if (!dv.ensure(vals.size() + 1)) return c->fail(GP_ERR_NOMEM, "equivalence filter: values");
        GP_CUDA_TRY(c, cudaMemcpyAsync(dv.p, vals.data(), vals.size(), cudaMemcpyHostToDevice, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    }
    const int64_t n0 = nvals / ps.W;
    if (n0 == 0) return GP_OK;
    if (n0 > INT32_MAX) return c->fail(GP_ERR_UNSUPPORTED, "equivalence filter: %lld pairs", (long long)n0);
    // ranks of the values that occur and of their negatives (images change signs)
    uint8_t code[256] = {};
    int used = 0;
    for (int v = -128; v < 128; ++v) {
        const int8_t neg = (int8_t)-v;
        if (((info.present[(v + 128) >> 5] >> (v & 31)) & 1u) || ((info.present[(neg + 128) >> 5] >> (neg & 31)) & 1u))
            code[(uint8_t)v] = (uint8_t)used++;
    }
    ps.bits = 1;
    while ((1 << ps.bits) < used) ++ps.bits;
    const int per = 32 / ps.bits;
    ps.Wk = (ps.W + per - 1) / per;
    ps.code = dcode.as<uint8_t>();
    GP_CUDA_TRY(c, cudaMemcpyAsync(dcode.p, code, 256, cudaMemcpyHostToDevice, s));
    DevBuf &didx = c->eq[kEqIdx], &dflag = c->eq[kEqFlag], &dpos = c->eq[kEqPos], &dout = c->eq[kEqOut],
           &drow = c->eq[kEqRows];
    if (!didx.ensure((size_t)n0 * 4) || !dflag.ensure((size_t)n0 * 4) || !dpos.ensure((size_t)n0 * 4) ||
        !dscan.ensure(gp::scan_tmp_bytes(n0)) || !dout.ensure((size_t)n0 * 4 + 4))
        return c->fail(GP_ERR_NOMEM, "equivalence filter: sort buffers");
    const int rc = sort_rows(ps, dv.as<int8_t>(), n0, didx.as<uint32_t>(), dflag.as<uint32_t>(), s);
    if (rc) return rc;
    uint32_t* d_cnt = dout.as<uint32_t>() + n0;
    GP_CUDA_TRY(c, gp::compact_flags(dflag.as<uint32_t>(), didx.as<uint32_t>(), dout.as<uint32_t>(), n0,
                                     dpos.as<uint32_t>(), dscan.as<uint32_t>(), d_cnt, s));
    uint32_t nu = 0;
    GP_CUDA_TRY(c, cudaMemcpyAsync(&nu, d_cnt, 4, cudaMemcpyDeviceToHost, s));
    GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    ps.np = nu;
    if (!drow.ensure((size_t)nu * ps.W)) return c->fail(GP_ERR_NOMEM, "equivalence filter: pairs");
    ps.rows = drow.as<int8_t>();
    gather_rows_kernel<<<grid_of((int64_t)nu * ps.W, 256), 256, 0, s>>>(dv.as<int8_t>(), dout.as<uint32_t>(), nu, ps.W,
                                                                        ps.rows);
    GP_CUDA_TRY(c, cudaGetLastError());
    return GP_OK;
}

// Class sizes and members of a pair set by canonical forms (canon_kernel):
// member_list[span[i].first .. span[i].second) are the pairs with the same
// least image as pair i (itself included), csize[i] is the group order over
// the number of elements fixing pair i.  L >= 3.
int canonical_classes(PairSet& ps, int L, int compress, std::vector<unsigned long long>& csize,
                      std::vector<uint32_t>& member_list, std::vector<std::pair<uint32_t, uint32_t>>& span,
                      cudaStream_t s) {
    gp_ctx* c = ps.c;
    const int W = 2 * L;
    const int64_t np = ps.np;
    const std::vector<int16_t> units = all_units(L);
    DevBuf &du = c->eq[kEqUnits], &dc = c->eq[kEqCanon], &df = c->eq[kEqFix], &didx = c->eq[kEqIdx],
           &dflag = c->eq[kEqFlag];
    if (!du.ensure(units.size() * 2) || !dc.ensure((size_t)np * W) || !df.ensure((size_t)np * 4))
        return c->fail(GP_ERR_NOMEM, "equivalence filter: device allocation");
    GP_CUDA_TRY(c, cudaMemcpyAsync(du.p, units.data(), units.size() * 2, cudaMemcpyHostToDevice, s));
    CanonArgs ca{};
    ca.pairs = ps.rows;
    ca.np = np;
    ca.L = L;
    ca.units = du.as<int16_t>();
    ca.nu = (int)units.size();
    ca.alt = !(compress > 1 || L % 2 == 1) ? 1 : 0;  // filter.cpp:83-87
    ca.canon = dc.as<int8_t>();
    ca.fixers = df.as<uint32_t>();
    const size_t smem = kCanonWarps * canon_layout(L, 2 * (ca.alt ? 4 : 1) * ca.nu).per_warp;
    const int64_t grid = std::min<int64_t>((np + kCanonWarps - 1) / kCanonWarps, (int64_t)c->num_sms * 16);
    canon_kernel<<<(unsigned)grid, 32 * kCanonWarps, smem, s>>>(ca);
    GP_CUDA_TRY(c, cudaGetLastError());
    // the classes: runs of equal least images
    std::vector<uint32_t> fixers(np), flags(np);
    if (ps.small) {
        std::vector<uint8_t> canon((size_t)np * W);
        GP_CUDA_TRY(c, cudaMemcpyAsync(fixers.data(), df.p, (size_t)np * 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(canon.data(), dc.p, canon.size(), cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        member_list = host_order(canon.data(), np, W);
        for (int64_t k = 0; k < np; ++k)
            flags[k] = k == 0 || std::memcmp(&canon[(size_t)member_list[k - 1] * W],
                                             &canon[(size_t)member_list[k] * W], (size_t)W) != 0;
    } else {
        const int rc = sort_rows(ps, ca.canon, np, didx.as<uint32_t>(), dflag.as<uint32_t>(), s);
        if (rc) return rc;
        member_list.resize(np);
        GP_CUDA_TRY(c, cudaMemcpyAsync(fixers.data(), df.p, (size_t)np * 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(flags.data(), dflag.p, (size_t)np * 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(member_list.data(), didx.p, (size_t)np * 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    }
    const uint64_t G = pair_group_size(L, compress);
    for (int64_t i = 0; i < np; ++i) {
        if (fixers[i] == 0 || G % fixers[i] != 0)
            return c->fail(GP_ERR_CUDA, "equivalence filter: %u of %llu elements fix pair %lld", fixers[i],
                           (unsigned long long)G, (long long)i);
        csize[i] = G / fixers[i];
    }
    for (int64_t r0 = 0; r0 < np;) {
        int64_t r1 = r0 + 1;
        while (r1 < np && !flags[r1]) ++r1;
        for (int64_t k = r0; k < r1; ++k) span[member_list[k]] = {(uint32_t)r0, (uint32_t)r1};
        r0 = r1;
    }
    return GP_OK;
}

// The kept pairs' lines, in order.
int pair_lines(PairSet& ps, const std::vector<char>& alive, std::string& out, cudaStream_t s) {
    gp_ctx* c = ps.c;
    out.clear();
    if (ps.np == 0) return GP_OK;
    const int64_t np = ps.np;
    if (ps.small) {
        const int W = ps.W, L = W / 2;
        for (int64_t i = 0; i < np; ++i) {
            if (!alive[i]) continue;
            for (int o = 0; o < W; ++o) {
                if (o == L) out.push_back(' ');
                gp::put_int_sp(out, ps.host[(size_t)i * W + o]);
            }
            out.push_back('\n');
        }
        return GP_OK;
    }
    // rows at a time: a block's text stays below 2^31 bytes (5 bytes a value at most)
    const int64_t step = std::min<int64_t>(np, (int64_t(1) << 31) / (5 * ps.W + 2));
    DevBuf &da = c->eq[kEqAlive], &db = c->eq[kEqBytes], &dat = c->eq[kEqPos], &dscan = c->eq[kEqScan],
           &dl = c->eq[kEqLine];
    if (!da.ensure((size_t)np) || !db.ensure((size_t)step * 4) || !dat.ensure((size_t)step * 4) ||
        !dscan.ensure(gp::scan_tmp_bytes(step)))
        return c->fail(GP_ERR_NOMEM, "equivalence filter: line buffers");
    GP_CUDA_TRY(c, cudaMemcpyAsync(da.p, alive.data(), (size_t)np, cudaMemcpyHostToDevice, s));
    for (int64_t r0 = 0; r0 < np; r0 += step) {
        const int64_t n = std::min(step, np - r0);
        const int8_t* rows = ps.rows + r0 * ps.W;
        const uint8_t* keep = da.as<uint8_t>() + r0;
        pair_line_bytes_kernel<<<grid_of(n, 256), 256, 0, s>>>(rows, keep, n, ps.W, db.as<uint32_t>());
        GP_CUDA_TRY(c, cudaGetLastError());
        GP_CUDA_TRY(c, gp::exclusive_scan_u32(db.as<uint32_t>(), dat.as<uint32_t>(), n, dscan.as<uint32_t>(), s));
        uint32_t last[2] = {0, 0};
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[0], dat.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaMemcpyAsync(&last[1], db.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
        const size_t bytes = (size_t)last[0] + last[1];
        if (!dl.ensure(bytes + 1)) return c->fail(GP_ERR_NOMEM, "equivalence filter: text buffer");
        pair_lines_kernel<<<grid_of(n, 8), 256, 0, s>>>(rows, keep, n, ps.W, dat.as<uint32_t>(), dl.as<char>());
        GP_CUDA_TRY(c, cudaGetLastError());
        const size_t at = out.size();
        out.resize(at + bytes);
        GP_CUDA_TRY(c, cudaMemcpyAsync(&out[at], dl.p, bytes, cudaMemcpyDeviceToHost, s));
        GP_CUDA_TRY(c, cudaStreamSynchronize(s));
    }
    return GP_OK;
}

// Size of the generator group: 4 phi(L) L^2, times 8 sign patterns with the
// alternating negation (exact for L >= 3, an upper bound at L = 2).
uint64_t pair_group_size(int L, int compress) {
    uint64_t phi = 0;
    for (int u = 1; u <= L; ++u)
        if (std::gcd(u, L) == 1) ++phi;
    const bool use_alt = !(compress > 1 || L % 2 == 1);
    return 4 * phi * (uint64_t)L * (uint64_t)L * (use_alt ? 8 : 1);
}

// The group's items take 2L int16 each on the host and again on the device.
extern const uint64_t kMaxGroupBytes = uint64_t(1) << 32;

}  // namespace

extern "C" {

// 1 when the affine parametrisation the canonical-form kernel enumerates
// (swap, e, signs, u, s_a, s_b) gives exactly the closure's group of length
// L at this compression, 0 when not, -1 when not applicable (L < 3 or too
// large).  Host only; a test hook.
int gp_debug_pair_group_check(int L, int compress) {
    if (L < 3 || 2 * L > kMaxW || compress < 1) return -1;
    if (pair_group_size(L, compress) * (uint64_t)(4 * L) > kMaxGroupBytes) return -1;
    const int W = 2 * L;
    const bool alt = !(compress > 1 || L % 2 == 1);
    const std::vector<int16_t> units = all_units(L);
    std::vector<std::vector<int16_t>> mine, closure;
    for (int swap = 0; swap < 2; ++swap)
        for (int e = 0; e < 2; ++e)
            for (int pat = 0; pat < (alt ? 8 : 1); ++pat)
                for (int16_t u : units)
                    for (int sa = 0; sa < L; ++sa)
                        for (int sb = 0; sb < L; ++sb) {
                            const int ha = swap ? L : 0, hb = swap ? 0 : L, ma = u, mb = e ? L - u : u;
                            const int alpha = pat & 1, ba = (pat >> 1) & 1, bb = (pat >> 2) & 1;
                            std::vector<int16_t> item(W);
                            for (int i = 0; i < L; ++i) {
                                const int sga = ((alpha & i) ^ ba) & 1 ? -1 : 1, sgb = ((alpha & i) ^ bb) & 1 ? -1 : 1;
                                item[i] = (int16_t)(sga * (ha + (int)(((long long)ma * i + sa) % L) + 1));
                                item[L + i] = (int16_t)(sgb * (hb + (int)(((long long)mb * i + sb) % L) + 1));
                            }
                            mine.push_back(std::move(item));
                        }
    const std::vector<int16_t> g = pair_generators(L, compress);
    for (size_t i = 0; i + W <= g.size(); i += W) closure.emplace_back(g.begin() + i, g.begin() + i + W);
    std::sort(mine.begin(), mine.end());
    std::sort(closure.begin(), closure.end());
    return mine == closure ? 1 : 0;
}

int64_t gp_debug_pair_generator_count(int L, int compress) {
    if (L < 1 || 2 * L > kMaxW || compress < 1) return -1;
    if (pair_group_size(L, compress) * (uint64_t)(4 * L) > kMaxGroupBytes) return -1;
    return (int64_t)(pair_generators(L, compress).size() / (size_t)(2 * L));
}

static int gp_equiv_filter_impl(gp_ctx* c, int order, int compress, const char* in_path, const char* out_path) {
    StageRange nvtx_range("gp_equiv_filter");
    if (!c || !in_path || !out_path) return GP_ERR_ARG;
    if (compress < 1 || order % compress) return c->fail(GP_ERR_ARG, "order %d not divisible by %d", order, compress);
    cudaSetDevice(c->device);
    const int L = order / compress;
    const int W = 2 * L;
    if (W > kMaxW) return c->fail(GP_ERR_UNSUPPORTED, "equivalence filter: length %d", L);
    if (L < 3 && pair_group_size(L, compress) * (uint64_t)(2 * W) > kMaxGroupBytes)  // the table path only
        return c->fail(GP_ERR_UNSUPPORTED, "equivalence filter: %llu generators at length %d exceed %llu bytes",
                       (unsigned long long)pair_group_size(L, compress), L, (unsigned long long)kMaxGroupBytes);
    // GP_EQUIV_TIMING=1 in the environment prints the phase times to stderr (diagnostics)
    static const bool timing = getenv("GP_EQUIV_TIMING") != nullptr;
    const auto t0 = std::chrono::steady_clock::now();
    auto lap = [&](const char* what) {
        if (timing)
            fprintf(stderr, "[equiv] %s %.4f s\n", what,
                    std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
    };
    FILE* out = fopen(out_path, "w");  // filter.cpp:24 opens the output first
    FILE* in = fopen(in_path, "rb");
    if (!in) {
        if (out) fclose(out);
        return GP_OK;  // filter.cpp:33-37: "Bad File." and success
    }
    // the generator group depends only on (L, compression): built on a host
    // thread while the pairs are read and sorted
    std::vector<int16_t> gens;
    bool group_failed = false;
    std::thread group_thread;
    if (L < 3)  // the table of every element (longer lengths use canonical forms)
        group_thread = std::thread([&] {
            try {
                gens = pair_generators(L, compress);
            } catch (const std::exception&) {
                group_failed = true;
            }
        });
    struct Joiner {
        std::thread& t;
        ~Joiner() {
            if (t.joinable()) t.join();
        }
    } joiner{group_thread};
    std::string text;
    {
        fseek(in, 0, SEEK_END);
        const long sz = ftell(in);
        fseek(in, 0, SEEK_SET);
        text.resize(sz > 0 ? (size_t)sz : 0);
        text.resize(sz > 0 ? fread(&text[0], 1, (size_t)sz, in) : 0);
        fclose(in);
    }
    lap("read");
    struct OutCloser {  // an error leaves the output empty, as opened
        FILE*& f;
        ~OutCloser() {
            if (f) fclose(f);
        }
    } out_closer{out};
    cudaStream_t s = c->s_comp;
    KeepSmall keep{c->eq};
    PairSet ps{c, W};
    int rc = load_pairs(ps, text.c_str(), text.size(), s);
    if (rc) return rc;
    std::string().swap(text);
    lap("pairs");
    const int64_t np = ps.np;
    std::vector<char> alive(np, 1);
    if (np > 0) {
        std::vector<unsigned long long> csize(np);
        // the input pairs of each pair's class: member_list[span[i].first .. span[i].second)
        std::vector<uint32_t> member_list;
        std::vector<std::pair<uint32_t, uint32_t>> span(np);
        if (L >= 3) {
            rc = canonical_classes(ps, L, compress, csize, member_list, span, s);
            if (rc) return rc;
            lap("classes");
        } else {
            group_thread.join();
            if (group_failed) return c->fail(GP_ERR_NOMEM, "equivalence filter: generator group of length %d", L);
            lap("group");
            const int64_t ng = (int64_t)(gens.size() / (size_t)W);
            std::vector<int16_t> items((size_t)ng * W);  // transposed: items[o * ng + g]
            // blocks of 64 generators: each thread writes whole cache lines of every row
            gp::par_for((size_t)((ng + 63) / 64), [&](size_t blk) {
                for (int64_t g = (int64_t)blk * 64; g < std::min<int64_t>((int64_t)blk * 64 + 64, ng); ++g) {
                    const auto src = as_sources(gens.data() + (size_t)g * W, L);
                    for (int o = 0; o < W; ++o) items[(size_t)o * ng + g] = src[o];
                }
            });
            lap("table");
            std::vector<int8_t> pairs = ps.host;
            if (!ps.small) {
                pairs.resize((size_t)np * W);
                GP_CUDA_TRY(c, cudaMemcpyAsync(pairs.data(), ps.rows, pairs.size(), cudaMemcpyDeviceToHost, s));
                GP_CUDA_TRY(c, cudaStreamSynchronize(s));
            }
            // hash set of the pairs (the image lookup), same hash as the kernel's
            uint32_t set_size = 1;
            while (set_size < 2 * (uint64_t)np) set_size <<= 1;
            std::vector<uint32_t> set_h(set_size, 0), set_i(set_size, 0xFFFFFFFFu);
            for (int64_t i = 0; i < np; ++i) {
                uint32_t h = kFnvBasis;
                for (int j = 0; j < W; ++j) h = fnv_step(h, pairs[i * W + j]);
                h = fnv_fold(h);
                uint32_t slot = h & (set_size - 1);
                while (set_i[slot] != 0xFFFFFFFFu) slot = (slot + 1) & (set_size - 1);
                set_h[slot] = h;
                set_i[slot] = (uint32_t)i;
            }
            const int64_t mcap = std::max<int64_t>(np * 64, 1 << 20);
            DevBuf di, dsh, dsi, dst, dm, dmisc;
            if (!di.ensure(items.size() * 2) || !dsh.ensure((size_t)set_size * 4) ||
                !dsi.ensure((size_t)set_size * 4) || !dst.ensure(np * 4) || !dm.ensure((size_t)mcap * 8) ||
                !dmisc.ensure(64))
                return c->fail(GP_ERR_NOMEM, "equivalence filter: device allocation");
            GP_CUDA_TRY(c, cudaMemcpyAsync(di.p, items.data(), items.size() * 2, cudaMemcpyHostToDevice, s));
            GP_CUDA_TRY(c, cudaMemcpyAsync(dsh.p, set_h.data(), (size_t)set_size * 4, cudaMemcpyHostToDevice, s));
            GP_CUDA_TRY(c, cudaMemcpyAsync(dsi.p, set_i.data(), (size_t)set_size * 4, cudaMemcpyHostToDevice, s));
            GP_CUDA_TRY(c, cudaMemsetAsync(dst.p, 0, np * 4, s));
            GP_CUDA_TRY(c, cudaMemsetAsync(dmisc.p, 0, 64, s));
            ClassArgs ca{};
            ca.srcT = di.as<int16_t>();
            ca.ng = ng;
            ca.pairs = ps.rows;
            ca.np = np;
            ca.W = W;
            ca.set_h = dsh.as<uint32_t>();
            ca.set_i = dsi.as<uint32_t>();
            ca.set_mask = set_size - 1;
            ca.stab = dst.as<uint32_t>();
            ca.members = dm.as<uint32_t>();
            ca.nmembers = dmisc.as<unsigned long long>();
            ca.mcap = mcap;
            ca.status = c->status.as<int>();
            const int64_t groups = (np + kPairsPerCta - 1) / kPairsPerCta;
            // generator shares per group: enough CTAs for eight per SM, each share
            // at least one generator per thread
            const int64_t want = std::max<int64_t>(1, (8 * (int64_t)c->num_sms + groups - 1) / groups);
            const int splits = (int)std::max<int64_t>(1, std::min<int64_t>(want, (ng + 255) / 256));
            for (int64_t g0 = 0; g0 < groups; g0 += (int64_t(1) << 20)) {  // grids of at most 2^20 groups
                const int64_t gn = std::min<int64_t>(groups - g0, int64_t(1) << 20);
                ClassArgs cb = ca;
                cb.group0 = g0;
                class_kernel<<<(unsigned)(gn * splits), 256, 0, s>>>(cb, splits);
            }
            GP_CUDA_TRY(c, cudaGetLastError());
            GP_CUDA_TRY(c, cudaStreamSynchronize(s));
            lap("classes");
            rc = c->check_status("equivalence filter");
            if (rc) return rc;
            std::vector<uint32_t> stab(np);
            unsigned long long nmem = 0;
            GP_CUDA_TRY(c, cudaMemcpy(stab.data(), dst.p, np * 4, cudaMemcpyDeviceToHost));
            GP_CUDA_TRY(c, cudaMemcpy(&nmem, dmisc.p, 8, cudaMemcpyDeviceToHost));
            // orbit-stabiliser: class size = group order / generators fixing the pair
            for (int64_t i = 0; i < np; ++i) {
                if (stab[i] == 0 || ng % stab[i] != 0)
                    return c->fail(GP_ERR_CUDA, "equivalence filter: stabiliser of pair %lld is %u of %lld generators",
                                   (long long)i, stab[i], (long long)ng);
                csize[i] = (unsigned long long)(ng / stab[i]);
            }
            std::vector<uint32_t> mem((size_t)nmem * 2);
            if (nmem) GP_CUDA_TRY(c, cudaMemcpy(mem.data(), dm.p, mem.size() * 4, cudaMemcpyDeviceToHost));
            std::vector<std::vector<uint32_t>> members(np);
            for (unsigned long long i = 0; i < nmem; ++i) members[mem[2 * i]].push_back(mem[2 * i + 1]);
            for (int64_t i = 0; i < np; ++i) {
                span[i].first = (uint32_t)member_list.size();
                member_list.insert(member_list.end(), members[i].begin(), members[i].end());
                span[i].second = (uint32_t)member_list.size();
            }
        }
        // filter.cpp:117-144, in set order
        int64_t n_alive = np;
        for (int64_t it = 0; it < np; ++it) {
            if (!alive[it]) continue;
            const uint32_t* mb = member_list.data() + span[it].first;
            const uint32_t* me = member_list.data() + span[it].second;
            if ((int64_t)csize[it] > n_alive) {
                for (const uint32_t* m = mb; m < me; ++m)
                    if ((int64_t)*m > it && alive[*m]) {
                        alive[*m] = 0;
                        --n_alive;
                    }
            } else {
                for (const uint32_t* m = mb; m < me; ++m)
                    if (alive[*m]) {
                        alive[*m] = 0;
                        --n_alive;
                    }
                if (!alive[it]) {
                    alive[it] = 1;
                    ++n_alive;
                }
            }
        }
    }
    lap("erase");
    if (out) {
        std::string lines;
        rc = pair_lines(ps, alive, lines, s);
        if (rc) return rc;
        const bool ok = lines.empty() || fwrite(lines.data(), 1, lines.size(), out) == lines.size();
        const int closed = fclose(out);
        out = nullptr;
        if (closed != 0 || !ok) return c->fail(GP_ERR_IO, "equivalence filter: write failed: %s", out_path);
    }
    lap("written");
    return GP_OK;
}

// No C++ exception (an allocation failure on a huge input) crosses the C ABI.
int gp_equiv_filter(gp_ctx* c, int order, int compress, const char* in_path, const char* out_path) {
    try {
        return gp_equiv_filter_impl(c, order, compress, in_path, out_path);
    } catch (const std::exception& e) {
        return c ? c->fail(GP_ERR_NOMEM, "equivalence filter: %s", e.what()) : GP_ERR_NOMEM;
    }
}

}  // extern "C"
