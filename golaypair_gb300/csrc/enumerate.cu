// enumerate.cu -- rank-window necklace enumerator (kernel (a)).
//
// Restates generate_necklaces_prefix / generate_necklaces_wrapper
// (src/utils/lyndon.cpp:47-121) and the row-sum gate of generate_hybrid
// (src/core/generate/generate_hybrid.cpp:35-41,139-154) for the GPU.
//
// The reference walks the FKM recursion over the sorted alphabet and sees
// every prenecklace of length L in lexicographic order, keeping those whose
// period divides L (necklaces).  Here the word space is cut into rank
// windows; each thread starts at the first prenecklace >= its window's first
// word and steps the FKM successor
//     i = last position whose digit is not maximal; a_i += 1;
//     a_j = a_{j-(i+1)} for j > i  (period i + 1)
// until it leaves the window.  Words are packed (see rows.cuh), so the
// successor is a handful of 64- or 128-bit bit operations.  One step takes a
// block of up to 64 words: those that share all but their last six bits, t
// digits.  Which of them are necklaces depends on the word's first t - 1
// digits only, so it is one table entry, and so are the ones whose digit sum
// matches a decomposition's row sum, by the sum of the other digits: a
// step's necklaces are counted and its candidates found without visiting
// them.  Candidates are appended (warp-aggregated) to a buffer with their A/B
// role bits.
//
// One launch serves several jobs (orders / compressions, each with its own
// length, alphabet, row-sum table and candidate buffer): every window names
// its job.  A window whose job's buffer has met its soft capacity is left
// with its position saved; the host drains the buffers and relaunches.
#include <type_traits>

#include "gp_device.cuh"
#include "enumerate.h"

namespace gp {

namespace {

struct W128 {
    uint64_t lo, hi;
};
__device__ __forceinline__ W128 w128(const U128p& v) { return {v.lo, v.hi}; }

__device__ __forceinline__ W128 shr(W128 a, int s) {
    if (s <= 0) return a;
    if (s >= 128) return {0, 0};
    if (s >= 64) return {a.hi >> (s - 64), 0};
    return {(a.lo >> s) | (a.hi << (64 - s)), a.hi >> s};
}
__device__ __forceinline__ W128 shl(W128 a, int s) {
    if (s <= 0) return a;
    if (s >= 128) return {0, 0};
    if (s >= 64) return {0, a.lo << (s - 64)};
    return {a.lo << s, (a.hi << s) | (a.lo >> (64 - s))};
}
__device__ __forceinline__ W128 band(W128 a, W128 b) { return {a.lo & b.lo, a.hi & b.hi}; }
__device__ __forceinline__ W128 bor(W128 a, W128 b) { return {a.lo | b.lo, a.hi | b.hi}; }
__device__ __forceinline__ W128 bxor(W128 a, W128 b) { return {a.lo ^ b.lo, a.hi ^ b.hi}; }
__device__ __forceinline__ bool is_zero(W128 a) { return (a.lo | a.hi) == 0; }
__device__ __forceinline__ bool lt(W128 a, W128 b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
__device__ __forceinline__ W128 low_mask(int bits) {  // 2^bits - 1
    if (bits >= 128) return {~0ull, ~0ull};
    if (bits >= 64) return {~0ull, bits == 64 ? 0ull : ((1ull << (bits - 64)) - 1ull)};
    return {bits == 0 ? 0ull : ((1ull << bits) - 1ull), 0ull};
}
__device__ __forceinline__ int ctz128(W128 a) {
    return a.lo ? __ffsll((long long)a.lo) - 1 : 64 + __ffsll((long long)a.hi) - 1;
}
__device__ __forceinline__ int digit(W128 w, int b, int L, int j) {
    const W128 s = shr(w, b * (L - 1 - j));
    return (int)(s.lo & ((1ull << b) - 1ull));
}

// Keeps the first p digits and repeats them with period p over L digits.
__device__ __forceinline__ W128 periodic_fill(W128 w, int b, int L, int p) {
    W128 x = band(w, bxor(low_mask(b * L), low_mask(b * (L - p))));
    for (int len = p; len < L; len <<= 1) x = bor(x, shr(x, b * len));
    return band(x, low_mask(b * L));
}

// The layout of a job's words, derived once per block (in shared memory).
struct JobView {
    int L, b;
    bool narrow;              // b * L <= 64: the word fits its low 64 bits
    uint32_t inv_b;           // floor(x / b) = (x * inv_b) >> 8 for 0 <= x < 128
    int lead_shift;           // a word's first t - 1 digits: word >> lead_shift
    uint32_t block;           // a block's words differ in these low bits
    W128 maxpat, full;        // full = low_mask(b * L)
    W128 ones;                // bit 0 of every digit; bit t of every digit = ones << t
    W128 divisors;            // bit p set iff p divides L (the necklace test, no division)
};

__device__ __forceinline__ JobView job_view(const EnumJob& j) {
    JobView v;
    v.L = j.L;
    v.b = j.b;
    v.maxpat = w128(j.maxpat);
    v.full = low_mask(j.b * j.L);
    v.ones = w128(j.plane[0]);
    v.lead_shift = j.b * (j.L - j.t + 1);
    v.block = (1u << (j.b * j.t)) - 1u;
    v.inv_b = (256u + (uint32_t)j.b - 1u) / (uint32_t)j.b;
    v.narrow = j.b * j.L <= 64;
    v.divisors = {0, 0};
    for (int p = 1; p <= j.L; ++p)
        if (j.L % p == 0) v.divisors = bor(v.divisors, shl({1ull, 0ull}, p));
    return v;
}

__device__ __forceinline__ bool divides_L(const JobView& a, int p) {
    return ((p < 64 ? (a.divisors.lo >> p) : (a.divisors.hi >> (p - 64))) & 1ull) != 0;
}

// FKM successor; returns the new period, or 0 when w was the last word.
__device__ __forceinline__ int fkm_next(W128& w, const JobView& a) {
    const W128 x = band(bxor(w, a.maxpat), a.full);
    if (is_zero(x)) return 0;
    const int r = (int)(((uint32_t)ctz128(x) * a.inv_b) >> 8);  // digits after the incremented one
    const int j = a.L - 1 - r;
    w = band(w, bxor(a.full, low_mask(a.b * r)));
    // increment digit j (it is below the maximum, so no carry)
    const W128 one = shl({1ull, 0ull}, a.b * r);
    w.lo += one.lo;
    w.hi += one.hi + (w.lo < one.lo ? 1ull : 0ull);
    const int p = j + 1;
    w = periodic_fill(w, a.b, a.L, p);
    return p;
}

// The same successor on words of at most 64 bits (native 64-bit shifts; no
// shift below reaches 64: b * len, b * r < b * L <= 64).
__device__ __forceinline__ uint64_t mask64(int bits) { return bits >= 64 ? ~0ull : ((1ull << bits) - 1ull); }

__device__ __forceinline__ int fkm_next64(uint64_t& w, const JobView& a) {
    const uint64_t x = (w ^ a.maxpat.lo) & a.full.lo;
    if (!x) return 0;
    const int r = (int)(((uint32_t)(__ffsll((long long)x) - 1) * a.inv_b) >> 8);
    const int p = a.L - r;  // the incremented digit is L - 1 - r; the new period is its index + 1
    w = (w & (a.full.lo ^ mask64(a.b * r))) + (1ull << (a.b * r));
    uint64_t y = w & (a.full.lo ^ mask64(a.b * r));
    for (int len = p; len < a.L; len <<= 1) y |= y >> (a.b * len);
    w = y & a.full.lo;
    return p;
}

// First prenecklace >= w (w a word of L digits); returns its period.
__device__ __forceinline__ int first_prenecklace(W128& w, int b, int L) {
    int p = 1;
    for (int i = 1; i < L; ++i) {
        const int d = digit(w, b, L, i), e = digit(w, b, L, i - p);
        if (d > e) {
            p = i + 1;
        } else if (d < e) {
            w = periodic_fill(w, b, L, p);
            return p;
        }
    }
    return p;
}

// The same on words of at most 63 bits.
__device__ __forceinline__ int first_prenecklace64(uint64_t& w, const JobView& a) {
    const uint64_t m = (1ull << a.b) - 1ull;
    int p = 1;
    for (int i = 1; i < a.L; ++i) {
        const uint64_t d = (w >> (a.b * (a.L - 1 - i))) & m, e = (w >> (a.b * (a.L - 1 - i + p))) & m;
        if (d > e) {
            p = i + 1;
        } else if (d < e) {
            const uint64_t full = a.full.lo;
            uint64_t y = w & (full ^ mask64(a.b * (a.L - p)));
            for (int len = p; len < a.L; len <<= 1) y |= y >> (a.b * len);
            w = y & full;
            return p;
        }
    }
    return p;
}

__device__ __forceinline__ int digit_sum64(uint64_t w, const JobView& a) {
    int s = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t)
        if (t < a.b) s += __popcll(w & (a.ones.lo << t)) << t;
    return s;
}

__device__ __forceinline__ int digit_sum(W128 w, const JobView& a) {
    int s = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (t < a.b) {
            const W128 m = band(w, shl(a.ones, t));
            s += (__popcll(m.lo) + __popcll(m.hi)) << t;
        }
    }
    return s;
}

__device__ __forceinline__ uint4 to_u4(W128 w) {
    return make_uint4((uint32_t)w.lo, (uint32_t)(w.lo >> 32), (uint32_t)w.hi, (uint32_t)(w.hi >> 32));
}
__device__ __forceinline__ W128 from_u4(uint4 v) {
    return {((uint64_t)v.y << 32) | v.x, ((uint64_t)v.w << 32) | v.z};
}
__device__ __forceinline__ bool job_full(const EnumJob& j) {
    return (int64_t)*reinterpret_cast<volatile unsigned long long*>(j.count) >= j.soft_cap;
}

// A warp takes windows from a global counter, up to 32 at a time: it loads
// them, drops finished ones and finds their first prenecklaces together, and
// hands them to its lanes as these run out of work.  A window whose job has
// reached its soft capacity is left (position saved), so one full job does not
// idle the others.
//
// Candidates go to a per-warp queue in shared memory first; the warp writes
// them out when kFlushAt or more are queued, with one counter atomic per
// job present.  What the atomic returns tells the warp when a job has met its
// soft capacity; warps that find few candidates look at the count every
// kCapCheck steps, on a load whose latency overlaps the steps in between.
//
// What bounds it: issue (67 %) once every lane has a dense window, the last
// windows' serial steps at the end.  An order-57 window of 2^32 words (2.3 G
// necklaces, 208 M candidates): 2.4 ms of kernel time, 9.4 when each lane took,
// loaded and checked its own windows and every 32 candidates took an atomic,
// 15.1 with blocks of two digits taken a row at a time; five orders: 16, 48 and
// 87 ms (27 with as many windows for all five as for one).  With that and
// queues of 192, blocks per SM 4, 5, 6: 2.56, 2.53, 2.70 and 27.0, 27.2, 30.4 ms.
//
// NARROW: every job's words fit 63 bits, so a word and its window end are
// 64-bit values (the high halves are zero and drop out of the registers).
constexpr int kCapCheck = 4;

template <bool NARROW>
struct EnumShared {
    using Word = typename std::conditional<NARROW, uint64_t, W128>::type;
    static constexpr int kQueue = NARROW ? kEnumQueue : kEnumQueueWide;
    EnumJob jobs[kMaxEnumJobs];
    JobView views[kMaxEnumJobs];
    unsigned long long visited[kMaxEnumJobs];  // necklaces, by job
    Word q_word[8][kQueue];                    // per warp: queued candidates and their jobs
    Word pool_w[8][32], pool_end[8][32];       // per warp: windows taken and not begun
    int64_t pool_win[8][32];
    uint8_t q_job[8][kQueue], pool_p[8][32], pool_job[8][32];
};

template <int MINB, bool NARROW>
__global__ void __launch_bounds__(256, MINB) enumerate_kernel(EnumArgs a) {
    __shared__ EnumShared<NARROW> sh;
    constexpr int kQueue = EnumShared<NARROW>::kQueue, kFlushAt = kQueue - 32;
    if (threadIdx.x < a.njobs) {
        sh.jobs[threadIdx.x] = a.jobs[threadIdx.x];
        sh.views[threadIdx.x] = job_view(sh.jobs[threadIdx.x]);
    }
    if (threadIdx.x < kMaxEnumJobs) sh.visited[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wq = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    // the same in every lane of the warp:
    int qlen = 0;             // queued candidates
    uint32_t full_jobs = 0;   // jobs seen at their soft capacity
    int pool = 0;             // windows in the pool
    bool open = true;         // windows may be left at the counter
    bool parked = false;      // (per lane) a window was left
    auto put = [](W128 v) {
        if constexpr (NARROW)
            return v.lo;
        else
            return v;
    };
    auto get = [](auto v) {
        if constexpr (NARROW)
            return W128{v, 0};
        else
            return v;
    };
    auto before = [](W128 x, W128 y) { return NARROW ? x.lo < y.lo : lt(x, y); };

    // writes the warp's queue out
    auto flush = [&]() {
        __syncwarp();
        uint32_t present = 0;  // jobs in the queue, one nearly always
        for (int e = lane; e < qlen; e += 32) present |= 1u << sh.q_job[wq][e];
        present = __reduce_or_sync(0xFFFFFFFFu, present);
        while (present) {
            const int jb = __ffs(present) - 1;
            present &= present - 1u;
            const EnumJob& J = sh.jobs[jb];
            unsigned mine = 0;
            for (int e = lane; e < qlen; e += 32) mine += sh.q_job[wq][e] == jb;
            const unsigned count = __reduce_add_sync(0xFFFFFFFFu, mine);
            unsigned long long pos = 0;
            if (lane == 0) pos = atomicAdd(J.count, (unsigned long long)count);
            pos = __shfl_sync(0xFFFFFFFFu, pos, 0);
            if ((int64_t)(pos + count) >= J.soft_cap) full_jobs |= 1u << jb;
            for (int base = 0; base < qlen; base += 32) {
                const int e = base + lane;
                const bool has = e < qlen && sh.q_job[wq][e] == jb;
                const uint32_t hm = __ballot_sync(0xFFFFFFFFu, has);
                const unsigned long long at = pos + __popc(hm & lt_mask);
                pos += __popc(hm);
                if (!has) continue;
                if ((int64_t)at < J.cap) {
                    const W128 word = get(sh.q_word[wq][e]);
                    J.words[at] = to_u4(word);
                    const int sum = NARROW ? digit_sum64(word.lo, sh.views[jb]) : digit_sum(word, sh.views[jb]);
                    J.out_roles[at] = __ldg(a.roles + jb * (kMaxDigitSum + 1) + sum);
                } else {
                    atomicCAS(a.status, 0, GP_KSTATUS_OVERFLOW);
                }
            }
        }
        qlen = 0;
        __syncwarp();
    };

    // takes windows into the (empty) pool: about as many as leave some for the
    // other warps
    int64_t taken = 0;  // of the counter's windows, as last seen
    auto refill = [&]() {
        if (full_jobs == a.win_jobs) {  // nothing more to visit this time
            parked = true;
            open = false;
            return;
        }
        int64_t n = (a.nwin - taken) / ((int64_t)gridDim.x * 8);
        n = n < 1 ? 1 : n > 32 ? 32 : n;
        long long w0 = 0;
        if (lane == 0) w0 = (long long)atomicAdd(a.next_win, (unsigned long long)n);
        w0 = __shfl_sync(0xFFFFFFFFu, w0, 0);
        taken = w0 + n;
        open = taken < a.nwin;
        const int64_t win = w0 + lane;
        bool ok = lane < n && win < a.nwin, full = false;
        int job = 0, p = 0;
        W128 w{}, end{};
        if (ok) {
            const uint4 c4 = a.cur[win], e4 = a.end[win];
            job = a.win_job[win];
            w = from_u4(c4);
            end = from_u4(e4);
            ok = lt(w, end);  // else finished
            full = ok && (((full_jobs >> job) & 1u) || job_full(sh.jobs[job]));
            if (full) {
                parked = true;  // untouched: it keeps its position
                ok = false;
            }
            if (ok) {
                const JobView& v = sh.views[job];
                if constexpr (NARROW)
                    p = first_prenecklace64(w.lo, v);
                else
                    p = first_prenecklace(w, v.b, v.L);
                ok = before(w, end);
                if (!ok) a.cur[win] = e4;  // no prenecklace in it
            }
        }
        // (a warp that went on through windows it may not begin, on its own,
        // would hold up the launch by milliseconds)
        full_jobs |= __reduce_or_sync(0xFFFFFFFFu, full ? 1u << job : 0u);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
        if (ok) {
            const int e = __popc(m & lt_mask);
            sh.pool_w[wq][e] = put(w);
            sh.pool_end[wq][e] = put(end);
            sh.pool_win[wq][e] = win;
            sh.pool_p[wq][e] = (uint8_t)p;
            sh.pool_job[wq][e] = (uint8_t)job;
        }
        pool = __popc(m);
        __syncwarp();
    };

    W128 w = {0, 0}, end = {0, 0};
    int64_t win = 0;
    int job = 0, p = 0;
    bool have = false;                 // w is a prenecklace to process, of window win
    unsigned long long necklaces = 0;  // of job `job`
    unsigned long long seen = 0;       // a count of the lane's job
    int seen_job = -1;
    for (int step = 1;; ++step) {
        // windows for idle lanes
        for (uint32_t idle; (idle = __ballot_sync(0xFFFFFFFFu, !have)) != 0 && (pool || open);) {
            if (!pool) refill();
            const int r = __popc(idle & lt_mask);
            if (!have && r < pool) {
                const int e = pool - 1 - r;
                const int nj = sh.pool_job[wq][e];
                if ((full_jobs >> nj) & 1u) {
                    parked = true;
                } else {
                    if (nj != job && necklaces) {
                        atomicAdd(&sh.visited[job], necklaces);
                        necklaces = 0;
                    }
                    job = nj;
                    w = get(sh.pool_w[wq][e]);
                    end = get(sh.pool_end[wq][e]);
                    win = sh.pool_win[wq][e];
                    p = sh.pool_p[wq][e];
                    have = true;
                }
            }
            pool = pool > __popc(idle) ? pool - __popc(idle) : 0;
            __syncwarp();
        }
        if (!__any_sync(0xFFFFFFFFu, have)) break;
        // One step takes the prenecklace w and the words after it that differ
        // from it in the last t digits only, x (t as the job's table has it,
        // L >= 2 t or t = 1).  Let a_0 a_1 .. be w's first digits.
        //  * A word with a larger x is a prenecklace iff no tail of x that is
        //    shorter than x is less than the a_0 a_1 .. of its length: tails
        //    that begin before x hold because w is one.
        //  * Its period is L, and it is a necklace, iff no such tail equals
        //    a_0 a_1 ..; else its period L - m, m < t the tail's length, does
        //    not divide L, as L > 2 m.
        //  * w itself is a necklace iff its period p divides L.
        // After the block comes FKM's successor of the word with the largest x,
        // every digit the maximum, which is a prenecklace too.
        W128 w0 = w;
        uint64_t cmask = 0;  // bit x: that word is a candidate
        if (have) {
            const EnumJob& J = sh.jobs[job];
            const JobView& v = sh.views[job];
            const uint32_t x0 = (uint32_t)w.lo & v.block;
            w0.lo = w.lo & ~(uint64_t)v.block;
            const uint32_t a0 = (uint32_t)(NARROW ? w.lo >> v.lead_shift : shr(w, v.lead_shift).lo);
            uint64_t in = J.strict[a0] & (~1ull << x0);
            bool done = false;
            if ((NARROW || end.hi == w.hi) && ((end.lo ^ w.lo) & ~(uint64_t)v.block) == 0) {
                in &= (1ull << ((uint32_t)end.lo & v.block)) - 1ull;  // the window ends here
                done = true;
            }
            if (divides_L(v, p)) in |= 1ull << x0;
            necklaces += (unsigned long long)__popcll(in);
            const int sum = (NARROW || v.narrow) ? digit_sum64(w0.lo, v) : digit_sum(w0, v);
            cmask = in & __ldg(J.cand + sum);
            if (!done) {
                w.lo = w0.lo | (v.maxpat.lo & v.block);
                if (NARROW || v.narrow) {
                    uint64_t wl = w.lo;
                    p = fkm_next64(wl, v);
                    w.lo = wl;
                } else {
                    p = fkm_next(w, v);
                }
                done = p == 0 || !before(w, end);
            }
            if (done) a.cur[win] = a.end[win];
            have = !done;
        }
        // the block's candidates into the queue, each lane's behind those of
        // the lanes before it; written out from kFlushAt on
        while (__any_sync(0xFFFFFFFFu, cmask != 0)) {
            const int n = __popcll(cmask);
            int to = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xFFFFFFFFu, to, o);
                if (lane >= o) to += y;
            }
            const int total = __shfl_sync(0xFFFFFFFFu, to, 31);
            for (int slot = qlen + to - n; cmask && slot < kQueue; ++slot) {
                W128 cand = w0;
                cand.lo |= (uint64_t)(__ffsll((long long)cmask) - 1);
                cmask &= cmask - 1ull;
                sh.q_word[wq][slot] = put(cand);
                sh.q_job[wq][slot] = (uint8_t)job;
            }
            qlen = qlen + total < kQueue ? qlen + total : kQueue;
            if (qlen >= kFlushAt) flush();
        }
        if ((step & (kCapCheck - 1)) == 0) {
            const bool met = have && seen_job == job && (int64_t)seen >= sh.jobs[job].soft_cap;
            full_jobs |= __reduce_or_sync(0xFFFFFFFFu, met ? 1u << job : 0u);
            if (have) {
                seen = *reinterpret_cast<volatile unsigned long long*>(sh.jobs[job].count);
                seen_job = job;
            }
        }
        // leave a window whose job has met its soft capacity
        if (have && ((full_jobs >> job) & 1u)) {
            a.cur[win] = to_u4(w);
            have = false;
            parked = true;
        }
    }
    flush();
    if (parked) *a.incomplete = 1;
    for (int j = 0; j < a.njobs; ++j) {
        unsigned long long v = job == j ? necklaces : 0ull;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
        if (lane == 0 && v) atomicAdd(&sh.visited[j], v);
    }
    __syncthreads();
    if (threadIdx.x < a.njobs && sh.visited[threadIdx.x]) atomicAdd(sh.jobs[threadIdx.x].necklaces, sh.visited[threadIdx.x]);
}

using u128d = unsigned __int128;

__device__ __forceinline__ u128d u128_of(U128p v) { return ((u128d)v.hi << 64) | v.lo; }

// Packed word of the word with rank r: the rank's base-k digits, by 32-bit
// pieces while it is longer than 64 bits.
__device__ __forceinline__ W128 word_of_rank(u128d r, const WinJobs::Job& j) {
    W128 w = {0, 0};
    const uint64_t k = (uint64_t)j.k;
    uint64_t lo = (uint64_t)r, hi = (uint64_t)(r >> 64);
    for (int q = 0; q < j.L; ++q) {
        uint64_t d;
        if (hi) {
            uint64_t piece[4] = {hi >> 32, hi & 0xFFFFFFFFull, lo >> 32, lo & 0xFFFFFFFFull};
            d = 0;
            for (int i = 0; i < 4; ++i) {
                const uint64_t x = (d << 32) | piece[i];
                piece[i] = x / k;
                d = x - piece[i] * k;
            }
            hi = (piece[0] << 32) | piece[1];
            lo = (piece[2] << 32) | piece[3];
        } else {
            const uint64_t x = lo / k;
            d = lo - x * k;
            lo = x;
        }
        w = bor(w, shl({d, 0}, j.b * q));
    }
    return w;
}

// A thread per window: two rank conversions, 33 us for 311,000 windows
// (2.5 to 3.5 ms on host threads, and their copy).
__global__ void window_words_kernel(WinJobs jobs, const WinRange* ranges, int64_t nranges, int64_t nwin, uint4* cur,
                                    uint4* end, uint8_t* win_job) {
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nwin; w += (int64_t)gridDim.x * blockDim.x) {
        int64_t a = 0, z = nranges;  // the last range whose first window is w or before
        while (z - a > 1) {
            const int64_t m = (a + z) / 2;
            if (ranges[m].first <= w)
                a = m;
            else
                z = m;
        }
        const WinRange& r = ranges[a];
        const WinJobs::Job& j = jobs.job[r.job];
        const u128d size = u128_of(r.wsize), last = u128_of(r.r1);
        const u128d lo = u128_of(r.r0) + (u128d)(w - r.first) * size;
        const u128d hi = last - lo > size ? lo + size : last;
        cur[w] = to_u4(word_of_rank(lo, j));
        end[w] = hi >= u128_of(j.space) ? to_u4(w128(j.past)) : to_u4(word_of_rank(hi, j));
        win_job[w] = (uint8_t)r.job;
    }
}

template <bool NARROW>
cudaError_t launch_enumerate_t(const EnumArgs& a, int num_sms, cudaStream_t st, int variant) {
    // one wave of resident blocks: windows are handed out dynamically
    static int resident[3] = {0, 0, 0};
    const int vi = variant == 1 ? 1 : variant == 2 ? 2 : 0;
    int& per_sm = resident[vi];
    if (per_sm == 0) {
        cudaError_t e = vi == 1   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<6, NARROW>, 256, 0)
                        : vi == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<5, NARROW>, 256, 0)
                                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<4, NARROW>, 256, 0);
        if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    }
    int64_t blocks = (a.nwin + 255) / 256;
    const int64_t maxb = (int64_t)num_sms * per_sm;
    if (blocks > maxb) blocks = maxb;
    if (vi == 1)
        enumerate_kernel<6, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    else if (vi == 2)
        enumerate_kernel<5, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    else
        enumerate_kernel<4, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_windows(const WinJobs& jobs, const WinRange* ranges, int64_t nranges, int64_t nwin, uint4* cur,
                           uint4* end, uint8_t* win_job, cudaStream_t st) {
    if (nwin <= 0 || nranges <= 0) return cudaSuccess;
    const int64_t blocks = (nwin + 255) / 256;
    window_words_kernel<<<(unsigned)(blocks < 65536 ? blocks : 65536), 256, 0, st>>>(jobs, ranges, nranges, nwin, cur,
                                                                                     end, win_job);
    return cudaGetLastError();
}

cudaError_t launch_enumerate(const EnumArgs& a, int num_sms, cudaStream_t st, int variant) {
    if (a.nwin <= 0) return cudaSuccess;
    if (a.njobs < 1 || a.njobs > kMaxEnumJobs) return cudaErrorInvalidValue;
    return a.narrow ? launch_enumerate_t<true>(a, num_sms, st, variant)
                    : launch_enumerate_t<false>(a, num_sms, st, variant);
}

}  // namespace gp
