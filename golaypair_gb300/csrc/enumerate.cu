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

// The layout of the job a thread is enumerating, held in registers.
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
// Digit sum of a word of a job, for its role.
__device__ __forceinline__ int word_sum(uint4 v, const EnumJob& j) {
    const W128 w = from_u4(v), ones = w128(j.plane[0]);
    int s = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (t < j.b) {
            const W128 m = band(w, shl(ones, t));
            s += (__popcll(m.lo) + __popcll(m.hi)) << t;
        }
    }
    return s;
}
__device__ __forceinline__ bool job_full(const EnumJob& j) {
    return (int64_t)*reinterpret_cast<volatile unsigned long long*>(j.count) >= j.soft_cap;
}

// Each thread takes windows from a global counter.  A window whose job
// has reached its soft capacity is left (position saved) and the thread goes
// on with its next window, so one full job does not idle the others.
// MINB = 3: 72 registers, no spills (3 CTAs of 256 per SM);
// MINB = 4: at most 64 registers (4 CTAs of 256 per SM); MINB = 8: capped
// at 32 registers for full occupancy (some spills).  The tuner picks.
//
// Candidates go to a per-warp queue in shared memory first; the warp writes
// them out when kFlushAt or more are queued, with one counter atomic per
// job present.  (An atomic per step, whose returned offset the whole warp waits
// for, made the kernel memory-latency bound.)  What the atomic returns tells
// the warp when a job has met its soft capacity.
//
// What bounds it: issue, of the steps where a word has few necklaces behind it
// and of the queue where many (windows of 2^32 words: order 57 9.4 ms, five
// orders 48 ms).
// A block of two digits, its rows taken one by one, needed four times
// the steps over an alphabet of four and longer ones: 15.1 and 87 ms.
constexpr int kFlushAt = kEnumQueue - 32;
constexpr int kQueue = kEnumQueue;  // per warp

// NARROW: every job's words fit 63 bits, so a word and its window end are
// 64-bit values (the high halves are zero and drop out of the registers).
template <int MINB, bool NARROW>
__global__ void __launch_bounds__(256, MINB) enumerate_kernel(EnumArgs a) {
    __shared__ uint8_t role_tab[kMaxEnumJobs][kMaxDigitSum + 1];
    __shared__ EnumJob jobs[kMaxEnumJobs];
    __shared__ uint4 q_word[8][kQueue];  // NARROW: the high half holds the job
    __shared__ uint8_t q_job[NARROW ? 1 : 8][NARROW ? 1 : kQueue];
    for (int i = threadIdx.x; i < a.njobs * (kMaxDigitSum + 1); i += blockDim.x)
        role_tab[i / (kMaxDigitSum + 1)][i % (kMaxDigitSum + 1)] = a.roles[i];
    if (threadIdx.x < a.njobs) jobs[threadIdx.x] = a.jobs[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wq = threadIdx.x >> 5;  // this warp's queue
    const uint32_t lt_mask = (1u << lane) - 1u;
    int qlen = 0;                     // queued candidates (the same in every lane)
    uint32_t full_jobs = 0;           // jobs whose count this warp has seen at the soft capacity
    // writes the warp's queue out (every lane of the warp calls it)
    auto flush = [&]() {
        __syncwarp();
        for (int base = 0; base < qlen; base += 32) {
            const int e = base + lane;
            const bool has = e < qlen;
            const uint32_t hm = __ballot_sync(0xFFFFFFFFu, has);
            uint32_t met = 0;
            if (has) {
                uint4 word = q_word[wq][e];
                int jb;
                if constexpr (NARROW) {
                    jb = (int)word.z;
                    word.z = 0;
                } else {
                    jb = q_job[wq][e];
                }
                const uint32_t grp = __match_any_sync(hm, jb);
                const int leader = __ffs(grp) - 1;
                const EnumJob& J = jobs[jb];
                unsigned long long pos0 = 0;
                if (lane == leader) pos0 = atomicAdd(J.count, (unsigned long long)__popc(grp));
                pos0 = __shfl_sync(grp, pos0, leader);
                if ((int64_t)pos0 + __popc(grp) >= J.soft_cap) met = 1u << jb;
                const unsigned long long pos = pos0 + __popc(grp & lt_mask);
                if ((int64_t)pos < J.cap) {
                    J.words[pos] = word;
                    J.out_roles[pos] = role_tab[jb][word_sum(word, J)];
                } else {
                    atomicCAS(a.status, 0, GP_KSTATUS_OVERFLOW);
                }
            }
            full_jobs |= __reduce_or_sync(0xFFFFFFFFu, met);
        }
        qlen = 0;
        __syncwarp();
    };
    // windows are handed out dynamically: a thread takes the next unvisited
    // one from a global counter when it needs work (long windows do not
    // hold up a statically assigned share)
    // The index of the window after the current one is fetched when the
    // current one starts, so the atomic's latency is hidden by its steps.
    int64_t pref = -1;
    auto take = [&]() -> int64_t {
        const int64_t w0 = pref >= 0 ? pref : (int64_t)atomicAdd(a.next_win, 1ull);
        pref = -1;
        return w0;
    };
    int64_t win = take();  // current window
    bool active = win < a.nwin;
    W128 w = {0, 0}, end = {0, 0};
    JobView jv{};
    int job = 0;
    int p = 0;
    bool have = false;  // w is a valid prenecklace to process
    bool parked_any = false;
    unsigned long long necklaces = 0;  // of job `job`, flushed when the job changes
    for (;;) {
        // (re)load a window when idle; skip windows whose job is full
        while (active && !have) {
            const int nj = a.win_job[win];
            if (nj != job && necklaces) {
                atomicAdd(jobs[job].necklaces, necklaces);
                necklaces = 0;
            }
            job = nj;
            if (job_full(jobs[job])) {
                parked_any = true;  // window untouched: it keeps its position
            } else {
                w = from_u4(a.cur[win]);
                end = from_u4(a.end[win]);
                if constexpr (NARROW) {
                    w.hi = 0;
                    end.hi = 0;
                }
                jv = job_view(jobs[job]);
                if (lt(w, end)) {
                    if constexpr (NARROW)
                        p = first_prenecklace64(w.lo, jv);
                    else
                        p = first_prenecklace(w, jv.b, jv.L);
                    have = lt(w, end);
                }
                if (have && pref < 0) pref = (int64_t)atomicAdd(a.next_win, 1ull);
                if (!have) a.cur[win] = a.end[win];  // window finished
            }
            if (!have) {
                win = take();
                active = win < a.nwin;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
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
        if (active) {
            const EnumJob& J = jobs[job];
            const uint32_t x0 = (uint32_t)w.lo & jv.block;
            w0.lo = w.lo & ~(uint64_t)jv.block;
            const uint32_t a0 = (uint32_t)(NARROW ? w.lo >> jv.lead_shift : shr(w, jv.lead_shift).lo);
            uint64_t in = J.strict[a0] & (~1ull << x0);
            bool done = false;
            if ((NARROW || end.hi == w.hi) && ((end.lo ^ w.lo) & ~(uint64_t)jv.block) == 0) {
                in &= (1ull << ((uint32_t)end.lo & jv.block)) - 1ull;  // the window ends here
                done = true;
            }
            if (divides_L(jv, p)) in |= 1ull << x0;
            necklaces += (unsigned long long)__popcll(in);
            const int sum = (NARROW || jv.narrow) ? digit_sum64(w0.lo, jv) : digit_sum(w0, jv);
            cmask = in & __ldg(J.cand + sum);
            if (!done) {
                w.lo = w0.lo | (jv.maxpat.lo & jv.block);
                if (NARROW || jv.narrow) {
                    uint64_t wl = w.lo;
                    p = fkm_next64(wl, jv);
                    w.lo = wl;
                } else {
                    p = fkm_next(w, jv);
                }
                done = p == 0 || !(NARROW ? w.lo < end.lo : lt(w, end));
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
                if constexpr (NARROW) {
                    cand.hi = (uint64_t)job;
                } else {
                    q_job[wq][slot] = (uint8_t)job;
                }
                q_word[wq][slot] = to_u4(cand);
            }
            qlen = qlen + total < kQueue ? qlen + total : kQueue;
            if (qlen >= kFlushAt) flush();
        }
        // leave a window whose job has met its soft capacity
        if (active && have && ((full_jobs >> job) & 1u)) {
            a.cur[win] = to_u4(w);
            have = false;
            parked_any = true;
        }
        if (active && !have) {
            win = take();
            active = win < a.nwin;
        }
    }
    flush();
    if (parked_any) *a.incomplete = 1;
    if (necklaces) atomicAdd(jobs[job].necklaces, necklaces);
}

template <bool NARROW>
cudaError_t launch_enumerate_t(const EnumArgs& a, int num_sms, cudaStream_t st, int variant) {
    // one wave of resident blocks: windows are handed out dynamically
    static int resident[3] = {0, 0, 0};
    const int vi = variant == 1 ? 1 : variant == 2 ? 2 : 0;
    int& per_sm = resident[vi];
    if (per_sm == 0) {
        cudaError_t e = vi == 1   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<8, NARROW>, 256, 0)
                        : vi == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<3, NARROW>, 256, 0)
                                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enumerate_kernel<4, NARROW>, 256, 0);
        if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    }
    int64_t blocks = (a.nwin + 255) / 256;
    const int64_t maxb = (int64_t)num_sms * per_sm;
    if (blocks > maxb) blocks = maxb;
    if (vi == 1)
        enumerate_kernel<8, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    else if (vi == 2)
        enumerate_kernel<3, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    else
        enumerate_kernel<4, NARROW><<<(unsigned)blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_enumerate(const EnumArgs& a, int num_sms, cudaStream_t st, int variant) {
    if (a.nwin <= 0) return cudaSuccess;
    if (a.njobs < 1 || a.njobs > kMaxEnumJobs) return cudaErrorInvalidValue;
    return a.narrow ? launch_enumerate_t<true>(a, num_sms, st, variant)
                    : launch_enumerate_t<false>(a, num_sms, st, variant);
}

}  // namespace gp
