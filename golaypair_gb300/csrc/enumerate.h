// enumerate.h -- arguments of the rank-window necklace enumerator.
//
// One launch enumerates the windows of up to kMaxEnumJobs jobs (orders /
// compressions of different lengths): every window carries its job, and each
// job has its own digit layout, row-sum table and output buffer.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "gp_internal.h"

namespace gp {

constexpr int kMaxDigitSum = 1023;
constexpr int kMaxEnumJobs = 8;
// Candidates a warp queues in shared memory (written out from 32 less on): 64-bit
// words, and wider ones (static shared memory stays under 48 KB).  Queues of 128,
// 192, 288 and 352: 16.4, 14.5, 13.5 and 13.2 ms of a five-order batch.
constexpr int kEnumQueue = 352, kEnumQueueWide = 192;

struct U128p {
    uint64_t lo, hi;
};

struct EnumJob {
    int L;                     // sequence length
    int b;                     // bits per digit
    U128p maxpat;              // digit k-1 at every position
    U128p plane[4];            // bit t of every digit
    uint4* words;              // out: candidate words
    uint8_t* out_roles;        // out: role bits per candidate
    unsigned long long* count; // out: candidates appended
    int64_t cap;               // hard capacity of words / out_roles
    int64_t soft_cap;          // stop when count reaches this
    unsigned long long* necklaces;  // out: necklaces visited
    // Blocks of words that differ in their last t digits x (b t <= 6 bits):
    int t;
    uint64_t strict[32];       // [first t - 1 digits]: x whose shorter tails all exceed them
    const uint64_t* cand;      // device, [sum of the other digits]: x with a digit sum that has a role
};

// t, and fills strict.
inline int enum_block(int k, int b, int L, uint64_t strict[32]) {
    const int t = L >= 2 * (6 / b) ? 6 / b : 1;
    for (uint32_t a = 0; a < 32; ++a) {
        strict[a] = 0;
        if (a >> (b * (t - 1))) continue;
        for (uint32_t x = 0; x < (1u << (b * t)); ++x) {
            bool in = true;
            for (int i = 0; i < t; ++i) in = in && (int)((x >> (b * i)) & ((1u << b) - 1u)) < k;
            for (int n = 1; n < t; ++n)  // tails of n digits
                in = in && (x & ((1u << (b * n)) - 1u)) > (a >> (b * (t - 1 - n)));
            if (in) strict[a] |= 1ull << x;
        }
    }
    return t;
}

// cand[s], s = 0 .. n - 1: bit x where s + the digit sum of x has a role
// (roles of digit sums 0 .. n - 1; none beyond); the largest number of bits set
// in one entry.
inline int enum_cand(int b, int t, const uint8_t* roles, int n, uint64_t* cand) {
    int most = 0;
    for (int s = 0; s < n; ++s) {
        cand[s] = 0;
        int bits = 0;
        for (uint32_t x = 0; x < (1u << (b * t)); ++x) {
            int d = s;
            for (int i = 0; i < t; ++i) d += (int)((x >> (b * i)) & ((1u << b) - 1u));
            if (d < n && roles[d]) {
                cand[s] |= 1ull << x;
                ++bits;
            }
        }
        most = bits > most ? bits : most;
    }
    return most;
}

struct EnumArgs {
    const EnumJob* jobs;       // device array of njobs jobs
    int njobs;
    const uint8_t* roles;      // [njobs][kMaxDigitSum+1]: bit0 = A row sum, bit1 = B row sum
    uint4* cur;                // per window: next word to visit (updated on exit)
    const uint4* end;          // per window: first word past the window
    const uint8_t* win_job;    // per window: its job
    uint32_t win_jobs;         // the jobs that have windows here, a bit each
    int64_t nwin;
    unsigned long long* next_win;  // window handout counter (zero before the launch)
    int* incomplete;           // out: 1 if some window is unfinished
    int* status;
    int narrow;                // 1: every job's word fits 63 bits (b * L <= 63): the 64-bit kernel
};

// The windows of a range of word ranks [r0, r1): wsize words each, the last
// one shorter; windows first, first + 1, ...
struct WinRange {
    U128p r0, r1, wsize;
    int64_t first;
    int64_t job;
};

struct WinJobs {
    struct Job {
        int k, b, L;
        U128p space, past;  // k^L; the number after the last word
    } job[kMaxEnumJobs];
};

// cur, end, win_job of windows 0 .. nwin - 1 (ranges: device, by first).
cudaError_t launch_windows(const WinJobs& jobs, const WinRange* ranges, int64_t nranges, int64_t nwin, uint4* cur,
                           uint4* end, uint8_t* win_job, cudaStream_t st);

// variant: 256-thread blocks per SM, 0: 4 (64 registers), 1: 6 (40), 2: 5 (48)
cudaError_t launch_enumerate(const EnumArgs& a, int num_sms, cudaStream_t st, int variant = 0);

}  // namespace gp
