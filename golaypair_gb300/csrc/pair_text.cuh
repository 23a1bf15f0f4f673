// pair_text.cuh -- numbers and lines as text on the device.  Pair lines: "%d "
// per entry of a, " ", "%d " per entry of b, newline (src/utils/io.cpp:75-95).
#pragma once
#include <cstdint>

namespace gp {

__device__ __forceinline__ int dec_digits(unsigned v) {
    int n = 1;
    while (v >= 10) {
        v /= 10;
        ++n;
    }
    return n;
}

// Writes v in decimal; returns the end.
__device__ __forceinline__ char* put_dec(char* o, unsigned v) {
    char tmp[10];
    int n = 0;
    do {
        tmp[n++] = (char)('0' + v % 10);
        v /= 10;
    } while (v);
    while (n) *o++ = tmp[--n];
    return o;
}

// Bytes of "%d ".
__device__ __forceinline__ int value_bytes(int v) {
    const int u = v < 0 ? -v : v;
    return (v < 0 ? 1 : 0) + (u >= 100 ? 3 : u >= 10 ? 2 : 1) + 1;
}

__device__ __forceinline__ int pair_line_bytes(const int8_t* a, const int8_t* b, int L) {
    int n = 2;
    for (int o = 0; o < L; ++o) n += value_bytes(a[o]) + value_bytes(b[o]);
    return n;
}

// The line of (a, b) at `line`, by a whole warp, 32 entries at a time.
__device__ __forceinline__ void put_pair_line(const int8_t* a, const int8_t* b, int L, char* line) {
    const int lane = threadIdx.x & 31, W = 2 * L;
    for (int o0 = 0; o0 < W; o0 += 32) {
        const int o = o0 + lane;
        const int v = o < L ? a[o] : o < W ? b[o - L] : 0;
        // the blank between the halves before entry L, the newline after the last
        const int mine = o < W ? value_bytes(v) + (o == L ? 1 : 0) + (o == W - 1 ? 1 : 0) : 0;
        int incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += y;
        }
        if (o < W) {
            char* q = line + incl - mine;
            if (o == L) *q++ = ' ';
            int u = v;
            if (v < 0) {
                *q++ = '-';
                u = -v;
            }
            if (u >= 100) *q++ = (char)('0' + u / 100);
            if (u >= 10) *q++ = (char)('0' + u / 10 % 10);
            *q++ = (char)('0' + u % 10);
            *q++ = ' ';
            if (o == W - 1) *q = '\n';
        }
        line += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
}

}  // namespace gp
