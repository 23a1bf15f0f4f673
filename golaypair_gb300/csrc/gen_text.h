// gen_text.h -- the generation stage's records as text, made on the device
// (gen_text.cu).
#pragma once
#include <cstdint>
#include <memory>

#include <cuda_runtime.h>

struct gp_ctx;

namespace gp {

// Lines of the A records, then of the B records, each in word order.
struct GenText {
    std::shared_ptr<char[]> p;  // null: not made
    size_t bytes_a = 0, bytes = 0;
    int64_t n_a = 0, n = 0;
};

struct GenRecords {  // device
    const uint4* words;
    const uint8_t* role;    // 1: A
    const uint16_t* sig;    // L - 1 each
    int64_t n;
    int L, b;
    int alpha[16];
};

// Leaves out.p null where the text needs more than 32-bit offsets or the
// device has no room for it; returns a GP code.
int records_to_text(gp_ctx* c, const GenRecords& r, GenText& out, cudaStream_t s);

}  // namespace gp
