// Calls a generation entry point, or the text export (host only), while large host allocations fail: all from
// the first-th on, `count` of them.  Prints the return code.  Exits with 2
// when an exception crosses the C ABI, with 3 when one ends a thread.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <new>
#include <string>

#include <unistd.h>

#include "golaypair_gb300.h"

static std::atomic<bool> armed{false};
static std::atomic<long> seen{0};
static long fail_from = 0, fail_count = 0;

void* operator new(std::size_t n) {
    if (armed && n >= 100000) {
        const long k = seen++;
        if (k >= fail_from && k < fail_from + fail_count) throw std::bad_alloc();
    }
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main(int argc, char** argv) {
    if (argc != 5) return 1;
    const std::string entry = argv[1], dir = argv[2];
    fail_from = std::atol(argv[3]);
    fail_count = std::atol(argv[4]);
    std::set_terminate([] { _exit(3); });
    gp_ctx* c = nullptr;
    if (entry != "export" && gp_ctx_create(&c, 0) != GP_OK) return 1;
    const std::string a = dir + "/a", b = dir + "/b", a2 = dir + "/a2", b2 = dir + "/b2";
    int rc = 1;
    armed = true;
    try {
        if (entry == "generate") {
            rc = gp_generate(c, 45, 3, -2, 0, 1, a.c_str(), b.c_str(), nullptr);
        } else if (entry == "export") {
            rc = gp_export_text(nullptr, (dir + "/in").c_str(), a.c_str());
        } else if (entry == "window") {
            rc = gp_generate_window(c, 45, 3, -2, 0, 0, 0, 1u << 30, a.c_str(), b.c_str(), nullptr);
        } else {
            gp_gen_job jobs[2] = {};
            jobs[0].order = 45, jobs[1].order = 39;
            for (auto& j : jobs) j.compress = 3, j.paf = -2, j.end_lo = 1u << 30;
            jobs[0].path_a = a.c_str(), jobs[0].path_b = b.c_str();
            jobs[1].path_a = a2.c_str(), jobs[1].path_b = b2.c_str();
            rc = gp_generate_batch(c, jobs, 2, 0, nullptr, nullptr);
        }
    } catch (...) {
        _exit(2);
    }
    armed = false;
    std::printf("%d\n", rc);
    if (c) gp_ctx_destroy(c);
    return 0;
}
