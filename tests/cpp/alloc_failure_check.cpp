// An entry point that looks a large array through on several host threads, with one of the calling
// thread's allocations failing: the call still finds the non-finite value at the end of the array.
// Prints the status codes, one per failing allocation.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <new>
#include <thread>
#include <vector>

#include "drifter_b200.h"

static thread_local int fail_in = -1;  // the allocation that fails, counted from here (-1: none)

void *operator new(std::size_t n) {
    if (fail_in >= 0 && fail_in-- == 0) throw std::bad_alloc();
    if (void *p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
    drf_bz_grid_desc g{};
    g.nx = g.ny = 725;  // 8.4 million samples
    g.Lx = g.Ly = 1e3;
    g.lambda = 1.0;
    std::vector<double> a((size_t)g.nx * g.ny * 16, 1.0);
    a.back() = std::numeric_limits<double>::infinity();
    // the list of threads, then one allocation per thread
    const int nt = (int)std::min(8u, std::max(1u, std::thread::hardware_concurrency()));
    for (int k = -1; k < (nt > 1 ? nt : 0); ++k) {
        fail_in = k;
        drf_bz *h = nullptr;
        const int rc = drf_bz_create(&g, a.data(), &h);
        fail_in = -1;
        std::printf("%d\n", rc);
    }
}
