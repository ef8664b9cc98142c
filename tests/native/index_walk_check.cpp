// index_walk over counts near 2^32: a walk ends after the entries that are its own.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <initializer_list>

#include "../../cumf_sgd_gb300/csrc/index_walk.h"

using u64 = unsigned long long;

static void check(u64 first, u64 step, u64 count) {
    const u64 own = first < count ? (count - first + step - 1) / step : 0;
    u64 visits = 0, at = first;
    bool in_order = true;
    cumf::index_walk((uint32_t)first, (uint32_t)step, (uint32_t)count, [&](u64 i) {
        in_order &= i == at;
        at += step;
        if (++visits > own) {
            printf("step %llu, count %llu: the walk from %llu does not end\n", step, count, first);
            exit(1);
        }
    });
    if (visits != own || !in_order) {
        printf("step %llu, count %llu, from %llu: %llu visits for %llu\n", step, count, first, visits, own);
        exit(1);
    }
}

int main() {
    const u64 grid = 152 * 64 * 256, last = 0xfffffffeull;  // threads of the largest grid, largest count
    for (u64 count : {last, last - 1, last + 2 - grid, last + 3 - grid, grid + 1, grid, grid - 1, 1ull, 0ull})
        for (u64 first : {0ull, 1ull, last % grid - 1, last % grid, grid - 1}) check(first, grid, count);
    for (u64 count : {last, last + 2 - 32, last + 3 - 32, 33ull, 32ull, 31ull})
        for (u64 first : {0ull, 29ull, 30ull, 31ull}) check(first, 32, count);
    printf("bad 0\n");
    return 0;
}
