// Which offset mappings the kernels may tabulate in 32 bits.
#include <cstdio>

#include "ltg_host.hpp"

using ltg::SubDims;

static SubDims dims(int n, const int32_t *ext, const int64_t *s0, const int64_t *s1) {
    SubDims d;
    d.n = n;
    for (int i = 0; i < n; i++) { d.ext[i] = ext[i]; d.s0[i] = s0[i]; d.s1[i] = s1[i]; }
    return d;
}

static int fails = 0;
static void check(const char *what, const SubDims &d, bool second, int64_t span, bool fits) {
    if (d.span(second) == span && d.fits_i32(second) == fits) return;
    std::printf("%s: span %lld, fits %d\n", what, (long long)d.span(second), (int)d.fits_i32(second));
    fails++;
}

int main() {
    const int64_t one[] = {1}, none[] = {0};
    const int32_t k[] = {100};
    // a 3e7 x 100 block (24 GB) contracted over its outer dimension, every
    // stride within 32 bits, against one contracted over its inner dimension
    const int64_t outer[] = {30000000};
    check("outer", dims(1, k, outer, one), false, 2970000000ll, false);
    check("outer, other tensor", dims(1, k, outer, one), true, 99, true);
    check("outer as second", dims(1, k, one, outer), true, 2970000000ll, false);
    // two steps of 2^30 reach 2^31, one element below them they do not
    const int32_t three[] = {3};
    const int64_t half[] = {1ll << 30};
    check("2^31", dims(1, three, half, none), false, 1ll << 31, false);
    const int32_t mixed[] = {2, 1073741824};
    const int64_t ms[] = {1ll << 30, 1};
    check("2^31 - 1", dims(2, mixed, ms, ms), false, (1ll << 31) - 1, true);
    check("empty", dims(0, k, one, one), false, 0, true);
    std::puts(fails ? "failed" : "ok");
    return fails != 0;
}
