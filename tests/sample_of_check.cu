// Prints "ok" when FastDiv (az_render.h) and sample_of (az_wave.cuh) give what plain 64-bit division gives: host code
// only, built and run by tests/test_sample_order.py.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "az_wave.cuh"

using namespace az;

static uint64_t rng_state = 0x9E3779B97F4A7C15ull;
static uint64_t rng() {   // xorshift64* (Vigna, "An experimental exploration of Marsaglia's xorshift generators", 2016)
    rng_state ^= rng_state >> 12;
    rng_state ^= rng_state << 25;
    rng_state ^= rng_state >> 27;
    return rng_state * 2685821657736338717ull;
}

static int fail(const char *what, uint64_t a, uint64_t b) {
    printf("%s: %llu %llu\n", what, (unsigned long long)a, (unsigned long long)b);
    return 1;
}

static int check_divisor(uint32_t d) {
    FastDiv f;
    f.set(d);
    std::vector<uint32_t> n = {0u, 1u, 2u, d - 1u, d, d + 1u, 0x7FFFFFFFu, 0x80000000u, 0xFFFFFFFEu, 0xFFFFFFFFu};
    for (int i = 0; i < 300; i++) {
        const uint32_t r = (uint32_t)rng(), k = r / d;
        for (uint32_t v : {r, r >> (i & 31), k * d, k * d - 1u, k * d + (d - 1u)}) n.push_back(v);
    }
    for (uint32_t v : n)
        if (f.quotient(v) != v / d) return fail("quotient", v, d);
    return 0;
}

static int check_samples(uint32_t wsc, uint32_t hsc, uint32_t root) {
    CameraParams cam{};
    cam.r0 = 3;
    cam.c0 = 5;
    cam.wsc = wsc;
    cam.hsc = hsc;
    cam.npix = (uint64_t)wsc * hsc;
    cam.sqrt_spp = root;
    cam.by_npix.set((uint32_t)cam.npix);
    cam.by_wsc.set(wsc);
    cam.by_sqrt.set(root);
    const uint64_t all = cam.npix * root * root, edge = (uint64_t)1 << 32;
    std::vector<uint64_t> s = {0, 1, cam.npix - 1, cam.npix, all - 1};
    for (int64_t k = -3; k <= 3; k++) s.push_back(edge + k);
    for (int i = 0; i < 2000; i++) s.push_back(rng() % all);
    for (uint64_t v : s) {
        if (v >= all) continue;
        uint32_t row, col, sx, sy;
        sample_of(cam, v, row, col, sx, sy);
        const uint64_t pix = v % cam.npix, k = v / cam.npix;
        if (row != 3 + pix / wsc || col != 5 + pix % wsc || sx != k % root || sy != k / root) return fail("sample", v, all);
    }
    return 0;
}

int main() {
    for (uint32_t d = 1; d <= 300; d++)
        if (check_divisor(d)) return 1;
    for (int b = 8; b < 32; b++)
        for (uint32_t d : {(1u << b) - 1u, 1u << b, (1u << b) + 1u})
            if (check_divisor(d)) return 1;
    for (uint32_t d : {1920u * 1080u, 65535u * 65535u, 0xFFFFFFFEu, 0xFFFFFFFFu})
        if (check_divisor(d)) return 1;
    for (int i = 0; i < 2000; i++)
        if (check_divisor((uint32_t)rng() >> (i & 31) | 1u)) return 1;
    const uint32_t sizes[][3] = {{1, 1, 1}, {1, 1, 255}, {97, 61, 2}, {13, 1, 3}, {1920, 1080, 46}, {1919, 1079, 64},
                                 {65535, 65535, 1}, {65535, 65535, 2}, {65535, 32771, 7}, {1, 65535, 300}};
    for (const auto &z : sizes)
        if (check_samples(z[0], z[1], z[2])) return 1;
    printf("ok\n");
    return 0;
}
