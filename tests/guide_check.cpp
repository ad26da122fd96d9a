// The sampling guide tables against their definition, record by record: {lo, hi, cdf[lo], cdf[lo + 1]} with lo
// the first entry that reaches (j - 1/2) / G (n - 1 at most) and hi the lo of record j + 2.
#include "scene_host.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

static uint32_t bits(float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
}

static int check(const std::vector<float> &cdf, const char *what) {
    const uint32_t n = (uint32_t)cdf.size(), G = wobgb::guide_records(n);
    const std::vector<uint32_t> rec = wobgb::build_guide(cdf);
    if (rec.size() != 4 * (size_t)G) return std::printf("%s n %u: %zu words\n", what, n, rec.size()), 1;
    std::vector<uint32_t> first(G + 2, n - 1);
    uint32_t i = 0;
    for (uint32_t j = 0; j < G; j++) {
        while (i + 1 < n && (double)cdf[i] < ((double)j - 0.5) / (double)G) i++;
        first[j] = i;
    }
    for (uint32_t j = 0; j < G; j++) {
        const uint32_t want[4] = {first[j], first[j + 2], bits(cdf[first[j]]), bits(cdf[std::min(first[j] + 1, n - 1)])};
        if (std::memcmp(want, &rec[4 * (size_t)j], sizeof want)) return std::printf("%s n %u record %u\n", what, n, j), 1;
    }
    return 0;
}

int main() {
    int bad = 0;
    for (uint32_t n : {1u, 2u, 3u, 7u, 64u, 1000u, 5120u, 70001u, 262144u, 262145u, 1100000u}) {
        std::mt19937 g(n);
        std::uniform_real_distribution<double> u(0.0, 1.0);
        for (int kind = 0; kind < 5; kind++) {
            std::vector<float> c(n);
            std::vector<double> w(n);
            for (uint32_t i = 0; i < n; i++)
                w[i] = kind == 0 ? 1.0 : kind == 1 ? u(g) : kind == 2 ? std::pow(u(g), 30.0)
                     : kind == 3 ? (u(g) < 0.01 ? 1.0 : 0.0) : (i == n / 2 ? 1e6 : 1e-3);  // even, spread, steep, plateaus, a step
            double t = 0.0;
            for (double x : w) t += x;
            if (!(t > 0.0)) w[0] = t = 1.0;
            double run = 0.0;
            for (uint32_t i = 0; i < n; i++) c[i] = (float)((run += w[i]) / t);
            bad += check(c, "random");
        }
        // entries on the thresholds themselves and next to them
        const uint32_t G = wobgb::guide_records(n);
        std::vector<float> c(n);
        for (uint32_t i = 0; i < n; i++) {
            const float at = (float)(((double)(uint32_t)((double)i * G / n) - 0.5) / (double)G);
            c[i] = i % 3 == 0 ? at : std::nextafter(at, i % 3 == 1 ? 2.0f : -2.0f);
            if (i && c[i] < c[i - 1]) c[i] = c[i - 1];
        }
        bad += check(c, "thresholds");
    }
    std::printf("%d bad\n", bad);
    return bad != 0;
}
