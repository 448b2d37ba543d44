// least_planes (csrc/z_chunks.h) against every split, and its time at the largest grids.
#include <stdio.h>
#include <stdlib.h>

#include <chrono>
#include <random>

#include "z_chunks.h"

static double product(long long xy, int nz, long long resident, int halo, int chunk)
{
    return (double)((xy * ((nz + chunk - 1) / chunk) + resident - 1) / resident) * (chunk + halo);
}

int main()
{
    std::mt19937 rng(1);
    auto log_int = [&](double bits) { return (long long)std::exp2(std::uniform_real_distribution<double>(0, bits)(rng)); };
    for (int i = 0; i < 20000; ++i) {
        const long long xy = log_int(17), resident = 152 << rng() % 4;
        const int nz = (int)log_int(11), halo = 2 + rng() % 5, least = rng() % 2 ? 2 : 4;
        double planes = 0;
        const int chunk = lgd::least_planes(xy, nz, resident, halo, &planes, least);
        if (chunk < 1 || chunk > nz || (chunk < least && chunk < nz)) return 2;
        if (planes != product(xy, nz, resident, halo, chunk)) return 3;
        double best = 1e300;
        for (int split = 1; split <= (nz / least > 1 ? nz / least : 1); ++split) {
            const double t = product(xy, nz, resident, halo, (nz + split - 1) / split);
            if (t < best) best = t;
        }
        if (planes > 1.02 * best) return 4;
    }
    const auto t0 = std::chrono::steady_clock::now();
    long long sum = 0;
    for (int i = 0; i < 1000; ++i) sum += lgd::least_planes(1 + i % 7, 1 << 30, 152, 4, nullptr);
    const double us = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() * 1e3;
    if (us > 50 || sum == 0) return 5;         // microseconds per call; every split would take seconds
    puts("ok");
    return 0;
}
