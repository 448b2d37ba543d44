// Planes per CTA of a launch whose CTAs march in z.
#ifndef LGD_Z_CHUNKS_H
#define LGD_Z_CHUNKS_H

namespace lgd {

// Over xy tiles per plane, the planes of a chunk with the least waves of
// resident CTAs times planes per CTA (its chunk and halo planes), chunks of at
// least min_chunk planes; that product into *planes (or null).  Per number of
// waves the most chunks are best, and more waves only add halo planes, so a few
// waves beyond the fewest suffice: a grid of thousands of planes is planned at
// each launch as fast as a small one (trying every split took 12 us per launch at
// 5000 planes, and finds at most 1% less).
inline int least_planes(long long xy, int nz, long long resident, int halo, double *planes, int min_chunk = 2)
{
    const long long cap = nz / min_chunk > 1 ? nz / min_chunk : 1;
    const long long fewest = (xy + resident - 1) / resident;
    int best_chunk = nz;
    double best = 1e300;
    for (long long w = fewest; w < fewest + 64; ++w) {
        const long long split = w * resident / xy < cap ? w * resident / xy : cap;
        const int chunk = (int)((nz + split - 1) / split);
        const long long waves = (xy * ((nz + chunk - 1) / chunk) + resident - 1) / resident;
        const double t = (double)waves * (chunk + halo);
        if (t < best * 0.999) {
            best = t;
            best_chunk = chunk;
        }
        if (split == cap) break;
    }
    if (planes) *planes = best;
    return best_chunk;
}

}  // namespace lgd

#endif
