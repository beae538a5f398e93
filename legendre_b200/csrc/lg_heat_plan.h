// How the marching heat kernel (lg_heat.cu) divides a grid.  Host code only.
#pragma once

#include <algorithm>
#include <cstdint>

namespace lg {

constexpr int kMaxPlanes = 256;  // planes a CTA marches over, at most

// Planes per CTA: of the heights that some number of chunks gives, the one
// whose waves of resident CTAs (`slots`) spend the fewest plane iterations, a
// CTA running zc + 2 halo planes plus about four iterations of start-up
// (address set-up and the first loads' latency).  It looks at no more than 2
// sqrt(planes) heights, 256 in all, and once a run: one chunk count after the
// other at every launch took 5 us on 1425 x 1001, where a launch takes 10.7,
// and 165 on 128 x 100000.
inline int march_planes(int64_t tiles, int64_t planes, int halo, int64_t slots) {
    int64_t best = -1;
    int best_zc = (int)std::min<int64_t>(planes, kMaxPlanes);
    for (int zc = best_zc; zc >= 1; --zc) {
        const int64_t chunks = (planes + zc - 1) / zc;
        zc = (int)((planes + chunks - 1) / chunks);  // the lowest height with as many chunks
        const int64_t ctas = tiles * chunks;
        const int64_t cost = (ctas + slots - 1) / slots * (zc + 2 * halo + 4);
        if (best < 0 || cost < best) {
            best = cost;
            best_zc = zc;
        }
        if (ctas > 64 * slots) break;  // many waves: the halo planes only add from here on
    }
    return best_zc;
}

// The length of a launch in which CTAs of `threads` threads with `rows` rows
// each march over zc planes: waves times iterations times an iteration's
// length, which grows with the rows that share the SM (a row and a half for
// each thread's first one) down to a latency of about a thousand of them.
// Forward Euler on cubes of 40^3 to 400^3 and on narrow grids (4 to 33 cells in
// one or two dimensions): the cheapest shape by this is the fastest one or
// within 4 %, 9 % at 4096 x 8 x 8; RungeKutta4 within 5 %.
inline double march_cost(int64_t tiles, int64_t planes, int zc, int halo, int64_t sms, int per_sm, int threads, int rows) {
    const int64_t ctas = tiles * ((planes + zc - 1) / zc), slots = sms * per_sm;
    const int64_t share = std::min<int64_t>(per_sm, (ctas + sms - 1) / sms);
    return (double)((ctas + slots - 1) / slots) * (zc + 2 * halo + 4) *
           std::max(1000.0, (double)share * threads * (rows + 0.5));
}

}  // namespace lg
