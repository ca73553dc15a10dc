// How the plane-marching kernels cut axis 0 into chunks, one CTA each.
#pragma once

namespace gb {

// Planes a CTA marches through (1 .. n) so that the launch ends soonest.  A
// chunk of c planes costs step * c + extra (extra: planes it reads beyond its
// own); per_sm CTAs fit an SM, and each beside the first slows them all by
// `share`.  A launch that fits the GPU at once takes as long as its busiest
// SM; a longer one its number of waves, an unfinished one counted as `tail` of
// the way from its fill to a whole one.  Ties go to the longer chunk (less is
// read twice).
// share and tail are fitted to the times at every chunk length, 21 shapes from
// one 24^3 grid to 16 x 96^3 and 128 x 56^3, both boundaries: the rule's choice is
// on average 1 to 2 % behind the best chunk, halving the chunk until the
// launch had 2 to 8 CTAs an SM 5 to 30 %, waves x planes alone (share 0) 2 to
// 24 %.
inline int balance_planes(int n, int step, int extra, long long tiles, int per_sm,
                          double share, double tail) {
    const long long slots = 148ll * per_sm;
    double best = -1.0;
    int chunk = n;
    for (int k = 1; k <= n; k++) {
        const int c = (n + k - 1) / k;
        if (k > 1 && c == (n + k - 2) / (k - 1)) continue;
        const long long ctas = tiles * ((n + c - 1) / c);
        const double fill = (double)ctas / slots;
        const double waves = fill + tail * ((double)((ctas + slots - 1) / slots) - fill);
        const double time = ctas <= slots ? 1.0 + share * ((ctas + 147) / 148 - 1)
                                          : (1.0 + share * (per_sm - 1)) * waves;
        const double cost = (step * (double)c + extra) * time;
        if (best < 0.0 || cost < 0.999 * best) {
            best = cost;
            chunk = c;
        }
        if (ctas > 64 * slots) break;     // finer splits only read more
    }
    return chunk;
}

// The chunk halved until `tiles` column tiles make `target` CTAs, at least
// `least` planes.
inline int halve_planes(int n, int least, long long tiles, long long target) {
    int c = n;
    while (c > least && tiles * ((n + c - 1) / c) < target) c = (c + 1) / 2;
    return c;
}

}  // namespace gb
