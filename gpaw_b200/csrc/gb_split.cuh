// How the plane-marching kernels cut axis 0 into chunks, one CTA each.
#pragma once

namespace gb {

// Planes a CTA marches through (1 .. n) so that waves x planes is least: a
// chunk of c planes costs step * c + extra (extra: planes it reads beyond
// its own), `tiles` column tiles share `slots` CTAs that run at once.  Ties
// go to the longer chunk (less is read twice).
inline int split_planes(int n, int step, int extra, long long tiles, long long slots) {
    long long best = -1;
    int chunk = n;
    for (int k = 1; k <= n; k++) {
        const int c = (n + k - 1) / k;
        if (k > 1 && c == (n + k - 2) / (k - 1)) continue;
        const long long ctas = tiles * ((n + c - 1) / c);
        const long long cost = (ctas + slots - 1) / slots * (step * (long long)c + extra);
        if (best < 0 || cost < best) {
            best = cost;
            chunk = c;
        }
        if (ctas > 64 * slots) break;     // finer splits only read more
    }
    return chunk;
}

// Planes a CTA marches through (1 .. n) so that the launch ends soonest.  A
// chunk of c planes costs step * c + extra (extra: planes it reads beyond its
// own); per_sm CTAs fit an SM, and each beside the first slows them all by
// `share` (measured: 0.2 for the stencils, 0.25 to 0.4 for the transfers).  A
// launch that fits the GPU at once takes as long as its busiest SM; a longer
// one its number of waves, the last of them between its fill and a whole one.
// Ties go to the longer chunk (less is read twice).
inline int balance_planes(int n, int step, int extra, long long tiles, int per_sm,
                          double share) {
    const long long slots = 148ll * per_sm;
    double best = -1.0;
    int chunk = n;
    for (int k = 1; k <= n; k++) {
        const int c = (n + k - 1) / k;
        if (k > 1 && c == (n + k - 2) / (k - 1)) continue;
        const long long ctas = tiles * ((n + c - 1) / c);
        const double waves = (double)ctas / slots;
        const double time = ctas <= slots
                                ? 1.0 + share * ((ctas + 147) / 148 - 1)
                                : (1.0 + share * (per_sm - 1)) * 0.5 *
                                      (waves + (double)((ctas + slots - 1) / slots));
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
