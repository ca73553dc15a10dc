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

// The chunk halved until `tiles` column tiles make `target` CTAs, at least
// `least` planes.
inline int halve_planes(int n, int least, long long tiles, long long target) {
    int c = n;
    while (c > least && tiles * ((n + c - 1) / c) < target) c = (c + 1) / 2;
    return c;
}

}  // namespace gb
