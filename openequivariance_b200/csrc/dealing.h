// How long the busiest of `workers` takes when units of work are dealt to them in turn: unit u, of cost part[u % n] + each, goes to
// worker u % workers.  A worker's costs repeat after at most n of its units, and how many units it has and which it starts with
// depends on its number only through its remainder by n and on which side of the last round's end it lies: no loop over units.
// (The choice of a cut looks at up to 31 cuts, on every call whose number of tiles is new: dealing 4,700 units one by one
// took 61 to 210 us.)
#pragma once

#include <algorithm>
#include <numeric>
#include <vector>

inline double busiest_load(long long units, int n, const double* part, double each, int workers) {
    const long long rounds = units / workers;
    const int rest = (int)(units % workers), period = n / std::gcd(n, workers);
    auto load = [&](int first, long long count) {   // `count` units from unit `first` on, `workers` apart
        double cycle = 0, tail = 0;
        for (int i = 0, at = first % n; i < period; ++i, at = (at + workers) % n) {
            if (i == count % period) tail = cycle;
            cycle += part[at] + each;
        }
        return count / period * cycle + tail;
    };
    double most = 0;
    for (int r = 0; r < std::min(n, rest); ++r) most = std::max(most, load(r, rounds + 1));
    for (int r = rest; rounds > 0 && r < std::min(rest + n, workers); ++r) most = std::max(most, load(r, rounds));
    return most;
}

// How a list of pieces of work is cut into parts, a piece never being cut: for S parts the boundaries that make the costliest part cheapest.
constexpr int kMaxParts = 16;
struct Cuts {
    std::vector<double> cost;                     // of every piece
    int n[kMaxParts + 1] = {0};                   // parts that S asks for (fewer where fewer are as good)
    int cut[kMaxParts + 1][kMaxParts + 1] = {{0}};
    double part[kMaxParts + 1][kMaxParts] = {{0}};
};
inline void cut_into_parts(Cuts& c) {
    const int G = (int)c.cost.size();
    double total = 0, big = 0;
    for (double v : c.cost) { total += v; big = std::max(big, v); }
    for (int S = 1; S <= kMaxParts; ++S) {
        double lo = big, hi = total + 1;
        auto fill = [&](double cap, bool keep) {
            int parts = 0;
            for (int g = 0; g < G;) {
                if (parts == S) return false;
                double sum = 0;
                if (keep) c.cut[S][parts] = g;
                do sum += c.cost[g++]; while (g < G && sum + c.cost[g] <= cap);
                if (keep) { c.part[S][parts] = sum; c.cut[S][parts + 1] = g; }
                ++parts;
            }
            if (keep) c.n[S] = parts;
            return true;
        };
        for (int it = 0; it < 24; ++it) (fill((lo + hi) / 2, false) ? hi : lo) = (lo + hi) / 2;
        fill(hi, true);
    }
}

// Parts for `tiles` tiles, and which of two lists of the same work is cut: whatever leaves the busiest worker least to do when units (a part of a tile)
// are dealt out in turn.  `each`: price of a unit beside its pieces; `extra`: price of having parts at all.
inline int best_parts(const Cuts* const lists[2], long long tiles, double each, double extra, int workers, int* list) {
    int best = 1;
    double best_time = 0;
    *list = 0;
    for (int l = 0; l < 2; ++l)
        for (int S = 1 + l; S <= kMaxParts; ++S) {
            if (lists[l]->n[S] != S) continue;    // (of four equal pieces three parts are two: the next number of parts may still pay)
            const double t = busiest_load(tiles * S, S, lists[l]->part[S], each, workers) + (S > 1 ? extra : 0.0);
            if ((l == 0 && S == 1) || t < 0.95 * best_time) { best = S; *list = l; best_time = t; }
        }
    return best;
}
