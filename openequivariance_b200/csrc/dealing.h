// How long the busiest of `workers` takes when units of work are dealt to them in turn: unit u, of cost part[u % n] + each, goes to
// worker u % workers.  A worker's costs repeat after at most n of its units, and how many units it has and which it starts with
// depends on its number only through its remainder by n and on which side of the last round's end it lies: no loop over units.
// (The choice of a cut looks at up to eight cuts, on every call whose number of tiles is new: dealing 4,700 units one by one
// took 61 to 210 us.)
#pragma once

#include <algorithm>
#include <numeric>

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
