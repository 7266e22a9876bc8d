// Drives the bookkeeping of deferred pairs (bie_fix64.cuh) on the host: rows x
// slices of pairs, some share of them deferred, in the order of a random
// interleaving.  Prints whether every deferred pair is either in the list once or
// gone through again, whether the counter is bounded by the list's length and one
// per (row, slice), and the final count.  Arguments: seed, rows, slices, pairs per
// slice, capacity, percentage deferred.
#include "bie_fix64.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include <utility>
#include <vector>

using namespace bie::fix64;

int main(int argc, char **argv) {
    if (argc < 7) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    const int rows = std::atoi(argv[2]), slices = std::atoi(argv[3]), per = std::atoi(argv[4]);
    const u64 cap = (u64)std::atoll(argv[5]);
    const int percent = std::atoi(argv[6]), lanes = rows * slices;
    u64 counter = 0;
    std::vector<std::pair<int, int>> list(cap, {-1, -1});
    std::vector<int> over((size_t)lanes, kNoOverflow), at((size_t)lanes, 0);
    std::vector<std::vector<int>> deferred((size_t)lanes);
    bool ok = true;
    std::vector<int> open;
    for (int l = 0; l < lanes; ++l) open.push_back(l);
    while (!open.empty()) {   // one pair of a random lane at a time
        const size_t j = gen() % open.size();
        const int l = open[j], s = l % slices, pe = s * per + at[l];
        if ((int)(gen() % 100) < percent) {
            deferred[l].push_back(pe);
            u64 slot = 0;
            if (defer_slot([&] { return counter++; }, cap, pe, over[l], slot)) {
                ok = ok && slot < cap && list[slot].first < 0;
                if (slot < cap) list[slot] = {l / slices, pe};
            }
        }
        if (++at[l] == per) {
            open[j] = open.back();
            open.pop_back();
        }
    }
    std::set<std::pair<int, int>> done;
    for (const auto &p : list)
        if (p.first >= 0) ok = ok && done.insert(p).second;
    if (counter > cap)   // the correction kernel's second part
        for (int l = 0; l < lanes; ++l)
            for (int pe : deferred[l])
                if (over[l] != kNoOverflow && pe >= over[l]) ok = ok && done.insert({l / slices, pe}).second;
    size_t total = 0;
    for (const auto &d : deferred) total += d.size();
    std::printf("%d %d %llu\n", ok && done.size() == total ? 1 : 0, counter <= cap + (u64)lanes ? 1 : 0,
                (unsigned long long)counter);
    return 0;
}
