// bt_plan.cpp -- which CTAs peel which graphs of a batched arena.
#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>

#include "bt_internal.h"

// A graph's peel is a chain of sub-rounds that does not get shorter with more
// CTAs (6.5 us each) beside the row positions walked and the edges scanned, which
// do.  Both are taken from the graph's butterflies B, which are counted before:
// about sqrt(B) sub-rounds, 0.017 us of one CTA per butterfly (4 positions,
// 1.5 to 10) and 0.027 per edge.  Measured sub-rounds against sqrt(B), and
// microseconds of one CTA beyond the chain against the estimate:
//   Chung-Lu, mean degree 8, 100k edges   1,798 / 2,128    77k / 80k
//   Chung-Lu of the bench, 400k           22,710 / 22,630  4.1M / 8.7M
//   hub-skewed, 500k                      21,301 / 26,186  20M / 12M
//   uniform, mean degree 8, 400k          3 / 34           11k / 11k
// Dense blocks have shorter chains than this (a uniform graph of density 1/4 and
// 100k edges 322 / 12,497, a hub-skewed one of 10k 120 / 3,071).  By the edges
// alone, with powers fitted to the first family, a 100k-edge hub graph
// beside ten uniform ones of 400k got the CTAs of a cheap one: 223 ms for the
// batch, and 39 one graph after the other.
double bt_peel_chain_us(const PeelJob &j) { return 6.5 * std::sqrt((double)j.butterflies); }
double bt_peel_walk_us(const PeelJob &j) { return 0.017 * (double)j.butterflies + 0.027 * (double)j.edges; }

// One graph takes all CTAs.  A batch is peeled by teams that take graphs one
// after another, in the order given.  Numbers of teams, with sizes in proportion to
// a power of their first graph's walk, are played through and the one that ends
// first is taken.  48 graphs of 1k to 100k edges: 23 ms, with the best equal sizes
// (8 or 9 CTAs) 26, as one chain of the union's sub-rounds 45.
std::vector<uint32_t> bt_plan_teams(const std::vector<PeelJob> &jobs, uint32_t ctas) {
    std::vector<uint32_t> best{ctas};
    if (jobs.size() < 2) return best;
    std::vector<double> chain, walk;
    for (const PeelJob &j : jobs) {
        chain.push_back(bt_peel_chain_us(j));
        walk.push_back(bt_peel_walk_us(j));
    }
    double best_us = 0;
    for (size_t q = 0; q < jobs.size(); q++) best_us += chain[q] + walk[q] / ctas;
    for (uint32_t teams = 2; teams <= ctas && teams <= jobs.size(); teams += std::max(1u, teams / 3)) {
        for (double power : {0.0, 0.5}) {
            std::vector<uint32_t> size(teams);
            double sum = 0;
            for (uint32_t t = 0; t < teams; t++) sum += std::pow(walk[t], power);
            uint32_t used = 0;
            for (uint32_t t = 0; t < teams; t++) {
                size[t] = std::max(1u, (uint32_t)(ctas * std::pow(walk[t], power) / sum));
                used += size[t];
            }
            for (uint32_t t = 0; used < ctas; t = (t + 1) % teams, used++) size[t]++;
            for (uint32_t t = 0; used > ctas; t = (t + 1) % teams)
                if (size[t] > 1) size[t]--, used--;
            std::priority_queue<std::pair<double, uint32_t>, std::vector<std::pair<double, uint32_t>>,
                                std::greater<std::pair<double, uint32_t>>> free_at;
            double last = 0;
            for (size_t q = 0; q < jobs.size() && (last < best_us); q++) {
                double at = 0;
                uint32_t t = (uint32_t)q;
                if (q >= teams) {
                    at = free_at.top().first;
                    t = free_at.top().second;
                    free_at.pop();
                }
                at += chain[q] + walk[q] / size[t];
                last = std::max(last, at);
                free_at.push({at, t});
            }
            if (last < best_us) {
                best_us = last;
                best = size;
            }
        }
    }
    return best;
}
