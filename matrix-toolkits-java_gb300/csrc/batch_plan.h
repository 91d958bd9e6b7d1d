// batch_plan.h -- how a batch's systems are handed to teams of CTAs
// (batch.cu).  Host only.
#pragma once

#include <algorithm>
#include <cstdint>
#include <functional>
#include <queue>
#include <vector>

namespace mtjg {

constexpr int kTeamSizes = 4;  // teams of 8, 4, 2 and 1 CTAs

// resident CTAs per SM the batched CG is compiled for (its register cap).
// Measured on GB300 (C4, FP64 / mixed): 3 (80 registers) 168.5 / 115.7 ms;
// 4 (64 registers) 200.9 / 128.0 ms; 5: 238.6 / 152.8 ms -- the rows a
// thread keeps in flight matter more than resident warps.
#ifndef MTJG_BATCH_MINB
#define MTJG_BATCH_MINB 3
#endif
constexpr int kBatchPerSm = MTJG_BATCH_MINB;

// CTAs of a system's team, as log2.  A share of 2048 rows or more is worth
// the team's three barriers and rank-order sums per iteration (about 6000
// cycles against 27,000 of FP64 work for 2048 rows of 19 entries).
inline int batch_team(int64_t rows) { return rows >= 16384 ? 3 : rows >= 8192 ? 2 : rows >= 4096 ? 1 : 0; }

// Puts the systems of each team size together, largest teams first, each
// keeping its order; counts[c]: systems of teams of 8 >> c CTAs.
inline void batch_teams(const int *sys_rows, std::vector<int> &order, int *counts)
{
    std::vector<int> by[kTeamSizes];
    for (int s : order) by[kTeamSizes - 1 - batch_team((int64_t)sys_rows[s + 1] - sys_rows[s])].push_back(s);
    order.clear();
    for (int c = 0; c < kTeamSizes; ++c) {
        counts[c] = (int)by[c].size();
        order.insert(order.end(), by[c].begin(), by[c].end());
    }
}

// Rows that `teams` teams at work at once get through, one after the other,
// until all systems of `order` (taken in that order) are done.
inline int64_t batch_makespan(const int *sys_rows, const int *order, int count, int64_t teams)
{
    std::priority_queue<int64_t, std::vector<int64_t>, std::greater<int64_t>> end;
    int64_t last = 0;
    for (int k = 0; k < count; ++k) {
        int64_t t = (int64_t)sys_rows[order[k] + 1] - sys_rows[order[k]];
        if ((int64_t)end.size() >= teams) {
            t += end.top();
            end.pop();
        }
        end.push(t);
        last = std::max(last, t);
    }
    return last;
}

// CTAs per SM of a launch that has the GPU to itself.  The CTAs of an SM
// share its FP64 pipe, so a round of teams takes as many times its rows as
// there are CTAs on an SM, and the last round takes that long however few
// systems are left for it.  Three a SM are best where there are many rounds;
// two where they need (almost) as many rounds as three: 300 systems of 6000
// rows of 19 entries are two rounds by 228 teams of two and two by 152.
// Measured, FP64, one CTA a system / three a SM / two, in ms (a butterfly per
// warp in the reductions): 300 such systems 5.51 / 7.86 / 5.66; 300 of 4200 rows
// 3.92 / 5.26 / 4.20; 250 of 7000 rows 6.32 / 8.47 / 6.49; 250 2D Poisson grids
// 90^2 31.8 / 36.8 / 30.3; 60 grids 129^2 69.9 / 27.6 / 24.4.  Where two a SM need
// more rounds: 1200 systems of 4200 rows 14.5 / 15.8 / 16.1, 300 of 17000 rows
// 16.3 / 17.7 / 20.0.
inline int batch_per_sm(const int *sys_rows, const int *order, int count, int team, int num_sms)
{
    const int64_t three = (int64_t)kBatchPerSm * num_sms / team, two = (int64_t)2 * num_sms / team;
    if (team == 1 || count <= two) return kBatchPerSm;
    const int64_t t3 = kBatchPerSm * batch_makespan(sys_rows, order, count, three);
    const int64_t t2 = 2 * batch_makespan(sys_rows, order, count, two);
    return t2 * 5 <= t3 * 4 ? 2 : kBatchPerSm;
}

}  // namespace mtjg
