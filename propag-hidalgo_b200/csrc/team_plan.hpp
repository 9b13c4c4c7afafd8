// How a batch is split over the device: the size of group-mode teams, several
// teams on a lone job, and the group modes an autotuner tries.  Host code
// without a device, so that a test can go through the rules.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <functional>
#include <vector>

#include "engine.cuh"

namespace propag {

// When the last of the jobs (sides, largest first) ends in `teams` teams of the
// CTAs, us: jobs go to the teams largest first, each to the team that is free
// first.  A job of s x s cells takes in the mean about 7.6 us x s on any team (its
// sweeps, each a chain of latencies) plus 0.229 us x s^2 / R on R CTAs; differ:
// times 2.25 u^1.25, the u spread evenly over (0, 1) (multiples of the golden
// ratio): mean 1, a quarter of the jobs below 0.4, the longest 2.2.
inline double batch_us(const std::vector<double> &side, int teams, int ctas, bool differ) {
  const int R = ctas / teams;
  std::vector<double> ends((size_t)teams, 0.0);  // a min-heap of the teams' finishing times
  double turn = 0.0;
  for (double s : side) {
    turn += 0.618034;
    turn -= std::floor(turn);
    std::pop_heap(ends.begin(), ends.end(), std::greater<double>());
    ends.back() += (7.6 * s + 0.229 * s * s / R) * (differ ? 2.25 * turn * std::sqrt(std::sqrt(turn)) : 1.0);
    std::push_heap(ends.begin(), ends.end(), std::greater<double>());
  }
  return *std::max_element(ends.begin(), ends.end());
}

// CTAs of a group-mode team for a batch on `ctas` co-resident CTAs; side: the
// jobs' sides (square roots of their cells), in any order.
//
// The number of teams decides between many jobs at once on few CTAs each and few
// at once on many.  Where jobs of one size take unequal time (a fire dies early or
// crosses the grid; the members of a weather ensemble do) fewer teams than jobs
// win: with a team per job the batch waits for its longest job on that job's few
// CTAs.  Where they take the same time, a team per job wins, and every number that
// does not divide the jobs into full rounds loses most.  Nothing tells the two
// apart before the run, so both are played through for the numbers that make
// full rounds (and a few small ones, for a batch of a few large jobs and many
// small ones), and the number is taken whose larger loss is the smallest, with
// 1.3 times the loss allowed where the jobs are alike, the rarer case.
//
// Measured, against the best number of teams: twelve batches of 5 to 256 ensemble
// members and unrelated scenarios (three seeds) 1.03; 32 sizes of ensembles of 5 to
// 50 members of 150^2 to 1024^2 (four seeds) 1.02, at most 1.10; the same with
// copies of one member 1.26, at most 1.77.  (56 sizes, 5 to 40 members of 80^2 to
// 668^2, five seeds: 1.03, at most 1.36 for 34 members of 139^2; copies 1.08, at
// most 1.71.)  The rule before, the number that ends
// first when the jobs differ, of 1, 2, 3, 4, 6, 8, 12, 16, 24, 37, 49 and 74 teams:
// 1.03, 1.12 (at most 1.55) and 1.64 (at most 1.90); a team per job up to 37: 1.41,
// 1.20 (1.78) and 1.02.  20 members of 400^2: 12.9 ms in 10 teams, 15.6 in 20;
// copies of one: 6.7 and 4.5 (7.7 in 16).  propag_autotune tries a team per job.
inline int team_size(std::vector<double> side, int ctas) {
  std::sort(side.begin(), side.end(), std::greater<double>());
  const int n = (int)std::min<size_t>(side.size(), 1u << 30), most = std::max(ctas / 2, 1);
  std::vector<int> counts;
  for (int t : {1, 2, 3, 4, 6})
    if (t <= n && t <= most) counts.push_back(t);
  const int k0 = std::max(1, (n + most - 1) / most);  // the fewest rounds
  for (int k = k0; k < k0 + 8 && k <= n; ++k) counts.push_back((n + k - 1) / k);
  std::sort(counts.begin(), counts.end());
  counts.erase(std::unique(counts.begin(), counts.end()), counts.end());
  std::vector<double> alike, differ;
  for (int t : counts) {
    alike.push_back(batch_us(side, t, ctas, false));
    differ.push_back(batch_us(side, t, ctas, true));
  }
  const double alike_best = *std::min_element(alike.begin(), alike.end());
  const double differ_best = *std::min_element(differ.begin(), differ.end());
  int best = ctas;
  double best_loss = 0.0, best_alike = 0.0;
  for (size_t i = 0; i < counts.size(); ++i) {
    const double loss = std::max(alike[i] / alike_best / 1.3, differ[i] / differ_best);
    if (i == 0 || loss < best_loss || (loss == best_loss && alike[i] < best_alike)) {
      best_loss = loss;
      best_alike = alike[i];
      best = ctas / counts[i];
    }
  }
  return std::max(best, 2);
}

// Several teams on one job (WaveDev in engine.cuh): how many, and the window
// within which launches keep their sequence; no teams when the job has too few
// tiles to run any of them at once.  A window of one tile of at least 257
// cells, two of 129, three of 86 holds every reference of up to 256 cells'
// offset: the longest lines of sight of the hilly and ridged scenarios are 160
// to 218 steps, and a job with a longer one is begun again in sequence.  The
// number of teams is what a simulation of the schedule with the sweep times
// measured then favoured (in sequence / 2 / 3 / 4 / 6 teams; 4096^2 with 20
// ignitions: 478 / 265 / 208 / 186 / 212 ms; 2048^2 with 20: 103 / 58 / 53 / 59 / 71,
// with one: 49 / 33 / 35 / 37 / 45).
//
// Measured, in sequence on all CTAs against these teams: ridged 4096^2 with 20
// ignitions (three seeds) 364 / 378 / 434 and 158 / 167 / 181 ms, hilly 2048^2 with
// 20: 184 and 98, 1024^2 with one: 14.1 and 13.8.  On constant ground, where lines
// of sight grow as wide as the fire, the run is begun twice: 1024^2 with one
// ignition 121 and 137 ms, stopped after 7200 s 8.9 and 16.6, 2048^2 803 and 821.
struct WavePlan {
  uint32_t teams = 0;
  int window = 0;
};
inline WavePlan wave_plan(uint32_t width, uint32_t height, int T, uint32_t n_ignitions) {
  WavePlan p;
  const uint32_t TX = (width + T - 1) / T, TY = (height + T - 1) / T;
  const uint64_t tiles = (uint64_t)TX * TY;
  const int window = T >= 257 ? 1 : T >= 129 ? 2 : 3;
  if (T < 86 || tiles > kWaveTiles || std::max(TX, TY) < 2u * window + 2u ||
      (uint64_t)width * height >= (1ull << 27))
    return p;
  p.window = window;
  p.teams = n_ignitions < 2 ? 2 : tiles >= 100 ? 4 : 3;
  return p;
}

// Teams (slots) and CTAs a team (group) of a batch in group mode on `ctas`
// co-resident CTAs: teams of at least `team` CTAs, as many as there are jobs at
// most, which share the CTAs evenly.
struct GroupSplit {
  uint32_t slots, group;
  bool operator==(const GroupSplit &o) const { return slots == o.slots && group == o.group; }
};
inline GroupSplit group_split(uint32_t n_jobs, int ctas, int team) {
  const uint32_t slots = std::min<uint32_t>(n_jobs, (uint32_t)std::max(1, ctas / team));
  return GroupSplit{slots, (uint32_t)ctas / slots};
}

// The group modes (PropagOptions.cluster) an autotuner times for a batch: the
// automatic one (0), a team per job, and teams of 24, 16, 8 and 4 CTAs, in case
// the jobs differ from what team_size takes them to be (20 copies of one 400^2
// scenario: 6.7 ms with its 10 teams, 4.5 with 20); of those that split
// the CTAs alike, one.  auto_team: the automatic team size, 0 when the automatic
// mode is another one (clusters, or several teams on a lone job).
inline std::vector<int> autotune_groups(uint32_t n_jobs, int ctas, int auto_team) {
  std::vector<int> modes{0};
  std::vector<GroupSplit> listed;
  if (auto_team > 0) listed.push_back(group_split(n_jobs, ctas, auto_team));
  const int own = n_jobs <= (uint32_t)ctas ? ctas / (int)n_jobs : 0;
  for (int team : {own, 24, 16, 8, 4}) {
    if (team < 2 || team > ctas) continue;
    const GroupSplit g = group_split(n_jobs, ctas, team);
    if (std::find(listed.begin(), listed.end(), g) != listed.end()) continue;
    listed.push_back(g);
    modes.push_back(-team);
  }
  return modes;
}

}  // namespace propag
