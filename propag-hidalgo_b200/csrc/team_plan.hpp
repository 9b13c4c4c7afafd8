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

// CTAs of a group-mode team for a batch on `ctas` co-resident CTAs.  Jobs go to
// the teams largest first, each to the team that is free first, so the number
// of teams decides between many jobs at once on few CTAs each and few at once
// on many.  A job of s x s cells takes in the mean about 7.6 us x s on any team
// (its sweeps, each a chain of latencies) plus 0.229 us x s^2 / R on R CTAs, but
// jobs of one size differ widely (a fire dies early or crosses the grid), and
// with as many teams as jobs the batch waits for the longest one on its few
// CTAs.  So the batch is played through with durations from a tenth of the mean
// to 1.9 times it, spread evenly over the jobs (multiples of the golden ratio),
// and the number of teams that ends first is taken.  Measured on twelve batches
// of 5 to 256 members of 100^2 to 2048^2, three seeds each: 2.7 % above the best
// number of teams in the mean, 13 % with every job at its mean.  64 members of
// 1024^2: 128 / 132 / 159 ms in 16 teams of 9, 128 / 157 / 254 in 37 of 4; 24
// members: 63 / 58 / 54 in 12 of 12, 94 / 90 / 83 in 24 of 6; 256 members of 512^2
// keep 37 teams of 4 (106 / 94 / 119; 140 / 112 / 145 in 16 of 9).
// Where members are alike the longest is no longer than the others, and teams as
// small as the jobs allow would be a sixth faster (64 copies of one 1024^2
// scenario: 126 ms in 16 of 9, 108 in 37 of 4; 64 of 512^2: 59 and 52; 200 of
// 300^2: 49 and 41), which is less than they lose where members differ.
//
// side: the jobs' sides (square roots of their cells), in any order.
inline int team_size(std::vector<double> side, int ctas) {
  std::sort(side.begin(), side.end(), std::greater<double>());
  int best = ctas;
  double best_us = 0.0;
  for (int teams : {1, 2, 3, 4, 6, 8, 12, 16, 24, 37, 49, 74}) {
    if (teams > 1 && ((size_t)teams > side.size() || ctas / teams < 2)) break;
    const int R = ctas / teams;
    std::vector<double> ends((size_t)teams, 0.0);  // a min-heap of the teams' finishing times
    double turn = 0.0;
    for (double s : side) {
      turn += 0.618034;
      turn -= std::floor(turn);
      std::pop_heap(ends.begin(), ends.end(), std::greater<double>());
      ends.back() += (7.6 * s + 0.229 * s * s / R) * (0.1 + 1.8 * turn);
      std::push_heap(ends.begin(), ends.end(), std::greater<double>());
    }
    const double us = *std::max_element(ends.begin(), ends.end());
    if (teams == 1 || us < best_us) {
      best_us = us;
      best = R;
    }
  }
  return std::max(best, 2);
}

// Several teams on one job (WaveDev in engine.cuh): how many, and the window
// within which launches keep their sequence; no teams when the job has too few
// tiles to run any of them at once.  A window of one tile of at least 257
// cells, two of 129, three of 86 holds every reference of up to 256 cells'
// offset: the longest lines of sight of the hilly and ridged scenarios are 160
// to 218 steps, and a job with a longer one is run twice.  The number of teams
// is what a simulation of the schedule with measured sweep times favours (in
// sequence / 2 / 3 / 4 / 6 teams; 4096^2 with 20 ignitions: 478 / 265 / 208 / 186 /
// 212 ms; 2048^2 with 20: 103 / 58 / 53 / 59 / 71, with one: 49 / 33 / 35 / 37 /
// 45).
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
// the jobs differ from what team_size takes them to be (64 copies of one 1024^2
// scenario: 126 ms with its teams of 9, 108 with teams of 4); of those that split
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
