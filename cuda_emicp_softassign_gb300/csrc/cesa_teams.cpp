// Which blocks of the launch run which of a batch's EM-ICP registrations
// (emicp_teams_kernel); host arithmetic. The blocks of a pair depend on the batch's
// sizes and schedules and on its own, not on where it stands, so that a pair's result
// does not either.
//
// A step of a registration on g blocks takes about lat(g) + M (N kTeamElemNs +
// kTeamRowNs) / g, an odd number of blocks above one kTeamOdd times as long for the
// division (no whole SMs, whose pairs of blocks split the sweep by pair_num): within 5%
// of 2000 x 2000, 4000 x 4000, 1000 x 3000 and 3000 x 1000 on 1 to 38 blocks, somewhat above 300 x
// 300. Two plans:
//   each    a team of its own for every pair that wants more than a block (plan_each);
//   packed  teams of one size take several pairs, one after the other (plan_packed),
//           looked at where there are more pairs than a quarter of the blocks, and taken
//           where it is modelled to save kPackedGain: pairs a few more than half of the
//           blocks, or than all of them, leave half of the chip idle with a team each,
//           and many uneven ones a sixth.
// ms, each -> packed (304 blocks): 160 pairs of 2000 x 2000 29.3 -> 20.8, 310 58.4 -> 42.5, 160 of 5000
// x 5000 161.9 -> 96.2, 120 80.5 -> 67.9, 500 of 500-4000 points 51.4 -> 45.6. In lock step over all
// pairs, as the Softassign pairs run what the series leaves, these took 18.8, 35.8, 105.1,
// 79.5 and 43.6 (with direct differences and poses that are not refined); 304 of 2000 x 2000
// 34.6, a team each 30.1.
#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "cesa_kernels.h"

namespace cesa {
namespace {

constexpr double kTeamElemNs = 0.093, kTeamRowNs = 12.0, kTeamOdd = 1.05;
constexpr double kTeamRounds[] = {1.0, 1.5, 2.0, 3.0, 4.0, 6.0, 8.0};
// Uneven pairs fill the teams' time as they are: with more shapes than this the first
// kTeamRoundsUneven of them are looked at.
constexpr int kTeamShapes = 16, kTeamRoundsUneven = 3;
constexpr double kTeamGrid = 1.1;  // t goes up by this until it can be kept, then is narrowed down

// A step's share by blocks g: lat, its barriers, completion and pose (one block alone
// does all of it itself), and div, what the work is multiplied with.
struct TeamModel {
  std::vector<double> lat, div;
  explicit TeamModel(int G) : lat((size_t)G + 1), div((size_t)G + 1) {
    for (int g = 1; g <= G; ++g) {
      lat[(size_t)g] = 12000.0 + 36000.0 * std::pow((double)g, -0.7);
      div[(size_t)g] = (g > 1 && g % 2 ? kTeamOdd : 1.0) / g;
    }
  }
};

struct TeamShape {  // registrations of one size and schedule
  double steps, work;
  int count, blocks;
  double own;  // time on `blocks` blocks
  double run(const TeamModel& m, int g) const { return steps * m.lat[(size_t)g] + work * m.div[(size_t)g]; }
  // the fewest blocks, up to `most`, that hold one to `slot`; false: none do
  bool fit(const TeamModel& m, double slot, int most) {
    const double left = slot - steps * m.lat[(size_t)most];
    if (left * most < work) return false;
    blocks = (int)(work / left);  // no fewer do
    if (blocks < 1) blocks = 1;
    while (blocks <= most && (own = run(m, blocks)) > slot) ++blocks;
    return blocks <= most;
  }
};

TeamShape shape_of(const EmTeamJob& J, int count) {
  const double steps = (double)J.nsteps;
  return TeamShape{steps, steps * (double)J.M * ((double)J.N * kTeamElemNs + kTeamRowNs), count, 1, 0.0};
}

// The teams for a time t, by shapes (the longest first): for every size of team what
// each has left of t (a heap), and each team's registrations, as places in the
// shapes' order. False where they want over G blocks.
struct TeamPacker {
  const TeamModel& model;
  std::vector<TeamShape>& shapes;
  int G;
  std::vector<std::vector<std::pair<double, int>>> left;  // by size: (time left, team)
  std::vector<double> sum;                                // by size
  std::vector<int> kinds;                                 // by size: shapes that want it
  std::vector<int> sizes;                                 // sizes that some shape wants
  std::vector<std::pair<int, std::vector<int>>> teams;    // (size, registrations)
  TeamPacker(const TeamModel& m, std::vector<TeamShape>& s, int g)
      : model(m), shapes(s), G(g), left((size_t)g + 1), sum((size_t)g + 1), kinds((size_t)g + 1) {}
  // the teams' times evenly divided, which any packing wants at least
  bool may(double t, double K) {
    for (int g : sizes) {
      sum[(size_t)g] = 0.0;
      kinds[(size_t)g] = 0;
      left[(size_t)g].clear();
    }
    sizes.clear();
    for (TeamShape& s : shapes) {
      if (!s.fit(model, t / K, G)) return false;
      const size_t g = (size_t)s.blocks;
      if (kinds[g]++ == 0) sizes.push_back(s.blocks);
      sum[g] += s.count * s.own;
    }
    double used = 0.0;
    for (int g : sizes) used += g * std::ceil(sum[(size_t)g] / t - 1e-9);
    return used <= G;
  }
  // build: with the teams' registrations, not only whether they fit
  bool pack(double t, double K, bool build) {
    if (!may(t, K)) return false;
    teams.clear();
    int used = 0, at = 0;
    for (const TeamShape& s : shapes) {
      if (!build && kinds[(size_t)s.blocks] == 1) {  // as many as fit, on every team
        const double each = std::floor(t / s.own * (1.0 - 1e-9));
        used += s.blocks * (int)std::ceil(s.count / (each < 1.0 ? 1.0 : each));
        if (used > G) return false;
        continue;
      }
      auto& h = left[(size_t)s.blocks];
      for (int c = 0; c < s.count; ++c, ++at) {
        if (!h.empty() && h.front().first >= s.own) {
          std::pop_heap(h.begin(), h.end());
          h.back().first -= s.own;
          if (build) teams[(size_t)h.back().second].second.push_back(at);
        } else {
          used += s.blocks;
          if (used > G) return false;
          h.emplace_back(t - s.own, (int)teams.size());
          if (build) teams.emplace_back(s.blocks, std::vector<int>{at});
        }
        std::push_heap(h.begin(), h.end());
      }
    }
    return true;
  }
};

TeamPlan plan_packed(const EmTeamJob* jobs, int n, int G, const TeamModel& model) {
  TeamPlan P;
  std::vector<std::pair<double, int>> key((size_t)n);  // the longest first, equal shapes together
  for (int i = 0; i < n; ++i) key[(size_t)i] = {shape_of(jobs[i], 1).run(model, 1), i};
  auto same = [&](int a, int b) {
    return jobs[a].N == jobs[b].N && jobs[a].M == jobs[b].M && jobs[a].nsteps == jobs[b].nsteps;
  };
  std::stable_sort(key.begin(), key.end(), [&](const auto& a, const auto& b) {
    if (a.first != b.first) return a.first > b.first;
    const EmTeamJob &x = jobs[a.second], &y = jobs[b.second];
    return x.nsteps != y.nsteps ? x.nsteps > y.nsteps : x.N != y.N ? x.N > y.N : x.M > y.M;
  });
  std::vector<TeamShape> shapes;
  double work = 0.0, all = 0.0, least = 0.0;
  for (int k = 0; k < n; ++k) {
    const int i = key[(size_t)k].second;
    if (k > 0 && same(i, key[(size_t)k - 1].second)) {
      shapes.back().count += 1;
    } else {
      shapes.push_back(shape_of(jobs[i], 1));
    }
    const TeamShape& s = shapes.back();
    work += s.work;
    all += s.run(model, 1);
    least = std::max(least, s.run(model, G));
  }
  TeamPacker T(model, shapes, G);
  const int nK = shapes.size() > kTeamShapes ? kTeamRoundsUneven : (int)(sizeof(kTeamRounds) / sizeof(double));
  double K = 1.0;
  auto keeps = [&](double t) {
    for (int k = 0; k < nK; ++k)
      if (T.pack(t, kTeamRounds[k], false)) {
        K = kTeamRounds[k];
        return true;
      }
    return false;
  };
  double t = std::max(least, work / G), lo = t;
  while (t < all && !keeps(t)) {
    lo = t;
    t *= kTeamGrid;
  }
  if (t >= all) {  // one block would take them all
    t = 1.0001 * all;
    K = 1.0;
  }
  for (int k = 0; k < 3; ++k) {
    const double mid = 0.5 * (lo + t);
    if (keeps(mid)) t = mid;
    else lo = mid;
  }
  while (!T.pack(t, K, true)) t *= 1.0001;  // (the count alone rounds differently at a whole number of runs)
  // even sizes (whole SMs), odd ones, single blocks
  auto rank = [](int g) { return g == 1 ? 2 : g % 2; };
  std::stable_sort(T.teams.begin(), T.teams.end(), [&](const auto& a, const auto& b) {
    return rank(a.first) != rank(b.first) ? rank(a.first) < rank(b.first) : a.first > b.first;
  });
  for (const auto& team : T.teams) {
    const int first = (int)P.order.size();
    for (int at : team.second) {
      P.order.push_back(key[(size_t)at].second);
      P.size.push_back(team.first);
    }
    for (int r = 0; r < team.first; ++r) P.blocks.push_back(TeamBlock{first, (int)team.second.size(), r, team.first});
  }
  P.time_ns = t;
  if ((int)P.blocks.size() < G) P.blocks.resize((size_t)G, TeamBlock{0, 0, 0, 0});  // the rest idle
  return P;
}

// For the least t that the blocks can keep, every registration that needs more than a
// block gets the fewest that hold it to t, and the others go to single blocks, as many
// on one as stay below t. The constants are a choice that serves batches of up to some
// 80 pairs best (40 mixed pairs of 500-20,000 points: 1-4% sooner than with the model
// above), not that model: teams of whole SMs are preferred. Those come first.
constexpr double kEachElemNs = 0.095, kEachRowNs = 30.0, kEachStepNs = 8000.0, kEachOdd = 1.2;

TeamPlan plan_each(const EmTeamJob* jobs, int n, int G) {
  TeamPlan P;
  std::vector<double> cost((size_t)n), need((size_t)n);  // need: time on one block
  P.order.resize((size_t)n);
  P.size.resize((size_t)n);
  double sum = 0.0;
  for (int i = 0; i < n; ++i) {
    const double steps = (double)jobs[i].nsteps;
    P.order[(size_t)i] = i;
    cost[(size_t)i] = steps * (double)jobs[i].M * ((double)jobs[i].N * kEachElemNs + kEachRowNs);
    need[(size_t)i] = kEachOdd * cost[(size_t)i] + steps * kEachStepNs;
  }
  std::stable_sort(P.order.begin(), P.order.end(), [&](int a, int b) { return need[(size_t)a] > need[(size_t)b]; });
  for (int j = 0; j < n; ++j) sum += need[(size_t)P.order[(size_t)j]];
  // sizes for a time t, and the blocks they take (more than G: not kept)
  auto fill = [&](double t) -> long {
    long used = 0;
    double left = 0.0;
    for (int j = 0; j < n && used <= G; ++j) {
      const size_t i = (size_t)P.order[(size_t)j];
      const double run = t - jobs[i].nsteps * kEachStepNs;
      int g = 1;
      if (need[i] > t) {
        const double e = run > 0.0 ? std::ceil(0.5 * cost[i] / run) * 2.0 : 2.0 * G;
        const double o = run > 0.0 ? std::ceil(kEachOdd * cost[i] / run) : 2.0 * G;
        g = (int)std::min(std::min(e, o), 2.0 * G);
        used += g;
      } else if (left >= need[i]) {
        left -= need[i];
      } else {
        left = t - need[i];
        used += 1;
      }
      P.size[(size_t)j] = g;
    }
    return used;
  };
  double lo = 0.0, hi = sum;  // all on one block
  for (int k = 0; k < 24; ++k) {
    const double t = 0.5 * (lo + hi);
    if (fill(t) <= G) hi = t;
    else lo = t;
  }
  fill(hi);
  for (int odd = 0; odd < 2; ++odd)
    for (int j = 0; j < n; ++j) {
      const int g = P.size[(size_t)j];
      if (g > 1 && (g & 1) == odd)
        for (int r = 0; r < g; ++r) P.blocks.push_back(TeamBlock{j, 1, r, g});
    }
  double left = -1.0;
  for (int j = 0; j < n; ++j) {  // single blocks: consecutive in the order
    if (P.size[(size_t)j] > 1) continue;
    const double w = need[(size_t)P.order[(size_t)j]];
    if (left >= w) {
      left -= w;
      P.blocks.back().njobs += 1;
    } else {
      left = hi - w;
      P.blocks.push_back(TeamBlock{j, 1, 0, 1});
    }
  }
  if ((int)P.blocks.size() < G) P.blocks.resize((size_t)G, TeamBlock{0, 0, 0, 0});  // the rest idle
  return P;
}

// The longest team's time by the model.
double modelled(const EmTeamJob* jobs, const TeamPlan& P, const TeamModel& model) {
  double most = 0.0;
  for (const TeamBlock& b : P.blocks) {
    if (b.njobs < 1 || b.rank > 0) continue;
    double t = 0.0;
    for (int k = 0; k < b.njobs; ++k) {
      const EmTeamJob& J = jobs[P.order[(size_t)(b.first + k)]];
      t += shape_of(J, 1).run(model, b.size);
    }
    most = std::max(most, t);
  }
  return most;
}

constexpr double kPackedGain = 0.92;

}  // namespace

TeamPlan plan_teams(const EmTeamJob* jobs, int n, int G) {
  const TeamModel model(G);
  TeamPlan P = plan_each(jobs, n, G);
  P.time_ns = modelled(jobs, P, model);
  if (4 * n <= G) return P;
  TeamPlan Q = plan_packed(jobs, n, G, model);
  return Q.time_ns < kPackedGain * P.time_ns ? Q : P;
}

}  // namespace cesa
