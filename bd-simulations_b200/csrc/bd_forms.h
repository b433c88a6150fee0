// Which form a step takes: rules on sizes, plain host code (no device calls;
// what the device holds comes in as numbers).
#pragma once

#include <algorithm>
#include <vector>

namespace bd {

// What the rules look at in a run.
struct FormRun {
  int N, Z;
  bool idgas;
  // work per CTA counts particles and a quarter of the mesh points
  double weight() const { return N + (idgas ? 0.0 : 0.25 * Z * Z); }
};

// Whether a call of nsteps steps of a single ideal-gas run (no mesh: sort and
// particle kernels only) takes the stage kernels from a graph. Measured, us per
// step (resident | stage kernels), particles, calls of many steps: 5000 11.0 |
// 12.8; 35 000 13.3 | 13.1; 60 000 12.9 | 13.5; 131 072 16.8 | 15.1; 500 000 32.1 |
// 29.5; adaptive dt: 60 000 16.7 | 18.0; 131 072 22.5 | 21.2; 500 000 48.0 | 45.5. A
// call per step, which pays the resident launch's start each time: 3000 12.4 |
// 14.4; 5000 14.4 | 14.7; 8000 15.9 | 14.4; 60 000 18.5 | 14.4; adaptive dt: 5000
// 31.5 | 36.8; 8000 37.6 | 35.3
inline bool idgas_stage_kernels(int N, long long nsteps) { return N > 65536 || (nsteps == 1 && N > 6000); }

// A batch's calls of several steps: launches per step (the pipelined or the
// stage kernels), one cluster of CTAs per run, or a group of CTAs of one
// cooperative grid per run.
enum BatchStep { BATCH_LAUNCHES, BATCH_CLUSTERS, BATCH_GROUPS };
struct BatchForm {
  BatchStep step = BATCH_LAUNCHES;
  std::vector<int> ctas;  // per run: CTAs of its cluster or group
};

// held(k, cs): clusters of cs CTAs for run k that the device holds at once (0:
// none). slots: CTAs to share out among groups (0: no groups). piped: the batch
// has the pipelined step.
template <class Held>
BatchForm choose_batch_form(const std::vector<FormRun>& runs, const Held& held, int slots, bool piped) {
  BatchForm out;
  const size_t n = runs.size();
  double particles = 0.0;
  for (const FormRun& r : runs) particles += r.N;
  // Clusters: every run on clusters of one size, the largest at which the
  // whole batch is resident at once; then larger clusters for runs that would
  // hold the others up, while there is room to spare (a batch that takes a mix
  // of cluster sizes fills the GPU less well: 0.8). The part of the GPU a
  // cluster takes comes from the device: clusters of 16 pack badly into GPCs.
  std::vector<int> clusters;
  double most_c = 0.0;
  auto part = [&](size_t k, int cs) {
    const int h = held(k, cs);
    return h > 0 ? 1.0 / h : 2.0;
  };
  for (int base = 16; base >= 1; base /= 2) {
    std::vector<int> cs(n, base);
    std::vector<double> used(n);
    double all = 0.0;
    for (size_t k = 0; k < n && all <= 1.0; k++) all += used[k] = part(k, base);
    if (all > 1.0) continue;
    auto load = [&](size_t k) { return runs[k].weight() / cs[k]; };
    size_t top = 0;
    for (;;) {
      for (size_t k = 0; k < n; k++)
        if (load(k) > load(top)) top = k;
      if (cs[top] >= 16) break;
      const double u = part(top, 2 * cs[top]);
      if (all + u - used[top] > 0.8) break;
      all += u - used[top];
      used[top] = u;
      cs[top] *= 2;
    }
    if (clusters.empty() || load(top) < 0.95 * most_c) {
      most_c = load(top);
      clusters = cs;
    }
  }
  // Groups: a CTA each, then a CTA at a time to the run with the largest load.
  std::vector<int> share;
  double most_g = 0.0;
  if (slots >= (int)n && n > 0) {
    share.assign(n, 1);
    auto top = [&]() {
      size_t t = 0;
      for (size_t k = 1; k < n; k++)
        if (runs[k].weight() / share[k] > runs[t].weight() / share[t]) t = k;
      return t;
    };
    for (int left = slots - (int)n; left > 0; left--) share[top()]++;
    const size_t t = top();
    most_g = runs[t].weight() / share[t];
  }
  // Estimates of a step in us, fitted to measurements of 1 to 128 runs of 1000
  // to 250 000 particles (clusters 12-60, groups 14-45, the pipelined step
  // 20-110; the stage kernels, 45-900, were never the fastest). A form that
  // does not fit is not compared.
  const double t_clusters = 8.0 + 0.025 * most_c, t_groups = 14.0 + 0.016 * most_g;
  double best = 19.0 + 8e-5 * particles;  // pipelined
  bool have = piped;
  auto consider = [&](BatchStep s, const std::vector<int>& ctas, double t) {
    if (ctas.empty() || (have && t > best)) return;
    have = true;
    best = t;
    out.step = s;
    out.ctas = ctas;
  };
  consider(BATCH_CLUSTERS, clusters, t_clusters);
  consider(BATCH_GROUPS, share, t_groups);
  return out;
}

}  // namespace bd
