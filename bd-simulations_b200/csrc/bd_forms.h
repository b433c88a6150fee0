// Which form a step takes: rules on sizes, plain host code (no device calls;
// what the device holds comes in as numbers).
#pragma once

#include <algorithm>
#include <set>
#include <vector>

namespace bd {

// What the rules look at in a run.
struct FormRun {
  int N, Z;
  bool idgas;
  bool adaptive = false;
  // work per CTA counts particles and a quarter of the mesh points
  double weight() const { return N + (idgas ? 0.0 : 0.25 * Z * Z); }
  double points() const { return idgas ? 0.0 : (double)Z * Z; }
  bool pow2() const { return (Z & (Z - 1)) == 0; }
  // a power of two, or 3 * 2^k with transforms of its own in the resident step
  bool compiled() const { return pow2() || (Z >= 48 && Z % 3 == 0 && ((Z / 3) & (Z / 3 - 1)) == 0); }
};

// us per step of a batch in the stage kernels' launches, which wait for one set
// of transforms after another (a set for every power of two, one for all meshes
// with a factor 3) and for the deposit tile of most particles.
inline double estimate_launches(const std::vector<FormRun>& runs) {
  double n = 0.0, m2 = 0.0, m3 = 0.0, tile = 0.0;
  std::set<int> sides;
  bool adaptive = false, factor3 = false;
  for (const FormRun& r : runs) {
    n += r.N;
    adaptive = adaptive || r.adaptive;
    if (r.idgas) continue;
    (r.pow2() ? m2 : m3) += r.points();
    if (r.pow2()) sides.insert(r.Z);
    else factor3 = true;
    int mt = 4;
    for (int c : {64, 48, 32, 24, 16, 12, 8, 6})
      if (r.Z % c == 0) {
        mt = c;
        break;
      }
    const double side = std::max(1, r.Z / mt);
    tile = std::max(tile, r.N / (side * side));
  }
  if (m2 + m3 == 0.0) return 12.0 + (adaptive ? 6.0 : 0.0) + 3.7e-5 * n;
  return 10.0 + (adaptive ? 6.0 : 0.0) + 18.0 * (double)sides.size() + (factor3 ? 34.0 : 0.0) +
         (adaptive ? 1.4e-4 : 1.3e-4) * n + 2.3e-5 * m2 + 5.7e-5 * m3 + 1.9e-3 * tile;
}

// us per step of a batch without the pipelined step whose run k has ctas[k] CTAs,
// that of the run that takes longest: clusters (two CTAs per SM once there are
// more than SMs, which slow each other down) or groups (a CTA per SM, up to
// 2048 particles in its shared memory).
inline double estimate_resident(const std::vector<FormRun>& runs, const std::vector<int>& ctas, bool clusters, int sms) {
  double most = 0.0, all = 0.0;
  bool adaptive = false, mesh = false;
  for (size_t k = 0; k < runs.size(); k++) {
    const FormRun& r = runs[k];
    const double n = (double)r.N / ctas[k], m = r.points() / ctas[k];
    adaptive = adaptive || r.adaptive;
    mesh = mesh || !r.idgas;
    all += ctas[k];
    const double per_point = clusters ? (r.compiled() ? 0.0055 : 0.0171) : (r.compiled() ? 0.0056 : 0.0129);
    const double per_n = clusters ? (r.adaptive ? 0.0176 : 0.0089) : (r.adaptive ? 0.0144 : 0.0061);
    most = std::max(most, per_n * n + per_point * m + (clusters ? 0.0 : 0.0011 * std::max(0.0, n - 2048.0)));
  }
  if (!clusters) return (mesh ? 16.8 : 10.4) + (adaptive ? 1.4 : 0.0) + most;
  const double full = std::min(1.0, std::max(0.0, all / sms - 1.0));
  return (mesh ? 12.9 : 7.8) + (adaptive ? 1.2 : 0.0) + most * (1.0 + 0.56 * full);
}

// more than k particles to a mesh point
inline bool many_per_point(double n, double points, double k) { return n > k * points; }

// A single run that steps pipelined when asked for several steps (on a mesh
// beyond the resident step's, always). Measured, us per step, 128 steps a call
// (resident | pipelined | a launch per step), particles, mesh side:
// 131 072, 256 27.5 | 29.3 | 31.0; 131 072, 512 32.5 | 31.6 | 35.4; 262 144, 512
// 45.1 | 41.0 | 51.4; 524 288, 512 64.2 | 57.4 | 71.9; 131 072, 1024 60.5 | 49.3 |
// 51.6; 262 144, 1024 72.9 | 59.9 | 64.1; 900 000, 1024 122 | 105 | 116.
// Not with many particles to a mesh point: the blocks under way hold
// neighbouring cells, and the deposits of all of them meet on a few points; in
// a launch per step every CTA has a share of its own. 1 000 000, 128 (61 a point)
// 122 | 127 | 115; 3 000 000, 256 (46) 364 | 324 | 346; 3 000 000, 128 352 | 628 |
// 340; 1 000 000, 64 167 | 299 | 159 to 200; 3 000 000, 64 588 | 2202 | 532.
// 4096: the accumulator does not stay in L2 between the move and the rows, and
// from 262 144 particles on the stage kernels (second) are ahead of what they
// were before their transforms went through registers (third) where the
// pipelined step (first) is not: 64 000 444 | 411 | 461; 300 000 501 | 443 | 497;
// 1 000 000 600 | 489 | 572; 4 000 000 792 | 732 | 857.
inline bool pipelined_single(int N, int Z) {
  if (Z > 1024) return Z < 4096 || N < 262144;
  if (many_per_point(N, (double)Z * Z, 48)) return false;
  return (N >= 131072 && Z >= 512) || N >= 262144;
}

// A single run with the one-step kernel that takes it, a launch per step, for
// calls of several steps too (where they are not pipelined). 1024^2: four
// elements per thread of half the CTAs' threads are short of the transforms'
// work, the launches cost less (65 536 particles, us per step: 55.6 resident,
// 43.9 a launch each). Many particles to a mesh point: as above (64 000 particles,
// 16^2 76.9 | 68.2; 131 072, 64^2 33.0 | 31.4; 500 000, 64^2 93 | 78).
inline bool launch_per_step_single(int N, int Z) {
  return Z == 1024 || (N >= 50000 && many_per_point(N, (double)Z * Z, 24));
}

// The particle kernel's form (k_step, AHEAD): for runs of 131 072 particles and
// more on average, whose arrays do not stay in L2 from one kernel to the next.
// Measured, us per step (that form | the other), runs x particles, mesh:
// 2 x 100 000, 256^2 36.7 | 35.6; 4 x 100 000 50.8 | 52.3; 2 x 250 000, 512^2
// 59.9 | 64.2; 8 x 250 000 200 | 258; 4 x 600 000 206 | 280; 1 x 2 000 000,
// 2048^2 247 | 351; the 256-run ensemble (24 000 on average) 562 | 537. But not
// with many particles to a mesh point: the blocks that it keeps under way are
// neighbours and deposit on the same few points (500 000, 64^2 106 | 87;
// 1 000 000, 128^2 127 | 112; 3 000 000, 64^2 2202 | 789).
// blocks: of 256 particles, all runs together.
inline bool step_kernel_prefetches(int blocks, int runs, double particles, double points) {
  return blocks >= runs * 512 && (points == 0.0 || !many_per_point(particles, points, 24));
}

// Whether a call of nsteps steps of a single ideal-gas run (no mesh: sort and
// particle kernels only) takes the stage kernels from a graph. Measured, us per
// step (resident | stage kernels), particles, calls of many steps: 5000 11.0 |
// 12.8; 35 000 13.3 | 13.1; 60 000 12.9 | 13.5; 131 072 16.8 | 15.1; 500 000 32.1 |
// 29.5; adaptive dt: 60 000 16.7 | 18.0; 131 072 22.5 | 21.2; 500 000 48.0 | 45.5. A
// call per step, which pays the resident launch's start each time: 3000 12.4 |
// 14.4; 5000 14.4 | 14.7; 8000 15.9 | 14.4; 60 000 18.5 | 14.4; adaptive dt: 5000
// 31.5 | 36.8; 8000 37.6 | 35.3
inline bool idgas_stage_kernels(int N, long long nsteps) { return N > 65536 || (nsteps == 1 && N > 6000); }

// us per step of a single resident run, about (to a factor of two: 64 000
// particles on 768^2 47, 262 144 on 1024^2 83, 3 000 000 on 1024^2 591).
inline double estimate_single(const FormRun& r) {
  return r.idgas ? 10.0 + 1e-4 * r.N : 15.0 + 1.9e-4 * r.N + (r.compiled() ? 5e-5 : 1.5e-4) * r.points();
}

// Steps of one resident launch: about 50 ms of the device's time, whatever the
// runs are (other work waits for a whole launch).
inline int steps_per_launch(double us) { return (int)std::max(1.0, std::min(1024.0, 5e4 / std::max(us, 1.0))); }

// A batch's calls of several steps: launches per step (the pipelined or the
// stage kernels), one cluster of CTAs per run, or a group of CTAs of one
// cooperative grid per run.
enum BatchStep { BATCH_LAUNCHES, BATCH_CLUSTERS, BATCH_GROUPS };
struct BatchForm {
  BatchStep step = BATCH_LAUNCHES;
  std::vector<int> ctas;  // per run: CTAs of its cluster or group
  double us = 0.0;        // estimate of a step
};

// held(k, cs): clusters of cs CTAs for run k that the device holds at once (0:
// none). slots: CTAs to share out among groups (0: no groups). piped: the batch
// has the pipelined step. sms: SMs of the device.
template <class Held>
BatchForm choose_batch_form(const std::vector<FormRun>& runs, const Held& held, int slots, bool piped, int sms = 148) {
  BatchForm out;
  const size_t n = runs.size();
  double particles = 0.0;
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
  double most;  // a resident form has to take less than this
  bool mesh = false;
  for (const FormRun& r : runs) {
    particles += r.N;
    mesh = mesh || !r.idgas;
  }
  if (piped) {
    // Estimates fitted to 1 to 128 runs of 1000 to 250 000 particles (clusters
    // 12-60 us, groups 14-45, the pipelined step 20-110). Of 171 batches of 2 to
    // 320 runs timed in every form, 5 took longer in the chosen one than in
    // launches (1.15 times at most).
    most = out.us = 19.0 + 8e-5 * particles;
  } else {
    // Estimates fitted to 864 batches of 2 to 320 runs of 300 to 100 000
    // particles on meshes of 32 to 1024 points a side, timed in every form (rms
    // errors of launches, groups and clusters 11, 12 and 23 %, hence the 0.9).
    // In the chosen form 7 of them take longer than in launches (by more than
    // 4 %; 1.44 times at most), and a step is 1.6 times as fast on average. The
    // piped batches' estimates, used for these too before, did not look at the
    // stage kernels: 157 took longer (256 adaptive runs on meshes of 32 to 1024
    // points: 6580 us a step on clusters of one CTA, 1464 in launches), 1.49
    // times as fast.
    out.us = estimate_launches(runs);
    most = (mesh ? 0.9 : 1.0) * out.us;
  }
  auto consider = [&](BatchStep s, const std::vector<int>& ctas, double t_piped) {
    if (ctas.empty()) return;
    const double t = piped ? t_piped : estimate_resident(runs, ctas, s == BATCH_CLUSTERS, sms);
    if (t >= most) return;
    most = out.us = t;
    out.step = s;
    out.ctas = ctas;
  };
  consider(BATCH_CLUSTERS, clusters, 8.0 + 0.025 * most_c);
  consider(BATCH_GROUPS, share, 14.0 + 0.016 * most_g);
  return out;
}

}  // namespace bd
