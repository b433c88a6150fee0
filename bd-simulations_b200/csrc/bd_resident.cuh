// Resident step: many steps of a run in one launch.
//
// The CTAs of one group (a thread-block cluster of up to 16 CTAs, one cluster
// per run; for one larger run, the whole cooperative grid; for few runs of
// uneven weight, a share of one) keep a run's step loop on the device: no launch, no drained grid and no reload of the
// run's description between steps, and a run's working set stays in L2 while
// its group advances. Many runs are independent groups, so the issue-bound
// particle phase of one overlaps the latency-bound transform and sort phases
// of its neighbours on the same SM.
//
// One step (the arithmetic of the stage kernels, same bits), the two halves
// of a CTA, each with a named barrier of its own, side by side:
//   I  inverse row transforms       |  WCA sums and noise of the CTA's share of
//                                   |  the particles, kept in shared memory
//   P  (all threads) mesh force, move, cell counts, the next density into
//      R.dacc; adaptive dt: forces and dt bound, barrier, then the move
//   S  next forward rows            |  scan of the cell counts
//   C  next columns + Green         |  scatter, step end
// with a group barrier after each. What bounds a step is the length of these
// chains (L2 round trips, one thread's instructions, the barriers: storing,
// meeting and loading again takes 1400 cycles in a cluster of 16 and 3400 on
// the grid), not bandwidth; about 30 % of the issue slots of its SMs are used.
// Measured, us per step of whole calls of many steps with the positions read
// behind them, one launch per step or eight before | here: 2000 particles, 128^2
// 20.4 | 15.2; 65 536, 512^2 27.8 | 27.6 (one launch per step already: no gain);
// 2204, 96^2 adaptive 48 | 18; 70 002, 768^2 88 | 47; a batch of 16 adaptive runs
// 179 | 57. The steps alone: 14.5, 25.2, 16.8 and 44.2; 4000, 384^2 adaptive 21.9.
//
// State between launches, as the prologue (deposit, forward rows, columns)
// leaves it: spec2 holds the column-transformed spectrum of the current
// positions and R.dacc is zero. Runs without an accumulator of their own
// (radix-3 meshes, adaptive dt) use spec2's memory for it: the inverse rows
// clear what they read, the density is deposited there and the forward rows
// read it before the column pass overwrites it.
#pragma once

#include <algorithm>

#include "bd_items.cuh"

namespace bd {

// ---- power-of-two meshes: the passes of fft2_rows_fwd_item, fft2_cols_item
// and fft2_rows_inv_item with four elements per thread. An item holds at most
// four elements per thread of the team, so every load and store loop is four
// predicated accesses issued together (a loop with a run-time trip count
// waited for each L2 round trip in turn).

template <int LZ, class Team>
__device__ __forceinline__ void res2_rows_fwd_item(const Team& T, const RunDesc& R, int row0, int lr, bool clear,
                                                   float2* s, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1, ln = LZ - 1;
  constexpr int ss = fft2_stride(n);
  const int tot = n << lr;
  ulonglong2* acc = reinterpret_cast<ulonglong2*>(R.dacc) + (size_t)row0 * n;
  float2* rho = reinterpret_cast<float2*>(R.rho) + (size_t)row0 * n;
  const double inv = pow2_double(-R.fx_shift);
  ulonglong2 a[4];
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    a[u] = make_ulonglong2(0ull, 0ull);
    if (i < tot) a[u] = acc[i];
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    if (i < tot) {
      const float2 v = make_float2((float)((double)(long long)a[u].x * inv), (float)((double)(long long)a[u].y * inv));
      s[(i >> ln) * ss + pad16(i & (n - 1))] = v;
      rho[i] = v;
      if (clear) acc[i] = make_ulonglong2(0ull, 0ull);
    }
  }
  T.sync();
  Fft4Sched<LZ - 1, 0>::run(T, s, ss, 1 << lr, tw, LZ, -1.f);
  // groups of up to four rows of one slot (fft2_rows_fwd_item)
  const int lrb = lr < 2 ? lr : 2;
  const int rbm = (1 << lrb) - 1;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    if (i < tot) {
      const int rest = i >> lrb;
      const int j = rest & (n - 1), b = ((rest >> ln) << lrb) + (i & rbm);
      const float2 zj = s[b * ss + pad16(j)];
      const float2 zc = s[b * ss + pad16((n - j) & (n - 1))];
      float2 out;
      if (j == 0) {
        out = make_float2(zj.x + zj.y, zj.x - zj.y);
      } else {
        // E = (zj + conj zc)/2, O = (zj - conj zc)/(2i), X = E + w^j O
        const float2 E = make_float2(0.5f * (zj.x + zc.x), 0.5f * (zj.y - zc.y));
        const float2 O = make_float2(0.5f * (zj.y + zc.y), -0.5f * (zj.x - zc.x));
        out = cadd(E, cmul(tw[j], O));
      }
      R.spec[(size_t)j * Z + row0 + b] = out;
    }
  }
  T.sync();
}

template <int LZ, class Team>
__device__ __forceinline__ void res2_cols_item(const Team& T, const RunDesc& R, int col0, int lw, float2* sA,
                                               const float2* tw, const float* sx) {
  constexpr int Z = 1 << LZ, n = Z >> 1;
  constexpr int ss = fft2_stride(Z);
  const int W = 1 << lw, tot = Z << lw;
  float2* sB = sA + W * ss;
  const float2* src = R.spec + (size_t)col0 * Z;
  {
    float2 v[4];
    float g[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = T.tid + u * T.nt();
      v[u] = make_float2(0.f, 0.f);
      if (i < tot) v[u] = src[i];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = T.tid + u * T.nt();
      if (i < tot) sA[(i >> LZ) * ss + pad16(i & (Z - 1))] = v[u];
    }
    // the Green's factors, requested ahead of the transform
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = T.tid + u * T.nt();
      g[u] = i < tot ? __ldg(&R.green[(size_t)col0 * Z + i]) : 0.f;
    }
    T.sync();
    Fft4Sched<LZ, 0>::run(T, sA, ss, W, tw, LZ, -1.f);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = T.tid + u * T.nt();
      const int c = i >> LZ, kx = i & (Z - 1), j = col0 + c;
      if (i < tot && j != 0) {
        const float gx = sx[kx] * g[u];
        const float gy = sx[Z + j] * g[u];
        const int a = c * ss + pad16(kx);
        const float2 v = sA[a];
        sA[a] = make_float2(-gx * v.y, gx * v.x);
        sB[a] = make_float2(-gy * v.y, gy * v.x);
      }
    }
  }
  if (col0 == 0) {
    // packed column (ky = 0, ky = Z/2): one thread handles kx and -kx
    const float sy0 = __ldg(&R.syt[0]), syn = __ldg(&R.syt[n]);
    for (int kx = T.tid; kx <= n; kx += T.nt()) {
      const int km = (Z - kx) & (Z - 1);
      const float2 Ck = sA[pad16(kx)], Cm = sA[pad16(km)];
      float2 P, Q;
      packed_green(R, kx, Ck, Cm, n, Z, sy0, syn, P, Q);
      sA[pad16(kx)] = P;
      sB[pad16(kx)] = Q;
      if (km != kx) {
        packed_green(R, km, Cm, Ck, n, Z, sy0, syn, P, Q);
        sA[pad16(km)] = P;
        sB[pad16(km)] = Q;
      }
    }
  }
  T.sync();
  if (2 * W * fft4_tps(LZ) <= T.nt()) {
    Fft4Sched<LZ, 0>::run(T, sA, ss, 2 * W, tw, LZ, 1.f);  // sB follows sA: 2W sequences
  } else {
    Fft4Sched<LZ, 0>::run(T, sA, ss, W, tw, LZ, 1.f);
    Fft4Sched<LZ, 0>::run(T, sB, ss, W, tw, LZ, 1.f);
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    if (i < tot) {
      const int k = i >> lw, c = i & (W - 1);
      const float2 a = sA[c * ss + pad16(k)], b = sB[c * ss + pad16(k)];
      R.spec2[(size_t)k * n + col0 + c] = make_float4(a.x, a.y, b.x, b.y);
    }
  }
  T.sync();
}

template <int LZ, class Team>
__device__ __forceinline__ void res2_rows_inv_item(const Team& T, const RunDesc& R, int row0, int lr, float2* s,
                                                   const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1;
  constexpr int ss = fft2_stride(Z);
  const int tot = Z << lr;
  float4 v[4];
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    const int b = i >> LZ, j = i & (Z - 1);
    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < tot) v[u] = R.spec2[(size_t)(row0 + b) * n + (j < n ? j : (Z - j) & (n - 1))];
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    const int b = i >> LZ, j = i & (Z - 1);
    float2 h;
    if (j == 0) h = make_float2(v[u].x, v[u].z);
    else if (j == n) h = make_float2(v[u].y, v[u].w);
    else if (j < n) h = make_float2(v[u].x - v[u].w, v[u].y + v[u].z);
    else h = make_float2(v[u].x + v[u].w, -v[u].y + v[u].z);
    if (i < tot) s[b * ss + pad16(j)] = h;
  }
  T.sync();
  Fft4Sched<LZ, 0>::run(T, s, ss, 1 << lr, tw, LZ, 1.f);
  float2* dst = R.H + (size_t)row0 * Z;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt();
    if (i < tot) dst[i] = s[(i >> LZ) * ss + pad16(i & (Z - 1))];
  }
  T.sync();
}

// ---- transforms of meshes with a factor 3, one item of a team ---------------
// (layouts and arithmetic of k_fft_rows_fwd, k_fft_cols, k_fft_rows_inv; the
// twiddle table tw is a copy in shared memory)

template <class Team>
__device__ __forceinline__ void gen_rows_fwd_item(const Team& T, const RunDesc& R, int row0, int lr, bool clear,
                                                  float2* s, const float2* tw) {
  const int Z = R.Z, n = Z >> 1, tot = n << lr;
  ulonglong2* acc = reinterpret_cast<ulonglong2*>(R.dacc) + (size_t)row0 * n;
  float2* rho = reinterpret_cast<float2*>(R.rho) + (size_t)row0 * n;
  const double inv = pow2_double(-R.fx_shift);
  for (int i = T.tid; i < tot; i += T.nt()) {
    const int b = i / n, m = i - b * n;
    const ulonglong2 a = acc[i];
    const float2 v = make_float2((float)((double)(long long)a.x * inv), (float)((double)(long long)a.y * inv));
    s[(m << lr) | b] = v;
    rho[i] = v;
    if (clear) acc[i] = make_ulonglong2(0ull, 0ull);
  }
  T.sync();
  fft_dif<true>(T, s, R.plan_half, lr, tw, 2, false);
  for (int i = T.tid; i < tot; i += T.nt()) {
    const int b = i / n, j = i - b * n;
    const float2 zj = s[(__ldg(&R.pos_half[j]) << lr) | b];
    const float2 zc = s[(__ldg(&R.pos_half[j == 0 ? 0 : n - j]) << lr) | b];
    float2 out;
    if (j == 0) {
      out = make_float2(zj.x + zj.y, zj.x - zj.y);
    } else {
      const float2 E = make_float2(0.5f * (zj.x + zc.x), 0.5f * (zj.y - zc.y));
      const float2 O = make_float2(0.5f * (zj.y + zc.y), -0.5f * (zj.x - zc.x));
      out = cadd(E, cmul(tw[j], O));
    }
    R.spec[(size_t)(row0 + b) * n + j] = out;
  }
  T.sync();
}

template <class Team>
__device__ __forceinline__ void gen_cols_item(const Team& T, const RunDesc& R, int col0, int lw, float2* sA,
                                              const float2* tw) {
  const int Z = R.Z, n = Z >> 1;
  const int W = 1 << lw;
  float2* sB = sA + ((size_t)Z << lw);
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int k = i >> lw, c = i & (W - 1);
    sA[i] = R.spec[(size_t)k * n + col0 + c];
  }
  T.sync();
  fft_dif<true>(T, sA, R.plan_full, lw, tw, 1, false);
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int pos = i >> lw, c = i & (W - 1);
    const int j = col0 + c;
    if (j == 0) continue;
    const int kx = __ldg(&R.freq_full[pos]);
    const float g = __ldg(&R.green[(size_t)j * Z + kx]);
    const float gx = __ldg(&R.sxt[kx]) * g;
    const float gy = __ldg(&R.syt[j]) * g;
    const float2 v = sA[i];
    sA[i] = make_float2(-gx * v.y, gx * v.x);
    sB[i] = make_float2(-gy * v.y, gy * v.x);
  }
  if (col0 == 0) {
    // packed column (ky = 0, ky = Z/2): one thread handles kx and -kx
    const float sy0 = __ldg(&R.syt[0]), syn = __ldg(&R.syt[n]);
    for (int kx = T.tid; kx <= n; kx += T.nt()) {
      const int km = kx == 0 ? 0 : Z - kx;
      const int pk = __ldg(&R.pos_full[kx]) << lw, pm = __ldg(&R.pos_full[km]) << lw;
      const float2 Ck = sA[pk], Cm = sA[pm];
      float2 P, Q;
      packed_green(R, kx, Ck, Cm, n, Z, sy0, syn, P, Q);
      sA[pk] = P;
      sB[pk] = Q;
      if (km != kx) {
        packed_green(R, km, Cm, Ck, n, Z, sy0, syn, P, Q);
        sA[pm] = P;
        sB[pm] = Q;
      }
    }
  }
  T.sync();
  fft_dit<true>(T, sA, R.plan_full, lw, tw, 1, true);
  fft_dit<true>(T, sB, R.plan_full, lw, tw, 1, true);
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int k = i >> lw, c = i & (W - 1);
    const float2 a = sA[i], b = sB[i];
    R.spec2[(size_t)k * n + col0 + c] = make_float4(a.x, a.y, b.x, b.y);
  }
  T.sync();
}

template <class Team>
__device__ __forceinline__ void gen_rows_inv_item(const Team& T, const RunDesc& R, int row0, int lr, float2* s,
                                                  const float2* tw) {
  const int Z = R.Z, n = Z >> 1;
  for (int i = T.tid; i < (Z << lr); i += T.nt()) {
    const int b = i / Z, j = i - b * Z;
    const size_t rb = (size_t)(row0 + b) * n;
    float2 h;
    if (j == 0) {
      const float4 v = R.spec2[rb];
      h = make_float2(v.x, v.z);
    } else if (j == n) {
      const float4 v = R.spec2[rb];
      h = make_float2(v.y, v.w);
    } else if (j < n) {
      const float4 v = R.spec2[rb + j];
      h = make_float2(v.x - v.w, v.y + v.z);
    } else {
      const float4 v = R.spec2[rb + (Z - j)];
      h = make_float2(v.x + v.w, -v.y + v.z);
    }
    s[(__ldg(&R.pos_full[j]) << lr) | b] = h;
  }
  T.sync();
  fft_dit<true>(T, s, R.plan_full, lr, tw, 1, true);
  for (int i = T.tid; i < (Z << lr); i += T.nt()) {
    const int b = i / Z, l = i - b * Z;
    R.H[(size_t)(row0 + b) * Z + l] = s[(l << lr) | b];
  }
  T.sync();
}

// Meshes of Z = 3 * 2^k points a side: the same passes, lengths known at
// compile time, a sequence's elements in order, the half spectrum by column
// (slot j of row k at j*Z + k, as the power-of-two meshes). An item holds at
// most eight elements per thread, accessed four at a time.
template <int Z, class Team>
__device__ __forceinline__ void tri_rows_fwd_item(const Team& T, const RunDesc& R, int row0, int lr, bool clear,
                                                  float2* s, const float2* tw) {
  constexpr int n = Z / 2;
  const int tot = n << lr;
  ulonglong2* acc = reinterpret_cast<ulonglong2*>(R.dacc) + (size_t)row0 * n;
  float2* rho = reinterpret_cast<float2*>(R.rho) + (size_t)row0 * n;
  const double inv = pow2_double(-R.fx_shift);
  for (int i0 = T.tid; i0 < tot; i0 += 4 * T.nt()) {
    ulonglong2 a[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      a[u] = make_ulonglong2(0ull, 0ull);
      if (i0 + u * T.nt() < tot) a[u] = acc[i0 + u * T.nt()];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * T.nt();
      if (i < tot) {
        const float2 v =
            make_float2((float)((double)(long long)a[u].x * inv), (float)((double)(long long)a[u].y * inv));
        s[i] = v;
        rho[i] = v;
        if (clear) acc[i] = make_ulonglong2(0ull, 0ull);
      }
    }
  }
  T.sync();
  FftcDif<n, 2>::run(T, s, 1 << lr, tw);
  const int lrb = lr < 2 ? lr : 2;
  const int rbm = (1 << lrb) - 1;
  for (int i = T.tid; i < tot; i += T.nt()) {
    const int rest = i >> lrb, bg = rest / n;
    const int j = rest - bg * n, b = (bg << lrb) + (i & rbm);
    const float2 zj = s[b * n + FftcDif<n, 2>::pos(j)];
    const float2 zc = s[b * n + FftcDif<n, 2>::pos(j == 0 ? 0 : n - j)];
    float2 out;
    if (j == 0) {
      out = make_float2(zj.x + zj.y, zj.x - zj.y);
    } else {
      const float2 E = make_float2(0.5f * (zj.x + zc.x), 0.5f * (zj.y - zc.y));
      const float2 O = make_float2(0.5f * (zj.y + zc.y), -0.5f * (zj.x - zc.x));
      out = cadd(E, cmul(tw[j], O));
    }
    R.spec[(size_t)j * Z + row0 + b] = out;
  }
  T.sync();
}

template <int Z, class Team>
__device__ __forceinline__ void tri_cols_item(const Team& T, const RunDesc& R, int col0, int lw, float2* sA,
                                              const float2* tw, const float* sx) {
  constexpr int n = Z / 2;
  const int W = 1 << lw, tot = Z << lw;
  float2* sB = sA + tot;
  const float2* src = R.spec + (size_t)col0 * Z;
  for (int i0 = T.tid; i0 < tot; i0 += 4 * T.nt()) {
    float2 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      v[u] = make_float2(0.f, 0.f);
      if (i0 + u * T.nt() < tot) v[u] = src[i0 + u * T.nt()];
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * T.nt() < tot) sA[i0 + u * T.nt()] = v[u];
  }
  // the Green's factors of the first elements, requested ahead of the transform
  float g[4];
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = T.tid + u * T.nt(), c = i / Z;
    g[u] = i < tot ? __ldg(&R.green[(size_t)(col0 + c) * Z + FftcDif<Z, 1>::freq(i - c * Z)]) : 0.f;
  }
  T.sync();
  FftcDif<Z, 1>::run(T, sA, W, tw);
  auto green = [&](int i, float gi) {
    const int c = i / Z, kx = FftcDif<Z, 1>::freq(i - c * Z);
    const int j = col0 + c;
    if (j == 0) return;
    const float gx = sx[kx] * gi;
    const float gy = sx[Z + j] * gi;
    const float2 v = sA[i];
    sA[i] = make_float2(-gx * v.y, gx * v.x);
    sB[i] = make_float2(-gy * v.y, gy * v.x);
  };
#pragma unroll
  for (int u = 0; u < 4; u++)
    if (T.tid + u * T.nt() < tot) green(T.tid + u * T.nt(), g[u]);
  for (int i = T.tid + 4 * T.nt(); i < tot; i += T.nt()) {
    const int c = i / Z;
    green(i, __ldg(&R.green[(size_t)(col0 + c) * Z + FftcDif<Z, 1>::freq(i - c * Z)]));
  }
  if (col0 == 0) {
    // packed column (ky = 0, ky = Z/2): one thread handles kx and -kx
    const float sy0 = __ldg(&R.syt[0]), syn = __ldg(&R.syt[n]);
    for (int kx = T.tid; kx <= n; kx += T.nt()) {
      const int km = kx == 0 ? 0 : Z - kx;
      const int pk = FftcDif<Z, 1>::pos(kx), pm = FftcDif<Z, 1>::pos(km);
      const float2 Ck = sA[pk], Cm = sA[pm];
      float2 P, Q;
      packed_green(R, kx, Ck, Cm, n, Z, sy0, syn, P, Q);
      sA[pk] = P;
      sB[pk] = Q;
      if (km != kx) {
        packed_green(R, km, Cm, Ck, n, Z, sy0, syn, P, Q);
        sA[pm] = P;
        sB[pm] = Q;
      }
    }
  }
  T.sync();
  FftcDit<Z, 1>::run(T, sA, 2 * W, tw);  // sB follows sA
  for (int i = T.tid; i < tot; i += T.nt()) {
    const int k = i >> lw, c = i & (W - 1);
    const float2 a = sA[c * Z + k], b = sB[c * Z + k];
    R.spec2[(size_t)k * n + col0 + c] = make_float4(a.x, a.y, b.x, b.y);
  }
  T.sync();
}

template <int Z, class Team>
__device__ __forceinline__ void tri_rows_inv_item(const Team& T, const RunDesc& R, int row0, int lr, float2* s,
                                                  const float2* tw) {
  constexpr int n = Z / 2;
  const int tot = Z << lr;
  for (int i0 = T.tid; i0 < tot; i0 += 4 * T.nt()) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * T.nt(), b = i / Z, j = i - b * Z;
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < tot) v[u] = R.spec2[(size_t)(row0 + b) * n + (j < n ? j : j == n ? 0 : Z - j)];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * T.nt(), b = i / Z, j = i - b * Z;
      float2 h;
      if (j == 0) h = make_float2(v[u].x, v[u].z);
      else if (j == n) h = make_float2(v[u].y, v[u].w);
      else if (j < n) h = make_float2(v[u].x - v[u].w, v[u].y + v[u].z);
      else h = make_float2(v[u].x + v[u].w, -v[u].y + v[u].z);
      if (i < tot) s[b * Z + FftcDif<Z, 1>::pos(j)] = h;
    }
  }
  T.sync();
  FftcDit<Z, 1>::run(T, s, 1 << lr, tw);
  for (int i = T.tid; i < tot; i += T.nt()) R.H[(size_t)row0 * Z + i] = s[i];
  T.sync();
}

// ---- the step's phases ------------------------------------------------------

// Scan of the counts of this CTA's contiguous share of the run's chunks. The
// counts are requested first; every warp sums the totals of the earlier
// chunks for itself, so one scan over the team is left.
template <int NT, class Team>
__device__ __forceinline__ void res_scan(const Team& T, const RunDesc& R, int b, int G, int nch, int* sh) {
  constexpr int PER = SCAN_CHUNK / NT;
  const int per = (nch + G - 1) / G, c0 = b * per, c1 = min(nch, c0 + per);
  if (c0 >= c1) return;
  const int ncells = R.C * R.C;
  int off = 0;
  for (int c = c0; c < c1; c++) {
    const int k0 = c * SCAN_CHUNK + T.tid * PER;
    int v[PER];
    if ((c + 1) * SCAN_CHUNK <= ncells) {
#pragma unroll
      for (int k = 0; k < PER; k += 4) {
        const int4 a = *reinterpret_cast<const int4*>(&R.count[k0 + k]);
        v[k] = a.x, v[k + 1] = a.y, v[k + 2] = a.z, v[k + 3] = a.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < PER; k++) v[k] = k0 + k < ncells ? R.count[k0 + k] : 0;
    }
    const int tot = R.chunk_sum[c];
    if (c == c0 && c0 > 0) {
      int loc = 0;
#pragma unroll 4
      for (int k = T.tid & 31; k < c0; k += 32) loc += R.chunk_sum[k];
      off = __reduce_add_sync(0xffffffffu, loc);
    }
    scan_chunk_store<PER>(T, R, c, ncells, v, off, sh);
    off += tot;
  }
}

// Records to their cells, four per thread at a time: src[0 .. n). noise: also
// the next step's noise of each, to the same place of that array (the half
// CTA that sorts waits for the transforms otherwise).
template <int NT, class Team>
__device__ __forceinline__ void res_scatter(const Team& T, const RunDesc& R, const Rec* src, int n, float2* noise,
                                            unsigned long long next) {
  for (int g = T.tid; g < n; g += 4 * NT) {
    Rec q[4] = {};
    int at[4] = {};
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (g + k * NT < n) q[k] = src[g + k * NT];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (g + k * NT < n) at[k] = R.start[q[k].cell] + atomicSub(&R.count[q[k].cell], 1) - 1;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (g + k * NT < n) R.recA[at[k]] = q[k];
    if (noise) {
#pragma unroll 1
      for (int k = 0; k < 4; k++)
        if (g + k * NT < n) noise[at[k]] = particle_noise(R.noise, R.seed, next, (uint32_t)q[k].pid);
    }
  }
}

// WCA force and noise of one particle.
__device__ __forceinline__ float2 res_wca(const RunDesc& R, const Rec& p, int gi) {
  if (R.flags & F_IDGAS) return make_float2(0.f, 0.f);
  int ic, jc;
  cell_ij(R, p.cell, ic, jc);
  return wca_direct<false>(R, p, ic, jc, gi, 7);
}
__device__ __forceinline__ float2 res_noise(const RunDesc& R, const Rec& p, unsigned long long step) {
  if (R.flags & F_NOWCA) return make_float2(0.f, 0.f);
  return particle_noise(R.noise, R.seed, step, (uint32_t)p.pid);
}
__device__ __forceinline__ float2 res_mesh(const RunDesc& R, const Rec& p) {
  if (R.flags & F_IDGAS) return make_float2(0.f, 0.f);
  int ic, jc;
  cell_ij(R, p.cell, ic, jc);
  return mesh_force<false>(R, p, ic, jc, R.scheme);
}

// The lanes of this thread's warp that work on one of n things, LANES lanes
// for each, i (< n) this thread's.
template <int LANES>
__device__ __forceinline__ unsigned lanes_below(int i, int n) {
  const int lane = (int)threadIdx.x & 31;
  const int k = (n - (i - lane / LANES)) * LANES;  // lanes of the warp in use
  return k >= 32 ? 0xffffffffu : (1u << k) - 1u;
}

// The move of particle p with its counts and its deposit, LANES lanes per
// particle: each computes the move, the lanes share the deposit's points and
// lane 0 counts. act: the lanes of the warp that call.
template <int LANES>
__device__ __forceinline__ Rec res_move(const RunDesc& R, RunDyn* D, const Rec& p, float2 F, float2 xi, float dt,
                                        float sq, bool mesh, int sub, unsigned act) {
  const Rec np = move_particle_sq(R, p, F, xi, dt, sq, &D->err, true, sub == 0);
  __syncwarp(act);
  if (sub == 0) {
    constexpr unsigned first = LANES == 1 ? 0xffffffffu : LANES == 2 ? 0x55555555u : 0x11111111u;
    count_into_cell(R, np.cell, act & first);
    if (np.cell != p.cell) atomicAdd(&D->moved[p.pid >= R.N1 ? 1 : 0], 1);
  }
  if (mesh) deposit_acc<LANES>(R, np, sub);
  return np;
}

// Adaptive dt: the forces stored by particle index (as the split step leaves
// them), the bits of this particle's dt bound (3e38 when it cannot win).
__device__ __forceinline__ unsigned res_bound(const RunDesc& R, const Rec& p, float2 Fw, float2 Fk, float2 xi) {
  R.Fw[p.pid] = Fw;
  R.Fk[p.pid] = Fk;
  R.Fn[p.pid] = xi;
  float bnd = fminf(dt_bound(Fw.x + Fk.x, xi.x, R.mrd, R.T), dt_bound(Fw.y + Fk.y, xi.y, R.mrd, R.T));
  if (!(bnd >= 0.f)) bnd = 3.0e38f;  // NaN never wins the minimum (std::min semantics)
  return __float_as_uint(bnd < R.dt_max ? bnd : 3.0e38f);
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// Dynamic shared memory of a CTA: the run's description, the twiddle table,
// the transforms' work space and, from part_off, up to pcap of the CTA's
// particles (records, WCA forces, noise). The phases name it themselves (a
// pointer parameter would be generic and every access a generic load).
extern __shared__ __align__(16) unsigned char res_smem[];
__device__ __forceinline__ const RunDesc& res_desc() { return *reinterpret_cast<const RunDesc*>(res_smem); }
__device__ __forceinline__ float2* res_tw() { return reinterpret_cast<float2*>(res_smem + RES_DESC_BYTES); }
// sin(q dx)/dx for kx in [0, Z), then for ky in [0, Z/2], behind the twiddles
__device__ __forceinline__ float* res_sx(int Z) { return reinterpret_cast<float*>(res_tw() + Z); }
__device__ __forceinline__ float2* res_work(int Z) {
  return reinterpret_cast<float2*>(res_smem + RES_DESC_BYTES + RES_TW_BYTES(Z));
}
struct ResPart {
  Rec* rec;
  float2 *F, *xi;
  __device__ __forceinline__ ResPart(int part_off, int pcap)
      : rec(reinterpret_cast<Rec*>(res_smem + part_off)),
        F(reinterpret_cast<float2*>(rec + pcap)),
        xi(F + pcap) {}
};

// The phases are functions of their own: inlined into the step loop, the
// compiler keeps the per-thread addresses of every transform pass live
// across it and spills. NT: threads of a half CTA.

// I, lower half: inverse rows; a shared accumulator is cleared behind them
template <int LZ, int NT>
__device__ __noinline__ void res_inv(int b, int G, int lri, bool alias) {
  const RunDesc& R = res_desc();
  const int Z = res_side(LZ) ? res_side(LZ) : R.Z, n = Z >> 1, nri = Z >> lri;
#pragma unroll 1
  for (int it = b; it < nri; it += G) {
    const HalfTeam<0, NT> T;
    if constexpr (LZ >= 16) tri_rows_inv_item<res_side(LZ)>(T, R, it << lri, lri, res_work(Z), res_tw());
    else if constexpr (LZ != 0) res2_rows_inv_item<LZ>(T, R, it << lri, lri, res_work(Z), res_tw());
    else gen_rows_inv_item(T, R, it << lri, lri, res_work(Z), res_tw());
    if (alias) {
      float4* q = R.spec2 + ((size_t)it << lri) * n;
      for (int i = T.tid; i < (n << lri); i += NT) q[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// I, upper half: WCA sums and noise of particles [g0, g0 + nc); noise: drawn
// already by the scatter that placed them, in their order. Few particles: the
// neighbour rows of one go to three of four lanes (the sum is an integer one,
// exact in any order).
template <int NT>
__device__ __noinline__ void res_pairs(unsigned long long step, int g0, int nc, const float2* noise, int part_off,
                                       int pcap) {
  const RunDesc& R = res_desc();
  const ResPart S(part_off, pcap);
  const int t = (int)threadIdx.x - NT;
  if (4 * nc <= NT && !(R.flags & F_IDGAS)) {
    const int i = t >> 2, row = t & 3;
    long long fx = 0, fy = 0;
    Rec p = {};
    if (i < nc) {
      p = ldrec<false>(&R.recA[g0 + i]);
      int ic, jc;
      cell_ij(R, p.cell, ic, jc);
      if (row < 3) wca_row(R, wca_params(R, p, 7), p, ic, jc, g0 + i, row - 1, fx, fy);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      fx += __shfl_xor_sync(0xffffffffu, fx, o);
      fy += __shfl_xor_sync(0xffffffffu, fy, o);
    }
    if (i < nc) {
      if (row == 0) S.rec[i] = p;
      if (row == 1) S.F[i] = wca_unfix(R, fx, fy);
      if (row == 3) S.xi[i] = noise ? noise[g0 + i] : res_noise(R, p, step);
    }
    return;
  }
  for (int i = t; i < nc; i += NT) {
    const Rec p = ldrec<false>(&R.recA[g0 + i]);
    S.rec[i] = p;
    S.xi[i] = noise ? noise[g0 + i] : res_noise(R, p, step);
    S.F[i] = res_wca(R, p, g0 + i);
  }
}

// P, fixed dt: the CTA's particles [g0, g1), the first nc from shared memory
template <int NT, int LANES>
__device__ __noinline__ void res_step(RunDyn* D, unsigned long long step, int g0, int g1, int nc, bool mesh,
                                      int part_off, int pcap) {
  const RunDesc& R = res_desc();
  const ResPart S(part_off, pcap);
  const float sq = sqrtf(2.0f * R.T * R.dt_max);
  const int sub = (int)threadIdx.x & (LANES - 1);
  for (int i = (int)threadIdx.x / LANES; i < nc; i += 2 * NT / LANES) {
    const Rec p = S.rec[i];
    const float2 Fk = res_mesh(R, p), Fw = S.F[i];
    const Rec np = res_move<LANES>(R, D, p, make_float2(Fw.x + Fk.x, Fw.y + Fk.y), S.xi[i], R.dt_max, sq, mesh, sub,
                                   lanes_below<LANES>(i, nc));
    if constexpr (LANES > 1) {
      // every lane of the particle has read its record
      const unsigned lane = threadIdx.x & 31u;
      __syncwarp(((1u << LANES) - 1u) << (lane & ~(unsigned)(LANES - 1)));
    }
    if (sub == 0) S.rec[i] = np;
  }
  if constexpr (LANES == 1)
    for (int gi = g0 + nc + (int)threadIdx.x; gi < g1; gi += 2 * NT) {
      if (mesh) step_particle<false, true>(R, *D, step, gi, lanes_below<1>(gi, g1));
      else step_particle<false, false>(R, *D, step, gi, lanes_below<1>(gi, g1));
    }
}

// P, adaptive dt, before its barrier: the rest of the forces, the dt bound
template <int NT>
__device__ __noinline__ void res_forces(RunDyn* D, unsigned long long step, int g0, int g1, int nc, int part_off,
                                        int pcap) {
  const RunDesc& R = res_desc();
  const ResPart S(part_off, pcap);
  unsigned bits = __float_as_uint(3.0e38f);
  for (int i = (int)threadIdx.x; i < nc; i += 2 * NT) {
    const Rec p = S.rec[i];
    const float2 Fk = res_mesh(R, p), Fw = S.F[i];
    S.F[i] = make_float2(Fw.x + Fk.x, Fw.y + Fk.y);
    bits = min(bits, res_bound(R, p, Fw, Fk, S.xi[i]));
  }
  for (int gi = g0 + nc + (int)threadIdx.x; gi < g1; gi += 2 * NT) {
    const Rec p = ldrec<false>(&R.recA[gi]);
    bits = min(bits, res_bound(R, p, res_wca(R, p, gi), res_mesh(R, p), res_noise(R, p, step)));
  }
  bits = __reduce_min_sync(0xffffffffu, bits);
  if ((threadIdx.x & 31) == 0 && bits < __float_as_uint(3.0e38f)) atomicMin(&D->dt_bits, bits);
}

// ... and after it: the move
template <int NT>
__device__ __noinline__ void res_adaptive_move(RunDyn* D, int g0, int g1, int nc, bool mesh, int part_off, int pcap) {
  const RunDesc& R = res_desc();
  const ResPart S(part_off, pcap);
  const float dt = fminf(R.dt_max, __uint_as_float(((volatile RunDyn*)D)->dt_bits));
  const float sq = sqrtf(2.0f * R.T * dt);
  for (int i = (int)threadIdx.x; i < nc; i += 2 * NT)
    S.rec[i] = res_move<1>(R, D, S.rec[i], S.F[i], S.xi[i], dt, sq, mesh, 0, lanes_below<1>(i, nc));
  for (int gi = g0 + nc + (int)threadIdx.x; gi < g1; gi += 2 * NT) {
    const Rec p = ldrec<false>(&R.recA[gi]);
    const float2 Fw = R.Fw[p.pid], Fk = R.Fk[p.pid];
    R.recB[gi] = res_move<1>(R, D, p, make_float2(Fw.x + Fk.x, Fw.y + Fk.y), R.Fn[p.pid], dt, sq, mesh, 0,
                             lanes_below<1>(gi, g1));
  }
}

// S, lower half: forward rows of the new density
template <int LZ, int NT>
__device__ __noinline__ void res_fwd(int b, int G, int lrf, bool alias) {
  const RunDesc& R = res_desc();
  const int Z = res_side(LZ) ? res_side(LZ) : R.Z, nrf = Z >> lrf;
#pragma unroll 1
  for (int it = G - 1 - b; it < nrf; it += G) {
    const HalfTeam<0, NT> T;
    if constexpr (LZ >= 16)
      tri_rows_fwd_item<res_side(LZ)>(T, R, it << lrf, lrf, !alias, res_work(Z), res_tw());
    else if constexpr (LZ != 0)
      res2_rows_fwd_item<LZ>(T, R, it << lrf, lrf, !alias, res_work(Z), res_tw());
    else
      gen_rows_fwd_item(T, R, it << lrf, lrf, !alias, res_work(Z), res_tw());
  }
}

// C, lower half: columns + Green
template <int LZ, int NT>
__device__ __noinline__ void res_cols(int b, int G, int lw) {
  const RunDesc& R = res_desc();
  const int Z = res_side(LZ) ? res_side(LZ) : R.Z, ncl = (Z >> 1) >> lw;
#pragma unroll 1
  for (int it = G - 1 - b; it < ncl; it += G) {
    const HalfTeam<0, NT> T;
    if constexpr (LZ >= 16) tri_cols_item<res_side(LZ)>(T, R, it << lw, lw, res_work(Z), res_tw(), res_sx(Z));
    else if constexpr (LZ != 0) res2_cols_item<LZ>(T, R, it << lw, lw, res_work(Z), res_tw(), res_sx(Z));
    else gen_cols_item(T, R, it << lw, lw, res_work(Z), res_tw());
  }
}

// S and C, upper half: scan; scatter and step end
template <int NT>
__device__ __noinline__ void res_scan_phase(int b, int G, int nch, int* sh) {
  res_scan<NT>(HalfTeam<1, NT>(), res_desc(), b, G, nch, sh);
}
template <int NT>
__device__ __noinline__ void res_place(RunDyn* D, int b, int g0, int g1, int nc, int nch, bool adaptive,
                                       float2* noise, unsigned long long next, int part_off, int pcap) {
  const RunDesc& R = res_desc();
  const HalfTeam<1, NT> T;
  res_scatter<NT>(T, R, ResPart(part_off, pcap).rec, nc, noise, next);
  res_scatter<NT>(T, R, R.recB + g0 + nc, g1 - g0 - nc, nullptr, 0ull);
  if (b == 0) {
    for (int c = T.tid; c < nch; c += NT) R.chunk_sum[c] = 0;
    if (T.tid == 0) end_step(R, *D, adaptive ? 1 : 0);
  }
}

// The transform phases with the mesh class known at run time (RES_GROUPS).
template <int LZ, int NT>
__device__ __forceinline__ void res_inv_of(int lz, int b, int G, int lri, bool alias) {
  if constexpr (LZ >= 0) res_inv<LZ, NT>(b, G, lri, alias);
  else switch (lz) {
#define BD_CASE(L) case L: res_inv<L, NT>(b, G, lri, alias); break;
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
  }
}
template <int LZ, int NT>
__device__ __forceinline__ void res_fwd_of(int lz, int b, int G, int lrf, bool alias) {
  if constexpr (LZ >= 0) res_fwd<LZ, NT>(b, G, lrf, alias);
  else switch (lz) {
#define BD_CASE(L) case L: res_fwd<L, NT>(b, G, lrf, alias); break;
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
  }
}
template <int LZ, int NT>
__device__ __forceinline__ void res_cols_of(int lz, int b, int G, int lw) {
  if constexpr (LZ >= 0) res_cols<LZ, NT>(b, G, lw);
  else switch (lz) {
#define BD_CASE(L) case L: res_cols<L, NT>(b, G, lw); break;
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
  }
}

// LZ: the mesh side as res_side gives it; 0: the other meshes with a factor 3
// and ideal-gas runs; -1 (RES_GROUPS): any, named by the items.
// KIND: RES_SINGLE: one run, described by the kernel parameter, on one cluster
// or on the whole cooperative grid, 1024 threads per CTA and one CTA per SM.
// RES_CLUSTERS: one cluster per entry of A.items, 512 threads and two CTAs per
// SM. RES_GROUPS: a cooperative grid shared out among the runs, a group of
// CTAs of any size for each with barrier words of its own: CTA k's items
// A.items[2k] (run, item sizes) and A.items[2k + 1] (mesh class, group, rank
// in it, its CTAs); for few runs of uneven weight, which clusters of at most
// 16 CTAs leave to the heaviest.
template <int LZ, int KIND>
__global__ void __launch_bounds__(res_threads(KIND), KIND == RES_CLUSTERS ? 2 : 1) k_resident(const __grid_constant__ ResArgs A) {
  constexpr int NT = res_threads(KIND) / 2;
  constexpr bool SINGLE = KIND == RES_SINGLE, GROUPS = KIND == RES_GROUPS;
  __shared__ int s_tmp[32];
  __shared__ int s_ok;
  const bool grid = GROUPS || (SINGLE && A.grid_mode);
  const Item J = GROUPS ? A.items[2 * blockIdx.x + 1] : Item{LZ, 0, 0, 0};
  const int G = GROUPS ? J.c : grid ? (int)gridDim.x : (int)cluster_size();
  const int b = GROUPS ? J.b : grid ? (int)blockIdx.x : (int)cluster_rank();
  const Item I = SINGLE ? A.one_item : GROUPS ? A.items[2 * blockIdx.x] : A.items[blockIdx.x / (unsigned)G];
  unsigned* bar = GROUPS ? A.bar + 2 * J.a : A.bar;
  {
    static_assert(sizeof(RunDesc) % 4 == 0 && sizeof(RunDesc) <= RES_DESC_BYTES, "copied by words");
    const int* src = SINGLE ? reinterpret_cast<const int*>(&A.one) : reinterpret_cast<const int*>(&A.runs[I.run]);
    for (int k = threadIdx.x; k < (int)(sizeof(RunDesc) / 4); k += 2 * NT) ((int*)res_smem)[k] = src[k];
    __syncthreads();
  }
  const RunDesc& R = res_desc();
  RunDyn* D = A.dyn + I.run;
  const int Z = res_side(LZ) ? res_side(LZ) : R.Z, n = Z >> 1;
  const bool mesh = LZ > 0 || !(R.flags & F_IDGAS);
  // the accumulator shares spec2's memory: its clearing moves to the inverse rows
  const bool alias = (const void*)R.dacc == (const void*)R.spec2;
  const bool adaptive = (R.flags & F_ADAPTIVE) != 0;
  const long long budget = ((volatile RunDyn*)D)->steps_left;
  // a run that failed takes no step (run_failed). One thread looks: a slow
  // CTA may start while a failure of this launch is being marked
  if (threadIdx.x == 0) s_ok = !(((volatile RunDyn*)D)->err & E_BARRIER_TIMEOUT);
  unsigned long long step = ((volatile RunDyn*)D)->step;
  if constexpr (SINGLE) {
    // what the phases read first is requested into L2 ahead of them
    if (threadIdx.x == 0 && mesh) {
      l2_prefetch_share(R.spec2, (size_t)Z * n * sizeof(float4), b, G);
      l2_prefetch_share(R.recA, (size_t)R.N * sizeof(Rec), b, G);
      l2_prefetch_share(R.start, ((size_t)R.C * R.C + 1) * sizeof(int), b, G);
      l2_prefetch_share(R.count, (size_t)R.C * R.C * sizeof(int), b, G);
      if (!alias) l2_prefetch_share(R.dacc, (size_t)Z * Z * sizeof(unsigned long long), b, G);
      l2_prefetch_share(R.green, (size_t)Z * (n + 1) * sizeof(float), b, G);
    }
  }
  if (mesh)
    for (int k = threadIdx.x; k < Z; k += 2 * NT) {
      res_tw()[k] = R.tw[k];
      res_sx(Z)[k] = R.sxt[k];
      if (k <= n) res_sx(Z)[Z + k] = R.syt[k];
    }
  const int nst = (int)min((long long)A.nsteps, budget);
  __syncthreads();
  if (!s_ok) return;
  const int nch = (R.C * R.C + SCAN_CHUNK - 1) / SCAN_CHUNK;
  // an equal contiguous share of the particles per CTA, the first pcap of
  // them in shared memory
  const int per = (R.N + G - 1) / G;
  const int g0 = min(R.N, b * per), g1 = min(R.N, g0 + per), nc = min(g1 - g0, A.pcap);
  // the next step's noise, drawn by the scatter; in recB's memory when no
  // particle of the run goes through it
  float2* noise = per <= A.pcap && !(R.flags & F_NOWCA) ? reinterpret_cast<float2*>(R.recB) : nullptr;
  unsigned ep = 0;
  const bool test = A.skip_barrier > 0 && (!GROUPS || J.a == A.skip_group);
  const unsigned maxp = test ? A.max_polls : BAR_MAX_POLLS;
  auto barrier = [&]() -> bool {
    if (!grid) {
      cluster_barrier();
      return true;
    }
    if (test && A.skip_barrier == (int)ep + 1 && b == A.skip_cta) return false;
    return grid_barrier(bar, ++ep * (unsigned)G, maxp, &D->err, &s_ok);
  };
  const bool rec = SINGLE && A.ts && b == 0 && threadIdx.x == 0;
  int ph = 0;
  if (rec) A.ts[0] = global_ns();
#define BD_BARRIER()      \
  if (!barrier()) return; \
  if (rec) A.ts[++ph] = global_ns()
  const bool lower = threadIdx.x < NT;
#pragma unroll 1
  for (int k = 0; k < nst; k++, step++) {
    if (!lower) res_pairs<NT>(step, g0, nc, k > 0 ? noise : nullptr, A.part_off, A.pcap);
    else if (mesh) res_inv_of<LZ, NT>(J.run, b, G, I.c, alias);
    BD_BARRIER();
    if (!adaptive) {
      // a few particles: several lanes for each
      if (4 * (g1 - g0) <= 2 * NT) res_step<NT, 4>(D, step, g0, g1, nc, mesh, A.part_off, A.pcap);
      else if (2 * (g1 - g0) <= 2 * NT) res_step<NT, 2>(D, step, g0, g1, nc, mesh, A.part_off, A.pcap);
      else res_step<NT, 1>(D, step, g0, g1, nc, mesh, A.part_off, A.pcap);
    } else {
      res_forces<NT>(D, step, g0, g1, nc, A.part_off, A.pcap);
      if (!barrier()) return;
      res_adaptive_move<NT>(D, g0, g1, nc, mesh, A.part_off, A.pcap);
    }
    BD_BARRIER();
    if (!lower) res_scan_phase<NT>(b, G, nch, s_tmp);
    else if (mesh) res_fwd_of<LZ, NT>(J.run, b, G, I.a, alias);
    BD_BARRIER();
    if (!lower) res_place<NT>(D, b, g0, g1, nc, nch, adaptive, k + 1 < nst ? noise : nullptr, step + 1, A.part_off, A.pcap);
    else if (mesh) res_cols_of<LZ, NT>(J.run, b, G, I.b);
    if (k + 1 < nst || (SINGLE && A.ts)) {
      BD_BARRIER();
    }
  }
#undef BD_BARRIER
  if (grid) grid_exit(bar, (unsigned)G);
}

// the kernel's attributes: its largest shared memory, clusters beyond eight CTAs
template <int LZ, int KIND>
int resident_attributes_t() {
  auto* f = k_resident<LZ, KIND>;
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)res_max_smem(KIND));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return (int)e;
}

// with the attributes set: grid mode (cs 0): fills *n with the CTAs that can
// be resident; cluster mode: with the clusters of cs CTAs. Returns 0 or a
// cudaError_t.
template <int LZ, int KIND>
int resident_held_t(size_t smem, int cs, int nsm, int* n) {
  auto* f = k_resident<LZ, KIND>;
  if (smem > res_max_smem(KIND)) return (int)cudaErrorInvalidValue;
  if (cs == 0) {
    int per = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, res_threads(KIND), smem);
    *n = per * nsm;
    return (int)e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(res_threads(KIND));
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaOccupancyMaxActiveClusters(n, f, &cfg);
}

template <int LZ, int KIND>
int launch_resident_t(const ResArgs& A, int nclusters, int cs, int grid, size_t smem, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs ? nclusters * cs : grid);
  cfg.blockDim = dim3(res_threads(KIND));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (cs) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, k_resident<LZ, KIND>, A);
}

#define BD_RES_INSTANTIATE_KIND(L, K)                           \
  template int resident_attributes_t<L, K>();                     \
  template int resident_held_t<L, K>(size_t, int, int, int*);     \
  template int launch_resident_t<L, K>(const ResArgs&, int, int, int, size_t, cudaStream_t);
#define BD_RES_INSTANTIATE(L)            \
  BD_RES_INSTANTIATE_KIND(L, RES_CLUSTERS) \
  BD_RES_INSTANTIATE_KIND(L, RES_SINGLE)

}  // namespace bd
