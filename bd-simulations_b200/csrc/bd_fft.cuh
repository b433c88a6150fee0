// Shared-memory FFT building blocks for the particle-mesh path.
//
// A CTA transforms `nseq` sequences of length n = 2^a 3^b that sit
// interleaved in shared memory: element e of sequence b is s[e*nseq + b]
// (nseq a power of two). Forward transforms use decimation in frequency
// (natural order in, digit-reversed order out), inverse transforms use
// decimation in time (digit-reversed order in, natural order out). A
// forward/inverse pair therefore needs no permutation pass: whatever acts
// between them (the Green's-function multiply) finds spectrum index k at
// position fft_pos(k).
//
// Stages use radix 4, 2 and 3 (FftPlan::r, in decimation-in-frequency
// order). Twiddles come from the run's table tw[t] = exp(-2 pi i t / Z); a
// length-n transform with n | Z reads it with stride Z/n.
#pragma once

#include <cuda_runtime.h>

namespace bd {

struct FftPlan {
  int n;
  int ns;
  int r[16];
  int pow2;    // every radix a power of two: block indices by shifts
  int lh[16];  // log2 of the butterfly span h = m/r of stage q (pow2 plans)
};

// The threads that work on one item together: a whole CTA, or half of one
// with a named barrier of its own, so that the two halves of a resident CTA
// work on different things between group barriers. tid: index in the team.
struct CtaTeam {
  static constexpr bool ONCE = false;  // no loop around the transforms
  int tid;
  __device__ __forceinline__ CtaTeam() : tid((int)threadIdx.x) {}
  __device__ __forceinline__ int nt() const { return (int)blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
};
// the CTA where no transform is in a loop: the values of idle threads need not
// be set (one-step launch after an L2 flush, 65 536 particles 32.2 -> 31.5 us)
struct OnceTeam : CtaTeam {
  static constexpr bool ONCE = true;
};
// half ID (0: the lower threads) of a CTA of 2*NT threads, NT a power of two
template <int ID, int NT>
struct HalfTeam {
  static constexpr bool ONCE = false;
  int tid;
  __device__ __forceinline__ HalfTeam() {
    // the index is opaque to the compiler: an item loop around a transform
    // would otherwise keep every pass's per-thread addresses live and spill
    unsigned t = threadIdx.x;
    asm volatile("" : "+r"(t));
    tid = (int)(t & (unsigned)(NT - 1));
  }
  __device__ __forceinline__ int nt() const { return NT; }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"n"(ID + 1), "n"(NT) : "memory"); }
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// frequency k -> storage position after the forward (DIF) transform
__device__ __forceinline__ int fft_pos(const FftPlan& P, int k) {
  int m = P.n, pos = 0;
  for (int q = 0; q < P.ns; q++) {
    const int r = P.r[q];
    m /= r;
    pos += (k % r) * m;
    k /= r;
  }
  return pos;
}

// storage position -> frequency
__device__ __forceinline__ int fft_freq(const FftPlan& P, int pos) {
  int m = P.n, k = 0, mul = 1;
  for (int q = 0; q < P.ns; q++) {
    const int r = P.r[q];
    m /= r;
    k += ((pos / m) % r) * mul;
    mul *= r;
  }
  return k;
}

// in-register DFT of radix r (2, 3, 4); sg = -1 forward, +1 inverse
__device__ __forceinline__ void dft_small(float2* v, int r, float sg) {
  if (r == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if (r == 4) {
    const float2 s0 = cadd(v[0], v[2]), d0 = csub(v[0], v[2]);
    const float2 s1 = cadd(v[1], v[3]), d1 = csub(v[1], v[3]);
    v[0] = cadd(s0, s1);
    v[2] = csub(s0, s1);
    // V1 = d0 + sg*i*d1, V3 = d0 - sg*i*d1
    v[1] = make_float2(d0.x - sg * d1.y, d0.y + sg * d1.x);
    v[3] = make_float2(d0.x + sg * d1.y, d0.y - sg * d1.x);
  } else {  // 3
    const float sn = sg * 0.866025403784438646763723f;
    const float2 t1 = cadd(v[1], v[2]);
    const float2 t2 = make_float2(v[0].x - 0.5f * t1.x, v[0].y - 0.5f * t1.y);
    const float2 t3 = make_float2(sn * (v[1].x - v[2].x), sn * (v[1].y - v[2].y));
    v[0] = cadd(v[0], t1);
    v[1] = make_float2(t2.x - t3.y, t2.y + t3.x);
    v[2] = make_float2(t2.x + t3.y, t2.y - t3.x);
  }
}

// Decimation-in-frequency stages. inv selects the sign (+1 when true).
// Caller syncs before; every stage ends with a sync of the team. TWS: tw is
// a copy in shared memory.
template <bool TWS, class Team>
__device__ __forceinline__ void fft_dif(const Team& T, float2* s, const FftPlan& P, int lognseq,
                                        const float2* tw, int twstride, bool inv) {
  const int n = P.n, nseq = 1 << lognseq;
  const float sg = inv ? 1.f : -1.f;
  int m = n;
  for (int q = 0; q < P.ns; q++) {
    const int r = P.r[q];
    const int h = m / r;
    const int tws = (n / m) * twstride;
    const int total = (n / r) << lognseq;
    for (int idx = T.tid; idx < total; idx += T.nt()) {
      const int b = idx & (nseq - 1);
      const int qq = idx >> lognseq;
      const int g = P.pow2 ? (qq >> P.lh[q]) : qq / h;
      const int e = qq - g * h;
      const int base = g * m + e;
      float2 v[4];
#pragma unroll
      for (int t = 0; t < 4; t++)
        if (t < r) v[t] = s[((base + t * h) << lognseq) | b];
      dft_small(v, r, sg);
#pragma unroll
      for (int u = 1; u < 4; u++)
        if (u < r) {
          float2 w = TWS ? tw[e * u * tws] : __ldg(&tw[e * u * tws]);
          if (inv) w.y = -w.y;
          v[u] = cmul(v[u], w);
        }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (u < r) s[((base + u * h) << lognseq) | b] = v[u];
    }
    T.sync();
    m = h;
  }
}

// Decimation-in-time stages: the forward stages undone in reverse order.
template <bool TWS, class Team>
__device__ __forceinline__ void fft_dit(const Team& T, float2* s, const FftPlan& P, int lognseq,
                                        const float2* tw, int twstride, bool inv) {
  const int n = P.n, nseq = 1 << lognseq;
  const float sg = inv ? 1.f : -1.f;
  int m = 1;
  for (int q = P.ns - 1; q >= 0; q--) {
    const int r = P.r[q];
    m *= r;  // block size of DIF stage q
    const int h = m / r;
    const int tws = (n / m) * twstride;
    const int total = (n / r) << lognseq;
    for (int idx = T.tid; idx < total; idx += T.nt()) {
      const int b = idx & (nseq - 1);
      const int qq = idx >> lognseq;
      const int g = P.pow2 ? (qq >> P.lh[q]) : qq / h;
      const int e = qq - g * h;
      const int base = g * m + e;
      float2 v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (u < r) v[u] = s[((base + u * h) << lognseq) | b];
#pragma unroll
      for (int u = 1; u < 4; u++)
        if (u < r) {
          float2 w = TWS ? tw[e * u * tws] : __ldg(&tw[e * u * tws]);
          if (inv) w.y = -w.y;
          v[u] = cmul(v[u], w);
        }
      dft_small(v, r, sg);
#pragma unroll
      for (int t = 0; t < 4; t++)
        if (t < r) s[((base + t * h) << lognseq) | b] = v[t];
    }
    T.sync();
  }
}

// The same transforms for a length known at compile time (the resident step's
// meshes of 3 * 2^k points a side): index arithmetic by constants, one
// butterfly per thread and stage where the team has enough threads. Sequence b
// starts at s + b*N, elements in order; the arithmetic of every butterfly is
// fft_dif's and fft_dit's, so are the results. tw: in shared memory, read with
// stride TWS (tw[t] = exp(-2 pi i t/(N*TWS))).
__host__ __device__ constexpr int fftc_radix(int m) { return m % 4 == 0 ? 4 : m % 2 == 0 ? 2 : 3; }

template <int N, int M, int TWS, bool DIT, class Team>
__device__ __forceinline__ void fftc_stage(const Team& T, float2* s, int nseq, const float2* tw) {
  constexpr int r = fftc_radix(M), h = M / r, per = N / r, st = (N / M) * TWS;
  constexpr float sg = DIT ? 1.f : -1.f;
  const int total = nseq * per;
  for (int idx = T.tid; idx < total; idx += T.nt()) {
    const int b = idx / per, qq = idx - b * per;
    const int g = qq / h, e = qq - g * h;
    float2* q = s + b * N + g * M + e;
    float2 v[4];
#pragma unroll
    for (int t = 0; t < r; t++) v[t] = q[t * h];
    if (!DIT) dft_small(v, r, sg);
#pragma unroll
    for (int u = 1; u < r; u++) {
      float2 w = tw[e * u * st];
      if (DIT) w.y = -w.y;
      v[u] = cmul(v[u], w);
    }
    if (DIT) dft_small(v, r, sg);
#pragma unroll
    for (int t = 0; t < r; t++) q[t * h] = v[t];
  }
  T.sync();
}
// Two stages of a transform in one pass: a thread holds the r1*r2 elements that
// stage M (radix r1) and the stage below it (radix r2, block M/r1) exchange
// among themselves, so shared memory is read and written once for both.
template <int N, int M, int TWS, bool DIT, class Team>
__device__ __forceinline__ void fftc_stage2(const Team& T, float2* s, int nseq, const float2* tw) {
  constexpr int r1 = fftc_radix(M), h1 = M / r1, r2 = fftc_radix(h1), h2 = h1 / r2, per = N / (r1 * r2);
  constexpr int st1 = (N / M) * TWS, st2 = (N / h1) * TWS;
  constexpr float sg = DIT ? 1.f : -1.f;
  const int total = nseq * per;
  for (int idx = T.tid; idx < total; idx += T.nt()) {
    const int b = idx / per, qq = idx - b * per;
    const int g = qq / h2, e2 = qq - g * h2;
    float2* q = s + b * N + g * M + e2;
    float2 v[r1][r2];
#pragma unroll
    for (int a = 0; a < r1; a++)
#pragma unroll
      for (int c = 0; c < r2; c++) v[a][c] = q[a * h1 + c * h2];
    auto upper = [&]() {  // stage M, over a, at e = e2 + c*h2
#pragma unroll
      for (int c = 0; c < r2; c++) {
        const int e = e2 + c * h2;
        float2 x[4];
#pragma unroll
        for (int a = 0; a < r1; a++) x[a] = v[a][c];
        if (!DIT) dft_small(x, r1, sg);
#pragma unroll
        for (int u = 1; u < r1; u++) {
          float2 w = tw[e * u * st1];
          if (DIT) w.y = -w.y;
          x[u] = cmul(x[u], w);
        }
        if (DIT) dft_small(x, r1, sg);
#pragma unroll
        for (int a = 0; a < r1; a++) v[a][c] = x[a];
      }
    };
    auto lower = [&]() {  // the stage below, over c, at e2
#pragma unroll
      for (int a = 0; a < r1; a++) {
        float2 x[4];
#pragma unroll
        for (int c = 0; c < r2; c++) x[c] = v[a][c];
        if (!DIT) dft_small(x, r2, sg);
#pragma unroll
        for (int u = 1; u < r2; u++) {
          float2 w = tw[e2 * u * st2];
          if (DIT) w.y = -w.y;
          x[u] = cmul(x[u], w);
        }
        if (DIT) dft_small(x, r2, sg);
#pragma unroll
        for (int c = 0; c < r2; c++) v[a][c] = x[c];
      }
    };
    if (DIT) {
      lower();
      upper();
    } else {
      upper();
      lower();
    }
#pragma unroll
    for (int a = 0; a < r1; a++)
#pragma unroll
      for (int c = 0; c < r2; c++) q[a * h1 + c * h2] = v[a][c];
  }
  T.sync();
}
// whether the pass at block m takes two stages: wherever a second one is left
// (70 000 particles on 768^2 52.6 -> 45.0 us per step, 16 adaptive runs 77 ->
// 69; a single stage a pass had a barrier and a round through shared memory
// for each)
__host__ __device__ constexpr bool fftc_pair(int m) { return m / fftc_radix(m) > 1; }

// forward, natural order in, digit-reversed out
template <int N, int TWS, int M = N>
struct FftcDif {
  template <class Team>
  static __device__ __forceinline__ void run(const Team& T, float2* s, int nseq, const float2* tw) {
    if constexpr (M > 1) {
      constexpr int M1 = M / fftc_radix(M);
      if constexpr (fftc_pair(M)) {
        fftc_stage2<N, M, TWS, false>(T, s, nseq, tw);
        FftcDif<N, TWS, M1 / fftc_radix(M1)>::run(T, s, nseq, tw);
      } else {
        fftc_stage<N, M, TWS, false>(T, s, nseq, tw);
        FftcDif<N, TWS, M1>::run(T, s, nseq, tw);
      }
    }
  }
  // frequency -> storage position, and back (fft_pos, fft_freq)
  static __device__ __forceinline__ int pos(int k) {
    if constexpr (M > 1) {
      constexpr int r = fftc_radix(M), h = M / r;
      return (k % r) * h + FftcDif<N, TWS, h>::pos(k / r);
    } else {
      return 0;
    }
  }
  static __device__ __forceinline__ int freq(int p) {
    if constexpr (M > 1) {
      constexpr int r = fftc_radix(M), h = M / r;
      return p / h + r * FftcDif<N, TWS, h>::freq(p % h);
    } else {
      return 0;
    }
  }
};
// inverse, digit-reversed in, natural order out
template <int N, int TWS, int M = N>
struct FftcDit {
  template <class Team>
  static __device__ __forceinline__ void run(const Team& T, float2* s, int nseq, const float2* tw) {
    if constexpr (M > 1) {
      constexpr int M1 = M / fftc_radix(M);
      if constexpr (fftc_pair(M)) {
        FftcDit<N, TWS, M1 / fftc_radix(M1)>::run(T, s, nseq, tw);
        fftc_stage2<N, M, TWS, true>(T, s, nseq, tw);
      } else {
        FftcDit<N, TWS, M1>::run(T, s, nseq, tw);
        fftc_stage<N, M, TWS, true>(T, s, nseq, tw);
      }
    }
  }
};

}  // namespace bd
