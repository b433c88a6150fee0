// Register-radix FFT for power-of-two lengths (the particle-mesh transforms
// of meshes with Z = 2^a).
//
// Stockham autosort formulation (Govindaraju et al., "High performance
// discrete Fourier transforms on graphics processors", SC 2008): a pass of
// radix R over a length-N sequence with sub-transform length Ns takes
// butterfly j from elements j + t*N/R, multiplies element t by
// exp(sg*2*pi*i*(j mod Ns)*t/(Ns*R)), transforms the R values in registers
// and writes them to (j div Ns)*Ns*R + (j mod Ns) + t*Ns. Input and output
// are in natural order, so no permutation pass is needed anywhere.
//
// Twiddles of a butterfly: the powers w^(2^b) come from the table, every
// other power is a product of at most four of them (a few ulp in FP32).
//
// Every thread holds E elements per pass (E/R butterflies of radix R), E
// the schedule's largest radix (16, or 8 for lengths 32, 64 and 512 whose
// passes are all radix 8 or less; N below 16: E = N), so a sequence needs
// N/E threads and one pass is: read all elements into registers, barrier,
// compute, write in place, barrier. The passes use radix 16 where possible:
// 2048 = 16*16*8 takes three passes. Which butterflies a thread holds does
// not change any butterfly's arithmetic, so E does not change the results.
//
// Shared-memory layout: sequence b starts at s + b*ss, element e sits at
// pad16(e) = e + e/16 (one float2 of padding per 16), which keeps the
// strided accesses of every pass free of bank conflicts. Twiddles come from
// the run's table tw[m] = exp(-2*pi*i*m/Z) with Z = 2^lz >= N.
#pragma once

#include <cuda_runtime.h>

#include "bd_fft.cuh"

namespace bd {

__device__ __forceinline__ int pad16(int e) { return e + (e >> 4); }

__host__ __device__ constexpr int fft2_stride(int n) { return n + (n >> 4) + 8; }

// Elements a thread holds in a length-2^logn transform: the radix of the
// schedule's first (largest) pass, 2^ceil(logn / ceil(logn / 4)) (Fft2Sched).
__host__ __device__ constexpr int fft2_e(int logn) {
  return logn < 4 ? (1 << logn) : (1 << ((logn + (logn + 3) / 4 - 1) / ((logn + 3) / 4)));
}
// threads one sequence of length 2^logn needs
__host__ __device__ constexpr int fft2_tps(int logn) { return (1 << logn) / fft2_e(logn); }

template <int R>
__device__ __forceinline__ void dftr(float2* v, float sg);

template <>
__device__ __forceinline__ void dftr<2>(float2* v, float) {
  const float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

// X[k] = sum_n v[n] w^(nk), w = exp(sg*2*pi*i/4) = sg*i
template <>
__device__ __forceinline__ void dftr<4>(float2* v, float sg) {
  const float2 s0 = cadd(v[0], v[2]), d0 = csub(v[0], v[2]);
  const float2 s1 = cadd(v[1], v[3]), d1 = csub(v[1], v[3]);
  v[0] = cadd(s0, s1);
  v[2] = csub(s0, s1);
  v[1] = make_float2(d0.x - sg * d1.y, d0.y + sg * d1.x);
  v[3] = make_float2(d0.x + sg * d1.y, d0.y - sg * d1.x);
}

// 8 = 4 x 2: two length-4 transforms of the even and odd elements, then
// X[k] = E[k] + w8^k O[k], X[k+4] = E[k] - w8^k O[k].
template <>
__device__ __forceinline__ void dftr<8>(float2* v, float sg) {
  constexpr float c = 0.70710678118654752440f;  // sqrt(1/2)
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  dftr<4>(e, sg);
  dftr<4>(o, sg);
  // o[k] *= exp(sg*2*pi*i*k/8)
  o[1] = make_float2(c * (o[1].x - sg * o[1].y), c * (o[1].y + sg * o[1].x));
  o[2] = make_float2(-sg * o[2].y, sg * o[2].x);
  o[3] = make_float2(-c * (o[3].x + sg * o[3].y), c * (sg * o[3].x - o[3].y));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = cadd(e[k], o[k]);
    v[k + 4] = csub(e[k], o[k]);
  }
}

// 16 = 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2. Length-4 transforms over n1 for
// each n2, twiddle w16^(n2 k1), length-4 transforms over n2.
template <>
__device__ __forceinline__ void dftr<16>(float2* v, float sg) {
  constexpr float c1 = 0.92387953251128675613f;  // cos(pi/8)
  constexpr float s1 = 0.38268343236508977173f;  // sin(pi/8)
  constexpr float h = 0.70710678118654752440f;   // sqrt(1/2)
  float2 y[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) {
    y[n2][0] = v[n2];
    y[n2][1] = v[n2 + 4];
    y[n2][2] = v[n2 + 8];
    y[n2][3] = v[n2 + 12];
    dftr<4>(y[n2], sg);
  }
  // w16^m = (cos(2 pi m/16), sg sin(2 pi m/16)) for m = n2*k1
  const float2 w1 = make_float2(c1, sg * s1), w2 = make_float2(h, sg * h);
  const float2 w3 = make_float2(s1, sg * c1), w6 = make_float2(-h, sg * h);
  const float2 w9 = make_float2(-c1, -sg * s1);
  y[1][1] = cmul(y[1][1], w1);
  y[1][2] = cmul(y[1][2], w2);
  y[1][3] = cmul(y[1][3], w3);
  y[2][1] = cmul(y[2][1], w2);
  y[2][2] = make_float2(-sg * y[2][2].y, sg * y[2][2].x);  // w16^4 = sg*i
  y[2][3] = cmul(y[2][3], w6);
  y[3][1] = cmul(y[3][1], w3);
  y[3][2] = cmul(y[3][2], w6);
  y[3][3] = cmul(y[3][3], w9);
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++) {
    float2 z[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
    dftr<4>(z, sg);
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++) v[k1 + 4 * k2] = z[k2];
  }
}

// One Stockham pass: radix 2^LOGR, sub-transform length 2^LOGNS, over nseq
// sequences of length 2^LOGN. Threads beyond nseq*N/E only join the barriers.
template <int LOGN, int LOGR, int LOGNS, bool TWS, class Team>
__device__ __forceinline__ void fft2_pass(const Team& T, float2* s, int ss, int nseq, const float2* __restrict__ tw,
                                          int lz, float sg) {
  constexpr int N = 1 << LOGN, R = 1 << LOGR;
  constexpr int E = fft2_e(LOGN);
  static_assert(E >= R && E % R == 0, "a thread holds whole butterflies");
  constexpr int TPS = N / E;  // threads per sequence
  constexpr int NB = E / R;   // butterflies per thread
  constexpr int NR = N / R;
  const int g = T.tid;
  const int b = g / TPS, i = g - b * TPS;
  const bool act = b < nseq;
  float2* q = s + b * ss;
  float2 v[E];
  // set before the branch: left undefined on the idle threads' path, v is kept
  // in local memory across the barrier wherever a loop surrounds the pass
  if constexpr (!Team::ONCE) {
#pragma unroll
    for (int t = 0; t < E; t++) v[t] = make_float2(0.f, 0.f);
  }
  if (act) {
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int t = 0; t < R; t++) v[u * R + t] = q[pad16(u * TPS + i + t * NR)];
  }
  T.sync();
  if (act) {
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int j = u * TPS + i;
      const int k = j & ((1 << LOGNS) - 1);
      if (LOGNS > 0) {
        // w^t for t = 2^b from the table, the others as products of at
        // most four table values (w^t = w^(top bit of t) * w^(rest))
        const int sh = lz - LOGNS - LOGR;
        float2 w[R];
#pragma unroll
        for (int t = 1; t < R; t++) {
          if ((t & (t - 1)) == 0) {
            w[t] = TWS ? tw[(k * t) << sh] : __ldg(&tw[(k * t) << sh]);
            if (sg > 0.f) w[t].y = -w[t].y;
          } else {
            const int hb = 1 << (31 - __clz(t));
            w[t] = cmul(w[hb], w[t - hb]);
          }
          v[u * R + t] = cmul(v[u * R + t], w[t]);
        }
      }
      dftr<R>(&v[u * R], sg);
      const int d = ((j >> LOGNS) << (LOGNS + LOGR)) + k;
#pragma unroll
      for (int t = 0; t < R; t++) q[pad16(d + (t << LOGNS))] = v[u * R + t];
    }
  }
  T.sync();
}

// Pass schedule: ceil(remaining bits / 4) passes left, the bits spread evenly.
// TWS: the twiddle table tw is a copy in shared memory (kernels that loop
// over items keep it there; global-memory twiddle loads would be hoisted
// out of the loop by the compiler and exhaust the registers).
template <int LOGN, int DONE, bool TWS = false>
struct Fft2Sched {
  template <class Team>
  static __device__ __forceinline__ void run(const Team& T, float2* s, int ss, int nseq, const float2* tw,
                                             int lz, float sg) {
    constexpr int rem = LOGN - DONE;
    constexpr int left = (rem + 3) / 4;
    constexpr int bits = (rem + left - 1) / left;
    fft2_pass<LOGN, bits, DONE, TWS>(T, s, ss, nseq, tw, lz, sg);
    Fft2Sched<LOGN, DONE + bits, TWS>::run(T, s, ss, nseq, tw, lz, sg);
  }
};
template <int LOGN, bool TWS>
struct Fft2Sched<LOGN, LOGN, TWS> {
  template <class Team>
  static __device__ __forceinline__ void run(const Team&, float2*, int, int, const float2*, int, float) {}
};

// Fft2Sched<LOGN, 0>::run transforms nseq sequences of length 2^LOGN in
// place (sg = -1 forward, +1 inverse, unnormalised) with nseq * N/E threads;
// the caller syncs before, the last pass ends with a barrier.

// The transform with its first pass reading through ld(b, e) (element e of
// sequence b, straight from global memory: no copy to shared memory and no
// barrier ahead of it) and its last one writing through st(b, e, value). The
// arithmetic is Fft2Sched's. ILV: neighbouring threads take the same elements
// of different sequences (b = thread mod nseq), for sources stored by column.
// OUT_SHARED: st writes shared memory (the reads of the last pass end first).
// 2^lseq sequences, 2^lseq * N/E threads at most; every thread calls; ends
// with a barrier unless the last pass leaves shared memory alone.
// IN_SHARED: the sequences are in shared memory already (ld is not used).
template <int LOGN, int DONE, bool ILV, bool IN_SHARED, bool OUT_SHARED, class Ld, class St>
__device__ __forceinline__ void fft2_through(float2* s, int ss, int lseq, const float2* __restrict__ tw, int lz,
                                             float sg, const Ld& ld, const St& st) {
  constexpr int rem = LOGN - DONE, left = (rem + 3) / 4, LOGR = (rem + left - 1) / left;
  constexpr bool FIRST = DONE == 0 && !IN_SHARED, LAST = DONE + LOGR == LOGN;
  constexpr int N = 1 << LOGN, R = 1 << LOGR, E = fft2_e(LOGN), TPS = N / E, NB = E / R, NR = N / R;
  const int g = threadIdx.x;
  const int b = ILV ? g & ((1 << lseq) - 1) : g / TPS, i = ILV ? g >> lseq : g - b * TPS;
  const bool act = ILV ? i < TPS : b < (1 << lseq);
  float2* q = s + b * ss;
  float2 v[E];
#pragma unroll
  for (int t = 0; t < E; t++) v[t] = make_float2(0.f, 0.f);
  if (act) {
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int t = 0; t < R; t++) {
        const int e = u * TPS + i + t * NR;
        if constexpr (FIRST) v[u * R + t] = ld(b, e);
        else v[u * R + t] = q[pad16(e)];
      }
  }
  if (!FIRST && (!LAST || OUT_SHARED)) __syncthreads();
  if (act) {
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int j = u * TPS + i;
      const int k = j & ((1 << DONE) - 1);
      if (DONE > 0) {
        const int sh = lz - DONE - LOGR;
        float2 w[R];
#pragma unroll
        for (int t = 1; t < R; t++) {
          if ((t & (t - 1)) == 0) {
            w[t] = __ldg(&tw[(k * t) << sh]);
            if (sg > 0.f) w[t].y = -w[t].y;
          } else {
            const int hb = 1 << (31 - __clz(t));
            w[t] = cmul(w[hb], w[t - hb]);
          }
          v[u * R + t] = cmul(v[u * R + t], w[t]);
        }
      }
      dftr<R>(&v[u * R], sg);
      const int d = ((j >> DONE) << (DONE + LOGR)) + k;
#pragma unroll
      for (int t = 0; t < R; t++) {
        const int e = d + (t << DONE);
        if constexpr (LAST) st(b, e, v[u * R + t]);
        else q[pad16(e)] = v[u * R + t];
      }
    }
  }
  if (!LAST || OUT_SHARED) __syncthreads();
  if constexpr (!LAST) fft2_through<LOGN, DONE + LOGR, ILV, IN_SHARED, OUT_SHARED>(s, ss, lseq, tw, lz, sg, ld, st);
}

// The same transform with four elements per thread (N/4 threads per
// sequence), for the resident step, whose transforms are bound by the length
// of one thread's instruction chain: a radix-16 butterfly is shared by four
// neighbouring lanes and a radix-8 one by two, each lane doing one length-4
// transform of dftr<16> / dftr<8> with the same twiddles and products, so
// the results are those of Fft2Sched bit for bit. tw: in shared memory. All
// threads of the team call (N >= 4; a warp's lanes past nseq only join).
// Products of fft4_pass, rounded as fft2_pass's and dftr<16>'s contracted
// products are: real part fma(x, c, -(y s)), imaginary part fma(y, c, x s)
// or (cmul_xs) fma(x, s, y c).
__device__ __forceinline__ float2 cmul_yc(float2 a, float2 w) {
  return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, __fmul_rn(a.x, w.y)));
}
__device__ __forceinline__ float2 cmul_xs(float2 a, float2 w) {
  return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}

template <int LOGN, int LOGR, int LOGNS, class Team>
__device__ __forceinline__ void fft4_pass(const Team& T, float2* s, int ss, int nseq, const float2* tw, int lz,
                                          float sg) {
  constexpr int N = 1 << LOGN, R = 1 << LOGR, NR = N / R, TPS = N / 4;
  constexpr int LB = R >= 4 ? R / 4 : 1;  // lanes per butterfly
  const int b = T.tid / TPS, i = T.tid - b * TPS;
  const bool act = b < nseq;
  float2* q = s + b * ss;
  const int sub = i & (LB - 1), j = i / LB;  // radix 2: butterflies i and i + N/4
  const int k = j & ((1 << LOGNS) - 1);
  constexpr int STEP = R == 2 ? N / 4 : LB * NR;  // between a lane's elements
  float2 v[4];
#pragma unroll
  for (int m = 0; m < 4; m++) v[m] = make_float2(0.f, 0.f);
  if (act) {
#pragma unroll
    for (int m = 0; m < 4; m++) v[m] = q[pad16(j + sub * NR + m * STEP)];
    if (LOGNS > 0) {
      const int sh = lz - LOGNS - LOGR;
      // products of two table values (conjugated for the inverse)
      auto ww = [&](float2 a, float2 c) { return sg < 0.f ? cmul_yc(a, c) : cmul_xs(a, c); };
      auto W = [&](int t) {
        float2 w = tw[(k * t) << sh];
        if (sg > 0.f) w.y = -w.y;
        return w;
      };
      if (R == 2) {
        // elements (i, i + N/2) and (i + N/4, i + 3N/4) of butterflies i and
        // i + N/4
        const int k2 = (j + N / 4) & ((1 << LOGNS) - 1);
        v[2] = cmul_yc(v[2], W(1));
        float2 w = tw[k2 << sh];
        if (sg > 0.f) w.y = -w.y;
        v[3] = cmul_yc(v[3], w);
      } else if (R == 4) {
        const float2 w1 = W(1), w2 = W(2);
        v[1] = cmul_yc(v[1], w1);
        v[2] = cmul_yc(v[2], w2);
        v[3] = cmul_yc(v[3], ww(w2, w1));
      } else if (R == 8) {
        const float2 w1 = W(1), w2 = W(2), w4 = W(4);
        const float2 x1 = sub ? ww(w2, w1) : w2, x2 = sub ? ww(w4, w1) : w4;
        if (sub) v[0] = cmul_yc(v[0], w1);
        v[1] = cmul_yc(v[1], x1);
        v[2] = cmul_yc(v[2], x2);
        v[3] = cmul_yc(v[3], ww(w4, x1));
      } else {
        const float2 w1 = W(1), w2 = W(2), w4 = W(4), w8 = W(8);
        const float2 w3 = ww(w2, w1);
        const float2 wn = sub == 1 ? w1 : sub == 2 ? w2 : w3;
        const float2 x1 = sub ? ww(w4, wn) : w4, x2 = sub ? ww(w8, wn) : w8;
        if (sub) v[0] = cmul_yc(v[0], wn);
        v[1] = cmul_yc(v[1], x1);
        v[2] = cmul_yc(v[2], x2);
        v[3] = cmul_yc(v[3], ww(w8, x1));
      }
    }
  }
  if (R == 2) {
    const float2 a = v[0], c = v[1];
    v[0] = cadd(a, v[2]);
    v[1] = csub(a, v[2]);
    v[2] = cadd(c, v[3]);
    v[3] = csub(c, v[3]);
  } else {
    dftr<4>(v, sg);
  }
  if (R == 8) {
    constexpr float c = 0.70710678118654752440f;  // sqrt(1/2)
    // the even lane keeps E + w O, the odd lane E - w O. The factor sqrt(1/2)
    // of w^1 and w^3 is applied inside the sum, fma(+-c, u, e), as dftr<8>'s
    // products are (contracted into its additions)
    if (sub) {
      v[1] = make_float2(v[1].x - sg * v[1].y, v[1].y + sg * v[1].x);
      v[2] = make_float2(-sg * v[2].y, sg * v[2].x);
      v[3] = make_float2(v[3].x + sg * v[3].y, sg * v[3].x - v[3].y);
    }
    const float cc = sub ? -c : c;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const float ox = __shfl_xor_sync(0xffffffffu, v[m].x, 1), oy = __shfl_xor_sync(0xffffffffu, v[m].y, 1);
      if (m & 1) {
        v[m] = make_float2(__fmaf_rn(m == 1 ? cc : -cc, sub ? v[m].x : ox, sub ? ox : v[m].x),
                           __fmaf_rn(cc, sub ? v[m].y : oy, sub ? oy : v[m].y));
      } else {
        v[m] = make_float2(ox + (sub ? -v[m].x : v[m].x), oy + (sub ? -v[m].y : v[m].y));
      }
    }
  }
  if (R == 16) {
    constexpr float c1 = 0.92387953251128675613f;  // cos(pi/8)
    constexpr float s1 = 0.38268343236508977173f;  // sin(pi/8)
    constexpr float h = 0.70710678118654752440f;   // sqrt(1/2)
    const float2 w1 = make_float2(c1, sg * s1), w2 = make_float2(h, sg * h);
    const float2 w3 = make_float2(s1, sg * c1), w6 = make_float2(-h, sg * h);
    const float2 w9 = make_float2(-c1, -sg * s1);
    if (sub) {
      // (products with dftr<16>'s constants: w1 and w3 of the forward
      // transform round as cmul_yc, the others as cmul_xs)
      auto mul = [](float2 a, float2 w, bool d) {
        const float2 p = cmul_xs(a, w), q = cmul_yc(a, w);
        return make_float2(p.x, d ? q.y : p.y);
      };
      const bool fw = sg < 0.f;
      const float2 r2 = make_float2(-sg * v[2].y, sg * v[2].x);  // w16^4 = sg*i
      v[1] = mul(v[1], sub == 1 ? w1 : sub == 2 ? w2 : w3, fw && sub != 2);
      v[2] = sub == 2 ? r2 : mul(v[2], sub == 1 ? w2 : w6, false);
      v[3] = mul(v[3], sub == 1 ? w3 : sub == 2 ? w6 : w9, fw && sub == 1);
    }
    // 4x4 transpose between the four lanes through their own slots
    if (act) {
#pragma unroll
      for (int m = 0; m < 4; m++) q[pad16(j + sub * NR + m * STEP)] = v[m];
    }
    __syncwarp();
    if (act) {
#pragma unroll
      for (int m = 0; m < 4; m++) v[m] = q[pad16(j + (m + 4 * sub) * NR)];
    }
    dftr<4>(v, sg);
  }
  T.sync();
  if (act) {
    if (R == 2) {
      const int j2 = j + N / 4, k2 = j2 & ((1 << LOGNS) - 1);
      const int d = ((j >> LOGNS) << (LOGNS + 1)) + k, d2 = ((j2 >> LOGNS) << (LOGNS + 1)) + k2;
      q[pad16(d)] = v[0];
      q[pad16(d + (1 << LOGNS))] = v[1];
      q[pad16(d2)] = v[2];
      q[pad16(d2 + (1 << LOGNS))] = v[3];
    } else {
      const int d = ((j >> LOGNS) << (LOGNS + LOGR)) + k;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int t = R == 16 ? sub + 4 * m : R == 8 ? m + 4 * sub : m;
        q[pad16(d + (t << LOGNS))] = v[m];
      }
    }
  }
  T.sync();
}

template <int LOGN, int DONE>
struct Fft4Sched {
  template <class Team>
  static __device__ __forceinline__ void run(const Team& T, float2* s, int ss, int nseq, const float2* tw,
                                             int lz, float sg) {
    constexpr int rem = LOGN - DONE;
    constexpr int left = (rem + 3) / 4;
    constexpr int bits = (rem + left - 1) / left;
    fft4_pass<LOGN, bits, DONE>(T, s, ss, nseq, tw, lz, sg);
    Fft4Sched<LOGN, DONE + bits>::run(T, s, ss, nseq, tw, lz, sg);
  }
};
template <int LOGN>
struct Fft4Sched<LOGN, LOGN> {
  template <class Team>
  static __device__ __forceinline__ void run(const Team&, float2*, int, int, const float2*, int, float) {}
};

__host__ __device__ constexpr int fft4_tps(int logn) { return (1 << logn) / 4; }

}  // namespace bd
