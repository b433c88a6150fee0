// Device functions of one step, shared by the stage kernels (bd_kernels.cu)
// and the resident step kernel (bd_resident.cuh): mesh transforms of one
// item, the physics of one particle, pieces of the cell sort, the grid
// barrier.
#pragma once

#include <cstdint>
#include <cuda/atomic>
#include <cuda_runtime.h>

#include "bd_common.cuh"
#include "bd_fft.cuh"
#include "bd_fft2.cuh"
#include "bd_kernels.h"

namespace bd {

__device__ __forceinline__ int wrapi(int a, int m) {
  a %= m;
  return a < 0 ? a + m : a;
}

// a in (-m, 2m) into [0, m)
__device__ __forceinline__ int wrap1(int a, int m) {
  return a < 0 ? a + m : (a >= m ? a - m : a);
}

// A bounded wait of a step of this run gave up: its cell counts, chunk totals
// and density sums may hold half a step. No step form and no sort touches the
// run until the host has put it back (Engine::recover_fused); a second move
// would count its particles twice and the scatter write past its records.
__device__ __forceinline__ bool run_failed(const RunDyn* dyn, int run) {
  return (dyn[run].err & E_BARRIER_TIMEOUT) != 0;
}

// One read of budget and error: looking at the error behind the budget cost
// every block a round trip more (us per step of a whole call, two reads | one:
// 2.1 M particles 267 | 259, 256-run ensemble 587 | 583).
__device__ __forceinline__ bool run_active(const RunDyn* dyn, int run) {
  const int4 v = *reinterpret_cast<const int4*>(&dyn[run].steps_left);
  const long long left = (long long)(((unsigned long long)(unsigned)v.y << 32) | (unsigned)v.x);
  return (left > 0) & ((v.z & E_BARRIER_TIMEOUT) == 0);
}

// Load of data that earlier kernels wrote: through the read-only cache when
// NC, or a plain (coherent) load where the same kernel also writes it (the
// resident step).
template <bool NC, class T>
__device__ __forceinline__ T ldm(const T* p) {
  if constexpr (NC) return __ldg(p);
  else return *p;
}

// 2^e for a normal exponent
__device__ __forceinline__ double pow2_double(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Exclusive scan over a team (any multiple of 32 threads up to 1024);
// sh: 32 ints of shared scratch. All threads must call it.
template <class Team>
__device__ __forceinline__ int team_excl_scan(const Team& T, int v, int* sh) {
  const int lane = T.tid & 31, w = T.tid >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  T.sync();
  if (w == 0) {
    int s = lane < (T.nt() >> 5) ? sh[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sh[lane] = s;
  }
  T.sync();
  const int base = w > 0 ? sh[w - 1] : 0;
  const int r = base + x - v;
  T.sync();
  return r;
}

__device__ inline int block_excl_scan(int v, int* sh) { return team_excl_scan(CtaTeam(), v, sh); }

// Integer adds whose old value nobody wants (atomicAdd was compiled to the
// form that returns it: 256-run ensemble, particle kernel 336 -> 328 us).
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v) : "memory");
}
__device__ __forceinline__ void red_add(int* p, int v) {
  asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}

// The same contributions as deposit_tile, of one particle, added straight to
// the accumulator R.dacc with 64-bit integer atomics (mesh point k*Z + l); the
// integer sums, and so the density, are those of the tiles. LANES lanes share
// a particle's nine points (neighbouring lanes take neighbouring points of a
// row, which the memory system merges); sub: this lane's index among them.
template <int LANES>
__device__ __forceinline__ void deposit_acc(const RunDesc& R, const Rec& p, int sub = 0) {
  int ic, jc;
  cell_ij(R, p.cell, ic, jc);
  int k, l;
  float tx, ty;
  mesh_axis(R, ic, p.ox, k, tx);
  mesh_axis(R, jc, p.oy, l, ty);
  const float scale = __int_as_float((127 + R.fx_shift) << 23);
  const float q = p.pid < R.N1 ? 1.0f : R.q2;
  unsigned long long* acc = R.dacc;
  if (R.scheme == NGP) {
    float c = R.drho;
    if (p.pid >= R.N1) c *= q;
    if (sub == 0)
      red_add(&acc[(size_t)k * R.Z + l], (unsigned long long)(long long)__float2int_rn(c * scale));
    return;
  }
  float wx[3], wy[3];
  axis_weights(R.scheme, tx, wx);
  axis_weights(R.scheme, ty, wy);
  if (LANES == 1) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const size_t row = (size_t)wrap1(k + a - 1, R.Z) * R.Z;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        float c = wx[a] * wy[b] * R.drho;
        if (p.pid >= R.N1) c *= q;
        red_add(&acc[row + wrap1(l + b - 1, R.Z)], (unsigned long long)(long long)__float2int_rn(c * scale));
      }
    }
    return;
  }
  const int ks[3] = {wrap1(k - 1, R.Z), k, wrap1(k + 1, R.Z)}, ls[3] = {wrap1(l - 1, R.Z), l, wrap1(l + 1, R.Z)};
#pragma unroll
  for (int t0 = 0; t0 < 9; t0 += LANES) {
    // point t0 + sub of the nine, row-major
    int row = ks[t0 / 3], col = ls[t0 % 3];
    float x = wx[t0 / 3], y = wy[t0 % 3];
#pragma unroll
    for (int u = 1; u < LANES; u++)
      if (sub == u) {
        const int t = t0 + u < 9 ? t0 + u : 8;
        row = ks[t / 3], col = ls[t % 3], x = wx[t / 3], y = wy[t % 3];
      }
    float c = x * y * R.drho;
    if (p.pid >= R.N1) c *= q;
    const int v = __float2int_rn(c * scale);
    // CIC weighs five of the nine points with zero: no atomic for those
    if (v != 0 && t0 + sub < 9) red_add(&acc[(size_t)row * R.Z + col], (unsigned long long)(long long)v);
  }
}

// ---------------------------------------------------------------------------
// Power-of-two meshes: the same three passes with the register-radix
// Stockham transform (bd_fft2.cuh), natural order throughout. Items are
// sized on the host so that one item's sequences need at most blockDim.x
// threads.

// Row pass, forward, of rows row0 .. row0 + 2^lr - 1 (layout as
// k_fft_rows_fwd). tw: the run's twiddle table, in shared memory when TWS.
// FROM_ACC (pipelined step): the rows come from the fixed-point accumulator
// R.dacc, converted as deposit_tile converts its sums; the density is also
// stored to R.rho and the accumulator words are cleared for the next step.
template <int LZ, bool TWS, bool FROM_ACC, class Team>
__device__ __forceinline__ void fft2_rows_fwd_item(const Team& T, const RunDesc& R, int row0, int lr, float2* s,
                                                   const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1, lz = LZ, ln = LZ - 1;
  constexpr int ss = fft2_stride(n);
  float2* src = reinterpret_cast<float2*>(R.rho) + (size_t)row0 * n;
  if (FROM_ACC) {
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(R.dacc) + (size_t)row0 * n;
    const double inv = 1.0 / (double)__int_as_float((127 + R.fx_shift) << 23);
    for (int i = T.tid; i < (n << lr); i += T.nt()) {
      const int b = i >> ln, m = i & (n - 1);
      const ulonglong2 a = acc[i];
      const float2 v = make_float2((float)((double)(long long)a.x * inv), (float)((double)(long long)a.y * inv));
      s[b * ss + pad16(m)] = v;
      src[i] = v;
      acc[i] = make_ulonglong2(0ull, 0ull);
    }
  } else {
    for (int i = T.tid; i < (n << lr); i += T.nt()) {
      const int b = i >> ln, m = i & (n - 1);
      s[b * ss + pad16(m)] = src[i];
    }
  }
  T.sync();
  Fft2Sched<LZ - 1, 0, TWS>::run(T, s, ss, 1 << lr, tw, lz, -1.f);
  // the half spectrum is stored by column (slot j of row k at spec[j*Z + k]),
  // so the column pass reads whole columns. Consecutive threads take groups
  // of rb = min(2^lr, 4) consecutive rows of one slot (a whole 32-byte sector
  // of a column from 4 rows on), then the next slot: at most rb-way bank
  // conflicts on the rows' shared-memory reads.
  const int lrb = lr < 2 ? lr : 2;
  const int rbm = (1 << lrb) - 1;
  for (int i = T.tid; i < (n << lr); i += T.nt()) {
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
      out = cadd(E, cmul(TWS ? tw[j] : __ldg(&tw[j]), O));
    }
    R.spec[(size_t)j * Z + row0 + b] = out;
  }
  T.sync();
}

// Green's multiply of the packed column (ky = 0 and ky = Z/2 travel as
// C = A + iB): split with the partner Cm = C[-kx], multiply A and B by
// i*s*g with their own factors, pack the Fx and Fy results again.
__device__ __forceinline__ void packed_green(const RunDesc& R, int kx, float2 Cv, float2 Cm, int n, int Z,
                                             float sy0, float syn, float2& P, float2& Q) {
  // A = (C + conj Cm)/2 ; B = (C - conj Cm)/(2i)
  const float2 A = make_float2(0.5f * (Cv.x + Cm.x), 0.5f * (Cv.y - Cm.y));
  const float2 Bv = make_float2(0.5f * (Cv.y + Cm.y), -0.5f * (Cv.x - Cm.x));
  const float gA = __ldg(&R.green[kx]);
  const float gB = __ldg(&R.green[(size_t)n * Z + kx]);
  const float sx = __ldg(&R.sxt[kx]);
  const float2 FxA = make_float2(-sx * gA * A.y, sx * gA * A.x);
  const float2 FxB = make_float2(-sx * gB * Bv.y, sx * gB * Bv.x);
  const float2 FyA = make_float2(-sy0 * gA * A.y, sy0 * gA * A.x);
  const float2 FyB = make_float2(-syn * gB * Bv.y, syn * gB * Bv.x);
  P = make_float2(FxA.x - FxB.y, FxA.y + FxB.x);
  Q = make_float2(FyA.x - FyB.y, FyA.y + FyB.x);
}

// Column pass (as k_fft_cols) of the 2^lw adjacent half-spectrum columns
// from col0; smem holds 2 * 2^lw sequences.
template <int LZ, bool TWS, class Team>
__device__ __forceinline__ void fft2_cols_item(const Team& T, const RunDesc& R, int col0, int lw, float2* sA, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1, lz = LZ;
  constexpr int ss = fft2_stride(Z);
  const int W = 1 << lw;
  float2* sB = sA + W * ss;
  // the row pass stored the half spectrum by column: whole columns are read
  const float2* src = R.spec + (size_t)col0 * Z;
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int c = i >> lz, k = i & (Z - 1);
    sA[c * ss + pad16(k)] = src[i];
  }
  T.sync();
  Fft2Sched<LZ, 0, TWS>::run(T, sA, ss, W, tw, lz, -1.f);
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int c = i >> lz, kx = i & (Z - 1);
    const int j = col0 + c;
    if (j == 0) continue;
    const float g = __ldg(&R.green[(size_t)j * Z + kx]);
    const float gx = __ldg(&R.sxt[kx]) * g;
    const float gy = __ldg(&R.syt[j]) * g;
    const int a = c * ss + pad16(kx);
    const float2 v = sA[a];
    sA[a] = make_float2(-gx * v.y, gx * v.x);
    sB[a] = make_float2(-gy * v.y, gy * v.x);
  }
  if (col0 == 0) {
    // packed column (ky = 0, ky = Z/2): C = A + iB. Element kx of A, B
    // needs C[kx] and C[-kx], so one thread handles both of a pair and
    // writes them in place.
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
  if (2 * W * fft2_tps(lz) <= T.nt()) {
    Fft2Sched<LZ, 0, TWS>::run(T, sA, ss, 2 * W, tw, lz, 1.f);  // sB follows sA: 2W sequences
  } else {
    Fft2Sched<LZ, 0, TWS>::run(T, sA, ss, W, tw, lz, 1.f);
    Fft2Sched<LZ, 0, TWS>::run(T, sB, ss, W, tw, lz, 1.f);
  }
  for (int i = T.tid; i < (Z << lw); i += T.nt()) {
    const int k = i >> lw, c = i & (W - 1);
    const float2 a = sA[c * ss + pad16(k)], b = sB[c * ss + pad16(k)];
    R.spec2[(size_t)k * n + col0 + c] = make_float4(a.x, a.y, b.x, b.y);
  }
  T.sync();
}

// Row pass, inverse (as k_fft_rows_inv), of rows row0 .. row0 + 2^lr - 1.
template <int LZ, bool TWS, class Team>
__device__ __forceinline__ void fft2_rows_inv_item(const Team& T, const RunDesc& R, int row0, int lr, float2* s, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1, lz = LZ;
  constexpr int ss = fft2_stride(Z);
  for (int i = T.tid; i < (Z << lr); i += T.nt()) {
    const int b = i >> lz, j = i & (Z - 1);
    const float4* rb = R.spec2 + (size_t)(row0 + b) * n;
    float2 h;
    if (j == 0) {
      const float4 v = rb[0];
      h = make_float2(v.x, v.z);
    } else if (j == n) {
      const float4 v = rb[0];
      h = make_float2(v.y, v.w);
    } else if (j < n) {
      const float4 v = rb[j];
      h = make_float2(v.x - v.w, v.y + v.z);
    } else {
      const float4 v = rb[Z - j];
      h = make_float2(v.x + v.w, -v.y + v.z);
    }
    s[b * ss + pad16(j)] = h;
  }
  T.sync();
  Fft2Sched<LZ, 0, TWS>::run(T, s, ss, 1 << lr, tw, lz, 1.f);
  float2* dst = R.H + (size_t)row0 * Z;
  for (int i = T.tid; i < (Z << lr); i += T.nt()) {
    const int b = i >> lz, l = i & (Z - 1);
    dst[i] = s[b * ss + pad16(l)];
  }
  T.sync();
}

// The three passes of meshes of 2048 and 4096 points a side (256 threads): the
// first transform pass of each reads global memory and the last one writes it
// (fft2_through), and spec2 is stored by column, point (slot j, row k) at
// j*Z + k, so that a column is written whole whatever number of columns an item
// has; the inverse rows read two rows of a column in one 32-byte sector.
// 2048^2, us per pass alone, columns 51 (1024 threads, four columns an item) and
// inverse rows 32 before.
template <int LZ, bool FROM_ACC>
__device__ __forceinline__ void big_rows_fwd_item(const RunDesc& R, int row0, int lr, float2* s, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1, ln = LZ - 1;
  constexpr int ss = fft2_stride(n);
  float2* rho = reinterpret_cast<float2*>(R.rho) + (size_t)row0 * n;
  ulonglong2* acc = reinterpret_cast<ulonglong2*>(R.dacc) + (size_t)row0 * n;
  const double inv = pow2_double(-R.fx_shift);
  auto ld = [&](int b, int m) {
    const int i = b * n + m;
    if constexpr (!FROM_ACC) return rho[i];
    const ulonglong2 a = acc[i];
    const float2 v = make_float2((float)((double)(long long)a.x * inv), (float)((double)(long long)a.y * inv));
    rho[i] = v;
    acc[i] = make_ulonglong2(0ull, 0ull);
    return v;
  };
  auto st = [&](int b, int j, float2 v) { s[b * ss + pad16(j)] = v; };
  fft2_through<LZ - 1, 0, false, false, true>(s, ss, lr, tw, LZ, -1.f, ld, st);
  const int lrb = lr < 2 ? lr : 2;
  const int rbm = (1 << lrb) - 1;
  for (int i = threadIdx.x; i < (n << lr); i += blockDim.x) {
    const int rest = i >> lrb;
    const int j = rest & (n - 1), b = ((rest >> ln) << lrb) + (i & rbm);
    const float2 zj = s[b * ss + pad16(j)];
    const float2 zc = s[b * ss + pad16((n - j) & (n - 1))];
    float2 out;
    if (j == 0) {
      out = make_float2(zj.x + zj.y, zj.x - zj.y);
    } else {
      const float2 E = make_float2(0.5f * (zj.x + zc.x), 0.5f * (zj.y - zc.y));
      const float2 O = make_float2(0.5f * (zj.y + zc.y), -0.5f * (zj.x - zc.x));
      out = cadd(E, cmul(__ldg(&tw[j]), O));
    }
    R.spec[(size_t)j * Z + row0 + b] = out;
  }
}

template <int LZ>
__device__ __forceinline__ void big_cols_item(const RunDesc& R, int col0, int lw, float2* sA, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1;
  constexpr int ss = fft2_stride(Z);
  const int W = 1 << lw;
  float2* sB = sA + W * ss;
  const float2* src = R.spec + (size_t)col0 * Z;
  auto ld = [&](int c, int k) { return src[c * Z + k]; };
  auto green = [&](int c, int kx, float2 v) {
    const int j = col0 + c, a = c * ss + pad16(kx);
    if (j == 0) {
      sA[a] = v;
      return;
    }
    const float g = __ldg(&R.green[(size_t)j * Z + kx]);
    const float gx = __ldg(&R.sxt[kx]) * g;
    const float gy = __ldg(&R.syt[j]) * g;
    sA[a] = make_float2(-gx * v.y, gx * v.x);
    sB[a] = make_float2(-gy * v.y, gy * v.x);
  };
  fft2_through<LZ, 0, false, false, true>(sA, ss, lw, tw, LZ, -1.f, ld, green);
  if (col0 == 0) {
    const float sy0 = __ldg(&R.syt[0]), syn = __ldg(&R.syt[n]);
    for (int kx = threadIdx.x; kx <= n; kx += blockDim.x) {
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
    __syncthreads();
  }
  // sequences 0 .. W-1 the x fields, W .. 2W-1 the y fields
  float2* dst = reinterpret_cast<float2*>(R.spec2 + (size_t)col0 * Z);
  auto inverse = [&](int s0, int ls) {
    auto st = [&](int b, int k, float2 v) {
      const int q = s0 + b;
      dst[2 * ((size_t)(q & (W - 1)) * Z + k) + (q >> lw)] = v;
    };
    fft2_through<LZ, 0, false, true, false>(sA + s0 * ss, ss, ls, tw, LZ, 1.f, ld, st);
  };
  if ((2 << lw) * fft2_tps(LZ) <= (int)blockDim.x) {
    inverse(0, lw + 1);
  } else {
    inverse(0, lw);
    inverse(W, lw);
  }
}

template <int LZ>
__device__ __forceinline__ void big_rows_inv_item(const RunDesc& R, int row0, int lr, float2* s, const float2* tw) {
  constexpr int Z = 1 << LZ, n = Z >> 1;
  constexpr int ss = fft2_stride(Z);
  const float4* src = R.spec2 + row0;
  auto ld = [&](int b, int j) {
    const float4 v = src[(size_t)(j < n ? j : (Z - j) & (n - 1)) * Z + b];
    return j == 0   ? make_float2(v.x, v.z)
           : j == n ? make_float2(v.y, v.w)
           : j < n  ? make_float2(v.x - v.w, v.y + v.z)
                    : make_float2(v.x + v.w, -v.y + v.z);
  };
  float2* dst = R.H + (size_t)row0 * Z;
  auto st = [&](int b, int l, float2 v) { dst[(size_t)b * Z + l] = v; };
  fft2_through<LZ, 0, true, false, false>(s, ss, lr, tw, LZ, 1.f, ld, st);
}

// ---------------------------------------------------------------------------
// Per-particle physics shared by the staged and the global neighbour paths.

// Interpolated capillary force (gridRoutinen.cpp:81-126, 284-407, 551-668).
template <bool NC>
__device__ inline float2 mesh_force(const RunDesc& R, const Rec& p, int ic, int jc, int scheme) {
  int k, l;
  float tx, ty;
  mesh_axis(R, ic, p.ox, k, tx);
  mesh_axis(R, jc, p.oy, l, ty);
  const bool sp2 = p.pid >= R.N1;
  if (scheme == NGP) {
    const float2 h = ldm<NC>(&R.H[(size_t)k * R.Z + l]);
    if (!sp2) return h;
    // species 2 reads the imaginary part of the x grid in the reference
    // (gridRoutinen.cpp:123), which is zero up to rounding
    if (R.flags & F_NGP_REFCOMPAT) return make_float2(R.q2 * h.x, 0.0f);
    return make_float2(R.q2 * h.x, R.q2 * h.y);
  }
  float wx[3], wy[3];
  axis_weights(scheme, tx, wx);
  axis_weights(scheme, ty, wy);
  const int km = k == 0 ? R.Z - 1 : k - 1, kp = k == R.Z - 1 ? 0 : k + 1;
  const int lm = l == 0 ? R.Z - 1 : l - 1, lp = l == R.Z - 1 ? 0 : l + 1;
  const int ks[3] = {km, k, kp};
  float fx = 0.f, fy = 0.f;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float2* row = R.H + (size_t)ks[a] * R.Z;
    const float2 h0 = ldm<NC>(&row[lm]), h1 = ldm<NC>(&row[l]), h2 = ldm<NC>(&row[lp]);
    fx += wx[a] * (wy[0] * h0.x + wy[1] * h1.x + wy[2] * h2.x);
    fy += wx[a] * (wy[0] * h0.y + wy[1] * h1.y + wy[2] * h2.y);
  }
  if (sp2) {
    fx *= R.q2;
    fy *= R.q2;
  }
  return make_float2(fx, fy);
}

// WCA parameters of one particle against neighbours of its own and of the
// other species (dynamik_methoden.cpp:679-686, 851-865, 1021-1035), held in
// registers for its pair loop. mask selects pair types (1: 11, 2: 22, 4: 12).
struct WcaP {
  float pre_s, sig_s, sig2_s;  // same species
  float pre_x, sig_x, sig2_x;  // other species
  float B, cut2, maxPair, L;
  float scale;                 // 2^wfx_shift: pair terms are summed in 64-bit fixed point
  int N1;
  bool sp, on_s, on_x, smallbox;
};

__device__ __forceinline__ WcaP wca_params(const RunDesc& R, const Rec& p, int mask) {
  WcaP W;
  W.sp = p.pid >= R.N1;
  const int ts = W.sp ? 1 : 0;
  W.pre_s = R.wpre[ts];
  W.sig_s = R.wsig[ts];
  W.sig2_s = R.wsig2[ts];
  W.pre_x = R.wpre[2];
  W.sig_x = R.wsig[2];
  W.sig2_x = R.wsig2[2];
  W.on_s = (mask & (W.sp ? 2 : 1)) != 0;
  W.on_x = (mask & 4) != 0;
  W.B = R.B;
  W.cut2 = R.cut2;
  W.maxPair = R.maxPair;
  W.L = R.L;
  W.N1 = R.N1;
  W.smallbox = (R.flags & F_SMALLBOX) != 0;
  W.scale = __int_as_float((127 + R.wfx_shift) << 23);
  return W;
}

// WCA contribution of neighbour q on particle p, added to the fixed-point
// sum (fx, fy): rounded once per pair term, the sum does not depend on the
// order in which neighbours are visited. da, db: cell step from p's cell to
// q's cell.
__device__ __forceinline__ void wca_pair(const WcaP& W, const Rec& p, const Rec& q, int da, int db, long long& fx,
                                         long long& fy) {
  const bool same = (q.pid >= W.N1) == W.sp;
  if (!(same ? W.on_s : W.on_x)) return;
  float dx = (p.ox - q.ox) - (float)da * W.B;
  float dy = (p.oy - q.oy) - (float)db * W.B;
  // minimum image, as abstand2_* (allgemeine_methoden.cpp:100-166). With
  // offsets in (-B, 2B] and neighbouring cells |d| < 3B, which is below L/2
  // from 7 cells per side on; only smaller boxes need the wrap.
  if (W.smallbox) {
    dx -= W.L * rintf(dx / W.L);
    dy -= W.L * rintf(dy / W.L);
  }
  const float a2 = dx * dx + dy * dy;
  const float a2s = a2 * (same ? W.sig2_s : W.sig2_x);
  if (a2s > W.cut2) return;
  const float coef = wca_coef(a2s, same ? W.pre_s : W.pre_x, W.maxPair);
  const float sg = same ? W.sig_s : W.sig_x;
  fx += __float2ll_rn(coef * (dx * sg) * W.scale);
  fy += __float2ll_rn(coef * (dy * sg) * W.scale);
}

// Re-binning of one axis after a move (refresh_erwNachbar,
// dynamik_methoden.cpp:216-325): the cell moves by floor(off/B) and the
// offset becomes fmod(off + B, B). For off in [-B, 0) the new offset is
// off + B, kept as is when FP32 rounds it to B (a legal offset) instead of
// wrapping to 0, which would move the particle by a whole cell. For
// off < -B the reference's fmod keeps a negative offset; reproduced.
__device__ inline void rebin_axis(float off, float B, int& n, float& no) {
  if (off >= 0.0f && off < B) {
    n = 0;
    no = off;
  } else if (off == B) {
    n = 1;
    no = 0.0f;
  } else if (off > B && off < 2.0f * B) {
    n = 1;
    no = off - B;
  } else if (off < 0.0f && off >= -B) {
    n = -1;
    no = off + B;
  } else if (off >= 2.0f * B) {
    const float fl = floorf(off / B);
    n = (int)fl;
    no = fmaf(-fl, B, off);
    if (no >= B) {
      no -= B;
      n++;
    } else if (no < 0.0f) {
      no += B;
      n--;
    }
  } else if (off < -B) {
    n = (int)floorf(off / B);
    no = fmodf(off + B, B);
  } else {  // NaN
    n = 0;
    no = off;
  }
}

// Euler-Maruyama update (zeitschritt, dynamik_methoden.cpp:117-157) and
// re-binning of one particle.
// sq = sqrt(2 T dt); note: whether this thread reports errors.
__device__ __forceinline__ Rec move_particle_sq(const RunDesc& R, Rec p, float2 F, float2 xi, float dt, float sq,
                                                int* err, bool apply, bool note) {
  if (apply) {
    // rounding stated, so that every kernel moves a particle to the same bits
    p.ox += __fmaf_rn(dt, F.x, __fmul_rn(sq, xi.x));
    p.oy += __fmaf_rn(dt, F.y, __fmul_rn(sq, xi.y));
  }
  if (apply && (R.flags & F_RADIAL) && p.pid >= R.N1) {
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    const double mitte = 0.5 * R.L_d;
    const double x = ic * R.B_d + (double)p.ox;
    const double y = jc * R.B_d + (double)p.oy;
    const double dxm = mitte - x, dym = mitte - y;
    const double abst = sqrt(dxm * dxm + dym * dym);
    const int t = p.pid - R.N1;
    // cos / sin of 2 pi t / N2 as sincospi (no large-argument reduction path)
    double sn, cs;
    sincospi(2.0 * t / R.N2, &sn, &cs);
    p.ox = (float)((double)p.ox + (mitte + abst * cs - x));
    p.oy = (float)((double)p.oy + (mitte + abst * sn - y));
  }
  if (!isfinite(p.ox) || !isfinite(p.oy)) {
    if (note) atomicOr(err, E_NONFINITE);
    return p;
  }
  if (p.ox < 0.0f || p.ox > R.B || p.oy < 0.0f || p.oy > R.B) {
    int nx, ny;
    float ox, oy;
    rebin_axis(p.ox, R.B, nx, ox);
    rebin_axis(p.oy, R.B, ny, oy);
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    const int icn = wrapi(ic + nx, R.C), jcn = wrapi(jc + ny, R.C);
    p.cell = icn * R.C + jcn;
    p.ox = ox;
    p.oy = oy;
  }
  return p;
}

__device__ inline Rec move_particle(const RunDesc& R, Rec p, float2 F, float2 xi, float dt, int* err,
                                    bool apply = true) {
  return move_particle_sq(R, p, F, xi, dt, apply ? sqrtf(2.0f * R.T * dt) : 0.f, err, apply, true);
}

// optimaler_zeitschritt bound of one component (dynamik_methoden.cpp:1420-1491):
// dt < (w-|u|)^2 with u = xi sqrt(T/2)/F, w = sqrt(u^2 + m/|F|). In FP32
// w - |u| cancels when u^2 >> m/|F|, so it is evaluated as the equal
// (m/|F|) / (w + |u|).
__device__ inline float dt_bound(float F, float nz, float mrd, float T) {
  if (fabsf(F) < 1.0e-5f) return mrd * mrd / (2.0f * T * nz * nz);
  const float u = nz * sqrtf(0.5f * T) / F;
  const float a = mrd / fabsf(F);
  const float w = sqrtf(u * u + a);
  const float d = a / (w + fabsf(u));
  return d * d;
}


template <bool NC>
__device__ inline void finish_particle(const RunDesc& R, RunDyn& D, const unsigned long long& step, int mode, int mask,
                                       const Rec& p, int ic, int jc, int gi, float2 Fw);

template <bool NC>
__device__ __forceinline__ Rec ldrec(const Rec* q) {
  const int4 v = ldm<NC>(reinterpret_cast<const int4*>(q));
  Rec r;
  r.ox = __int_as_float(v.x);
  r.oy = __int_as_float(v.y);
  r.cell = v.z;
  r.pid = v.w;
  return r;
}

// The fixed-point sum as a force: 2^-wfx_shift, exact in FP64 (built from its
// exponent: a division per particle cost more than a pair).
__device__ __forceinline__ float2 wca_unfix(const RunDesc& R, long long fx, long long fy) {
  const double inv = pow2_double(-R.wfx_shift);
  return make_float2((float)((double)fx * inv), (float)((double)fy * inv));
}

// WCA sum of particle p (at global index self, cell (ic, jc)) over the 3x3
// neighbour cells, read straight from the cell-sorted array: per neighbour
// row the cells jc-1, jc, jc+1 form one contiguous range unless the row
// wraps. The fixed-point sum makes the result independent of the order of
// the particles within a cell.
template <bool NC>
__device__ inline float2 wca_direct(const RunDesc& R, const Rec& p, int ic, int jc, int self, int m) {
  long long fx = 0, fy = 0;
  const WcaP W = wca_params(R, p, m);
  const int C = R.C;
  const Rec* rec = R.recA;
  const int* start = R.start;
  if (jc >= 1 && jc <= C - 2) {
    // per neighbour row one contiguous range (cells jc-1 .. jc+1); the six
    // bounds are loaded together
    int beg[3], end[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int row = wrap1(ic + a - 1, C) * C;
      beg[a] = ldm<NC>(&start[row + jc - 1]);
      end[a] = ldm<NC>(&start[row + jc + 2]);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int cmid = wrap1(ic + a - 1, C) * C + jc;
      if constexpr (!NC) {
        // resident step: the next record is requested
        // before the current pair is evaluated
        Rec q;
        if (beg[a] < end[a]) q = ldrec<NC>(&rec[beg[a]]);
        for (int j = beg[a]; j < end[a]; j++) {
          Rec qn = q;
          if (j + 1 < end[a]) qn = ldrec<NC>(&rec[j + 1]);
          if (j != self) wca_pair(W, p, q, a - 1, q.cell - cmid, fx, fy);
          q = qn;
        }
      } else {
        for (int j = beg[a]; j < end[a]; j++) {
          if (j == self) continue;
          const Rec q = ldrec<NC>(&rec[j]);
          wca_pair(W, p, q, a - 1, q.cell - cmid, fx, fy);
        }
      }
    }
  } else {
#pragma unroll 1
    for (int da = -1; da <= 1; da++) {
      const int row = wrap1(ic + da, C) * C;
#pragma unroll 1
      for (int db = -1; db <= 1; db++) {
        const int g = row + wrap1(jc + db, C);
        const int beg = ldm<NC>(&start[g]), end = ldm<NC>(&start[g + 1]);
        for (int j = beg; j < end; j++) {
          if (j == self) continue;
          wca_pair(W, p, ldrec<NC>(&rec[j]), da, db, fx, fy);
        }
      }
    }
  }
  return wca_unfix(R, fx, fy);
}

// The part of wca_direct's sum from neighbour row da (-1, 0, 1), for particles
// whose rows are shared out over lanes.
__device__ __forceinline__ void wca_row(const RunDesc& R, const WcaP& W, const Rec& p, int ic, int jc, int self,
                                        int da, long long& fx, long long& fy) {
  const int C = R.C, row = wrap1(ic + da, C) * C;
  const Rec* rec = R.recA;
  if (jc >= 1 && jc <= C - 2) {
    const int beg = R.start[row + jc - 1], end = R.start[row + jc + 2];
    Rec q = {};
    if (beg < end) q = ldrec<false>(&rec[beg]);
    for (int j = beg; j < end; j++) {
      Rec qn = q;
      if (j + 1 < end) qn = ldrec<false>(&rec[j + 1]);
      if (j != self) wca_pair(W, p, q, da, q.cell - row - jc, fx, fy);
      q = qn;
    }
  } else {
#pragma unroll 1
    for (int db = -1; db <= 1; db++) {
      const int g = row + wrap1(jc + db, C);
      const int beg = R.start[g], end = R.start[g + 1];
      for (int j = beg; j < end; j++)
        if (j != self) wca_pair(W, p, ldrec<false>(&rec[j]), da, db, fx, fy);
    }
  }
}

// Forces of the particle at sorted index gi in the mode asked for.
template <bool NC>
__device__ __forceinline__ void particle_item(const RunDesc& R, RunDyn& D, const unsigned long long& step, int gi, int mode,
                                              int mask) {
  const Rec p = ldrec<NC>(&R.recA[gi]);
  int ic, jc;
  cell_ij(R, p.cell, ic, jc);
  int m = mask;
  if (mode == MODE_SET) m &= p.pid >= R.N1 ? 2 : 1;
  if (R.flags & F_IDGAS) m = 0;
  const float2 Fw = m ? wca_direct<NC>(R, p, ic, jc, gi, m) : make_float2(0.f, 0.f);
  finish_particle<NC>(R, D, step, mode, mask, p, ic, jc, gi, Fw);
}

// Count a particle into its new cell (an add whose result nobody waits for;
// the scatter takes the slots) and into the per-chunk total for the scan,
// added once per group of lanes in the same chunk (neighbouring particles of
// the cell-sorted order mostly share one). The cell is the key: the scatter
// reads it from the record recB[gi].
// act: the lanes of the warp that call, converged.
__device__ __forceinline__ void count_into_cell(const RunDesc& R, int key, unsigned act) {
  red_add(&R.count[key], 1);
  const int ch = key / SCAN_CHUNK;
  const unsigned grp = __match_any_sync(act, ch);
  if ((threadIdx.x & 31) == __ffs(grp) - 1) red_add(&R.chunk_sum[ch], __popc(grp));
}

// Everything after the WCA sum: store it (MODE_SET, MODE_ADD), or store it with
// the mesh force and the noise and take the dt bound (MODE_FORCES).
template <bool NC>
__device__ inline void finish_particle(const RunDesc& R, RunDyn& D, const unsigned long long& step, int mode, int mask,
                                       const Rec& p, int ic, int jc, int gi, float2 Fw) {
  const bool sp2 = p.pid >= R.N1;
  if (mode == MODE_SET) {
    if ((mask & (sp2 ? 2 : 1))) R.Fw[p.pid] = Fw;
    return;
  }
  if (mode == MODE_ADD) {
    float2 f = R.Fw[p.pid];
    f.x += Fw.x;
    f.y += Fw.y;
    R.Fw[p.pid] = f;
    return;
  }
  const float2 Fk = (R.flags & F_IDGAS) ? make_float2(0.f, 0.f) : mesh_force<NC>(R, p, ic, jc, R.scheme);
  float2 xi = make_float2(0.f, 0.f);
  if (!(R.flags & F_NOWCA)) xi = particle_noise(R.noise, R.seed, step, (uint32_t)p.pid);
  R.Fw[p.pid] = Fw;
  R.Fk[p.pid] = Fk;
  R.Fn[p.pid] = xi;
  float bnd = fminf(dt_bound(Fw.x + Fk.x, xi.x, R.mrd, R.T), dt_bound(Fw.y + Fk.y, xi.y, R.mrd, R.T));
  if (!(bnd >= 0.f)) bnd = 3.0e38f;  // NaN never wins the minimum (std::min semantics)
  if (bnd < R.dt_max) atomicMin(&D.dt_bits, __float_as_uint(bnd));
}

// Forces, noise and move of the particle at sorted index gi, its counts and
// (DEP) its deposit. act: the lanes of the warp that call. The lanes are
// brought together again behind the neighbour loops, the noise's rejections
// and the re-binning: left to the compiler, what follows ran for parts of the
// warp in turn (lanes that leave a loop early going ahead).
template <bool NC, bool DEP>
__device__ __forceinline__ void step_particle(const RunDesc& R, RunDyn& D, const unsigned long long& step, int gi,
                                              unsigned act) {
  const Rec p = ldrec<NC>(&R.recA[gi]);
  int ic, jc;
  cell_ij(R, p.cell, ic, jc);
  const bool gas = (R.flags & F_IDGAS) != 0;
  const float2 Fw = gas ? make_float2(0.f, 0.f) : wca_direct<NC>(R, p, ic, jc, gi, 7);
  __syncwarp(act);
  const float2 Fk = gas ? make_float2(0.f, 0.f) : mesh_force<NC>(R, p, ic, jc, R.scheme);
  float2 xi = make_float2(0.f, 0.f);
  if (!(R.flags & F_NOWCA)) xi = particle_noise(R.noise, R.seed, step, (uint32_t)p.pid);
  __syncwarp(act);
  const Rec np = move_particle(R, p, make_float2(Fw.x + Fk.x, Fw.y + Fk.y), xi, R.dt_max, &D.err);
  __syncwarp(act);
  R.recB[gi] = np;
  count_into_cell(R, np.cell, act);
  // the resident and the pipelined step: the next step's density
  if constexpr (DEP) deposit_acc<1>(R, np);
  if (np.cell != p.cell) atomicAdd(&D.moved[p.pid >= R.N1 ? 1 : 0], 1);  // num_Zellwechsel of TimestepInfo
}

// End of a step (one thread per run): advance the Philox step counter, the
// simulated time and the steps budget; re-arm the adaptive dt reduction.
__device__ inline void end_step(const RunDesc& R, RunDyn& D, int adaptive) {
  double dt = R.dt_max_d;
  if (adaptive && (R.flags & F_ADAPTIVE)) {
    const float b = __uint_as_float(D.dt_bits);
    dt = b < R.dt_max ? (double)b : R.dt_max_d;
  }
  D.dt = (float)dt;
  D.t += dt;
  D.step++;
  D.steps_left--;
  D.dt_bits = __float_as_uint(3.0e38f);
  D.moved_last[0] = D.moved[0];
  D.moved_last[1] = D.moved[1];
  D.moved[0] = D.moved[1] = 0;
}

// start[] of one chunk from its counts v (PER per thread, PER * threads =
// SCAN_CHUNK) and its offset. The counts stay: the scatter counts them down
// to zero as it takes slots. All threads of the team call; sh: 32 ints.
template <int PER, class Team>
__device__ __forceinline__ void scan_chunk_store(const Team& T, const RunDesc& R, int chunk, int ncells,
                                                 const int* v, int off, int* sh) {
  static_assert(PER % 4 == 0, "whole int4 vectors per thread");
  const int base = chunk * SCAN_CHUNK;
  const int c0 = base + T.tid * PER;
  int loc = 0;
#pragma unroll
  for (int k = 0; k < PER; k++) loc += v[k];
  int acc = team_excl_scan(T, loc, sh) + off;
  int w[PER];
#pragma unroll
  for (int k = 0; k < PER; k++) {
    w[k] = acc;
    acc += v[k];
  }
  if (base + SCAN_CHUNK <= ncells) {
#pragma unroll
    for (int k = 0; k < PER; k += 4)
      *reinterpret_cast<int4*>(&R.start[c0 + k]) = make_int4(w[k], w[k + 1], w[k + 2], w[k + 3]);
  } else {
#pragma unroll
    for (int k = 0; k < PER; k++)
      if (c0 + k < ncells) R.start[c0 + k] = w[k];
  }
  if (base + SCAN_CHUNK >= ncells && T.tid == 0) R.start[ncells] = R.N;
  T.sync();  // sh is reused by the next scan
}

// Particle gi of the old order to start[cell] + slot, the slot taken by
// counting the cell's count down (which leaves it zero for the next sort).
__device__ __forceinline__ void scatter_particle(const RunDesc& R, int gi) {
  const Rec q = R.recB[gi];
  const int slot = atomicSub(&R.count[q.cell], 1) - 1;
  R.recA[R.start[q.cell] + slot] = q;
}

constexpr unsigned BAR_MAX_POLLS = 1u << 22;
// set in the arrival counter by a CTA whose wait gave up: every CTA that
// sees it fails the barrier
constexpr unsigned BAR_POISON = 0x80000000u;

// Grid-wide barrier: bar[0] counts arrivals (a release add; waiters poll it
// with acquire loads until it reaches target = barriers so far x grid), so
// the writes of every CTA before the barrier are visible to all after it.
// bar[1] counts CTAs leaving the launch; the last one clears both words for
// the next launch. A wait gives up after max_polls polls: it sets the poison
// bit with a compare-and-swap that succeeds only while the count is short of
// the target, so either the last arrival comes first and every CTA passes,
// or the poison comes first and every CTA (late arrivals included) fails
// this barrier and returns: no CTA runs past a failed barrier. The failure
// is reported as E_BARRIER_TIMEOUT; the host clears the words.
__device__ inline bool grid_barrier(unsigned* bar, unsigned target, unsigned max_polls, int* err, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> c(bar[0]);
    c.fetch_add(1u, cuda::memory_order_release);
    int ok = 1;
    for (unsigned polls = 0;; polls++) {
      unsigned v = c.load(cuda::memory_order_acquire);
      if (v & BAR_POISON) {
        ok = 0;
        break;
      }
      if (v >= target) break;
      if (polls >= max_polls) {
        while (!(v & BAR_POISON) && v < target)
          if (c.compare_exchange_weak(v, v | BAR_POISON, cuda::memory_order_acq_rel, cuda::memory_order_acquire))
            v |= BAR_POISON;
        if (v & BAR_POISON) {
          ok = 0;
          atomicOr(err, E_BARRIER_TIMEOUT);
        }
        break;
      }
      __nanosleep(20);
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// G: the CTAs that share the words
__device__ inline void grid_exit(unsigned* bar, unsigned G) {
  if (threadIdx.x == 0 && atomicAdd(&bar[1], 1u) == G - 1) {
    atomicExch(&bar[0], 0u);
    atomicExch(&bar[1], 0u);
  }
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bring this CTA's share (1/G, 256-byte aligned pieces) of a device array
// into L2 with one bulk prefetch (no data moves to the SM; the base must be
// 16-byte aligned, as cudaMalloc's are). Issued by one thread.
__device__ __forceinline__ void l2_prefetch_share(const void* base, size_t bytes, int b, int G) {
  const size_t per = ((bytes + G - 1) / G + 255) & ~(size_t)255;
  const size_t off = (size_t)b * per;
  if (off >= bytes) return;
  const size_t len = (bytes - off < per ? bytes - off : per) & ~(size_t)15;
  if (len == 0) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char*)base + off), "r"((unsigned)len)
               : "memory");
}

}  // namespace bd
