// Device kernels of the force-and-integrate step.
//
// One step of every run in a batch is the launch sequence
//   deposit -> fft_rows_fwd -> fft_cols -> fft_rows_inv      (capillary mesh)
//   integrate                                                (WCA + mesh force
//                                                             + noise + update
//                                                             + re-binning)
//   scan_partial -> scan_final -> scatter -> fixup -> step_end (cell sort)
// Each kernel walks a list of work items (run, a, b, c) so that runs of
// different sizes share one launch. All reductions are order-independent or
// run in a fixed order, so results do not depend on scheduling.
#include <algorithm>
#include <cstdio>
#include <cstdint>
#include <cuda_runtime.h>

#include "bd_common.cuh"
#include "bd_fft.cuh"
#include "bd_fft2.cuh"
#include "bd_items.cuh"
#include "bd_kernels.h"

namespace bd {

// In-place exclusive scan of n counts stored with a stride: a[k*stride] ->
// out[k*stride + 1]; writes the total to out[n*stride]. All threads call it.
__device__ inline void block_scan_strided(const int* cnt, int* out, int n, int stride, int* tmp32) {
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int s0 = threadIdx.x * per;
  int loc = 0;
  for (int q = 0; q < per; q++)
    if (s0 + q < n) loc += cnt[(s0 + q) * stride];
  int ex = block_excl_scan(loc, tmp32);
  for (int q = 0; q < per; q++)
    if (s0 + q < n) {
      out[(s0 + q) * stride] = ex;
      ex += cnt[(s0 + q) * stride];
    }
  if (threadIdx.x == blockDim.x - 1) out[n * stride] = ex;
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Charge assignment (gridRoutinen.cpp:31-76, 131-280, 412-547).
// One CTA owns a MT x MT tile of mesh points and gathers every particle whose
// stencil can reach it (the cell rows covering the tile plus halo, located
// through the cell-sorted order). Contributions are rounded to fixed point
// (|value| <= 2^30 units of 2^-fx_shift) and accumulate in shared memory as
// 64-bit sums kept in two 32-bit words (fx_add), so the sum is exact and
// independent of the order in which threads add; the owner writes its tile
// once, without global atomics.

// 64-bit fixed-point add from 32-bit shared-memory atomics (much faster on
// this GPU than 64-bit ones): the carry out of the low word is read off the
// returned old value, so lo/hi always hold the exact sum modulo 2^64,
// whatever the order of the additions.
__device__ __forceinline__ void fx_add(unsigned* lo, unsigned* hi, int a, int v) {
  const unsigned u = (unsigned)v;
  const unsigned old = atomicAdd(&lo[a], u);
  const unsigned h = (unsigned)(v >> 31) + (old + u < old ? 1u : 0u);
  if (h) atomicAdd(&hi[a], h);
}

// Deposit of the MT x MT tile at mesh (x0, y0); smem holds the 2*MT*MT
// accumulator words and the segment table, s_tmp 32 ints. All threads call.
__device__ inline void deposit_tile(const RunDesc& R, int scheme, int x0, int y0, int MT, unsigned char* smem,
                                    int* s_tmp) {
  unsigned* acc_lo = (unsigned*)smem;
  unsigned* acc_hi = acc_lo + MT * MT;
  int* seg = (int*)(acc_hi + MT * MT);  // [nseg][3]: global begin, length, prefix
  for (int i = threadIdx.x; i < 2 * MT * MT; i += blockDim.x) acc_lo[i] = 0u;
  // cell rows/columns that can reach this tile: offsets lie in (-B, 2B]
  const float rB = R.dx * R.invB;
  int ilo = (int)floorf((x0 - 1) * rB) - 2, ihi = (int)floorf((x0 + MT + 1) * rB) + 1;
  int jlo = (int)floorf((y0 - 1) * rB) - 2, jhi = (int)floorf((y0 + MT + 1) * rB) + 1;
  if (ihi - ilo + 1 >= R.C) ilo = 0, ihi = R.C - 1;
  if (jhi - jlo + 1 >= R.C) jlo = 0, jhi = R.C - 1;
  const int ncx = ihi - ilo + 1;
  // per cell row at most two contiguous particle segments (periodic wrap)
  const int jl = wrapi(jlo, R.C);
  const int ncy = jhi - jlo + 1;
  const bool split = jl + ncy > R.C;
  const int nseg = ncx * (split ? 2 : 1);
  for (int s = threadIdx.x; s < nseg; s += blockDim.x) {
    const int row = split ? s >> 1 : s;
    const int part = split ? (s & 1) : 0;
    const int ic = wrapi(ilo + row, R.C);
    int a, b;
    if (!split) {
      a = jl;
      b = jl + ncy;
    } else if (part == 0) {
      a = jl;
      b = R.C;
    } else {
      a = 0;
      b = jl + ncy - R.C;
    }
    const int gb = R.start[ic * R.C + a];
    const int ge = R.start[ic * R.C + b];
    seg[3 * s] = gb;
    seg[3 * s + 1] = ge - gb;
  }
  __syncthreads();
  block_scan_strided(seg + 1, seg + 2, nseg, 3, s_tmp);
  const int total = seg[3 * nseg + 2];
  const float scale = __int_as_float((127 + R.fx_shift) << 23);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (seg[3 * mid + 2] <= t) lo = mid;
      else hi = mid - 1;
    }
    const Rec p = R.recA[seg[3 * lo] + (t - seg[3 * lo + 2])];
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    int k, l;
    float tx, ty;
    mesh_axis(R, ic, p.ox, k, tx);
    mesh_axis(R, jc, p.oy, l, ty);
    const float q = p.pid < R.N1 ? 1.0f : R.q2;
    if (scheme == NGP) {
      const int lk = wrap1(k - x0, R.Z), ll = wrap1(l - y0, R.Z);
      if (lk < MT && ll < MT) {
        float c = R.drho;
        if (p.pid >= R.N1) c *= q;
        fx_add(acc_lo, acc_hi, lk * MT + ll, __float2int_rn(c * scale));
      }
      continue;
    }
    float wx[3], wy[3];
    axis_weights(scheme, tx, wx);
    axis_weights(scheme, ty, wy);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int lk = wrap1(k + a - 1 - x0, R.Z);
      if (lk >= MT) continue;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const int ll = wrap1(l + b - 1 - y0, R.Z);
        if (ll >= MT) continue;
        float c = wx[a] * wy[b] * R.drho;
        if (p.pid >= R.N1) c *= q;
        fx_add(acc_lo, acc_hi, lk * MT + ll, __float2int_rn(c * scale));
      }
    }
  }
  __syncthreads();
  const double inv = 1.0 / (double)scale;
  for (int i = threadIdx.x; i < MT * MT; i += blockDim.x) {
    const int lk = i / MT, ll = i - (i / MT) * MT;
    const long long acc = (long long)(((unsigned long long)acc_hi[i] << 32) | acc_lo[i]);
    R.rho[(size_t)(x0 + lk) * R.Z + y0 + ll] = (float)((double)acc * inv);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_deposit(const RunDesc* __restrict__ runs,
                                                 const RunDyn* __restrict__ dyn,
                                                 const Item* __restrict__ items, int nitems,
                                                 int scheme_override, int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_tmp[32];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active && !run_active(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int scheme = scheme_override >= 0 ? scheme_override : R.scheme;
    const int MT = I.c;
    deposit_tile(R, scheme, I.a * MT, I.b * MT, MT, smem, s_tmp);
  }
}

// ---------------------------------------------------------------------------
// Row pass, forward: each mesh row (fixed x index k) is real; it is packed as
// Z/2 complex values z[m] = rho[2m] + i rho[2m+1], transformed, and unpacked
// into the half spectrum X[j], j in [0, Z/2]. The two purely real bins j = 0
// and j = Z/2 share slot 0 as (X[0], X[Z/2]).
__global__ void __launch_bounds__(FFT_THREADS) k_fft_rows_fwd(const RunDesc* __restrict__ runs,
                                                      const RunDyn* __restrict__ dyn,
                                                      const Item* __restrict__ items, int nitems,
                                                      int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = (float2*)smem;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active && !run_active(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int Z = R.Z, n = Z >> 1;
    const int lr = I.c;  // log2(rows in this item)
    const int row0 = I.a;
    for (int i = threadIdx.x; i < (n << lr); i += blockDim.x) {
      const int b = i / n, m = i - b * n;
      const float2 v = *reinterpret_cast<const float2*>(&R.rho[(size_t)(row0 + b) * Z + 2 * m]);
      s[(m << lr) | b] = v;
    }
    __syncthreads();
    fft_dif<false>(CtaTeam(), s, R.plan_half, lr, R.tw, 2, false);
    for (int i = threadIdx.x; i < (n << lr); i += blockDim.x) {
      const int b = i / n, j = i - b * n;
      const float2 zj = s[(__ldg(&R.pos_half[j]) << lr) | b];
      const float2 zc = s[(__ldg(&R.pos_half[j == 0 ? 0 : n - j]) << lr) | b];
      float2 out;
      if (j == 0) {
        out = make_float2(zj.x + zj.y, zj.x - zj.y);
      } else {
        // E = (zj + conj zc)/2, O = (zj - conj zc)/(2i), X = E + w^j O
        const float2 E = make_float2(0.5f * (zj.x + zc.x), 0.5f * (zj.y - zc.y));
        const float2 O = make_float2(0.5f * (zj.y + zc.y), -0.5f * (zj.x - zc.x));
        out = cadd(E, cmul(__ldg(&R.tw[j]), O));
      }
      R.spec[(size_t)(row0 + b) * n + j] = out;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Column pass: forward transform over x of W spectrum columns, multiply by
// i*sin(q dx)/dx*G(q) for both force components (dynamik_methoden.cpp:
// 1210-1216 with the tables of :585-593), inverse transform over x of both
// fields. Column 0 holds the packed real pair (ky = 0, ky = Z/2): its
// transform C = A + iB is split into A and B, each multiplied by its own
// Green's factor and packed again for the inverse.
__global__ void __launch_bounds__(FFT_THREADS) k_fft_cols(const RunDesc* __restrict__ runs,
                                                  const RunDyn* __restrict__ dyn,
                                                  const Item* __restrict__ items, int nitems,
                                                  int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active && !run_active(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int Z = R.Z, n = Z >> 1;
    const int lw = I.c, W = 1 << lw;
    const int col0 = I.a;
    float2* sA = (float2*)smem;
    float2* sB = sA + ((size_t)Z << lw);
    for (int i = threadIdx.x; i < (Z << lw); i += blockDim.x) {
      const int k = i >> lw, c = i & (W - 1);
      sA[i] = R.spec[(size_t)k * n + col0 + c];
    }
    __syncthreads();
    fft_dif<false>(CtaTeam(), sA, R.plan_full, lw, R.tw, 1, false);
    // columns other than the packed one: independent per element
    for (int i = threadIdx.x; i < (Z << lw); i += blockDim.x) {
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
      // packed column: read partners before anyone overwrites column 0
      constexpr int MAXIT = 16;
      float2 P[MAXIT], Q[MAXIT];
      int cnt = 0;
      for (int pos = threadIdx.x; pos < Z && cnt < MAXIT; pos += blockDim.x, cnt++) {
        const int kx = __ldg(&R.freq_full[pos]);
        const int km = kx == 0 ? 0 : Z - kx;
        const float2 Cv = sA[pos << lw];
        const float2 Cm = sA[__ldg(&R.pos_full[km]) << lw];
        // A = (C + conj Cm)/2 ; B = (C - conj Cm)/(2i)
        const float2 A = make_float2(0.5f * (Cv.x + Cm.x), 0.5f * (Cv.y - Cm.y));
        const float2 Bv = make_float2(0.5f * (Cv.y + Cm.y), -0.5f * (Cv.x - Cm.x));
        const float gA = __ldg(&R.green[kx]);
        const float gB = __ldg(&R.green[(size_t)n * Z + kx]);
        const float sx = __ldg(&R.sxt[kx]);
        const float syA = __ldg(&R.syt[0]), syB = __ldg(&R.syt[n]);
        // i*s*g*A, then P = FxA + i FxB, Q = FyA + i FyB
        const float2 FxA = make_float2(-sx * gA * A.y, sx * gA * A.x);
        const float2 FxB = make_float2(-sx * gB * Bv.y, sx * gB * Bv.x);
        const float2 FyA = make_float2(-syA * gA * A.y, syA * gA * A.x);
        const float2 FyB = make_float2(-syB * gB * Bv.y, syB * gB * Bv.x);
        P[cnt] = make_float2(FxA.x - FxB.y, FxA.y + FxB.x);
        Q[cnt] = make_float2(FyA.x - FyB.y, FyA.y + FyB.x);
      }
      __syncthreads();
      cnt = 0;
      for (int pos = threadIdx.x; pos < Z && cnt < MAXIT; pos += blockDim.x, cnt++) {
        sA[pos << lw] = P[cnt];
        sB[pos << lw] = Q[cnt];
      }
    }
    __syncthreads();
    fft_dit<false>(CtaTeam(), sA, R.plan_full, lw, R.tw, 1, true);
    fft_dit<false>(CtaTeam(), sB, R.plan_full, lw, R.tw, 1, true);
    for (int i = threadIdx.x; i < (Z << lw); i += blockDim.x) {
      const int k = i >> lw, c = i & (W - 1);
      const float2 a = sA[i], b = sB[i];
      R.spec2[(size_t)k * n + col0 + c] = make_float4(a.x, a.y, b.x, b.y);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Row pass, inverse: both force grids are real, so one complex inverse
// transform of H = Fx' + i Fy' over the full y spectrum (Hermitian
// extension of the half spectra) yields Fx + i Fy, stored as float2.
__global__ void __launch_bounds__(FFT_THREADS) k_fft_rows_inv(const RunDesc* __restrict__ runs,
                                                      const RunDyn* __restrict__ dyn,
                                                      const Item* __restrict__ items, int nitems,
                                                      int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = (float2*)smem;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active && !run_active(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int Z = R.Z, n = Z >> 1;
    const int lr = I.c;
    const int row0 = I.a;
    for (int i = threadIdx.x; i < (Z << lr); i += blockDim.x) {
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
    __syncthreads();
    fft_dit<false>(CtaTeam(), s, R.plan_full, lr, R.tw, 1, true);
    for (int i = threadIdx.x; i < (Z << lr); i += blockDim.x) {
      const int b = i / Z, l = i - b * Z;
      R.H[(size_t)(row0 + b) * Z + l] = s[(l << lr) | b];
    }
    __syncthreads();
  }
}

// The three passes as kernels, one item per CTA (an item loop around the
// transform with twiddles from global memory makes the compiler hoist the
// twiddle loads of every pass and spill). Meshes of 2048 and more: bounded for
// four CTAs per SM, 64 registers (columns 55 -> 47 us at 2048^2). Smaller ones
// name no number of CTAs: told that one is enough, the compiler took 128, 94
// and 55 registers for columns, inverse and forward rows of 1024 points
// instead of 80, 64 and 40 (200 meshes of 1024^2, us per pass 2608, 1863 and 868
// instead of 2053, 1216 and 704).
template <int LZ>
__global__ void __launch_bounds__(FFT2_THREADS, LZ >= 11 ? 4 : 0) k_fft2_rows_fwd(const RunDesc* __restrict__ runs,
                                                         const RunDyn* __restrict__ dyn,
                                                         const Item* __restrict__ items, int nitems,
                                                         int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x >= nitems) return;
  const Item I = items[blockIdx.x];
  if (require_active && !run_active(dyn, I.run)) return;
  const RunDesc& R = runs[I.run];
  if constexpr (LZ >= 11) big_rows_fwd_item<LZ, false>(R, I.a, I.c, (float2*)smem, R.tw);
  else fft2_rows_fwd_item<LZ, false, false>(OnceTeam(), R, I.a, I.c, (float2*)smem, R.tw);
}

template <int LZ>
__global__ void __launch_bounds__(FFT2_THREADS, LZ >= 11 ? 4 : 0) k_fft2_cols(const RunDesc* __restrict__ runs,
                                                     const RunDyn* __restrict__ dyn,
                                                     const Item* __restrict__ items, int nitems,
                                                     int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x >= nitems) return;
  const Item I = items[blockIdx.x];
  if (require_active && !run_active(dyn, I.run)) return;
  const RunDesc& R = runs[I.run];
  if constexpr (LZ >= 11) big_cols_item<LZ>(R, I.a, I.c, (float2*)smem, R.tw);
  else fft2_cols_item<LZ, false>(OnceTeam(), R, I.a, I.c, (float2*)smem, R.tw);
}

template <int LZ>
__global__ void __launch_bounds__(FFT2_THREADS, LZ >= 11 ? 4 : 0) k_fft2_rows_inv(const RunDesc* __restrict__ runs,
                                                         const RunDyn* __restrict__ dyn,
                                                         const Item* __restrict__ items, int nitems,
                                                         int require_active) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x >= nitems) return;
  const Item I = items[blockIdx.x];
  if (require_active && !run_active(dyn, I.run)) return;
  const RunDesc& R = runs[I.run];
  if constexpr (LZ >= 11) big_rows_inv_item<LZ>(R, I.a, I.c, (float2*)smem, R.tw);
  else fft2_rows_inv_item<LZ, false>(OnceTeam(), R, I.a, I.c, (float2*)smem, R.tw);
}

// The step's particle kernel: forces, noise, move, re-binning and counts, one
// thread per particle of the cell-sorted array. DEP: the move adds the next
// step's density to each run's accumulator R.dacc (the pipelined stage step,
// whose forward row pass reads it). A kernel of its own, not a mode of
// k_particles: the pair loop tests no mask and less code is fetched.
// MINB: CTAs per SM the compiler keeps registers for (4: at most 64
// registers; 5: at most 51, more warps resident, a few values reloaded from
// local memory); the batch autotuner picks one, the arithmetic is the same.
// AHEAD > 0: every block requests into L2 what the block AHEAD items on reads
// first. A large run's arrays stream through memory with the cell order, and
// each of a particle's dependent reads (record, cell starts, neighbours, force
// grid, accumulator) waited for DRAM: 2.1 M particles, 2048^2, 207 -> 143 us.
// Runs of a batch that fit L2 gain nothing and pay for the requests (256-run
// ensemble 333 -> 343 us).

// Part of an array of `total` elements, [at, at + n), into L2.
__device__ __forceinline__ void l2_prefetch_part(const void* base, size_t elem, size_t at, size_t n, size_t total) {
  if (at >= total) return;
  const size_t lo = (at * elem) & ~(size_t)15, hi = (min(at + n, total) * elem) & ~(size_t)15;
  if (hi <= lo) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char*)base + lo), "r"((unsigned)(hi - lo)));
}

// What block a (256 particles) of run R reads first. Its cells and mesh points
// are guessed from its place in the cell order, as for a uniform density (a
// wrong guess costs the request); the rows behind them are in L2 already.
template <bool DEP>
__device__ __forceinline__ void prefetch_block(const RunDesc& R, int a) {
  const size_t g = (size_t)a * 256, cc = (size_t)R.C * R.C;
  const float f = (float)g / (float)R.N, w = 256.f / (float)R.N;
  l2_prefetch_part(R.recA, sizeof(Rec), g, 256, R.N);
  const size_t c0 = (size_t)(f * (float)cc), cn = (size_t)(w * (float)cc) + 8;
  l2_prefetch_part(R.start, sizeof(int), c0 + R.C, cn, cc + 1);
  l2_prefetch_part(R.count, sizeof(int), c0, cn, cc);
  if (R.flags & F_IDGAS) return;
  const size_t zz = (size_t)R.Z * R.Z, z0 = (size_t)(f * (float)zz), zn = (size_t)(w * (float)zz) + 8;
  l2_prefetch_part(R.H, sizeof(float2), z0 + 2 * R.Z, zn, zz);
  if (DEP) l2_prefetch_part(R.dacc, sizeof(unsigned long long), z0 + 2 * R.Z, zn, zz);
}

template <int MINB, bool DEP, int AHEAD>
__global__ void __launch_bounds__(256, MINB) k_step(const RunDesc* __restrict__ runs, RunDyn* __restrict__ dyn,
                                                    const Item* __restrict__ items, int nitems) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (AHEAD > 0 && threadIdx.x == 32 && it + AHEAD < nitems) {
      const Item J = items[it + AHEAD];
      prefetch_block<DEP>(runs[J.run], J.a);
    }
    const bool on = run_active(dyn, I.run);
    // the pipelined step: the run's first block records whether the run takes
    // part in this step, for the sort and transform kernels that follow (the
    // step end changes the budget while they run)
    if (DEP && I.a == 0 && threadIdx.x == 0) dyn[I.run].sorting = on ? 1 : 0;
    if (!on) continue;
    const RunDesc& R = runs[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, gi < R.N);
    if (gi < R.N) step_particle<true, DEP>(R, dyn[I.run], dyn[I.run].step, gi, act);
  }
}

// Forces only, stored by particle index: the drop-in WCA routines (MODE_SET,
// MODE_ADD with their pair mask) and the adaptive step's (MODE_FORCES).
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k_particles(const RunDesc* __restrict__ runs,
                                                   RunDyn* __restrict__ dyn,
                                                   const Item* __restrict__ items, int nitems,
                                                   int mode, int mask, int require_active) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active && !run_active(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    if (gi >= R.N) continue;
    particle_item<true>(R, dyn[I.run], dyn[I.run].step, gi, mode, mask);
  }
}

// Move from stored forces (adaptive dt: the reduced bound; fixed dt: dt_max),
// or with refresh_only re-bin the current positions without moving
// (refresh_erwNachbar on caller-modified offsets).
__global__ void __launch_bounds__(256) k_move(const RunDesc* __restrict__ runs,
                                              RunDyn* __restrict__ dyn,
                                              const Item* __restrict__ items, int nitems,
                                              int require_active, int refresh_only) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (require_active ? !run_active(dyn, I.run) : run_failed(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    RunDyn& D = dyn[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, gi < R.N);
    if (gi >= R.N) continue;
    const Rec p = R.recA[gi];
    Rec np;
    if (refresh_only) {
      np = move_particle(R, p, make_float2(0.f, 0.f), make_float2(0.f, 0.f), 0.f, &D.err, false);
    } else {
      const float2 Fw = R.Fw[p.pid], Fk = R.Fk[p.pid], xi = R.Fn[p.pid];
      const float dt = (R.flags & F_ADAPTIVE) ? fminf(R.dt_max, __uint_as_float(D.dt_bits)) : R.dt_max;
      np = move_particle(R, p, make_float2(Fw.x + Fk.x, Fw.y + Fk.y), xi, dt, &D.err);
    }
    R.recB[gi] = np;
    __syncwarp(act);
    count_into_cell(R, np.cell, act);
    if (np.cell != p.cell) atomicAdd(&D.moved[p.pid >= R.N1 ? 1 : 0], 1);
  }
}

// Keys of an unsorted upload in recB (initial sort).
__global__ void __launch_bounds__(256) k_count(const RunDesc* __restrict__ runs, const RunDyn* __restrict__ dyn,
                                               const Item* __restrict__ items, int nitems) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (run_failed(dyn, I.run)) continue;
    const RunDesc& R = runs[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, gi < R.N);
    if (gi < R.N) count_into_cell(R, R.recB[gi].cell, act);
  }
}

// ---------------------------------------------------------------------------
// Counting sort by cell: exclusive scan of the counts (the per-chunk totals
// come from the counting kernels; one CTA per run scans them, then every
// chunk of SCAN_CHUNK cells scans its counts from its offset), scatter by
// (start + atomic slot), then a fix-up that orders every cell holding two or
// more particles by particle index. The result is the order a stable sort by
// cell of the particle-index order gives, which is the reference's
// neighbour-list order after WCA_init (ascending index).

// Exclusive scan of one run's chunk totals into chunk_off; clears the
// totals. With end_step (a step's sort) its thread 0 also ends the
// run's step: the particle kernels that read the step counter and the dt
// bound are done, the scan and the scatter do not read them.
__global__ void __launch_bounds__(1024) k_chunk_scan(const RunDesc* __restrict__ runs, RunDyn* __restrict__ dyn,
                                                     int run0, int nruns, int end_step_flag, int adaptive,
                                                     int require_active) {
  __shared__ int sh[32];
  // up to 1024 * CPT chunks: C <= 4095 gives at most 8188
  constexpr int CPT = 8;
  for (int run = run0 + blockIdx.x; run < run0 + nruns; run += gridDim.x) {
    // the scan and the scatter of this sort follow this decision, taken
    // before end_step changes the steps budget
    const bool on = require_active ? run_active(dyn, run) : !run_failed(dyn, run);
    __syncthreads();
    if (threadIdx.x == 0) dyn[run].sorting = on ? 1 : 0;
    if (!on) continue;
    const RunDesc& R = runs[run];
    const int nch = (R.C * R.C + SCAN_CHUNK - 1) / SCAN_CHUNK;
    const int k0 = threadIdx.x * CPT;
    int v[CPT];
    int loc = 0;
#pragma unroll
    for (int k = 0; k < CPT; k++) {
      v[k] = k0 + k < nch ? R.chunk_sum[k0 + k] : 0;
      loc += v[k];
    }
    int ex = block_excl_scan(loc, sh);
#pragma unroll
    for (int k = 0; k < CPT; k++)
      if (k0 + k < nch) {
        R.chunk_off[k0 + k] = ex;
        R.chunk_sum[k0 + k] = 0;
        ex += v[k];
      }
    if (end_step_flag && threadIdx.x == 0) end_step(R, dyn[run], adaptive);
    __syncthreads();
  }
}

// Scan of one chunk's counts from its offset into start[]; clears the
// counts for the next sort. CTAs stride over the chunks and load the next
// chunk's counts before scanning the current one, so loads stay in flight.
struct ScanChunk {
  const RunDesc* R;
  int chunk, ncells;
  bool on;
  int v[SCAN_CHUNK / 256];
};

__device__ __forceinline__ void scan_load(const RunDesc* __restrict__ runs, const RunDyn* __restrict__ dyn,
                                          const Item& I, ScanChunk& S) {
  constexpr int PER = SCAN_CHUNK / 256;
  S.R = &runs[I.run];
  S.chunk = I.a;
  S.on = dyn[I.run].sorting;
  S.ncells = S.R->C * S.R->C;
  const int base = I.a * SCAN_CHUNK;
  const int c0 = base + threadIdx.x * PER;
  const int* cnt = S.R->count;
  if (base + SCAN_CHUNK <= S.ncells) {
    const int4 a = __ldcg(reinterpret_cast<const int4*>(&cnt[c0]));
    const int4 b = __ldcg(reinterpret_cast<const int4*>(&cnt[c0 + 4]));
    S.v[0] = a.x, S.v[1] = a.y, S.v[2] = a.z, S.v[3] = a.w;
    S.v[4] = b.x, S.v[5] = b.y, S.v[6] = b.z, S.v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < PER; k++) S.v[k] = c0 + k < S.ncells ? __ldcg(&cnt[c0 + k]) : 0;
  }
}

__global__ void __launch_bounds__(256) k_scan(const RunDesc* __restrict__ runs, const RunDyn* __restrict__ dyn,
                                              const Item* __restrict__ items, int nitems) {
  static_assert(SCAN_CHUNK == 2048, "eight counts per thread");
  __shared__ int sh[32];
  int it = blockIdx.x;
  if (it >= nitems) return;
  ScanChunk cur, nxt;
  scan_load(runs, dyn, items[it], cur);
  for (;;) {
    const int itn = it + gridDim.x;
    if (itn < nitems) scan_load(runs, dyn, items[itn], nxt);
    if (cur.on) scan_chunk_store<SCAN_CHUNK / 256>(CtaTeam(), *cur.R, cur.chunk, cur.ncells, cur.v, cur.R->chunk_off[cur.chunk], sh);
    if (itn >= nitems) break;
    it = itn;
    cur = nxt;
  }
}

// Places every particle at start[cell] + slot (slots in atomic order: the
// order within a cell is arbitrary and no result depends on it).
__global__ void __launch_bounds__(256) k_scatter(const RunDesc* __restrict__ runs,
                                                 const RunDyn* __restrict__ dyn,
                                                 const Item* __restrict__ items, int nitems) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    if (!dyn[I.run].sorting) continue;
    const RunDesc& R = runs[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    if (gi >= R.N) continue;
    scatter_particle(R, gi);
  }
}

// ---------------------------------------------------------------------------
// Pipelined stage step: any number of runs on power-of-two meshes with a
// fixed dt, six launches per step. As in the resident step, the move deposits
// the next step's density (the same fixed-point integers as the tiles, into
// each run's R.dacc), and the transform of the new density runs beside the
// cell sort:
//   k_step          forces, noise, move, re-binning, counts, next density;
//                   marks the runs that take part (`sorting`)
//   then, on two streams joined at the step's end:
//   k_pipe_scan -> k_pipe_scatter (step end)
//   k_pipe_fft<1> forward rows -> k_pipe_fft<2> columns + Green
//                 -> k_pipe_fft<0> inverse rows (the next step's force grids)
// Each kernel keeps its own registers and shared memory. Every transform CTA
// takes one item, of any mesh size (log2 Z in Item.b): no loop wraps a
// transform, whose per-thread offsets and twiddles the compiler would
// otherwise keep live across iterations.
#define BD_PIPE_SIZES(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

// pass 0: inverse rows, 1: forward rows from R.dacc, 2: columns + Green
template <int PASS, int L>
__device__ __forceinline__ void pipe_fft_sized(const RunDesc& R, const Item& I, float2* s) {
  if constexpr (L >= 11) {
    if (PASS == 0) big_rows_inv_item<L>(R, I.a, I.c, s, R.tw);
    else if (PASS == 1) big_rows_fwd_item<L, true>(R, I.a, I.c, s, R.tw);
    else big_cols_item<L>(R, I.a, I.c, s, R.tw);
  } else {
    if (PASS == 0) fft2_rows_inv_item<L, false>(CtaTeam(), R, I.a, I.c, s, R.tw);
    else if (PASS == 1) fft2_rows_fwd_item<L, false, true>(CtaTeam(), R, I.a, I.c, s, R.tw);
    else fft2_cols_item<L, false>(CtaTeam(), R, I.a, I.c, s, R.tw);
  }
}

template <int PASS>
__device__ __forceinline__ void pipe_fft_item(const RunDesc& R, const Item& I, float2* s) {
  switch (I.b) {
#define BD_CASE(L)                   \
  case L:                            \
    pipe_fft_sized<PASS, L>(R, I, s); \
    break;
    BD_PIPE_SIZES(BD_CASE)
#undef BD_CASE
    default:
      break;
  }
}

// One transform item per CTA, of any mesh size (pass as pipe_fft_item).
// Every pass checks `sorting` (whether the run takes part in this step,
// recorded by the particle kernel): the passes run beside the cell sort,
// whose last kernel ends the step and changes the step budget.
// Registers bounded for four CTAs per SM (64; a few values spill): the
// passes are bound by load latency, and the fourth CTA hides more of it
// (256-run ensemble: three passes 0.138 -> 0.129 ms).
template <int PASS>
__global__ void __launch_bounds__(FFT2_THREADS, 4) k_pipe_fft(const RunDesc* __restrict__ runs,
                                                            RunDyn* __restrict__ dyn,
                                                            const Item* __restrict__ items, int nitems) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x >= nitems) return;
  const Item I = items[blockIdx.x];
  if (!((volatile const RunDyn*)dyn)[I.run].sorting) return;
  pipe_fft_item<PASS>(runs[I.run], I, (float2*)smem);
}

// Scan chunk c of run R (256 threads, all call): its offset is the sum of
// the run's earlier chunk totals, formed here (no separate chunk scan).
__device__ __forceinline__ void scan_chunk_item(const RunDesc& R, int c, int* s_tmp) {
  static_assert(SCAN_CHUNK == 2048, "eight counts per thread");
  const int ncells = R.C * R.C;
  int loc = 0;
  for (int k = threadIdx.x; k < c; k += blockDim.x) loc += R.chunk_sum[k];
  const int ex = block_excl_scan(loc, s_tmp);
  if (threadIdx.x == blockDim.x - 1) s_tmp[0] = ex + loc;
  __syncthreads();
  const int off = s_tmp[0];
  __syncthreads();
  constexpr int PER = SCAN_CHUNK / 256;
  const int c0 = c * SCAN_CHUNK + threadIdx.x * PER;
  int cv[PER];
#pragma unroll
  for (int k = 0; k < PER; k++) cv[k] = c0 + k < ncells ? R.count[c0 + k] : 0;
  scan_chunk_store<SCAN_CHUNK / 256>(CtaTeam(), R, c, ncells, cv, off, s_tmp);
}

// PIPE_SCAN_GROUP chunks of one run per CTA (Item.a: the first): the counts
// (8 per chunk and thread) are requested before the offset, the sum of the run's
// earlier chunk totals, so both round trips overlap; one exclusive scan over
// the group. The starts are those of the per-chunk scan (one exclusive scan
// of the run's counts), so the group size is a free choice.
__global__ void __launch_bounds__(256) k_pipe_scan(const RunDesc* __restrict__ runs,
                                                   RunDyn* __restrict__ dyn,
                                                   const Item* __restrict__ groups, int ngroup) {
  constexpr int PER = PIPE_SCAN_GROUP * SCAN_CHUNK / 256;
  static_assert(PER % 4 == 0, "whole int4 vectors per thread");
  __shared__ int s_tmp[32];
  if ((int)blockIdx.x >= ngroup) return;
  const Item I = groups[blockIdx.x];
  if (!dyn[I.run].sorting) return;
  const RunDesc& R = runs[I.run];
  const int ncells = R.C * R.C, c0 = I.a;
  const int g0 = c0 * SCAN_CHUNK;
  const int base = g0 + threadIdx.x * PER;
  int v[PER];
  if (base + PER <= ncells) {
#pragma unroll
    for (int k = 0; k < PER; k += 4) {
      const int4 q = *reinterpret_cast<const int4*>(&R.count[base + k]);
      v[k] = q.x;
      v[k + 1] = q.y;
      v[k + 2] = q.z;
      v[k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < PER; k++) v[k] = base + k < ncells ? R.count[base + k] : 0;
  }
  int pre = 0;
  for (int k = threadIdx.x; k < c0; k += blockDim.x) pre += R.chunk_sum[k];
  int tot = 0;
#pragma unroll
  for (int k = 0; k < PER; k++) tot += v[k];
  // the offset: the block's sum of pre, read after the scan of pre
  const int ex_pre = block_excl_scan(pre, s_tmp);
  if (threadIdx.x == blockDim.x - 1) s_tmp[0] = ex_pre + pre;
  __syncthreads();
  const int off = s_tmp[0];
  __syncthreads();
  int acc = block_excl_scan(tot, s_tmp) + off;
  if (base + PER <= ncells) {
#pragma unroll
    for (int k = 0; k < PER; k += 4) {
      int4 w;
      w.x = acc;
      acc += v[k];
      w.y = acc;
      acc += v[k + 1];
      w.z = acc;
      acc += v[k + 2];
      w.w = acc;
      acc += v[k + 3];
      *reinterpret_cast<int4*>(&R.start[base + k]) = w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < PER; k++) {
      if (base + k < ncells) R.start[base + k] = acc;
      acc += v[k];
    }
  }
  if (g0 + PIPE_SCAN_GROUP * SCAN_CHUNK >= ncells && threadIdx.x == 0) R.start[ncells] = R.N;
}

// Scatter of particles [a * PIPE_SCATTER_UNIT, +PIPE_SCATTER_UNIT) of run R:
// four per thread, their loads and slot atomics issued together.
__device__ __forceinline__ void scatter_unit(const RunDesc& R, int a) {
  constexpr int Q = PIPE_SCATTER_UNIT / 256;
  const int g0 = a * PIPE_SCATTER_UNIT + threadIdx.x;
  Rec q[Q];
  int slot[Q], st[Q];
#pragma unroll
  for (int k = 0; k < Q; k++)
    if (g0 + 256 * k < R.N) q[k] = R.recB[g0 + 256 * k];
#pragma unroll
  for (int k = 0; k < Q; k++)
    if (g0 + 256 * k < R.N) {
      slot[k] = atomicSub(&R.count[q[k].cell], 1) - 1;
      st[k] = R.start[q[k].cell];
    }
#pragma unroll
  for (int k = 0; k < Q; k++)
    if (g0 + 256 * k < R.N) R.recA[st[k] + slot[k]] = q[k];
}

// One scatter unit per CTA, then, spread over all threads of the launch, the
// chunk totals of every sorting run cleared and (by its first chunk's
// thread) the run's step ended.
__global__ void __launch_bounds__(256) k_pipe_scatter(const RunDesc* __restrict__ runs, RunDyn* __restrict__ dyn,
                                                      const Item* __restrict__ units, int nunit,
                                                      const Item* __restrict__ chunks, int nchunk) {
  if ((int)blockIdx.x < nunit) {
    const Item I = units[blockIdx.x];
    if (dyn[I.run].sorting) scatter_unit(runs[I.run], I.a);
  }
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nchunk; c += gridDim.x * blockDim.x) {
    const Item I = chunks[c];
    if (!dyn[I.run].sorting) continue;
    runs[I.run].chunk_sum[I.a] = 0;
    if (I.a == 0) end_step(runs[I.run], dyn[I.run], 0);
  }
}

// ---------------------------------------------------------------------------
// Drop-in single routines.

// inv_gridDensity_*: Fk[pid] from the current force grid with `scheme`.
__global__ void __launch_bounds__(256) k_interp(const RunDesc* __restrict__ runs,
                                                const Item* __restrict__ items, int nitems,
                                                int scheme) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    const RunDesc& R = runs[I.run];
    const int gi = I.a * blockDim.x + threadIdx.x;
    if (gi >= R.N) continue;
    const Rec p = R.recA[gi];
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    R.Fk[p.pid] = (R.flags & F_IDGAS) ? make_float2(0.f, 0.f) : mesh_force<true>(R, p, ic, jc, scheme);
  }
}

// berechne_zufallskraefte: Fn[pid] for the current step.
__global__ void __launch_bounds__(256) k_noise(const RunDesc* __restrict__ runs,
                                               const RunDyn* __restrict__ dyn,
                                               const Item* __restrict__ items, int nitems) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    const RunDesc& R = runs[I.run];
    const int pid = I.a * blockDim.x + threadIdx.x;
    if (pid >= R.N) continue;
    R.Fn[pid] = (R.flags & F_NOWCA) ? make_float2(0.f, 0.f)
                                    : particle_noise(R.noise, R.seed, dyn[I.run].step, (uint32_t)pid);
  }
}

// optimaler_zeitschritt over the stored force/noise buffers.
__global__ void __launch_bounds__(256) k_dtbound(const RunDesc* __restrict__ runs,
                                                 RunDyn* __restrict__ dyn,
                                                 const Item* __restrict__ items, int nitems) {
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item I = items[it];
    const RunDesc& R = runs[I.run];
    const int pid = I.a * blockDim.x + threadIdx.x;
    if (pid >= R.N) continue;
    const float2 Fw = R.Fw[pid], Fk = R.Fk[pid], xi = R.Fn[pid];
    float bnd = fminf(dt_bound(Fw.x + Fk.x, xi.x, R.mrd, R.T), dt_bound(Fw.y + Fk.y, xi.y, R.mrd, R.T));
    if (!(bnd >= 0.f)) bnd = 3.0e38f;
    if (bnd < R.dt_max) atomicMin(&dyn[I.run].dt_bits, __float_as_uint(bnd));
  }
}

// Green's function tables in FP64 (kapkraefte_init and G,
// dynamik_methoden.cpp:585-593, 1384-1394), stored FP32:
//   green[ky][kx] = kapillar_vorfaktor * G(kx, ky) / Z^2, ky in [0, Z/2] (stored by
//   column, so a column pass reads it contiguously)
//   sxt[kx] = sin(qx dx)/dx, syt[ky] = sin(qy dx)/dx
__global__ void k_green(float* __restrict__ green, float* __restrict__ sxt,
                        float* __restrict__ syt, int Z, double kap, double lambda, double L) {
  const int n = Z / 2;
  const double dx = L / Z, dq = 2.0 * 3.14159265358979323846 / L;
  const long long total = (long long)Z * (n + 1);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ky = (int)(i / Z), kx = (int)(i - (long long)ky * Z);
    const double qx = dq * (((kx + n) % Z) - 0.5 * Z);
    const double qy = dq * (((ky + n) % Z) - 0.5 * Z);
    double G;
    if (kx == 0 && ky == 0 && lambda > 0.2 * L) G = 0.0;
    else {
      const double sx = sin(0.5 * qx * dx), sy = sin(0.5 * qy * dx);
      G = 1.0 / (4 * sx * sx / dx / dx + 4 * sy * sy / dx / dx + 1.0 / (lambda * lambda));
    }
    green[i] = (float)(kap * G / Z / Z);
    if (ky == 0) sxt[kx] = (float)(sin(qx * dx) / dx);
    if (kx == 0) syt[ky] = (float)(sin(qy * dx) / dx);
  }
}

// ---------------------------------------------------------------------------
// Two-launch pipelined step (any number of runs on power-of-two meshes with a
// fixed dt): the particle kernel, then one cooperative launch that holds the
// rest of the step and the start of the next, its phases separated by grid
// barriers:
//   C  scan chunks and the next forward row items (of the runs the particle
//      kernel marked as taking part)
//   D  scatter (PIPE_SCATTER_UNIT particles per unit) and the next column +
//      Green items; chunk totals cleared and steps ended
//   A  inverse row items of the runs that took part (the next step's force
//      grids; a run that did not keeps its spectrum and its grids)
// Unit u of a phase goes to CTA u mod G. The host interleaves transform
// items with scan chunks (and with scatter units) in one list, so every CTA
// holds a share of both kinds and on every SM the latency-bound transforms
// run beside the bandwidth-bound sort, which two kernels on two streams did
// not: the first kernel's CTAs filled the GPU before the second's started.

// meshes of the two-launch form (the host keeps larger ones on six launches)
#define BD_TAIL_FFT_SIZES(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

// A transform item called from the unit loops: not inlined, so the compiler
// cannot hoist the per-thread offsets and twiddle addresses of every pass
// and mesh size out of the loop (kept live across it, they spill).
// The dynamic shared memory is named here, not passed: a pointer parameter
// would be generic and every transform access a generic load.
template <int PASS, int L>
__device__ __noinline__ void tail_fft_sized(const RunDesc* R, int a, int c) {
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = (float2*)smem;
  if (PASS == 0) fft2_rows_inv_item<L, false>(CtaTeam(), *R, a, c, s, R->tw);
  else if (PASS == 1) fft2_rows_fwd_item<L, false, true>(CtaTeam(), *R, a, c, s, R->tw);
  else fft2_cols_item<L, false>(CtaTeam(), *R, a, c, s, R->tw);
}

template <int PASS>
__device__ __forceinline__ void tail_fft_item(const RunDesc* R, const Item& I) {
  switch (I.b) {
#define BD_CASE(L)                                \
  case L:                                         \
    tail_fft_sized<PASS, L>(R, I.a, I.c);         \
    break;
    BD_TAIL_FFT_SIZES(BD_CASE)
#undef BD_CASE
    default:
      break;
  }
}

// ts (optional, 4 entries): CTA 0 records the global timer at the start and
// after phases C, D and A (a barrier closes A when ts is given).
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k_pipe_tail(const RunDesc* __restrict__ runs, RunDyn* dyn,
                                                          const __grid_constant__ PipeTail P, unsigned* bar,
                                                          unsigned long long* ts) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_tmp[32];
  __shared__ int s_ok;
  const unsigned G = gridDim.x;
  const int b = blockIdx.x, nt = blockDim.x;
  unsigned ep = 0;
  const bool rec = ts && b == 0 && threadIdx.x == 0;
  if (rec) ts[0] = global_ns();
  const unsigned maxp = P.max_polls ? P.max_polls : BAR_MAX_POLLS;
  // which runs take part in this step: recorded by the particle kernel
  // before this launch; read with volatile loads (the run's state line may
  // sit in this SM's L1 while the step end in phase D changes it)
  volatile const RunDyn* dv = dyn;
  // a failed barrier leaves every run that took part in mid-step: all of them
  // are marked, so that no other form steps them before the host's recovery
  auto barrier = [&]() -> bool {
    if (P.skip_barrier == (int)ep + 1 && b == P.skip_cta) return false;
    if (grid_barrier(bar, ++ep * G, maxp, &dyn[0].err, &s_ok)) return true;
    for (int c = threadIdx.x; c < P.nchunk; c += nt) {
      const Item I = P.chunks[c];
      if (I.a == 0 && dv[I.run].sorting) atomicOr(&dyn[I.run].err, E_BARRIER_TIMEOUT);
    }
    return false;
  };
  for (int u = b; u < P.ncu; u += G) {
    const Item I = P.cunits[u];
    if (!dv[I.run].sorting) continue;
    const RunDesc& R = runs[I.run];
    if (I.b < 0) scan_chunk_item(R, I.a, s_tmp);
    else tail_fft_item<1>(&R, I);
  }
  if (!barrier()) return;
  if (rec) ts[1] = global_ns();
  for (int u = b; u < P.ndu; u += G) {
    const Item I = P.dunits[u];
    if (!dv[I.run].sorting) continue;
    const RunDesc& R = runs[I.run];
    if (I.b < 0) scatter_unit(R, I.a);
    else tail_fft_item<2>(&R, I);
  }
  for (int c = b * nt + threadIdx.x; c < P.nchunk; c += (int)G * nt) {
    const Item I = P.chunks[c];
    if (!dv[I.run].sorting) continue;
    runs[I.run].chunk_sum[I.a] = 0;
    if (I.a == 0) end_step(runs[I.run], dyn[I.run], 0);
  }
  if (!barrier()) return;
  if (rec) ts[2] = global_ns();
  for (int u = b; u < P.ninv; u += G) {
    const Item I = P.inv[u];
    if (dv[I.run].sorting) tail_fft_item<0>(&runs[I.run], I);
  }
  if (ts) {
    if (!barrier()) return;
    if (rec) ts[3] = global_ns();
  }
  grid_exit(bar, G);
}

#define BD_TAIL_SHAPES(X) X(2) X(3) X(4)

int pipe_tail_configure(PipeTail& P, int device) {
  int nsm = 0, per = 0;
  cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return (int)e;
  switch (P.minb) {
#define BD_CASE(M)                                                                                   \
  case M:                                                                                            \
    e = cudaFuncSetAttribute(k_pipe_tail<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem); \
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pipe_tail<M>, 256, P.smem); \
    break;
    BD_TAIL_SHAPES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return (int)e;
  if (per <= 0) return (int)cudaErrorInvalidConfiguration;
  P.grid = std::min(per, P.minb) * nsm;
  return 0;
}

int launch_pipe_tail(const RunDesc* runs, RunDyn* dyn, const PipeTail& P, unsigned* bar, cudaStream_t s,
                     unsigned long long* ts) {
  cudaError_t e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.grid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  switch (P.minb) {
#define BD_CASE(M)                                                         \
  case M:                                                                  \
    e = cudaLaunchKernelEx(&cfg, k_pipe_tail<M>, runs, dyn, P, bar, ts); \
    break;
    BD_TAIL_SHAPES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
  return (int)e;
}

// ---------------------------------------------------------------------------
// TimestepInfo diagnostics (zeitschritt_debug, dynamik_methoden.cpp:168-211,
// and the *_debug force routines) plus the WCA potential energy and virial
// in FP64. One thread per particle of the sorted array, after the forces of
// the current positions are in Fw/Fk/Fn (per particle index):
//  - the largest |F| of each force kind, as (|F|^2 bits << 32 | index) maxima;
//  - the pairs the reference's WCA loops examine: same-species neighbours of
//    every particle (i != j) and type-2 neighbours of every type-1 particle
//    (berechne_WCA11/22 and addiere_WCA12 loop over the 3x3 cells);
//  - over all pairs within the cutoff, each seen from both ends and halved:
//    U = 4 eps (s^-12 - s^-6) + eps with s = r*sigma (the potential whose
//    gradient is the uncapped WCA force), and r.F with the force the step
//    uses (capped at maxPairWCA).
struct DiagAcc {
  double energy, virial;
  unsigned long long maxF[3];  // WCA, capillary, noise
  unsigned long long pairs;
};

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}

__global__ void __launch_bounds__(256) k_diag(const RunDesc* __restrict__ runs, DiagAcc* __restrict__ acc) {
  const RunDesc& R = runs[0];
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0, w = 0.0;
  unsigned long long pairs = 0, mx[3] = {0, 0, 0};
  if (gi < R.N) {
    const Rec p = R.recA[gi];
    const float2* Fs[3] = {R.Fw, R.Fk, R.Fn};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float2 f = Fs[k][p.pid];
      const float m = f.x * f.x + f.y * f.y;
      mx[k] = ((unsigned long long)__float_as_uint(m) << 32) | (unsigned)p.pid;
    }
    if (!(R.flags & F_IDGAS)) {
      const int C = R.C;
      int ic, jc;
      cell_ij(R, p.cell, ic, jc);
      const bool sp = p.pid >= R.N1;
      for (int da = -1; da <= 1; da++) {
        const int row = wrap1(ic + da, C) * C;
        for (int db = -1; db <= 1; db++) {
          const int g = row + wrap1(jc + db, C);
          for (int j = R.start[g]; j < R.start[g + 1]; j++) {
            if (j == gi) continue;
            const Rec q = R.recA[j];
            const bool sq = q.pid >= R.N1;
            if (sp == sq || !sp) pairs++;
            const int t = sp == sq ? (sp ? 1 : 0) : 2;
            double dx = ((double)p.ox - (double)q.ox) - da * R.B_d;
            double dy = ((double)p.oy - (double)q.oy) - db * R.B_d;
            if (R.flags & F_SMALLBOX) {
              dx -= R.L_d * rint(dx / R.L_d);
              dy -= R.L_d * rint(dy / R.L_d);
            }
            const double sig = R.wsig[t];
            const double a2s = (dx * dx + dy * dy) * sig * sig;
            if (a2s > (double)R.cut2) continue;
            const double eps = (double)R.wpre[t] / (24.0 * sig);
            const double i2 = 1.0 / a2s, i6 = i2 * i2 * i2;
            e += 4.0 * eps * (i6 * i6 - i6) + eps;
            double f = (double)R.wpre[t] * i6 * i2 * (2.0 * i6 - 1.0);  // 24 eps sigma (2 s^-14 - s^-8)
            if (f > (double)R.maxPair) f = R.maxPair;
            w += f * a2s / sig;  // r . F = f * sigma * r^2
          }
        }
      }
    }
  }
  // block reductions, one atomic per block and quantity
  __shared__ double s_e[8], s_w[8];
  __shared__ unsigned long long s_p[8], s_m[3][8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_xor_sync(0xffffffffu, e, o);
    w += __shfl_xor_sync(0xffffffffu, w, o);
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) mx[k] = warp_max_u64(mx[k]);
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_e[wid] = e;
    s_w[wid] = w;
    s_p[wid] = pairs;
    for (int k = 0; k < 3; k++) s_m[k][wid] = mx[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double te = 0.0, tw = 0.0;
    unsigned long long tp = 0, tm[3] = {0, 0, 0};
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
      te += s_e[k];
      tw += s_w[k];
      tp += s_p[k];
      for (int q = 0; q < 3; q++) tm[q] = s_m[q][k] > tm[q] ? s_m[q][k] : tm[q];
    }
    atomicAdd(&acc->energy, 0.5 * te);
    atomicAdd(&acc->virial, 0.5 * tw);
    atomicAdd(&acc->pairs, tp);
    for (int q = 0; q < 3; q++) atomicMax(&acc->maxF[q], tm[q]);
  }
}

int launch_diag(const RunDesc* runs, int N, void* acc, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(acc, 0, sizeof(DiagAcc), s);
  if (e != cudaSuccess) return (int)e;
  k_diag<<<(N + 255) / 256, 256, 0, s>>>(runs, (DiagAcc*)acc);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

size_t diag_bytes() { return sizeof(DiagAcc); }

// ---------------------------------------------------------------------------
// Observables computed from the resident state (the reference's in-run
// auswertung.cpp, validation tools here).

// Pair-distance histogram for g11 / g12 / g22 (record_korrelationsfunktion11/
// 12/22, auswertung.cpp:110-188): every pair once (11, 22: the lower particle
// index of the pair counts; 12: type 1 against type 2), minimum-image
// distance in FP64 from the cell and offset, bin (int)(r / dr). One thread
// per particle of the sorted array searches the cells within `range` of its
// own (the whole box when the range covers it); the CTA counts in shared
// memory and adds to hist[bins] once.
__global__ void __launch_bounds__(256) k_korr(const RunDesc* __restrict__ runs, int which, int bins, double dr,
                                              int range, unsigned long long* __restrict__ hist) {
  extern __shared__ unsigned sh_hist[];
  const RunDesc& R = runs[0];
  for (int b = threadIdx.x; b < bins; b += blockDim.x) sh_hist[b] = 0u;
  __syncthreads();
  const int C = R.C;
  const bool all_rows = 2 * range + 1 >= C;
  for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < R.N; gi += gridDim.x * blockDim.x) {
    const Rec p = R.recA[gi];
    const int si = p.pid >= R.N1;
    if ((which == 0 && si != 0) || (which == 1 && si != 0) || (which == 2 && si != 1)) continue;
    const int want = which == 1 ? 1 : si;
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    const double xi = ic * R.B_d + (double)p.ox, yi = jc * R.B_d + (double)p.oy;
    const int nrows = all_rows ? C : 2 * range + 1;
    for (int a = 0; a < nrows; a++) {
      const int row = all_rows ? a : wrapi(ic - range + a, C);
      // columns jc-range .. jc+range as at most two contiguous runs
      int segs[2][2];
      int ns = 1;
      if (all_rows) {
        segs[0][0] = 0, segs[0][1] = C;
      } else {
        const int j0 = wrapi(jc - range, C), len = 2 * range + 1;
        if (j0 + len <= C) {
          segs[0][0] = j0, segs[0][1] = j0 + len;
        } else {
          segs[0][0] = j0, segs[0][1] = C, segs[1][0] = 0, segs[1][1] = j0 + len - C;
          ns = 2;
        }
      }
      for (int sgi = 0; sgi < ns; sgi++) {
        const int beg = R.start[row * C + segs[sgi][0]], end = R.start[row * C + segs[sgi][1]];
        for (int j = beg; j < end; j++) {
          const Rec q = R.recA[j];
          const int sj = q.pid >= R.N1;
          if (sj != want) continue;
          if (which != 1 && q.pid >= p.pid) continue;  // each pair once
          int qi, qj;
          cell_ij(R, q.cell, qi, qj);
          double dx = xi - (qi * R.B_d + (double)q.ox);
          double dy = yi - (qj * R.B_d + (double)q.oy);
          dx -= R.L_d * rint(dx / R.L_d);
          dy -= R.L_d * rint(dy / R.L_d);
          const int idx = (int)(sqrt(dx * dx + dy * dy) / dr);
          if (idx >= 0 && idx < bins) atomicAdd(&sh_hist[idx], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += blockDim.x)
    if (sh_hist[b]) atomicAdd(&hist[b], (unsigned long long)sh_hist[b]);
}

// Density Fourier sums of one species on the lattice k = dq (i, j),
// 0 <= i, j < qbins, i^2 + j^2 <= qbins^2 (record_ftrho_unkorrigiert,
// auswertung.cpp:307-380): re + i im = sum over particles of exp(i k.r), in
// FP64. Each thread owns up to FT_KPT lattice points and sums over the
// particles its CTA stages in shared memory; one atomic add per CTA and point.
constexpr int FT_KPT = 16;
__global__ void __launch_bounds__(256) k_ftrho(const RunDesc* __restrict__ runs, int species, int qbins, double dq,
                                               double* __restrict__ re, double* __restrict__ im) {
  __shared__ double sx[256], sy[256];
  __shared__ int sn;
  const RunDesc& R = runs[0];
  const int nk = qbins * qbins;
  double ar[FT_KPT], ai[FT_KPT];
#pragma unroll
  for (int m = 0; m < FT_KPT; m++) ar[m] = ai[m] = 0.0;
  for (int base = blockIdx.x * 256; base < R.N; base += gridDim.x * 256) {
    if (threadIdx.x == 0) sn = 0;
    __syncthreads();
    const int gi = base + threadIdx.x;
    if (gi < R.N) {
      const Rec p = R.recA[gi];
      if ((p.pid >= R.N1) == (species == 1)) {
        int ic, jc;
        cell_ij(R, p.cell, ic, jc);
        const int slot = atomicAdd(&sn, 1);
        sx[slot] = ic * R.B_d + (double)p.ox;
        sy[slot] = jc * R.B_d + (double)p.oy;
      }
    }
    __syncthreads();
    const int n = sn;
#pragma unroll
    for (int m = 0; m < FT_KPT; m++) {
      const int k = threadIdx.x + m * 256;
      if (k >= nk) break;
      const int i = k / qbins, j = k - (k / qbins) * qbins;
      if (i * i + j * j > qbins * qbins) continue;
      for (int t = 0; t < n; t++) {
        double sn_, cs;
        sincos(dq * (sx[t] * i + sy[t] * j), &sn_, &cs);
        ar[m] += cs;
        ai[m] += sn_;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < FT_KPT; m++) {
    const int k = threadIdx.x + m * 256;
    if (k >= nk) break;
    if (ar[m] != 0.0 || ai[m] != 0.0) {
      atomicAdd(&re[k], ar[m]);
      atomicAdd(&im[k], ai[m]);
    }
  }
}

int launch_korr(const RunDesc* runs, int N, int which, int bins, double dr, int range, unsigned long long* hist,
                cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(hist, 0, (size_t)bins * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return (int)e;
  const int grid = std::max(1, std::min((N + 255) / 256, 148 * 8));
  k_korr<<<grid, 256, (size_t)bins * sizeof(unsigned), s>>>(runs, which, bins, dr, range, hist);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

int launch_ftrho(const RunDesc* runs, int N, int species, int qbins, double dq, double* re, double* im,
                 cudaStream_t s) {
  const size_t nk = (size_t)qbins * qbins;
  cudaError_t e = cudaMemsetAsync(re, 0, nk * sizeof(double), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(im, 0, nk * sizeof(double), s);
  if (e != cudaSuccess) return (int)e;
  const int grid = std::max(1, std::min((N + 255) / 256, 148 * 4));
  k_ftrho<<<grid, 256, 0, s>>>(runs, species, qbins, dq, re, im);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// Local densities of the offline analysis (main_auswertung.cpp:182-390),
// from the resident state. Lattice of n x n cells of width w = L/n; each
// particle adds w_x w_y drho (drho = 1/w^2) to nine cells with FP64 atomic
// adds. A fixed-point sum would be order-independent, but its absolute
// resolution turns cells holding only the tail of a TSC weight (values near
// 1e-19) into empty cells, and the reference counts such a cell in the
// |rho1 - rho2| / rho thresholds; FP64 adds keep every cell's value to a few
// ulp of itself. All weight arithmetic is written with explicit
// round-to-nearest operations, so no product is fused into a following add
// and each contribution equals the reference's FP64 expression.
__device__ __forceinline__ void snap_tsc(double x, double w, int n, int* kk, double* wt) {
  int k = __double2int_rz(__ddiv_rn(x, w));  // (int)(x/width)
  k = k % n;
  if (k < 0) k += n;  // x < 0 (never from the integrator) stays on the lattice
  kk[0] = (k - 1 + n) % n;
  kk[1] = k;
  kk[2] = (k + 1) % n;
  const double d = __dsub_rn(x, __dmul_rn((double)k + 0.5, w));
  wt[1] = __dsub_rn(0.75, __ddiv_rn(__dmul_rn(d, d), __dmul_rn(w, w)));
  double t = 1.5 - fabs(__ddiv_rn(__dadd_rn(d, w), w));
  wt[0] = __dmul_rn(__dmul_rn(0.5, t), t);
  t = 1.5 - fabs(__ddiv_rn(__dsub_rn(d, w), w));
  wt[2] = __dmul_rn(__dmul_rn(0.5, t), t);
}

__global__ void __launch_bounds__(256) k_lokdens(const RunDesc* __restrict__ runs, LdSnap sp,
                                                 double* __restrict__ grid) {
  const RunDesc& R = runs[0];
  const size_t cells = (size_t)sp.n * sp.n;
  for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < R.N; gi += gridDim.x * blockDim.x) {
    const Rec p = R.recA[gi];
    const int s = p.pid >= R.N1;
    int ic, jc;
    cell_ij(R, p.cell, ic, jc);
    const double x = __dadd_rn(__dmul_rn((double)ic, R.B_d), (double)p.ox);
    const double y = __dadd_rn(__dmul_rn((double)jc, R.B_d), (double)p.oy);
    int kx[3], ky[3];
    double wx[3], wy[3];
    snap_tsc(x, sp.w, sp.n, kx, wx);
    snap_tsc(y, sp.w, sp.n, ky, wy);
    double* G = grid + s * cells;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int b = 0; b < 3; b++)
        atomicAdd(&G[(size_t)kx[a] * sp.n + ky[b]], __dmul_rn(__dmul_rn(wx[a], wy[b]), sp.drho));
  }
}

// Histogram bin of main_auswertung.cpp:337-355: (int) truncation of v,
// clamped to [0, bins); values at or above bins are clamped before the
// conversion.
__device__ __forceinline__ int snap_bin(double v, int bins) {
  if (v >= (double)bins) return bins - 1;
  const int b = __double2int_rz(v);
  return b < 0 ? 0 : b;
}

// Histograms and threshold counts over the lattice (main_auswertung.cpp:
// 302-390). hist: [4][bins] counts (rho1, rho2, rho1+rho2, rho1-rho2), then
// [7] threshold counts.
__global__ void __launch_bounds__(256) k_rhohist(const LdHist hp, const double* __restrict__ grid,
                                                 unsigned* __restrict__ hist) {
  extern __shared__ unsigned sh_rh[];
  const int bins = hp.bins, nb = 4 * bins + 7;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sh_rh[i] = 0u;
  __syncthreads();
  const size_t cells = (size_t)hp.n * hp.n;
  unsigned over[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += (size_t)gridDim.x * blockDim.x) {
    const double rho1 = grid[c], rho2 = grid[cells + c];
    const double rho = __dadd_rn(rho1, rho2), drho = __dsub_rn(rho1, rho2);
#pragma unroll
    for (int t = 0; t < 3; t++) over[t] += rho > hp.rho_thresh[t];
    const double q = __ddiv_rn(fabs(drho), rho);  // 0/0 for an empty cell: never over
#pragma unroll
    for (int t = 0; t < 4; t++) over[3 + t] += q > hp.drho_thresh[t];
    atomicAdd(&sh_rh[0 * bins + snap_bin(__dsub_rn(__ddiv_rn(rho1, hp.dbin), 0.5), bins)], 1u);
    atomicAdd(&sh_rh[1 * bins + snap_bin(__dsub_rn(__ddiv_rn(rho2, hp.dbin), 0.5), bins)], 1u);
    atomicAdd(&sh_rh[2 * bins + snap_bin(__dsub_rn(__ddiv_rn(rho, hp.dbin), 0.5), bins)], 1u);
    atomicAdd(&sh_rh[3 * bins + snap_bin(__dadd_rn(__dsub_rn(__ddiv_rn(drho, hp.dbin), 0.5), (double)(bins / 2)),
                                         bins)],
              1u);
  }
#pragma unroll
  for (int t = 0; t < 7; t++) {
    const unsigned v = __reduce_add_sync(0xffffffffu, over[t]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&sh_rh[4 * bins + t], v);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    if (sh_rh[i]) atomicAdd(&hist[i], sh_rh[i]);
}

int launch_lokdens(const RunDesc* runs, int N, const LdSnap& sp, const LdHist& hp, double* grid, unsigned* hist,
                   cudaStream_t s) {
  const size_t cells = (size_t)sp.n * sp.n;
  cudaError_t e = cudaMemsetAsync(grid, 0, 2 * cells * sizeof(double), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(hist, 0, (4 * (size_t)hp.bins + 7) * sizeof(unsigned), s);
  if (e != cudaSuccess) return (int)e;
  if (N > 0) k_lokdens<<<std::max(1, std::min((N + 255) / 256, 148 * 8)), 256, 0, s>>>(runs, sp, grid);
  const int g2 = (int)std::max<size_t>(1, std::min<size_t>((cells + 255) / 256, 148 * 4));
  k_rhohist<<<g2, 256, (4 * (size_t)hp.bins + 7) * sizeof(unsigned), s>>>(hp, grid, hist);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------------------
// host-side launchers

#define BD_LAUNCH_CHECK()                                                                    \
  do {                                                                                       \
    cudaError_t e__ = cudaGetLastError();                                                    \
    if (e__ != cudaSuccess) {                                                                \
      std::fprintf(stderr, "bd: %s:%d: launch: %s\n", __FILE__, __LINE__, cudaGetErrorString(e__)); \
      return (int)e__;                                                                       \
    }                                                                                        \
  } while (0)

static inline int grid_for(int n, int cap) { return n < cap ? (n > 0 ? n : 1) : cap; }

// SMs of the current device (asked once per device)
static int sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

size_t deposit_smem(int mt_max, int rows_max) {
  return (size_t)mt_max * mt_max * 8 + (size_t)(3 * 2 * rows_max + 4) * 4;  // lo + hi words, segments
}

int launch_deposit(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, int mt_max,
                   int rows_max, int scheme_override, int require_active, cudaStream_t s) {
  if (n <= 0) return 0;
  const size_t sm = deposit_smem(mt_max, rows_max);
  k_deposit<<<grid_for(n, 65535), 256, sm, s>>>(runs, dyn, items, n, scheme_override, require_active);
  BD_LAUNCH_CHECK();
  return 0;
}

// the power-of-two kernels of every mesh size 8..4096, by log2(Z)
#define BD_FFT2_SIZES(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

static int launch_fft2(int pass, int lz, const RunDesc* runs, const RunDyn* dyn, const FftPass& p,
                       int require_active, cudaStream_t s) {
  if (p.n <= 0) return 0;
  switch (lz) {
#define BD_CASE(L)                                                                                      \
  case L:                                                                                               \
    if (pass == 0)                                                                                      \
      k_fft2_rows_fwd<L><<<p.n, p.threads, p.smem, s>>>(runs, dyn, p.items, p.n, require_active);      \
    else if (pass == 1)                                                                                 \
      k_fft2_cols<L><<<p.n, p.threads, p.smem, s>>>(runs, dyn, p.items, p.n, require_active);        \
    else                                                                                                \
      k_fft2_rows_inv<L><<<p.n, p.threads, p.smem, s>>>(runs, dyn, p.items, p.n, require_active);      \
    break;
    BD_FFT2_SIZES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_fft(const RunDesc* runs, const RunDyn* dyn, const FftPass gen[3], const Fft2Group* g2, int ng2,
               int require_active, cudaStream_t s, cudaEvent_t* ev, int first, int last) {
  for (int pass = first; pass <= last; pass++) {
    const FftPass& g = gen[pass];
    if (g.n > 0) {
      if (pass == 0)
        k_fft_rows_fwd<<<grid_for(g.n, 65535), FFT_THREADS, g.smem, s>>>(runs, dyn, g.items, g.n, require_active);
      else if (pass == 1)
        k_fft_cols<<<grid_for(g.n, 65535), FFT_THREADS, g.smem, s>>>(runs, dyn, g.items, g.n, require_active);
      else
        k_fft_rows_inv<<<grid_for(g.n, 65535), FFT_THREADS, g.smem, s>>>(runs, dyn, g.items, g.n, require_active);
      BD_LAUNCH_CHECK();
    }
    for (int k = 0; k < ng2; k++) {
      const int e = launch_fft2(pass, g2[k].lz, runs, dyn, g2[k].pass[pass], require_active, s);
      if (e) return e;
    }
    if (ev) cudaEventRecord(ev[pass], s);
  }
  return 0;
}

int launch_particles(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int mode,
                     int mask, int require_active, cudaStream_t s, int shape) {
  if (n <= 0) return 0;
  const int g = grid_for(n, 65535);
  if (shape == PART_SHAPE_5CTA)
    k_particles<5><<<g, 256, 0, s>>>(runs, dyn, items, n, mode, mask, require_active);
  else
    k_particles<4><<<g, 256, 0, s>>>(runs, dyn, items, n, mode, mask, require_active);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_step(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int deposit, int large,
                cudaStream_t s, int shape) {
  if (n <= 0) return 0;
  const bool five = shape == PART_SHAPE_5CTA;
  if (large) {
    // one CTA per item, four per SM: the block that starts when this one ends
    constexpr int ahead = 592;
    const int g = grid_for(n, 65535);
    if (deposit) k_step<4, true, ahead><<<g, 256, 0, s>>>(runs, dyn, items, n);
    else k_step<4, false, ahead><<<g, 256, 0, s>>>(runs, dyn, items, n);
  } else {
    // one wave of resident CTAs, each taking items blockIdx.x, +gridDim.x, ...
    // (256-run ensemble: 398 us with one CTA per item, 333 us)
    // resident CTAs per SM of each shape, asked once per process (every
    // device of one process is taken to be the same GPU model)
    static int resident[2] = {0, 0};
    if (!resident[five]) {
      int per = 0;
      const cudaError_t e = five ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_step<5, true, 0>, 256, 0)
                                 : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_step<4, true, 0>, 256, 0);
      resident[five] = (e == cudaSuccess && per > 0) ? per : 1;
    }
    const int g = deposit ? grid_for(n, resident[five] * sm_count()) : grid_for(n, 65535);
    if (deposit) {
      if (five) k_step<5, true, 0><<<g, 256, 0, s>>>(runs, dyn, items, n);
      else k_step<4, true, 0><<<g, 256, 0, s>>>(runs, dyn, items, n);
    } else {
      if (five) k_step<5, false, 0><<<g, 256, 0, s>>>(runs, dyn, items, n);
      else k_step<4, false, 0><<<g, 256, 0, s>>>(runs, dyn, items, n);
    }
  }
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_pipe_fft(int pass, const RunDesc* runs, RunDyn* dyn, const Item* items, int n, size_t smem,
                    cudaStream_t s) {
  if (n <= 0) return 0;
  if (pass == 0) k_pipe_fft<0><<<n, FFT2_THREADS, smem, s>>>(runs, dyn, items, n);
  else if (pass == 1) k_pipe_fft<1><<<n, FFT2_THREADS, smem, s>>>(runs, dyn, items, n);
  else k_pipe_fft<2><<<n, FFT2_THREADS, smem, s>>>(runs, dyn, items, n);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_pipe_scan(const RunDesc* runs, RunDyn* dyn, const Item* groups, int ngroup, cudaStream_t s) {
  if (ngroup <= 0) return 0;
  k_pipe_scan<<<ngroup, 256, 0, s>>>(runs, dyn, groups, ngroup);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_pipe_scatter(const RunDesc* runs, RunDyn* dyn, const Item* units, int nunit, const Item* chunks,
                        int nchunk, cudaStream_t s) {
  if (nunit + nchunk <= 0) return 0;
  k_pipe_scatter<<<nunit > 0 ? nunit : 1, 256, 0, s>>>(runs, dyn, units, nunit, chunks, nchunk);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_move(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int require_active,
                int refresh_only, cudaStream_t s) {
  if (n <= 0) return 0;
  k_move<<<grid_for(n, 65535), 256, 0, s>>>(runs, dyn, items, n, require_active, refresh_only);
  BD_LAUNCH_CHECK();
  return 0;
}

// Records in particle-index order (dst[pid] = src[i]), for the copy of a
// run's positions to the host: the host then writes the caller's arrays in
// order instead of at scattered indices.
__global__ void __launch_bounds__(256) k_records_by_pid(const Rec* __restrict__ src, Rec* __restrict__ dst, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Rec q = src[i];
    if ((unsigned)q.pid < (unsigned)n) dst[q.pid] = q;  // every pid of a run is in [0, n)
  }
}

int launch_records_by_pid(const Rec* src, Rec* dst, int n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_records_by_pid<<<std::min((n + 255) / 256, 4096), 256, 0, s>>>(src, dst, n);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_count(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_count<<<grid_for(n, 65535), 256, 0, s>>>(runs, dyn, items, n);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_sort(const RunDesc* runs, RunDyn* dyn, int run0, int nruns, const Item* chunks, int nchunks,
                const Item* parts, int nparts, int end_step_flag, int adaptive, int require_active, cudaStream_t s,
                cudaEvent_t* ev) {
  if (nchunks > 0) {
    k_chunk_scan<<<nruns, 1024, 0, s>>>(runs, dyn, run0, nruns, end_step_flag, adaptive, require_active);
    BD_LAUNCH_CHECK();
    k_scan<<<grid_for(nchunks, 148 * 8), 256, 0, s>>>(runs, dyn, chunks, nchunks);
    BD_LAUNCH_CHECK();
  }
  if (ev) cudaEventRecord(ev[0], s);
  if (nparts > 0) {
    k_scatter<<<grid_for(nparts, 65535), 256, 0, s>>>(runs, dyn, parts, nparts);
    BD_LAUNCH_CHECK();
  }
  if (ev) {
    cudaEventRecord(ev[1], s);
    cudaEventRecord(ev[2], s);
  }
  return 0;
}

int launch_interp(const RunDesc* runs, const Item* items, int n, int scheme, cudaStream_t s) {
  if (n <= 0) return 0;
  k_interp<<<grid_for(n, 65535), 256, 0, s>>>(runs, items, n, scheme);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_noise(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_noise<<<grid_for(n, 65535), 256, 0, s>>>(runs, dyn, items, n);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_dtbound(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_dtbound<<<grid_for(n, 65535), 256, 0, s>>>(runs, dyn, items, n);
  BD_LAUNCH_CHECK();
  return 0;
}

int launch_green(float* green, float* sxt, float* syt, int Z, double kap, double lambda,
                 double L, cudaStream_t s) {
  const long long total = (long long)Z * (Z / 2 + 1);
  const int blocks = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  k_green<<<blocks, 256, 0, s>>>(green, sxt, syt, Z, kap, lambda, L);
  BD_LAUNCH_CHECK();
  return 0;
}

int set_kernel_attributes() {
  cudaError_t e;
  e = cudaFuncSetAttribute(k_fft_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(k_fft_rows_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(k_fft_rows_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
#define BD_ATTR(L)                                                                                     \
  e = cudaFuncSetAttribute(k_fft2_rows_fwd<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM); \
  if (e != cudaSuccess) return (int)e;                                                                  \
  e = cudaFuncSetAttribute(k_fft2_cols<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);     \
  if (e != cudaSuccess) return (int)e;                                                                  \
  e = cudaFuncSetAttribute(k_fft2_rows_inv<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM); \
  if (e != cudaSuccess) return (int)e;
  BD_FFT2_SIZES(BD_ATTR)
#undef BD_ATTR
  e = cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(k_pipe_fft<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(k_pipe_fft<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(k_pipe_fft<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_FFT_SMEM);
  if (e != cudaSuccess) return (int)e;
  return 0;
}

}  // namespace bd
