// A call of one step of a run on a power-of-two mesh with a fixed dt, in one
// cooperative launch: the phases of the resident step (bd_resident.cuh) from
// the same state to the same state and bits, two CTAs of 256 threads per SM.
//
// A launch of one step pays the resident kernel's start (a description copied
// to shared memory, the step budget before the first phase) and gains nothing
// from its loop, and with 1024 threads per CTA and the halves apart its phases
// are built to overlap in steady state. Here everything a phase reads first is
// in flight before the first transform, the budget is looked at after it, the
// run's description is in the parameter bank and the kernel is a third of the
// code (fetched from memory again when other work has used the L2). What
// bounds it is the chain of launch, four phases and three grid barriers.
// Measured, us per call of one step, L2 flushed before it (resident kernel |
// this one): 2000 particles, 128^2 34.0 | 25.4; 16 384, 256^2 34.8 | 28.6; 65 536,
// 512^2 42.4 | 31.5; 262 144, 1024^2 97.8 | 76.0; not flushed 23.2 | 25.2, 29.0 |
// 27.6, 37.4 | 31.2, 86.0 | 67.9. Every size takes this kernel: for the smallest
// the resident launch is 2 us ahead where calls follow each other directly and
// 8.6 behind where other work has used the L2 in between.
#include <algorithm>

#include "bd_items.cuh"

namespace bd {

constexpr size_t ONE_TW_BYTES(int lz) { return (((size_t)8 << lz) + 255) & ~(size_t)255; }

// ts (optional, FUSED_PHASES + 1 entries): CTA 0 records the global timer at
// the start and after every phase's barrier.
template <int LZ>
__global__ void __launch_bounds__(256, 2) k_one_step(const __grid_constant__ RunDesc R, RunDyn* __restrict__ dyn,
                                                     const __grid_constant__ OneStepPlan P, unsigned* bar,
                                                     unsigned long long* ts) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_tmp[32];
  __shared__ int s_ok;
  constexpr int Z = 1 << LZ, nZ = Z / 2 + 1;
  RunDyn& D = dyn[0];
  const int b = blockIdx.x, G = gridDim.x;
  // the spectrum rows of this CTA's inverse row item go to L2 first
  if (threadIdx.x == 0 && b < P.nri)
    l2_prefetch_share(R.spec2 + ((size_t)b << P.lri) * (Z / 2), ((size_t)1 << P.lri) * (Z / 2) * sizeof(float4), 0, 1);
  constexpr int TWR = (Z + 255) / 256;
  float2 twr[TWR];
#pragma unroll
  for (int k = 0; k < TWR; k++)
    if (threadIdx.x + 256 * k < Z) twr[k] = R.tw[threadIdx.x + 256 * k];
  // looked at after the inverse row pass, which only rebuilds the force grid
  // from the unchanged spectrum: its load does not hold up the start
  const long long steps_left = ((volatile RunDyn*)dyn)->steps_left;
  if (threadIdx.x == 0) {
    l2_prefetch_share(R.green, (size_t)Z * nZ * sizeof(float), b, G);
    l2_prefetch_share(R.recA, (size_t)R.N * sizeof(Rec), b, G);
    l2_prefetch_share(R.start, ((size_t)R.C * R.C + 1) * sizeof(int), b, G);
    l2_prefetch_share(R.count, (size_t)R.C * R.C * sizeof(int), b, G);
    l2_prefetch_share(R.dacc, (size_t)Z * Z * sizeof(unsigned long long), b, G);
    if (b == 0) {
      l2_prefetch_share(R.sxt, (size_t)Z * sizeof(float), 0, 1);
      l2_prefetch_share(R.syt, (size_t)nZ * sizeof(float), 0, 1);
    }
  }
  float2* tws = (float2*)smem;
  float2* work = (float2*)(smem + ONE_TW_BYTES(LZ));
#pragma unroll
  for (int k = 0; k < TWR; k++)
    if (threadIdx.x + 256 * k < Z) tws[threadIdx.x + 256 * k] = twr[k];
  // an equal contiguous share of the particles per CTA (the busiest SM then
  // holds two shares, not two full CTAs of 256 while others hold one)
  const int per = (R.N + G - 1) / G;
  const int g0 = min(R.N, b * per), g1 = min(R.N, g0 + per);
  unsigned ep = 0;
  const bool rec = ts && b == 0 && threadIdx.x == 0;
  int ph = 0;
  if (rec) ts[0] = global_ns();
  // after a barrier that failed in an earlier launch the words still hold its
  // poison: this launch ends at its first barrier, before anything moves
  auto barrier = [&]() -> bool {
    if (P.skip_barrier == (int)ep + 1 && b == P.skip_cta) return false;
    return grid_barrier(bar, ++ep * (unsigned)G, P.max_polls ? P.max_polls : BAR_MAX_POLLS, &D.err, &s_ok);
  };
#define BD_BARRIER()      \
  if (!barrier()) return; \
  if (rec) ts[++ph] = global_ns()
  // A transform item runs at most once per call site and CTA (the host sizes
  // them so): in a loop the compiler keeps the addresses of all its passes.
  if (b < P.nri) fft2_rows_inv_item<LZ, true>(OnceTeam(), R, b << P.lri, P.lri, work, tws);
  BD_BARRIER();
  if (steps_left <= 0) {  // the same for every CTA
    grid_exit(bar, (unsigned)G);
    return;
  }
  const unsigned long long step = D.step;
  for (int i0 = g0 + (threadIdx.x & ~31u); i0 < g1; i0 += 256) {
    const int gi = i0 + (threadIdx.x & 31);
    const unsigned act = __ballot_sync(0xffffffffu, gi < g1);
    if (gi < g1) step_particle<false, true>(R, D, step, gi, act);
    __syncwarp();
  }
  BD_BARRIER();
  // the next step's forward rows from the top CTA down, beside the scan's
  // chunks on the lowest ones; each CTA sums the totals before its chunk (few
  // chunks), else CTA 0 scans them first
  const int ncells = R.C * R.C;
  const bool own = P.nch <= 512;
  if (!own) {
    if (b == 0) {
      int loc = 0;
      const int pc = (P.nch + blockDim.x - 1) / blockDim.x, k0 = threadIdx.x * pc;
      for (int k = 0; k < pc; k++)
        if (k0 + k < P.nch) loc += R.chunk_sum[k0 + k];
      int ex = block_excl_scan(loc, s_tmp);
      for (int k = 0; k < pc; k++)
        if (k0 + k < P.nch) {
          const int v = R.chunk_sum[k0 + k];
          R.chunk_off[k0 + k] = ex;
          ex += v;
        }
    }
    if (!barrier()) return;
  }
  for (int c = b; c < P.nch; c += G) {
    int off;
    if (own) {
      int loc = 0;
      for (int k = threadIdx.x; k < c; k += blockDim.x) loc += R.chunk_sum[k];
      const int ex = block_excl_scan(loc, s_tmp);
      __syncthreads();  // every thread has read s_tmp
      if (threadIdx.x == blockDim.x - 1) s_tmp[0] = ex + loc;
      __syncthreads();
      off = s_tmp[0];
      __syncthreads();
    } else {
      off = ((volatile int*)R.chunk_off)[c];
    }
    constexpr int PER = SCAN_CHUNK / 256;
    const int c0 = c * SCAN_CHUNK + threadIdx.x * PER;
    int v[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) v[k] = c0 + k < ncells ? R.count[c0 + k] : 0;
    scan_chunk_store<PER>(CtaTeam(), R, c, ncells, v, off, s_tmp);
  }
  {
    const int it = G - 1 - b;
    if (it < P.nrf) fft2_rows_fwd_item<LZ, true, true>(OnceTeam(), R, it << P.lrf, P.lrf, work, tws);
  }
  BD_BARRIER();
  for (int gi = g0 + threadIdx.x; gi < g1; gi += blockDim.x) scatter_particle(R, gi);
  {
    const int it = G - 1 - b;
    if (it < P.ncl) fft2_cols_item<LZ, true>(OnceTeam(), R, it << P.lw, P.lw, work, tws);
  }
  if (b == 0) {
    for (int k = threadIdx.x; k < P.nch; k += blockDim.x) R.chunk_sum[k] = 0;
    if (threadIdx.x == 0) end_step(R, D, 0);
  }
  if (ts) {
    // the last phase ends when every CTA has scattered and transformed
    BD_BARRIER();
  }
  grid_exit(bar, (unsigned)G);
#undef BD_BARRIER
}

#define BD_ONE_SIZES(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

// The items are sized so that a CTA handles at most one of each kind; two
// CTAs per SM once the particles fill a CTA per SM, a small run takes fewer
// (at least 32), so that its barriers wait on fewer arrivals.
int one_step_plan(OneStepPlan& P, int Z, int N, int C, int device) {
  P = OneStepPlan{};
  if (Z < 8 || Z > 1024 || (Z & (Z - 1))) return (int)cudaErrorInvalidValue;
  while ((1 << P.lz) < Z) P.lz++;
  int nsm = 0, fit = 0;
  cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return (int)e;
  const int blocks = (N + 255) / 256;
  const int gmin = blocks >= nsm ? 2 * nsm : std::max(32, blocks);
  auto size_items = [&](int count, int tps, int& l, int& n) {
    l = 0;
    while ((count >> l) > gmin && ((2 << l) * tps) <= 256) l++;
    n = count >> l;
  };
  size_items(Z, fft2_tps(P.lz - 1), P.lrf, P.nrf);
  size_items(Z / 2, fft2_tps(P.lz), P.lw, P.ncl);
  size_items(Z, fft2_tps(P.lz), P.lri, P.nri);
  P.nch = (int)(((long long)C * C + SCAN_CHUNK - 1) / SCAN_CHUNK);
  // forward row items run beside the scan chunks, on the other CTAs where the
  // threads allow
  while (P.nrf + P.nch > gmin && P.nrf > 1 && ((2 << P.lrf) * fft2_tps(P.lz - 1)) <= 256) {
    P.lrf++;
    P.nrf >>= 1;
  }
  const size_t rf = (size_t)(1 << P.lrf) * fft2_stride(Z / 2) * 8;
  const size_t cl = (size_t)2 * (1 << P.lw) * fft2_stride(Z) * 8;
  const size_t ri = (size_t)(1 << P.lri) * fft2_stride(Z) * 8;
  P.smem = ONE_TW_BYTES(P.lz) + std::max(rf, std::max(cl, ri));
  switch (P.lz) {
#define BD_CASE(L)                                                                                                \
  case L:                                                                                                         \
    if (P.smem > 48 * 1024)                                                                                       \
      e = cudaFuncSetAttribute(k_one_step<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);            \
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_one_step<L>, 256, P.smem);    \
    break;
    BD_ONE_SIZES(BD_CASE)
#undef BD_CASE
  }
  if (e != cudaSuccess) return (int)e;
  // two CTAs per SM: more make every grid barrier slower than they gain
  P.grid = std::min(std::min(fit, 2) * nsm, std::max(gmin, std::max(P.nrf, std::max(P.ncl, P.nri))));
  if (P.smem > 96 * 1024 || P.grid <= 0 || P.nrf > P.grid || P.ncl > P.grid || P.nri > P.grid)
    return (int)cudaErrorInvalidConfiguration;
  return 0;
}

int launch_one_step(const RunDesc& run, RunDyn* dyn, const OneStepPlan& P, unsigned* bar, cudaStream_t s,
                    unsigned long long* ts) {
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
  switch (P.lz) {
#define BD_CASE(L) \
  case L: return (int)cudaLaunchKernelEx(&cfg, k_one_step<L>, run, dyn, P, bar, ts);
    BD_ONE_SIZES(BD_CASE)
#undef BD_CASE
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace bd
