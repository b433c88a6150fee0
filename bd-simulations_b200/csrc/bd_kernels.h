// Host-visible declarations of the kernel launchers (bd_kernels.cu).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

#include "bd_common.cuh"

namespace bd {

// Work item of a batched launch: run index plus up to three coordinates
// whose meaning depends on the kernel (tile, row group, block, chunk).
struct Item {
  int run, a, b, c;
};

enum CellblockMode { MODE_SET = 1, MODE_ADD = 2, MODE_FORCES = 3 };

constexpr int SCAN_CHUNK = 2048;
constexpr int FFT_THREADS = 512;
constexpr int FFT2_THREADS = 256;  // power-of-two path (register-radix transform)
constexpr int MAX_FFT_SMEM = 200 * 1024;

// One FFT launch: its items, dynamic shared memory and threads per CTA.
struct FftPass {
  const Item* items;
  int n;
  size_t smem;
  int threads;
};

size_t deposit_smem(int mt_max, int rows_max);

int set_kernel_attributes();
int launch_deposit(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, int mt_max,
                   int rows_max, int scheme_override, int require_active, cudaStream_t s);
// the three power-of-two passes of all runs with mesh 2^lz
struct Fft2Group {
  int lz;
  FftPass pass[3];
};

// rows forward, columns + Green, rows inverse: gen[] the kernels for meshes
// with a factor 3 (radix 4/2/3), g2[] one group per power-of-two mesh size;
// ev[0..2] (optional) recorded after each pass; passes first .. last of 0 .. 2
int launch_fft(const RunDesc* runs, const RunDyn* dyn, const FftPass gen[3], const Fft2Group* g2, int ng2,
               int require_active, cudaStream_t s, cudaEvent_t* ev = nullptr, int first = 0, int last = 2);
// shape: the compiled form of a particle kernel (same arithmetic):
// PART_SHAPE_DEFAULT (registers for four 256-thread CTAs per SM) or
// PART_SHAPE_5CTA (for five)
enum PartShape { PART_SHAPE_DEFAULT = 0, PART_SHAPE_5CTA = 1 };
// forces only: MODE_SET, MODE_ADD (mask: pair types) and MODE_FORCES
int launch_particles(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int mode,
                     int mask, int require_active, cudaStream_t s, int shape = PART_SHAPE_DEFAULT);
// forces and move of the runs whose step budget is not used up; deposit: also
// add the new positions to each run's R.dacc; large: the form for runs whose
// arrays do not stay in L2 (shape is not used)
int launch_step(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int deposit, int large,
                cudaStream_t s, int shape = PART_SHAPE_DEFAULT);
// Pipelined stage step (power-of-two meshes, fixed dt, every run with its
// R.dacc): particles (launch_step with deposit), then the scan and the
// scatter with the step end beside the transform of the new density:
// forward rows (pass 1), columns + Green (pass 2), inverse rows (pass 0).
// Transform items carry log2 Z in Item.b; smem is the largest item's shared
// memory; runs whose `sorting` flag is clear are skipped.
int launch_pipe_fft(int pass, const RunDesc* runs, RunDyn* dyn, const Item* items, int n, size_t smem,
                    cudaStream_t s);
// the six-launch form's scan: one CTA per group of PIPE_SCAN_GROUP chunks of
// one run (Item.a: its first chunk), and its scatter: one CTA per unit of
// PIPE_SCATTER_UNIT particles (Item.a: the unit's index in the run), then
// the chunk totals cleared and the steps ended
// two chunks per CTA: 41 us for the 256-run ensemble's scan, four: 55 us
constexpr int PIPE_SCAN_GROUP = 2;
constexpr int PIPE_SCATTER_UNIT = 1024;
int launch_pipe_scan(const RunDesc* runs, RunDyn* dyn, const Item* groups, int ngroup, cudaStream_t s);
int launch_pipe_scatter(const RunDesc* runs, RunDyn* dyn, const Item* units, int nunit, const Item* chunks,
                        int nchunk, cudaStream_t s);
// Two-launch form of the pipelined step: launch_step (with deposit),
// then one cooperative launch of the sort and the transforms, phases C (scan
// chunks and next forward rows), D (scatter, next columns + Green, step end)
// and A (inverse rows: the next step's force grids). Unit lists:
// Item.b >= 3 a transform item (log2 Z), Item.b < 0 a scan chunk (C, Item.a)
// or a scatter unit of PIPE_SCATTER_UNIT particles (D, Item.a).
struct PipeTail {
  const Item* cunits;
  int ncu;
  const Item* dunits;
  int ndu;
  const Item* chunks;  // every chunk of every run (totals cleared, steps ended)
  int nchunk;
  const Item* inv;     // inverse row items
  int ninv;
  unsigned max_polls;  // grid-barrier poll bound (0: the default, about a second)
  int skip_barrier, skip_cta;  // recovery-path test, as ResArgs
  size_t smem;    // the largest transform item's shared memory
  int minb;       // CTAs per SM the registers are bounded for (2, 3 or 4)
  int grid;       // filled by pipe_tail_configure
};
int pipe_tail_configure(PipeTail& P, int device);
// bar: the two grid-barrier words (zero; each launch leaves them zero); ts
// (optional): 4 device timestamps (ns), start and the ends of C, D and A
int launch_pipe_tail(const RunDesc* runs, RunDyn* dyn, const PipeTail& P, unsigned* bar, cudaStream_t s,
                     unsigned long long* ts = nullptr);
int launch_move(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, int require_active,
                int refresh_only, cudaStream_t s);
int launch_count(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, cudaStream_t s);
// dst[src[i].pid] = src[i] for the n records of one run
int launch_records_by_pid(const Rec* src, Rec* dst, int n, cudaStream_t s);
// scan of the cell counts (chunk offsets of runs run0 .. run0+nruns-1, then
// chunks) and scatter (particles); end_step_flag: also end the step of every
// run (adaptive: take the reduced dt bound)
int launch_sort(const RunDesc* runs, RunDyn* dyn, int run0, int nruns, const Item* chunks, int nchunks,
                const Item* parts, int nparts, int end_step_flag, int adaptive, int require_active, cudaStream_t s,
                cudaEvent_t* ev = nullptr);
// phases of one step whose ends a single run's launch of one step can time:
// [0] inverse row FFT [1] particles (forces, noise, move, next density)
// [2] cell-count scan + next row FFT [3] scatter + next column FFT + Green
constexpr int FUSED_PHASES = 4;
// Resident step (bd_resident.cuh): A.nsteps steps (at most each run's step
// budget) of one run (SINGLE) or of every run of A.items in one launch.
enum ResKind { RES_CLUSTERS = 0, RES_SINGLE = 1, RES_GROUPS = 2 };
__host__ __device__ constexpr int res_threads(int kind) { return kind == RES_CLUSTERS ? 512 : 1024; }
constexpr size_t res_max_smem(int kind) { return (kind == RES_CLUSTERS ? 112 : 200) * 1024; }  // two CTAs per SM, or one
constexpr int res_pcap(int kind) { return kind == RES_CLUSTERS ? 1536 : 2048; }  // particles of a CTA kept in shared memory
__host__ __device__ constexpr int res_side(int lz) { return lz >= 16 ? 3 << (lz - 16) : lz > 0 ? 1 << lz : 0; }
constexpr size_t RES_DESC_BYTES = 1024;   // the run's description
__host__ __device__ constexpr size_t RES_TW_BYTES(int Z) {  // twiddles and sine tables
  return ((size_t)8 * Z + 4 * (Z + Z / 2 + 1) + 255) & ~(size_t)255;
}
// mesh classes with kernels of their own (res_side); 0: the rest, ideal gas
#define BD_RES_SIZES(X) \
  X(0) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(20) X(21) X(22) X(23) X(24)
struct ResArgs {
  RunDesc one;             // the single run (its dacc set)
  Item one_item;           // its item: run 0, a/b/c = log2 rows forward, columns, rows inverse per item
  const RunDesc* runs;     // run table (descriptions with dacc set)
  RunDyn* dyn;
  const Item* items;       // one per cluster: run, item sizes as above; groups: two per CTA (k_resident)
  int nsteps;
  int part_off, pcap;      // the particles' place in shared memory and their number
  int grid_mode;           // single run: the whole cooperative grid instead of one cluster
  unsigned* bar;           // grid mode's two barrier words (zero; each launch leaves them zero)
  // grid-barrier waits give up after this many polls (0: the default bound,
  // about a second); a wait that gives up fails that barrier for every CTA
  unsigned max_polls;
  // recovery-path test: CTA skip_cta (of group skip_group) returns instead of
  // arriving at barrier skip_barrier (1-based; 0: none), so every other CTA's
  // wait gives up; max_polls then bounds that group's waits only
  int skip_barrier, skip_cta, skip_group;
  unsigned long long* ts;  // single run: FUSED_PHASES + 1 timestamps of one step (may be null)
};
// kind: one run, one cluster per run, or groups of CTAs of one cooperative grid.
// lz: the mesh side: 2^lz (3..10), 3 * 2^(lz - 16) (20..24: 48 to 768), 0:
// other meshes with a factor 3 and ideal-gas runs, -1: any (groups). cs: CTAs per cluster, 0: cooperative grid (single run).
// resident_held, once resident_attributes has set the kernel's: *n: resident
// CTAs (cs 0) or clusters the device can hold at once
int resident_attributes(int lz, int kind);
int resident_held(int lz, int kind, size_t smem, int cs, int device, int* n);
int launch_resident(int lz, int kind, const ResArgs& A, int nclusters, int cs, int grid, size_t smem,
                    cudaStream_t s);
// One step of one run on a power-of-two mesh up to 1024^2 with a fixed dt in
// one launch of its own (bd_onestep.cu); run: its description, dacc set. bar:
// two barrier words, zero before and after each launch. Starts and ends with
// the resident step's state.
struct OneStepPlan {
  int lz;
  int lrf, nrf;  // forward row items: 2^lrf rows, nrf items
  int lw, ncl;   // column items
  int lri, nri;  // inverse row items
  int nch;       // scan chunks
  unsigned max_polls;          // as ResArgs
  int skip_barrier, skip_cta;
  size_t smem;   // dynamic shared memory
  int grid;      // CTAs (all resident: cooperative launch); 0: no plan
};
int one_step_plan(OneStepPlan& P, int Z, int N, int C, int device);
int launch_one_step(const RunDesc& run, RunDyn* dyn, const OneStepPlan& P, unsigned* bar, cudaStream_t s,
                    unsigned long long* ts);
// TimestepInfo reductions of run 0 into acc (diag_bytes() of device memory):
// energy, virial (double), largest |F|^2 << 32 | index of WCA, capillary,
// noise forces (uint64 x 3), examined WCA pairs (uint64)
int launch_diag(const RunDesc* runs, int N, void* acc, cudaStream_t s);
size_t diag_bytes();
// observables of run 0: pair-distance counts hist[bins] (which 0: 11,
// 1: 12, 2: 22; cells searched within `range` of each particle's) and the
// density Fourier sums re/im[qbins*qbins] of one species
int launch_korr(const RunDesc* runs, int N, int which, int bins, double dr, int range, unsigned long long* hist,
                cudaStream_t s);
int launch_ftrho(const RunDesc* runs, int N, int species, int qbins, double dq, double* re, double* im,
                 cudaStream_t s);
// local densities of run 0 (main_auswertung.cpp:182-390): the TSC lattice
// grid[2][n*n] (FP64, species 1 then 2), then the histograms hist[4][bins]
// and threshold counts hist[4*bins .. +7]
struct LdSnap {
  int n;
  double w, drho;
};
struct LdHist {
  int n, bins;
  double dbin;
  double rho_thresh[3];
  double drho_thresh[4];
};
int launch_lokdens(const RunDesc* runs, int N, const LdSnap& sp, const LdHist& hp, double* grid, unsigned* hist,
                   cudaStream_t s);
int launch_interp(const RunDesc* runs, const Item* items, int n, int scheme, cudaStream_t s);
int launch_noise(const RunDesc* runs, const RunDyn* dyn, const Item* items, int n, cudaStream_t s);
int launch_dtbound(const RunDesc* runs, RunDyn* dyn, const Item* items, int n, cudaStream_t s);
int launch_green(float* green, float* sxt, float* syt, int Z, double kap, double lambda,
                 double L, cudaStream_t s);

}  // namespace bd
