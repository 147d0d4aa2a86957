// particles.cuh -- argument blocks of the particle kernels (particles.cu).
#pragma once

#include "common.cuh"

namespace aprl_gpu {

constexpr int kMaxMagnets = 4;

// ParticleCPMLRegion + ParticleOpenBoundary geometry of the current window
// (src/particle_boundary.cpp:56-85, 251-283), evaluated on the host.
struct DRegion {
  double outer_lower[3], outer_upper[3];
  double physical_lower[3], physical_upper[3], tolerance[3];
  double max_rate[3];     // maximumConductivityRate per axis
  double thickness[3];    // cells*spacing per axis (0 when no CPML)
  int cells[3];
  double global_lower[3], global_upper[3], global_tolerance[3];
  double order;           // polynomial order of the grading
};

// Particle SoA (RelativisticParticleSI without the diagnostics).  Storage
// is sorted by cell (x fastest) for gather/deposit locality; `order` keeps
// each particle's rank in the reference's list order, which the ABI
// restores on read-out.
struct DParticles {
  double *x, *y, *z, *ux, *uy, *uz, *q, *m;
  unsigned long long* id;
  unsigned long long* order;
  unsigned char* frozen;  // held lab-plane injection state
  double* beta;           // frozenBetaZ
};

constexpr int kTileShift = 0;  // sort granularity: single cells (2^0)

// CPML carriers.  `key` = (birth step + 1) << 32 | rank of the parent in
// the particle list, so sorting by key restores the reference's carrier
// order (survivors first, then newborns in particle order); storage order
// is free.
struct DCarriers {
  double *px, *py, *pz, *vx, *vy, *vz, *q, *w;
  unsigned long long* key;
};

// Per-trial counters of the boundary bookkeeping (src/simulation.cpp:
// 4841-4901, 4375-4383); cumulative counters live on the host.
struct TrialCounters {
  unsigned long long exits;
  double exit_charge;
  unsigned long long cpml[6];
  double cpml_charge[6];
  unsigned long long direct[6];
  double direct_charge[6];
  unsigned long long carrier_outer[6];
  double carrier_outer_charge[6];
  unsigned long long cropped;     // carriers beyond the window upper edge
  double cropped_charge;
  unsigned long long activations; // held particles crossing the activation plane
  unsigned long long held;        // held particles retained by the trial
  // Compaction sizes, so the commit needs no further host round trip.
  unsigned long long lost;        // particles with action 1 or 2
  unsigned long long born_kept;   // newborn carriers kept
  unsigned long long carriers_kept;  // existing carriers kept
  unsigned events;                // particles listed for push_events_kernel
};

struct ResidualSums {
  unsigned long long force_bits;  // max over particles (non-negative double bits)
  double defect;
  double scale;
  unsigned long long calls;       // pushed (seen) slots
};

// One trial's results, and a step's block of them: read back in one copy.
struct TrialResult {
  ResidualSums sums;
  TrialCounters counters;
};
constexpr int kTrialSlots = 3;  // trials issued before the host reads any (run.cu)
struct TrialBlock {
  TrialResult trial[kTrialSlots];
  int stop;             // verdict of the trials issued ahead
  DeviceStatus status;
};

// Per-slot record of one trial push (ConservativeSourceCoupling::Impl::Slot,
// src/source_coupling.cpp:19): where and when the push started and its dt
// (a held particle released mid-step is pushed from its activation kink for
// the remaining fraction of the step).
struct DSlots {
  double *x0, *y0, *z0;
  double* dt;
  unsigned char* seen;
};

// What the gathers read.  W is the arithmetic type of the gathers.
struct GatherArrays {
  const void* filtered[3];   // W: the filtered orbit sum (layout of j_index)
  const double* sum[3];      // the unfiltered current-free orbit sum (ring layout of E)
  const void* magnetic[3];   // W: the filtered B (layout of bf_index), when dense
};

// The argument blocks of the particle kernels are templated on the type F
// of J in the grid view (binary64 in both modes of this library).  Particle
// state, the push, the deposit and the boundary logic are binary64.
template <class F>
struct PushArgs {
  GridT<F> g;
  GatherArrays src;
  DFrame frame;
  DRegion region;
  DMagnet magnets[kMaxMagnets];
  int n_magnets;
  int shape;
  int substeps;
  double time;           // box time at the start of the step
  double exit_lab_z;
  double activation_plane_lab_z;
  long long count;
  DParticles p;          // state at the start of the step (read only)
  double *x1, *y1, *z1, *ux1, *uy1, *uz1;  // state after the trial push
  unsigned char* frozen1;                  // held state after the trial
  DSlots slot;
  double* used_e;        // 3*count: the first-trial gather's or the previous
  double* used_b;        // residual's fields (zeroed where there is no push)
  double* abs_grid_work; // sum over substeps of |grid work|
  unsigned char* action; // 0 retain, 1 CPML/exit carrier, 2 outer exit
  DCarriers born;        // carrier created by a CPML entry (when kept)
  unsigned char* plain;  // 1: chord_deposit_kernel deposits the chord start -> end
  unsigned* events;      // the other particles, for push_events_kernel
  double crop_upper;     // as in CarrierArgs, for newborn carriers
  unsigned long long key_base;  // (step + 1) << 32 for newborn carrier keys
  unsigned char* born_keep;
  TrialCounters* counters;
  DeviceStatus* status;
};

template <class F>
struct CarrierArgs {
  GridT<F> g;
  DRegion region;
  int shape;
  long long count;
  double crop_upper;     // carriers at or above it are cropped by this step's shift
  DCarriers in;          // carriers at the start of the step
  DCarriers out;         // after this step's segment
  unsigned char* keep;
  TrialCounters* counters;
  DeviceStatus* status;
};

template <class F>
struct ResidualArgs {
  GridT<F> g;
  GatherArrays src;
  int shape;
  long long count;
  DParticles p;
  DSlots slot;
  const double *x1, *y1, *z1;
  const double* used_e;
  const double* used_b;
  double* next_e;
  double* next_b;
  const double* abs_grid_work;
  ResidualSums* sums;
  // defect and scale per block; the last block to finish sums them in block
  // order (ticket counts the finished blocks and is left at zero) and, for a
  // trial issued ahead, applies the stopping rule.
  double* partial;
  unsigned* ticket;
  unsigned iterations;      // this trial's number, from 1
  double force_tolerance, work_tolerance;
  int* stop;                // null: no verdict
  DeviceStatus* status;
};

// The chords of a trial that chord_deposit_kernel deposits.
struct ChordArgs {
  GridT<double> g;
  long long count;
  const unsigned char* plain;
  DParticles p;                 // chord starts and charges
  const double *x1, *y1, *z1;   // chord ends
  DeviceStatus* status;
};

// Occupancy of the hot particle kernels (blocks of 128 threads that must fit
// one SM), measured on the 128x128x512 dipole grid with 1M particles (FP64),
// on the 128x128x2048 undulator grid with 4M (FP32-mixed) and on smaller runs.
//
// push_kernel (push_deposit in the profile) is bound by FP64 issue (Newton,
// divisions) with long serial chains: 8 blocks (64 registers) 0.074 and 0.295 ms against 0.075 and 0.297
// at 7, 0.078 and 0.323 at 6.  (While the kernel carried the boundary events'
// pieces, 6 were best.)
#ifndef APRL_PUSH_MIN_BLOCKS
#define APRL_PUSH_MIN_BLOCKS 8
#endif
// The gathers are bound by load latency.  The binary32 narrow stencils fit 64
// registers: residual 0.308 ms at 8 blocks against 0.325 at 7 and 0.360 at 6,
// guess gather 0.209, 0.214 and 0.265.  The binary64 ones and the wide stencils
// of sparse runs spill there: residual 0.107 ms (FP64) at 8, 0.101 at 7, 0.104
// at 6, but 0.0212, 0.0198 and 0.0189 with 84k particles; guess gather 0.072,
// 0.069 and 0.068; wide binary32 residual 0.073, 0.070 and 0.064: 6 blocks.
// (With the wide stencils these launches took 0.296 and 0.231 ms.)
#ifndef APRL_RESIDUAL_MIN_BLOCKS
#define APRL_RESIDUAL_MIN_BLOCKS 6
#endif
#ifndef APRL_GATHER_MIN_BLOCKS
#define APRL_GATHER_MIN_BLOCKS 6
#endif
#ifndef APRL_NARROW32_MIN_BLOCKS
#define APRL_NARROW32_MIN_BLOCKS 8
#endif
// The quintic gathers keep 24 spline values: 4 blocks (128 registers).  With
// that, and with the visits' range tests made once a particle (Near), the
// residual of 265k particles takes 0.106 ms (0.269 before; 0.110 at 3 blocks,
// 0.152 at 5, 0.191 at 6), the guess gather 0.091 (0.260).
#ifndef APRL_QUINTIC_MIN_BLOCKS
#define APRL_QUINTIC_MIN_BLOCKS 4
#endif
// chord_deposit is bound by issue and the scan's shuffles (6.5 L2 reductions a
// particle, a quarter of their ceiling rate): 0.101 and 0.375 ms at 8 blocks
// against 0.105 and 0.397 at 7, 0.114 and 0.439 at 6 (the wide stencils' 64
// nodes a piece took 0.307 ms).  The quintic one is left to the compiler (0: 168
// registers, 3 blocks).  Launches with 77k, 247k and 939k particles: 0.060, 0.157
// and 0.539 ms; at 4 blocks (128 registers, 0.2 KB spilled) 0.061, 0.141 and
// 0.475, at 5 0.063, 0.156 and 0.503, at 6 0.070, 0.172 and 0.544.  With the
// fixed-point sum 0.105, 0.262 and 0.876; at 4 blocks 0.110, 0.237 and 0.768.
#ifndef APRL_CHORD_MIN_BLOCKS
#define APRL_CHORD_MIN_BLOCKS 8
#endif
#define APRL_CHORD_BOUNDS(S) __launch_bounds__(128, (S) == 0 ? APRL_CHORD_MIN_BLOCKS : 0)
#define APRL_GATHER_BLOCKS(W, S, D, BLOCKS) \
  ((S) != 0 ? APRL_QUINTIC_MIN_BLOCKS       \
            : sizeof(W) == 4 && !(D) ? APRL_NARROW32_MIN_BLOCKS : BLOCKS)
#define APRL_GATHER_BOUNDS(W, S, D) \
  __launch_bounds__(128, APRL_GATHER_BLOCKS(W, S, D, APRL_GATHER_MIN_BLOCKS))
#define APRL_RESIDUAL_BOUNDS(W, S, D) \
  __launch_bounds__(128, APRL_GATHER_BLOCKS(W, S, D, APRL_RESIDUAL_MIN_BLOCKS))
#define APRL_PUSH_BOUNDS __launch_bounds__(128, APRL_PUSH_MIN_BLOCKS)
// W: arithmetic of the gathers (double, or float in the FP32-mixed mode).
// S: the particle shape, 0 linear-binomial3, 1 quintic-compensated.
// D, DB: read the wide stencils directly (linear-binomial3, sparse runs).
template <class W, class F, int S, bool D> __global__ void guess_gather_kernel(const __grid_constant__ PushArgs<F> a);
template <class F> __global__ void APRL_PUSH_BOUNDS push_kernel(const __grid_constant__ PushArgs<F> a);
// Q: the deterministic mode's fixed-point current sum.
template <class F, int S, bool Q>
__global__ void push_events_kernel(const __grid_constant__ PushArgs<F> a);
template <class F, int S, bool Q> __global__ void carrier_kernel(const __grid_constant__ CarrierArgs<F> a);
template <int S, bool Q>
__global__ void APRL_CHORD_BOUNDS(S) chord_deposit_kernel(const __grid_constant__ ChordArgs a);
template <class W, class F, int S, bool DB>
__global__ void APRL_RESIDUAL_BOUNDS(W, S, DB) residual_kernel(const __grid_constant__ ResidualArgs<F> a);

// RelativisticBorisPusher::push of `count` particles (SoA, in place) with
// per-particle E and B (3 values each).
struct BorisArgs {
  long long count;
  double *x, *y, *z, *ux, *uy, *uz;
  const double *q, *m, *e, *b;
  double dt;
};
__global__ void boris_push_kernel(BorisArgs a);

// Stable compaction helpers (warp ballot + block scan + block-offset scan).
constexpr int kScanBlock = 256;
// Up to three flagged lists compacted together: one count launch, one scan
// launch (a block per list), then a gather per kind.
struct FlagList {
  const unsigned char* flag;
  long long n;
  unsigned blocks;         // of kScanBlock
  unsigned first;          // its first block in block_count and block_offset
  unsigned char want;
};
struct FlagLists {
  FlagList list[3];
  unsigned* block_count;
  unsigned* block_offset;
};
__global__ void flag_count_kernel(FlagLists a);
__global__ void flag_scan_kernel(FlagLists a);
// Exclusive scan of n counts by one block of 1024 threads.
__global__ void block_offset_scan_kernel(const unsigned* block_count, int blocks,
                                         unsigned* block_offset);
__global__ void gather_particles_kernel(DParticles out, DParticles src,
                                        const double* x1, const double* y1,
                                        const double* z1, const double* ux1,
                                        const double* uy1, const double* uz1,
                                        const unsigned char* frozen1,
                                        const unsigned char* flag, unsigned char want,
                                        long long n, const unsigned* block_offset);
__global__ void gather_carriers_kernel(DCarriers out, DCarriers src,
                                       const unsigned char* flag, unsigned char want,
                                       long long n, const unsigned* block_offset,
                                       unsigned long long base);
// Stable radix sort of the particle storage by cell (8-bit digits).
constexpr int kRadixBins = 256;
constexpr int kRadixThreads = 256;  // one thread per digit in the scatter's prefix
constexpr int kRadixItems = 8;
constexpr int kRadixTile = kRadixThreads * kRadixItems;
static_assert(kRadixThreads == kRadixBins, "radix_scatter_kernel: one thread per digit");
__global__ void sort_key_kernel(DParticles p, long long n, DGrid g, int tiles_x, int tiles_y,
                                unsigned* key, unsigned* index);
// Keys of a sort by list order: bits [shift, shift + 32) of order[index[i]]
// (of order[i], with index filled by i, when index_in is null).
__global__ void order_key_kernel(const unsigned long long* order, const unsigned* index_in,
                                 long long n, int shift, unsigned* key, unsigned* index);
__global__ void iota_kernel(unsigned long long* out, long long n);
__global__ void radix_count_kernel(const unsigned* key, long long n, int shift, unsigned* count);
__global__ void radix_scatter_kernel(const unsigned* key_in, const unsigned* index_in,
                                     unsigned* key_out, unsigned* index_out, long long n,
                                     int shift, const unsigned* offset);
__global__ void permute_particles_kernel(DParticles out, DParticles src, long long n,
                                         const unsigned* index);
__global__ void chunk_scan_kernel(const unsigned* in, long long n, unsigned* out,
                                  unsigned* chunk_sum);
__global__ void chunk_add_kernel(unsigned* data, long long n, const unsigned* chunk_offset);
// Pending queue (PendingParticleQueue) on the device: particles sorted by
// their due step, initial state.
struct DPending {
  double *x, *y, *z, *ux, *uy, *uz, *q, *m, *beta;
  unsigned long long* id;
};
__global__ void admit_kernel(DParticles out, long long first_slot, DPending src,
                             long long begin, long long count, unsigned long long steps,
                             double held_distance_per_beta, unsigned long long first_order);
template <class F>
struct SupportArgs {
  GridT<F> g;
  int shape;
  DPending src;
  long long begin, count;
  unsigned long long steps;      // step - initial step
  double held_distance_per_beta; // c*dt
  DeviceStatus* status;
};
template <class F, int S, bool Q> __global__ void frozen_support_kernel(const __grid_constant__ SupportArgs<F> a);
__global__ void crop_flags_kernel(DCarriers c, long long n, double upper,
                                  double lower, unsigned char* keep,
                                  TrialCounters* counters, DeviceStatus* status);
// finishMovingWindowStep's guard (src/simulation_moving_window.cpp:358-359):
// an active particle may not fall behind the inlet; held ones may.
// Carriers may not either; `cz` counts on from n.
__global__ void inlet_check_kernel(const double* z, const unsigned char* frozen, long long n,
                                   const double* cz, long long nc, double origin,
                                   DeviceStatus* status);
// The inlet-layer charge of the charge-matched inlet (ChargeMatchedInlet::particle,
// src/charge_matched_inlet.h:31-53) from the stored particles and the
// pending entries [pbegin, pbegin + pcount) at their held positions of step
// `steps` after the queue's first.
struct InletMatchArgs {
  DParticles p;
  long long np;
  DPending src;
  long long pbegin, pcount;
  unsigned long long steps;
  double held_distance_per_beta;
  double origin[3];
  double dx, dy, dz;
  int nx, ny, shape;
  double* rho;                 // (nx+1) x (ny+1) node plane
  // Deterministic mode: the charge goes into these (lo, hi) word pairs
  // instead (fixed_add with rho_scale), converted by fixed_convert_kernel.
  unsigned long long* rho_pairs;
  double rho_scale;
  DeviceStatus* status;
};
__global__ void inlet_charge_kernel(InletMatchArgs a);

// A trial's start: the raw current's marked columns, the trial counters and
// the residual sums cleared (skipped with the trial).
// clear_current: 1 clears the current; in the deterministic mode 2 clears its
// fixed-point pairs instead (it is then written by current_convert_kernel).
// reset_stop: a step's first trial, clearing the verdict of the step before.
__global__ void trial_clear_kernel(GridT<double> g, TrialResult* result, int clear_current,
                                   int* reset_stop);
// Deterministic mode: the raw current from its fixed-point pairs, in the
// marked columns.
__global__ void current_convert_kernel(GridT<double> g, double unscale);
// out[i] = value of pair i (fixed_value), for i < n.
__global__ void fixed_convert_kernel(const unsigned long long* pairs, double* out, long long n,
                                     double unscale);
// solveConservativeSourceStep's stopping rule (src/simulation_source_coupling.cpp:50)
// applied to trial `iterations`' residual sums: on convergence *stop = iterations.
__global__ void trial_verdict_kernel(const ResidualSums* sums, unsigned iterations,
                                     double force_tolerance, double work_tolerance, int* stop);

}  // namespace aprl_gpu
