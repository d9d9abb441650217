// engine_kernels.h -- launchers shared between the engine translation units.
// Templates over the flight precision R are instantiated for double (plain
// FP64 path) and float (FP32 flight) in flight_kernels.cu.
#pragma once

#include <cuda_runtime.h>

#include "device_state.cuh"

namespace mcb200 {

template <typename R>
struct FlightCtxT;
using FlightCtx = FlightCtxT<double>;

// Flight launches: the drift pass over the store's n particles (device
// count; n.max sizes the grids), which flies those without an event and
// lists the others, and the persistent flight of the listed ones; with
// draws_apart (by `expected`, the host's idea of the count: it changes the
// launches, not the result) that one leaves the particles that come to a
// final-state draw, and a third launch flies these.  `lists` has room for
// n.max particles; returns the kernels launched.  tickets: zeroed device counters the
// persistent blocks take indices from, one a launch (kFlightTickets: these
// two, then the child generations); a child generation reads its own count;
// n_hint bounds the copies a generation holds.
constexpr int kFlightTickets = 2 + kChildGenerations;
bool draws_apart(bool fp32, long long particles);
template <typename R>
int launch_flight(const FlightCtxT<R> &F, const DevParticlesT<R> &P, const FlightListsT<R> &lists, DevCount n,
                  long long expected, unsigned int *tickets, int sm_count, cudaStream_t s);
template <typename R>
void launch_child_flight(const FlightCtxT<R> &F, const DevChildrenT<R> &in, int n_hint, unsigned int *ticket,
                         int sm_count, cudaStream_t s);
// The drift pass of the simulations k < ninst with bit k of `members` set, in
// one launch (before their flight).  Returns 0 on success.
template <typename R>
struct BatchInstT;
template <typename R>
int launch_batch_drift(const FlightCtxT<R> &F, const BatchInstT<R> *inst, int ninst, uint64_t members, int sm_count,
                       cudaStream_t s);
// One persistent launch flying the listed particles, those left to the draws,
// or the copies of one generation, of the simulations k < ninst with bit k
// of `members` set (inst: device table of BatchInstT, steps: their step
// numbers); blocks_per_sm <= 0: as many as fit.  Returns 0 on success.
// kFlight: the listed particles, draws included; kFlightFirst and kDraws: the
// same in two launches.
enum class BatchPart : int { kFlight = 0, kFlightFirst = 1, kDraws = 2, kChildren = 3 };
template <typename R>
int launch_batch_flight(const FlightCtxT<R> &F, const BatchInstT<R> *inst, int ninst, uint64_t members,
                        const uint32_t *steps, BatchPart part, unsigned int *ticket, int blocks_per_sm, int sm_count,
                        cudaStream_t s, bool smem_table);
// steps[k] += 1 and the step field of simulation k in `ntab` consecutive
// tables of n simulations (the tables the batched flights read in place).
template <typename R>
void launch_advance_batch_steps(uint32_t *steps, BatchInstT<R> *tab, int n, int ntab, cudaStream_t s);

// The step's surviving copies (all generations) ranked by (parent uid, sub),
// given uids from *next_uid on, and appended to `dst` after its *n
// particles, in one launch; *appended (zeroed by the step reset) counts them,
// *overflow is set if the store is full.
template <typename R>
void launch_append_children(const ChildSetT<R> &set, unsigned int *next_uid, const DevParticlesT<R> &dst,
                            const unsigned int *n, int capacity, unsigned int *appended, unsigned int *overflow,
                            int grid, cudaStream_t s);
// The counters a step starts from, zeroed in one launch: the flight tickets,
// the copy count of every generation and of the sink, and the appended count.
struct StepCounters {
  unsigned int *tickets;  // [kFlightTickets]
  unsigned int *count[kChildGenerations + 1];
  unsigned int *appended;  // copies appended to the store this step
  unsigned int *listed;    // [2] the flight's list counts (FlightListsT::count)
};
// The flight's per-cell records (DevMesh::cell32, [cells][3] float4, or
// cell64, [cells][3] double2) and the step reset of z, in one launch.
void launch_records_and_reset(const DevTables &T, const DevMesh &M, float4 *out, int cells, const StepCounters &z,
                              cudaStream_t s);
void launch_records_and_reset(const DevTables &T, const DevMesh &M, double2 *out, int cells, const StepCounters &z,
                              cudaStream_t s);
// The end of a step, done by the last block of the sort's scatter (n null:
// none): *particle_steps += *n; *n = *sorted_total; *next_uid += *appended.
// blocks, scan_blocks: counters that are zero between launches.  A sort
// with a StepFinish leaves `offsets` as tile-local cell ends (nothing reads
// them after the step's sort) and `hist` zero, and expects it zero (the
// refresh's sort, without one, zeroes it first and the refresh zeroes it
// again when done).
struct StepFinish {
  unsigned int *n = nullptr;
  const unsigned int *sorted_total = nullptr;
  unsigned int *next_uid = nullptr;
  const unsigned int *appended = nullptr;
  unsigned long long *particle_steps = nullptr;
  unsigned int *blocks = nullptr;
  unsigned int *scan_blocks = nullptr;
};
// One member's part of a batch's step kernels (device table): its cell
// records and step counters, and its step's tail (the copies of `set` join
// `src`, which is sorted into `dst`).
template <typename R>
struct BatchTailT {
  DevMesh M;
  void *records;  // float4 or double2 [cells][3]
  StepCounters counters;
  DevParticlesT<R> src, dst;
  ChildSetT<R> set;
  StepFinish finish;
  unsigned int *overflow, *hist, *offsets, *tile_sums, *total;
  unsigned long long *bounds;
  int cells, buckets, capacity, nx, nz, shift;
};
// The records of the members in `members` (tiles: of 256 cells, of all
// members), which also zeroes the batch's `ntickets` work tickets; their tails in four launches (scan_tiles: of 1024 buckets, of
// all members; tile_first: device scratch of n + 1 ints).  Return 0 on
// success.
template <typename R>
int launch_batch_records(const DevTables &T, const BatchTailT<R> *tails, int n, uint64_t members, int tiles,
                         unsigned int *tickets, int ntickets, cudaStream_t s);
template <typename R>
int launch_batch_tails(const BatchTailT<R> *tails, int n, uint64_t members, int scan_tiles, int *tile_first,
                       int sm_count, cudaStream_t s);
// The members' counts (a context's dev_counts[3]) to out, pinned host memory.
template <typename R>
int launch_batch_counts(const BatchTailT<R> *tails, int n, unsigned int *out, cudaStream_t s);
template <typename R>
void launch_seed(const FlightCtx &F, const DevParticlesT<R> &P, int offset, int n, const int *cell_of,
                 const double *charge, int type, uint32_t uid0, int grid, cudaStream_t s);
void launch_exclusive_scan(const unsigned int *in, unsigned int *out, unsigned int *tile_sums, unsigned int *total,
                           int n, cudaStream_t s);
// Counting sort of the live particles among the first n (device count) of
// `src` by cell into `dst`; *total = live particles, offsets = cell starts
// (after the scatter: cell ends).  With shift > 0 the keys are buckets of
// 2^shift consecutive cells (hist and offsets per bucket).  bounds (or
// null): the sorted store's charge bounds, as launch_charge_bounds writes.
template <typename R>
void launch_cell_sort(const DevParticlesT<R> &src, DevCount n, const DevParticlesT<R> &dst, int ncells, int nx,
                      int nz, unsigned int *hist, unsigned int *offsets, unsigned int *tile_sums, unsigned int *total,
                      int shift, unsigned long long *bounds, int grid, cudaStream_t s,
                      const StepFinish &finish = StepFinish{});

}  // namespace mcb200
