// flight_kernels.cu -- free-flight kernels and the per-step particle
// bookkeeping (mid-step copies, removal of caught particles, counting sort
// by mesh cell).
//
// Step structure (replaces MeshQuantities::update_particle +
// local_migrate, src/mcmodel.cpp:1460-1505 and :1615-1638):
//   1. drift_kernel: the particles that have no event in the step fly it
//      at once and the others are listed; flight_kernel: the listed ones
//      fly dt on their own random streams; caught particles are marked dead
//      in their meta word.
//   2. child_flight_kernel, repeated: copies made by GENERATE / GENREF fly
//      the rest of the step (they may make copies of their own).
//   3. append_children_kernel: surviving copies join the store with uids
//      next_uid + rank of (parent, sub).
//   4. cell_histogram / scan_tiles / cell_scatter: survivors and copies are
//      counting-sorted by cell into the second particle buffer; the
//      scatter's last block makes the sorted count the particle count.
#include <algorithm>
#include <type_traits>

#include "engine_kernels.h"
#include "flight_physics.cuh"
#include "pdl.cuh"
#include "flight_physics_impl.cuh"

namespace mcb200 {

// Resident blocks of 256 threads per SM the flight kernels are compiled for
// (the register budget per thread follows: 2 -> 128, 3 -> 80).
#ifndef MCB200_FLIGHT_BLOCKS_F32
#define MCB200_FLIGHT_BLOCKS_F32 2
#endif
#ifndef MCB200_FLIGHT_BLOCKS_F64
#define MCB200_FLIGHT_BLOCKS_F64 2
#endif
template <typename R>
constexpr int kFlightBlocks = sizeof(R) == 4 ? MCB200_FLIGHT_BLOCKS_F32 : MCB200_FLIGHT_BLOCKS_F64;
// The flight without draws fits FP32 in 80 registers (2M electrons: 610 us at
// two blocks per SM, 541 at three).
template <typename R>
constexpr int kNoDrawBlocks = sizeof(R) == 4 ? 3 : MCB200_FLIGHT_BLOCKS_F64;
// Resident blocks per SM of the drift pass (measured best: FP32 of 4 to 6, 80 us
// for 2M electrons; FP64 of 2 to 4, 155 us).
#ifndef MCB200_DRIFT_BLOCKS_F32
#define MCB200_DRIFT_BLOCKS_F32 4
#endif
#ifndef MCB200_DRIFT_BLOCKS_F64
#define MCB200_DRIFT_BLOCKS_F64 3
#endif
template <typename R>
constexpr int kDriftBlocks = sizeof(R) == 4 ? MCB200_DRIFT_BLOCKS_F32 : MCB200_DRIFT_BLOCKS_F64;

// The expected particle count from which a step's final-state draws are left
// to a launch of their own (draws_apart; tuning defines).  Without the draws
// the flight's loop has two thirds of the code and no register spills (FP64),
// or fits three blocks per SM (FP32); the second launch costs the latency of
// a draw and the rest of its particles' steps, 30-40 us.  Measured, a whole
// step in us with one launch and with two (bulk boxes at 1 to 100 kV/cm, n-FinFETs;
// per cent by which two are slower):
//   FP64  bulk   5k 92-97 / 118-122 (+23 to +30)   20k 131-140 / 146-155 (+11)
//                40k +4 to 0   65,536 +1 to -6   100k -2 to -11   400k -14 to -16
//                2M 1570-1814 / 1213-1362 (-23 to -25)
//         FinFET 192k -7   487k -14   1.26M -15
//   FP32  bulk   5k 70-73 / 98-101 (+39)   100k +12 to +23   400k +1 to -1
//                700k -3 to -8   1M 492-579 / 455-515 (-8 to -11)
//                2M 907-1070 / 807-923 (-11 to -14)
//         FinFET 192k +7   285k +5   487k -4   1.26M -11
// FP64's line lies where a cold box gains nothing yet; FP32's above the crossing
// (400k-500k), where every ensemble gains: up to it one launch gives away 3-8 %.
#ifndef MCB200_DRAWS_APART_F32
#define MCB200_DRAWS_APART_F32 1000000
#endif
#ifndef MCB200_DRAWS_APART_F64
#define MCB200_DRAWS_APART_F64 65536
#endif

constexpr uint32_t kMetaDead = 1u << 16;
constexpr uint32_t kMetaUnfinished = 1u << 17;

template <typename R>
__device__ void load_sym(SymSmemT<R> &S, const DevTables &T) {
  for (int i = threadIdx.x; i < 48; i += blockDim.x) S.sym[i] = T.sym_packed[i];
  for (int i = threadIdx.x; i < 5 * 48; i += blockDim.x) S.newisym[i] = T.newisym[i];
  for (int i = threadIdx.x; i < 3 * 5 * 48; i += blockDim.x) S.bz[i] = (R)T.bz[i];
  for (int i = threadIdx.x; i < 3 * 48; i += blockDim.x) S.refl[i] = T.reflect_isym[i];
  __syncthreads();
}

// Loading and storing the flown particles of the main store (StoreIO: those
// that drift_kernel listed or, kResume, those a launch without draws left to
// them) and of a child generation (ChildIO).  load takes the q-th particle
// to fly, with the state its flight is in, and returns where store puts it
// (-1: none); defer leaves a particle to the draws.
template <typename R, bool kResume>
struct StoreIO {
  DevParticlesT<R> P;
  FlightListsT<R> lists;
  double dt;
  uint32_t step;  // the particles' step number (their random streams)
  // particle p of the store; false: not to be flown
  __device__ __forceinline__ bool read(int p, FlyerT<R> &f) const {
    const uint32_t meta = P.meta[p];
    if (meta & kMetaDead) return false;
    f.step_ = step;
    f.x = P.x[p]; f.y = P.y[p]; f.z = P.z[p];
    f.kx = P.kx[p]; f.ky = P.ky[p]; f.kz = P.kz[p];
    f.energy = P.energy[p];
    f.charge = P.charge[p];
    const uint32_t c = P.cell[p];
    f.ic = c & 1023; f.jc = (c >> 10) & 1023; f.kc = (c >> 20) & 1023;
    f.itet = P.itet[p];
    f.isym = meta & 255;
    f.type = (meta >> 8) & 255;
    f.start_stream(P.uid[p], 0);
    f.nchild = 0;
    f.left_time = dt;
    return true;
  }
  __device__ int load(int q, FlyerT<R> &f, int &state) const {
    const int p = (int)(kResume ? lists.draws : lists.list)[q];
    if (!read(p, f)) return -1;
    if constexpr (kResume) {
      f.resume(lists, p);
      state = FlyerT<R>::kDraw;
    } else {
      f.begin();
      state = FlyerT<R>::kGoOn;
    }
    return p;
  }
  __device__ void defer(int p, const FlyerT<R> &f) const {
    f.save(lists, p);
    store(p, f, 0);
    lists.draws[atomicAdd(lists.count + 1, 1u)] = (uint32_t)p;
  }
  __device__ void store(int p, const FlyerT<R> &f, int r) const {
    P.x[p] = f.x; P.y[p] = f.y; P.z[p] = f.z;
    P.kx[p] = f.kx; P.ky[p] = f.ky; P.kz[p] = f.kz;
    P.energy[p] = f.energy;
    P.cell[p] = pack_cell(f.ic, f.jc, f.kc);
    P.itet[p] = f.itet;
    uint32_t m = (uint32_t)f.isym | ((uint32_t)f.type << 8);
    if (r == 1) m |= kMetaDead;
    if (r == 2) m |= kMetaUnfinished;
    P.meta[p] = m;
  }
};
template <typename R>
struct ChildIO {
  DevChildrenT<R> C;
  uint32_t step;
  __device__ int load(int p, FlyerT<R> &f, int &state) const {
    f.step_ = step;
    f.x = C.x[p]; f.y = C.y[p]; f.z = C.z[p];
    f.kx = C.kx[p]; f.ky = C.ky[p]; f.kz = C.kz[p];
    f.energy = C.energy[p];
    f.charge = C.charge[p];
    const uint32_t c = C.cell[p];
    f.ic = c & 1023; f.jc = (c >> 10) & 1023; f.kc = (c >> 20) & 1023;
    f.itet = C.itet[p];
    f.isym = C.meta[p] & 255;
    f.type = (C.meta[p] >> 8) & 255;
    f.start_stream(C.parent_uid[p], C.sub[p]);
    f.nchild = 0;
    f.left_time = C.left_time[p];
    f.begin();
    state = FlyerT<R>::kGoOn;
    return p;
  }
  __device__ void store(int p, const FlyerT<R> &f, int r) const {
    C.x[p] = f.x; C.y[p] = f.y; C.z[p] = f.z;
    C.kx[p] = f.kx; C.ky[p] = f.ky; C.kz[p] = f.kz;
    C.energy[p] = f.energy;
    C.cell[p] = pack_cell(f.ic, f.jc, f.kc);
    C.itet[p] = f.itet;
    uint32_t m = (uint32_t)f.isym | ((uint32_t)f.type << 8);
    if (r == 1) m |= kMetaDead;
    if (r == 2) m |= kMetaUnfinished;
    C.meta[p] = m;
  }
};

// Persistent flight: each lane holds one particle at a time; a lane whose
// particle has finished its step stores it and takes the next index of the
// warp's chunk of consecutive particles, and the warp takes its next chunk
// from `ticket` (fetched one chunk ahead, so no lane waits for the atomic).
// Every particle's draws come from its own stream, so the result does not
// depend on which lane flies it or when.
//
// A pass of the loop advances every lane to its next event and then runs the
// work that events left: an impurity event's new k and k-space searches by
// the lanes that have some, final-state draws by the whole warp.  (Keeping
// the lanes' work back until 8, 16 or 24 lanes have some was measured slower
// on bulk boxes and no faster on FinFETs: it takes the lanes out of the next
// advances, and a warp that alternates between two long pieces of code
// misses the instruction cache more.)
//
// With fewer particles than the grid has lanes, a warp uses only as many
// lanes as it takes to give every particle one: a warp's passes are the
// union of its lanes' work, so fewer lanes a warp finish sooner.
//
// kLaneEvents (launches of one simulation): the event count of each finished
// particle is summed in the lane and the warp adds its total to the
// simulation's counter once, at the end, instead of one atomic on that one
// address per particle.  A batched launch counts per particle (its particles
// belong to different simulations).
#ifndef MCB200_FLIGHT_CHUNK
#define MCB200_FLIGHT_CHUNK 64
#endif
template <typename R, bool kLaneEvents, bool kDraws, class IO>
__device__ __forceinline__ void fly_interleaved(const FlightCtxT<R> &F, const SymSmemT<R> &S, const IO &io, int n,
                                                unsigned int *ticket) {
  __shared__ R ring[FlyerT<R>::kRing * FlyerT<R>::kRingStride];
  FlyerT<R> f(F, S, ring + threadIdx.x);
  f.n_ph = f.n_imp = 0;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned warps = gridDim.x * (blockDim.x >> 5), count = (unsigned)n;
  const unsigned lanes = min(32u, (count + warps - 1) / warps);
  // a warp's chunk: what its lanes hold when there are few particles, else a
  // quarter of its share, 8 to MCB200_FLIGHT_CHUNK
  const unsigned chunk = lanes < 32u ? lanes : max(8u, min((unsigned)MCB200_FLIGHT_CHUNK, count / (4u * warps)));
  const bool working = lane < lanes;
  auto take = [&]() {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(ticket, chunk);
    return base;  // lane 0's value counts
  };
  unsigned ahead = take(), next = 0, end = 0;
  int p = -1;
  int state = FlyerT<R>::kGoOn;
  bool exhausted = false;
  uint32_t events = 0;  // < 2^31 + kMaxEvents: flushed whenever it passes 2^31 (it bounds n_ph and n_imp)
  auto flush = [&]() {
    atomicAdd(&F.Y.counters[kCntEvents], (unsigned long long)events);
    atomicAdd(&F.Y.counters[kCntPhonon], (unsigned long long)f.n_ph);
    atomicAdd(&F.Y.counters[kCntImpurity], (unsigned long long)f.n_imp);
    events = f.n_ph = f.n_imp = 0;
  };
  auto count_events = [&]() {
    if constexpr (kLaneEvents) {
      events += (uint32_t)(f.loop - f.counted);
      if (events >= 0x80000000u) flush();
    } else {
      f.count_events();
    }
  };
  auto done = [&]() {
    count_events();
    return f.finish();
  };
  for (;;) {
    if (!exhausted) {
      const bool wants = p < 0 && working;
      unsigned need = __ballot_sync(0xffffffffu, wants);
      if (need) {
        unsigned mine = __popc(need & ((1u << lane) - 1u)), left = __popc(need);  // rank among those that still need one
        int q = -1;
        while (left) {
          if (next >= end) {
            next = __shfl_sync(0xffffffffu, ahead, 0);
            end = min(next + chunk, count);
            if (next >= count) {
              exhausted = true;
              break;
            }
            ahead = take();
          }
          const unsigned give = min(left, end - next);
          if (wants && mine < give) q = (int)(next + mine);
          mine -= give;  // wraps past zero once served: no second turn
          left -= give;
          next += give;
        }
        if (q >= 0) {
          p = io.load(q, f, state);
          // (a resumed particle's draw is due even when its event came at the
          // very end of the step)
          if (p >= 0 && state == FlyerT<R>::kGoOn && !(f.left_time > 0)) {
            io.store(p, f, done());
            p = -1;
          }
        }
      }
    }
    const unsigned held = __ballot_sync(0xffffffffu, p >= 0);
    if (!held) {
      if (exhausted) break;
      continue;
    }
    if (p >= 0 && state == FlyerT<R>::kGoOn) state = f.advance();
    if constexpr (kDraws) {
      const unsigned draws = __ballot_sync(0xffffffffu, p >= 0 && state == FlyerT<R>::kDraw);
      if (draws) f.final_states(draws);
    } else if (p >= 0 && state == FlyerT<R>::kDraw) {
      io.defer(p, f);
      count_events();
      p = -1;
    }
    if (p >= 0 && state >= FlyerT<R>::kPending) {
      if (state == FlyerT<R>::kPending) f.run_pending();
      state = f.settle() ? FlyerT<R>::kStepOver : FlyerT<R>::kGoOn;
    }
    if (p >= 0 && state == FlyerT<R>::kStepOver) {
      io.store(p, f, done());
      p = -1;
    }
  }
  if constexpr (kLaneEvents) {
    const uint32_t mine[3] = {events, f.n_ph, f.n_imp};
    const int to[3] = {kCntEvents, kCntPhonon, kCntImpurity};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      unsigned long long sum = mine[c];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
      if (lane == 0 && sum) atomicAdd(&F.Y.counters[to[c]], sum);
    }
  }
}

// The drift pass: every particle that certainly has no event in the step
// (FlyerT::no_event) flies it here, on the fields of its cell with the
// velocity of its tetrahedron, and the others are listed for the flight.
// About half of the particles of a bulk step and four fifths of a FinFET's
// have no event; in the flight's loop each costs a whole pass of the general
// code, here a fifth of its instructions, in a kernel small enough for the
// instruction cache and without its divergence.  Measured (drift + flight
// against the flight of every particle): FinFET FP32 25 + 110 against 165 us
// per launch of 530k particles, bulk FP32 80 + 707 against 823 us per launch
// of 2M; the drift pass itself is bound by the latency of its loads (its
// 112 bytes a particle would take 35 us from HBM in the bulk case).
//
// n: the store's count; *listed (zeroed by the step reset) counts the list.
// A block takes 256 consecutive particles at a time and places its
// unfinished ones with one atomic.
template <typename R, class IO>
__device__ __forceinline__ int drift_block(const FlightCtxT<R> &F, FlyerT<R> &f, const IO &io, int p, bool in,
                                           bool &unfinished) {
  unfinished = false;
  if (!in || !io.read(p, f)) return 0;
  f.load_cell_fields();
  f.iband = f.tf(f.itet).band;
  f.GetV();
  if (f.left_time > kMyZero && f.no_event() && f.drift()) {
    const DevParticlesT<R> &P = io.P;
    P.x[p] = f.x; P.y[p] = f.y; P.z[p] = f.z;
    P.kx[p] = f.kx; P.ky[p] = f.ky; P.kz[p] = f.kz;
    P.energy[p] = f.energy;
    return 1;
  }
  unfinished = true;
  return 0;
}

// The warp's particles that drifted to the step's end: a pass of the event
// loop each.
__device__ __forceinline__ void count_drifted(const DevTallies &Y, unsigned int done) {
  if ((threadIdx.x & 31u) != 0 || done == 0) return;
  atomicAdd(&Y.counters[kCntEvents], (unsigned long long)done);
  if constexpr (MCB200_FLIGHT_EVENT_STATS != 0) atomicAdd(&Y.counters[kStatStepEnd], (unsigned long long)done);
}

// Places the block's marked threads: each gets a consecutive index from *counter.
__device__ __forceinline__ unsigned place_in_list(bool mine, unsigned int *counter) {
  __shared__ unsigned warp_base[kFlightThreads / 32 + 1];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned votes = __ballot_sync(0xffffffffu, mine);
  if (lane == 0) warp_base[warp] = (unsigned)__popc(votes);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kFlightThreads / 32; ++w) {
      const unsigned c = warp_base[w];
      warp_base[w] = run;
      run += c;
    }
    warp_base[kFlightThreads / 32] = run ? atomicAdd(counter, run) : 0u;
  }
  __syncthreads();
  const unsigned at = warp_base[kFlightThreads / 32] + warp_base[warp] + (unsigned)__popc(votes & ((1u << lane) - 1u));
  __syncthreads();  // the counts are reused by the next call
  return at;
}

template <typename R>
__global__ void __launch_bounds__(kFlightThreads, kDriftBlocks<R>) drift_kernel(const __grid_constant__ FlightCtxT<R> F,
                                                               const __grid_constant__ DevParticlesT<R> P, DevCount n,
                                                               uint32_t *list, unsigned int *listed) {
  __shared__ SymSmemT<R> S;  // its operations only
  for (int i = threadIdx.x; i < 48; i += blockDim.x) S.sym[i] = F.T.sym_packed[i];
  __syncthreads();
  pdl_wait();
  const int count = n.get();
  const uint32_t step = F.step_dev ? *F.step_dev : F.step;
  const StoreIO<R, false> io{P, FlightListsT<R>{}, F.dt, step};
  unsigned int done = 0;
  for (int base = blockIdx.x * kFlightThreads; base < count; base += gridDim.x * kFlightThreads) {
    const int p = base + (int)threadIdx.x;
    FlyerT<R> f(F, S, nullptr);
    bool unfinished;
    done += drift_block(F, f, io, p, p < count, unfinished);
    const unsigned at = place_in_list(unfinished, listed);
    if (unfinished) list[at] = (uint32_t)p;
  }
  done = __reduce_add_sync(0xffffffffu, done);
  count_drifted(F.Y, done);
}

template <typename R, bool kDraws, bool kResume>
__global__ void __launch_bounds__(kFlightThreads, kDraws ? kFlightBlocks<R> : kNoDrawBlocks<R>)
    flight_kernel(FlightCtxT<R> F, DevParticlesT<R> P, FlightListsT<R> lists, unsigned int *ticket) {
  __shared__ SymSmemT<R> S;
  if constexpr (!kResume) load_sym(S, F.T);  // the band tables: nothing the kernel ahead writes
  pdl_wait();
  const int count = (int)lists.count[kResume ? 1 : 0];
  if (count == 0) return;
  if constexpr (kResume) load_sym(S, F.T);
  const uint32_t step = F.step_dev ? *F.step_dev : F.step;
  fly_interleaved<R, true, kDraws>(F, S, StoreIO<R, kResume>{P, lists, F.dt, step}, count, ticket);
}

// Copies made during the previous pass (buffer `in`) fly the rest of their
// step; copies they make go to `F.C`.
template <typename R>
__global__ void __launch_bounds__(kFlightThreads, kFlightBlocks<R>) child_flight_kernel(FlightCtxT<R> F, DevChildrenT<R> in,
                                                              unsigned int *ticket) {
  pdl_wait();
  const int count = min((int)*in.count, in.capacity);
  if (count == 0) return;
  __shared__ SymSmemT<R> S;
  load_sym(S, F.T);
  const uint32_t step = F.step_dev ? *F.step_dev : F.step;
  fly_interleaved<R, true, true>(F, S, ChildIO<R>{in, step}, count, ticket);
}

// ---- batched flight ------------------------------------------------------
// Many simulations in one persistent launch.  Each block copies the batch's
// table of simulations (BatchInstT, one per simulation) into shared memory
// and forms the prefix of their particle counts, read on the device; a lane
// that takes ticket q flies particle q - prefix[k] of simulation k, the
// largest k with prefix[k] <= q, with that simulation's mesh, fields,
// tallies, copy buffer, dt, seed and step (FlyerT::I).  A particle's draws
// still come from its own stream (seed, uid, step), so it flies exactly as
// in a launch of its simulation alone.

// The simulation of a batch's ticket or tile: the prefix of the members'
// counts, in shared memory.  One warp reads the counts, a lane or two per
// member: read one after another by one thread they cost 16 us a launch for
// 32 members (a copy flight without copies took 17.3 us and takes 2.5 this way).
struct MemberPrefix {
  int *first;  // [n + 1]
  int n;
  // count(k) for k < n; by every thread of the block
  template <class Count>
  __device__ __forceinline__ void fill(Count &&count) {
    static_assert(kMaxBatch <= 64, "two members a lane");
    if (threadIdx.x < 32) {
      const int k = (int)threadIdx.x;
      const int a = k < n ? count(k) : 0, b = k + 32 < n ? count(k + 32) : 0;
      int upto_a = a, upto_b = b;
      for (int off = 1; off < 32; off <<= 1) {
        const int ta = __shfl_up_sync(0xffffffffu, upto_a, off), tb = __shfl_up_sync(0xffffffffu, upto_b, off);
        if (k >= off) {
          upto_a += ta;
          upto_b += tb;
        }
      }
      upto_b += __shfl_sync(0xffffffffu, upto_a, 31);
      if (k < n) first[k] = upto_a - a;
      if (k + 32 < n) first[k + 32] = upto_b - b;
      if (k == 31) first[n] = upto_b;
    }
    __syncthreads();
  }
  __device__ __forceinline__ int total() const { return first[n]; }
  // the last k with first[k] <= t (members without a count are passed over)
  __device__ __forceinline__ int find(int t) const {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
};

template <typename R, bool kChild, bool kResume>
struct BatchIO {
  const BatchInstT<R> *I;  // shared memory
  MemberPrefix members;
  __device__ int load(int q, FlyerT<R> &f, int &state) const {
    const int k = members.find(q);
    const BatchInstT<R> &b = I[k];
    f.I = &b;
    const int p = q - members.first[k];
    if constexpr (kChild) return ChildIO<R>{b.in, b.step}.load(p, f, state);
    else return StoreIO<R, kResume>{b.P, b.lists, b.dt, b.step}.load(p, f, state);
  }
  __device__ void defer(int p, const FlyerT<R> &f) const {
    const BatchInstT<R> *b = static_cast<const BatchInstT<R> *>(f.I);
    StoreIO<R, false>{b->P, b->lists, b->dt, b->step}.defer(p, f);
  }
  __device__ void store(int p, const FlyerT<R> &f, int r) const {
    const BatchInstT<R> *b = static_cast<const BatchInstT<R> *>(f.I);
    if constexpr (kChild) ChildIO<R>{b->in, b->step}.store(p, f, r);
    else StoreIO<R, kResume>{b->P, b->lists, b->dt, b->step}.store(p, f, r);
  }
};

// Dynamic shared memory of a batched launch over `ninst` simulations: the
// table of simulations (when it is copied there) and the prefix of their
// particle counts.
template <typename R>
constexpr size_t batch_smem_bytes(int ninst, bool table) {
  return (table ? (size_t)ninst * sizeof(BatchInstT<R>) : 0) + (size_t)(ninst + 1) * sizeof(int);
}

// F holds the band tables (its per-simulation part is unused); steps[k] is
// simulation k's step number (device memory, advanced between steps).
// Simulations whose bit in `members` is clear contribute no particles.
// kSmemTable: every block copies the table into shared memory (about 0.8 KB
// per simulation, taken from the SM's L1 share) and takes the step numbers
// from `steps`; otherwise lanes read the table where it lies (global memory,
// through L1), whose step fields advance_batch_steps keeps current.
template <typename R, bool kChild, bool kDraws, bool kResume, bool kSmemTable>
__global__ void __launch_bounds__(kFlightThreads, kFlightBlocks<R>) batch_flight_kernel(const __grid_constant__ FlightCtxT<R> F,
                                                                             const BatchInstT<R> *inst,
                                                                             int ninst, uint64_t members,
                                                                             const uint32_t *steps,
                                                                             unsigned int *ticket) {
  extern __shared__ __align__(16) unsigned char batch_smem[];
  __shared__ SymSmemT<R> S;
  MemberPrefix prefix{reinterpret_cast<int *>(batch_smem + (kSmemTable ? ninst * sizeof(BatchInstT<R>) : 0)), ninst};
  prefix.fill([&](int k) {
    if (!((members >> k) & 1ull)) return 0;
    return kChild ? min((int)*inst[k].in.count, inst[k].in.capacity) : (int)inst[k].lists.count[kResume ? 1 : 0];
  });
  const int total = prefix.total();
  if (total == 0) return;
  const BatchInstT<R> *I = inst;
  if constexpr (kSmemTable) {
    BatchInstT<R> *T = reinterpret_cast<BatchInstT<R> *>(batch_smem);
    static_assert(sizeof(BatchInstT<R>) % 8 == 0, "the table is copied in 8-byte words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(inst);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(T);
    const int words = ninst * (int)(sizeof(BatchInstT<R>) / 8);
    for (int w = threadIdx.x; w < words; w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    for (int k = threadIdx.x; k < ninst; k += blockDim.x) T[k].step = steps[k];
    I = T;
  }
  load_sym(S, F.T);  // ends with a barrier: the table is visible
  fly_interleaved<R, false, kDraws>(F, S, BatchIO<R, kChild, kResume>{I, prefix}, total, ticket);
}

// The drift pass of many simulations in one launch: the blocks take 256
// particles of one simulation at a time.
template <typename R>
__global__ void __launch_bounds__(kFlightThreads, kDriftBlocks<R>) batch_drift_kernel(const __grid_constant__ FlightCtxT<R> F,
                                                                     const BatchInstT<R> *inst, int ninst,
                                                                     uint64_t members) {
  __shared__ SymSmemT<R> S;
  __shared__ int first[kMaxBatch + 1];  // the tiles before each simulation's
  for (int i = threadIdx.x; i < 48; i += blockDim.x) S.sym[i] = F.T.sym_packed[i];
  MemberPrefix prefix{first, ninst};
  prefix.fill([&](int k) {
    return (members >> k) & 1ull ? (min((int)*inst[k].n, inst[k].capacity) + kFlightThreads - 1) / kFlightThreads : 0;
  });
  const int tiles = prefix.total();
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int k = prefix.find(t);  // uniform over the block
    const BatchInstT<R> &b = inst[k];
    const int count = min((int)*b.n, b.capacity);
    const int p = (t - first[k]) * kFlightThreads + (int)threadIdx.x;
    FlyerT<R> f(F, S, nullptr);
    f.I = &b;
    bool unfinished;
    const StoreIO<R, false> io{b.P, FlightListsT<R>{}, b.dt, b.step};
    const unsigned done = __reduce_add_sync(0xffffffffu, drift_block(F, f, io, p, p < count, unfinished));
    count_drifted(b.Y, done);
    const unsigned at = place_in_list(unfinished, b.lists.count);
    if (unfinished) b.lists.list[at] = (uint32_t)p;
  }
}

// Step numbers of a batch: steps[k] += 1, and the step field of simulation
// k in each of the `ntab` tables of n simulations.
template <typename R>
__global__ void advance_batch_steps(uint32_t *steps, BatchInstT<R> *tab, int n, int ntab) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t v = steps[k] + 1;
  steps[k] = v;
  for (int t = 0; t < ntab; ++t) tab[(size_t)t * n + k].step = v;
}
template <typename R>
void launch_advance_batch_steps(uint32_t *steps, BatchInstT<R> *tab, int n, int ntab, cudaStream_t s) {
  advance_batch_steps<R><<<(n + 63) / 64, 64, 0, s>>>(steps, tab, n, ntab);
}

// FP32 flight's per-cell records (DevMesh::cell32): the fields in float and
// the Brooks-Herring factors of GetImpScRate / GetImpScGamma /
// EleImpScUpdateK (src/ElectronImpurityScatter.cpp:6-306) evaluated once per
// cell in FP64 from the cell's screening density and doping.
//
// The step's counters are reset in the same launch (block 0: zeroed work
// tickets, copy counts and appended count), which the flight then reads.
__device__ __forceinline__ void reset_step_counters(const StepCounters &z, int t) {
  if (t < kFlightTickets) z.tickets[t] = 0u;
  if (t < 1 + kChildGenerations) *z.count[t] = 0u;
  if (t == 0) *z.appended = 0u;
  if (t < 2) z.listed[t] = 0u;
}
// FP64 flight's records (DevMesh::cell64): the factors of the reference's
// expressions that hold no particle value, each rounded as there.
__device__ __forceinline__ void cell_record(const DevTables &T, const DevMesh &M, double2 *out, int c) {
  const double rho = M.rho[c], da = M.da[c];
  // a surface-impurity cell: the reference's formula is commented out there
  // and leaves the rate unset; the engine treats it as zero
  const bool on = (da * T.conc0 >= 1e22) && !(M.surface_scatter && M.surface_impurity && M.in_surf[c]);
  const double eebeta = T.frickel * 4 * kPiD * rho / (2.0 * T.meld * T.eps_si);
  const double fr = T.frickel * rho;
  out[3 * (size_t)c + 0] = make_double2(on ? da * T.meld : 0.0, eebeta * T.meld);
  out[3 * (size_t)c + 1] =
      make_double2(kPiD * (fr * fr), T.frickel * 4 * kPiD * rho / (8.0 * T.melt * T.eps_si));
  out[3 * (size_t)c + 2] = make_double2(T.frickel * 4 * kPiD * rho / T.eps_si, 0.0);
}
__device__ __forceinline__ void cell_record(const DevTables &T, const DevMesh &M, float4 *out, int c) {
  const double rho = M.rho[c], da = M.da[c];
  const bool on = (da * T.conc0 >= 1e22) && !(M.surface_scatter && M.surface_impurity && M.in_surf[c]);
  const double eebeta = T.frickel * 4 * kPiD * rho / (2.0 * T.meld * T.eps_si);
  const double fr = T.frickel * rho;
  const float bh_a = on ? (float)(da * T.meld * sqrt(2.0 * T.meld) / (kPiD * (fr * fr))) : 0.0f;
  const float bh_b = on ? (float)(4.0 * T.melt / (eebeta * T.meld)) : 0.0f;
  const double *e = M.efield + 3 * (size_t)c, *h = M.hfield + 3 * (size_t)c;
  out[3 * (size_t)c + 0] = make_float4((float)e[0], (float)e[1], (float)e[2], bh_a);
  out[3 * (size_t)c + 1] = make_float4((float)h[0], (float)h[1], (float)h[2], bh_b);
  out[3 * (size_t)c + 2] = make_float4((float)(T.frickel * 4 * kPiD * rho / (8.0 * T.melt * T.eps_si)),
                                       (float)(T.frickel * 4 * kPiD * rho / T.eps_si), (float)(0.120 / T.eV0), 0.0f);
}

template <typename Rec>
__global__ void cell_records_kernel(DevTables T, DevMesh M, Rec *out, int cells, StepCounters z) {
  pdl_wait();
  if (blockIdx.x == 0) reset_step_counters(z, threadIdx.x);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < cells) cell_record(T, M, out, c);
}

// ---- counting sort by cell ------------------------------------------------
__device__ __forceinline__ int cell_linear(uint32_t c, int nx, int nz) {
  return (int)((((c >> 10) & 1023) * nx + (c & 1023)) * nz + ((c >> 20) & 1023));
}

// Buckets of 2^shift consecutive cells of the linear order (z fastest):
// shift 0 sorts by cell; wider buckets make the histogram and its scan
// shorter and leave the particles of a bucket in arrival order.  When the
// scatter will compute the sorted store's charge bounds, they start from
// zero here.
__device__ __forceinline__ void histogram_warp(const uint32_t *cell, const uint32_t *meta, int n, int nx, int nz,
                                               unsigned int *hist, int shift, int p) {
  // a warp takes 32 consecutive particles; lanes of the same bucket (a
  // cell-sorted store holds runs of them) add their count with one atomic
  const unsigned lane = threadIdx.x & 31u;
  unsigned int key = 0xffffffffu;
  if (p < n && !(meta[p] & kMetaDead)) key = (unsigned int)(cell_linear(cell[p], nx, nz) >> shift);
  const unsigned int peers = __match_any_sync(0xffffffffu, key);
  if (key != 0xffffffffu && (int)lane == __ffs(peers) - 1) atomicAdd(&hist[key], (unsigned int)__popc(peers));
}
__global__ void cell_histogram(const uint32_t *cell, const uint32_t *meta, DevCount count, int nx, int nz,
                               unsigned int *hist, int shift, unsigned long long *bounds) {
  pdl_wait();
  const int n = count.get();
  if (bounds && blockIdx.x == 0 && threadIdx.x < 4) bounds[threadIdx.x] = 0ull;
  const int lane = (int)(threadIdx.x & 31u);
  for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x)
    histogram_warp(cell, meta, n, nx, nz, hist, shift, base + lane);
}

// Exclusive scan of `count` values, single pass per 1024-wide tile plus a
// tile-sum pass (cells are at most ~10^6, so three small launches suffice).
// Blocks of 256 threads, four consecutive values a thread: shuffles within
// the warps and one exchange of the warps' sums (a block of 1024 threads that
// doubled its reach in shared memory met 20 barriers a tile: 1M buckets 25.5
// us, here 13.1; 16k buckets 5.6, here 3.1).
constexpr int kScanThreads = 256;
constexpr int kScanTile = 4 * kScanThreads;
// The sum of the values of the threads before this one; all: of the block's.
__device__ __forceinline__ unsigned int scan_block(unsigned int mine, unsigned int *all) {
  __shared__ unsigned int sums[kScanThreads / 32];
  const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
  unsigned int upto = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned int t = __shfl_up_sync(0xffffffffu, upto, off);
    if (lane >= off) upto += t;
  }
  if (lane == 31) sums[warp] = upto;
  __syncthreads();
  unsigned int before = 0, run = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w == warp) before = run;
    run += sums[w];
  }
  __syncthreads();  // the sums are reused by the next call
  *all = run;
  return before + upto - mine;
}
// Exclusive scan of the tile sums in place by one block, 1024 tiles per pass
// with the running total carried between passes.
__device__ void scan_tile_sums_block(unsigned int *tile_sums, int ntiles, unsigned int *total) {
  unsigned int carry = 0;
  for (int base = 0; base < ntiles; base += kScanTile) {
    const int t = base + 4 * (int)threadIdx.x;
    unsigned int v[4], all;
#pragma unroll
    for (int e = 0; e < 4; ++e)  // other blocks' writes: read at L2
      v[e] = t + e < ntiles ? __ldcg(tile_sums + t + e) : 0u;
    unsigned int at = carry + scan_block(v[0] + v[1] + v[2] + v[3], &all);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (t + e < ntiles) tile_sums[t + e] = at;
      at += v[e];
    }
    carry += all;
  }
  if (threadIdx.x == 0) *total = carry;
}

// Exclusive scan of each 1024-wide tile, and its sum into tile_sums.  With
// `blocks` (a counter that is zero between launches) the last block to
// finish then scans the tile sums too (scan_tile_sums' work, one launch
// fewer).  clear (or null): the input, zeroed once read (the step's sort
// keeps its histogram zero between sorts, so no memset precedes it).
__device__ void scan_tile(const unsigned int *in, unsigned int *out, unsigned int *tile_sums, int n,
                          unsigned int *blocks, unsigned int *total, unsigned int *clear, int tile, int ntiles) {
  __shared__ bool last;
  const int i = tile * kScanTile + 4 * (int)threadIdx.x;
  // 16-byte accesses where the arrays start on 16 bytes and all four values exist
  const bool whole =
      i + 3 < n && (((uintptr_t)in | (uintptr_t)out | (uintptr_t)clear) & 15) == 0;
  unsigned int v[4] = {0u, 0u, 0u, 0u}, all;
  if (whole) {
    const uint4 q = *reinterpret_cast<const uint4 *>(in + i);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    if (clear) *reinterpret_cast<uint4 *>(clear + i) = make_uint4(0u, 0u, 0u, 0u);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (i + e < n) {
        v[e] = in[i + e];
        if (clear) clear[i + e] = 0u;
      }
  }
  const unsigned int at = scan_block(v[0] + v[1] + v[2] + v[3], &all);
  const uint4 o = make_uint4(at, at + v[0], at + v[0] + v[1], at + v[0] + v[1] + v[2]);
  if (whole) {
    *reinterpret_cast<uint4 *>(out + i) = o;
  } else {
    if (i < n) out[i] = o.x;
    if (i + 1 < n) out[i + 1] = o.y;
    if (i + 2 < n) out[i + 2] = o.z;
    if (i + 3 < n) out[i + 3] = o.w;
  }
  if (threadIdx.x == 0) tile_sums[tile] = all;
  if (blocks == nullptr) return;  // uniform over the grid
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(blocks, 1u) == (unsigned)ntiles - 1u;
  }
  __syncthreads();
  if (!last) return;  // uniform over the block
  __threadfence();
  scan_tile_sums_block(tile_sums, ntiles, total);
  if (threadIdx.x == 0) *blocks = 0u;
}
__global__ void __launch_bounds__(kScanThreads) scan_tiles(const unsigned int *in, unsigned int *out, unsigned int *tile_sums, int n,
                           unsigned int *blocks, unsigned int *total, unsigned int *clear) {
  pdl_wait();
  scan_tile(in, out, tile_sums, n, blocks, total, clear, (int)blockIdx.x, (int)gridDim.x);
}
__global__ void __launch_bounds__(kScanThreads) scan_tile_sums(unsigned int *tile_sums, int ntiles, unsigned int *total) {
  scan_tile_sums_block(tile_sums, ntiles, total);
}
__global__ void scan_add(unsigned int *out, const unsigned int *tile_sums, int n) {
  const int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += tile_sums[blockIdx.x];
}

// bounds (optional, zeroed by the histogram): the sorted store's charge
// bounds in charge_bounds_kernel's layout, {max |q| bits of electrons, of
// holes, electron count, hole count}, from the particles this pass moves.
// finish (optional): the end of the step, by the grid's last block to
// finish (every block has read the count by then).
// tile_base (optional): cursor holds tile-local offsets and the tile's
// exclusive prefix is added (scan_add's work, one launch fewer; the cursor
// then ends as tile-local cell ends).
// One warp's 32 particles, p this lane's; mx and cnt collect the bounds.
template <typename R>
__device__ __forceinline__ void scatter_warp(const DevParticlesT<R> &src, const DevParticlesT<R> &dst, int n,
                                             unsigned int *cursor, int nx, int nz, int shift,
                                             const unsigned int *tile_base, int p, unsigned long long *mx,
                                             unsigned long long *cnt) {
  // lanes of the same bucket take consecutive slots with one atomic
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t m = p < n ? src.meta[p] : kMetaDead;
  const bool live = !(m & kMetaDead);
  // (the particle is on its way while its slot is drawn: loaded after the
  // atomic, 5k electrons took 7.5 us, 2M 76, 32 batched members 37.9; this way
  // 5.9, 72 and 33.7)
  const int from = live ? p : 0;
  const uint32_t cell = src.cell[from];
  const R x = src.x[from], y = src.y[from], z = src.z[from];
  const R kx = src.kx[from], ky = src.ky[from], kz = src.kz[from];
  const double energy = src.energy[from], charge = src.charge[from];
  const int itet = src.itet[from];
  const uint32_t uid = src.uid[from];
  const unsigned int key = live ? (unsigned int)(cell_linear(cell, nx, nz) >> shift) : 0xffffffffu;
  const unsigned int peers = __match_any_sync(0xffffffffu, key);
  const int leader = __ffs(peers) - 1;
  unsigned int first = 0;
  if (live && (int)lane == leader) first = atomicAdd(&cursor[key], (unsigned int)__popc(peers));
  first = __shfl_sync(0xffffffffu, first, leader);
  if (!live) return;
  const unsigned int q = first + (unsigned int)__popc(peers & ((1u << lane) - 1u)) +
                         (tile_base ? tile_base[key >> 10] : 0u);
  dst.x[q] = x; dst.y[q] = y; dst.z[q] = z;
  dst.kx[q] = kx; dst.ky[q] = ky; dst.kz[q] = kz;
  dst.energy[q] = energy; dst.charge[q] = charge;
  dst.cell[q] = cell;
  dst.itet[q] = itet;
  dst.meta[q] = m & 0xffffu;
  dst.uid[q] = uid;
  const int t = ((m >> 8) & 255) == 0 ? 0 : 1;
  const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(charge));
  mx[t] = b > mx[t] ? b : mx[t];
  cnt[t] += 1;
}
// The block's bounds into the store's (every thread of a block of up to 256 calls it).
__device__ __forceinline__ void scatter_bounds(unsigned long long *mx, unsigned long long *cnt,
                                               unsigned long long *bounds) {
  __shared__ unsigned long long red[4][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = 0; t < 2; ++t) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long om = __shfl_down_sync(0xffffffffu, mx[t], o);
      mx[t] = om > mx[t] ? om : mx[t];
      cnt[t] += __shfl_down_sync(0xffffffffu, cnt[t], o);
    }
    if (lane == 0) {
      red[t][warp] = mx[t];
      red[2 + t][warp] = cnt[t];
    }
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const int v = threadIdx.x;
    unsigned long long a = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a = v < 2 ? (red[v][w] > a ? red[v][w] : a) : a + red[v][w];
    if (v < 2) {
      if (a) atomicMax(bounds + v, a);
    } else if (a) {
      atomicAdd(bounds + v, a);
    }
  }
}
// The end of the step, by the last of `parts` (thread 0 of each calls it
// once its block is done with the count).
__device__ __forceinline__ void finish_step(const StepFinish &finish, unsigned int parts) {
  __threadfence();
  const unsigned int done = atomicAdd(finish.blocks, 1u);
  if (done == parts - 1u) {  // every part has read the count
    __threadfence();
    *finish.particle_steps += *finish.n;
    *finish.n = *finish.sorted_total;
    *finish.next_uid += *finish.appended;
    *finish.blocks = 0u;
  }
}
template <typename R>
__global__ void __launch_bounds__(256) cell_scatter(DevParticlesT<R> src, DevCount count, DevParticlesT<R> dst,
                                                    unsigned int *cursor, int nx, int nz, int shift,
                                                    unsigned long long *bounds, StepFinish finish,
                                                    const unsigned int *tile_base) {
  pdl_wait();
  const int n = count.get();
  unsigned long long mx[2] = {0, 0}, cnt[2] = {0, 0};
  const int lane = (int)(threadIdx.x & 31u);
  for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x)
    scatter_warp(src, dst, n, cursor, nx, nz, shift, tile_base, base + lane, mx, cnt);
  if (bounds != nullptr) scatter_bounds(mx, cnt, bounds);  // uniform over the grid
  if (finish.n != nullptr) {                               // uniform over the grid
    __syncthreads();  // every thread of the block has read the count
    if (threadIdx.x == 0) finish_step(finish, gridDim.x);
  }
}

// The surviving copies of every generation (already flown) join the store
// after its *n particles, in one launch.  A copy's uid is *next_uid + the
// number of surviving copies with a smaller (parent uid, sub) key, over all
// generations (the key set is the concatenation of the generations).  A
// block ranks 32 copies at a time, one a lane: the keys of all copies are
// staged through shared memory in chunks, each of the eight warps counts
// the smaller live keys of every eighth one (a broadcast read per compare),
// and the eight counts of a lane are added.  The place in the store is
// taken from `appended` (order does not matter: the cell sort follows); a
// copy that would land beyond the store's capacity is dropped and raises
// *overflow (the host reports it).
template <typename R>
struct CopyRef {
  const ChildSetT<R> &set;
  int cnt[kChildGenerations];
  __device__ explicit CopyRef(const ChildSetT<R> &s) : set(s) {
#pragma unroll
    for (int q = 0; q < kChildGenerations; ++q) cnt[q] = min((int)*set.g[q].count, set.g[q].capacity);
  }
  // generation and index of copy i of the concatenation
  __device__ __forceinline__ void locate(int i, int &gen, int &local) const {
    gen = 0;
    local = i;
#pragma unroll
    for (int q = 0; q + 1 < kChildGenerations; ++q)
      if (gen == q && local >= cnt[q]) {
        local -= cnt[q];
        ++gen;
      }
  }
  __device__ __forceinline__ void key(int i, uint64_t &k, bool &alive) const {
    int gen, local;
    locate(i, gen, local);
    const DevChildrenT<R> &c = set.g[gen];
    k = ((uint64_t)c.parent_uid[local] << 32) | c.sub[local];
    alive = !(c.meta[local] & kMetaDead);
  }
};

template <typename R>
__device__ __forceinline__ int copy_count(const ChildSetT<R> &set) {
  int total = 0;
#pragma unroll
  for (int q = 0; q < kChildGenerations; ++q) total += min((int)*set.g[q].count, set.g[q].capacity);
  return total;
}

// Block `block` of `blocks` (256 threads).
template <typename R>
__device__ __forceinline__ void append_block(const ChildSetT<R> &set, const unsigned int *next_uid,
                                             const DevParticlesT<R> &dst, const unsigned int *n, int capacity,
                                             unsigned int *appended, unsigned int *overflow, int block, int blocks) {
  constexpr int kChunk = 2048;
  __shared__ uint64_t keys[kChunk];
  __shared__ uint32_t part[8][32];
  const CopyRef<R> ref(set);
  int total = 0;
#pragma unroll
  for (int q = 0; q < kChildGenerations; ++q) total += ref.cnt[q];
  if (total == 0) return;
  const uint32_t uid0 = *next_uid;
  const unsigned int n0 = *n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base_i = block * 32; base_i < total; base_i += blocks * 32) {
    const int i = base_i + lane;
    uint64_t my = ~0ull;
    bool my_alive = false;
    if (i < total) ref.key(i, my, my_alive);
    uint32_t rank = 0;
    for (int base = 0; base < total; base += kChunk) {
      const int m = min(kChunk, total - base);
      __syncthreads();  // the previous chunk (and the previous group's counts) are consumed
      for (int j = threadIdx.x; j < m; j += 256) {
        uint64_t kj;
        bool aj;
        ref.key(base + j, kj, aj);
        keys[j] = aj ? kj : ~0ull;  // a dead copy ranks after every live one
      }
      __syncthreads();
      for (int q = warp; q < m; q += 8) rank += keys[q] < my ? 1u : 0u;
    }
    part[warp][lane] = rank;
    __syncthreads();
    if (warp == 0 && i < total && my_alive) {
      uint32_t r = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) r += part[w][lane];
      int gen, local;
      ref.locate(i, gen, local);
      const DevChildrenT<R> &c = set.g[gen];
      const unsigned long long q = (unsigned long long)n0 + atomicAdd(appended, 1u);
      if (q >= (unsigned long long)capacity) {
        *overflow = 1u;
      } else {
        dst.x[q] = c.x[local]; dst.y[q] = c.y[local]; dst.z[q] = c.z[local];
        dst.kx[q] = c.kx[local]; dst.ky[q] = c.ky[local]; dst.kz[q] = c.kz[local];
        dst.energy[q] = c.energy[local]; dst.charge[q] = c.charge[local];
        dst.cell[q] = c.cell[local];
        dst.itet[q] = c.itet[local];
        dst.meta[q] = c.meta[local] & 0xffffu;
        dst.uid[q] = uid0 + r;
      }
    }
  }
}

template <typename R>
__global__ void __launch_bounds__(256) append_children_kernel(ChildSetT<R> set, const unsigned int *next_uid,
                                                              DevParticlesT<R> dst, const unsigned int *n,
                                                              int capacity, unsigned int *appended,
                                                              unsigned int *overflow) {
  pdl_wait();
  append_block(set, next_uid, dst, n, capacity, appended, overflow, (int)blockIdx.x, (int)gridDim.x);
}

// ---- the members' step kernels of a batch ------------------------------------
// The cell records, the copies' append and the sort of every batched member
// in one launch each, in place of five launches per member: 32 members of
// 5k-50k particles took 160 launches a step, most of them shorter than their
// launch.  32 members of FP32 stores of up to 50k particles: 89 us a step
// (records 27, append 2, histogram 10, scan 13, scatter 37) where the 160
// launches took some 220.  `tails` is the
// batch's table (BatchTailT), `members` the members taken (bit k).
template <typename R, typename Rec>
__global__ void __launch_bounds__(256) batch_records_kernel(const __grid_constant__ DevTables T,
                                                            const BatchTailT<R> *tails, int n, uint64_t members,
                                                            unsigned int *tickets, int ntickets) {
  __shared__ int first[kMaxBatch + 1];
  if (blockIdx.x == 0 && (int)threadIdx.x < ntickets) tickets[threadIdx.x] = 0u;
  MemberPrefix tp{first, n};
  tp.fill([&](int k) { return (members >> k) & 1ull ? (tails[k].cells + 255) / 256 : 0; });
  for (int t = blockIdx.x; t < first[n]; t += gridDim.x) {
    const int k = tp.find(t), tile = t - first[k];
    const BatchTailT<R> &b = tails[k];
    if (tile == 0) reset_step_counters(b.counters, threadIdx.x);
    const int c = tile * 256 + (int)threadIdx.x;
    if (c < b.cells) cell_record(T, b.M, static_cast<Rec *>(b.records), c);
  }
}
// The members' copies, 32 a block, whatever their numbers: ranking a member's
// copies is quadratic in them, so those of one with many are spread over the
// grid like those of a step of it alone.  Four members of 500k FP32 carriers
// with 471, 1857 and 6521 copies each: 20, 75 and 532 us with eight blocks a
// member, 10, 16 and 80 this way (one member alone: 8, 13, 55).
template <typename R>
__global__ void __launch_bounds__(256) batch_append_kernel(const BatchTailT<R> *tails, int n, uint64_t members) {
  __shared__ int first[kMaxBatch + 1];
  MemberPrefix tp{first, n};
  tp.fill([&](int k) { return (members >> k) & 1ull ? (copy_count(tails[k].set) + 31) / 32 : 0; });
  for (int t = blockIdx.x; t < first[n]; t += gridDim.x) {
    const int k = tp.find(t);
    const BatchTailT<R> &b = tails[k];
    append_block(b.set, b.finish.next_uid, b.src, b.finish.n, b.capacity, b.counters.appended, b.overflow,
                 t - first[k], first[k + 1] - first[k]);
  }
}
template <typename R>
__device__ __forceinline__ int tail_count(const BatchTailT<R> &b) {
  const unsigned long long v = (unsigned long long)*b.finish.n + *b.counters.appended;
  return (int)(v < (unsigned long long)b.capacity ? v : (unsigned long long)b.capacity);
}
// Also leaves the prefix of the members' tiles for the scatter, which ends
// the members' steps while it runs (their counts change under it).
template <typename R>
__global__ void __launch_bounds__(256) batch_histogram_kernel(const BatchTailT<R> *tails, int n, uint64_t members,
                                                              int *tile_first) {
  __shared__ int first[kMaxBatch + 1];
  MemberPrefix tp{first, n};
  tp.fill([&](int k) { return (members >> k) & 1ull ? max(1, (tail_count(tails[k]) + 255) / 256) : 0; });
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k <= n; k += blockDim.x) tile_first[k] = first[k];
  for (int t = blockIdx.x; t < first[n]; t += gridDim.x) {
    const int k = tp.find(t), tile = t - first[k];
    const BatchTailT<R> &b = tails[k];
    if (tile == 0 && threadIdx.x < 4) b.bounds[threadIdx.x] = 0ull;
    histogram_warp(b.src.cell, b.src.meta, tail_count(b), b.nx, b.nz, b.hist, b.shift, tile * 256 + (int)threadIdx.x);
  }
}
template <typename R>
__global__ void __launch_bounds__(kScanThreads) batch_scan_kernel(const BatchTailT<R> *tails, int n, uint64_t members) {
  __shared__ int first[kMaxBatch + 1];
  MemberPrefix tp{first, n};
  tp.fill([&](int k) { return (members >> k) & 1ull ? (tails[k].buckets + 1023) / 1024 : 0; });
  if ((int)blockIdx.x >= first[n]) return;
  const int k = tp.find((int)blockIdx.x);
  const BatchTailT<R> &b = tails[k];
  scan_tile(b.hist, b.offsets, b.tile_sums, b.buckets, b.finish.scan_blocks, b.total, b.hist,
            (int)blockIdx.x - first[k], first[k + 1] - first[k]);
}
template <typename R>
__global__ void __launch_bounds__(256) batch_scatter_kernel(const BatchTailT<R> *tails, int n, const int *tile_first) {
  __shared__ int first[kMaxBatch + 1];
  for (int k = threadIdx.x; k <= n; k += blockDim.x) first[k] = tile_first[k];
  __syncthreads();
  const MemberPrefix tp{first, n};
  for (int t = blockIdx.x; t < first[n]; t += gridDim.x) {
    const int k = tp.find(t), tile = t - first[k];
    const BatchTailT<R> &b = tails[k];
    const int count = tail_count(b);  // (this tile is not done: the member's count still stands)
    unsigned long long mx[2] = {0, 0}, cnt[2] = {0, 0};
    scatter_warp(b.src, b.dst, count, b.offsets, b.nx, b.nz, b.shift, b.tile_sums, tile * 256 + (int)threadIdx.x, mx,
                 cnt);
    scatter_bounds(mx, cnt, b.bounds);
    __syncthreads();  // every thread has read the count, and the bounds are read from shared memory
    if (threadIdx.x == 0) finish_step(b.finish, (unsigned)(first[k + 1] - first[k]));
  }
}

// Every member's device counts (n, next uid, store-full flag) into pinned host
// memory: one launch in place of a copy and a wait per member (20 steps of 32
// members and their tallies: 12.2 ms with the copies, 11.8 this way).
template <typename R>
__global__ void batch_counts_kernel(const BatchTailT<R> *tails, int n, unsigned int *out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 3 * n) out[t] = tails[t / 3].finish.n[t % 3];
}

// ---- initial ensemble ---------------------------------------------------------
// New particle q (uid = uid0 + q) of carrier `type` in cell cell_of[q]:
// position uniform in the cell (init_particle_data,
// src/particle_init.cpp:185-207) and k-state from select_kstate
// (src/mcmodel.cpp:3006-3057): energy from the Boltzmann distribution,
// accepted against the DOS, band by the DOS share, k uniform on the
// iso-energy surface.  Draws: stream (seed, uid, kSeedStreamStep, 0).
// The sampling runs in FP64 for both stores, so an FP32 store starts from
// the same ensemble as an FP64 one (rounded once, positions made
// cell-relative).

template <typename R>
__global__ void __launch_bounds__(kFlightThreads) seed_kernel(FlightCtx F, DevParticlesT<R> P, int offset, int n,
                                                   const int *cell_of, const double *charge, int type,
                                                   uint32_t uid0) {
  __shared__ SymSmem S;
  __shared__ double ring[Flyer::kRing * Flyer::kRingStride];
  load_sym(S, F.T);
  const DevTables &T = F.T;
  const double tmp_const = 1 - exp(-T.emax);
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    Flyer f(F, S, ring + threadIdx.x);
    const int c = cell_of[q];
    const int kc = c % F.M.nz, ic = (c / F.M.nz) % F.M.nx, jc = c / (F.M.nz * F.M.nx);
    f.ic = ic; f.jc = jc; f.kc = kc;
    f.type = type;
    f.start_stream(uid0 + q, 0);
    f.stock(3);
    double lamda = f.Random();
    f.x = lamda * F.M.lx[ic] + (1 - lamda) * F.M.lx[ic + 1];
    lamda = f.Random();
    f.y = lamda * F.M.ly[jc] + (1 - lamda) * F.M.ly[jc + 1];
    lamda = f.Random();
    f.z = lamda * F.M.lz[kc] + (1 - lamda) * F.M.lz[kc + 1];
    f.itet = 0;
    f.kx = f.ky = f.kz = 0;
    bool ok = false;
    for (int attempt = 0; attempt < 100000 && !ok; ++attempt) {
      f.stock(3);
      f.energy = -log(1 - f.Random() * tmp_const);
      // CALDOSSUM (src/Band.cpp:2267-2295) and CALDOS (:2234-2264)
      const TabPos p = tab_pos(T, f.energy);
      const double ddos = tab_at_strided(T.sumdos + type, 3, p);
      double rdos = f.Random() * T.dosmax[type];
      if (rdos > ddos) continue;
      for (f.iband = T.bandof[type]; f.iband < T.bandof[type] + T.nband[type]; f.iband++) {
        rdos -= tab_at(T.dos + (size_t)f.iband * kNT, p);
        if (rdos < 0) break;
      }
      f.isym = ((int)(f.Random() * 48)) % 48;
      if (f.iband >= T.bandof[type] + T.nband[type]) continue;  // rounding left no band: draw again
      f.get_state();
      if (f.self) continue;
      ok = true;
    }
    if (!ok) count(F.Y, kCntNoTet);
    const int o = offset + q;
    if constexpr (FlightReal<R>::kCellRelative) {
      P.x[o] = (R)(f.x - F.M.lx[ic]); P.y[o] = (R)(f.y - F.M.ly[jc]); P.z[o] = (R)(f.z - F.M.lz[kc]);
    } else {
      P.x[o] = f.x; P.y[o] = f.y; P.z[o] = f.z;
    }
    P.kx[o] = (R)f.kx; P.ky[o] = (R)f.ky; P.kz[o] = (R)f.kz;
    P.energy[o] = f.energy;
    P.charge[o] = charge[q];
    P.cell[o] = pack_cell(ic, jc, kc);
    P.itet[o] = f.itet;
    P.meta[o] = (uint32_t)f.isym | ((uint32_t)type << 8) | (ok ? 0u : kMetaDead);
    P.uid[o] = f.uid;
  }
}

// ---- host-side launchers ----------------------------------------------------
template <typename R>
void launch_seed(const FlightCtx &F, const DevParticlesT<R> &P, int offset, int n, const int *cell_of,
                 const double *charge, int type, uint32_t uid0, int grid, cudaStream_t s) {
  if (n > 0) seed_kernel<R><<<grid, kFlightThreads, 0, s>>>(F, P, offset, n, cell_of, charge, type, uid0);
}
// Blocks of the persistent flight kernels: enough to fill every SM at the
// kernel's occupancy, fewer when there are fewer particles than warps.
// Launch settings are looked up once per device (the current device at the
// launch) and kept: a process may drive several GPUs.
constexpr int kMaxDevices = 64;
inline int current_device() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= kMaxDevices) d = 0;
  return d;
}
template <typename R>
int flight_grid(int n, int block, int sm_count) {
  static int per_sm_of[kMaxDevices] = {};
  int &per_sm = per_sm_of[current_device()];
  if (per_sm == 0) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, flight_kernel<R, true, false>, block, 0) != cudaSuccess || b < 1) b = 1;
    per_sm = b;
  }
  const long long want = ((long long)n + block / 32 - 1) / (block / 32);
  return (int)std::max<long long>(1, std::min<long long>(want, (long long)per_sm * sm_count));
}

template <typename R>
int drift_grid(long long tiles, int sm_count) {
  static int per_sm_of[kMaxDevices] = {};
  int &per_sm = per_sm_of[current_device()];
  if (per_sm == 0) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, drift_kernel<R>, kFlightThreads, 0) != cudaSuccess || b < 1)
      b = 1;
    per_sm = b;
  }
  return (int)std::max<long long>(1, std::min<long long>(tiles, (long long)per_sm * sm_count));
}
bool draws_apart(bool fp32, long long particles) {
  return particles >= (fp32 ? MCB200_DRAWS_APART_F32 : MCB200_DRAWS_APART_F64);
}
template <typename R>
int launch_flight(const FlightCtxT<R> &F, const DevParticlesT<R> &P, const FlightListsT<R> &lists, DevCount n,
                  long long expected, unsigned int *tickets, int sm_count, cudaStream_t s) {
  launch_pdl(drift_kernel<R>, drift_grid<R>(((long long)n.max + kFlightThreads - 1) / kFlightThreads, sm_count),
             kFlightThreads, 0, s, F, P, n, lists.list, lists.count);
  const int grid = flight_grid<R>(n.max, kFlightThreads, sm_count);
  if (!draws_apart(sizeof(R) == 4, expected)) {
    launch_pdl(flight_kernel<R, true, false>, grid, kFlightThreads, 0, s, F, P, lists, tickets);
    return 2;
  }
  const int first = (int)std::min<long long>(((long long)n.max + kFlightThreads / 32 - 1) / (kFlightThreads / 32),
                                             (long long)kNoDrawBlocks<R> * sm_count);
  launch_pdl(flight_kernel<R, false, false>, std::max(first, 1), kFlightThreads, 0, s, F, P, lists, tickets);
  launch_pdl(flight_kernel<R, true, true>, grid, kFlightThreads, 0, s, F, P, lists, tickets + 1);
  return 3;
}
template <typename R>
int launch_batch_drift(const FlightCtxT<R> &F, const BatchInstT<R> *inst, int ninst, uint64_t members, int sm_count,
                       cudaStream_t s) {
  if (ninst < 1 || ninst > kMaxBatch) return 1;
  batch_drift_kernel<R><<<drift_grid<R>(1 << 30, sm_count), kFlightThreads, 0, s>>>(F, inst, ninst, members);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
template <typename R>
void launch_child_flight(const FlightCtxT<R> &F, const DevChildrenT<R> &in, int n_hint, unsigned int *ticket,
                         int sm_count, cudaStream_t s) {
  // One block per SM: a step's copies are few (their lanes refill from the
  // same counter however many there are), and most generations are empty.
  const int n = (int)std::min<long long>(n_hint, (long long)sm_count * (kFlightThreads / 32));
  launch_pdl(child_flight_kernel<R>, flight_grid<R>(n, kFlightThreads, sm_count), kFlightThreads, 0, s, F, in, ticket);
}
template <typename R>
int launch_batch_flight(const FlightCtxT<R> &F, const BatchInstT<R> *inst, int ninst, uint64_t members,
                        const uint32_t *steps, BatchPart part, unsigned int *ticket, int blocks_per_sm, int sm_count,
                        cudaStream_t s, bool smem_table) {
  if (ninst < 1 || ninst > kMaxBatch) return 1;
  const size_t smem = batch_smem_bytes<R>(ninst, smem_table);
  auto pick = [&](auto table) {
    constexpr bool T = decltype(table)::value;
    return part == BatchPart::kFlight        ? batch_flight_kernel<R, false, true, false, T>
           : part == BatchPart::kFlightFirst ? batch_flight_kernel<R, false, false, false, T>
           : part == BatchPart::kDraws       ? batch_flight_kernel<R, false, true, true, T>
                                             : batch_flight_kernel<R, true, true, false, T>;
  };
  auto kernel = smem_table ? pick(std::true_type{}) : pick(std::false_type{});
  if (smem_table) {
    // the opt-in to more than 48 KB of dynamic shared memory holds per device
    static bool opted[kMaxDevices][4] = {};
    bool &done = opted[current_device()][(int)part];
    if (!done) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)batch_smem_bytes<R>(kMaxBatch, true)) != cudaSuccess)
        return 1;
      done = true;
    }
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kFlightThreads, smem) != cudaSuccess ||
      per_sm < 1)
    return 1;
  if (blocks_per_sm > 0) per_sm = std::min(per_sm, blocks_per_sm);
  kernel<<<per_sm * sm_count, kFlightThreads, smem, s>>>(F, inst, ninst, members, steps, ticket);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
void launch_records_and_reset(const DevTables &T, const DevMesh &M, float4 *out, int cells, const StepCounters &z,
                              cudaStream_t s) {
  launch_pdl(cell_records_kernel<float4>, std::max((cells + 255) / 256, 1), 256, 0, s, T, M, out, cells, z);
}
void launch_records_and_reset(const DevTables &T, const DevMesh &M, double2 *out, int cells, const StepCounters &z,
                              cudaStream_t s) {
  launch_pdl(cell_records_kernel<double2>, std::max((cells + 255) / 256, 1), 256, 0, s, T, M, out, cells, z);
}
template <typename R>
int launch_batch_records(const DevTables &T, const BatchTailT<R> *tails, int n, uint64_t members, int tiles,
                         unsigned int *tickets, int ntickets, cudaStream_t s) {
  using Rec = std::conditional_t<sizeof(R) == 4, float4, double2>;
  batch_records_kernel<R, Rec><<<std::max(tiles, 1), 256, 0, s>>>(T, tails, n, members, tickets, ntickets);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
template <typename R>
int launch_batch_tails(const BatchTailT<R> *tails, int n, uint64_t members, int scan_tiles, int *tile_first,
                       int sm_count, cudaStream_t s) {
  batch_append_kernel<R><<<4 * sm_count, 256, 0, s>>>(tails, n, members);
  batch_histogram_kernel<R><<<8 * sm_count, 256, 0, s>>>(tails, n, members, tile_first);
  batch_scan_kernel<R><<<std::max(scan_tiles, 1), kScanThreads, 0, s>>>(tails, n, members);
  batch_scatter_kernel<R><<<8 * sm_count, 256, 0, s>>>(tails, n, tile_first);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
template <typename R>
int launch_batch_counts(const BatchTailT<R> *tails, int n, unsigned int *out, cudaStream_t s) {
  batch_counts_kernel<R><<<(3 * n + 63) / 64, 64, 0, s>>>(tails, n, out);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
template <typename R>
void launch_append_children(const ChildSetT<R> &set, unsigned int *next_uid, const DevParticlesT<R> &dst,
                            const unsigned int *n, int capacity, unsigned int *appended, unsigned int *overflow,
                            int grid, cudaStream_t s) {
  launch_pdl(append_children_kernel<R>, grid, 256, 0, s, set, next_uid, dst, n, capacity, appended, overflow);
}
void launch_exclusive_scan(const unsigned int *in, unsigned int *out, unsigned int *tile_sums, unsigned int *total,
                           int n, cudaStream_t s) {
  const int tiles = (n + 1023) / 1024;
  scan_tiles<<<tiles, kScanThreads, 0, s>>>(in, out, tile_sums, n, nullptr, nullptr, nullptr);
  scan_tile_sums<<<1, kScanThreads, 0, s>>>(tile_sums, tiles, total);
  scan_add<<<tiles, 1024, 0, s>>>(out, tile_sums, n);
}
template <typename R>
void launch_cell_sort(const DevParticlesT<R> &src, DevCount n, const DevParticlesT<R> &dst, int ncells, int nx,
                      int nz, unsigned int *hist, unsigned int *offsets, unsigned int *tile_sums, unsigned int *total,
                      int shift, unsigned long long *bounds, int grid, cudaStream_t s, const StepFinish &finish) {
  const int buckets = (ncells + (1 << shift) - 1) >> shift;
  const int tiles = (buckets + 1023) / 1024;
  if (finish.n != nullptr) {
    // the step's sort: the histogram starts from the zeros the last one
    // left, the tile sums are scanned by scan_tiles' last block (which also
    // clears the histogram), the tile prefixes added by the scatter, the
    // step ended by its last block
    launch_pdl(cell_histogram, grid, 256, 0, s, src.cell, src.meta, n, nx, nz, hist, shift, bounds);
    launch_pdl(scan_tiles, tiles, kScanThreads, 0, s, (const unsigned int *)hist, offsets, tile_sums, buckets,
               finish.scan_blocks, total, hist);
    launch_pdl(cell_scatter<R>, grid, 256, 0, s, src, n, dst, offsets, nx, nz, shift, bounds, finish, tile_sums);
    return;
  }
  cudaMemsetAsync(hist, 0, sizeof(unsigned int) * buckets, s);
  cell_histogram<<<grid, 256, 0, s>>>(src.cell, src.meta, n, nx, nz, hist, shift, bounds);
  scan_tiles<<<tiles, kScanThreads, 0, s>>>(hist, offsets, tile_sums, buckets, nullptr, nullptr, nullptr);
  scan_tile_sums<<<1, kScanThreads, 0, s>>>(tile_sums, tiles, total);
  scan_add<<<tiles, 1024, 0, s>>>(offsets, tile_sums, buckets);
  cell_scatter<R><<<grid, 256, 0, s>>>(src, n, dst, offsets, nx, nz, shift, bounds, finish, nullptr);
}

#define MCB200_INSTANTIATE(R)                                                                                   \
  template void launch_seed<R>(const FlightCtx &, const DevParticlesT<R> &, int, int, const int *,            \
                               const double *, int, uint32_t, int, cudaStream_t);                             \
  template int launch_flight<R>(const FlightCtxT<R> &, const DevParticlesT<R> &, const FlightListsT<R> &,        \
                                DevCount, long long, unsigned int *, int, cudaStream_t);                        \
  template int launch_batch_drift<R>(const FlightCtxT<R> &, const BatchInstT<R> *, int, uint64_t, int,          \
                                     cudaStream_t);                                                             \
  template void launch_child_flight<R>(const FlightCtxT<R> &, const DevChildrenT<R> &, int, unsigned int *, int, \
                                       cudaStream_t);                                                           \
  template void launch_append_children<R>(const ChildSetT<R> &, unsigned int *, const DevParticlesT<R> &,     \
                                          const unsigned int *, int, unsigned int *, unsigned int *, int,       \
                                          cudaStream_t);                                                        \
  template int launch_batch_flight<R>(const FlightCtxT<R> &, const BatchInstT<R> *, int, uint64_t,             \
                                      const uint32_t *, BatchPart, unsigned int *, int, int, cudaStream_t, bool); \
  template int launch_batch_records<R>(const DevTables &, const BatchTailT<R> *, int, uint64_t, int,            \
                                       unsigned int *, int, cudaStream_t);                                      \
  template int launch_batch_tails<R>(const BatchTailT<R> *, int, uint64_t, int, int *, int, cudaStream_t);       \
  template int launch_batch_counts<R>(const BatchTailT<R> *, int, unsigned int *, cudaStream_t);              \
  template void launch_advance_batch_steps<R>(uint32_t *, BatchInstT<R> *, int, int, cudaStream_t);           \
  template void launch_cell_sort<R>(const DevParticlesT<R> &, DevCount, const DevParticlesT<R> &, int, int, int, \
                                    unsigned int *, unsigned int *, unsigned int *, unsigned int *, int,        \
                                    unsigned long long *, int, cudaStream_t, const StepFinish &);
MCB200_INSTANTIATE(double)
MCB200_INSTANTIATE(float)
#undef MCB200_INSTANTIATE

}  // namespace mcb200
