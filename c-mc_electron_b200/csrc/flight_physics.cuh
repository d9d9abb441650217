// flight_physics.cuh -- per-particle full-band free flight on the device.
//
// A lane flies one particle at a time through the reference's event loop
// (MeshQuantities::particle_fly, src/mcmodel.cpp:1874-2161), with every
// routine it calls restated as device code below; final states are drawn by
// the whole warp for one lane after another.  Each routine cites
// the reference lines it follows.  Arithmetic is IEEE double in the
// reference's operand order and this code is compiled without FMA
// contraction, so with the same random draws (include/mcb200_rng.h) the
// discrete outcomes (tetrahedron, wedge, cell, event type, final state) are
// the reference's; only libm transcendentals (log, sincos) and the impurity
// event's 1 / (q q), the reference's pow(q, -2.0), may differ from glibc by an
// ulp or so.
//
// Device-side differences from the reference, each deliberate:
//  * no process exit: conditions where the reference calls exit() or loops
//    forever set a counter in the tally block and end the particle's step;
//  * the free-flight loop is capped (kMaxEvents) instead of only printing
//    TOO_MANY_LOOPS (src/mcmodel.cpp:2156);
//  * surface-phonon mechanism choice uses drand = Random() * sum(rates): the
//    reference reads an uninitialised local there (src/ParSurfaceScatter.cpp:94,149);
//  * FP32 flight (R = float) runs the same event loop with float kinematics:
//    positions relative to the cell's low corner, k, velocities, fields,
//    event times and rate lookups in float; energy, charge and the
//    remaining step time stay double.  Its own random stream (four float
//    uniforms per Philox block, mcb200_uniform_f32) and a rounding-tolerant
//    event clock (a zero event time is taken as an event now, not as the
//    reference's "Tf < MY_ZERO" catch) make it statistically, not bitwise,
//    equal to the FP64 path;
//  * the tetrahedron search after an impurity event (Getisym,
//    src/ParticleUtils.cpp:395-625) walks the mesh from the current
//    tetrahedron through face neighbours, falling back to a uniform k-grid
//    lookup, instead of scanning the reference's lists; both return the
//    tetrahedron of the band that contains k (they could differ only for a
//    k within 1e-13 of a face shared by two tetrahedra).
#pragma once

#include "device_state.cuh"
#include "mcb200_rng.h"

namespace mcb200 {

constexpr double kMyZero = 1e-13;          // MY_ZERO, include/defs.h
constexpr double kPiD = 3.141592653589793238462643e0;
constexpr int kMaxEvents = 1000000;  // fits in 20 bits (FlyerT::save)
constexpr int kMaxStateTries = 10000;
// FP32 flight: consecutive zero-length events after which a particle is
// taken as stuck (counted in kCntZeroTime and caught).
constexpr int kMaxZeroTimeEvents = 64;
// Threads per block of the kernels that fly or seed particles (a tuning define
// like those of flight_kernels.cu; whole warps, at most 512: a column of the
// draws' ring each).
#ifndef MCB200_FLIGHT_THREADS
#define MCB200_FLIGHT_THREADS 256
#endif
constexpr int kFlightThreads = MCB200_FLIGHT_THREADS;
static_assert(kFlightThreads % 32 == 0 && kFlightThreads <= 512, "whole warps, the ring in shared memory");
// Opt-in event census (build with -DMCB200_FLIGHT_EVENT_STATS=1): counters
// 10-15 of the tallies count the flight loop's passes by the event that
// ended them and the work of the rare shared tails, for the design record
// (mcb200.flight_events); one atomic per counted event, so never in a
// timed build.
#ifndef MCB200_FLIGHT_EVENT_STATS
#define MCB200_FLIGHT_EVENT_STATS 0
#endif
enum EventStat : int {
  kStatTetFace = 10,    // passes ended at a tetrahedron face
  kStatCellFace = 11,   // at a cell face
  kStatScatter = 12,    // at a phonon, impurity or surface event (real or self-scattering)
  kStatStepEnd = 13,    // at the end of the step
  kStatStateTries = 14, // get_state draws (tetrahedra tried, accepted or not)
  kStatWalkSteps = 15,  // tetrahedra visited by the k-space walks
};

// Arithmetic of the two flight precisions.
template <typename R> struct FlightReal;
template <> struct FlightReal<double> {
  using V4 = double4;
  static constexpr bool kCellRelative = false;  // absolute positions, reference arithmetic
  static constexpr double kContain = kMyZero;   // face test d >= -kContain (unnormalised faces)
  static constexpr double kBig = 1e99;
};
template <> struct FlightReal<float> {
  using V4 = float4;
  static constexpr bool kCellRelative = true;   // positions relative to the cell's low corner
  static constexpr float kContain = 2e-5f;      // unit face normals: a k-space distance, ~10 float ulps at the BZ edge
  static constexpr float kBig = 1e30f;
};

__device__ __forceinline__ double m_abs(double v) { return fabs(v); }
__device__ __forceinline__ float m_abs(float v) { return fabsf(v); }
__device__ __forceinline__ double m_sqrt(double v) { return sqrt(v); }
__device__ __forceinline__ float m_sqrt(float v) { return sqrtf(v); }
__device__ __forceinline__ double m_log(double v) { return log(v); }
__device__ __forceinline__ float m_log(float v) { return logf(v); }
__device__ __forceinline__ double m_floor(double v) { return floor(v); }
__device__ __forceinline__ float m_floor(float v) { return floorf(v); }
__device__ __forceinline__ void m_sincos(double v, double *s, double *c) { sincos(v, s, c); }
__device__ __forceinline__ void m_sincos(float v, float *s, float *c) { sincosf(v, s, c); }

// v times +-1: the sign flipped where the top bit of `neg` is set.
__device__ __forceinline__ float m_flip(float v, uint32_t neg) {
  return __uint_as_float(__float_as_uint(v) ^ (neg & 0x80000000u));
}
__device__ __forceinline__ double m_flip(double v, uint32_t neg) {
  return __hiloint2double(__double2hiint(v) ^ (int)(neg & 0x80000000u), __double2loint(v));
}
template <typename R>
__device__ __forceinline__ R m_pick3(uint32_t which, R a, R b, R c) {
  which &= 3u;
  return which == 0u ? a : (which == 1u ? b : c);
}

// mcb200_philox4x32_10 (include/mcb200_rng.h) unrolled, for the stream's one
// hot place.
__device__ __forceinline__ void philox_rounds(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0,
                                              uint32_t k1, uint32_t *w) {
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint64_t p0 = (uint64_t)MCB200_PHILOX_M0 * c0, p1 = (uint64_t)MCB200_PHILOX_M1 * c2;
    c0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
    c1 = (uint32_t)p1;
    c2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
    c3 = (uint32_t)p0;
    k0 += MCB200_PHILOX_W0;
    k1 += MCB200_PHILOX_W1;
  }
  w[0] = c0; w[1] = c1; w[2] = c2; w[3] = c3;
}

// Table views per precision (the FP64 tables or their FP32 copies).
template <typename R> struct Tab;
template <> struct Tab<double> {
  static __device__ __forceinline__ const TetFlightT<double> *tf(const DevTables &T) { return T.tf; }
  static __device__ __forceinline__ const TetShapeT<double> *ts(const DevTables &T) { return T.ts; }
  static __device__ __forceinline__ const double4 *knode(const DevTables &T) { return T.knode; }
  static __device__ __forceinline__ const FlightConstT<double> &k(const DevTables &T) { return T.k64; }
  static __device__ __forceinline__ const double *energy(const DevTables &T) { return T.energy; }
  static __device__ __forceinline__ const double *sumscatt(const DevTables &T) { return T.sumscatt; }
  static __device__ __forceinline__ const double *scatte(const DevTables &T) { return T.scatte; }
  static __device__ __forceinline__ const double *dose(const DevTables &T) { return T.dose; }
  static __device__ __forceinline__ const double *scattiie(const DevTables &T) { return T.scattiie; }
  static __device__ __forceinline__ const double *scatth(const DevTables &T) { return T.scatth; }
  static __device__ __forceinline__ const double *dosh(const DevTables &T) { return T.dosh; }
  static __device__ __forceinline__ const double *scattiih(const DevTables &T) { return T.scattiih; }
  static __device__ __forceinline__ const double *dostetmax(const DevTables &T) { return T.dostetmax; }
};
template <> struct Tab<float> {
  static __device__ __forceinline__ const TetFlightT<float> *tf(const DevTables &T) { return T.f32.tf; }
  static __device__ __forceinline__ const TetShapeT<float> *ts(const DevTables &T) { return T.f32.ts; }
  static __device__ __forceinline__ const float4 *knode(const DevTables &T) { return T.f32.knode; }
  static __device__ __forceinline__ const FlightConstT<float> &k(const DevTables &T) { return T.k32; }
  static __device__ __forceinline__ const float *energy(const DevTables &T) { return T.f32.energy; }
  static __device__ __forceinline__ const float *sumscatt(const DevTables &T) { return T.f32.sumscatt; }
  static __device__ __forceinline__ const float *scatte(const DevTables &T) { return T.f32.scatte; }
  static __device__ __forceinline__ const float *dose(const DevTables &T) { return T.f32.dose; }
  static __device__ __forceinline__ const float *scattiie(const DevTables &T) { return T.f32.scattiie; }
  static __device__ __forceinline__ const float *scatth(const DevTables &T) { return T.f32.scatth; }
  static __device__ __forceinline__ const float *dosh(const DevTables &T) { return T.f32.dosh; }
  static __device__ __forceinline__ const float *scattiih(const DevTables &T) { return T.f32.scattiih; }
  static __device__ __forceinline__ const float *dostetmax(const DevTables &T) { return T.f32.dostetmax; }
};

// Symmetry tables staged in shared memory (one copy per block).
template <typename R>
struct SymSmemT {
  uint32_t sym[48];   // DevTables::sym_packed
  int newisym[5 * 48];
  R bz[3 * 5 * 48];
  int refl[3 * 48];
};
using SymSmem = SymSmemT<double>;

template <typename R>
struct FlightInstT {  // one simulation: its mesh and fields, tallies, copy buffer and step
  DevMesh M;
  DevTallies Y;
  DevChildrenT<R> C;
  double dt;
  uint64_t seed;
  uint32_t step;
  // when set, the step number is read here on the device instead (launches
  // captured in a CUDA graph and replayed at later steps)
  const uint32_t *step_dev = nullptr;
};
template <typename R>
struct FlightCtxT : FlightInstT<R> {  // plus the band tables, shared by every simulation
  DevTables T;
};

// One simulation of a batched flight launch: its flight context, its
// current particle store and device count (main flight), or the copies it
// flies (child flights).
template <typename R>
struct BatchInstT : FlightInstT<R> {
  DevParticlesT<R> P;
  DevChildrenT<R> in;
  const unsigned int *n;
  FlightListsT<R> lists;
  int capacity;
  int pad_;
};
constexpr int kMaxBatch = 64;  // simulations per batched launch (their table fits in shared memory)
using FlightCtx = FlightCtxT<double>;

__device__ __forceinline__ void tally_add_i64(long long *p, double v, double scale) {
  atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)__double2ll_rn(v * scale));
}
__device__ __forceinline__ void count(const DevTallies &Y, int which) { atomicAdd(&Y.counters[which], 1ull); }

template <typename R>
struct FlyerT {
  using Real = FlightReal<R>;
  using V4 = typename Real::V4;
  using TB = Tab<R>;
  const FlightCtxT<R> &F;      // the tables (F.T)
  const SymSmemT<R> &S;
  const FlightInstT<R> *I;     // the simulation of the current particle (F itself unless batched)
  // random stream (uid, step_, sub; step_ set by the launch's IO from the
  // simulation's step): n draws made, draws [n, stocked) ready in the lane's
  // ring of kRing entries (shared memory, entry d % kRing of thread t at
  // [d % kRing * kRingStride + t])
  uint32_t uid, sub, n, step_, stocked;
  R *ring;
  // particle registers (MeshQuantities members, include/mcmodel.h:215-233)
  R x, y, z, kx, ky, kz;
  double energy, charge, left_time;
  int ic, jc, kc, itet, isym, type, iband;
  R Ex, Ey, Ez, vx, vy, vz;
  // The cell's Brooks-Herring constants (its record): FP32 the rate is
  // imp_a sqrt(e) / (1 + imp_b e) below imp_ecut; FP64 imp_a = doping meld (0:
  // no rate), imp_b = eebeta meld, imp_c = pi (frickel rho)^2
  R imp_a, imp_b, imp_c, imp_ecut, imp_emax, imp_beta;
  int itetdir, idir;
  bool catch_, self;
  R rough_rate, sphon_rate, surf_gamma, imp_gamma;
  int nchild;
  uint32_t n_ph, n_imp;  // real phonon and impurity events since they were last added to the counters
  int ev;                // the event that ended the last advance()
  // Work an event left: an impurity event's new k and / or a k-point search
  // (run_pending, lane by lane), or a final-state draw (final_states, by the
  // whole warp): for a phonon or surface event whose mechanism is to be
  // searched with pick_drand or with a draw of its own, or for Diffuse.
  bool imp_pending;
  int loc_mode;
  int draw_kind;
  R pick_drand;
  enum : int { kLocNone = 0, kLocBZ = 1, kLocImpurity = 2 };
  enum : int { kDrawNone = 0, kDrawPick = 1, kDrawPickSurface = 2, kDrawDiffuse = 3 };

  __device__ FlyerT(const FlightCtxT<R> &f, const SymSmemT<R> &s, R *r) : F(f), S(s), I(&f), step_(f.step), ring(r) {}

  __device__ __forceinline__ void start_stream(uint32_t u, uint32_t sb) {
    uid = u;
    sub = sb;
    n = 0;
    stocked = 0;
  }

  // Draw n of the particle's stream (include/mcb200_rng.h).  FP64: the
  // 52-bit uniforms of mcb200_uniform, two per Philox block; FP32: the
  // 23-bit uniforms of mcb200_uniform_f32, four per block.  stock(k) makes
  // sure of the next k <= kRing / 2 draws, Random takes one of them.  The
  // draws of an event pass come at several places, where other lanes may or
  // may not draw; one stock per pass computes the block once for all lanes
  // that need one, instead of at each place for the lanes that do there.
  static constexpr uint32_t kRing = 8, kRingStride = kFlightThreads;
  static constexpr uint32_t kBlockDraws = sizeof(R) == 4 ? 4 : 2;
  __device__ __forceinline__ void stock(uint32_t k) {
#pragma unroll 1
    while (n + k > stocked) {
      uint32_t w[4];
      philox_rounds(stocked / kBlockDraws, uid, step_, sub, (uint32_t)I->seed, (uint32_t)(I->seed >> 32), w);
      R *e = ring + (stocked & (kRing - 1u)) * kRingStride;
      if constexpr (sizeof(R) == 8) {
        e[0] = mcb200_bits_to_unit(w[1], w[0]);
        e[kRingStride] = mcb200_bits_to_unit(w[3], w[2]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) e[q * kRingStride] = mcb200_bits_to_unit_f32(w[q]);
      }
      stocked += kBlockDraws;
    }
  }
  __device__ __forceinline__ R Random() { return ring[(n++ & (kRing - 1u)) * kRingStride]; }
  // Draws up to n - 1 were made elsewhere (final_states): what the ring
  // holds from n on is still good.
  __device__ __forceinline__ void skip_to(uint32_t at) {
    n = at;
    if (n > stocked) stocked = n & ~(kBlockDraws - 1u);
  }

  __device__ __forceinline__ int cell_index() const { return (jc * I->M.nx + ic) * I->M.nz + kc; }
  __device__ __forceinline__ int cell_index(int i, int j, int k) const { return (j * I->M.nx + i) * I->M.nz + k; }
  __device__ __forceinline__ const TetFlightT<R> &tf(int it) const { return TB::tf(F.T)[it]; }
  __device__ __forceinline__ const TetShapeT<R> &ts(int it) const { return TB::ts(F.T)[it]; }

  // in_wedge, src/ParticleUtils.cpp:295-305: BZ vector -> irreducible wedge of isym.
  __device__ __forceinline__ void in_wedge(R &xo, R &yo, R &zo, R xi, R yi, R zi) const {
    const uint32_t w = S.sym[isym];
    const R a = m_flip(xi, w), b = m_flip(yi, w << 1), c = m_flip(zi, w << 2);
    xo = m_pick3(w >> 6, a, b, c);
    yo = m_pick3(w >> 8, a, b, c);
    zo = m_pick3(w >> 10, a, b, c);
  }
  // Band::OutWedge, src/Band.cpp:555-570: wedge vector -> BZ, with operation `w`.
  static __device__ __forceinline__ void out_wedge(uint32_t w, R &xo, R &yo, R &zo, R xi, R yi, R zi) {
    xo = m_flip(m_pick3(w, xi, yi, zi), w);
    yo = m_flip(m_pick3(w >> 2, xi, yi, zi), w << 1);
    zo = m_flip(m_pick3(w >> 4, xi, yi, zi), w << 2);
  }
  __device__ __forceinline__ void out_wedge(R &xo, R &yo, R &zo, R xi, R yi, R zi) const {
    out_wedge(S.sym[isym], xo, yo, zo, xi, yi, zi);
  }
  // GetV, src/ParticleUtils.cpp:307-313.
  __device__ __forceinline__ void GetV() {
    const V4 v = *reinterpret_cast<const V4 *>(tf(itet).v);
    out_wedge(vx, vy, vz, v.x, v.y, v.z);
  }
  // GetEnergy, src/ParticleUtils.cpp:315-329.
  __device__ void GetEnergy() {
    R dx, dy, dz;
    in_wedge(dx, dy, dz, kx, ky, kz);
    const TetFlightT<R> &t = tf(itet);
    const V4 k0 = TB::knode(F.T)[t.node0];
    dx -= k0.x;
    dy -= k0.y;
    dz -= k0.z;
    const R *v = t.v;
    energy = v[3] + v[0] * dx + v[1] * dy + v[2] * dz;
  }
  __device__ __forceinline__ R face_dist(int it, int f, R a, R b, R c) const {
    const R *nn = tf(it).n[f];
    return nn[0] * a + nn[1] * b + nn[2] * c - nn[3];
  }
  __device__ __forceinline__ bool tet_contains(int it, R a, R b, R c) const {
    const R tol = -Real::kContain;
    return face_dist(it, 0, a, b, c) >= tol && face_dist(it, 1, a, b, c) >= tol &&
           face_dist(it, 2, a, b, c) >= tol && face_dist(it, 3, a, b, c) >= tol;
  }

  // TetTime, src/TetHit.cpp:4-106: time to the tet face the drift reaches first.
  __device__ R TetTime() {
    R xkl, ykl, zkl, xfl, yfl, zfl;
    in_wedge(xkl, ykl, zkl, kx, ky, kz);
    in_wedge(xfl, yfl, zfl, Ex, Ey, Ez);
    const TetFlightT<R> &t = tf(itet);
    R num[4], den[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      den[f] = t.n[f][0] * xfl + t.n[f][1] * yfl + t.n[f][2] * zfl;
      num[f] = t.n[f][3] - (t.n[f][0] * xkl + t.n[f][1] * ykl + t.n[f][2] * zkl);
    }
    const unsigned valid = (den[0] < 0 ? 1u : 0u) | (den[1] < 0 ? 2u : 0u) | (den[2] < 0 ? 4u : 0u) |
                           (den[3] < 0 ? 8u : 0u);
    itetdir = 0;
    return least_quotient<4>(num, den, valid, (R)0, itetdir);
  }

  // The least of the quotients num / den of the `valid` indices, each taken
  // as at least `low`, and its index (the lowest of equal ones); kBig and
  // `which` unchanged when none is valid.  FP64 divides only those that a
  // fast estimate (a few ulp of float) leaves in question, one division's
  // code in place of N: bulk flight 1446 -> 1326 us per launch of 2M
  // electrons (in FP32, whose divisions are short, 707 -> 750 us: all are
  // divided there).
  template <int N>
  static __device__ __forceinline__ R least_quotient(const R *num, const R *den, unsigned valid, R low, int &which) {
    R best = Real::kBig;
    if constexpr (sizeof(R) == 4) {
      bool any = false;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        if (!((valid >> q) & 1u)) continue;
        R v = num[q] / den[q];
        if (v < low) v = low;
        if (!any || v < best) {
          best = v;
          which = q;
        }
        any = true;
      }
      return best;
    } else {
      float est[N], least = 3.0e38f;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        est[q] = fmaxf(__fdividef((float)num[q], (float)den[q]), (float)low);
        if ((valid >> q) & 1u) least = fminf(least, est[q]);
      }
      const float bar = least + fabsf(least) * 1e-4f + 1e-25f;
      unsigned open = 0;
#pragma unroll
      for (int q = 0; q < N; ++q)
        if (((valid >> q) & 1u) && !(est[q] > bar)) open |= 1u << q;
      bool any = false;
#pragma unroll 1
      for (; open; open &= open - 1u) {
        const int q = __ffs(open) - 1;
        R a = num[0], b = den[0];
#pragma unroll
        for (int w = 1; w < N; ++w)
          if (q == w) { a = num[w]; b = den[w]; }
        R v = a / b;
        if (v < low) v = low;
        if (!any || v < best) {
          best = v;
          which = q;
        }
        any = true;
      }
      return best;
    }
  }

  // CellTime, src/CellHit.cpp:4-93: time to the real-space cell face.  FP32
  // positions are offsets from the cell's low corner, so the gaps are
  // (width - x) and x.
  __device__ R CellTime() {
    const DevMesh &M = I->M;
    R gap[3];
    if constexpr (Real::kCellRelative) {
      gap[0] = vx > 0 ? M.dxf[ic] - x : -x;
      gap[1] = vy > 0 ? M.dyf[jc] - y : -y;
      gap[2] = vz > 0 ? M.dzf[kc] - z : -z;
    } else {
      gap[0] = vx > 0 ? M.lx[ic + 1] - x : -(x - M.lx[ic]);
      gap[1] = vy > 0 ? M.ly[jc + 1] - y : -(y - M.ly[jc]);
      gap[2] = vz > 0 ? M.lz[kc + 1] - z : -(z - M.lz[kc]);
    }
    const R v[3] = {vx, vy, vz};
    const unsigned moving = (vx > 0 || vx < 0 ? 1u : 0u) | (vy > 0 || vy < 0 ? 2u : 0u) | (vz > 0 || vz < 0 ? 4u : 0u);
    int axis = 0;
    R t = least_quotient<3>(gap, v, moving, -Real::kBig, axis);
    // faces come in pairs per axis, the odd one towards larger coordinates
    idir = 2 * axis + (m_pick3((uint32_t)axis, vx, vy, vz) > 0 ? 1 : 0);
    if constexpr (Real::kCellRelative) {
      if (t < 0) t = 0;  // a position rounded just past the face
    } else {
      if (t < -kMyZero) t = 0;
    }
    return t;
  }

  // Band::CONFBZ, src/Band.cpp:573-616: fold k back into the first BZ.
  __device__ void CONFBZ(R &a, R &b, R &c) const {
    const R p = TB::k(F.T).a0pi;
#pragma unroll 1
    for (int guard = 0; guard < 64; ++guard) {
      bool out = m_abs(a) > p || m_abs(b) > p || m_abs(c) > p || m_abs(a) + m_abs(b) + m_abs(c) > (R)1.50 * p;
      if (!out) return;
      a = a > (R)0 ? a - p : a + p;
      b = b > (R)0 ? b - p : b + p;
      c = c > (R)0 ? c - p : c + p;
    }
  }

  // Point location by walking the tetrahedral mesh: from `start`, repeatedly
  // step through the face whose plane the point lies furthest outside of,
  // until every face test passes (the reference's containment test,
  // d >= -MY_ZERO).  Returns -1 when the walk reaches a wedge boundary or
  // does not settle within the step cap; the caller then uses the k-grid.
  __device__ int walk_to(int start, R a, R b, R c) const {
    int it = start;
#pragma unroll 1
    for (int s = 0; s < 64; ++s) {
      if constexpr (MCB200_FLIGHT_EVENT_STATS != 0) count(I->Y, kStatWalkSteps);
      int fmin = -1;
      R dmin = -Real::kContain;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const R d = face_dist(it, f, a, b, c);
        if (d < dmin) {
          dmin = d;
          fmin = f;
        }
      }
      if (fmin < 0) return it;
      const int nb = tf(it).neib[fmin];
      if (nb < 0) return -1;
      it = nb;
    }
    return -1;
  }

  // Getisym, src/ParticleUtils.cpp:395-625: wedge from k, then the tet of
  // band iband that contains the wedge vector (k-grid lookup, see file note).
  __device__ void Getisym() {
    int mink, maxk;
    R tmin, tmax;
    if (m_abs(kx) > m_abs(ky)) { tmin = m_abs(ky); tmax = m_abs(kx); mink = 1; maxk = 0; }
    else { tmin = m_abs(kx); tmax = m_abs(ky); mink = 0; maxk = 1; }
    if (m_abs(kz) < tmin) mink = 2;
    else if (m_abs(kz) > tmax) maxk = 2;
    // pos[mink] = 2, pos[maxk] = 0, else 1 (mink != maxk always)
    const int p0 = maxk == 0 ? 0 : (mink == 0 ? 2 : 1);
    const int p1 = maxk == 1 ? 0 : (mink == 1 ? 2 : 1);
    const int p2 = maxk == 2 ? 0 : (mink == 2 ? 2 : 1);
    int sx, sy, sz;
    if constexpr (sizeof(R) == 8) {
      auto sgn = [](double v) { return (int)(fabs(v) / v); };  // utils.cpp sign()
      sx = sgn(kx) + 1; sy = sgn(ky) + 1; sz = sgn(kz) + 1;
    } else {
      // a component rounded to exactly zero lies on a wedge plane: either
      // side's wedge contains it, take the positive one
      sx = kx < 0 ? 0 : 2; sy = ky < 0 ? 0 : 2; sz = kz < 0 ? 0 : 2;
    }
    if (sx < 0 || sx > 2 || sy < 0 || sy > 2 || sz < 0 || sz > 2) {  // a zero component: sign() is NaN in the reference
      count(I->Y, kCntNoTet);
      catch_ = true;
      return;
    }
    isym = F.T.indmat[((((sx * 3 + sy) * 3 + sz) * 3 + p0) * 3 + p1) * 3 + p2];
    R a, b, c;
    in_wedge(a, b, c, kx, ky, kz);
    const bool same_band = iband == tf(itet).band;
    if (same_band && tet_contains(itet, a, b, c)) return;
    int start = same_band ? itet : -1;
    if (iband == F.T.bandof[0]) {  // lowest conduction band: start next to the point
      const int sg = kSeedGridN;
      const int si = min(max((int)m_floor((a - TB::k(F.T).grid_lo[0]) * TB::k(F.T).seed_inv[0]), 0), sg - 1);
      const int sj = min(max((int)m_floor((b - TB::k(F.T).grid_lo[1]) * TB::k(F.T).seed_inv[1]), 0), sg - 1);
      const int sk = min(max((int)m_floor((c - TB::k(F.T).grid_lo[2]) * TB::k(F.T).seed_inv[2]), 0), sg - 1);
      const int s0 = F.T.seed_grid[((size_t)si * sg + sj) * sg + sk];
      if (s0 >= 0) start = s0;
    }
    if (start >= 0) {
      const int w = walk_to(start, a, b, c);
      if (w >= 0) {
        itet = w;
        return;
      }
    }
    const int g = F.T.grid_n;
    int gi = (int)m_floor((a - TB::k(F.T).grid_lo[0]) * TB::k(F.T).grid_inv[0]);
    int gj = (int)m_floor((b - TB::k(F.T).grid_lo[1]) * TB::k(F.T).grid_inv[1]);
    int gk = (int)m_floor((c - TB::k(F.T).grid_lo[2]) * TB::k(F.T).grid_inv[2]);
    gi = min(max(gi, 0), g - 1);
    gj = min(max(gj, 0), g - 1);
    gk = min(max(gk, 0), g - 1);
    const int *st = F.T.grid_start + (size_t)iband * (g * g * g + 1);
    const int cell = (gi * g + gj) * g + gk;
#pragma unroll 1
    for (int q = st[cell]; q < st[cell + 1]; ++q) {
      const int it = F.T.grid_tets[q];
      if (tet_contains(it, a, b, c)) {
        itet = it;
        return;
      }
    }
    count(I->Y, kCntNoTet);
    catch_ = true;
  }

  // GetisymBZ, src/ParticleUtils.cpp:331-392, first part: after a
  // BZ-boundary crossing, the current tet or one of the BZ-surface tets of
  // the particle's energy bin; false leaves the search to Getisym.
  __device__ bool bz_surface_search() {
    R a, b, c;
    in_wedge(a, b, c, kx, ky, kz);
    if (iband == tf(itet).band && tet_contains(itet, a, b, c)) return true;
    int ie = (int)(energy * F.T.dlist);
    if (ie < 0) ie = 0;
    if (ie >= kMWLE) ie = kMWLE - 1;
    const int p = F.T.pslist[ie * kMNB + iband], cnt = F.T.nslist[ie * kMNB + iband];
#pragma unroll 1
    for (int itl = p; itl <= p + cnt - 1; ++itl) {
      const int it = F.T.slist[itl];
      if (iband == tf(it).band && tet_contains(it, a, b, c)) {
        itet = it;
        return true;
      }
    }
    return false;
  }

  // HitTet, src/TetHit.cpp:109-142.  After a BZ-boundary crossing the tet
  // search and GetEnergy run in run_locate.
  __device__ void HitTet() {
    const int nb = tf(itet).neib[itetdir];
    if (nb >= 0) {
      itet = nb;
    } else if (nb == -5 || nb == -6) {
      const int ii = -nb - 2;
      kx = kx + S.bz[(0 * 5 + ii) * 48 + isym];
      ky = ky + S.bz[(1 * 5 + ii) * 48 + isym];
      kz = kz + S.bz[(2 * 5 + ii) * 48 + isym];
      isym = S.newisym[ii * 48 + isym];
      loc_mode = kLocBZ;
    } else {
      isym = S.newisym[(-nb - 2) * 48 + isym];
    }
  }

  // The k-point search after a BZ crossing (GetisymBZ, then GetEnergy unless
  // the particle was caught: src/TetHit.cpp:129-134) or after an accepted
  // impurity event (Getisym, then GetEnergy:
  // src/ElectronImpurityScatter.cpp:291-296).
  __device__ void run_locate() {
    const bool bz = loc_mode == kLocBZ;
    loc_mode = kLocNone;
    if (!(bz && bz_surface_search())) Getisym();
    if (bz && catch_) return;
    GetEnergy();
  }

  // TALIND, src/ParticleUtils.cpp:626-748: the final valley (1..6) of a
  // transition of type ityp (1: the same valley, 2: the opposite one, 3: one
  // of the four others) from k.  The reference's talend[] lookups are
  // written as arithmetic on the drawn index (1..4); an index of 5 (u*4+1
  // rounding up to 5, possible only for u within 2^-51 of 1) reads past the
  // reference's table and is clamped to 4 here.
  template <class Draw>
  static __device__ __forceinline__ int final_valley(int ityp, R qx, R qy, R qz, Draw &&draw) {
    const R ax = m_abs(qx), ay = m_abs(qy), az = m_abs(qz);
    int valley = 1;
#pragma unroll 1
    for (int axis = 0; axis < 3; ++axis) {
      const bool here = axis == 0 ? ax >= ay && ax >= az : (axis == 1 ? ay >= az && ay >= ax : az > ay && az > ax);
      if (!here) continue;
      const R q = axis == 0 ? qx : (axis == 1 ? qy : qz);
      if (ityp == 3) {  // {3,4,5,6}, {1,2,5,6}, {1,2,3,4}
        const int i = min((int)(draw() * (R)4.0 + (R)1.0), 4);
        valley = i > 2 * axis ? i + 2 : i;
      } else {
        valley = 2 * axis + ((q >= (R)0) == (ityp == 1) ? 1 : 2);
      }
    }
    return valley;
  }

  // Band::CALDOSTETMAX, src/Band.cpp:2298-2320.
  __device__ R CALDOSTETMAX(R eed, int ib) const {
    const R *d = TB::dostetmax(F.T) + (size_t)ib * kNT;
    if (eed <= (R)0) return d[0];
    if (eed >= TB::k(F.T).emax) return d[kNT - 1];
    const int itab = min((int)(eed / TB::k(F.T).dtable), kNT - 2);  // eed just below emax may round to the last point
    return d[itab] > d[itab + 1] ? d[itab] : d[itab + 1];
  }

  // Band::SURF, src/Band.cpp:194-332 (only reached by FASTSURF for
  // tetrahedra whose two lowest nodes are degenerate).
  static __device__ R SURF(const DevTables &T, R eps, int it);
  // Band::FASTSURF, src/Band.cpp:665-704.
  __device__ R FASTSURF(R eps, int it) const {
    const TetShapeT<R> &s = ts(it);
    const R e0 = s.e[0], e1 = s.e[1], e2 = s.e[2], e3 = s.e[3];
    if (eps > e0 && eps < e3) {
      if (eps <= e1) return s.fac[0] * (eps - e0) * (eps - e0);
      if (eps < e2) {
        if (e1 - e0 > (R)1e-10) return s.fac[0] * (eps - e0) * (eps - e0) - s.fac[1] * (eps - e1) * (eps - e1);
        return SURF(F.T, eps, it);
      }
      return s.fac[2] * (eps - e3) * (eps - e3);
    }
    return 0;
  }

  // The tetrahedra of band ib whose energy bin holds e: lst[0, count).
  __device__ __forceinline__ const int *energy_list(R e, int ib, int &count) const {
    int itab = (int)(e * TB::k(F.T).dlists);
    const bool fine = itab < kMWLES;
    if (!fine) {
      itab = (int)(e * TB::k(F.T).dlist);
      if (itab >= kMWLE) itab = kMWLE - 1;
    }
    const int at = itab * kMNB + ib;
    count = fine ? F.T.ntlists[at] : F.T.ntlist[at];
    return fine ? F.T.tlists + F.T.ptlists[at] : F.T.tlist + F.T.ptlist[at];
  }
  static __device__ __forceinline__ int list_pick(R u, int count) {
    const int pick = (int)(count * u);
    return sizeof(R) == 4 ? min(pick, count - 1) : pick;
  }

  // get_state, src/ParticleUtils.cpp:48-120: random final state on the
  // iso-energy surface of band iband (rejection on the tet's DOS share),
  // one lane for itself (seeding); the flight draws with the whole warp
  // (final_states).
  __device__ void get_state() {
    self = true;
    if (energy <= 0.0) return;
    const R e = (R)energy;
    const R maxdostet = CALDOSTETMAX(e, iband);
    int nted;
    const int *lst = energy_list(e, iband, nted);
    if (nted == 0) return;
    int count2 = 0;
    for (;;) {
      stock(2);
      itet = lst[list_pick(Random(), nted)];
      count2++;
      const TetShapeT<R> &s = ts(itet);
      if ((count2 < kMaxStateTries) && !((s.e[0] < e) && (s.e[3] > e))) continue;
      const R dostet = FASTSURF(e, itet) / s.vgt;
      if (((Random() * maxdostet) > dostet) && (count2 < kMaxStateTries)) continue;
      break;
    }
    if (count2 >= kMaxStateTries) return;
    self = false;
    R a, b, c;
    stock(4);
    point_on_surface(itet, energy, [this]() { return Random(); }, a, b, c);
    out_wedge(kx, ky, kz, a, b, c);
  }

  // getK, src/ParticleUtils.cpp:122-284: uniform point (in the wedge) on the
  // iso-energy triangle / quadrangle of tet it.
  template <class Draw>
  __device__ void point_on_surface(int it, double &en, Draw &&draw, R &xo, R &yo, R &zo) const;

  // Band::CALSCATTSUM, src/Band.cpp:1999-2033.
  __device__ R CALSCATTSUM(R eed, int ib) const {
    const R *s = TB::sumscatt(F.T);
    const R *E = TB::energy(F.T);
    if (eed <= (R)0) return s[ib];
    if (eed >= TB::k(F.T).emax) return s[(size_t)(kNT - 1) * kMNB + ib];
    const int itab = min((int)(eed / TB::k(F.T).dtable), kNT - 2);
    const R intp = (eed - E[itab]) / (E[itab + 1] - E[itab]);
    return s[(size_t)itab * kMNB + ib] + intp * (s[(size_t)(itab + 1) * kMNB + ib] - s[(size_t)itab * kMNB + ib]);
  }

  // heat_to_point, src/heat.cpp:169-196 (CIC onto the cell's 8 nodes).
  __device__ void heat_to_point(double e, long long *heat) const {
    const DevMesh &M = I->M;
    R rx, ry, rz;
    if constexpr (Real::kCellRelative) {
      rx = x / M.dxf[ic];
      ry = y / M.dyf[jc];
      rz = z / M.dzf[kc];
    } else {
      rx = (x - M.lx[ic]) / M.dx[ic];
      ry = (y - M.ly[jc]) / M.dy[jc];
      rz = (z - M.lz[kc]) / M.dz[kc];
    }
    const int px = M.nx + 1, pz = M.nz + 1;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      const int dx = c & 1, dz = (c >> 1) & 1, dy = c >> 2;
      const R wx = dx ? rx : 1 - rx, wy = dy ? ry : 1 - ry, wz = dz ? rz : 1 - rz;
      tally_add_i64(heat + ((size_t)(jc + dy) * px + ic + dx) * pz + kc + dz, e * wy * wx * wz, kEnergyScale);
    }
  }

  // ---- final states ----------------------------------------------------
  // The reference draws a final state inside EPSCAT / ESCATII (electrons),
  // HPSCAT / HSCATII (holes) and Diffuse.  Here the event handlers only say
  // which draw is due (draw_kind), and final_states makes it with the whole
  // warp, in the reference's order: the mechanism, the wedge (TALIND or a
  // random isym), get_state, and the routine's epilogue.

  // FEKLOEM / FEKLOAB / FEKTOEM / FEKTOAB / FEKLAEM / FEKLAAB
  // (src/ElectronPhononScatter.cpp:633-1022), table-driven: the final energy
  // of an LO / TO / LA phonon event under quantum correction.  The energy in
  // phonon quanta selects a column of the dispersion table (per-range
  // offset, scale and spacing edeta); one draw walks the column's
  // cumulative sum to a row i, and the final energy is the phonon energy
  // shifted by +-(i / 2) steps of c * edeta.  Below one quantum the emission
  // tables return at once, without a draw.  `which` follows kDispNames.
  template <class Draw>
  __device__ double fek(int which, double eet, Draw &&draw) const {
    const DevTables &T = F.T;
    const bool emit = (which & 1) == 0;
    const int phon = which >> 1;  // 0 LO, 1 TO, 2 LA
    const double e = phon == 0 ? T.templog : (phon == 1 ? T.temptof : T.templaf);
    const double ie = eet / e;
    if (emit && ie < 1.0) return phon == 2 ? -1.0e-10 : 1.0e-10;
    // energy ranges: upper bound, offset, scale, first column, edeta
    double shift, mult, edeta;
    int base;
    bool last = false;
    if (phon == 0 && emit) {  // FEKLOEM
      if (ie < 3.05) { shift = 1.0; mult = 10.0; base = 0; edeta = 1.0; }
      else if (ie < 5.625) { shift = 3.0; mult = 4.0; base = 20; edeta = 2.0; }
      else if (ie < 13.25) { shift = 5.5; mult = 2.0; base = 30; edeta = 4.0; }
      else if (ie < 28.5) { shift = 13.0; mult = 1.0; base = 45; edeta = 8.0; }
      else { shift = 28.0; mult = 1.0; base = 60; edeta = 12.0; last = true; }
    } else if (phon == 0) {  // FEKLOAB
      if (ie < 1.05) { shift = 0.0; mult = 10.0; base = 0; edeta = 1.0; }
      else if (ie < 3.625) { shift = 1.0; mult = 4.0; base = 10; edeta = 2.0; }
      else if (ie < 11.25) { shift = 3.5; mult = 2.0; base = 20; edeta = 4.0; }
      else if (ie < 26.5) { shift = 11.0; mult = 1.0; base = 35; edeta = 8.0; }
      else { shift = 26.0; mult = 1.0; base = 50; edeta = 12.0; last = true; }
    } else if (emit) {  // FEKTOEM, FEKLAEM
      if (ie < 3.05) { shift = 1.0; mult = 10.0; base = 0; edeta = 0.25; }
      else if (ie < 5.625) { shift = 3.0; mult = 4.0; base = 20; edeta = 0.5; }
      else if (ie < 13.25) { shift = 5.5; mult = 2.0; base = 30; edeta = 0.5; }
      else { shift = 13.0; mult = 1.0; base = 45; edeta = 1.0; last = true; }
    } else {  // FEKTOAB, FEKLAAB
      if (ie < 1.05) { shift = 0.0; mult = 10.0; base = 0; edeta = 0.25; }
      else if (ie < 3.625) { shift = 1.0; mult = 4.0; base = 10; edeta = 0.25; }
      else if (ie < 11.25) { shift = 3.5; mult = 2.0; base = 20; edeta = 0.5; }
      else { shift = 11.0; mult = 1.0; base = 35; edeta = 1.0; last = true; }
    }
    int it = (int)((ie - shift) * mult + 0.5);
    if (it < 1) it = 1;
    if (last) {  // the last range's cap
      if (phon == 0) { if (it > 60) it = 60; }
      else if (emit) { if (it > 115) it = 115; }
      else if (it > 60) it = 115;  // as the reference: past 60 the column jumps to 150
    }
    const int ei = base + it;
    const int cols = phon == 0 ? (emit ? 120 : 110) : (emit ? 160 : 150);
    const int rows = phon == 0 ? 201 : 51;
    const double *tab = T.disp + T.disp_off[which] + (ei - 1);
    const double ran = (double)draw();
    // The walk down the column, by the whole warp (its lanes all call this
    // with the same arguments): 32 rows are loaded at once and added in
    // order.  FEKLOEM wraps before the last row is added, the others after.
    const int lane = (int)(threadIdx.x & 31u);
    const int last_row = which == 0 ? rows - 1 : rows;
    int i = 1;
    double ksum = 0.0;
    bool open = true;
#pragma unroll 1
    for (int base = 0; open && base < last_row; base += 32) {
      const double mine = base + lane < last_row ? tab[(size_t)(base + lane) * cols] : 0.0;
#pragma unroll 1
      for (int t = 0; t < 32 && base + t < last_row; ++t) {
        ksum += __shfl_sync(0xffffffffu, mine, t);
        if (!(ksum < ran)) {
          i = base + t + 1;
          open = false;
          break;
        }
      }
    }
    if (open || i == rows) i = 1;
    const int j = i % 2, k = i / 2;
    const double c = phon == 0 ? 0.01 : 0.04;
    double ef;
    if (emit) ef = j == 1 ? eet - e * (1.0 - c * edeta * k) : eet - e * (1.0 + c * edeta * k);
    else ef = j == 1 ? eet + e * (1.0 + c * edeta * k) : eet + e * (1.0 - c * edeta * k);
    if (phon == 2 && ef <= 0.0) ef = 1.0e-5 * e;
    return ef;
  }

  // Set-up of EPSCAT (src/ElectronPhononScatter.cpp:98-195; with
  // Flag_QuantumCorrection the LO / LA / TO events take their final energy
  // from fek, :152-167), ESCATII (:406-497, seciifl = false), HPSCAT
  // (src/HolePhononScatter.cpp:86-146) and HSCATII (:149-234) for mechanism
  // iscat: the final band and energy, and the wedge rule of the draw (tal:
  // 1..3 = TALIND(tal), 0 = a random isym, -1 = none).  Returns whether the
  // event is a phonon's.
  template <class Draw>
  __device__ __forceinline__ bool scatter_setup(int iscat, int carrier, bool quantum, double &en, int &ib, int &tal,
                                                Draw &&draw) const {
    const DevTables &T = F.T;
    const int per = carrier == 0 ? T.scpre : T.scprh;
    ib = iscat / per + T.bandof[carrier == 0 ? 0 : 1];
    const int m = iscat % per;
    tal = 0;
    if (m + 1 == per) {  // ESCATII, HSCATII
      en = (en - T.sieg) / 3.0;
      return false;
    }
    if (carrier != 0) {
      if (m == 1) en = en + T.temphop;
      else if (m == 2) en = en - T.temphop;
      return true;
    }
    if (m == 0) {
      tal = 1;
      return true;
    }
    tal = m > 12 ? -1 : (m <= 6 ? 2 : 3);
    if (m > 12) return true;
    if (quantum && (m == 5 || m == 6 || m >= 9)) {
      // the dispersion table of the event: LO 5 / 6, LA 9 / 10, TO 11 / 12
      // (absorption / emission); the energy before the event
      en = fek(m <= 6 ? 6 - m : 14 - m, en, draw);
      return true;
    }
    const int q = (m - 1) >> 1;  // absorption (m odd) and emission of each phonon
    const double ph = q == 0 ? T.temptag : q == 1 ? T.templag : q == 2 ? T.templog : q == 3 ? T.temptaf
                      : q == 4 ? T.templaf : T.temptof;
    en = (m & 1) ? en + ph : en - ph;
    return true;
  }

  // The final-state draws of the lanes in `owners` (draw_kind), one owner at
  // a time by the whole warp; every lane of the warp calls it.
  __device__ __forceinline__ void final_states(unsigned owners);

  // GetImpScRate, src/ElectronImpurityScatter.cpp:62-126 (Brooks-Herring,
  // bhmrtfl = false).  FP32: the same rate written as
  // imp_a * sqrt(e) / (1 + imp_b * e) with the cell's constants (load_cell_fields).
  __device__ R GetImpScRate(R eel) const {
    if constexpr (sizeof(R) == 4) {
      return eel < imp_ecut ? imp_a * m_sqrt(eel) / ((R)1 + imp_b * eel) : (R)0;
    } else {
      const DevTables &T = F.T;
      if (!(eel * T.eV0 < 0.120) || imp_a == 0.0) return 0.0;
      return imp_a * sqrt(2.0 * T.meld * eel) / (imp_c * (1.0 + 4.0 * eel * T.melt / imp_b));
    }
  }

  // GetImpScGamma, src/ElectronImpurityScatter.cpp:6-59: majorant of the
  // BH rate over the tet's energy span.
  __device__ R GetImpScGamma() const {
    const DevTables &T = F.T;
    const R eemax = imp_emax;
    const TetFlightT<R> &s = tf(itet);
    // the rate at the energy of the span nearest its peak (one evaluation)
    const R gammax = GetImpScRate(eemax < s.e0 ? s.e0 : (eemax > s.e3 ? s.e3 : eemax));
    const R floor_ = TB::k(T).gamma_floor;
    return gammax > floor_ ? gammax : floor_;
  }

  // EleImpScUpdateK, src/ElectronImpurityScatter.cpp:188-306.
  __device__ void EleImpScUpdateK();

  // GetSurfScRate, src/ParSurfaceScatter.cpp:3-45.
  __device__ void GetSurfScRate() {
    const int c = cell_index();
    if (type == 0) { rough_rate = (R)I->M.e_rough[c]; sphon_rate = (R)I->M.e_sphon[c]; }
    else { rough_rate = (R)I->M.h_rough[c]; sphon_rate = (R)I->M.h_sphon[c]; }
    surf_gamma = rough_rate + sphon_rate;
  }

  __device__ void reflect_axis(int axis) {
    if (axis == 0) kx = -kx;
    else if (axis == 1) ky = -ky;
    else kz = -kz;
    isym = S.refl[axis * 48 + isym];
  }
  // Reflect, src/CellHit.cpp:214-240.
  __device__ void Reflect() {
    if (idir == kUp || idir == kDown) reflect_axis(0);
    else if (idir == kRight || idir == kLeft) reflect_axis(1);
    else if (idir == kFront || idir == kBack) reflect_axis(2);
  }
  __device__ bool inside_mesh(int i, int j, int k) const {
    return i >= 0 && j >= 0 && k >= 0 && i < I->M.nx && j < I->M.ny && k < I->M.nz;
  }
  // Pass, src/CellHit.cpp:389-413.  A PASS rule on the outer x / z boundary
  // would move the particle off the mesh (the reference indexes out of its
  // arrays there); the engine removes such a particle and counts it.
  __device__ void Pass() {
    int ni, nj, nk;
    neighbour(ni, nj, nk);
    if (!inside_mesh(ni, nj, nk)) {
      count(I->Y, kCntUnfinished);
      catch_ = true;
      return;
    }
    // the face, in the new cell's frame (FP32) or absolute; faces come in
    // pairs per axis, the odd one towards larger coordinates
    const DevMesh &M = I->M;
    const int axis = idir >> 1, up = idir & 1;
    const int old = axis == 0 ? ic : (axis == 1 ? jc : kc), to = up ? old + 1 : old - 1;
    R at;
    if constexpr (Real::kCellRelative) {
      const float *w = axis == 0 ? M.dxf : (axis == 1 ? M.dyf : M.dzf);
      at = up ? (R)0 : w[to];
    } else {
      const double *l = axis == 0 ? M.lx : (axis == 1 ? M.ly : M.lz);
      at = l[old + up];
    }
    if (axis == 0) { x = at; ic = to; }
    else if (axis == 1) {
      y = at;
      jc = to;
      tally_add_i64((up ? I->Y.rcurrent : I->Y.lcurrent) + old + up, charge, kChargeScale);
    } else { z = at; kc = to; }
  }
  // Period, src/CellHit.cpp:416-432.
  __device__ void Period() {
    const DevMesh &M = I->M;
    if constexpr (Real::kCellRelative) {
      if (idir == kUp) x = M.dxf[ic];
      else if (idir == kDown) x = 0;
      else if (idir == kLeft) y = M.dyf[jc];
      else if (idir == kRight) y = 0;
      else if (idir == kFront) z = M.dzf[kc];
      else if (idir == kBack) z = 0;
    } else {
      if (idir == kUp) x = M.lx[ic + 1];
      else if (idir == kDown) x = M.lx[ic];
      else if (idir == kLeft) y = M.ly[jc + 1];
      else if (idir == kRight) y = M.ly[jc];
      else if (idir == kFront) z = M.lz[kc + 1];
      else if (idir == kBack) z = M.lz[kc];
    }
  }
  __device__ void neighbour(int &i, int &j, int &k) const {
    i = ic; j = jc; k = kc;
    switch (idir) {
      case kUp: i = ic - 1; break;
      case kDown: i = ic + 1; break;
      case kLeft: j = jc - 1; break;
      case kRight: j = jc + 1; break;
      case kFront: k = kc - 1; break;
      case kBack: k = kc + 1; break;
    }
  }
  __device__ void contact_add(int icont, int slot, double v, double scale) const {
    if (icont < 0 || icont >= kMaxContacts) return;
    tally_add_i64(I->Y.contact + icont * 6 + slot, v, scale);
  }
  // Generate, src/CellHit.cpp:435-501: tally, then a copy of the particle
  // enters the neighbour cell and finishes the step there.
  __device__ void Generate() {
    count(I->Y, kCntGenerated);
    const int icont = I->M.contact[cell_index()] - 1;
    if (icont >= 0) {
      atomicAdd(reinterpret_cast<unsigned long long *>(I->Y.contact + icont * 6 + 0), 1ull);
      contact_add(icont, 1, charge, kChargeScale);
      contact_add(icont, 2, energy, kEnergyScale);
    }
    if (idir == kRight) tally_add_i64(I->Y.rcurrent + jc + 1, charge, kChargeScale);
    if (idir == kLeft) tally_add_i64(I->Y.lcurrent + jc, charge, kChargeScale);
    int i, j, k;
    neighbour(i, j, k);
    if (!inside_mesh(i, j, k)) {
      count(I->Y, kCntUnfinished);
      return;
    }
    const DevChildrenT<R> &C = I->C;
    const unsigned slot = atomicAdd(C.count, 1u);
    const uint32_t csub = sub * 16u + 1u + (uint32_t)nchild++;
    if ((int)slot >= C.capacity) {
      count(I->Y, kCntChildOverflow);
      return;
    }
    R cx = x, cy = y, cz = z;
    if constexpr (Real::kCellRelative) {  // the same point in the neighbour cell's frame
      const DevMesh &M = I->M;
      switch (idir) {
        case kUp: cx = x + M.dxf[i]; break;
        case kDown: cx = x - M.dxf[ic]; break;
        case kLeft: cy = y + M.dyf[j]; break;
        case kRight: cy = y - M.dyf[jc]; break;
        case kFront: cz = z + M.dzf[k]; break;
        case kBack: cz = z - M.dzf[kc]; break;
      }
    }
    C.x[slot] = cx; C.y[slot] = cy; C.z[slot] = cz;
    C.kx[slot] = kx; C.ky[slot] = ky; C.kz[slot] = kz;
    C.energy[slot] = energy; C.charge[slot] = charge; C.left_time[slot] = left_time;
    C.cell[slot] = pack_cell(i, j, k);
    C.itet[slot] = itet;
    C.meta[slot] = (uint32_t)isym | ((uint32_t)type << 8);
    C.parent_uid[slot] = uid;
    C.sub[slot] = csub;
  }
  // CatchAtContact / CatchAtGate, src/CellHit.cpp:504-574.
  __device__ void Catch(bool with_current) {
    int i, j, k;
    neighbour(i, j, k);
    const int icont = inside_mesh(i, j, k) ? I->M.contact[cell_index(i, j, k)] - 1 : -1;
    if (with_current) {
      if (idir == kRight) tally_add_i64(I->Y.rcurrent + jc + 1, charge, kChargeScale);
      if (idir == kLeft) tally_add_i64(I->Y.lcurrent + jc, charge, kChargeScale);
    }
    if (icont >= 0 && icont < kMaxContacts) {
      atomicAdd(reinterpret_cast<unsigned long long *>(I->Y.contact + icont * 6 + 3), 1ull);
      contact_add(icont, 4, charge, kChargeScale);
      contact_add(icont, 2, energy, kEnergyScale);  // the reference adds to EnergyGen here (src/CellHit.cpp:542)
    }
  }
  __device__ void load_cell_fields() {
    const int c = cell_index();
    const DevMesh &M = I->M;
    if constexpr (sizeof(R) == 8) {
      const double *f = (type == 0 ? M.efield : M.hfield) + 3 * (size_t)c;
      Ex = f[0];
      Ey = f[1];
      Ez = f[2];
      if (type == 0) {
        const double2 *r = M.cell64 + 3 * (size_t)c;
        const double2 a = r[0], b = r[1], m = r[2];
        imp_a = a.x;
        imp_b = a.y;
        imp_c = b.x;
        imp_emax = b.y;
        imp_beta = m.x;
      }
    } else {
      const float4 *r = M.cell32 + 3 * (size_t)c;
      if (type == 0) {
        const float4 a = r[0], b = r[1], m = r[2];
        Ex = a.x; Ey = a.y; Ez = a.z;
        imp_a = a.w;
        imp_b = b.w;
        imp_emax = m.x;
        imp_beta = m.y;
        imp_ecut = m.z;
      } else {
        const float4 b = r[1];
        Ex = b.x; Ey = b.y; Ez = b.z;
      }
    }
  }
  // HitCell, src/CellHit.cpp:96-211.  Returns false when the particle would
  // leave the device through a PASS / GENERATE face on the outer y boundary.
  // imot: the face's rule; u: the draw of a SCATTOX face without surface scattering.
  __device__ bool HitCell(int imot, R u) {
    if (imot == kPass || imot == kGenerate || imot == kGenRef) {
      if ((idir == kLeft && jc == 0) || (idir == kRight && jc == I->M.ny - 1)) return false;
    }
    if (imot == kPass) Pass();
    else if (imot == kReflect) Reflect();
    else if (imot == kScattOx) {
      if (I->M.surface_scatter) Reflect();
      else {
        if (u > (R)F.T.difpr[type]) Reflect();
        else draw_kind = kDrawDiffuse;
      }
    } else if (imot == kPeriod) Period();
    else if (imot == kGenerate || imot == kGenRef) {
      Generate();
      Reflect();
    } else if (imot == kCatch) {
      Catch(true);
      catch_ = true;
    } else if (imot == kCatchGate) {
      Catch(false);
      catch_ = true;
    } else {
      catch_ = true;  // no such rule: the reference exits
      count(I->Y, kCntNoTet);
    }
    load_cell_fields();
    return true;
  }
  // One particle, one step: particle_fly, src/mcmodel.cpp:1874-2161, split
  // into begin (the set-up before the event loop), one pass of the loop as
  // advance (to the next event, and the events that are done on the spot),
  // run_pending and final_states (the work the others left) and settle (the
  // end of the pass; true when the particle's step is over), and finish (the
  // tallies after the loop), so a kernel can interleave particles on one
  // lane and keep a lane's pending work until other lanes have some too.
  // Loop state (particle_fly's locals):
  bool get_tet, get_cell, get_ph, get_imp, get_surf, too_far;
  R ssnl, imprnl, phrnl, TetTf, CellTf;
  int loop, zero_run;
  int counted;  // of `loop`, the events already added to the counters

  __device__ void begin() {
    catch_ = false;
    imp_pending = false;
    draw_kind = kDrawNone;
    loc_mode = kLocNone;
    get_tet = get_cell = get_ph = get_imp = get_surf = true;
    ssnl = imprnl = phrnl = 0;
    TetTf = CellTf = 0;
    too_far = false;
    zero_run = 0;
    load_cell_fields();
    iband = tf(itet).band;
    GetV();
    loop = counted = 0;
    surf_gamma = 0;
    imp_gamma = 0;
  }

  // The drift pass (no begin(): the cell's fields, band and velocity are
  // loaded).  no_event: whether the step certainly ends before the first
  // event, from the same times as advance() compares but without forming
  // the quotients: an event at num / rate > T, for every rounding of it, is
  // num > rate T with a margin.  drift: the step's motion as advance() makes
  // it; false (nothing changed) when the energy would turn negative.
  __device__ __forceinline__ bool no_event() const;
  __device__ __forceinline__ bool drift() {
    const R T = (R)left_time;
    const double e = energy + (vx * Ex + vy * Ey + vz * Ez) * T;
    if (e < 0) return false;
    energy = e;
    kx += Ex * T;
    ky += Ey * T;
    kz += Ez * T;
    x += vx * T;
    y += vy * T;
    z += vz * T;
    return true;
  }

  // The flight's state while it waits for a final-state draw.
  __device__ __forceinline__ void save(const FlightListsT<R> &m, int p) const {
    m.phrnl[p] = phrnl;
    m.imprnl[p] = imprnl;
    m.ssnl[p] = ssnl;
    m.tet_time[p] = TetTf;
    m.cell_time[p] = CellTf;
    m.pick_drand[p] = pick_drand;
    m.left_time[p] = left_time;
    m.progress[p] = make_uint2(n, (uint32_t)loop | (uint32_t)zero_run << 20);
    m.info[p] = (get_tet ? 1u : 0u) | (get_ph ? 2u : 0u) | (get_imp ? 4u : 0u) | (get_surf ? 8u : 0u) |
                (self ? 16u : 0u) | (imp_pending ? 32u : 0u) | (uint32_t)loc_mode << 6 | (uint32_t)draw_kind << 8 |
                (uint32_t)idir << 10 | (uint32_t)itetdir << 13 | (uint32_t)ev << 15;
    m.copies[p] = nchild;
  }
  // After the store's part is loaded.
  __device__ __forceinline__ void resume(const FlightListsT<R> &m, int p) {
    phrnl = m.phrnl[p];
    imprnl = m.imprnl[p];
    ssnl = m.ssnl[p];
    TetTf = m.tet_time[p];
    CellTf = m.cell_time[p];
    pick_drand = m.pick_drand[p];
    left_time = m.left_time[p];
    const uint2 c = m.progress[p];
    n = c.x;
    stocked = n & ~(kBlockDraws - 1u);
    loop = counted = (int)(c.y & 0xfffffu);
    zero_run = (int)(c.y >> 20);
    const uint32_t w = m.info[p];
    get_tet = get_cell = w & 1u;
    get_ph = w & 2u;
    get_imp = w & 4u;
    get_surf = w & 8u;
    self = w & 16u;
    imp_pending = w & 32u;
    loc_mode = (int)(w >> 6 & 3u);
    draw_kind = (int)(w >> 8 & 3u);
    idir = (int)(w >> 10 & 7u);
    itetdir = (int)(w >> 13 & 3u);
    ev = (int)(w >> 15 & 7u);
    nchild = m.copies[p];
    catch_ = too_far = false;
    surf_gamma = imp_gamma = 0;
    load_cell_fields();
    iband = tf(itet).band;
  }

  // What is left after an advance().
  enum : int { kGoOn = 0, kStepOver = 1, kPending = 2, kDraw = 3 };
  __device__ int advance() {
    GetV();
    if (++loop > kMaxEvents) {
      count(I->Y, kCntTooManyEvents);
      catch_ = true;
      return kStepOver;
    }
    if (get_tet) { TetTf = TetTime(); get_tet = false; }
    if (get_cell) { CellTf = CellTime(); get_cell = false; }
    const bool impurities = iband == F.T.bandof[0];
    const bool surface = I->M.surface_scatter && I->M.in_surf[cell_index()];
    // the clocks that are to be drawn, in the reference's order (rolled: one
    // copy of the stream and the logarithm in the loop's code)
    unsigned clocks = (get_ph ? 1u : 0u) | (impurities && get_imp ? 2u : 0u) | (surface && get_surf ? 4u : 0u);
    // FP32: a block serves the pass's four draws at most; FP64: its clocks
    stock(sizeof(R) == 4 ? 4u : (uint32_t)__popc(clocks));
#pragma unroll 1
    while (clocks) {
      const R v = -m_log(Random());
      if (clocks & 1u) { phrnl = v; get_ph = false; }
      else if (clocks & 2u) { imprnl = v; get_imp = false; }
      else { ssnl = v; get_surf = false; }
      clocks &= clocks - 1u;
    }
    const R g = tf(itet).gam;
    R PhScTf, ImpScTf, SurfScTf, Tf;
    PhScTf = phrnl / g;
    if (impurities) {
      imp_gamma = GetImpScGamma();
      ImpScTf = imprnl / imp_gamma;
    } else {
      ImpScTf = (R)(2 * I->dt);
      imp_gamma = TB::k(F.T).gamma_floor;
    }
    SurfScTf = (R)(2 * I->dt);
    if (surface) {
      GetSurfScRate();
      if (surf_gamma > 0 && ssnl > 0) SurfScTf = ssnl / surf_gamma;
    }
    // Min(..., flag), src/Constant_GlobalVariable_MathFunction.cpp:92-118
    int flag = 1;
    Tf = TetTf;
    if (Tf > CellTf) { Tf = CellTf; flag = 2; }
    if (Tf > PhScTf) { Tf = PhScTf; flag = 3; }
    if (Tf > ImpScTf) { Tf = ImpScTf; flag = 4; }
    if (Tf > SurfScTf) { Tf = SurfScTf; flag = 5; }
    if ((double)Tf > left_time) { Tf = (R)left_time; flag = 6; }
    if constexpr (sizeof(R) == 8) {
      if (Tf < kMyZero) {
        catch_ = true;
        return kStepOver;
      }
    } else {
      // float event times that round to zero (or below) are events now
      if (!(Tf > (R)0)) {
        Tf = 0;
        if (++zero_run > kMaxZeroTimeEvents) {
          count(I->Y, kCntZeroTime);
          catch_ = true;
          return kStepOver;
        }
      } else {
        zero_run = 0;
      }
    }
    TetTf -= Tf;
    CellTf -= Tf;
    PhScTf -= Tf;
    ImpScTf -= Tf;
    SurfScTf -= Tf;
    if constexpr (MCB200_FLIGHT_EVENT_STATS != 0)
      count(I->Y, flag == 1 ? kStatTetFace : flag == 2 ? kStatCellFace : flag == 6 ? kStatStepEnd : kStatScatter);
    if (flag == 6) left_time = 0;  // Tf == left_time: the step is used up
    else left_time -= Tf;
    phrnl -= g * Tf;
    imprnl -= imp_gamma * Tf;
    ssnl -= surf_gamma * Tf;
    kx += Ex * Tf;
    ky += Ey * Tf;
    kz += Ez * Tf;
    energy += (vx * Ex + vy * Ey + vz * Ez) * Tf;
    x += vx * Tf;
    y += vy * Tf;
    z += vz * Tf;
    if (energy < 0) {
      catch_ = true;
      return kStepOver;
    }
    ev = flag;
    int imot = 0;
    if (flag == 2) imot = I->M.motion[(size_t)cell_index() * 6 + idir];
    R u = 0;  // the event's draw
    if ((flag >= 3 && flag <= 5) || (imot == kScattOx && !I->M.surface_scatter)) {
      if constexpr (sizeof(R) == 8) stock(1);
      u = Random();
    }
    switch (flag) {
      case 1:
        HitTet();
        get_tet = true;
        get_cell = true;
        break;
      case 2:
        if (HitCell(imot, u)) {
          get_tet = true;
          get_cell = true;
        } else {
          // trace_back, src/mcmodel.cpp:1774-1783
          kx -= Ex * Tf;
          ky -= Ey * Tf;
          kz -= Ez * Tf;
          energy -= (vx * Ex + vy * Ey + vz * Ez) * Tf;
          x -= vx * Tf;
          y -= vy * Tf;
          z -= vz * Tf;
          left_time += Tf;
          too_far = true;
        }
        break;
      case 3: {
        // ElectronPhononScatter (src/ElectronPhononScatter.cpp:5-95) and
        // HolePhononScatter (src/HolePhononScatter.cpp:4-83): real or
        // self-scattering against the variable-gamma majorant
        const R scasum = CALSCATTSUM((R)energy, iband);
        pick_drand = u * (scasum > g ? scasum : g);
        self = scasum < pick_drand;
        if (!self) draw_kind = kDrawPick;
        break;
      }
      case 4:
        // ElectronImpurityScatter, src/ElectronImpurityScatter.cpp:128-185
        // (electrons: a hole's impurity time is past the step's end)
        if (GetImpScRate((R)energy) < u * imp_gamma) self = true;
        else imp_pending = true;
        break;
      case 5:
        // ParticleSurfaceScatter, src/ParSurfaceScatter.cpp:48-61, with the
        // surface-phonon branches' drand defined (see file note)
        if (u * surf_gamma < rough_rate) {
          idir = I->M.surface_dir[min(max(I->M.nearest_surf[cell_index()], 0), kMaxSurfaces - 1)];
          draw_kind = kDrawDiffuse;
        } else {
          draw_kind = kDrawPickSurface;
        }
        break;
    }
    if (draw_kind != kDrawNone) return kDraw;
    if (imp_pending || loc_mode != kLocNone) return kPending;
    return settle() ? kStepOver : kGoOn;
  }

  __device__ void run_pending() {
    if (imp_pending) {
      imp_pending = false;
      EleImpScUpdateK();
    }
    if (loc_mode != kLocNone) run_locate();
  }

  __device__ __forceinline__ bool settle() {
    if (ev == 3) {
      if (!self) {
        get_tet = true;
        get_cell = true;
        ++n_ph;
      }
      get_ph = true;
    } else if (ev == 4) {
      if (!self) {
        get_tet = true;
        get_cell = true;
        ++n_imp;
      }
      get_imp = true;
    } else if (ev == 5) {
      if (!self) {
        get_tet = true;
        get_cell = true;
      }
      get_surf = true;
    }
    if (too_far || catch_) return true;
    return !(left_time > 0);
  }

  // The particle's events into the simulation's counters (a caller that sums
  // them itself, one simulation per launch, does not call it).
  __device__ void count_events() {
    atomicAdd(&I->Y.counters[kCntEvents], (unsigned long long)(loop - counted));
    if (n_ph) atomicAdd(&I->Y.counters[kCntPhonon], (unsigned long long)n_ph);
    if (n_imp) atomicAdd(&I->Y.counters[kCntImpurity], (unsigned long long)n_imp);
    n_ph = n_imp = 0;
  }
  // Returns 0 done, 1 caught, 2 unfinished (outer-boundary PASS).
  __device__ int finish() {
    if (catch_) {
      count(I->Y, kCntCaught);
      return 1;
    }
    if (too_far) {
      count(I->Y, kCntUnfinished);
      return 2;
    }
    return 0;
  }
};
using Flyer = FlyerT<double>;

}  // namespace mcb200
