// stat_kernels.cu -- the per-step statistics the reference writes every
// stat_step steps (MeshQuantities::statistic, src/mcmodel.cpp:1167-1408):
// per node and carrier type the CIC-weighted |q| v_x, |q| v_y, |q| v_z,
// |q| and |q| E of every particle, per cell the particle count, and per node
// the potential; summed over the steps of a statistics window.  Also the
// current one contact carries by induction (Ramo-Shockley, a tally of the
// transport step): sum over particles of q v . E_w.
//
// Node sums are int64 fixed point (order independent).  A window's scales
// are fixed when it starts, from bounds every sum respects for the whole
// window: |q| sums <= (particles of the type) x max|q| x steps x 4 (the
// factor leaves room for GENERATE copies and refreshes), |v| <= the
// largest group-velocity component of the band tables, |E| <= the energy
// table's top.
#include <algorithm>

#include "stat_kernels.h"
#include "field_kernels.h"
#include "warp_segments.cuh"

namespace mcb200 {

constexpr uint32_t kStatDead = 1u << 16;

__device__ __forceinline__ long long st_fx(double v, double scale) { return __double2ll_rn(v * scale); }
__device__ __forceinline__ void st_put(long long *p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}

// GetV (src/ParticleUtils.cpp:307-313) from the FP64 tables: the wedge
// velocity of itet mapped out of the wedge of isym.
__device__ __forceinline__ void group_velocity(const DevTables &T, int itet, int isym, double &vx, double &vy,
                                               double &vz) {
  const double *v = T.tf[itet].v;
  const int *m = T.symi + isym * 6;  // matsym[c][isym] at isym * 6 + c
  const int p0 = m[0] - 1, p1 = m[1] - 1, p2 = m[2] - 1;
  vx = (p0 == 0 ? v[0] : (p0 == 1 ? v[1] : v[2])) * (double)m[3];
  vy = (p1 == 0 ? v[0] : (p1 == 1 ? v[1] : v[2])) * (double)m[4];
  vz = (p2 == 0 ? v[0] : (p2 == 1 ? v[1] : v[2])) * (double)m[5];
}

// Runs of particles of the same cell and carrier type add up before their
// atomics (warp_segments.cuh).  A node's five sums lie side by side, so the
// ten of two corners (b, a, k) and (b, a, k + 1) are consecutive words: row
// 10 (2 b + a) + 5 d + t holds tally t of corner (i + a, j + b, k + d).
// Lane l owns row l, and lanes 0-7 rows 32-39 too.
//
// Bound by the latency of about 800 instructions a chunk at 20 warps per SM and
// by shared memory (issue slots at 47 %, the SM's memory pipes at 77, DRAM at
// 10), with short runs also by their ends.  One
// wave of blocks, each warp with its share of chunks, and the next particles
// fetched ahead took 142 us for 2M electrons of a bulk box to 93; shuffles
// took 231.  A 20 nm FinFET (511k carriers): 53 us, 40 here; a bar of 4k: 9.0, 5.9.
constexpr int kStatThreads = 128, kStatBlocks = 5;  // four warps' 40 rows: 42.5 KB; blocks per SM
template <typename R>
__global__ void __launch_bounds__(kStatThreads, kStatBlocks) statistic_kernel(DevParticlesT<R> P, DevCount count, DevMesh M,
                                                                 DevTables T, StatScales S, StatBuffers B) {
  __shared__ __align__(16) long long rows[kStatThreads / 32][40 * kRunRow];
  const int n = count.get();
  const int px = M.nx + 1, pz = M.nz + 1;
  const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
  long long *terms = rows[warp];
  const int row[2] = {lane, 32 + (lane & 7)};
  long long *word[2];  // the row's sum at node 0
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const int ab = row[w] / 10;
    word[w] = B.node + 5 * (((size_t)(ab >> 1) * px + (ab & 1)) * pz) + row[w] % 10;
  }
  auto flush = [&](unsigned node, unsigned cell, int particles, const long long (&sum)[2]) {
    st_put(word[0] + 5 * (size_t)node, sum[0]);
    if (lane < 8) st_put(word[1] + 5 * (size_t)node, sum[1]);
    if (lane == 8) atomicAdd(B.cell_count + cell, (unsigned long long)particles);
  };
  // the warp's chunks of 32 follow one another, so that a run goes on
  const int chunks = (n + 31) / 32, warps = (int)gridDim.x * (kStatThreads / 32);
  const int each = (chunks + warps - 1) / warps;
  const int from = ((int)blockIdx.x * (kStatThreads / 32) + warp) * each, to = min(from + each, chunks);
  if (from >= to) return;
  RunWalk<2> walk;
  // the next chunk's particles are on their way while this one's rows are walked
  struct Particle {
    uint32_t meta = kStatDead, cell = 0;
    int itet = 0;
    R x = 0, y = 0, z = 0;
    double charge = 0, energy = 0;
  };
  auto fetch = [&](int chunk) {
    Particle f;
    const int p = chunk * 32 + lane;
    if (chunk < to && p < n) {
      f.meta = P.meta[p];
      f.cell = P.cell[p];
      f.itet = P.itet[p];
      f.x = P.x[p]; f.y = P.y[p]; f.z = P.z[p];
      f.charge = P.charge[p];
      f.energy = P.energy[p];
    }
    return f;
  };
  Particle next = fetch(from);
  for (int chunk = from; chunk < to; ++chunk) {
    const Particle f = next;
    next = fetch(chunk + 1);
    const uint32_t meta = f.meta;
    const bool live = !(meta & kStatDead);
    const uint32_t c = live ? f.cell : 0u;
    const int type = ((meta >> 8) & 255) == 0 ? 0 : 1;
    const int i = c & 1023, j = (c >> 10) & 1023, k = (c >> 20) & 1023;
    double vx = 0, vy = 0, vz = 0, rx = 0, ry = 0, rz = 0, q = 0, e = 0;
    if (live) {
      group_velocity(T, f.itet, meta & 255, vx, vy, vz);
      if constexpr (sizeof(R) == 4) {
        rx = (double)f.x / M.dx[i];
        ry = (double)f.y / M.dy[j];
        rz = (double)f.z / M.dz[k];
      } else {
        rx = (f.x - M.lx[i]) / M.dx[i];
        ry = (f.y - M.ly[j]) / M.dy[j];
        rz = (f.z - M.lz[k]) / M.dz[k];
      }
      q = f.charge;
      e = f.energy;
    }
    const double sq = type ? S.q[1] : S.q[0], sv = type ? S.v[1] : S.v[0], se = type ? S.e[1] : S.e[0];
    auto put = [&](int a, int b, int d, double w) {
      const double aq = fabs(q * w);
      long long *t = terms + (10 * (2 * b + a) + 5 * d) * kRunRow + lane;
      t[0 * kRunRow] = st_fx(vx * aq, sv);
      t[1 * kRunRow] = st_fx(vy * aq, sv);
      t[2 * kRunRow] = st_fx(vz * aq, sv);
      t[3 * kRunRow] = st_fx(aq, sq);
      t[4 * kRunRow] = st_fx(aq * e, se);
    };
    // the eight corners in the reference's order and weights
    put(0, 0, 0, (1 - rx) * (1 - ry) * (1 - rz));
    put(1, 0, 0, rx * (1 - ry) * (1 - rz));
    put(0, 0, 1, (1 - rx) * (1 - ry) * rz);
    put(1, 0, 1, rx * (1 - ry) * rz);
    put(0, 1, 0, (1 - rx) * ry * (1 - rz));
    put(1, 1, 0, rx * ry * (1 - rz));
    put(0, 1, 1, (1 - rx) * ry * rz);
    put(1, 1, 1, rx * ry * rz);
    walk.chunk(terms, row, live ? (c | ((unsigned)type << 30)) : kNoRun,
               (unsigned)type * (unsigned)B.nodes + (unsigned)((j * px + i) * pz + k),
               (unsigned)((j * M.nx + i) * M.nz + k), chunk * 32, flush);
  }
  walk.end(to * 32, flush);
}

// Sums out of fixed point, every stride-th word.
__global__ void fixed_values_kernel(int n, const long long *sums, int stride, double scale, double *out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) out[p] = (double)sums[(size_t)stride * p] / scale;
}

// The counters, the contact sums and the currents' rows, one after another
// into pinned host memory: one launch in place of four copies, of which two
// were waited for one by one (20 batched steps of 32 members and their
// tallies: 13.2 ms, 12.3 this way).
__global__ void small_tallies_kernel(DevTallies y, int rows, double *out) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < kCntNumCounters) {
    reinterpret_cast<unsigned long long *>(out)[t] = y.counters[t];
    return;
  }
  out += kCntNumCounters;
  t -= kCntNumCounters;
  if (t < kMaxContacts * 6) {  // per contact and direction: particles, charge, energy
    const int what = t % 3;
    out[t] = what == 0 ? (double)y.contact[t] : (double)y.contact[t] / (what == 1 ? kChargeScale : kEnergyScale);
    return;
  }
  out += kMaxContacts * 6;
  t -= kMaxContacts * 6;
  if (t < 2 * rows) out[t] = (double)(t < rows ? y.lcurrent[t] : y.rcurrent[t - rows]) / kChargeScale;
}

// stat_pot += pot: one thread per node, so the FP64 sum is exact to the
// reference's order (step by step).
__global__ void add_potential_kernel(int nodes, const double *pot, double *sum) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nodes) sum[p] += pot[p];
}

// The fixed-point unit of one step's induced-current terms: sum |q v . E_w|
// <= (electrons + holes) * max|q| * sqrt(3) vmax * sqrt(3) emax.
__device__ __forceinline__ double induced_unit(const unsigned long long *b, double vmax, double emax) {
  const double qmax = fmax(__longlong_as_double((long long)b[0]), __longlong_as_double((long long)b[1]));
  const double bound = fmax((double)(b[2] + b[3]) * qmax * vmax * emax * 3.0, 1e-300);
  return ldexp(1.0, 62 - (int)ceil(log2(bound)));
}

template <typename R>
__global__ void __launch_bounds__(256) induced_current_kernel(DevParticlesT<R> P, DevCount count, DevMesh M,
                                                              DevTables T, InducedBuffers B) {
  const int n = count.get();
  const double unit = induced_unit(B.bounds, B.vmax, B.emax);
  long long t = 0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const uint32_t meta = P.meta[p];
    if (meta & kStatDead) continue;
    const uint32_t c = P.cell[p];
    const int i = c & 1023, j = (c >> 10) & 1023, k = (c >> 20) & 1023;
    double vx, vy, vz;
    group_velocity(T, P.itet[p], meta & 255, vx, vy, vz);
    const double *ew = B.field + 3 * (size_t)((j * M.nx + i) * M.nz + k);
    t += st_fx(P.charge[p] * (vx * ew[0] + vy * ew[1] + vz * ew[2]), unit);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
  if ((threadIdx.x & 31u) == 0 && t) st_put(B.acc, t);
}
__global__ void induced_finish_kernel(InducedBuffers B) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    B.sum[0] += (double)*B.acc / induced_unit(B.bounds, B.vmax, B.emax);
    B.sum[1] += 1.0;
    *B.acc = 0;
  }
}

template <typename R>
void launch_statistic(const DevParticlesT<R> &P, DevCount n, const DevMesh &M, const DevTables &T, const StatScales &S,
                      const StatBuffers &B, int sm_count, cudaStream_t s) {
  const int grid = std::max(1, std::min((n.max + kStatThreads - 1) / kStatThreads, kStatBlocks * sm_count));
  statistic_kernel<R><<<grid, kStatThreads, 0, s>>>(P, n, M, T, S, B);
}
void launch_fixed_values(int n, const void *sums, int stride, double scale, double *out, cudaStream_t s) {
  if (n > 0)
    fixed_values_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, static_cast<const long long *>(sums), stride, scale, out);
}
void launch_small_tallies(const DevTallies &y, int rows, double *out, cudaStream_t s) {
  const int n = kCntNumCounters + kMaxContacts * 6 + 2 * rows;
  small_tallies_kernel<<<(n + 127) / 128, 128, 0, s>>>(y, rows, out);
}
void launch_add_potential(int nodes, const double *pot, double *sum, cudaStream_t s) {
  if (nodes > 0 && pot) add_potential_kernel<<<(nodes + 255) / 256, 256, 0, s>>>(nodes, pot, sum);
}

template <typename R>
void launch_induced_current(const DevParticlesT<R> &P, DevCount n, const DevMesh &M, const DevTables &T,
                            const InducedBuffers &B, int grid, cudaStream_t s) {
  induced_current_kernel<R><<<grid, 256, 0, s>>>(P, n, M, T, B);
  induced_finish_kernel<<<1, 32, 0, s>>>(B);
}
template void launch_induced_current<double>(const DevParticlesT<double> &, DevCount, const DevMesh &,
                                             const DevTables &, const InducedBuffers &, int, cudaStream_t);
template void launch_induced_current<float>(const DevParticlesT<float> &, DevCount, const DevMesh &,
                                            const DevTables &, const InducedBuffers &, int, cudaStream_t);
template void launch_statistic<double>(const DevParticlesT<double> &, DevCount, const DevMesh &, const DevTables &,
                                       const StatScales &, const StatBuffers &, int, cudaStream_t);
template void launch_statistic<float>(const DevParticlesT<float> &, DevCount, const DevMesh &, const DevTables &,
                                      const StatScales &, const StatBuffers &, int, cudaStream_t);

}  // namespace mcb200
