// quantum_kernels.cu -- the effective potential of the quantum region
// (quantum_setup.h; MeshQuantities::effective_potential / quantumPotential,
// src/mcmodel.cpp:2337-2403).
#include "quantum_setup.h"

namespace mcb200 {

namespace {

__global__ void copy_potential_kernel(int nodes, const double *pot, double *out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < nodes) out[n] = pot[n];
}

__global__ void erf_differences_kernel(const double2 *edge, const double *target, const int2 *window, int n, int width,
                                       double *out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n * width * kBoxKinds) return;
  const int kind = q % kBoxKinds, w = (q / kBoxKinds) % width, t = q / (kBoxKinds * width);
  const int from = window[t].x + w;
  if (from > window[t].y) {
    out[q] = 0.0;
    return;
  }
  const double2 e = edge[from * kBoxKinds + kind];
  out[q] = erf(e.y - target[t]) - erf(e.x - target[t]);
}

// A group of lanes per quantum node.  The window's terms are taken in the
// reference's order (x outer, z inner), eight at a time: lane g forms term
// f + g, the product of the three tabulated erf differences in the reference's
// association ((V + Eb) * dz) * dy) * dx, and every lane adds the eight to its
// running sum one after another, so the sum is the reference's to the last
// bit (a node outside adds a zero, which changes no sum).  Every term reads
// `pot`, never `out`, so no node sees another's corrected value.
//
// A 20 nm FinFET's 52k targets of up to 500 terms: 145 us; one thread per
// target, without the shuffles, takes as long there and longer where there are
// fewer targets (36k: 94 against 136), and six erf per term in place of the
// tables took 1.24 ms.  (Eight partial sums, each over every eighth row, took
// 85 us but moved the potential in its last digits, and with it the
// trajectories of the steps that follow.)
constexpr int kLanes = 8;
__global__ void __launch_bounds__(256) effective_potential_kernel(const __grid_constant__ QuantumDevice q,
                                                                  const double *pot, double *out) {
  const int g = threadIdx.x % kLanes;
  const unsigned mask = 0xffu << (threadIdx.x & 31 & ~(kLanes - 1));
  static_assert(kLanes == 8, "the group's mask");
  const int groups = gridDim.x * blockDim.x / kLanes;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes; t < q.n_list; t += groups) {
    const int n = q.list[t];
    const int pk = n % q.pz, r = n / q.pz, pi = r % q.px, pj = r / q.px;
    const int2 wx = q.window[pi], wy = q.window[q.px + pj], wz = q.window[q.px + q.py + pk];
    // (a window can be empty, its end before its start: under a negative ratio)
    const int nx = max(wx.y - wx.x + 1, 0), ny = max(wy.y - wy.x + 1, 0), nz = max(wz.y - wz.x + 1, 0);
    const int terms = nx * ny * nz;
    const double *ex = q.erf_diff[0] + (size_t)pi * q.width[0] * kBoxKinds;
    const double *ey = q.erf_diff[1] + (size_t)pj * q.width[1] * kBoxKinds;
    const double *ez = q.erf_diff[2] + (size_t)pk * q.width[2] * kBoxKinds;
    double ret = 0.0;
    int i = 0, j = 0, k = g;  // the lane's term
#pragma unroll 2
    for (int f = 0; f < terms; f += kLanes) {
      for (; k >= nz; k -= nz)
        if (++j == ny) {
          j = 0;
          ++i;
        }
      double term = 0.0;
      if (f + g < terms) {
        const size_t m = ((size_t)(wy.x + j) * q.px + wx.x + i) * q.pz + wz.x + k;
        const unsigned box = q.inside[m];
        const double v = pot[m] + q.eb[m];
        const unsigned kinds = box - 1u;
        if (box)
          term = v * ez[k * kBoxKinds + ((kinds >> 4) & 3u)] * ey[j * kBoxKinds + ((kinds >> 2) & 3u)] *
                 ex[i * kBoxKinds + (kinds & 3u)];
      }
      k += kLanes;
#pragma unroll
      for (int s = 0; s < kLanes; ++s) ret += __shfl_sync(mask, term, s, kLanes);
    }
    if (g == 0) out[n] = ret * 0.125;
  }
}

}  // namespace

void launch_effective_potential(const QuantumDevice &q, const double *pot, double *out, cudaStream_t s) {
  const int nodes = q.px * q.py * q.pz;
  if (nodes <= 0) return;
  copy_potential_kernel<<<(nodes + 255) / 256, 256, 0, s>>>(nodes, pot, out);
  if (q.n_list > 0) {
    const long long threads = (long long)q.n_list * kLanes;
    effective_potential_kernel<<<(int)((threads + 255) / 256), 256, 0, s>>>(q, pot, out);
  }
}

void launch_erf_differences(const double2 *edge, const double *target, const int2 *window, int n, int width,
                            double *out, cudaStream_t s) {
  const int total = n * width * kBoxKinds;
  if (total > 0) erf_differences_kernel<<<(total + 255) / 256, 256, 0, s>>>(edge, target, window, n, width, out);
}

}  // namespace mcb200
