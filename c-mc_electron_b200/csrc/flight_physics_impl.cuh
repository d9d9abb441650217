// flight_physics_impl.cuh -- out-of-line members of FlyerT (flight_physics.cuh).
#pragma once

#include "flight_physics.cuh"

namespace mcb200 {

template <typename R>
__device__ __forceinline__ R dfii(R x1, R y1, R z1, R x2, R y2, R z2, R x3, R y3, R z3) {
  // Band::FII, src/Band.cpp:335-353
  const R sbx = (y2 - y1) * (z3 - z1) - (y3 - y1) * (z2 - z1);
  const R sby = (x3 - x1) * (z2 - z1) - (x2 - x1) * (z3 - z1);
  const R sbz = (x2 - x1) * (y3 - y1) - (x3 - x1) * (y2 - y1);
  return (R)0.50 * m_sqrt(sbx * sbx + sby * sby + sbz * sbz);
}

// Band::SURF, src/Band.cpp:194-332.
template <typename R>
__device__ __noinline__ R FlyerT<R>::SURF(const DevTables &T, R eps, int it) {
  const int4 nd = T.tnode[it];
  const V4 *kn = TB::knode(T);
  const V4 k0 = kn[nd.x], k1 = kn[nd.y], k2 = kn[nd.z], k3 = kn[nd.w];
  const R e0 = k0.w, e1 = k1.w, e2 = k2.w, e3 = k3.w;
  if (!(eps > e0 && eps < e3)) return 0;
  auto rel = [&](const V4 &p, const V4 &q, R &ox, R &oy, R &oz) {
    const R r = (eps - p.w) / (q.w - p.w);
    ox = r * (q.x - p.x);
    oy = r * (q.y - p.y);
    oz = r * (q.z - p.z);
  };
  auto abs_ = [&](const V4 &p, const V4 &q, R &ox, R &oy, R &oz) {
    const R r = (eps - p.w) / (q.w - p.w);
    ox = r * (q.x - p.x) + p.x;
    oy = r * (q.y - p.y) + p.y;
    oz = r * (q.z - p.z) + p.z;
  };
  R ax, ay, az, bx, by, bz, cx, cy, cz, dx, dy, dz;
  if (eps <= e1) {
    rel(k0, k1, ax, ay, az);
    rel(k0, k2, bx, by, bz);
    rel(k0, k3, cx, cy, cz);
    return dfii(ax, ay, az, bx, by, bz, cx, cy, cz);
  }
  if (eps > e1 && eps < e2) {
    abs_(k0, k2, ax, ay, az);
    abs_(k1, k2, bx, by, bz);
    abs_(k0, k3, cx, cy, cz);
    abs_(k1, k3, dx, dy, dz);
    const R a1 = dfii(ax, ay, az, bx, by, bz, cx, cy, cz);
    const R a2 = dfii(dx, dy, dz, bx, by, bz, cx, cy, cz);
    const R a3 = dfii(ax, ay, az, dx, dy, dz, cx, cy, cz);
    const R a4 = dfii(ax, ay, az, bx, by, bz, dx, dy, dz);
    return (R)0.50 * (a1 + a2 + a3 + a4);
  }
  if (eps > e2 && eps < e3) {
    rel(k3, k0, ax, ay, az);
    rel(k3, k1, bx, by, bz);
    rel(k3, k2, cx, cy, cz);
    return dfii(ax, ay, az, bx, by, bz, cx, cy, cz);
  }
  return 0;
}

// getK, src/ParticleUtils.cpp:122-284.
template <typename R>
template <class Draw>
__device__ void FlyerT<R>::point_on_surface(int it, double &en, Draw &&draw, R &xkl, R &ykl, R &zkl) const {
  const R rv1 = (R)1.0 - m_sqrt(draw());
  const R rv2 = draw() * ((R)1.0 - rv1);
  const int4 nd = F.T.tnode[it];
  const V4 *kn = TB::knode(F.T);
  const V4 k0 = kn[nd.x], k1 = kn[nd.y], k2 = kn[nd.z], k3 = kn[nd.w];
  R e = (R)en;
  if ((e < k0.w) || (e > k3.w)) {
    e = k0.w + (k3.w - k0.w) * draw();
    en = e;
  }
  if (e <= k1.w) {
    R r = (e - k0.w) / (k1.w - k0.w);
    const R ax = r * (k1.x - k0.x), ay = r * (k1.y - k0.y), az = r * (k1.z - k0.z);
    r = (e - k0.w) / (k2.w - k0.w);
    const R bx = r * (k2.x - k0.x), by = r * (k2.y - k0.y), bz = r * (k2.z - k0.z);
    r = (e - k0.w) / (k3.w - k0.w);
    const R cx = r * (k3.x - k0.x), cy = r * (k3.y - k0.y), cz = r * (k3.z - k0.z);
    xkl = rv1 * (bx - ax) + rv2 * (cx - ax) + ax + k0.x;
    ykl = rv1 * (by - ay) + rv2 * (cy - ay) + ay + k0.y;
    zkl = rv1 * (bz - az) + rv2 * (cz - az) + az + k0.z;
  } else if (e < k2.w) {
    R r = (e - k0.w) / (k2.w - k0.w);
    const R ax = r * (k2.x - k0.x) + k0.x, ay = r * (k2.y - k0.y) + k0.y, az = r * (k2.z - k0.z) + k0.z;
    r = (e - k1.w) / (k2.w - k1.w);
    const R bx = r * (k2.x - k1.x) + k1.x, by = r * (k2.y - k1.y) + k1.y, bz = r * (k2.z - k1.z) + k1.z;
    r = (e - k0.w) / (k3.w - k0.w);
    const R cx = r * (k3.x - k0.x) + k0.x, cy = r * (k3.y - k0.y) + k0.y, cz = r * (k3.z - k0.z) + k0.z;
    r = (e - k1.w) / (k3.w - k1.w);
    const R dx = r * (k3.x - k1.x) + k1.x, dy = r * (k3.y - k1.y) + k1.y, dz = r * (k3.z - k1.z) + k1.z;
    const R a1 = dfii(ax, ay, az, bx, by, bz, cx, cy, cz);
    const R a2 = dfii(dx, dy, dz, bx, by, bz, cx, cy, cz);
    const R a3 = dfii(ax, ay, az, dx, dy, dz, cx, cy, cz);
    const R a4 = dfii(ax, ay, az, bx, by, bz, dx, dy, dz);
    const R ar = draw() * (a1 + a2 + a3 + a4);
    if (ar < a1) {
      xkl = rv1 * (bx - ax) + rv2 * (cx - ax) + ax;
      ykl = rv1 * (by - ay) + rv2 * (cy - ay) + ay;
      zkl = rv1 * (bz - az) + rv2 * (cz - az) + az;
    } else if (ar < (a1 + a2)) {
      xkl = rv1 * (bx - dx) + rv2 * (cx - dx) + dx;
      ykl = rv1 * (by - dy) + rv2 * (cy - dy) + dy;
      zkl = rv1 * (bz - dz) + rv2 * (cz - dz) + dz;
    } else if (ar < (a1 + a2 + a3)) {
      xkl = rv1 * (dx - ax) + rv2 * (cx - ax) + ax;
      ykl = rv1 * (dy - ay) + rv2 * (cy - ay) + ay;
      zkl = rv1 * (dz - az) + rv2 * (cz - az) + az;
    } else {
      xkl = rv1 * (bx - ax) + rv2 * (dx - ax) + ax;
      ykl = rv1 * (by - ay) + rv2 * (dy - ay) + ay;
      zkl = rv1 * (bz - az) + rv2 * (dz - az) + az;
    }
  } else {
    R r = (e - k3.w) / (k0.w - k3.w);
    const R ax = r * (k0.x - k3.x), ay = r * (k0.y - k3.y), az = r * (k0.z - k3.z);
    r = (e - k3.w) / (k1.w - k3.w);
    const R bx = r * (k1.x - k3.x), by = r * (k1.y - k3.y), bz = r * (k1.z - k3.z);
    r = (e - k3.w) / (k2.w - k3.w);
    const R cx = r * (k2.x - k3.x), cy = r * (k2.y - k3.y), cz = r * (k2.z - k3.z);
    xkl = rv1 * (bx - ax) + rv2 * (cx - ax) + ax + k3.x;
    ykl = rv1 * (by - ay) + rv2 * (cy - ay) + ay + k3.y;
    zkl = rv1 * (bz - az) + rv2 * (cz - az) + az + k3.z;
  }
}

// Interpolation weight of the energy tables (CALSCATTE / CALSCATTH prologue).
template <typename R>
struct TabPosT {
  int mode;  // 0: below table, 1: above, 2: interior
  int itab;
  R intp;
};
using TabPos = TabPosT<double>;
template <typename R>
__device__ __forceinline__ TabPosT<R> tab_pos(const DevTables &T, R eed) {
  TabPosT<R> p;
  const R *E = Tab<R>::energy(T);
  if (eed <= (R)0) { p.mode = 0; p.itab = 0; p.intp = 0; }
  else if (eed >= Tab<R>::k(T).emax) { p.mode = 1; p.itab = kNT - 1; p.intp = 0; }
  else {
    p.mode = 2;
    p.itab = min((int)(eed / Tab<R>::k(T).dtable), kNT - 2);
    p.intp = (eed - E[p.itab]) / (E[p.itab + 1] - E[p.itab]);
  }
  return p;
}
template <typename R>
__device__ __forceinline__ R tab_at(const R *tab, const TabPosT<R> &p) {
  if (p.mode != 2) return tab[p.itab];
  return tab[p.itab] + p.intp * (tab[p.itab + 1] - tab[p.itab]);
}
template <typename R>
__device__ __forceinline__ R tab_at_strided(const R *tab, int stride, const TabPosT<R> &p) {
  if (p.mode != 2) return tab[(size_t)p.itab * stride];
  const R a = tab[(size_t)p.itab * stride], b = tab[(size_t)(p.itab + 1) * stride];
  return a + p.intp * (b - a);
}

// Entry idx of Band::CALSCATTE (src/Band.cpp:2165-2231, electrons) or
// Band::CALSCATTH (:2098-2162, holes) for initial band ini.
template <typename R>
__device__ __forceinline__ R scatter_rate(const DevTables &T, const TabPosT<R> &p, int carrier, int ini, int idx) {
  const int per = carrier == 0 ? T.scpre : T.scprh, nb = carrier == 0 ? 4 : 3;
  const int f = idx / per, is = idx % per;
  const bool ion = is == per - 1;
  const R *tab = carrier == 0 ? (ion ? Tab<R>::scattiie(T) : Tab<R>::dose(T))
                              : (ion ? Tab<R>::scattiih(T) : Tab<R>::dosh(T));
  const R v = tab_at(tab + (size_t)(ion ? f * nb + ini : is * nb + f) * kNT, p);
  if (ion) return v;
  return (carrier == 0 ? Tab<R>::scatte(T) : Tab<R>::scatth(T))[(is * nb + f) * nb + ini] * v;
}

// The final-state draws of a warp's lanes, one owner at a time.
//
// A draw made by its lane alone is a serial chain of dependent loads (the
// mechanism's running sum over up to 56 tabulated rates, then about 11
// rejected tetrahedra) that the warp's other lanes wait for.  Here lane l
// evaluates rates l and l + 32, and, since draw n of a particle's stream is
// a function of n alone, lane l also holds draw first + l and tests the
// tetrahedron that draw would pick; the reference's sequence is then read
// off the lanes' votes, with the same draws used for the same decisions.
template <typename R>
__device__ __forceinline__ void FlyerT<R>::final_states(unsigned owners) {
  const DevTables &T = F.T;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned all = 0xffffffffu;
#pragma unroll 1
  for (; owners; owners &= owners - 1u) {
    const int src = __ffs(owners) - 1;
    const uint32_t o_uid = __shfl_sync(all, uid, src), o_sub = __shfl_sync(all, sub, src);
    const uint32_t o_step = __shfl_sync(all, step_, src);
    const unsigned long long o_seed = __shfl_sync(all, (unsigned long long)I->seed, src);
    // the owner's draws from `at` on; lane l holds draw first + l
    uint32_t at = __shfl_sync(all, n, src), first = at;
    R ahead = (R)0;
    auto look_ahead = [&]() {
      first = at;
      if constexpr (sizeof(R) == 8) ahead = mcb200_uniform(o_seed, o_uid, o_step, o_sub, first + lane);
      else ahead = mcb200_uniform_f32(o_seed, o_uid, o_step, o_sub, first + lane);
    };
    auto draw = [&]() -> R {
      const R v = __shfl_sync(all, ahead, (int)(at - first));
      ++at;
      return v;
    };
    look_ahead();
    const int kind = __shfl_sync(all, draw_kind, src);
    const int carrier = __shfl_sync(all, type, src);
    const double e_old = __shfl_sync(all, energy, src);
    const R q_x = __shfl_sync(all, kx, src), q_y = __shfl_sync(all, ky, src), q_z = __shfl_sync(all, kz, src);
    int ib = __shfl_sync(all, iband, src), is = __shfl_sync(all, isym, src), it = __shfl_sync(all, itet, src);
    double e_new = e_old;
    R o_x = (R)0, o_y = (R)0, o_z = (R)0;
    bool real = true, phonon = false;
    int tal = 1;  // Diffuse: TALIND(1)
    if (kind != kDrawDiffuse) {
      // the mechanism (src/ElectronPhononScatter.cpp:47-63,
      // src/HolePhononScatter.cpp:49-66): the first whose running sum of
      // rates reaches drand, added in the reference's order
      const TabPosT<R> pos = tab_pos(T, (R)e_old);
      const int count = carrier == 0 ? T.scpre * T.nband[0] : T.scprh * T.nband[1];  // at most 14 x 4
      const int ini = ib - T.bandof[carrier == 0 ? 0 : 1];
      R r0 = (R)0, r1 = (R)0;
      if ((int)lane < count) r0 = scatter_rate<R>(T, pos, carrier, ini, (int)lane);
      if ((int)lane + 32 < count) r1 = scatter_rate<R>(T, pos, carrier, ini, (int)lane + 32);
      R drand = __shfl_sync(all, pick_drand, src);
      if (kind == kDrawPickSurface) {
        R sum = (R)0;
        for (int i = 0; i < count; ++i) sum += __shfl_sync(all, i < 32 ? r0 : r1, i & 31);
        drand = draw() * sum;
      }
      int iscat = -1;
      R dscat = (R)0;
#pragma unroll 1
      while (drand > dscat) {
        if (++iscat >= count) {
          iscat = -1;
          break;
        }
        dscat = dscat + __shfl_sync(all, iscat < 32 ? r0 : r1, iscat & 31);
      }
      real = iscat >= 0;
      if (real) {
        const bool quantum = __shfl_sync(all, (int)I->M.quantum, src) != 0;
        phonon = scatter_setup(iscat, carrier, quantum, e_new, ib, tal, draw);
      }
    }
    if (real) {
      if (tal == 0) is = ((int)((R)48 * draw()) % 48);
      else if (tal > 0) {
        const int valley = final_valley(tal, q_x, q_y, q_z, draw);
        is = (int)(draw() * (R)8.0) + 8 * (valley - 1);
      }
      // get_state, src/ParticleUtils.cpp:48-120
      real = false;
      const R e = (R)e_new;
      int nted = 0;
      const int *lst = nullptr;
      if (e_new > 0.0) lst = energy_list(e, ib, nted);
      if (nted > 0) {
        const R most = CALDOSTETMAX(e, ib);
        int tries = 0;
#pragma unroll 1
        for (bool open = true; open;) {
          look_ahead();
          const int mine = lst[list_pick(ahead, nted)];
          const TetShapeT<R> &s = ts(mine);
          const bool holds = (s.e[0] < e) && (s.e[3] > e);
          const R next = __shfl_down_sync(all, ahead, 1);
          const bool kept = holds && !(next * most > FASTSURF(e, mine) / s.vgt);
          const unsigned hold = __ballot_sync(all, holds), keep = __ballot_sync(all, kept);
          // the sequence of tries: one draw for a tetrahedron off the energy,
          // two for one that is tested (the last lane's test needs the next
          // draws: it opens the next round)
          unsigned q = 0;
#pragma unroll 1
          while (q < 31u) {
            ++tries;
            const bool last = tries >= kMaxStateTries;
            if (!last && !((hold >> q) & 1u)) {
              ++q;
              continue;
            }
            q += 2;
            if (last || ((keep >> (q - 2u)) & 1u)) {
              it = __shfl_sync(all, mine, (int)q - 2);
              open = false;
              break;
            }
          }
          at = first + q;
        }
        if constexpr (MCB200_FLIGHT_EVENT_STATS != 0)
          if ((int)lane == src) atomicAdd(&I->Y.counters[kStatStateTries], (unsigned long long)tries);
        real = tries < kMaxStateTries;
        if (real) {
          look_ahead();
          R a, b, c;
          point_on_surface(it, e_new, draw, a, b, c);
          out_wedge(S.sym[is], o_x, o_y, o_z, a, b, c);
        }
      }
    }
    if ((int)lane != src) continue;
    skip_to(at);
    draw_kind = kDrawNone;
    self = !real;
    if (kind != kDrawDiffuse) {
      if (!real) continue;
      kx = o_x; ky = o_y; kz = o_z;
      energy = e_new;
      iband = ib; itet = it; isym = is;
      if (phonon && I->M.heat)
        heat_to_point((e_new - e_old) * fabs(charge), type == 0 ? I->Y.heat_e : I->Y.heat_h);
      continue;
    }
    // Diffuse, src/CellHit.cpp:243-386: the old state again when the new one
    // does not move across the face's axis, mirrored when it moves out
    if (real) energy = e_new;
    const int axis = idir >> 1;
    const V4 w = *reinterpret_cast<const V4 *>(tf(real ? it : itet).v);
    R wx, wy, wz;
    out_wedge(S.sym[real ? is : isym], wx, wy, wz, w.x, w.y, w.z);
    const R across = m_pick3((uint32_t)axis, wx, wy, wz);
    if (real && across != (R)0) {
      kx = o_x; ky = o_y; kz = o_z;
      itet = it; isym = is;
    }
    if ((idir & 1) ? across > (R)0 : across < (R)0) reflect_axis(axis);
  }
}

// EleImpScUpdateK, src/ElectronImpurityScatter.cpp:188-306: Brooks-Herring
// final state in the ellipsoidal-valley picture, accepted by rejection (the
// reference's pow(q, -2.0) as 1 / q^2: half an ulp twice).
template <typename R>
__device__ void FlyerT<R>::EleImpScUpdateK() {
  const FlightConstT<R> &K = TB::k(F.T);
  stock(3);
  const R u0 = Random(), u1 = Random(), u2 = Random();
  R xkl, ykl, zkl;
  in_wedge(xkl, ykl, zkl, kx, ky, kz);
  xkl = xkl - K.shift;
  xkl = xkl * K.in_l;
  ykl = ykl * K.in_t;
  zkl = zkl * K.in_t;
  const R betaq = imp_beta;
  const R eebeta = betaq / K.two_meld;
  const R alfa = eebeta * K.meld / ((R)2.0 * (R)energy * K.melt);
  R pr = u0 / ((R)1.0 + (R)0.5 * alfa);
  const R costr = (R)1.0 - alfa * pr / ((R)1.0 - pr);
  const R sintr = m_sqrt((R)1.0 - costr * costr);
  pr = (R)(2.0 * kPiD) * u1;
  R cospr, sinpr;
  m_sincos(pr, &sinpr, &cospr);
  const R ca = m_sqrt(xkl * xkl + ykl * ykl);
  const R cb = m_sqrt(ca * ca + zkl * zkl);
  const R xkll = cb * sintr * cospr, ykll = cb * sintr * sinpr, zkll = cb * costr;
  const R cosphi = xkl / ca, sinphi = ykl / ca, costheta = zkl / cb, sintheta = ca / cb;
  const R xklll = cosphi * costheta * xkll - sinphi * ykll + cosphi * sintheta * zkll;
  const R yklll = sinphi * costheta * xkll + cosphi * ykll + sinphi * sintheta * zkll;
  const R zklll = -sintheta * xkll + costheta * zkll;
  const R dx = xkl - xklll, dy = ykl - yklll, dz = zkl - zklll;
  const R q = betaq + K.ml * dx * dx + K.mt * (dy * dy + dz * dz);
  const R qmax = betaq + K.mt * dx * dx + K.mt * (dy * dy + dz * dz);
  const R dn = (R)1 / (q * q), dnmax = (R)1 / (qmax * qmax);
  if (dn > u2 * dnmax) {
    xkl = xklll * K.out_l;
    ykl = yklll * K.out_t;
    zkl = zklll * K.out_t;
    xkl = xkl + K.shift;
    out_wedge(kx, ky, kz, xkl, ykl, zkl);
    CONFBZ(kx, ky, kz);
    loc_mode = kLocImpurity;  // Getisym + GetEnergy in run_locate
    self = false;
  } else {
    self = true;
  }
}

template <typename R>
__device__ __forceinline__ bool FlyerT<R>::no_event() const {
  // The margins: the products below are rounded once or twice, the quotients
  // advance() compares once; the clocks' logarithm is the fast one (absolute
  // error below 2^-21 near 1, a few ulp elsewhere) and the impurity majorant
  // and rates are in float, all well inside 2^-16 and 2^-18.
  const R T = (R)left_time;
  const R Ts = T * (R)(sizeof(R) == 4 ? 1.0 + 0x1p-18 : 1.0 + 0x1p-40);
  R xkl, ykl, zkl, xfl, yfl, zfl;
  in_wedge(xkl, ykl, zkl, kx, ky, kz);
  in_wedge(xfl, yfl, zfl, Ex, Ey, Ez);
  const TetFlightT<R> &t = tf(itet);
  bool stays = true;
#pragma unroll
  for (int f = 0; f < 4; ++f) {  // TetTime
    const R nf = t.n[f][0] * xfl + t.n[f][1] * yfl + t.n[f][2] * zfl;
    const R num = t.n[f][3] - (t.n[f][0] * xkl + t.n[f][1] * ykl + t.n[f][2] * zkl);
    stays = stays && (!(nf < 0) || num < nf * Ts);
  }
  const DevMesh &M = I->M;
  auto axis = [&](R v, R up, R down) { return (v > 0 ? up : down) > m_abs(v) * Ts; };  // CellTime
  if constexpr (Real::kCellRelative) {
    stays = stays && axis(vx, M.dxf[ic] - x, x) && axis(vy, M.dyf[jc] - y, y) && axis(vz, M.dzf[kc] - z, z);
  } else {
    stays = stays && axis(vx, M.lx[ic + 1] - x, x - M.lx[ic]) && axis(vy, M.ly[jc + 1] - y, y - M.ly[jc]) &&
            axis(vz, M.lz[kc + 1] - z, z - M.lz[kc]);
  }
  if (!stays) return false;
  // the clocks: draws 0, 1 (, 2) as advance() takes them in its first pass
  const float tf32 = (float)T;
  uint32_t w[4];
  philox_rounds(0u, uid, step_, sub, (uint32_t)I->seed, (uint32_t)(I->seed >> 32), w);
  auto clock = [](float u) { return -__logf(u) * (1.0f - 0x1p-16f) - 0x1p-18f; };
  float u0, u1;
  if constexpr (sizeof(R) == 4) {
    u0 = mcb200_bits_to_unit_f32(w[0]);
    u1 = mcb200_bits_to_unit_f32(w[1]);
  } else {
    u0 = (float)mcb200_bits_to_unit(w[1], w[0]);
    u1 = (float)mcb200_bits_to_unit(w[3], w[2]);
  }
  if (!(clock(u0) > (float)t.gam * tf32)) return false;
  const bool impurities = iband == F.T.bandof[0];
  const int c = cell_index();
  if (impurities) {  // GetImpScGamma
    float rate = 0.0f;
    if constexpr (sizeof(R) == 4) {
      const float e = imp_emax < t.e0 ? t.e0 : (imp_emax > t.e3 ? t.e3 : imp_emax);
      const float d = 1.0f + imp_b * e;
      if (e < imp_ecut) rate = __fdividef(imp_a * sqrtf(e), d);
      if (d > 0x1p126f) return false;  // where the fast quotient is zero: a density next to none
    } else {
      const float e = fminf(fmaxf((float)imp_emax, (float)t.e0), (float)t.e3);
      if (e * (float)F.T.eV0 < 0.120f * (1.0f + 0x1p-16f))
        rate = __fdividef((float)imp_a * sqrtf(2.0f * F.T.k32.meld * e),
                          (float)imp_c * (1.0f + __fdividef(4.0f * e * F.T.k32.melt, (float)imp_b)));
    }
    // (a rate that is no number, from a density no float holds, is an event)
    const float c1 = clock(u1);
    if (!(c1 > rate * tf32 && c1 > (float)TB::k(F.T).gamma_floor * tf32)) return false;
  }
  if (M.surface_scatter && M.in_surf[c]) {
    float u = impurities ? 0.0f : u1;
    if (impurities) {
      if constexpr (sizeof(R) == 4) {
        u = mcb200_bits_to_unit_f32(w[2]);
      } else {
        philox_rounds(1u, uid, step_, sub, (uint32_t)I->seed, (uint32_t)(I->seed >> 32), w);
        u = (float)mcb200_bits_to_unit(w[1], w[0]);
      }
    }
    const float rate = type == 0 ? (float)M.e_rough[c] + (float)M.e_sphon[c] : (float)M.h_rough[c] + (float)M.h_sphon[c];
    if (!(clock(u) > rate * tf32)) return false;
  }
  return true;
}

}  // namespace mcb200
