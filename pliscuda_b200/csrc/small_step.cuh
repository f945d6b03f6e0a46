// small_step.cuh — the leap and the classification of a small model (SmallModel: at most kSmallR
// reactions and kSmallS species, one set of rate constants, tables in the kernel arguments).
//
// Both kernels are bound by instruction issue, not by memory (the counts of a 64^3 lattice are
// 1 MB per species and sit in L2), so this file spends as few instructions per subvolume as it can
// while every floating-point result keeps the bits of the generic phases (engine_kernels.cuh).
// Measured on one B200, Schlogl 64^3 in binary64, against the generic loops over byte tables: the
// leap went from 17.8 M to 11.1 M warp instructions and from 31.6 to 19.8 us a launch, the
// classification from 10.7 M to 5.6 M and from 29.2 to 13.2 us (both cold), the step from 51.3 to
// 27.2 us; 1,000 subvolumes (A/B network) 30.8 to 10.2 us a step (in k_steps); 256 Brusselator
// replicas 2.7 to 1.15 ms a round.
//   * the tables are whole words at compile-time offsets (constant-bank operands: no byte loads);
//     criticality is one compare per reactant species against a threshold made at set-up;
//   * the inversion searches count the CDF terms a uniform exceeds (u > F_0, u > F_1, ...) instead of
//     keeping an open flag, a select and a close test per draw, and they run on uniforms and CDFs
//     both scaled by a power of two (exact), so that a uniform is one subtraction from its word;
//   * a subvolume with all six neighbours takes the six words of its diffusion blocks in place;
//   * neighbour terms divide by the neighbour's own neighbour count with a product and one exact
//     remainder step (div_small) instead of a full division.
// Firings fit 32 bits there (an inversion search stops below 201); the draws with means of
// PLIS_LEAP_INV_MAX and more keep 64-bit counts and guards.
#ifndef PLIS_SMALL_STEP_CUH_
#define PLIS_SMALL_STEP_CUH_

namespace plis {

// a / b for b = 1..6 given y = 1/b rounded to nearest: q = RN(a y), r = a - b q (exact by fma),
// RN(q + r y) (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).  Correctly rounded here: the value added is off by at most 2^-52 ulp of the
// result, while a/b, a multiple of 1/b of an ulp, is never closer than 1/10 ulp to a rounding
// boundary.  Needs a = 0 or a well inside the normal range (SmallModel::on).
__device__ __forceinline__ double div_small(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ float div_small(float a, float b, float y) {
  const float q = a * y;
  return fmaf(fmaf(-b, q, a), y, q);
}

// Uniforms of the inversion searches, and the CDF they are compared with, scaled by 2^32 (binary64:
// w + 1/2, built by planting w in the low bits of 2^52) or 2^23 (binary32: the top 23 bits + 1/2).
template <typename Real> struct Scaled;
template <> struct Scaled<double> {
  static constexpr double scale = 4294967296.0;
  static constexpr int kmax = 200;
  static __device__ __forceinline__ double uniform(uint32_t w) {
    return __hiloint2double(0x43300000, (int)w) - 4503599627370495.5;
  }
  static __device__ __forceinline__ bool top(uint32_t) { return false; }  // no tail test (DiffTraits<double>)
};
template <> struct Scaled<float> {
  static constexpr float scale = 8388608.0f;
  static constexpr int kmax = 100;
  static __device__ __forceinline__ float uniform(uint32_t w) { return (float)(w >> 9) + 0.5f; }
  // The binary32 search also stops where p <= F 2^-25.  That can only happen with F above 1 - 2^-15
  // (the mass beyond is below 2^-24 and the rounding of F below 200 x 2^-24), so a uniform below it
  // has stopped on u <= F before; the words above it take the search with the tail test.
  static __device__ __forceinline__ bool top(uint32_t w) { return w >= 0xFFFE0000u; }
};

// the searches with the tail test for binary32 uniforms next to 1 (about one warp in a hundred)
template <typename Real>
__device__ __noinline__ int search_top(uint32_t w, Real lam) {
  return (int)RT<Real>::inv_word(w, lam);
}

// Up to four draws by inversion, word w[i] and mean lam[i] < PLIS_LEAP_INV_MAX (0: no draw).
template <typename Real>
__device__ __forceinline__ void search4(const uint32_t w[4], const Real lam[4], int k[4]) {
  Real u[4], p[4], F[4];
  bool open[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    u[i] = Scaled<Real>::uniform(w[i]);
    p[i] = RT<Real>::emlam(lam[i]) * Scaled<Real>::scale;
    F[i] = p[i];
    k[i] = 0;
    open[i] = u[i] > F[i];  // lam 0: F = scale, above every uniform
  }
  int ki = 0;
  while (open[0] || open[1] || open[2] || open[3]) {
    const Real ik1 = (Real)plis_inv_k_tab[ki + 1];
    const Real ik2 = (Real)plis_inv_k_tab[ki + 2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      k[i] += open[i] ? 1 : 0;
      p[i] = (p[i] * lam[i]) * ik1;
      F[i] += p[i];
      k[i] += u[i] > F[i] ? 1 : 0;
      p[i] = (p[i] * lam[i]) * ik2;
      F[i] += p[i];
      open[i] = u[i] > F[i];
    }
    ki += 2;
    if (ki >= Scaled<Real>::kmax) break;  // never reached: F has passed every uniform long before
  }
  if (Scaled<Real>::top(w[0]) || Scaled<Real>::top(w[1]) || Scaled<Real>::top(w[2]) || Scaled<Real>::top(w[3])) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (lam[i] > (Real)0) k[i] = search_top<Real>(w[i], lam[i]);
  }
}

// Six draws of one mean 0 < lam < PLIS_LEAP_INV_MAX; draw d only where bit d of `on` is set.
template <typename Real>
__device__ __forceinline__ void search6(const uint32_t w[6], uint32_t on, Real lam, int k[6]) {
  Real u[6];
  uint32_t wm = 0;
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    const bool a = (on >> d) & 1u;
    u[d] = a ? Scaled<Real>::uniform(w[d]) : (Real)0;
    wm = a && w[d] > wm ? w[d] : wm;
    k[d] = 0;
  }
  const Real um = Scaled<Real>::uniform(wm);
  Real p = RT<Real>::emlam(lam) * Scaled<Real>::scale, F = p;
  int ki = 0;
  while (um > F) {
#pragma unroll
    for (int d = 0; d < 6; ++d) k[d] += u[d] > F ? 1 : 0;
    ki += 1;
    if (ki >= Scaled<Real>::kmax) break;  // never reached
    p = (p * lam) * (Real)plis_inv_k_tab[ki];
    F += p;
  }
  if (Scaled<Real>::top(wm)) {
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if ((on >> d) & 1u) k[d] = search_top<Real>(w[d], lam);
  }
}

// Propensities and the critical bits (bit r: some reactant species is below its threshold) of a
// subvolume.  Corrected semantics call a reaction critical only when its propensity is positive;
// every use below adds or tests a propensity that is zero otherwise, so the bit alone serves both.
template <typename Real, int MAXS>
__device__ __forceinline__ uint32_t small_rates(const SmallModel& t, const int32_t x[MAXS], Real a[kSmallR]) {
  uint32_t crit = 0;
  if constexpr (MAXS == 1) {
    const Real f1 = (Real)x[0];
    const Real f2 = f1 * (f1 - (Real)1), f3 = f2 * (f1 - (Real)2);
#pragma unroll
    for (int r = 0; r < kSmallR; ++r) {
      const int m = t.ord[r][0];
      const Real prod = m == 0 ? (Real)1 : m == 1 ? f1 : m == 2 ? f2 : f3;
      a[r] = (sm_rate<Real>(t, r) * prod) * (Real)t.inv_denom[r];
      crit |= x[0] < t.thr[r][0] ? 1u << r : 0u;
    }
  } else {
#pragma unroll
    for (int r = 0; r < kSmallR; ++r) {
      Real prod = (Real)1;
#pragma unroll
      for (int s = 0; s < MAXS; ++s) {
        const int m = t.ord[r][s];
        if (m > 0) {
          const Real xs = (Real)x[s];
          prod = prod * xs;
          if (m > 1) {
            prod = prod * (xs - (Real)1);
            if (m > 2) prod = prod * (xs - (Real)2);
          }
        }
        crit |= x[s] < t.thr[r][s] ? 1u << r : 0u;
      }
      a[r] = (sm_rate<Real>(t, r) * prod) * (Real)t.inv_denom[r];
    }
  }
  return crit;
}

// ------------------------------------------------------------------------------------------------
// leap of one brick (leap_step, leap.cu:3-65)
// ------------------------------------------------------------------------------------------------
// Lattice directions of a subvolume that have a neighbour, bit d of 0..5 = -x,+x,-y,+y,-z,+z.
__device__ __forceinline__ uint32_t lattice_dirs(const DevModel& m, const Cell& cl) {
  return (cl.x > 0 ? 1u : 0u) | (cl.x + 1 < m.X ? 2u : 0u) | (cl.y > 0 ? 4u : 0u) | (cl.y + 1 < m.Y ? 8u : 0u) |
         (cl.z > 0 ? 16u : 0u) | (cl.z + 1 < m.Z ? 32u : 0u);
}

// One subvolume's leap from its counts x and flag f.
// LAT: a lattice (directions by coordinates), else a neighbour table (slot j = direction j).
// RK: group blocks from the round keys in the kernel arguments.
template <typename Real, int MAXS, bool LOG, bool LAT, bool RK>
__device__ __forceinline__ void leap_cell_small(const KArgs& A, const SmallModel& t, const Cell& cl, const int32_t x[MAXS],
                                                uint8_t f, const LeapCtx& L, Real tl, long long& ev_out, int& big) {
  const DevModel& m = A.m;
  const int nc = A.o.nc, mode = A.o.mode;
  const int S = (int)m.S;
  const uint32_t c = cl.c;
  int32_t dl[MAXS];
  long long dbig[MAXS];  // net changes of the draws counted in 64 bits
  bool wide = false;
#pragma unroll
  for (int s = 0; s < MAXS; ++s) {
    dl[s] = 0;
    dbig[s] = 0;
  }
  if (f == F_LEAP_CR || f == F_LEAP_NOCR) {  // leap.cu:9-10
    uint32_t ev = 0;  // at most 6 x 2^27 per species: a jump of 2^27 or more rolls the attempt back
    {
      Real a[kSmallR], lam[4];
      const uint32_t crit = small_rates<Real, MAXS>(t, x, a);
      uint32_t need = 0, large = 0;
#pragma unroll
      for (int r = 0; r < kSmallR; ++r) {
        lam[r] = (crit >> r) & 1u ? (Real)0 : tl * a[r];  // rate constants of reactions >= R are 0
        if (!(lam[r] > (Real)0)) lam[r] = (Real)0;
        else if (lam[r] < (Real)PLIS_LEAP_INV_MAX) need = 1u;
        else large |= 1u << r;
      }
      if (large) {  // PTRS, one inlined sampler
        wide = true;
        for (uint32_t todo = large; todo; todo &= todo - 1u) {
          const int r = __ffs(todo) - 1;
          Real lr = lam[0];
#pragma unroll
          for (int j = 1; j < 4; ++j)
            if (r == j) lr = lam[j];
          plis_stream st = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_react(r));
          const long long k = RT<Real>::count(RT<Real>::poisson(&st, lr));
          ev_out += k;
          if (LOG && k > 0) ev_put(A.b.ev, L.t, L.step, L.attempt, c, c, k, r, PLIS_EVENT_LEAP_REACTION);
#pragma unroll
          for (int s = 0; s < MAXS; ++s) {
            int nu = t.nu[0][s];
#pragma unroll
            for (int j = 1; j < 4; ++j)
              if (r == j) nu = t.nu[j][s];
            const long long v = k * (long long)nu;
            if (v >= kBigDraw || v <= -kBigDraw) big = 1;
            dbig[s] += v;
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if ((large >> r) & 1u) lam[r] = (Real)0;
      }
      if (need) {
        const plis_stream g = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_rgroup(0));
        plis_u32x4 b;
        if constexpr (RK) b = plis_group_block_rk(&g, 0, A.o.rk0, A.o.rk1);
        else b = plis_group_block(&g, 0);
        const uint32_t w[4] = {b.x, b.y, b.z, b.w};
        int k[4];
        search4<Real>(w, lam, k);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          ev += (uint32_t)k[r];
          if (LOG && k[r] > 0) ev_put(A.b.ev, L.t, L.step, L.attempt, c, c, k[r], r, PLIS_EVENT_LEAP_REACTION);
#pragma unroll
          for (int s = 0; s < MAXS; ++s) dl[s] += k[r] * t.nu[r][s];
        }
      }
    }
    uint32_t on;  // directions with a neighbour
    int n;
    uint32_t nb[6];
    if constexpr (LAT) {
      on = lattice_dirs(m, cl);
      n = __popc(on);
      const uint32_t XY = m.X * m.Y;
      nb[0] = c - 1; nb[1] = c + 1; nb[2] = c - m.X; nb[3] = c + m.X; nb[4] = c - XY; nb[5] = c + XY;
    } else {
      n = m.ncount[c];
      on = (1u << n) - 1u;
#pragma unroll
      for (int d = 0; d < 6; ++d) nb[d] = m.canon[(size_t)c * 6 + d];
    }
    bool mark = false;
#pragma unroll
    for (int s = 0; s < MAXS; ++s) {
      if (s >= S || x[s] < nc || n == 0) continue;  // is_critical_diffusion, tau.cu:42-45
      mark = true;
      const Real lam = tl * (sm_drate<Real>(t, s) * (Real)x[s]);
      if (!(lam > (Real)0)) continue;
      int k[6];
      if (lam < (Real)PLIS_LEAP_INV_MAX) {
        const plis_stream g = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_dgroup(s));
        uint32_t w[6];
        {
          plis_u32x4 b;
          if constexpr (RK) b = plis_group_block_rk(&g, 0, A.o.rk0, A.o.rk1);
          else b = plis_group_block(&g, 0);
          w[0] = b.x; w[1] = b.y; w[2] = b.z; w[3] = b.w;
          if constexpr (RK) b = plis_group_block_rk(&g, 1, A.o.rk0, A.o.rk1);
          else b = plis_group_block(&g, 1);
          w[4] = b.x; w[5] = b.y;
        }
        if (LAT && on != 63u) {  // slot j belongs to the j-th present direction
#pragma unroll
          for (int d = 0; d < 5; ++d)
            if (!((on >> d) & 1u)) {
#pragma unroll
              for (int e = 5; e > d; --e) w[e] = w[e - 1];
            }
        }
        search6<Real>(w, on, lam, k);
      } else {
#pragma unroll
        for (int d = 0; d < 6; ++d) k[d] = 0;
        int j = 0;
#pragma unroll 1
        for (int d = 0; d < 6; ++d) {  // one inlined PTRS for the slots
          if (!((on >> d) & 1u)) continue;
          plis_stream st = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_diff(s, j));
          ++j;
          const long long kj = plis_count_d(plis_poisson_d(&st, (double)lam));
          const int v = (int)(kj < kBigJump ? kj : kBigJump);  // a jump of 2^27 or more rolls the attempt back
          if (v >= kBigJump) big = 1;
#pragma unroll
          for (int e = 0; e < 6; ++e)
            if (e == d) k[e] = v;
        }
      }
      int32_t* row = L.Xt + (size_t)s * m.Npad;
      int out = 0;
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if (k[d] > 0) {
          atomicAdd(&row[nb[d]], k[d]);
          if (LOG) ev_put(A.b.ev, L.t, L.step, L.attempt, c, nb[d], k[d], s, PLIS_EVENT_LEAP_DIFFUSION);
        }
        out += k[d];
      }
      if (mode == 1 && !L.ff_free) {
#pragma unroll
        for (int d = 0; d < 6; ++d)
          if (k[d] > 0 && L.flag[nb[d]] == F_SSA_FF) L.flag[nb[d]] = F_SSA;
      }
      dl[s] -= out;
      ev += (uint32_t)out;
    }
    if (mode == 0 && mark && !L.ff_free) {  // leap.cu:54-56: every receiver leaves fast-forward
#pragma unroll
      for (int d = 0; d < 6; ++d)
        if (((on >> d) & 1u) && L.flag[nb[d]] == F_SSA_FF) L.flag[nb[d]] = F_SSA;
    }
    ev_out += ev;
  }
#pragma unroll
  for (int s = 0; s < MAXS; ++s) {
    if (s >= S) continue;
    // |dl| <= 6 x 2^27 + 4 x 200 x 127 and 0 <= x < 2^30: no 32-bit sum wraps below 2^31
    long long tv = (long long)x[s] + dl[s];
    if (wide) tv += dbig[s];
    if (tv >= kBigTile || tv <= -kBigTile) big = 1;
    atomicAdd(&L.Xt[(size_t)s * m.Npad + c], (int)tv);
  }
}

template <typename Real, int MAXS, bool LOG, bool LAT, bool RK>
__device__ __forceinline__ void leap_tile_small(const KArgs& A, const SmallModel& t, uint32_t tile, const LeapCtx& L,
                                                Real tl, long long& ev_out, int& big) {
  const DevModel& m = A.m;
  ev_out = 0;
  big = 0;
  Cell cl;
  if (!cell_of(A, tile, cl)) return;
  const uint8_t f = L.flag[cl.c];
  int32_t x[MAXS];
#pragma unroll
  for (int s = 0; s < MAXS; ++s) x[s] = s < (int)m.S ? L.Xc[(size_t)s * m.Npad + cl.c] : 0;
  leap_cell_small<Real, MAXS, LOG, LAT, RK>(A, t, cl, x, f, L, tl, ev_out, big);
}

// ------------------------------------------------------------------------------------------------
// classification of one subvolume (compute_taus, tau.cu:68-195): cell_tau_parts for a small model
// ------------------------------------------------------------------------------------------------
template <typename Real, int MAXS, bool LAT>
__device__ __forceinline__ void small_tau_parts(const KArgs& A, const SmallModel& t, const Cell& cl, const int32_t x[MAXS],
                                                const int32_t* Xe, Real& tau_ncr_out, Real& rate_cr_out) {
  const DevModel& m = A.m;
  const int mode = A.o.mode, nc = A.o.nc;
  const int S = (int)m.S;
  const uint32_t c = cl.c;
  uint32_t on, nb[6];
  int nn[6];  // the neighbours' own neighbour counts (reference semantics)
  int n;
  bool deep = false;  // all six neighbours, each with six
  if constexpr (LAT) {
    const uint32_t X = m.X, Y = m.Y, Z = m.Z, XY = X * Y;
    on = lattice_dirs(m, cl);
    n = __popc(on);
    nb[0] = c - 1; nb[1] = c + 1; nb[2] = c - X; nb[3] = c + X; nb[4] = c - XY; nb[5] = c + XY;
    deep = cl.x > 1 && cl.x + 2 < X && cl.y > 1 && cl.y + 2 < Y && cl.z > 1 && cl.z + 2 < Z;
    // along its own axis a neighbour lacks the far side only when it is the first or the last there
    nn[0] = n - (int)((on >> 1) & 1u) + 1 - (cl.x > 1 ? 0 : 1);
    nn[1] = n - (int)(on & 1u) + 1 - (cl.x + 2 < X ? 0 : 1);
    nn[2] = n - (int)((on >> 3) & 1u) + 1 - (cl.y > 1 ? 0 : 1);
    nn[3] = n - (int)((on >> 2) & 1u) + 1 - (cl.y + 2 < Y ? 0 : 1);
    nn[4] = n - (int)((on >> 5) & 1u) + 1 - (cl.z > 1 ? 0 : 1);
    nn[5] = n - (int)((on >> 4) & 1u) + 1 - (cl.z + 2 < Z ? 0 : 1);
  } else {
    n = m.ncount[c];
    on = (1u << n) - 1u;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      nb[d] = m.canon[(size_t)c * 6 + d];
      nn[d] = (on >> d) & 1u ? (int)m.ncount[nb[d]] : 1;
    }
  }
  Real a[kSmallR];
  const uint32_t crit = small_rates<Real, MAXS>(t, x, a);
  uint32_t pos = 0;
  if (mode != 0) {
#pragma unroll
    for (int r = 0; r < kSmallR; ++r) pos |= a[r] > (Real)0 ? 1u << r : 0u;
  }
  Real tau_ncr = RT<Real>::inf();
#pragma unroll
  for (int s = 0; s < MAXS; ++s) {
    if (s >= S) continue;
    const int32_t xs = x[s];
    const Real dr = sm_drate<Real>(t, s);
    bool include;
    if (mode == 0) include = !((crit & t.rmask[s]) != 0u && xs < nc);  // tau.cu:165
    else include = (pos & ~crit & t.rmask[s]) != 0u || (xs >= nc && dr > (Real)0 && n > 0);
    if (!include) continue;
    int32_t xb[6];
    const int32_t* row = Xe + (size_t)s * m.Npad;
#pragma unroll
    for (int d = 0; d < 6; ++d) xb[d] = (on >> d) & 1u ? row[nb[d]] : 0;
    const Real g = gfun<Real>(t.hor[s], t.hmult[s], (Real)xs);
    Real mu = (Real)0, s2 = (Real)0;
#pragma unroll
    for (int r = 0; r < kSmallR; ++r) {
      const int nu = t.nu[r][s];  // 0 for reactions >= R
      if (nu == 0) continue;
      if ((crit >> r) & 1u) continue;
      mu = mu + (Real)nu * a[r];
      s2 = s2 + (Real)(nu * nu) * a[r];
    }
    const Real d0 = dr * (Real)xs;
    if (mode == 0) {
      if (xs >= nc) { mu = mu + d0; s2 = s2 + d0; }
      if (deep) {
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          const Real q = div_small(dr * (Real)xb[d], (Real)6, (Real)(1.0 / 6.0));
          mu = mu - q;
          s2 = s2 + q;
        }
      } else {
#pragma unroll
        for (int d = 0; d < 6; ++d) {  // an absent direction has count 0: q = 0 leaves mu and s2
          const Real q = div_small(dr * (Real)xb[d], (Real)nn[d], (Real)plis_inv_k_tab[nn[d]]);
          mu = mu - q;
          s2 = s2 + q;
        }
      }
    } else {
      if (xs >= nc && n > 0) {
        const Real dout = (Real)n * d0;
        mu = mu - dout;
        s2 = s2 + dout;
      }
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if (xb[d] >= nc && ((on >> d) & 1u)) {
          const Real q = dr * (Real)xb[d];
          mu = mu + q;
          s2 = s2 + q;
        }
      }
    }
    Real mm = ((Real)A.o.eps * (Real)xs) / g;
    if (!(mm > (Real)1)) mm = (Real)1;
    const Real t1 = mm / fabs(mu);
    const Real t2 = (mm * mm) / s2;
    const Real ts = t1 < t2 ? t1 : t2;
    if (ts < tau_ncr) tau_ncr = ts;
  }
  // critical (or, corrected SSA subvolume: total) rate, compute_tau_cr tau.cu:176-195
  Real rsum = (Real)0, dsum = (Real)0;
  if (mode == 0 || !plis_isinf_d((double)tau_ncr)) {
    if (crit) {
#pragma unroll
      for (int r = 0; r < kSmallR; ++r)
        if ((crit >> r) & 1u) rsum = rsum + a[r];
    }
#pragma unroll
    for (int s = 0; s < MAXS; ++s) {
      if (s >= S) continue;
      if (x[s] < nc) {
        const Real d = sm_drate<Real>(t, s) * (Real)x[s];
        dsum = dsum + (mode == 0 ? d : (Real)n * d);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < kSmallR; ++r) rsum = rsum + a[r];
#pragma unroll
    for (int s = 0; s < MAXS; ++s)
      if (s < S) dsum = dsum + (Real)n * (sm_drate<Real>(t, s) * (Real)x[s]);
  }
  tau_ncr_out = tau_ncr;
  rate_cr_out = (rsum == (Real)0 && dsum == (Real)0) ? (Real)0 : rsum + dsum;
}

}  // namespace plis

#endif
