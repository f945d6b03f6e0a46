// net_step.cuh — the leap, the critical events and the classification of a network that is too large
// for the small-model kernels (or has several sets of rate constants, or draws pooled) but fits NetTab:
// at most kNetR reactions and kNetS species.
//
// These phases are bound by instruction issue and by the latency of what a thread looks up.  The
// generic phases (engine_kernels.cuh) read byte and word tables from global memory for every value,
// keep counts indexed by species in local memory and evaluate a propensity wherever they need it.  Here
//   * the tables are words in the kernel arguments (NetTab), read through the constant bank with an
//     index that is the same in every lane;
//   * a thread keeps its counts, already converted to the working precision, its propensities and its
//     net changes in its own column of shared memory (no bank conflicts: lanes are adjacent);
//   * every propensity is evaluated once, with the criticality of its reaction as one bit;
//   * neighbour terms divide with div_small, searches count as in small_step.cuh.
// Every floating-point value is formed by the same operations in the same order as in the generic
// phases, which larger networks keep.
// Measured on one B200 against the generic phases (us a step): 10 species and 20 reactions on 128^3 in
// binary64 2130 -> 826 (leap 767 -> 331, exact events 168 -> 62, classification 1053 -> 417), on
// 64^3 in binary32 279 -> 121; a cell of 9,300 subvolumes as a table with two compartments 71.6 -> 27.4
// (there in the persistent kernel, k_steps).
#ifndef PLIS_NET_STEP_CUH_
#define PLIS_NET_STEP_CUH_

namespace plis {

template <typename Real> __device__ __forceinline__ const NetTab<Real>& net_tab(const NetArgs& A);
template <> __device__ __forceinline__ const NetTab<double>& net_tab<double>(const NetArgs& A) { return A.net.d; }
template <> __device__ __forceinline__ const NetTab<float>& net_tab<float>(const NetArgs& A) { return A.net.f; }

// shared memory of one CTA, rows of kNetCols: S rows of counts, R of propensities, and for the leap S
// of net changes
template <typename Real>
constexpr size_t net_smem(uint32_t S, uint32_t R, bool leap) {
  return (size_t)kNetCols * (sizeof(Real) * (S + R) + (leap ? sizeof(int32_t) * S : 0u));
}

// One thread's column: byte offsets of the tables, or row numbers, from its first row.
template <typename T> struct Column {
  unsigned char* p;
  __device__ __forceinline__ T& at(uint32_t off) const { return *reinterpret_cast<T*>(p + off); }
  __device__ __forceinline__ T& operator[](int row) const { return at((uint32_t)row * (kNetCols * (uint32_t)sizeof(T))); }
};
template <typename T>
__device__ __forceinline__ Column<T> column(unsigned char* base, size_t row_bytes) {
  return Column<T>{base + row_bytes * kNetCols + threadIdx.x * sizeof(T)};
}

// f(s, count) for every species of subvolume c, the counts of five species loaded together: what f
// stores may alias the counts for all the compiler knows, so loads between stores would wait one by one.
template <class F>
__device__ __forceinline__ void net_rows(const DevModel& m, const int32_t* X, uint32_t c, int S, F&& f) {
  for (int s0 = 0; s0 < S; s0 += 5) {
    int32_t v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = s0 + i < S ? X[(size_t)(s0 + i) * m.Npad + c] : 0;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (s0 + i < S) f(s0 + i, v[i]);
  }
}

template <typename Real, bool COMP>
__device__ __forceinline__ Real net_drate(const NetTab<Real>& T, const DevModel& m, uint32_t comp, int s) {
  if constexpr (COMP) return __ldg((const Real*)m.dr + (size_t)comp * m.S + s);
  else return T.drate[s];
}

// Propensity of reaction r from the counts (prop()), and whether a reactant species is below its
// threshold (crit_ref(); crit_fix() but for its test that the propensity is positive, see small_rates).
template <typename Real, bool COMP>
__device__ __forceinline__ Real net_prop(const NetTab<Real>& T, const DevModel& m, uint32_t comp, Column<Real> sx, int r,
                                         bool& crit) {
  const uint32_t nf = T.nf[r];
  Real prod = (Real)1;
  bool cr = false;
  if (nf > 0) {
    const Real x0 = sx.at(T.fac[r][0].off);
    cr = x0 < T.fac[r][0].thr;
    prod = x0;  // the first factor has j = 0
    if (nf > 1) {
      const Real x1 = sx.at(T.fac[r][1].off);
      cr = cr || x1 < T.fac[r][1].thr;
      prod = prod * (x1 - T.fac[r][1].j);
      if (nf > 2) {
        const Real x2 = sx.at(T.fac[r][2].off);
        cr = cr || x2 < T.fac[r][2].thr;
        prod = prod * (x2 - T.fac[r][2].j);
      }
    }
  }
  crit = cr;
  Real rate;
  if constexpr (COMP) rate = __ldg((const Real*)m.rr + (size_t)comp * m.R + r);
  else rate = T.rate[r];
  return (rate * prod) * T.inv_denom[r];
}

// one draw by inversion (search4 for a single draw)
template <typename Real>
__device__ __forceinline__ int search1(uint32_t w, Real lam) {
  if (Scaled<Real>::top(w)) return search_top<Real>(w, lam);
  const Real u = Scaled<Real>::uniform(w);
  Real p = RT<Real>::emlam(lam) * Scaled<Real>::scale, F = p;
  int k = 0;
  while (u > F && k < Scaled<Real>::kmax) {
    ++k;
    p = (p * lam) * (Real)plis_inv_k_tab[k];
    F += p;
  }
  return k;
}

// The neighbours of a subvolume by direction (lattice) or slot (table).
struct Dirs {
  uint32_t on;     // bit d: there is a neighbour in direction (slot) d
  int n;
  uint32_t nb[6];
};
template <bool LAT>
__device__ __forceinline__ void net_dirs(const DevModel& m, const Cell& cl, Dirs& q) {
  const uint32_t c = cl.c;
  if constexpr (LAT) {
    const uint32_t XY = m.X * m.Y;
    q.on = lattice_dirs(m, cl);
    q.n = __popc(q.on);
    q.nb[0] = c - 1; q.nb[1] = c + 1; q.nb[2] = c - m.X; q.nb[3] = c + m.X; q.nb[4] = c - XY; q.nb[5] = c + XY;
  } else {
    q.n = m.ncount[c];
    q.on = (1u << q.n) - 1u;
#pragma unroll
    for (int d = 0; d < 6; ++d) q.nb[d] = m.canon[(size_t)c * 6 + d];
  }
}

// ------------------------------------------------------------------------------------------------
// leap of one brick (leap_step, leap.cu:3-65), pooled or not
// ------------------------------------------------------------------------------------------------
// One subvolume's leap.  fresh: the rows still hold the counts and, 0 for critical reactions, the
// propensities that its classification put there; else they are read and formed here.
template <typename Real, bool LOG, bool LAT, bool COMP>
__device__ __forceinline__ void leap_cell_net(const KArgs& A, const NetTab<Real>& T, const Cell& cl, uint8_t f, bool fresh,
                                              const LeapCtx& L, Real tl, unsigned char* smem, long long& ev_out, int& big) {
  const DevModel& m = A.m;
  const int nc = A.o.nc, mode = A.o.mode;
  const int S = (int)m.S, R = (int)m.R;
  const uint32_t c = cl.c;
  const Column<Real> sx = column<Real>(smem, 0);                                       // [S] counts
  const Column<Real> sl = column<Real>(smem, sizeof(Real) * (size_t)S);                // [R] means of the firing reactions
  const Column<int32_t> sd = column<int32_t>(smem, sizeof(Real) * (size_t)(S + R));    // [S] net changes
  if (!(f == F_LEAP_CR || f == F_LEAP_NOCR)) {  // leap.cu:9-10
    net_rows(m, L.Xc, c, S, [&](int s, int32_t xs) {
      if (xs >= kBigTile) big = 1;
      atomicAdd(&L.Xt[(size_t)s * m.Npad + c], xs);
    });
    return;
  }
  if (!fresh) net_rows(m, L.Xc, c, S, [&](int s, int32_t xs) { sx[s] = (Real)xs; });
  for (int s = 0; s < S; ++s) sd[s] = 0;
  // Net changes of 2^24 and more go to 64-bit sums in local memory; the others, at most one per
  // reaction and species and one of jumps, stay below 2^30 in the 32-bit column.
  long long wide[kNetS];
  bool has_wide = false;
  auto add = [&](int s, long long v) {
    if (v < (1 << 24) && v > -(1 << 24)) {
      sd[s] += (int32_t)v;
    } else {
      if (!has_wide) {
        for (int i = 0; i < kNetS; ++i) wide[i] = 0;
        has_wide = true;
      }
      wide[s] += v;
    }
  };
  const uint32_t comp = COMP ? (uint32_t)m.comp[c] : 0u;
  const bool pool_on = A.o.pool != 0;
  Real pool = (Real)0;
  uint32_t pool_r = 0, pool_s = 0;  // members of the pool
  auto pool_join = [&](Real unit, Real w) -> bool {
    if (!pool_on || !(unit < (Real)PLIS_POOL_CUT) || !(pool + w <= (Real)PLIS_POOL_MAX)) return false;
    pool = pool + w;
    return true;
  };
  auto fired = [&](int r, long long k) {
    ev_out += k;
    if (LOG) ev_put(A.b.ev, L.t, L.step, L.attempt, c, c, k, r, PLIS_EVENT_LEAP_REACTION);
    for (uint32_t e = T.net_off[r]; e < T.net_off[r + 1]; ++e) {
      const long long v = k * (long long)T.net_nu[e];
      if (v >= kBigDraw || v <= -kBigDraw) big = 1;
      add((int)T.net_s[e], v);
    }
  };
  for (int r0 = 0; r0 < R; r0 += 4) {
    Real lam[4];
    uint32_t need = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + i;
      lam[i] = (Real)0;
      if (r < R) {
        bool crit = false;
        const Real a = fresh ? sl[r] : net_prop<Real, COMP>(T, m, comp, sx, r, crit);
        Real lr = crit ? (Real)0 : tl * a;
        if (!(lr > (Real)0)) lr = (Real)0;
        sl[r] = lr;
        if (lr > (Real)0) {
          if (pool_join(lr, lr)) pool_r |= 1u << r;
          else {
            lam[i] = lr;
            need |= lr < (Real)PLIS_LEAP_INV_MAX ? 1u << i : 16u << i;
          }
        }
      }
    }
    for (uint32_t todo = need >> 4; todo; todo &= todo - 1u) {  // PTRS, one inlined sampler
      const int i = __ffs(todo) - 1;
      Real li = lam[0];
#pragma unroll
      for (int j = 1; j < 4; ++j)
        if (i == j) li = lam[j];
      plis_stream st = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_react(r0 + i));
      const long long k = RT<Real>::count(RT<Real>::poisson(&st, li));
      if (k > 0) fired(r0 + i, k);
    }
    if (need & 15u) {  // few of a network's channels are drawn on their own: one search at a time
      const plis_stream g =
          plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_rgroup((uint32_t)r0 >> 2));
      const plis_u32x4 b = plis_group_block_rk(&g, 0, A.o.rk0, A.o.rk1);
      for (uint32_t todo = need & 15u; todo; todo &= todo - 1u) {
        const int i = __ffs(todo) - 1;
        const Real li = i == 0 ? lam[0] : i == 1 ? lam[1] : i == 2 ? lam[2] : lam[3];
        const int k = search1<Real>(i == 0 ? b.x : i == 1 ? b.y : i == 2 ? b.z : b.w, li);
        if (k) fired(r0 + i, k);
      }
    }
  }
  Dirs q;
  net_dirs<LAT>(m, cl, q);
  const int n = q.n;
  bool mark = false;
  auto jumps = [&](int s, int k, uint32_t b) {  // k > 0 molecules of species s to subvolume b
    atomicAdd(&L.Xt[(size_t)s * m.Npad + b], k);
    if (mode == 1 && !L.ff_free && L.flag[b] == F_SSA_FF) L.flag[b] = F_SSA;
    if (LOG) ev_put(A.b.ev, L.t, L.step, L.attempt, c, b, k, s, PLIS_EVENT_LEAP_DIFFUSION);
  };
  for (int s = 0; s < S; ++s) {
    const Real xs = sx[s];
    if (xs < (Real)nc || n == 0) continue;  // is_critical_diffusion, tau.cu:42-45
    mark = true;
    const Real lam = tl * (net_drate<Real, COMP>(T, m, comp, s) * xs);
    if (!(lam > (Real)0)) continue;
    if (pool_join(lam, (Real)n * lam)) {
      pool_s |= 1u << s;
      continue;
    }
    int k[6];
    if (lam < (Real)PLIS_LEAP_INV_MAX) {
      const plis_stream g = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, plis_ch_dgroup(s));
      uint32_t w[6];
      {
        plis_u32x4 b = plis_group_block_rk(&g, 0, A.o.rk0, A.o.rk1);
        w[0] = b.x; w[1] = b.y; w[2] = b.z; w[3] = b.w;
        b = plis_group_block_rk(&g, 1, A.o.rk0, A.o.rk1);
        w[4] = b.x; w[5] = b.y;
      }
      if (LAT && q.on != 63u) {  // slot j belongs to the j-th present direction
#pragma unroll
        for (int d = 0; d < 5; ++d)
          if (!((q.on >> d) & 1u)) {
#pragma unroll
            for (int e = 5; e > d; --e) w[e] = w[e - 1];
          }
      }
      search6<Real>(w, q.on, lam, k);
    } else {
#pragma unroll
      for (int d = 0; d < 6; ++d) k[d] = 0;
      int j = 0;
#pragma unroll 1
      for (int d = 0; d < 6; ++d) {  // one inlined PTRS for the slots
        if (!((q.on >> d) & 1u)) continue;
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
    int out = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      if (k[d] > 0) jumps(s, k[d], q.nb[d]);
      out += k[d];
    }
    if (out) {
      add(s, -(long long)out);
      ev_out += out;
    }
  }
  if (pool > (Real)0) {  // the pool's events: total by inversion, then one walk over its members per event
    const plis_stream g = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_LEAP, L.step, L.attempt, PLIS_CH_POOL);
    const uint32_t w0 = plis_group_block_rk(&g, 0, A.o.rk0, A.o.rk1).x;
    // e^-pool >= 1 - pool > u leaves no event without the exponential (2^-20 covers every rounding)
    long long K = 0;
    if (!(RT<Real>::word_uniform(w0) < (Real)1 - pool - (Real)9.5367431640625e-07))
      K = RT<Real>::count(RT<Real>::inv_word(w0, pool));
    for (long long e = 0; e < K; ++e) {
      const plis_u32x4 w = plis_group_block_rk(&g, (uint32_t)(e + 1), A.o.rk0, A.o.rk1);
      const Real target = RT<Real>::word_uniform(w.x) * pool;
      Real acc = (Real)0;
      int pick_r = -1, pick_s = -1, last = -1;
      for (uint32_t todo = pool_r; todo && pick_r < 0; todo &= todo - 1u) {
        last = __ffs(todo) - 1;
        acc = acc + sl[last];
        if (target < acc) pick_r = last;
      }
      if (pick_r < 0) {
        for (uint32_t todo = pool_s; todo && pick_s < 0; todo &= todo - 1u) {
          const int s = __ffs(todo) - 1;
          acc = acc + (Real)n * (tl * (net_drate<Real, COMP>(T, m, comp, s) * sx[s]));
          if (target < acc) pick_s = s;
        }
        if (pick_s < 0) {  // rounding left the target at the total: the last member
          if (pool_s) pick_s = 31 - __clz(pool_s);
          else pick_r = last;
        }
      }
      if (pick_r >= 0) {
        fired(pick_r, 1);
      } else {
        int j = (int)plis_pool_slot(w.y, (uint32_t)n);
        if constexpr (LAT) j = __fns(q.on, 0, j + 1);  // the j-th present direction
        uint32_t b = q.nb[0];
#pragma unroll
        for (int d = 1; d < 6; ++d)
          if (d == j) b = q.nb[d];
        ev_out += 1;
        jumps(pick_s, 1, b);
        sd[pick_s] -= 1;
      }
    }
  }
  if (mode == 0 && mark && !L.ff_free) {  // leap.cu:54-56: every receiver leaves fast-forward
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if (((q.on >> d) & 1u) && L.flag[q.nb[d]] == F_SSA_FF) L.flag[q.nb[d]] = F_SSA;
  }
  net_rows(m, L.Xc, c, S, [&](int s, int32_t xs) {
    long long tv = (long long)xs + sd[s];
    if (has_wide) tv += wide[s];
    if (tv >= kBigTile || tv <= -kBigTile) big = 1;
    atomicAdd(&L.Xt[(size_t)s * m.Npad + c], (int)tv);
  });
}

template <typename Real, bool LOG, bool LAT, bool COMP>
__device__ __forceinline__ void leap_tile_net(const KArgs& A, const NetTab<Real>& T, uint32_t tile, const LeapCtx& L,
                                              Real tl, unsigned char* smem, long long& ev_out, int& big) {
  ev_out = 0;
  big = 0;
  Cell cl;
  if (!cell_of(A, tile, cl)) return;
  leap_cell_net<Real, LOG, LAT, COMP>(A, T, cl, L.flag[cl.c], false, L, tl, smem, ev_out, big);
}

// ------------------------------------------------------------------------------------------------
// classification of one subvolume (compute_taus, tau.cu:68-195): cell_tau_parts
// ------------------------------------------------------------------------------------------------
// The leap bound of one species from its drift mu and spread s2 (tau.cu:127-143).
template <typename Real>
__device__ __forceinline__ Real net_tau_species(const KArgs& A, int hor, int hmult, Real xs, Real mu, Real s2) {
  Real mm = ((Real)A.o.eps * xs) / gfun<Real>(hor, hmult, xs);
  if (!(mm > (Real)1)) mm = (Real)1;
  const Real t1 = mm / fabs(mu);
  const Real t2 = (mm * mm) / s2;
  return t1 < t2 ? t1 : t2;
}
// The same to about 1e-6 in binary32 (0, inf or NaN outside its range).
template <typename Real>
__device__ __forceinline__ float net_tau_near(float eps, int hor, int hmult, Real xs, Real mu, Real s2) {
  const float x = (float)xs;
  float mm = eps * x;
  if (hor != 1) {
    float g;
    if (hor == 0) g = __int_as_float(0x7f800000);
    else if (hmult == 1) g = hor == 2 ? 2.f : 3.f;
    else {
      const float i1 = __fdividef(1.f, x - 1.f);
      g = hor == 2 ? 2.f + i1 : hmult == 2 ? 1.5f * (2.f + i1) : 3.f + i1 + __fdividef(2.f, x - 2.f);
    }
    mm = __fdividef(mm, g);
  }
  mm = fmaxf(mm, 1.f);
  return fminf(__fdividef(mm, fabsf((float)mu)), __fdividef(mm * mm, (float)s2));
}

template <typename Real, bool LAT, bool COMP>
__device__ __forceinline__ void net_tau_parts(const KArgs& A, const NetTab<Real>& T, const Cell& cl, Column<Real> sx,
                                              Column<Real> sa, const int32_t* Xe, Real& tau_ncr_out, Real& rate_cr_out) {
  const DevModel& m = A.m;
  const int mode = A.o.mode, nc = A.o.nc;
  const int S = (int)m.S, R = (int)m.R;
  Dirs q;
  net_dirs<LAT>(m, cl, q);
  const int n = q.n;
  uint32_t nn = 0;     // the neighbours' own neighbour counts, 4 bits each (reference semantics)
  uint32_t ncomp = 0;  // their compartments, 5 bits each
  bool deep = false;   // all six neighbours, each with six
  if constexpr (LAT) {
    const uint32_t on = q.on;
    deep = cl.x > 1 && cl.x + 2 < m.X && cl.y > 1 && cl.y + 2 < m.Y && cl.z > 1 && cl.z + 2 < m.Z;
    nn = (uint32_t)(n - (int)((on >> 1) & 1u) + (cl.x > 1)) | (uint32_t)(n - (int)(on & 1u) + (cl.x + 2 < m.X)) << 4 |
         (uint32_t)(n - (int)((on >> 3) & 1u) + (cl.y > 1)) << 8 | (uint32_t)(n - (int)((on >> 2) & 1u) + (cl.y + 2 < m.Y)) << 12 |
         (uint32_t)(n - (int)((on >> 5) & 1u) + (cl.z > 1)) << 16 | (uint32_t)(n - (int)((on >> 4) & 1u) + (cl.z + 2 < m.Z)) << 20;
  } else {
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if ((q.on >> d) & 1u) nn |= (uint32_t)m.ncount[q.nb[d]] << (4 * d);
  }
  const uint32_t comp = COMP ? (uint32_t)m.comp[cl.c] : 0u;
  if constexpr (COMP) {
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if ((q.on >> d) & 1u) ncomp |= (uint32_t)m.comp[q.nb[d]] << (5 * d);
  }
  // the rows keep the propensities of the non-critical reactions, 0 for the others: a critical reaction
  // then adds nothing to mu and s2, as if left out
  uint32_t critm = 0, posm = 0;
  Real rcrit = (Real)0, rall = (Real)0;
#pragma unroll 2
  for (int r = 0; r < R; ++r) {
    bool crit;
    const Real a = net_prop<Real, COMP>(T, m, comp, sx, r, crit);
    sa[r] = crit ? (Real)0 : a;
    if (crit) {
      critm |= 1u << r;
      rcrit = rcrit + a;
    } else if (a > (Real)0) {
      posm |= 1u << r;
    }
    if (mode != 0) rall = rall + a;
  }
  // The bound is a min over species.  Each species' bound is first formed in binary32; only the
  // smallest, and any within 1e-4 of it or outside binary32's range, is then computed in full.
  Real tau_ncr = RT<Real>::inf();
  const float eps = (float)A.o.eps;
  float near_ = __int_as_float(0x7f800000);
  Real b_mu = (Real)0, b_s2 = (Real)0;
  int b_s = -1;
#pragma unroll 1
  for (int s = 0; s < S; ++s) {
    const Real xs = sx[s];
    const Real dr = net_drate<Real, COMP>(T, m, comp, s);
    const uint32_t rmask = T.rmask[s];
    const bool leaps = !(xs < (Real)nc);
    bool include;
    if (mode == 0) include = (critm & rmask) == 0u || leaps;  // tau.cu:165
    else include = (posm & rmask) != 0u || (leaps && dr > (Real)0 && n > 0);
    if (!include) continue;
    int32_t xb[6];
    const int32_t* row = Xe + (size_t)s * m.Npad;
#pragma unroll
    for (int d = 0; d < 6; ++d) xb[d] = (q.on >> d) & 1u ? row[q.nb[d]] : 0;
    Real mu = (Real)0, s2 = (Real)0;
    const uint32_t e1 = T.sp_off[s + 1];
#pragma unroll 2
    for (uint32_t e = T.sp_off[s]; e < e1; ++e) {
      const Real a = sa.at(T.sp[e].off);
      mu = mu + T.sp[e].nu * a;
      s2 = s2 + T.sp[e].nu2 * a;
    }
    const Real d0 = dr * xs;
    if (mode == 0) {
      if (leaps) { mu = mu + d0; s2 = s2 + d0; }
      if (deep && !COMP) {
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          const Real v = div_small(dr * (Real)xb[d], (Real)6, (Real)(1.0 / 6.0));
          mu = mu - v;
          s2 = s2 + v;
        }
      } else {
#pragma unroll
        for (int d = 0; d < 6; ++d) {  // an absent direction has count 0: v = 0 leaves mu and s2
          const Real db = COMP ? net_drate<Real, COMP>(T, m, (ncomp >> (5 * d)) & 31u, s) : dr;
          const Real* by = T.by[(nn >> (4 * d)) & 7u];
          const Real v = div_small(db * (Real)xb[d], by[0], by[1]);
          mu = mu - v;
          s2 = s2 + v;
        }
      }
    } else {
      if (leaps && n > 0) {
        const Real dout = (Real)n * d0;
        mu = mu - dout;
        s2 = s2 + dout;
      }
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if (xb[d] >= nc && ((q.on >> d) & 1u)) {
          const Real v = (COMP ? net_drate<Real, COMP>(T, m, (ncomp >> (5 * d)) & 31u, s) : dr) * (Real)xb[d];
          mu = mu + v;
          s2 = s2 + v;
        }
      }
    }
    const float t = net_tau_near<Real>(eps, T.hor[s], T.hmult[s], xs, mu, s2);
    const bool sane = t > 1e-30f && t < 1e30f;
    if (sane && t < near_ * 0.9999f) {
      near_ = t;
      b_mu = mu;
      b_s2 = s2;
      b_s = s;
    } else if (!sane || t < near_ * 1.0001f) {
      const Real ts = net_tau_species<Real>(A, T.hor[s], T.hmult[s], xs, mu, s2);
      if (ts < tau_ncr) tau_ncr = ts;
    }
  }
  if (b_s >= 0) {
    const Real ts = net_tau_species<Real>(A, T.hor[b_s], T.hmult[b_s], sx[b_s], b_mu, b_s2);
    if (ts < tau_ncr) tau_ncr = ts;
  }
  // critical (or, corrected SSA subvolume: total) rate, compute_tau_cr tau.cu:176-195
  Real rsum, dsum = (Real)0;
  if (mode == 0 || !plis_isinf_d((double)tau_ncr)) {
    rsum = rcrit;
    for (int s = 0; s < S; ++s) {
      const Real xs = sx[s];
      if (xs < (Real)nc) {
        const Real d = net_drate<Real, COMP>(T, m, comp, s) * xs;
        dsum = dsum + (mode == 0 ? d : (Real)n * d);
      }
    }
  } else {
    rsum = rall;
    for (int s = 0; s < S; ++s) dsum = dsum + (Real)n * (net_drate<Real, COMP>(T, m, comp, s) * sx[s]);
  }
  tau_ncr_out = tau_ncr;
  rate_cr_out = (rsum == (Real)0 && dsum == (Real)0) ? (Real)0 : rsum + dsum;
}

// ------------------------------------------------------------------------------------------------
// critical event of one LEAP_CR subvolume, reference semantics (leap.cu:86-199): critical_event_ref
// with its propensities evaluated once
// ------------------------------------------------------------------------------------------------
// sx holds the subvolume's counts.  (Finding the critical reactions first and evaluating only theirs was
// slower: 25.9 against 23.4 us for the events of the 10-species network on 64^3.)
template <typename Real, bool LOG, bool COMP>
__device__ __forceinline__ int critical_event_net(const KArgs& A, const NetTab<Real>& T, uint32_t c, Column<Real> sx,
                                                  Column<Real> sa, const int32_t* Xt, uint64_t step, uint32_t attempt, int32_t* D,
                                                  uint8_t* flag) {
  const DevModel& m = A.m;
  const int nc = A.o.nc;
  const int S = (int)m.S, R = (int)m.R;
  const uint32_t comp = COMP ? (uint32_t)m.comp[c] : 0u;
  plis_stream su = plis_stream_make(A.o.seed, A.o.replica, c, PLIS_PHASE_CRIT, step, attempt, 0);
  const Real u = RT<Real>::uniform(&su);
  uint32_t critm = 0;
  Real rsum = (Real)0, dsum = (Real)0;
#pragma unroll 2
  for (int r = 0; r < R; ++r) {
    bool crit;
    const Real a = net_prop<Real, COMP>(T, m, comp, sx, r, crit);
    sa[r] = a;
    critm |= (uint32_t)crit << r;
    if (crit) rsum = rsum + a;
  }
  uint32_t dcrit = 0;
  for (int s = 0; s < S; ++s) {
    const Real xs = sx[s];
    if (xs < (Real)nc) {
      dcrit |= 1u << s;
      dsum = dsum + net_drate<Real, COMP>(T, m, comp, s) * xs;
    }
  }
  if (rsum + dsum == (Real)0) return 0;
  if (u < rsum / (rsum + dsum)) {
    const Real scaled = rsum * u;
    Real partial = (Real)0;
    int ric = 0;
    while (partial <= scaled && ric < R) {
      if ((critm >> ric) & 1u) partial = partial + sa[ric];
      ++ric;
    }
    int ri = 0;
    for (ri = 0; ri < R && ric > 0; ++ri)
      if ((critm >> ri) & 1u) --ric;
    ri = ri - 1;  // leap.cu:121-126 as written
    if (ri < 0) ri = 0;
    // feasible: every reactant species has its molecules before and after the leap, and no species
    // went below zero in the leap
    bool fire = true;
    net_rows(m, Xt, c, S, [&](int s, int32_t xt) {
      int need = 0;
      for (uint32_t w = T.need[ri]; w; w >>= 10)
        if ((w & 31u) == (uint32_t)s) need = (int)((w >> 5) & 31u);
      fire = fire && !(sx[s] < (Real)need) && xt >= need;
    });
    if (!fire) return 0;
    for (uint32_t e = T.net_off[ri]; e < T.net_off[ri + 1]; ++e)
      atomicAdd(&D[(size_t)T.net_s[e] * m.Npad + c], T.net_nu[e]);
    touch(A, c);
    if (LOG) ev_put(A.b.ev, A.b.ctrl->t, step, attempt, c, c, 1, ri, PLIS_EVENT_CRITICAL_REACTION);
    return 1;
  }
  const Real scaled = dsum * u;
  Real partial = (Real)0;
  int spic = 0;
  while (partial <= scaled && spic < S) {
    if ((dcrit >> spic) & 1u) partial = partial + net_drate<Real, COMP>(T, m, comp, spic) * sx[spic];
    ++spic;
  }
  int spi = 0;
  for (spi = 0; spi < S && spic > 0; ++spi)
    if ((dcrit >> spi) & 1u) --spic;
  spi = spi - 1;  // leap.cu:160-166
  if (spi < 0) spi = 0;
  return critical_jump_ref<Real, LOG>(A, c, spi, sx[spi] > (Real)0, Xt, step, attempt, D, flag);
}

}  // namespace plis

#endif
