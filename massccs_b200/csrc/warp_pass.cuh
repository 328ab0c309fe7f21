// warp_pass.cuh -- the warp pass of the trajectory engine: parked
// trajectories, one per CTA, at the lowest latency per integration step.
//
// A captured orbit runs up to 3e5 steps one after another, so a run ends with
// the longest chain of steps: the time of one step is what this pass is built
// for, and the sums of a step are spread over the SM's four sub-partitions.
// The terms of one force evaluation fall into independent sums (a site's
// force, the dipole's field, the field's gradient); each group of sums is a
// role, and each role is a warp that walks the whole candidate list.  A sum's
// order (which candidates a lane adds, and when) is that of one warp doing
// all of them, so the split changes no result.  Measured on the 1231-atom N2
// globule (about 1100 candidates a step): see the figures at warp_pass_kernel.
#pragma once

#include "ccs_device.cuh"

namespace ccs {

// The roles of a gas shape: role r sums the row entries [k0(r), k1(r)) at one site.
template <int GAS, bool HASQ> struct Roles {
  static constexpr bool ATOM = GAS == GAS_ATOM;
  // atoms: force + field, gradient; N2: the two N, the charge's force + field,
  // gradient; CO2: the three sites, field + gradient
  static constexpr int N = ATOM ? (HASQ ? 2 : 1) : HASQ ? 4 : GAS == GAS_N2 ? 2 : 3;
  static constexpr int E = Row<GAS>::E, G = Row<GAS>::G, U = Row<GAS>::U;
  static constexpr int k0(int r) { return ATOM ? (r == 0 ? 0 : G) : r < 3 ? 3 * r : GAS == GAS_N2 ? G : E; }
  static constexpr int k1(int r) {
    return ATOM ? (r == 0 ? (HASQ ? G : E) : U) : r < 2 ? 3 * r + 3 : r == 2 ? (GAS == GAS_N2 ? G : E) : U;
  }
  static constexpr int site(int r) { return ATOM ? 0 : r < 3 ? r : GasShape<GAS>::DIP; }
  static constexpr bool force(int r) { return ATOM ? r == 0 : r < 3; }
  static constexpr bool field(int r) { return HASQ && (ATOM ? r == 0 : GAS == GAS_N2 ? r == 2 : r == 3); }
  static constexpr bool grad(int r) { return HASQ && r == N - 1; }
};

// One candidate's terms of role R, in the order and with the roundings of
// visit_atom.  LJ: the candidate may be inside the LJ cutoff (a group of
// candidates that all lie beyond it adds exact zeros, and is passed by).
template <typename T, int GAS, bool HASQ, int R, bool LJ>
__device__ __forceinline__ void visit_role(const KParams &kp, const T (&p)[3], const Atom<T> &a, bool dipf, T (&f)[3],
                                           T (&E)[3], T (&G)[6]) {
  using RO = Roles<GAS, HASQ>;
  constexpr int s = RO::site(R);
  constexpr int lj = site_lj<GAS>(s);
  const KConst<T> &kc = kconst<T>(kp);
  const T dx = p[0] - a.x, dy = p[1] - a.y, dz = p[2] - a.z;
  const T r2 = dx * dx + dy * dy + dz * dz;
  const T ir = Real<T>::rsq(r2);
  const T ir2 = ir * ir;
  if constexpr (RO::force(R) && lj != 0 && LJ) {
    const bool in_lj = r2 < kc.rlj2;
    const T A = lj == 2 ? a.Ac : a.A, B = lj == 2 ? a.Bc : a.B;
    const T ir6 = ir2 * ir2 * ir2;
    const T fl = in_lj ? ir6 * (T(12) * A * ir6 - T(6) * B) * ir2 : T(0);
    f[0] += fl * dx; f[1] += fl * dy; f[2] += fl * dz;
  }
  if constexpr (HASQ) {
    const bool in_c = r2 < kc.rc2;
    const T ir3 = Real<T>::mul(ir, ir2);
    const T ir3s = Real<T>::add(ir3, -kc.rc3inv);
    if constexpr (RO::force(R) && site_coul<GAS>(s)) {
      T ir3c = Real<T>::fma(ir, ir2, -kc.rc3inv);
      if constexpr (s == GasShape<GAS>::DIP) ir3c = dipf ? ir3c : ir3s;
      const T fc = in_c ? kc.kq[s] * a.q * ir3c : T(0);
      f[0] += fc * dx; f[1] += fc * dy; f[2] += fc * dz;
    }
    if constexpr (RO::field(R) || RO::grad(R)) {
      const T sq = in_c ? a.q * ir3s : T(0);
      if constexpr (RO::field(R)) { E[0] += sq * dx; E[1] += sq * dy; E[2] += sq * dz; }
      if constexpr (RO::grad(R)) {
        const T tq = in_c ? T(-3) * a.q * ir3 * ir2 : T(0);
        const T tx = tq * dx, ty = tq * dy;
        G[0] += sq + tx * dx;
        G[1] += sq + ty * dy;
        G[2] += sq + tq * dz * dz;
        G[3] += tx * dy;
        G[4] += tx * dz;
        G[5] += ty * dz;
      }
    }
  }
}

// Where a step's candidates are: packed in shared memory in list order
// (FP32), or atoms of the global tables, by index or all of them.
template <typename T> struct Cand {
  const float4 *pos;   // packed x, y, z, q (nullptr: not packed)
  const float2 *ab, *abc;
  const int *list;     // atom indices (nullptr: atom t is candidate t)
  const unsigned *ljm; // one bit per 32 candidates of this virtual warp: some may be inside the LJ cutoff
  int m;
};

template <typename T, int GAS, bool PACK, bool LJ>
__device__ __forceinline__ Atom<T> fetch(const KParams &kp, const Cand<T> &c, int t) {
  Atom<T> a;
  if constexpr (PACK) {
    const float4 q = c.pos[t];
    a.x = q.x; a.y = q.y; a.z = q.z; a.q = q.w;
    if constexpr (LJ) {
      const float2 ab = c.ab[t];
      a.A = ab.x; a.B = ab.y;
      if constexpr (GAS == GAS_CO2) { const float2 v = c.abc[t]; a.Ac = v.x; a.Bc = v.y; }
    }
    return a;
  } else {
    const int i = c.list ? c.list[t] : t;
    if constexpr (sizeof(T) == 4) {
      const float4 q = __ldg(&kp.xyzq32[i]);
      a.x = q.x; a.y = q.y; a.z = q.z; a.q = q.w;
      if constexpr (LJ) {
        const float2 ab = __ldg(&kp.ab32[i]);
        a.A = ab.x; a.B = ab.y;
        if constexpr (GAS == GAS_CO2) { const float2 v = __ldg(&kp.abc32[i]); a.Ac = v.x; a.Bc = v.y; }
      }
    } else {
      const double4 q = kp.xyzq64[i];
      a.x = q.x; a.y = q.y; a.z = q.z; a.q = q.w;
      if constexpr (LJ) {
        const double2 ab = kp.ab64[i];
        a.A = ab.x; a.B = ab.y;
        if constexpr (GAS == GAS_CO2) { const double2 v = kp.abc64[i]; a.Ac = v.x; a.Bc = v.y; }
      }
    }
    return a;
  }
}

// How many of a lane's candidates are in flight at once.  A lone warp per
// sub-partition hides the ~100 cycles of load, rsqrt and products behind
// other candidates' work.
constexpr int WP_ILP = 4;

// Role R's sums over the candidates of virtual thread vt (vt, vt + NT, ...).
template <typename T, int GAS, bool HASQ, int R, int NT, bool PACK>
__device__ __forceinline__ void role_visits(const KParams &kp, const T (&p)[3], const Cand<T> &c, int vt, T (&f)[3],
                                            T (&E)[3], T (&G)[6]) {
  using RO = Roles<GAS, HASQ>;
  constexpr bool HASLJ = RO::force(R) && site_lj<GAS>(RO::site(R)) != 0;
  constexpr bool PF = sizeof(T) == 4 && GAS == GAS_CO2;  // see visit_atom's DIPF
  const int cnt = vt < c.m ? (c.m - vt + NT - 1) / NT : 0;
  int k = 0, t = vt;
  for (; k + WP_ILP <= cnt; k += WP_ILP, t += WP_ILP * NT) {
    const bool lj = HASLJ && (!c.ljm || ((c.ljm[k >> 5] >> (k & 31)) & ((1u << WP_ILP) - 1u)) != 0);
    if (lj) {
      Atom<T> a[WP_ILP];
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) a[i] = fetch<T, GAS, PACK, HASLJ>(kp, c, t + i * NT);
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) visit_role<T, GAS, HASQ, R, HASLJ>(kp, p, a[i], PF, f, E, G);
    } else if (HASQ) {
      Atom<T> a[WP_ILP];
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) a[i] = fetch<T, GAS, PACK, false>(kp, c, t + i * NT);
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) visit_role<T, GAS, HASQ, R, false>(kp, p, a[i], PF, f, E, G);
    }
  }
#pragma unroll 1
  for (; k < cnt; k++, t += NT) {
    const Atom<T> a = fetch<T, GAS, PACK, HASLJ>(kp, c, t);
    visit_role<T, GAS, HASQ, R, HASLJ>(kp, p, a, PF && !(NT == 32 && (cnt & 1) && k == cnt - 1), f, E, G);
  }
}

// The sums of one role over its candidates, reduced over the warp into row
// (the part of it that is the role's).
template <typename T, int GAS, bool HASQ, int R> __device__ __forceinline__ void role_reduce(const T (&f)[3], const T (&E)[3],
                                                                                            const T (&G)[6], int lane, T *row) {
  using RO = Roles<GAS, HASQ>;
  constexpr int K0 = RO::k0(R), K1 = RO::k1(R);
  warp_sum_rows<K1 - K0, T>(
      [&](int k) { return k >= Row<GAS>::G ? G[(k - Row<GAS>::G) % 6] : k >= Row<GAS>::E ? E[(k - Row<GAS>::E) % 3] : f[k % 3]; },
      K0, lane, row);
}

// Atom i as packed candidate t.
template <typename T, int GAS>
__device__ __forceinline__ void pack_atom(const KParams &kp, int i, int t, float4 *pos, float2 *ab, float2 *abc) {
  if constexpr (sizeof(T) == 4) {
    pos[t] = __ldg(&kp.xyzq32[i]);
    ab[t] = __ldg(&kp.ab32[i]);
    if constexpr (GAS == GAS_CO2) abc[t] = __ldg(&kp.abc32[i]);
  }
}

// This warp's role in one force evaluation.
template <typename T, int GAS, bool HASQ, int NT, int R = 0>
__device__ __forceinline__ void step_visits(const KParams &kp, int role, const T (&p)[GasShape<GAS>::NS][3],
                                            unsigned actbits, const Cand<T> &c, int vt, T (&f)[3], T (&E)[3], T (&G)[6]) {
  using RO = Roles<GAS, HASQ>;
  if constexpr (R < RO::N) {
    if (role == R) {
      constexpr int s = RO::site(R);
      if (!((actbits >> s) & 1u) || (!RO::force(R) && !kp.dip_on)) return;  // the site feels nothing
      if constexpr (sizeof(T) == 4) {
        if (c.pos) { role_visits<T, GAS, HASQ, R, NT, true>(kp, p[s], c, vt, f, E, G); return; }
      }
      role_visits<T, GAS, HASQ, R, NT, false>(kp, p[s], c, vt, f, E, G);
    } else {
      step_visits<T, GAS, HASQ, NT, R + 1>(kp, role, p, actbits, c, vt, f, E, G);
    }
  }
}
template <typename T, int GAS, bool HASQ, int R = 0>
__device__ __forceinline__ void step_reduce(int role, const T (&f)[3], const T (&E)[3], const T (&G)[6], int lane, T *row) {
  if constexpr (R < Roles<GAS, HASQ>::N) {
    if (role == R) role_reduce<T, GAS, HASQ, R>(f, E, G, lane, row);
    else step_reduce<T, GAS, HASQ, R + 1>(role, f, E, G, lane, row);
  }
}

// Shared memory of the pass besides the candidate lists.
template <typename T, int GAS, int NT> struct WarpShared {
  static constexpr int NW = NT / 32;
  static constexpr int ROWP = (Row<GAS>::N + 3) / 4 * 4;
  alignas(16) T red[2][NW][ROWP];  // reduced sums per virtual warp, alternating
  unsigned ljm[NW][LCAP_MAX / 32 / NW / 32 > 0 ? LCAP_MAX / 32 / NW / 32 : 1];
  int wsum[NW];
  unsigned long long blk[8];
  unsigned long long idx;
  int kind, stop;
};

// Exclusive scan of the run lengths of the NT threads of role 0 (every thread
// of the CTA calls; the others pass len = 0 and get no position).  Two
// barriers: wsum may be rewritten after it.
template <int NT>
__device__ __forceinline__ int role_scan(int len, bool lead, int lane, int v, int *wsum, int &total) {
  constexpr int NW = NT / 32;
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lead && lane == 31) wsum[v] = incl;
  __syncthreads();
  int wofs = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < NW; k++) {
    const int ws = wsum[k];
    wofs += k < v ? ws : 0;
    total += ws;
  }
  __syncthreads();
  return incl + wofs - len;
}

// The candidates of a step whose list would not fit: the runs of the reach
// sphere around c, flattened chunk by chunk; each chunk goes to visit(list, m).
template <typename T, int NT, bool RF, typename F>
__device__ __forceinline__ uint32_t for_chunks(const KParams &kp, T cx, T cy, T cz, T R, bool lead, int lane, int v,
                                               int *list, int lcap, int *wsum, const F &visit) {
  int i0, j0, nj;
  float inv_nj;
  uint32_t nvis = 0;
  const int vt = v * 32 + lane;
  const int ncol = column_range(kp, cx, cy, R, i0, j0, nj, inv_nj);
  for (int base = 0; base < ncol; base += NT) {
    int b = 0, len = 0, total;
    if (lead) column_run<RF>(kp, base + vt, ncol, i0, j0, nj, inv_nj, cx, cy, cz, R, b, len);
    const int excl = role_scan<NT>(len, lead, lane, v, wsum, total);
    for (int cs = 0; cs < total; cs += lcap) {
      // this thread's run, as far as it falls into the chunk [cs, cs + lcap)
      const int lo = max(excl, cs), hi = min(excl + len, cs + lcap);
      for (int q = lo; q < hi; q++) list[q - cs] = b + (q - excl);
      __syncthreads();
      visit(list, min(lcap, total - cs));
      __syncthreads();  // the chunk is rewritten next
    }
    nvis += (uint32_t)total;
  }
  return nvis;
}

// The sites' energies of a step that begins or ends a try, one warp per
// virtual warp (the lead role's) in the order of the force sums, into
// row[v][U..U + NS) of the reduction buffer.  Out of line: once or twice a try.
// chunked: the candidates are the runs of the sphere (c, R); else list/m.
template <typename T, int GAS, bool HASQ, int NT, bool RF>
__device__ __noinline__ void warp_energy(const KParams *__restrict__ kpg, const ProbeSites<T, GAS> ps, bool chunked,
                                         T cx, T cy, T cz, T R, int *list, int m, int lcap, bool lead, int lane, int v,
                                         int *wsum, T *row) {
  const KParams &kp = *kpg;
  Acc<T, GasShape<GAS>::NS> acc;
  acc.zero();
  auto visit = [&](const int *l, int n) {
    if (!lead) return;
    for (int t = v * 32 + lane; t < n; t += NT)
      visit_atom<T, GAS, HASQ, false, false, true>(kp, ps.p, ps.act, load_atom<T, GAS>(kp, l ? l[t] : t), acc);
  };
  if (chunked) for_chunks<T, NT, RF>(kp, cx, cy, cz, R, lead, lane, v, list, lcap, wsum, visit);
  else visit(list, m);
  if (lead) reduce_group_row<T, 32, GAS, Row<GAS>::U, Row<GAS>::N>(acc, lane, 0xffffffffu, row);
}

// CTAs per SM that the register allocation allows: FP32 512 threads (128
// registers), FP64 unconstrained.
#ifndef CCS_WARP_THREADS_PER_SM
#define CCS_WARP_THREADS_PER_SM 512
#endif
template <typename T, int GAS, bool HASQ, int NT> struct WarpShape {
  static constexpr int THREADS = NT * Roles<GAS, HASQ>::N;
  static constexpr int MINB = sizeof(T) == 8 ? 1 : (CCS_WARP_THREADS_PER_SM / THREADS > 0 ? CCS_WARP_THREADS_PER_SM / THREADS : 1);
};

// The warp pass.  See the speculative retries in ccs_device.cuh for the hand-
// over of failed tries; the launch's phases and counters are described there.
template <typename T, int GAS, bool HASQ, int NT, bool BATCH>
__global__ void __launch_bounds__(WarpShape<T, GAS, HASQ, NT>::THREADS, WarpShape<T, GAS, HASQ, NT>::MINB)
    warp_pass_kernel(KParams kp, const KParams *__restrict__ kpg) {
  using S = Sites<GAS>;
  using RO = Roles<GAS, HASQ>;
  constexpr int NS = S::NS, NW = NT / 32, NTHREADS = WarpShape<T, GAS, HASQ, NT>::THREADS;
  constexpr bool PACKS = sizeof(T) == 4;
  constexpr bool RF = sizeof(T) == 4 && GAS != GAS_ATOM && NT != 32 && !BATCH;  // see column_run
  constexpr int NF = Row<GAS>::forces(HASQ);
  __shared__ WarpShared<T, GAS, NT> sm;
  __shared__ __align__(16) unsigned char sm_kp[BATCH ? sizeof(KParams) : 16];  // this trajectory's ion
  extern __shared__ __align__(16) unsigned char dyn[];
  // candidate list: indices, then (kp.wp_pack) the packed candidates in list order
  int *const sm_list = reinterpret_cast<int *>(dyn);
  float4 *const sm_pos = reinterpret_cast<float4 *>(dyn + (((size_t)kp.wp_cap * 4 + 15) & ~size_t(15)));
  float2 *const sm_ab = reinterpret_cast<float2 *>(sm_pos + kp.wp_cap);
  float2 *const sm_abc = sm_ab + kp.wp_cap;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // the roles of a virtual warp sit on different sub-partitions; a second
  // virtual warp starts two further on, so light and heavy roles mix
  const int v = w / RO::N, role = (w + 2 * v) % RO::N;
  const int vt = v * 32 + lane;
  const bool lead = role == 0;
  if (tid < 8) sm.blk[tid] = 0ull;
  __syncthreads();
  int red = 0;
  const bool spec_launch = kp.spec_phase != 0;
  const unsigned long long deadline = *(volatile const unsigned long long *)kp.deadline;
  unsigned long long np;
  if (spec_launch) {
    np = *(volatile unsigned long long *)kp.spec_count;
    if (np > kp.spec_cap) np = kp.spec_cap;
    np *= SPEC_ITEMS;
  } else {
    np = *(volatile unsigned long long *)kp.park_count;
    if (np > kp.park_cap) np = kp.park_cap;
  }
  unsigned long long *next = spec_launch ? kp.spec_next : kp.park_next;
  const bool may_spec = kp.spec_rec && !spec_launch;
  bool park_done = spec_launch;
  for (;;) {
    if (tid == 0) {
      int kind;
      sm.idx = claim_item(kp, np, next, spec_launch, may_spec, deadline, park_done, kind);
      sm.kind = kind;
    }
    __syncthreads();
    const unsigned long long idx = sm.idx;
    bool spec = sm.kind != 0;  // this item is a speculative try
    __syncthreads();
    if (idx == ~0ull) break;
    LaneState<T> L;
    unsigned long long rec = 0;
    if (spec) {  // try k of record rec, from the trajectory's initial state
      rec = idx / SPEC_ITEMS;
      if (tid == 0) sm.stop = *(volatile int *)&kp.spec_rec[rec].stop;
      __syncthreads();
      const int stop = sm.stop;
      __syncthreads();
      const SpecRec R = load_spec_rec(kp.spec_rec + rec);
      const int k = R.tries + 1 + (int)(idx % SPEC_ITEMS);
      if (k > 8 || k > stop) continue;  // beyond the last try, or decided before it (block-uniform)
      L.j = R.j;
      L.ion = R.ion;
      load_init<T, GAS>(L, lane_setup<T, GAS>(ion_params_ptr<BATCH>(kp, kpg, L.ion), L.j));
      L.Ei = T(R.Ei);
      L.tries = k;
      L.maxTries = R.maxTries;
      L.dt = T(ion_params<BATCH>(kp, L.ion).dt / (k + 1));
      L.mode = M_RESTART;
      L.nsteps = 0;
      L.nvis = 0;
    } else {
      L = reinterpret_cast<const LaneState<T> *>(kp.park)[idx];
    }
    const KParams *Kg = ion_params_ptr<BATCH>(kp, kpg, L.ion);
    if constexpr (BATCH) {  // the ion's parameters, read every step
      for (int i = tid; i < (int)(sizeof(KParams) / 4); i += NTHREADS)
        reinterpret_cast<unsigned *>(sm_kp)[i] = reinterpret_cast<const unsigned *>(Kg)[i];
      __syncthreads();
    }
    const KParams &K = [&]() -> const KParams & {
      if constexpr (BATCH) return *reinterpret_cast<const KParams *>(sm_kp); else return kp;
    }();
    const KConst<T> &kc = kconst<T>(K);
    const int lcap = kp.lcap;
    // A target of at most two atoms per virtual thread is all candidates at every step
    const bool small = K.natoms <= 2 * NT;
    const bool packs = PACKS && kp.wp_pack;
    if (packs && small) {
      for (int t = tid; t < K.natoms; t += NTHREADS) pack_atom<T, GAS>(K, t, t, sm_pos, sm_ab, sm_abc);
      __syncthreads();
    }
    int list_n = -1;  // this trajectory's candidate list (none yet)
    T list_c[3] = {T(0), T(0), T(0)};
    T inv_dt = Real<T>::div(T(1), L.dt);
    // From spec_from failed tries on, the remaining ones run at once as soon
    // as the pass is short of work; the one at hand goes on here.
    auto try_record = [&]() {
      if (tid == 0) sm.idx = record_spec(kp, np, L);
      __syncthreads();
      const unsigned long long slot = sm.idx;
      __syncthreads();
      if (slot != ~0ull) {
        spec = true;
        rec = slot;
        L.nsteps = L.nvis = 0;  // the record holds those so far
      }
    };
    if (may_spec && !spec && L.tries >= kp.spec_from) try_record();
    for (unsigned it = 1;; it++) {
      int r = S_CONTINUE;
      double omc = 0.0;
      if ((it & 255u) == 0) {
        if (tid == 0) {
          sm.stop = (global_ns() > deadline || *(volatile int *)kp.error)                   ? 1
                    : spec && L.tries > *(volatile int *)&kp.spec_rec[rec].stop ? 2
                                                                                : 0;
        }
        __syncthreads();
        const int e = sm.stop;
        __syncthreads();
        if (e == 2) break;  // the trajectory is decided by an earlier try
        if (e) {
          if (tid == 0) atomicExch(kp.error, 1);
          r = S_CAPPED;
        } else if (may_spec && !spec && L.tries >= kp.spec_from) {
          try_record();
        }
      }
      if (r == S_CONTINUE) {
        bool out = false;
        if (L.mode == M_STEP) {
          first_half<T, GAS>(K, L, inv_dt);
          out = step_leaves(K, L);
        }
        const bool want_u = L.mode == M_INIT || out;
        L.U = T(0);
        T p[NS][3], fs[NS][3];
        site_positions<T, GAS>(L, p);
        unsigned actbits;
        if (probe_near<T, GAS>(K, p, actbits)) {
          bool act[NS];
#pragma unroll
          for (int s = 0; s < NS; s++) act[s] = (actbits >> s) & 1u;
          const T off = site_offset<T, GAS>(p);
          const T R = K.allpairs ? T(INFINITY) : kc.reach + off + T(1e-3);
          const T cx = p[S::cs][0], cy = p[S::cs][1], cz = p[S::cs][2];
          const T ex = fmax(fmax(kc.bb_lo[0] - cx, cx - kc.bb_hi[0]), T(0));
          const T ey = fmax(fmax(kc.bb_lo[1] - cy, cy - kc.bb_hi[1]), T(0));
          const T ez = fmax(fmax(kc.bb_lo[2] - cz, cz - kc.bb_hi[2]), T(0));
          const T fx = fmax(cx - kc.bb_lo[0], kc.bb_hi[0] - cx);
          const T fy = fmax(cy - kc.bb_lo[1], kc.bb_hi[1] - cy);
          const T fz = fmax(cz - kc.bb_lo[2], kc.bb_hi[2] - cz);
          Cand<T> cd{nullptr, sm_ab, sm_abc, nullptr, nullptr, 0};
          bool chunked = false;
          if (small || fx * fx + fy * fy + fz * fz <= R * R) {
            // the whole target inside the reach sphere, or a small target:
            // every atom is a candidate (the cutoff tests are exact)
            cd.m = K.natoms;
            if (packs && small) cd.pos = sm_pos;
          } else if (ex * ex + ey * ey + ez * ez <= R * R) {
            const T dcx = cx - list_c[0], dcy = cy - list_c[1], dcz = cz - list_c[2];
            const T moved2 = Real<T>::fma(dcz, dcz, Real<T>::fma(dcx, dcx, Real<T>::mul(dcy, dcy)));
            if (list_n < 0 || moved2 > T(LSKIN) * T(LSKIN)) {
              // rebuild the list for the sphere of radius R + LSKIN around the centre
              const T RL = R + T(LSKIN);
              int i0, j0, nj;
              float inv_nj;
              const int ncol = column_range(K, cx, cy, RL, i0, j0, nj, inv_nj);
              int filled = 0;  // block-uniform
              for (int i = tid; i < (int)(sizeof(sm.ljm) / 4); i += NTHREADS) (&sm.ljm[0][0])[i] = 0u;
              for (int base = 0; base < ncol; base += NT) {
                int b = 0, len = 0, total;
                if (lead) column_run<RF>(K, base + vt, ncol, i0, j0, nj, inv_nj, cx, cy, cz, RL, b, len);
                const int excl = role_scan<NT>(len, lead, lane, v, sm.wsum, total);
                if (filled + total <= lcap)
                  for (int q = 0; q < len; q++) sm_list[filled + excl + q] = b + q;
                filled += total;
              }
              list_n = filled <= lcap ? filled : -1;
              list_c[0] = cx; list_c[1] = cy; list_c[2] = cz;
              __syncthreads();  // the runs are in place
              if (list_n >= 0) {
                // pack, and mark the groups of 32 candidates that can come inside the LJ
                // cutoff of a site while this list is in use
                const T rl = T(sqrt(kc.rlj2)) + T(LSKIN) + off + T(0.05);
                for (int g = w; g * 32 < list_n; g += NTHREADS / 32) {
                  const int t = g * 32 + lane;
                  bool in = false;
                  if (t < list_n) {
                    const int i = sm_list[t];
                    if (packs) pack_atom<T, GAS>(K, i, t, sm_pos, sm_ab, sm_abc);
                    T x, y, z;
                    if constexpr (sizeof(T) == 4) { const float4 q = __ldg(&K.xyzq32[i]); x = q.x; y = q.y; z = q.z; }
                    else { const double4 q = K.xyzq64[i]; x = q.x; y = q.y; z = q.z; }
                    in = (x - cx) * (x - cx) + (y - cy) * (y - cy) + (z - cz) * (z - cz) <= rl * rl;
                  }
                  if (__any_sync(0xffffffffu, in) && lane == 0)
                    atomicOr(&sm.ljm[g % NW][g / NW >> 5], 1u << (g / NW & 31));
                }
                __syncthreads();
              }
            }
            if (list_n >= 0) {
              cd.list = sm_list;
              cd.ljm = sm.ljm[v];
              cd.m = list_n;
              if (packs) cd.pos = sm_pos;
            } else {
              chunked = true;
            }
          }
          T af[3] = {T(0), T(0), T(0)}, aE[3] = {T(0), T(0), T(0)}, aG[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
          uint32_t nvis;
          if (chunked) {
            nvis = for_chunks<T, NT, RF>(K, cx, cy, cz, R, lead, lane, v, sm_list, lcap, sm.wsum, [&](int *l, int n) {
              Cand<T> cc{nullptr, nullptr, nullptr, l, nullptr, n};
              step_visits<T, GAS, HASQ, NT>(K, role, p, actbits, cc, vt, af, aE, aG);
            });
          } else {
            step_visits<T, GAS, HASQ, NT>(K, role, p, actbits, cd, vt, af, aE, aG);
            nvis = (uint32_t)cd.m;
          }
          T *const row = sm.red[red][v];
          step_reduce<T, GAS, HASQ>(role, af, aE, aG, lane, row);
          if (want_u) {
            ProbeSites<T, GAS> ps;
#pragma unroll
            for (int s = 0; s < NS; s++) {
              ps.act[s] = act[s];
#pragma unroll
              for (int k = 0; k < 3; k++) ps.p[s][k] = p[s][k];
            }
            if (chunked) __syncthreads();  // the list is rewritten by the energy's chunks
            warp_energy<T, GAS, HASQ, NT, RF>(Kg, ps, chunked, cx, cy, cz, R, chunked || cd.list ? sm_list : nullptr, cd.m,
                                          lcap, lead, lane, v, sm.wsum, row);
          }
          __syncthreads();
          // every thread sums the virtual warps' partials in the same fixed order
          T sum[Row<GAS>::N];
#pragma unroll
          for (int k = 0; k < NF; k++) {
            sum[k] = sm.red[red][0][k];
#pragma unroll
            for (int q = 1; q < NW; q++) sum[k] += sm.red[red][q][k];
          }
          if constexpr (GAS == GAS_N2 && !HASQ) sum[6] = sum[7] = sum[8] = T(0);  // the centre has no terms
          finish_row<T, GAS, HASQ>(K, sum, act, fs);
          if (want_u) {
#pragma unroll
            for (int k = Row<GAS>::U; k < Row<GAS>::N; k++) {
              sum[k] = sm.red[red][0][k];
#pragma unroll
              for (int q = 1; q < NW; q++) sum[k] += sm.red[red][q][k];
            }
            L.U = finish_energy<T, GAS, HASQ>(K, sum, act);
          }
          red ^= 1;
          L.nvis += nvis;
        } else {
#pragma unroll
          for (int s = 0; s < NS; s++) fs[s][0] = fs[s][1] = fs[s][2] = T(0);
        }
        absorb_forces<T, GAS>(K, fs, L);
        if (L.mode == M_INIT) { L.Ei += L.U; L.mode = M_STEP; continue; }
        if (L.mode == M_RESTART) { L.mode = M_STEP; continue; }
        r = second_half<T, GAS>(K, L, out);
        if (r == S_CONTINUE) continue;
        if (r == S_SCATTER)
          omc = lane_chi<T, GAS>(Kg, L.j, exit_velocity<T, GAS>(L, 0), exit_velocity<T, GAS>(L, 1),
                                 exit_velocity<T, GAS>(L, 2));
      }
      // the try has ended: scatter, capped (or watchdog), or a failed test
      if (spec) {
        if (tid == 0) write_spec_out(kp, rec, L, r, omc);
        break;
      }
      if (r == S_SCATTER) {
        if (tid == 0) write_result(K, L, 1, omc, sm.blk);
        break;
      }
      if (r == S_CAPPED) {
        if (tid == 0) write_result(K, L, 3, 0.0, sm.blk);
        break;
      }
      L.tries++;
      if (r == S_RETRY_ENERGY) L.maxTries++;
      L.dt = T(K.dt / (L.tries + 1));
      inv_dt = Real<T>::div(T(1), L.dt);
      if (!(L.tries < L.maxTries && L.maxTries < 10)) {
        if (tid == 0) write_result(K, L, 2, 0.0, sm.blk);
        break;
      }
      if (may_spec && L.tries >= kp.spec_from) try_record();
      load_init<T, GAS>(L, lane_setup<T, GAS>(Kg, L.j));
      L.mode = M_RESTART;
      list_n = -1;
    }
    // a parked trajectory has ended (or its record is published): one fewer running
    if (tid == 0 && !spec && may_spec) {
      __threadfence();
      atomicAdd(kp.park_active, ~0ull);
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid < 6 && sm.blk[tid]) atomicAdd(&kp.stats[tid], sm.blk[tid]);
}

}  // namespace ccs
