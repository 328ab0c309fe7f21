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
// all of them (NT "virtual threads": thread t adds candidates t, t + NT, ...),
// so the split changes no result.
//
// What bounds it: alone, the latency of a step (an instruction every 3.2
// cycles and warp); with the SM full, instruction fetch and issue (0.59 a
// cycle).  One step of one trajectory alone on the GPU, us: 32 (N2, CO2) or 64
// threads doing all sums, the energies at every step among them -> this pass:
//   He, 60 atoms 0.48 -> 0.25; He, 1231 atoms 1.08 -> 0.74; Ar, 777 atoms,
//   LJ 0.78 -> 0.53; N2, 1231 atoms, +4 e 6.7 -> 1.34; CO2, 1001 atoms 6.7 ->
//   1.18; N2, 20,000 atoms 6.7 -> 2.14; N2 in FP64 5.5 -> 2.2; N2 without
//   cutoffs, 333 atoms 3.8 -> 1.26; He, shell of 5e5 atoms 5.3 -> 2.8.
// (Without the energies at every step the former took 3.3 us for the N2 one.)
// Tried and left out: one integrating warp per CTA with the others waiting for
// positions (N2 1.62 -> 1.76 us: its two hand-overs cost more than the copies
// of the integrator), two candidates per instruction in packed FP32 (no gain:
// the step is not short of multiply-adds), 2 or 8 candidates side by side
// (2: 10 % slower on lists of thousands), 5 CTAs an SM (the registers spill).
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
  // the first role of the same shape (a molecule's two like atoms): the two
  // run one code, since instruction fetch is what a full SM waits for
  static constexpr int code(int r) { return GAS == GAS_N2 && r == 1 ? 0 : GAS == GAS_CO2 && r == 2 ? 0 : r; }
};

// One candidate's terms of role R, in the order and with the roundings of
// visit_atom.  LJ: the candidate may be inside the LJ cutoff (a group of
// candidates that all lie beyond it adds exact zeros, and is passed by).
// p, kq: position and charge factor of the role's site.
template <typename T, int GAS, bool HASQ, int R, bool LJ>
__device__ __forceinline__ void visit_role(const KParams &kp, const T (&p)[3], T kq, const Atom<T> &a, bool dipf,
                                           T (&f)[3], T (&E)[3], T (&G)[6]) {
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
    // (an ion without Coulomb forces has no charges in its table: ccs_set_target)
    if constexpr (RO::force(R) && site_coul<GAS>(s)) {
      T ir3c = Real<T>::fma(ir, ir2, -kc.rc3inv);
      if constexpr (s == GasShape<GAS>::DIP) ir3c = dipf ? ir3c : ir3s;
      const T fc = in_c ? kq * a.q * ir3c : T(0);
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
// (FP32; every address a shared one), or atoms of the global tables, by index
// or all of them.
enum : int { C_NONE = 0, C_PACK = 1, C_LIST = 2, C_ALL = 3 };
struct Cand {
  const float4 *pos;   // packed x, y, z, q; far atoms up to the end of the last block
  const float2 *ab, *abc;
  const int *list;     // atom indices
  const unsigned *ljm; // one bit per 32 candidates of this virtual warp: some may be inside the LJ cutoff
  bool masked;         // ljm is valid (else every candidate may be)
  int m;
};

template <typename T, int GAS, int MODE, bool LJ>
__device__ __forceinline__ Atom<T> fetch(const KParams &kp, const Cand &c, int t) {
  Atom<T> a;
  a.A = a.B = a.Ac = a.Bc = T(0);
  if constexpr (MODE == C_PACK) {
    const float4 q = c.pos[t];
    a.x = q.x; a.y = q.y; a.z = q.z; a.q = q.w;
    if constexpr (LJ) {
      const float2 ab = c.ab[t];
      a.A = ab.x; a.B = ab.y;
      if constexpr (GAS == GAS_CO2) { const float2 v = c.abc[t]; a.Ac = v.x; a.Bc = v.y; }
    }
  } else {
    const int i = MODE == C_LIST ? c.list[t] : t;
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
  }
  return a;
}

// An atom whose every term is an exact zero: it fills a lane's place past the
// end of the candidates, so that the last ones run side by side as well
// (one at a time they cost up to three full latencies a step).
template <typename T> __device__ __forceinline__ Atom<T> far_atom() {
  Atom<T> a;
  a.x = T(1e18);
  a.y = a.z = a.q = a.A = a.B = a.Ac = a.Bc = T(0);
  return a;
}

// How many of a lane's candidates are in flight at once.  A lone warp per
// sub-partition hides the ~100 cycles of load, rsqrt and products behind
// other candidates' work.
constexpr int WP_ILP = 4;

// Role R's sums over the candidates of virtual thread vt (vt, vt + NT, ...),
// WP_ILP of them side by side.  The packed list ends in far atoms, so its
// blocks are all whole; the others mask their last block.
template <typename T, int GAS, bool HASQ, int R, int NT, int MODE>
__device__ __forceinline__ void role_visits(const KParams &kp, const T (&p)[3], T kq, const Cand &c, int vt, T (&f)[3],
                                            T (&E)[3], T (&G)[6]) {
  using RO = Roles<GAS, HASQ>;
  constexpr bool HASLJ = RO::force(R) && site_lj<GAS>(RO::site(R)) != 0;
  constexpr bool PF = sizeof(T) == 4 && GAS == GAS_CO2;  // see visit_atom's DIPF
  constexpr bool TAILF = PF && NT == 32 && RO::force(R) && RO::site(R) == GasShape<GAS>::DIP;
  const int wbase = vt & ~31;  // the same count of rounds for the whole warp
  const int rounds = wbase < c.m ? (c.m - wbase + NT - 1) / NT : 0;
  const int cnt = (MODE != C_PACK || TAILF) && vt < c.m ? (c.m - vt + NT - 1) / NT : 0;
#pragma unroll 1
  for (int k = 0, t = vt; k < rounds; k += WP_ILP, t += WP_ILP * NT) {
    Atom<T> a[WP_ILP];
    bool lj = false;
    if constexpr (HASLJ) lj = !c.masked || ((c.ljm[k >> 5] >> (k & 31)) & ((1u << WP_ILP) - 1u)) != 0;
    if (HASLJ && lj) {
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) {
        if constexpr (MODE != C_PACK) a[i] = far_atom<T>();
        if (MODE == C_PACK || k + i < cnt) a[i] = fetch<T, GAS, MODE, HASLJ>(kp, c, t + i * NT);
      }
#pragma unroll
      for (int i = 0; i < WP_ILP; i++)
        visit_role<T, GAS, HASQ, R, HASLJ>(kp, p, kq, a[i], PF && !(TAILF && (cnt & 1) && k + i == cnt - 1), f, E, G);
    } else if constexpr (HASQ) {
#pragma unroll
      for (int i = 0; i < WP_ILP; i++) {
        if constexpr (MODE != C_PACK) a[i] = far_atom<T>();
        if (MODE == C_PACK || k + i < cnt) a[i] = fetch<T, GAS, MODE, false>(kp, c, t + i * NT);
      }
#pragma unroll
      for (int i = 0; i < WP_ILP; i++)
        visit_role<T, GAS, HASQ, R, false>(kp, p, kq, a[i], PF && !(TAILF && (cnt & 1) && k + i == cnt - 1), f, E, G);
    }
  }
}

// The sums of one role over its candidates, reduced over the warp into row
// (the part of it that is the role's).
template <typename T, int GAS, bool HASQ, int R>
__device__ __forceinline__ void role_reduce(int role, const T (&f)[3], const T (&E)[3], const T (&G)[6], int lane, T *row) {
  using RO = Roles<GAS, HASQ>;
  constexpr int K0 = RO::k0(R), K1 = RO::k1(R);
  if (RO::force(R)) row += 3 * (role - R);  // a role that shares this code: its own site's entries
  warp_sum_rows<K1 - K0, T>(
      [&](int k) { return k >= Row<GAS>::G ? G[(k - Row<GAS>::G) % 6] : k >= Row<GAS>::E ? E[(k - Row<GAS>::E) % 3] : f[k % 3]; },
      K0, lane, row);
}

// Far atoms in the packed places from n to the end of its last block.
template <int GAS, int NT>
__device__ __forceinline__ void pack_end(int n, int tid, int nthreads, float4 *pos, float2 *ab, float2 *abc) {
  const int end = (n + WP_ILP * NT - 1) / (WP_ILP * NT) * (WP_ILP * NT);
  for (int t = n + tid; t < end; t += nthreads) {
    pos[t] = make_float4(1e18f, 0.f, 0.f, 0.f);
    ab[t] = make_float2(0.f, 0.f);
    if constexpr (GAS == GAS_CO2) abc[t] = make_float2(0.f, 0.f);
  }
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

// This warp's role in one force evaluation.  sa: atomic gases, a small
// target's atoms of this virtual thread, held in registers (C_NONE: they are
// the candidates).
template <typename T, int GAS, bool HASQ, int NT, int R = 0>
__device__ __forceinline__ void step_visits(const KParams &kp, int role, const T (&p)[GasShape<GAS>::NS][3],
                                            unsigned actbits, int mode, const Cand &c, const Atom<T> (&sa)[2], int vt,
                                            T (&f)[3], T (&E)[3], T (&G)[6]) {
  using RO = Roles<GAS, HASQ>;
  if constexpr (R < RO::N && RO::code(R < RO::N ? R : 0) != R) {
    step_visits<T, GAS, HASQ, NT, R + 1>(kp, role, p, actbits, mode, c, sa, vt, f, E, G);
  } else if constexpr (R < RO::N) {
    if (RO::code(role) == R) {
      const int s = RO::site(R) + (role - R);
      if (!((actbits >> s) & 1u) || (!RO::force(R) && !kp.dip_on)) return;  // the site feels nothing
      T ps[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        ps[k] = p[RO::site(R)][k];
#pragma unroll
        for (int q = R + 1; q < RO::N; q++)
          if (RO::code(q) == R && role == q) ps[k] = p[RO::site(q)][k];
      }
      const T kq = kconst<T>(kp).kq[RO::site(R)];  // roles of one code: equal charges
      if constexpr (GAS == GAS_ATOM) {
        if (mode == C_NONE) {
          visit_role<T, GAS, HASQ, R, true>(kp, ps, kq, sa[0], false, f, E, G);
          if (c.m > NT) visit_role<T, GAS, HASQ, R, true>(kp, ps, kq, sa[1], false, f, E, G);
          return;
        }
      }
      if constexpr (sizeof(T) == 4) {
        if (mode == C_PACK) { role_visits<T, GAS, HASQ, R, NT, C_PACK>(kp, ps, kq, c, vt, f, E, G); return; }
      }
      if (mode == C_LIST) role_visits<T, GAS, HASQ, R, NT, C_LIST>(kp, ps, kq, c, vt, f, E, G);
      else role_visits<T, GAS, HASQ, R, NT, C_ALL>(kp, ps, kq, c, vt, f, E, G);
    } else {
      step_visits<T, GAS, HASQ, NT, R + 1>(kp, role, p, actbits, mode, c, sa, vt, f, E, G);
    }
  }
}
template <typename T, int GAS, bool HASQ, int R = 0>
__device__ __forceinline__ void step_reduce(int role, const T (&f)[3], const T (&E)[3], const T (&G)[6], int lane, T *row) {
  using RO = Roles<GAS, HASQ>;
  if constexpr (R < RO::N && RO::code(R < RO::N ? R : 0) != R) {
    step_reduce<T, GAS, HASQ, R + 1>(role, f, E, G, lane, row);
  } else if constexpr (R < RO::N) {
    if (RO::code(role) == R) role_reduce<T, GAS, HASQ, R>(role, f, E, G, lane, row);
    else step_reduce<T, GAS, HASQ, R + 1>(role, f, E, G, lane, row);
  }
}

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
  T ang[2];     // the usual steps' angle and whether it is left to angle3, alternating like red
  int wide[2];
};

// The rounded square root of x without a branch (the usual call has one for
// the ends of the range): a Newton step from the approximate reciprocal root,
// then Tuckerman's test on the exact remainder (Agarwal et al. 1986) moves
// the result to the neighbour if that is nearer.  For 1e-18 <= x <= 1e18.
__device__ __forceinline__ float sqrt_mid(float x) {
  const float y = rsqrtf(x);
  float s = __fmul_rn(x, y);
  s = __fmaf_rn(__fmaf_rn(-s, s, x), __fmul_rn(0.5f, y), s);
  const float r = __fmaf_rn(-s, s, x);
  const float up = __int_as_float(__float_as_int(s) + 1), dn = __int_as_float(__float_as_int(s) - 1);
  return r > __fmul_rn(s, up - s) ? up : r <= -__fmul_rn(s, s - dn) ? dn : s;
}

// angle3 of a usual step, without branches; wide: it is not the small angle
// of the series (or too small for the root), and is left to angle3.
template <typename T> __device__ __forceinline__ T small_angle(const T a[3], const T b[3], bool &wide) {
  if constexpr (sizeof(T) == 8) {
    wide = false;
    return angle3(a, b);
  } else {
    const float cx = a[1] * b[2] - a[2] * b[1], cy = a[2] * b[0] - a[0] * b[2],
                cz = a[0] * b[1] - a[1] * b[0];
    const float c2 = cx * cx + cy * cy + cz * cz, cs = dot3(a, b);
    const float sn = sqrt_mid(c2);
    wide = !((c2 >= 1e-18f) & (c2 <= 1e18f) & (cs > 0.f) & (sn < 0.125f * cs));
    const float t = __fdividef(sn, cs), t2 = t * t;
    return t * (1.f + t2 * (-1.f / 3.f + t2 * (1.f / 5.f + t2 * (-1.f / 7.f + t2 * (1.f / 9.f)))));
  }
}

// The sums of a step from the virtual warps' partials, in a fixed order, and
// the forces from them.
template <typename T, int GAS, bool HASQ, int NT>
__device__ __forceinline__ void step_forces(const KParams &kp, const T (*red)[WarpShared<T, GAS, NT>::ROWP],
                                            const bool (&act)[GasShape<GAS>::NS], LaneState<T> &L, T *sum) {
#pragma unroll
  for (int k = 0; k < Row<GAS>::forces(HASQ); k++) {
    sum[k] = red[0][k];
#pragma unroll
    for (int q = 1; q < NT / 32; q++) sum[k] += red[q][k];
  }
  if constexpr (GAS == GAS_N2 && !HASQ) sum[6] = sum[7] = sum[8] = T(0);  // the centre has no terms
  T fs[GasShape<GAS>::NS][3];
  finish_row<T, GAS, HASQ>(kp, sum, act, fs);
  absorb_forces<T, GAS>(kp, fs, L);
}

// A ball in which every step is usual, however it is rounded: all sites
// inside the reference grid, the probe inside the box and the ellipsoid and
// within reach of the target, its candidates those at hand.  Each of these
// is a bound on a function of the centre that changes by at most its
// displacement, so one distance replaces all the tests of a step.
template <typename T> struct Usual {
  T c[3], rho2;        // the ball (rho2 < 0: none)
  T hd2lo, hd2hi;      // the pair distance within half a percent of its constrained value
};

// The ball around c for the candidates at hand: a list (built around c, good
// within LSKIN of it), or all atoms; everyone: all atoms whatever the distance.
template <typename T, int GAS>
__device__ __noinline__ T usual_radius2(const KParams *__restrict__ kpg, T cx, T cy, T cz, bool list, bool everyone) {
  const KParams &kp = *kpg;
  const KConst<T> &kc = kconst<T>(kp);
  const T offm = GAS == GAS_ATOM ? T(0) : T(0.5) * T(sqrt(kc.d2)), offlo = offm * T(0.995), offhi = offm * T(1.005);
  const T c[3] = {cx, cy, cz};
  T e2 = T(0), f2 = T(0), u2 = T(0), rho = T(1e6);
  const T half[3] = {kc.lx, kc.ly, kc.lz}, inv[3] = {kc.inv_a, kc.inv_b, kc.inv_c};
  for (int k = 0; k < 3; k++) {
    const T lo = kc.bb_lo[k] - c[k], hi = c[k] - kc.bb_hi[k];
    const T e = fmax(fmax(lo, hi), T(0)), f = fmax(-lo, -hi);
    e2 += e * e;
    f2 += f * f;
    u2 += c[k] * inv[k] * c[k] * inv[k];
    rho = fmin(rho, fmin(kp.ref_check ? kc.ref_lim[k] - offhi : T(1e6), half[k]) - fabs(c[k]));
  }
  rho = fmin(rho, (T(1) - sqrt(u2)) / fmax(fmax(inv[0], inv[1]), inv[2]));
  if (!kp.allpairs) {
    const T rin = kc.reach + offlo, rout = kc.reach + offhi + T(0.01);
    rho = fmin(rho, rin - sqrt(e2));
    if (list) rho = fmin(rho, sqrt(f2) - rout);
    else if (!everyone) rho = fmin(rho, rin - sqrt(f2));
  }
  rho -= T(2e-3);  // far more than any rounding here or there
  if (!(rho > T(0))) return T(-1);
  return list && rho >= T(LSKIN) ? T(LSKIN) * T(LSKIN) : rho * rho;
}

enum : int { F_OTHER = 0, F_TEST = 1, F_WIDE = 2 };

// Usual steps, one after another: the probe in the ball, its candidates
// known (mode), no end of the try.  Few branches, so that little stands
// between the forces and the next positions.  One copy of the integrator for
// all roles: every warp of the CTA computes the same bits and takes the same
// turns; only the step's angle, which nothing waits for, is one warp's (the
// role with the least to sum) and reaches the others with the forces.
// Returns F_OTHER: a step whose move is done and which is not usual; F_TEST:
// after a step, an exit test or the periodic check is due; F_WIDE: the same
// with the step's angle still to do.
template <typename T, int GAS, bool HASQ, int NT>
__device__ __forceinline__ int usual_steps(int role, const KParams &kp, LaneState<T> &L, T inv_dt, const Usual<T> &us,
                                           int mode, const Cand &cd, const Atom<T> (&sa)[2], int vt, int lane, int v,
                                           WarpShared<T, GAS, NT> &sm, int &red, unsigned &it) {
  constexpr int NS = GasShape<GAS>::NS;
  constexpr int ANGLE_ROLE = GAS == GAS_N2 && HASQ ? 2 : 0;
  for (;;) {
    first_half_move<T, GAS>(kp, L, inv_dt);
    const T c[3] = {centre<T, GAS>(L, 0), centre<T, GAS>(L, 1), centre<T, GAS>(L, 2)};
    const T dcx = c[0] - us.c[0], dcy = c[1] - us.c[1], dcz = c[2] - us.c[2];
    const T moved2 = Real<T>::fma(dcz, dcz, Real<T>::fma(dcx, dcx, Real<T>::mul(dcy, dcy)));
    bool ok = moved2 <= us.rho2;
    if constexpr (GAS != GAS_ATOM) {
      const T hd[3] = {L.r1[0] - L.r2[0], L.r1[1] - L.r2[1], L.r1[2] - L.r2[2]};
      const T hd2 = dot3(hd, hd);
      ok &= (hd2 >= us.hd2lo) & (hd2 <= us.hd2hi);
    }
    if (!ok) return F_OTHER;
    T p[NS][3];
    site_positions<T, GAS>(L, p);
    T f[3] = {T(0), T(0), T(0)}, E[3] = {T(0), T(0), T(0)}, G[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    step_visits<T, GAS, HASQ, NT>(kp, role, p, (1u << NS) - 1u, mode, cd, sa, vt, f, E, G);
    if (role == ANGLE_ROLE && v == 0) {
      bool wide;
      const T ang = small_angle(c, L.rold, wide);
      if (lane == 0) {
        sm.ang[red] = ang;
        sm.wide[red] = wide;
      }
    }
    step_reduce<T, GAS, HASQ>(role, f, E, G, lane, sm.red[red][v]);
    __syncthreads();
    bool act[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) act[k] = true;
    T sum[Row<GAS>::N];
    step_forces<T, GAS, HASQ, NT>(kp, sm.red[red], act, L, sum);
    const T ang = sm.ang[red];
    const bool wide = sm.wide[red] != 0;
    red ^= 1;
    L.nvis += (uint32_t)cd.m;
    second_kick<T, GAS>(kp, L);
    it++;
    if (wide) return F_WIDE;
    L.dtheta += ang;
#pragma unroll
    for (int k = 0; k < 3; k++) L.rold[k] = c[k];
    if ((L.dtheta > T(1.5 * PI_D)) | (L.stepcount >= kp.max_steps) | ((it & 255u) == 0)) return F_TEST;
  }
}

// The ball around c in which the probe is out of reach of the whole target
// and inside the box and the ellipsoid: a free flight.
template <typename T, int GAS>
__device__ __noinline__ T free_radius2(const KParams *__restrict__ kpg, T cx, T cy, T cz) {
  const KParams &kp = *kpg;
  const KConst<T> &kc = kconst<T>(kp);
  if (kp.allpairs) return T(-1);
  const T c[3] = {cx, cy, cz};
  T e2 = T(0), u2 = T(0), rho = T(1e6);
  const T half[3] = {kc.lx, kc.ly, kc.lz}, inv[3] = {kc.inv_a, kc.inv_b, kc.inv_c};
  for (int k = 0; k < 3; k++) {
    const T e = fmax(fmax(kc.bb_lo[k] - c[k], c[k] - kc.bb_hi[k]), T(0));
    e2 += e * e;
    u2 += c[k] * inv[k] * c[k] * inv[k];
    rho = fmin(rho, half[k] - fabs(c[k]));
  }
  const T offhi = GAS == GAS_ATOM ? T(0) : T(0.5 * 1.005) * T(sqrt(kc.d2));
  rho = fmin(rho, (T(1) - sqrt(u2)) / fmax(fmax(inv[0], inv[1]), inv[2]));
  rho = fmin(rho, sqrt(e2) - (kc.reach + offhi + T(0.01))) - T(2e-3);
  return rho > T(0) ? rho * rho : T(-1);
}

// Steps of a free flight: no force, no barrier.  Returns as usual_steps.
template <typename T, int GAS>
__device__ __forceinline__ int free_steps(const KParams &kp, LaneState<T> &L, T inv_dt, const Usual<T> &us, unsigned &it) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    L.f1[k] = T(0);
    if constexpr (GAS != GAS_ATOM) L.f2[k] = T(0);
  }
  for (;;) {
    first_half_move<T, GAS>(kp, L, inv_dt);
    const T c[3] = {centre<T, GAS>(L, 0), centre<T, GAS>(L, 1), centre<T, GAS>(L, 2)};
    const T dcx = c[0] - us.c[0], dcy = c[1] - us.c[1], dcz = c[2] - us.c[2];
    bool ok = dcx * dcx + dcy * dcy + dcz * dcz <= us.rho2;
    if constexpr (GAS != GAS_ATOM) {
      const T hd[3] = {L.r1[0] - L.r2[0], L.r1[1] - L.r2[1], L.r1[2] - L.r2[2]};
      const T hd2 = dot3(hd, hd);
      ok &= (hd2 >= us.hd2lo) & (hd2 <= us.hd2hi);
    }
    if (!ok) return F_OTHER;
    bool wide;
    const T ang = small_angle(c, L.rold, wide);
    second_kick<T, GAS>(kp, L);
    it++;
    if (wide) return F_WIDE;
    L.dtheta += ang;
#pragma unroll
    for (int k = 0; k < 3; k++) L.rold[k] = c[k];
    if ((L.dtheta > T(1.5 * PI_D)) | (L.stepcount >= kp.max_steps) | ((it & 255u) == 0)) return F_TEST;
  }
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

// CTAs per SM that the register allocation must allow, FP32: CTAs of up to
// 128 threads share an SM by threes (168 registers: four candidates side by
// side and the integrator's state fit), larger ones by twos (128).  Measured
// against 512 threads an SM throughout: one lone step of N2 1.52 -> 1.33 us,
// CO2 1.33 -> 1.19, He globule 0.81 -> 0.74; warp pass of n2_protein_3k 41 ->
// 35 ms, co2_protein_9k 93 -> 82, n2_protein_150k (queue full for a third of
// it) 360 -> 363; one CTA of 256 threads an SM takes n2_complex_20k from 260
// to 300.  FP64 is unconstrained.
template <typename T, int GAS, bool HASQ, int NT> struct WarpShape {
  static constexpr int THREADS = NT * Roles<GAS, HASQ>::N;
  static constexpr int MINB = sizeof(T) == 8 ? 1 : THREADS <= 128 ? 384 / THREADS : THREADS <= 256 ? 2 : 1;
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
  __shared__ WarpShared<T, GAS, NT> sm;
  __shared__ __align__(16) unsigned char sm_kp[BATCH ? sizeof(KParams) : 16];  // this trajectory's ion
  extern __shared__ __align__(16) unsigned char dyn[];
  // candidate list: indices, then (kp.wp_pack) the packed candidates in list order
  int *const sm_list = reinterpret_cast<int *>(dyn);
  float4 *const sm_pos = reinterpret_cast<float4 *>(dyn + (((size_t)kp.wp_cap * 4 + 15) & ~size_t(15)));
  float2 *const sm_ab = reinterpret_cast<float2 *>(sm_pos + kp.wp_pack);
  float2 *const sm_abc = sm_ab + kp.wp_pack;
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
    // its atoms stay in registers (atomic gases) or, as without cutoffs, packed
    const bool insmall = GAS == GAS_ATOM && small;
    const bool packall = packs && !insmall && (small || K.allpairs) && K.natoms <= kp.wp_cap;
    Atom<T> sa[2] = {far_atom<T>(), far_atom<T>()};
    Cand cd{sm_pos, sm_ab, sm_abc, sm_list, sm.ljm[v], false, 0};
    if (insmall) {
#pragma unroll
      for (int i = 0; i < 2; i++)
        if (vt + i * NT < K.natoms) sa[i] = fetch<T, GAS, C_ALL, true>(K, cd, vt + i * NT);
    }
    if (packall) {
      for (int t = tid; t < K.natoms; t += NTHREADS) pack_atom<T, GAS>(K, t, t, sm_pos, sm_ab, sm_abc);
      pack_end<GAS, NT>(K.natoms, tid, NTHREADS, sm_pos, sm_ab, sm_abc);
      __syncthreads();
    }
    Usual<T> us;
    us.rho2 = T(-1);
    us.c[0] = us.c[1] = us.c[2] = T(0);
    us.hd2lo = kc.d2 * T(0.995 * 0.995);
    us.hd2hi = kc.d2 * T(1.005 * 1.005);
    int mode = C_NONE;
    bool usual = false;  // the next step may be a usual one
    bool us_list = false, us_free = false;
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
      if (r == S_CONTINUE && usual && L.mode == M_STEP) {
        const int u = us_free ? free_steps<T, GAS>(K, L, inv_dt, us, it)
                              : usual_steps<T, GAS, HASQ, NT>(role, K, L, inv_dt, us, mode, cd, sa, vt, lane, v, sm,
                                                              red, it);
        if (u == F_WIDE) turn<T, GAS>(L);
        if (u != F_OTHER) {
          it--;  // the loop's own count
          r = exit_test<T, GAS>(K, L, false);
          if (r == S_CONTINUE) continue;
        }
      }
      if (r == S_CONTINUE) {
        bool out = false;
        if (L.mode == M_STEP) {
          if (!usual) first_half_move<T, GAS>(K, L, inv_dt);
          turn<T, GAS>(L);
          out = step_leaves(K, L);
        }
        usual = false;
        const bool want_u = L.mode == M_INIT || out;
        L.U = T(0);
        T p[NS][3];
        site_positions<T, GAS>(L, p);
        const T cx = p[S::cs][0], cy = p[S::cs][1], cz = p[S::cs][2];
        const T ex = fmax(fmax(kc.bb_lo[0] - cx, cx - kc.bb_hi[0]), T(0));
        const T ey = fmax(fmax(kc.bb_lo[1] - cy, cy - kc.bb_hi[1]), T(0));
        const T ez = fmax(fmax(kc.bb_lo[2] - cz, cz - kc.bb_hi[2]), T(0));
        const T fx = fmax(cx - kc.bb_lo[0], kc.bb_hi[0] - cx);
        const T fy = fmax(cy - kc.bb_lo[1], kc.bb_hi[1] - cy);
        const T fz = fmax(cz - kc.bb_lo[2], kc.bb_hi[2] - cz);
        const T e2 = ex * ex + ey * ey + ez * ez, f2 = fx * fx + fy * fy + fz * fz;
        const T dcx = cx - list_c[0], dcy = cy - list_c[1], dcz = cz - list_c[2];
        const T moved2 = Real<T>::fma(dcz, dcz, Real<T>::fma(dcx, dcx, Real<T>::mul(dcy, dcy)));
        const bool keep = list_n >= 0 && !(moved2 > T(LSKIN) * T(LSKIN));
        unsigned actbits;
        bool chunked = false;
        T R = T(0);
        cd.m = K.natoms;
        const bool near = probe_near<T, GAS>(K, p, actbits);
        if (near) {
          const T off = site_offset<T, GAS>(p);
          R = K.allpairs ? T(INFINITY) : kc.reach + off + T(1e-3);
          if (small || f2 <= R * R) {
            // the whole target inside the reach sphere, or a small target:
            // every atom is a candidate (the cutoff tests are exact)
            mode = insmall ? C_NONE : packall ? C_PACK : C_ALL;
            cd.masked = false;
          } else if (e2 <= R * R) {
            if (!keep) {
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
                if (packs) pack_end<GAS, NT>(list_n, tid, NTHREADS, sm_pos, sm_ab, sm_abc);
                __syncthreads();
              }
            }
            mode = packs ? C_PACK : C_LIST;
            cd.masked = true;
            cd.m = list_n;
            chunked = list_n < 0;
          } else {
            mode = C_ALL;
            cd.m = 0;  // no atom in reach
          }
        }
        if (near) {
          bool act[NS];
#pragma unroll
          for (int s = 0; s < NS; s++) act[s] = (actbits >> s) & 1u;
          T af[3] = {T(0), T(0), T(0)}, aE[3] = {T(0), T(0), T(0)}, aG[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
          uint32_t nvis;
          if (chunked) {
            nvis = for_chunks<T, NT, RF>(K, cx, cy, cz, R, lead, lane, v, sm_list, lcap, sm.wsum, [&](int *l, int n) {
              Cand cc = cd;
              cc.masked = false;
              cc.m = n;
              step_visits<T, GAS, HASQ, NT>(K, role, p, actbits, C_LIST, cc, sa, vt, af, aE, aG);
            });
          } else {
            step_visits<T, GAS, HASQ, NT>(K, role, p, actbits, mode, cd, sa, vt, af, aE, aG);
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
            warp_energy<T, GAS, HASQ, NT, RF>(Kg, ps, chunked, cx, cy, cz, R, chunked || cd.masked ? sm_list : nullptr, cd.m,
                                          lcap, lead, lane, v, sm.wsum, row);
          }
          __syncthreads();
          T sum[Row<GAS>::N];
          step_forces<T, GAS, HASQ, NT>(K, sm.red[red], act, L, sum);
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
          // the ball for the next steps: around the list's centre, or this position
          usual = !chunked && cd.m > 0 && L.mode == M_STEP;
          if (usual && (!cd.masked || us_free || list_c[0] != us.c[0] || list_c[1] != us.c[1] || list_c[2] != us.c[2] || !us_list)) {
            us_list = cd.masked;
            us_free = false;
            us.c[0] = us_list ? list_c[0] : cx;
            us.c[1] = us_list ? list_c[1] : cy;
            us.c[2] = us_list ? list_c[2] : cz;
            us.rho2 = usual_radius2<T, GAS>(Kg, us.c[0], us.c[1], us.c[2], us_list, small);
          }
          usual = usual && us.rho2 > T(0);
        } else {
          T fs[NS][3];
#pragma unroll
          for (int s = 0; s < NS; s++) fs[s][0] = fs[s][1] = fs[s][2] = T(0);
          absorb_forces<T, GAS>(K, fs, L);
          if (L.mode == M_STEP && !out) {
            us_free = true;
            us.c[0] = cx; us.c[1] = cy; us.c[2] = cz;
            us.rho2 = free_radius2<T, GAS>(Kg, cx, cy, cz);
            usual = us.rho2 > T(0);
          }
        }
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
      usual = false;
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
