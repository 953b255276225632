// The active particles' substeps of one MPCD step in a single kernel (both forms).
//
// Between two SRD collisions only the particles whose straight path may meet a sphere need
// the colloids' positions substep by substep; every other particle is streamed through the
// whole step by the free-flight pass.  k_near_step64 / k_near_step32 take the active ones
// (a few per cent of the fluid) through all n_sub substeps: one block per SM, launched
// cooperatively, each with its share of the active particles in shared memory and its share
// of the colloids.  A block has two groups of warps that meet only at grid-wide counters:
//
//   particle warps, substep l                  colloid warps, substep l
//     wait: every colloid has moved to X(l)      wait: the same
//     the listed particles' exact collisions     WCA forces at X(l)
//     count the block in (BAR_COLL)              wait: every block is through its collisions
//     stream to l + 1, list what may collide     exchange, V, Omega, X(l + 1)
//     (FP32 test against X(l) + margin)          count the block in (BAR_MOVE)
//     their draws, which no position enters
//
// A launch per stage (near pass, event pass, colloid finish) spends 3 to 4 us per substep and
// stage on launch latency and ramps, and reads the particles' state again each time; here a
// stage boundary is one counter in L2 (about 1 us), the state stays on the SM, and the
// streaming of l + 1 runs while the colloids of l are finished.  Bound: the latency of that
// cycle (fence and counter 1.2 us twice, exact collisions 2 us FP32 / 4 us FP64, colloid finish
// 2 us), and with that the rate at which the code of a cycle is fetched: what is rarely taken is
// out of line, and the common test runs two particles at a time without a branch.  Measured per
// step, before it -> with it and the passes around it as they are now: 24^3 FP32 system (30
// colloids) 204 -> 131 us, 20^3 FP64 (20 colloids) 251 -> 164 us, 64^3 (500 colloids) FP32
// 390 -> 269 us, FP64 605 -> 450 us, 128^3 FP32 (2,000 colloids, 20 substeps) 3.08 -> 1.41 ms;
// 32 FP32 systems of 16^3 to 48^3 stepped together, each on blocks of its own, 2.29 -> 1.59 ms.
// Which systems take it: near_sized in context.cu.
//
// The arithmetic is that of the per-substep passes, in their order: the results are theirs
// bit for bit.  The candidates of a particle come from the flight table of its cell (every
// colloid that can come near in the step) with the reference's box rule (in_block) instead of
// a cell table rebuilt each substep (where a cell lists more than it holds, with it: near_list).
// Waits are bounded: one that runs out sets ERRB_WAIT and its group returns.
#pragma once
#include "device.cuh"

namespace bgb {

constexpr int NEAR_CW = 3;         // colloid warps of a block (and one for the orientations)

// a particle's candidate colloids for the rest of the step, packed: up to two ids (0xFFFF:
// none); NEAR_WILD: look the tables up in every substep (near_list); NEAR_GONE: kept elsewhere
constexpr unsigned NEAR_NONE = 0xFFFFFFFFu, NEAR_WILD = 0xFFFEFFFEu, NEAR_GONE = 0xFFFDFFFDu,
                   NEAR_STALE = 0xFFFCFFFCu;  // (after a collision: to be looked up)

// ---------------------------------------------------------------- waiting

static __device__ __forceinline__ void group_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// counts the block in; called by one thread after a group_sync, so that what the group's
// threads did before it is visible to whoever sees the count
static __device__ __forceinline__ void bar_arrive(unsigned *c) {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
}

static __device__ __forceinline__ bool bar_wait(const unsigned *c, unsigned target, int polls) {
  for (int it = 0; it < polls; ++it) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
    if (v >= target) return true;
  }
  return false;
}

// one thread polls, the group follows; false where the wait ran out.  At least one group_sync
// lies between two calls of a group (the flag is read after the first one).
static __device__ __forceinline__ bool group_wait(const SysF64 &S, int which, unsigned target, int t, int id, int n,
                                                  volatile int *flag) {
  if (t == 0) {
    const bool ok = bar_wait(S.bar + which, target, S.near_polls);
    if (!ok) atomicOr(&S.ss->err, ERRB_WAIT);
    *flag = ok ? 1 : 0;
  }
  group_sync(id, n);
  return *flag != 0;
}

// lets the kernel behind this one (the free-flight pass) start: it then finds every block of this
// one on its SM, and fills what room they leave instead of taking theirs
static __device__ __forceinline__ void near_let_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- candidates

// The colloids that may matter to a particle of cell lin in substep g of this step: the flight table's, or
// where it lists more than it holds, the cell table's of that substep, which such a step builds;
// brute: all colloids (an aliased cell).  (Scanning all of them in crowded cells, too: 300 spheres of
// radius 0.5 in a cube of side 12, 5,532 us a step FP64 and 2,882 FP32; this 395 and 333, a launch per
// stage 357 and 250.  With 28 ids a flight cell, whose lists are longer than the cell tables', 411 and 352.)
struct NearList {
  const uint16_t *ids;
  int cnt;
  bool brute;
};

// the cell table's (rare, out of line)
static __device__ __noinline__ int near_table(const SysF64 &S, long long g, int lin) {
  return min(tcount(S.Tcnt[g & 1][lin], g), TCAP);
}

static __device__ __forceinline__ NearList near_list(const SysF64 &S, long long step, long long g, int lin, bool alias) {
  NearList q;
  q.ids = nullptr;
  q.cnt = 0;
  q.brute = alias || lin >= S.C;
  if (!q.brute) {
    const FlightCell *fc = S.ftab + lin;
    q.ids = fc->id;
    q.cnt = tcount(fc->tc, step);
    if (q.cnt > FLIGHT_CAP) {
      q.ids = S.Tlist[g & 1] + (size_t)lin * TCAP;
      q.cnt = near_table(S, g, lin);
    }
  }
  return q;
}

// the next colloid after `last`, in ascending order, whose neighbour boxes (of its cell in the
// substep before, buffer prev) hold the cell lin = (ix, iy, iz), or -1; alias: lin is not that
// cell's number, and the box rule goes by the numbers
struct NearCell {
  int lin, ix, iy, iz;
  bool alias;
};

static __device__ __forceinline__ bool near_in_block(const SysF64 &S, int j, const NearCell &c, int prev) {
  return c.alias ? in_block(S, S.cbox[prev][j], c.lin) : in_block3(S, S.ccell[prev][j], c.ix, c.iy, c.iz);
}

static __device__ __forceinline__ int near_next(const SysF64 &S, const NearList &q, int last, const NearCell &c,
                                                int prev) {
  if (q.brute) {
    for (int j = last + 1; j < S.Nc; ++j)
      if (near_in_block(S, j, c, prev)) return j;
    return -1;
  }
  for (;;) {
    int best = 0x7FFFFFFF;
    for (int k = 0; k < q.cnt; ++k) {
      const int j = q.ids[k];
      if (j > last && j < best) best = j;
    }
    if (best == 0x7FFFFFFF) return -1;
    if (near_in_block(S, best, c, prev)) return best;
    last = best;
  }
}

// radius a particle's straight path over `rem` substeps must reach to need the substeps: the
// sphere, what a colloid may move meanwhile (and a substep more on either side, the margins
// of the FP32 tests), and a slack for FP32 rounding
static __device__ __forceinline__ float near_radius(const SysF64 &S, float cm, int rem) {
  return S.r_coll + (float)(rem + 2) * cm + 0.02f;
}

// does the path r + t w, t in [0, 1], come within rad of the origin (true for what is not finite)
static __device__ __forceinline__ bool path_meets(float rx, float ry, float rz, float wx, float wy, float wz,
                                                  float rad) {
  const float ww = wx * wx + wy * wy + wz * wz, rw = rx * wx + ry * wy + rz * wz;
  float t = ww > 0.f ? -rw / ww : 0.f;
  t = fminf(fmaxf(t, 0.f), 1.f);
  const float dx = rx + t * wx, dy = ry + t * wy, dz = rz + t * wz;
  return !(dx * dx + dy * dy + dz * dz > rad * rad);
}

// add colloid j to a packed candidate pair
static __device__ __forceinline__ unsigned near_add(unsigned cand, int j) {
  if (cand == NEAR_WILD || j >= 0xFFFC) return NEAR_WILD;
  if ((cand & 0xFFFFu) == 0xFFFFu) return (cand & 0xFFFF0000u) | (unsigned)j;
  if ((cand >> 16) == 0xFFFFu) return (cand & 0xFFFFu) | ((unsigned)j << 16);
  return NEAR_WILD;
}

// An asynchronous 16-byte copy from global to shared memory (through L2: what the grid-wide
// counters have made visible there is what arrives), and the wait for this thread's copies
static __device__ __forceinline__ void near_copy16(void *to, const void *from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}
static __device__ __forceinline__ void near_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The colloids around a block's active particles, kept in shared memory for the tests of the next
// substep: seeing BAR_MOVE empties the SM's L1, so each test would otherwise wait for L2 again
// (three to four dependent 0.4 us reads a substep).  T: what a test needs of a colloid.  The first
// MAX colloids noted are kept; any other is read from global memory.
template <typename T>
struct NearCols {
  static constexpr int MAX = 192, TAB = 2048;
  T d[MAX];
  int at_[TAB];  // colloid -> slot (-1: none)
  uint16_t id[MAX];
  int n;
  __device__ __forceinline__ void clear(const SysF64 &S, int t, int nt) {
    if (t == 0) n = 0;
    for (int j = t; j < min(S.Nc, TAB); j += nt) at_[j] = -1;
  }
  // the candidates of a packed pair get slots
  __device__ __forceinline__ void note(unsigned cand) {
    if (cand == NEAR_WILD) return;
    for (int k = 0; k < 2; ++k, cand >>= 16) {
      const int j = (int)(cand & 0xFFFFu);
      if (j >= TAB || at_[j] != -1 || atomicCAS(&at_[j], -1, -2) != -1) continue;  // (none is beyond the table)
      const int i = atomicAdd(&n, 1);
      if (i >= MAX) continue;
      id[i] = (uint16_t)j;
      at_[j] = i;
    }
  }
  // the pair by slots; NEAR_WILD where one has none
  __device__ __forceinline__ unsigned slots(unsigned cand) const {
    if (cand == NEAR_WILD) return NEAR_WILD;
    unsigned r = NEAR_NONE;
    for (int k = 0; k < 2; ++k, cand >>= 16) {
      const int j = (int)(cand & 0xFFFFu);
      if (j == 0xFFFF) continue;
      const int i = j < TAB ? at_[j] : -1;
      if (i < 0) return NEAR_WILD;
      r = near_add(r, i);
    }
    return r;
  }
  __device__ __forceinline__ int kept() const { return min(n, MAX); }
  __device__ __forceinline__ void load(const SysF64 &S, int b, int t, int nt) {
    for (int i = t; i < kept(); i += nt) d[i] = T::get(S, b, id[i]);
  }
  __device__ __forceinline__ void copy(const SysF64 &S, int b, int t, int nt) {
    for (int i = t; i < kept(); i += nt) T::copy(S, b, id[i], &d[i]);
  }
  // colloid j (positions in buffer b)
  __device__ __forceinline__ T at(const SysF64 &S, int b, int j) const {
    const int i = j < TAB ? at_[j] : -1;
    return i >= 0 ? d[i] : T::get(S, b, j);
  }
};

// append run() candidate records, one atomic per warp (the whole warp calls it)
static __device__ __forceinline__ void near_record(const SysF64 &S, const ShellRec &rec, bool has) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(FULL, has);
  if (!m) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(&S.ss->nshell, __popc(m));
  base = __shfl_sync(FULL, base, 0);
  if (!has) return;
  const int i = base + __popc(m & ((1u << lane) - 1u));
  if (i < S.shell_cap) S.shell[i] = rec;
  else atomicOr(&S.ss->err, ERRB_SHELL);
}

// ---------------------------------------------------------------- colloids

// The forces of a block's colloids, their pairs packed into full warps.
struct NearPairs {
  static constexpr int CAP = 96, COL = 32;  // pairs of a round, and its colloids
  double f[CAP][3];
  uint16_t j[CAP], k[CAP];  // the colloid (its number in the round) and its partner
  uint8_t hit[CAP];
  int first[COL], cnt[COL];  // a colloid's pairs (cnt < 0: it was summed by itself)
  int n;
};

// compute_force_md at X[cur] for the block's colloids s (VB + G s), by the colloid group.  An FP64
// instruction takes the SM's FP64 unit for 16 cycles however few of its lanes are active, and a
// colloid has a partner or two within the cutoff: a warp per colloid (wca_force_vlist) spends 110 such
// instructions on one or two lanes.  So the partners that pass the FP32 test are listed first, the
// pairs then take a lane each, and each colloid's thread adds its own in ascending partner order:
// wca_force_vlist's terms in its order.  (One colloid: that directly, without the two barriers.  A
// colloid with more than 32 listed partners, or beyond the round's room: itself, too.)
// Measured, us a step once the colloids are in contact (from about 1,000 steps on), with the listed
// second spheres of the collisions: 64^3 FP32 (3 colloids a block) 303 -> 281, 128^3 FP32 (13) 1,661 ->
// 1,566, 53x37x41 FP64 at volume fraction 0.2 (3) 353 -> 344.
static __device__ __forceinline__ void near_forces(const SysF64 &S, NearPairs &pr, int VB, int G, int M, int cur, int t,
                                                   int bar_id) {
  constexpr int NT = 32 * NEAR_CW;
  const int lane = t & 31, w = t >> 5;
  if (!S.vlist) {  // (no list: one colloid)
    if (t == 0) stv(S.fnew, VB, mk(0, 0, 0));
    group_sync(bar_id, NT);
    return;
  }
  if (M == 1) {
    if (w == 0) {
      const d3 fn = wca_force_vlist(S, S.X[cur], S.Xf[cur], VB, lane);
      if (lane == 0) stv(S.fnew, VB, fn);
    }
    group_sync(bar_id, NT);
    return;
  }
  const float Lx = S.Lxf, Ly = S.Lyf, Lz = S.Lzf, rc2 = S.rcf * S.rcf;
  const float iLx = __frcp_rn(Lx), iLy = __frcp_rn(Ly), iLz = __frcp_rn(Lz);
  const float4 *Xf = S.Xf[cur];
  for (int s0 = 0; s0 < M; s0 += NearPairs::COL) {
    const int m = min(NearPairs::COL, M - s0);
    if (t == 0) pr.n = 0;
    group_sync(bar_id, NT);
    for (int c = w; c < m; c += NEAR_CW) {
      const int j = VB + G * (s0 + c), n = min(S.nbr_n[j], NBR_CAP);
      bool cand = false;
      int k = 0;
      if (lane < n) {
        k = S.nbr[(size_t)j * NBR_CAP + lane];
        const float4 xj = Xf[j], xk = Xf[k];
        const float dx = wrapf_r(xj.x - xk.x, Lx, iLx), dy = wrapf_r(xj.y - xk.y, Ly, iLy),
                    dz = wrapf_r(xj.z - xk.z, Lz, iLz);
        cand = dx * dx + dy * dy + dz * dz < rc2;
      }
      const unsigned mc = __ballot_sync(FULL, cand);
      const int cnt = __popc(mc);
      int first = 0;
      if (lane == 0 && cnt && n <= 32) first = atomicAdd(&pr.n, cnt);
      first = __shfl_sync(FULL, first, 0);
      const bool self = n > 32 || first + cnt > NearPairs::CAP;
      if (cand && n <= 32) {
        const int at = first + __popc(mc & ((1u << lane) - 1u));
        if (at < NearPairs::CAP) {
          pr.j[at] = (uint16_t)(self ? 0xFFFF : c);  // (0xFFFF: room that a colloid summed by itself had taken)
          pr.k[at] = (uint16_t)k;
        }
      }
      if (lane == 0) {
        pr.first[c] = first;
        pr.cnt[c] = self ? -1 : cnt;
      }
      if (self) {
        const d3 fn = wca_force_vlist(S, S.X[cur], Xf, j, lane);
        if (lane == 0) stv(S.fnew, j, fn);
      }
    }
    group_sync(bar_id, NT);
    for (int i = t; i < min(pr.n, NearPairs::CAP); i += NT) {
      const int c = pr.j[i];
      if (c == 0xFFFF) continue;
      d3 ff = mk(0, 0, 0);
      double pt = 0;
      pr.hit[i] = wca_pair(S, ldv(S.X[cur], VB + G * (s0 + c)), S.X[cur], pr.k[i], false, ff, pt);
      pr.f[i][0] = ff.x; pr.f[i][1] = ff.y; pr.f[i][2] = ff.z;
    }
    group_sync(bar_id, NT);
    if (t < m && pr.cnt[t] >= 0) {
      d3 f = mk(0, 0, 0);
      for (int i = pr.first[t]; i < pr.first[t] + pr.cnt[t]; ++i)
        if (pr.hit[i]) f = add3(f, mk(pr.f[i][0], pr.f[i][1], pr.f[i][2]));
      stv(S.fnew, VB + G * (s0 + t), f);
    }
    group_sync(bar_id, NT);
  }
}

// The colloid group of a block (t: thread of the group): colloids VB, VB + G, ... through the
// substeps.  A colloid has eight lanes (four colloids a warp): lane k < 3 the linear component
// k, lane 3 + k the angular one, so that an FP64 instruction, which occupies the SM's FP64 unit
// for 16 cycles however few lanes are active, serves four colloids; k_fin's operations in its
// order.  *fin: the last substep whose Omega the orientation warp may use.
static __device__ __forceinline__ void near_colloids(const SysF64 &S, NearPairs &pr, const int VB, const int G, const int t,
                                                     const int bar_id, volatile int *flag, volatile int *fin) {
  constexpr int NT = 32 * NEAR_CW;
  const int M = VB < S.Nc ? (S.Nc - VB + G - 1) / G : 0;
  if (M == 0) return;
  const int n = S.n_sub, lane = t & 31, w = t >> 5;
  const int k8 = lane & 7;
  const bool lin = k8 < 3;
  const int k = lin ? k8 : (k8 < 6 ? k8 - 3 : 0);
  const unsigned Gm = (unsigned)(G < S.Nc ? G : S.Nc);
  const long long step = S.ss->step, g0 = step * n;
  const double cm2 = S.ss->cm2;
  const bool crowd = S.ss->crowd == step + 1;
  const Dim &D = k == 0 ? S.dx : (k == 1 ? S.dy : S.dz);
  const int Lk = k == 0 ? S.Lx : (k == 1 ? S.Ly : S.Lz);
  for (int l = 1; l <= n; ++l) {
    const long long g = g0 + (l - 1);
    const int cur = (int)(g & 1), nxt = cur ^ 1;
    if (l > 1 && !group_wait(S, BAR_MOVE, Gm * (unsigned)(l - 1), t, bar_id, NT, flag)) break;
    // compute_force_md at X(l)
    near_forces(S, pr, VB, G, M, cur, t, bar_id);
    if (!group_wait(S, BAR_COLL, (unsigned)G * (unsigned)l, t, bar_id, NT, flag)) break;
    // end of fluid_colloid_collision, update_velocity_colloid, then update_pos_md of l + 1
    for (int s0 = 4 * w; s0 < M; s0 += 4 * NEAR_CW) {
      const int s = s0 + (lane >> 3);
      const bool on = s < M && k8 < 6;
      const int j = VB + G * (s < M ? s : 0);
      double v = 0, f = 0, xo = 0;
      if (on) {
        v = lin ? S.V[3 * j + k] : S.W[3 * j + k];
        if (lin) {
          f = S.f[3 * j + k];
          xo = S.X[cur][3 * j + k];
        }
        ExchAcc *e = S.exch + j;
        const double x = __dadd_rn((double)e->hi[k8] * 0x1p-20, (double)e->lo[k8] * 0x1p-72);
        e->hi[k8] = 0;
        e->lo[k8] = 0;
        const double dp = __dmul_rn(x, S.mass_fl);
        S.xacc[6 * j + k8] += dp;
        v = __dadd_rn(v, __dmul_rn(dp, lin ? S.inv_mc : S.inv_ic));
        if (lin) {
          const double fn = S.fnew[3 * j + k];
          v = __dadd_rn(v, __dmul_rn(__dadd_rn(f, fn), S.dtb2));
          f = fn;
        }
      }
      if (on) {
        if (lin) {
          S.V[3 * j + k] = v;
          S.f[3 * j + k] = f;
        } else {
          S.W[3 * j + k] = v;
          S.w_all[(size_t)(l - 1) * 3 * S.Nc + 3 * j + k] = v;
        }
      }
      if (l == n) continue;
      double xn = 0, e2 = 0;
      float oc = 0.f, of = 0.f;
      if (on && lin) {
        xn = ref_mod(__dadd_rn(xo, __dadd_rn(__dmul_rn(v, S.dt), __dmul_rn(f, S.ddt))), D);
        const double ex = ref_img(__dsub_rn(xn, xo), D);
        e2 = __dmul_rn(ex, ex);
        S.X[nxt][3 * j + k] = xn;
        // the FP32 form's copy: integer cell and offset (colloid_q, one component per lane)
        const double fl = floor(xn);
        of = (float)(xn - fl);
        int ci = (int)fl;
        if (of >= 1.f) { of = 0.f; ci += 1; }
        if (ci < 0 || ci >= Lk) {
          ci %= Lk;
          if (ci < 0) ci += Lk;
        }
        oc = (float)ci;
      }
      const double d2 = __shfl_sync(FULL, e2, 0, 8) + __shfl_sync(FULL, e2, 1, 8) + __shfl_sync(FULL, e2, 2, 8);
      const d3 Xn = mk(__shfl_sync(FULL, xn, 0, 8), __shfl_sync(FULL, xn, 1, 8), __shfl_sync(FULL, xn, 2, 8));
      const float c1 = __shfl_sync(FULL, oc, 1, 8), c2 = __shfl_sync(FULL, oc, 2, 8);
      const float o1 = __shfl_sync(FULL, of, 1, 8), o2 = __shfl_sync(FULL, of, 2, 8);
      if (on && k8 == 0) {
        if (d2 > cm2) atomicOr(&S.ss->err, ERRB_DISPLACE);
        S.Xf[nxt][j] = make_float4((float)Xn.x, (float)Xn.y, (float)Xn.z, 0.f);
        const int cb = colloid_cell(S, Xn);
        S.cbox[nxt][j] = cb;
        S.ccell[nxt][j] = cell_coords(S, cb);
        S.Xcq[nxt][j] = make_float4(oc, c1, c2, 0.f);
        S.Xco[nxt][j] = make_float4(of, o1, o2, 0.f);
      }
    }
    group_sync(bar_id, NT);
    if (t == 0) {
      __threadfence_block();
      *fin = l;  // (the orientation warp follows)
    }
    if (l == n) return;
    // the cell table of substep g + 2 (those of the step's first two are k_fin's): near_list reads it once this
    // count is complete, and its capacity is checked as in the per-substep passes.  (It takes the place of
    // substep g's, whose collisions are over in every block.)
    if (crowd) {
      for (int j = VB; j < S.Nc; j += G) table_of(S, j, g + 2, t, NT);
      group_sync(bar_id, NT);
    }
    if (t == 0) bar_arrive(S.bar + BAR_MOVE);
  }
  if (t == 0) *fin = -1;  // (a wait ran out)
}

// The orientations of the block's colloids (one warp, lane of it: lane): update_activity_direction
// of every substep in turn, as soon as the colloid warps have finished it.  Nothing before the
// end of the step reads the orientation, so its chain (60 dependent FP64 operations a substep)
// runs at its own pace beside theirs.  Lane k < 3 of a colloid's eight takes component k, with
// activity_rot's operations for it.
static __device__ __forceinline__ void near_orient(const SysF64 &S, const int VB, const int G, const int lane,
                                                   volatile int *fin) {
  const int M = VB < S.Nc ? (S.Nc - VB + G - 1) / G : 0;
  const int k8 = lane & 7, k = k8 < 3 ? k8 : 0;
  for (int l = 1; l <= S.n_sub && M > 0; ++l) {
    int f = 0;
    for (int it = 0; it < S.orient_polls; ++it) {
      f = *fin;
      if (f < 0 || f >= l) break;
      __nanosleep(64);
    }
    if (!__all_sync(FULL, f >= l)) {
      // this wait ran out, or (f < 0, reported already) one of the colloid warps'
      if (lane == 0) atomicOr(&S.ss->err, ERRB_WAIT);
      return;
    }
    __threadfence_block();
    for (int s0 = 0; s0 < M; s0 += 4) {
      const int s = s0 + (lane >> 3);
      const bool on = s < M && k8 < 3;
      const int j = VB + G * (s < M ? s : 0);
      const size_t at = (size_t)(l - 1) * 3 * S.Nc + 3 * j + k;
      double sn = 0, co = 0, ra = 0, xi = 0;
      if (on) {
        sincos_small(__dmul_rn(S.w_all[at], S.dt), &sn, &co);
        ra = S.ra[3 * j + k];
        if (S.Dr > 0) xi = S.xi_all[at];
      }
      const d3 sb = mk(__shfl_sync(FULL, sn, 0, 8), __shfl_sync(FULL, sn, 1, 8), __shfl_sync(FULL, sn, 2, 8));
      const d3 cb = mk(__shfl_sync(FULL, co, 0, 8), __shfl_sync(FULL, co, 1, 8), __shfl_sync(FULL, co, 2, 8));
      d3 r3 = mk(__shfl_sync(FULL, ra, 0, 8), __shfl_sync(FULL, ra, 1, 8), __shfl_sync(FULL, ra, 2, 8));
      d3 m;
      if (k == 0) {
        m = mk(__dmul_rn(cb.y, cb.z), __dmul_rn(-cb.y, sb.z), sb.y);
      } else {
        // rows 2 and 3: (-+p sb.y) with p the sine / cosine of x, as activity_rot writes them
        const double p = k == 1 ? sb.x : -cb.x, q = k == 1 ? cb.x : sb.x;
        m = mk(__dadd_rn(__dmul_rn(__dmul_rn(p, sb.y), cb.z), __dmul_rn(q, sb.z)),
               __dadd_rn(__dmul_rn(__dmul_rn(-p, sb.y), sb.z), __dmul_rn(q, cb.z)),
               k == 1 ? __dmul_rn(-sb.x, cb.y) : __dmul_rn(cb.x, cb.y));
      }
      ra = dot_ref(m, r3);
      if (S.Dr > 0) {
        r3 = mk(__shfl_sync(FULL, ra, 0, 8), __shfl_sync(FULL, ra, 1, 8), __shfl_sync(FULL, ra, 2, 8));
        const d3 x3 = mk(__shfl_sync(FULL, xi, 0, 8), __shfl_sync(FULL, xi, 1, 8), __shfl_sync(FULL, xi, 2, 8));
        const double xa = dot_ref(x3, r3);
        const double a = __dadd_rn(ra, __dmul_rn(__dsub_rn(xi, __dmul_rn(ra, xa)), S.rotdiff_s));
        const d3 a3 = mk(__shfl_sync(FULL, a, 0, 8), __shfl_sync(FULL, a, 1, 8), __shfl_sync(FULL, a, 2, 8));
        ra = __ddiv_rn(a, __dsqrt_rn(norm2_ref(a3.x, a3.y, a3.z)));
      }
      if (on) S.ra[3 * j + k] = ra;
    }
  }
}

// completes a step: bumps the step counter (tables: the cell table of the next step's first substep is built)
static __device__ __forceinline__ void k_end_step_body(const SysF64 &S, const int VB, bool tables) {
  if (VB != 0) return;
  if (threadIdx.x == 0 && tables) S.ss->tab = (S.ss->step + 1) * S.n_sub;
  // run()'s shell counts start from zero for the next step (its rear-shell test runs beside
  // the next step's cell pass, so the cell pass cannot clear them)
  for (int j = threadIdx.x; j < S.Nc; j += blockDim.x) S.shell_cnt[j] = 0;
  if (S.Nc > 0) {
    // the next step's colloid margin: twice the largest displacement a substep gives at
    // the colloids' present speeds, within [0.005, the static bound], and never below the
    // move the FP64 form's next first streaming pass assumes (from the last substep's
    // positions to the present ones, already checked against this step's margin; from the
    // FP32 copies of the positions, plus 2e-5 for their rounding).  A colloid that moves
    // further in a substep fails the step (the finish checks every move), so the FP32
    // form's free-flight classification may take n_sub times it as the colloids' move.
    __shared__ float s_vm[32], s_dm[32];
    const long long g = (S.ss->step + 1) * S.n_sub;  // the substep the colloids are at
    const float4 *Fc = S.Xf[g & 1], *Fp = S.Xf[(g - 1) & 1];
    float vm = 0.f, dm = 0.f;
    for (int j = threadIdx.x; j < S.Nc; j += blockDim.x) {
      const float vx = (float)S.V[3 * j], vy = (float)S.V[3 * j + 1], vz = (float)S.V[3 * j + 2];
      vm = fmaxf(vm, vx * vx + vy * vy + vz * vz);
      const float4 a = Fc[j], b = Fp[j];
      const float ex = wrapf(a.x - b.x, S.Lxf), ey = wrapf(a.y - b.y, S.Lyf), ez = wrapf(a.z - b.z, S.Lzf);
      dm = fmaxf(dm, ex * ex + ey * ey + ez * ez);
    }
    for (int o = 16; o > 0; o >>= 1) {
      vm = fmaxf(vm, __shfl_xor_sync(0xFFFFFFFFu, vm, o));
      dm = fmaxf(dm, __shfl_xor_sync(0xFFFFFFFFu, dm, o));
    }
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) {
      s_vm[w] = vm;
      s_dm[w] = dm;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < nw; ++k) {
        vm = fmaxf(vm, s_vm[k]);
        dm = fmaxf(dm, s_dm[k]);
      }
      float cm = fminf(fmaxf(2.f * (float)S.dt * sqrtf(vm), 0.005f), S.cmarginf);
      // (capped: in a step that has failed a colloid may have moved anywhere, and the steps enqueued behind it
      // would take that for the reach of their tables)
      cm = fmaxf(cm, fminf(sqrtf(dm) + 2e-5f, fmaxf(2.f * S.cmarginf, 0.1f)));
      S.ss->cm = cm;
      S.ss->cm2 = (double)cm * (double)cm;
    }
  }
  if (threadIdx.x == 0) S.ss->step += 1;
}

// rotational-diffusion normals of colloid j in every substep of the step (rotdiff_draw's
// operations), one thread per substep, colloid and pair of normals: full warps, so the FP64
// logarithms, sines and cosines cost 1/16 of what they do at two lanes per colloid
static __device__ __forceinline__ void rotdiff_step(const SysF64 &S, long long i) {
  const long long q = i >> 1;
  if (q >= (long long)S.Nc * S.n_sub) return;
  const int l = (int)(q / S.Nc), j = (int)(q % S.Nc), pair = (int)(i & 1);
  const long long g = S.ss->step * S.n_sub + l;
  const uint4 r = draw4(S.key, DOM_ROTDIFF, 0, (uint32_t)(j + 1), 0, (uint32_t)g);
  const uint32_t ur = pair == 0 ? r.x : r.z, ut = pair == 0 ? r.y : r.w;
  const double rr = sqrt(-2.0 * log(u01(ur)));
  double sn, cs;
  sincos(__dmul_rn(S.two_pi, u01(ut)), &sn, &cs);
  double *o = S.xi_all + 3 * q;
  if (pair == 0) {
    o[0] = __dmul_rn(rr, cs);
    o[1] = __dmul_rn(rr, sn);
  } else {
    o[2] = __dmul_rn(rr, cs);
  }
}

}  // namespace bgb
