// FP64 form of the MPCD + active-colloid step (sm_103a).
//
// Data layout (HBM, structure of arrays): fluid positions px/py/pz and per-substep
// displacements w = v*dt (wx/wy/wz) in double; one int per particle for the cell
// of the next SRD binning; per-cell exact sums (CellAcc); the 3x3 map and offset
// of each cell's SRD collision (cell_ab); colloid arrays of a few KB.
//
// Kernels of one MPCD step (one CUDA graph):
//   k_cell_prep   per cell: mean, thermostat factor, random axis -> w' = A w + b
//   k_rotate      per particle: w' = A w + b                      rotation_mpcd
//   k_run_shell   per run() candidate: rear-shell test and count   run
//   k_run_kick    per run() candidate: compensating fluid kick     run
//   k_fin         per colloid (one thread): run()'s colloid kick, update_pos_md
//   then per substep g:
//   k_stream      per particle: streaming, wall collisions with the colloids its cell
//                 table lists, and (last substep) run() candidates and the next SRD
//                 binning (update_pos_mpcd, neighbour_list_mpcd, fluid_colloid_collision);
//                 its first blocks meanwhile compute the WCA forces at the substep's
//                 colloid positions and the cell table of the next substep
//   k_fin         per colloid: end of fluid_colloid_collision, update_activity_direction,
//                 update_velocity_colloid, then update_pos_md of the next substep
#include "../../include/brownian_gb300.h"
#include "near_step.cuh"

namespace bgb {
// One particle's part of the SRD binning for the next step: its cell (recorded
// in rotcell) and the fixed-point w and |w|^2 the exact cell sums add up
struct BinTerm {
  int c;
  long long fx, fy, fz, f2;
};

// (rr: the grid shift of that binning)
__device__ __forceinline__ BinTerm bin_term(const SysF64 &S, const double *rr, int p, double x, double y, double z,
                                            double wx, double wy, double wz) {
  // (1 + mod(pos + rr, len).cell(len), cpp/rotation_mpcd.cpp:11)
  double ax = ref_mod(__dadd_rn(x, rr[0]), S.dx), ay = ref_mod(__dadd_rn(y, rr[1]), S.dy),
         az = ref_mod(__dadd_rn(z, rr[2]), S.dz);
  bool alias;
  BinTerm t;
  t.c = cell_of_pos(S, ax, ay, az, alias);
  S.rotcell[p] = t.c;
  long long ax_ = dbits(wx) & 0x7FFFFFFFFFFFFFFFll, ay_ = dbits(wy) & 0x7FFFFFFFFFFFFFFFll,
            az_ = dbits(wz) & 0x7FFFFFFFFFFFFFFFll;
  if (ax_ > S.wlim_bits || ay_ > S.wlim_bits || az_ > S.wlim_bits) atomicOr(&S.ss->err, ERRB_VRANGE);
  t.fx = to_fix(wx, S.kw); t.fy = to_fix(wy, S.kw); t.fz = to_fix(wz, S.kw);
  t.f2 = sq_fix(t.fx, S.kw) + sq_fix(t.fy, S.kw) + sq_fix(t.fz, S.kw);
  return t;
}

// the exact sums of the SRD binning for the next step: cell number, count, w, |w|^2
__device__ __forceinline__ void bin_for_rotation(const SysF64 &S, int p, double x, double y, double z, double wx,
                                                 double wy, double wz) {
  const BinTerm t = bin_term(S, S.ss->rr, p, x, y, z, wx, wy, wz);
  bin_add(S.acc + t.c, 1, t.fx, t.fy, t.fz, t.f2);
}

// FLAGS: F_* bits.  l: substep (1..n_sub) whose streaming this is; 0 for the
// set-up pass (no streaming; bins for the first step).  fb: the fluid buffer.
//
// Per particle: streaming, then an FP32 scan of the colloids its cell table
// lists.  A particle that may be inside a sphere (or is on the edge of a run()
// shell, or sits in an aliased cell) goes to the event list, which k_events then
// processes with the reference's exact FP64 arithmetic, one event per lane; all
// other particles finish here (shell record, SRD binning on the last substep).
// U particles per thread (thread t of block b: particles b * 256 U + t + 256 u),
// their loads issued together so more memory requests are in flight.  The pass
// that also lists run() shell members keeps more state per particle and one
// particle per thread, for its register count.
#ifndef STREAM64_U
#define STREAM64_U 2
#endif
#ifndef STREAM64_U_SHELL
#define STREAM64_U_SHELL 1
#endif
static constexpr __host__ __device__ int stream64_u(int flags) { return (flags & F_SHELL) ? STREAM64_U_SHELL : STREAM64_U; }
// One chunk of 256 U particles: i = chunk * 256 U + threadIdx.x + 256 u below `count`,
// slot i of the fluid (NEAR false) or slot near[i] (NEAR true: the free-flight schedule's
// passes over the near list).  The whole block calls it.
template <int FLAGS, bool NEAR>
static __device__ __forceinline__ void stream64_chunk(const SysF64 &S, const int chunk, const int count, int l,
                                                      int fb) {
  constexpr int flags = FLAGS;
  constexpr int U = stream64_u(FLAGS);
  const long long step = S.ss->step;
  const long long gs = step * S.n_sub + (l - 1);
  const Fluid F = fluid_at(S, fb);
  const int i0 = chunk * (256 * U) + threadIdx.x;
  const int buf = (int)(gs & 1);
  // F_PIPE: the colloid positions of the previous substep (this substep's are being
  // computed meanwhile) and the displacement bound as margin; pending particles
  // belong to the event passes and are skipped
  const int xb = (flags & F_PIPE) ? (int)((gs - 1) & 1) : buf;
  const float mg = (flags & F_PIPE) ? S.ss->cm : 0.f;

  double x[U], y[U], z[U], wx[U], wy[U], wz[U];
  bool valid[U], ev[U];
  unsigned members[U];  // run() shell members among the cell-table slots
  int cnt[U], lin[U], pp[U];
  uint8_t pd[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int i = i0 + 256 * u;
    valid[u] = i < count;
    ev[u] = false;
    members[u] = 0;
    cnt[u] = 0;
    lin[u] = 0;
    pd[u] = 0;
    pp[u] = i;
    wx[u] = wy[u] = wz[u] = 0;
    if (valid[u]) {
      const int p = NEAR ? S.near[i] : i;
      pp[u] = p;
      x[u] = F.x[p]; y[u] = F.y[p]; z[u] = F.z[p];
      if (flags & (F_STREAM | F_BINROT | F_COLLIDE)) { wx[u] = F.wx[p]; wy[u] = F.wy[p]; wz[u] = F.wz[p]; }
      if (flags & F_PIPE) pd[u] = S.pend[p];
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) valid[u] = valid[u] && pd[u] == 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!valid[u]) continue;
    if (flags & F_STREAM) {
      // update_pos_mpcd: pos = mod(pos + vel*dt, len)   cpp/update.cpp:56-60
      x[u] = ref_mod(__dadd_rn(x[u], wx[u]), S.dx);
      y[u] = ref_mod(__dadd_rn(y[u], wy[u]), S.dy);
      z[u] = ref_mod(__dadd_rn(z[u], wz[u]), S.dz);
    }
    if (flags & (F_COLLIDE | F_SHELL)) {
      bool alias;
      lin[u] = cell_of_pos(S, x[u], y[u], z[u], alias);
      ev[u] = alias;
      if (!alias) cnt[u] = tcount(S.Tcnt[buf][lin[u]], gs);
    }
  }
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (valid[u] && (flags & (F_COLLIDE | F_SHELL)) && cnt[u] > 0) {
      cnt[u] = cnt[u] < TCAP ? cnt[u] : TCAP;
      const uint16_t *lst = S.Tlist[buf] + (size_t)lin[u] * TCAP;
      const float4 *Xf = S.Xf[xb];
      const float px = d2f_trunc(x[u]), py = d2f_trunc(y[u]), pz = d2f_trunc(z[u]);
      const float ch = S.r_coll + 1e-3f + mg, sl = S.r_shell - 1e-3f - mg, sh = S.r_shell + 1e-3f + mg;
      for (int k = 0; k < cnt[u]; ++k) {
        const float4 c = Xf[lst[k]];
        const float dx = wrap_half(c.x - px, S.Lxf), dy = wrap_half(c.y - py, S.Lyf), dz = wrap_half(c.z - pz, S.Lzf);
        const float d2 = dx * dx + dy * dy + dz * dz;
        if (flags & F_COLLIDE) ev[u] |= d2 <= ch * ch;
        if (flags & F_SHELL) {
          if (d2 < sl * sl) members[u] |= 1u << k;
          else ev[u] |= d2 <= sh * sh;
        }
      }
    }
    const int p = pp[u];
    if (valid[u]) {
      if (!ev[u] && (flags & F_BINROT)) bin_for_rotation(S, p, x[u], y[u], z[u], wx[u], wy[u], wz[u]);
      if (flags & F_STREAM) { F.x[p] = x[u]; F.y[p] = y[u]; F.z[p] = z[u]; }
    }
    // the event record, one atomic per warp (no block barrier), written while the
    // particle's state is still in registers
    const unsigned mev = __ballot_sync(FULL, ev[u]);
    int bev = 0;
    if (lane == 0 && mev) bev = atomicAdd(&S.ss->nnew[buf], __popc(mev));
    bev = __shfl_sync(FULL, bev, 0);
    if (ev[u]) {
      const int i = bev + __popc(mev & lt);
      if (i < S.events_cap) {
        EventRec r;
        r.xy = make_double2(x[u], y[u]); r.zwx = make_double2(z[u], wx[u]); r.wywz = make_double2(wy[u], wz[u]);
        r.p = p; r.id = F.id[p];
        S.newrec[buf][i] = r;
        if (flags & F_PIPE) S.pend[p] = 1;
      } else {
        atomicOr(&S.ss->err, ERRB_EVENTS);
      }
    }
  }
  // run() candidate records (last substep), one atomic per block
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!(flags & F_SHELL)) break;
    const int p = pp[u];
    const bool has_rec = valid[u] && !ev[u] && members[u] != 0;
    const unsigned mrec = __ballot_sync(FULL, has_rec);
    const int brec = block_base(&S.ss->nshell, mrec, lane);
    if (has_rec) {
      const int i = brec + __popc(mrec & lt);
      if (i < S.shell_cap) {
        // colloids in ascending index, the order run() visits them
        const uint16_t *lst = S.Tlist[buf] + (size_t)lin[u] * TCAP;
        ShellRec *r = S.shell + i;
        r->p = F.id[p];
        r->pass = 0;
        int n = 0, last = -1;
        for (int it = 0; it < cnt[u] && n < SHELL_J; ++it) {
          int best = 0x7FFFFFFF;
          for (int k = 0; k < cnt[u]; ++k) {
            const int j = lst[k];
            if (((members[u] >> k) & 1u) && j > last && j < best) best = j;
          }
          if (best == 0x7FFFFFFF) break;
          r->j[n++] = (uint16_t)best;
          last = best;
        }
        if (__popc(members[u]) > SHELL_J) atomicOr(&S.ss->err, ERRB_SHELLSLOTS);
        r->n = (uint8_t)n;
      } else {
        atomicOr(&S.ss->err, ERRB_SHELL);
      }
    }
  }
}

// Five blocks per SM (48 registers, a few spilled to L1) measured faster than four
// without spills.
template <int FLAGS>
__global__ void __launch_bounds__(256, 5) k_stream(const SysF64 S, int l, int fb) {
  stream64_chunk<FLAGS, false>(S, blockIdx.x, S.N, l, fb);
}

// the same over the near list of the free-flight schedule (grid-stride over chunks)
template <int FLAGS>
__global__ void __launch_bounds__(256, 5) k_stream_near(const SysF64 S, int l, int fb) {
  const int count = S.ss->nnear;
  constexpr int per = 256 * stream64_u(FLAGS);
  for (int chunk = blockIdx.x; chunk * per < count; chunk += gridDim.x)
    stream64_chunk<FLAGS, true>(S, chunk, count, l, fb);
}

int stream64_per_thread(int flags) { return stream64_u(flags); }

// The particles the streaming pass listed: wall collisions in colloid order with
// the reference's exact arithmetic (and, on the last substep, their run() record
// and SRD binning).  Per round of up to blockDim.x particles (one per thread):
// each thread loads its particle and finds its first collision; then the block's
// collisions are gathered onto its first threads, rank by rank (a particle's
// second collision follows its first), and each particle is finished by its own
// thread.  blockDim.x <= 128.
template <int FLAGS>
static __device__ __forceinline__ void k_events_body(const SysF64 &S, const int VB, const int NVB, int l, int fb) {
  constexpr int flags = FLAGS;
  __shared__ EvState sst[128];
  __shared__ int stask[128];
  __shared__ int sntask;
  __shared__ CollScratch scs[32];
  const long long step = S.ss->step;
  const long long gs = step * S.n_sub + (l - 1);
  const int buf = (int)(gs & 1);
  const Fluid F = fluid_at(S, fb);
  // F_PIPE: items 0..np-1 are the particles pending from earlier substeps of this
  // step (their streaming of this substep is done here), items np.. the ones this
  // substep's streaming pass listed; every item's state goes back to prec[i]
  const int nn = min(S.ss->nnew[buf], S.events_cap);
  const int np = (flags & F_PIPE) ? S.ss->npend : 0;
  int n = np + nn;
  if ((flags & F_PIPE) && n > S.pend_cap) {
    if (VB == 0 && threadIdx.x == 0) atomicOr(&S.ss->err, ERRB_EVENTS);
    n = S.pend_cap;
  }
  // item i goes to block i % NVB: the items of a substep spread over all SMs
  EvState &st = sst[threadIdx.x];
  for (int base = 0;; base += blockDim.x) {
    const int i = VB + NVB * (threadIdx.x + base);
    const bool valid = i < n;
    if (!__syncthreads_or(valid)) break;  // block-uniform trip count
    const bool old = i < np;
    st.j = -1;
    if (valid) {
      const EventRec r = old ? S.prec[i] : S.newrec[buf][i - np];
      double x = r.xy.x, y = r.xy.y, z = r.zwx.x;
      const double wx = r.zwx.y, wy = r.wywz.x, wz = r.wywz.y;
      if ((flags & F_PIPE) && old) {
        // update_pos_mpcd of a pending particle (as the streaming pass does it)
        x = ref_mod(__dadd_rn(x, wx), S.dx);
        y = ref_mod(__dadd_rn(y, wy), S.dy);
        z = ref_mod(__dadd_rn(z, wz), S.dz);
      }
      bool alias;
      const int lin = cell_of_pos(S, x, y, z, alias);
      int cnt = 0;
      if (!alias) {
        cnt = tcount(S.Tcnt[buf][lin], gs);
        cnt = cnt < TCAP ? cnt : TCAP;
      }
      st.x = x; st.y = y; st.z = z; st.wx = wx; st.wy = wy; st.wz = wz;
      st.x0 = x; st.y0 = y; st.z0 = z;
      st.vdx = st.vdy = st.vdz = 0.0;
      st.p = r.p; st.id = r.id; st.lin = lin; st.last = -1; st.cnt = cnt;
      st.alias = alias; st.dumped = false; st.changed = false;
      if (flags & F_COLLIDE) st.j = ev_next_hit(S, st, buf);
    }
    if (flags & F_COLLIDE) {
      for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sntask = 0;
        __syncthreads();
        if (st.j >= 0) stask[atomicAdd(&sntask, 1)] = threadIdx.x;
        __syncthreads();
        const int nt = sntask;
        if (nt == 0) break;
        if (blockDim.x == 128) {
          for (int k0 = 0; k0 < nt; k0 += 32) ev_collide_coop(S, sst, stask, k0, nt, gs, buf, scs);
          if ((int)threadIdx.x < nt) {
            EvState &t = sst[stask[threadIdx.x]];
            t.j = ev_next_hit(S, t, buf);
          }
        } else if ((int)threadIdx.x < nt) {
          EvState &t = sst[stask[threadIdx.x]];
          ev_collide(S, t, t.j, gs, buf);
          t.j = ev_next_hit(S, t, buf);
        }
      }
    }
    __syncthreads();
    if (valid) {
      const int p = st.p;
      if (flags & F_SHELL) {
        ShellRec rec;
        ev_shell(S, st, buf, rec);
        if (rec.n) {
          int idx = atomicAdd(&S.ss->nshell, 1);
          if (idx < S.shell_cap) S.shell[idx] = rec;
          else atomicOr(&S.ss->err, ERRB_SHELL);
        }
      }
      if (flags & F_BINROT) bin_for_rotation(S, p, st.x, st.y, st.z, st.wx, st.wy, st.wz);
      if ((flags & F_PIPE) || st.changed) {
        F.x[p] = st.x; F.y[p] = st.y; F.z[p] = st.z;
        F.wx[p] = st.wx; F.wy[p] = st.wy; F.wz[p] = st.wz;
      }
      if (flags & F_PIPE) {
        EventRec o;
        o.xy = make_double2(st.x, st.y); o.zwx = make_double2(st.z, st.wx); o.wywz = make_double2(st.wy, st.wz);
        o.p = p; o.id = st.id;
        S.prec[i] = o;
      }
    }
    __syncthreads();  // the next round reuses the shared state
  }
}

template <int FLAGS>
__global__ void __launch_bounds__(128) k_events(const SysF64 S, int l, int fb) {
  k_events_body<FLAGS>(S, blockIdx.x, gridDim.x, l, fb);
}

// the event pass (blocks 0..nevb-1) and, after them, the colloid side work of the same
// substep (colloid_aux: forces and orientation, two colloids per block of four warps),
// which needs only the positions the colloid finish of the substep before computed: one
// launch where the side work would take a second stream per substep
template <int FLAGS>
__global__ void __launch_bounds__(128) k_events_aux(const SysF64 S, int l, int fb, int nevb, int act) {
  if ((int)blockIdx.x < nevb) {
    k_events_body<FLAGS>(S, blockIdx.x, nevb, l, fb);
    return;
  }
  const int j = 2 * ((int)blockIdx.x - nevb) + (threadIdx.x >> 6);
  const long long gs = S.ss->step * S.n_sub + (l - 1);
  if (j < S.Nc) colloid_aux(S, gs, j, act != 0, (threadIdx.x >> 5) & 1, 2, S.vlist != 0);
}

// The SRD binning of the particles the last streaming pass of a step finished
// (the pending ones are binned by the event pass): a pass of its own, so that
// its atomics run beside that substep's event pass and colloid finish.  Pending
// marks stay set until the next step's rotation clears them.
// Particles sit in cell order (sorted every sort_every steps), so a warp's particles
// fall into a few cells of the shifted grid: their terms are summed per cell across the
// warp first (bin_add_warp), one set of atomics per cell and warp.
__global__ void __launch_bounds__(256) k_bin(const SysF64 S, int fb) {
  const Fluid F = fluid_at(S, fb);
  for (int base = blockIdx.x * blockDim.x; base < S.N; base += gridDim.x * blockDim.x) {
    const int p = base + threadIdx.x;
    BinTerm t{-1, 0, 0, 0, 0};
    if (p < S.N && !S.pend[p]) t = bin_term(S, S.ss->rr, p, F.x[p], F.y[p], F.z[p], F.wx[p], F.wy[p], F.wz[p]);
    bin_add_warp(S.acc, t.c, t.fx, t.fy, t.fz, t.f2);
  }
}

// ------------------------------------------------------------ free-flight schedule
// (the FP64 form's kernels; the schedule and the flight table are described with the FP32
// form's, kernels_fp32c.cu)

// the last substep's binning of the near particles the streaming pass finished (pending
// ones are binned by the event pass)
__global__ void __launch_bounds__(256) k_bin_near(const SysF64 S, int fb) {
  const Fluid F = fluid_at(S, fb);
  const int count = S.ss->nnear;
  for (int base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    BinTerm t{-1, 0, 0, 0, 0};
    if (i < count) {
      const int p = S.near[i];
      if (!S.pend[p]) t = bin_term(S, S.ss->rr, p, F.x[p], F.y[p], F.z[p], F.wx[p], F.wy[p], F.wz[p]);
    }
    bin_add_warp(S.acc, t.c, t.fx, t.fy, t.fz, t.f2);
  }
}

// rotation_mpcd of one particle (w' = A w + b of its cell, as k_rotate; ROT false: a
// counting-sort step, whose scatter rotated it) and its classification against the flight
// table: a near particle is flagged and listed (one atomic per block).  SPLIT: of the near
// ones, those whose straight path may meet a sphere are also listed as active (k_near_step64).
template <bool ROT, bool SPLIT>
__global__ void __launch_bounds__(256) k_rotate_classify(const SysF64 S, int fb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < S.N;
  const Fluid F = fluid_at(S, fb);
  const long long step = S.ss->step;
  const int b0 = (int)((step * S.n_sub - 1) & 1);
  bool near = false;
  unsigned cand = NEAR_NONE;  // (SPLIT: the colloids its path comes near)
  if (valid) {
    if (!SPLIT) S.pend[p] = 0;  // no particle is pending at the start of a step
    const int c = ROT ? S.rotcell[p] : S.C;
    double wx = F.wx[p], wy = F.wy[p], wz = F.wz[p];
    const float px = d2f_trunc(F.x[p]), py = d2f_trunc(F.y[p]), pz = d2f_trunc(F.z[p]);
    int cx = (int)px, cy = (int)py, cz = (int)pz;  // positions in (0, L]: L is cell 0
    cx -= cx == S.Lx ? S.Lx : 0; cy -= cy == S.Ly ? S.Ly : 0; cz -= cz == S.Lz ? S.Lz : 0;
    // a position outside the box (a state that is not finite) reads no table: near
    const bool inb = cx >= 0 && cx < S.Lx && cy >= 0 && cy < S.Ly && cz >= 0 && cz < S.Lz;
    const FlightCell *fc = S.ftab + (inb ? cx + S.Lx * (cy + S.Ly * cz) : 0);
    const uint4 w0 = reinterpret_cast<const uint4 *>(fc)[0];
    if (c < S.C) {
      const double2 *ab = reinterpret_cast<const double2 *>(S.cell_ab + (size_t)c * 12);
      double2 a01 = ab[0], a23 = ab[1], a45 = ab[2], a67 = ab[3], a8b0 = ab[4], b12 = ab[5];
      const double nx = fma(a01.x, wx, fma(a01.y, wy, fma(a23.x, wz, a8b0.y)));
      const double ny = fma(a23.y, wx, fma(a45.x, wy, fma(a45.y, wz, b12.x)));
      const double nz = fma(a67.x, wx, fma(a67.y, wy, fma(a8b0.x, wz, b12.y)));
      wx = nx; wy = ny; wz = nz;
      F.wx[p] = wx; F.wy[p] = wy; F.wz[p] = wz;
    }
    // n_sub |w| = ndt |v| (FP32 copies by truncation, on the integer pipe: below 2^-23 of
    // the travel under it, which the slack covers)
    const float fx = d2f_trunc(wx), fy = d2f_trunc(wy), fz = d2f_trunc(wz);
    const float travel = (float)S.n_sub * sqrtf(fx * fx + fy * fy + fz * fz);
    int cnt = tcount(((unsigned long long)w0.y << 32) | w0.x, step);
    if (!inb || !(travel <= S.flight_rv) || cnt > FLIGHT_CAP) {
      near = true;  // faster than the table allows (or not finite), or a crowded cell
      cand = NEAR_WILD;
    } else if (cnt > 0) {
      const float r = S.r_shell + travel + (float)S.n_sub * S.ss->cm + 0.01f, r2 = r * r;
      const float rad = near_radius(S, S.ss->cm, S.n_sub), fn = (float)S.n_sub;
      if (r > S.near_img) {  // (a box as narrow as that: other copies of the spheres matter)
        near = true;
        cand = NEAR_WILD;
        cnt = 0;
      }
      // (four ids lie in the first half of the record)
      const uint4 w1 = cnt > 4 ? reinterpret_cast<const uint4 *>(fc)[1] : make_uint4(0, 0, 0, 0);
      const unsigned ids[6] = {w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      const float4 *Xf = S.Xf[b0];
      for (int k = 0; k < cnt; ++k) {
        const int j = (int)((ids[k >> 1] >> (16 * (k & 1))) & 0xFFFFu);
        const float4 q = Xf[j];
        const float dx = wrap_half(q.x - px, S.Lxf), dy = wrap_half(q.y - py, S.Lyf), dz = wrap_half(q.z - pz, S.Lzf);
        if (!(dx * dx + dy * dy + dz * dz > r2)) {
          near = true;
          if (SPLIT && path_meets(-dx, -dy, -dz, fn * fx, fn * fy, fn * fz, rad)) cand = near_add(cand, j);
        }
      }
    }
    S.fnear[p] = near ? (SPLIT && cand != NEAR_NONE ? FN_ACTIVE : FN_NEAR) : FN_FREE;
  }
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(FULL, near);
  const unsigned lt = (1u << lane) - 1u;
  int base, ba;
  if (SPLIT) {
    const bool active = cand != NEAR_NONE;
    const unsigned ma = __ballot_sync(FULL, active);
    block_base2(&S.ss->nnear, __popc(m), __popc(ma), lane, &base, &ba);
    if (active) {
      S.act[ba + __popc(ma & lt)] = p;
      S.actc[ba + __popc(ma & lt)] = cand;
    }
  } else {
    base = block_base_n(&S.ss->nnear, __popc(m), lane);
  }
  if (near) S.near[base + __popc(m & lt)] = p;
}

// n substeps of update_pos_mpcd along one axis for a free particle: x = mod(x + w, L) n
// times (cpp/update.cpp:56-60), with the result of the additions one by one.  x > 0 has
// the unit u = ulp(x) of its binade [2^e, 2^(e+1)); w/u = Mw 2^-s (Mw the significand of w).
// While an exact sum x + w lies inside that binade, the nearest double to it is x plus the
// multiple of u nearest to w, k u with k = round(Mw 2^-s), the same k at every addition
// unless w/u is exactly halfway between two integers (then ties-to-even would depend on x).
// So while the results x + j k u stay at least u inside the binade (the exact sums then lie
// inside it) and inside [2^-30 L, L), where mod is the identity, j additions give x + j k u,
// built here on the integer pipe from the bits (the FP64 units stay free for the substeps'
// chains).

// the additions one by one, as the reference does them
static __device__ __forceinline__ double seq(double x, double w, int n, const Dim &D) {
#pragma unroll 1
  for (int q = 0; q < n; ++q) x = ref_mod(__dadd_rn(x, w), D);
  return x;
}

// All n steps at once where they lie in one run, without a branch: with x1 = fl(x + w) in the
// binade of x (and no tie), x1 - x is the k u of the run above, as a difference of bit patterns
// k, and the result's pattern is x's plus n k, if that too lies inside the binade (not on its
// lower edge) and inside [2^-30 L, L).  Else x stays and the result is false.  One FP64 addition
// and about 30 integer instructions an axis, the three axes independent of one another; it
// applies to 98.9 % of axis moves, and the rest take the additions one by one (seq, a single
// copy of it: the pass runs at the rate its instructions are fetched).  Measured, the 64^3
// system's step (density 10, 500 colloids; the pass beside the substeps' kernel): runs of steps
// between crossings, with branches and inlined per axis, 593 us; this 461 us.
static __device__ __forceinline__ bool free_jump(double &x, double w, int n, const Dim &D) {
  const long long bx = dbits(x), b1 = dbits(__dadd_rn(x, w)), aw = dbits(w) & 0x7FFFFFFFFFFFFFFFll;
  const long long bn = (long long)((unsigned long long)bx + ((unsigned long long)b1 - (unsigned long long)bx) * n);
  // (the same sign and exponent, x1's checked so that n k cannot have wrapped)
  const bool in = (((b1 ^ bx) | (bn ^ bx)) >> 52) == 0 && (bn & 0xFFFFFFFFFFFFFll) != 0 && bx >= D.lo_bits &&
                  bn >= D.lo_bits && bx < D.L_bits && bn < D.L_bits && n <= 1024;
  // w / u halfway between two integers: the fraction of w's significand below u is one half
  const int sh = (int)(bx >> 52) - (int)(aw >> 52);
  const unsigned long long mw = ((unsigned long long)aw & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const bool tie = sh >= 1 && sh <= 53 && (mw << (64 - sh)) == 0x8000000000000000ull;
  const bool ok = in && !tie;
  if (ok) x = __longlong_as_double(bn);
  return ok;
}

// the free particles' whole step: update_pos_mpcd of every substep (free_jump, or seq on the axes
// it does not cover: the streaming passes' operations in order, or their exact result) and the
// binning of the last substep with the next step's grid shift, beside the near particles'
// substeps, which touch none of its particles.  A grid of a few blocks per SM walks the fluid
// (it shares the SMs with the substeps' latency-bound chain), each thread's next particle loaded
// while this one is worked on.
// (thr: the flag from which on a particle is not this pass's: 1, or 2 where the near ones that
// no sphere can reach are streamed here too)
__global__ void __launch_bounds__(256, 4) k_free_flight(const SysF64 S, int fb, int thr) {
  const Fluid F = fluid_at(S, fb);
  const int n = S.n_sub, stride = gridDim.x * blockDim.x;
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  double x = 0, y = 0, z = 0, wx = 0, wy = 0, wz = 0;
  int fn = 255;
  auto load = [&](int q) {
    fn = 255;
    if (q < S.N) {
      fn = S.fnear[q];
      x = F.x[q]; y = F.y[q]; z = F.z[q];
      wx = F.wx[q]; wy = F.wy[q]; wz = F.wz[q];
    }
  };
  load(p);
  for (int p0 = p - (int)threadIdx.x; p0 < S.N; p0 += stride, p += stride) {
    const bool free = fn < thr;
    double ax = x, ay = y, az = z;
    const double bx = wx, by = wy, bz = wz;
    load(p + stride);
    BinTerm t{-1, 0, 0, 0, 0};
    if (free) {
      const bool ox = free_jump(ax, bx, n, S.dx), oy = free_jump(ay, by, n, S.dy), oz = free_jump(az, bz, n, S.dz);
      // the axes it does not cover, one a lane at a time
      unsigned left = (ox ? 0u : 1u) | (oy ? 0u : 2u) | (oz ? 0u : 4u);
      while (left) {
        const int a = __ffs(left) - 1;
        left &= left - 1;
        const double sel = a == 0 ? ax : a == 1 ? ay : az, sw = a == 0 ? bx : a == 1 ? by : bz;
        const Dim &D = a == 0 ? S.dx : a == 1 ? S.dy : S.dz;
        const double r = seq(sel, sw, n, D);
        if (a == 0) ax = r;
        else if (a == 1) ay = r;
        else az = r;
      }
      t = bin_term(S, S.ss->rrn, p, ax, ay, az, bx, by, bz);
      F.x[p] = ax; F.y[p] = ay; F.z[p] = az;
    }
    bin_add_warp(S.acc, t.c, t.fx, t.fy, t.fz, t.f2);  // the whole warp
  }
}

EventAuxKernel event_aux_kernel(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE | F_PIPE: return k_events_aux<F_COLLIDE | F_PIPE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT | F_PIPE: return k_events_aux<F_COLLIDE | F_SHELL | F_BINROT | F_PIPE>;
  }
  return nullptr;
}

ClassifyKernel classify_kernel(bool rotate, bool split) {
  return rotate ? (split ? k_rotate_classify<true, true> : k_rotate_classify<true, false>)
                : (split ? k_rotate_classify<false, true> : k_rotate_classify<false, false>);
}

StreamKernel stream_kernel_near(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE | F_PIPE: return k_stream_near<F_STREAM | F_COLLIDE | F_PIPE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT | F_PIPE:
      return k_stream_near<F_STREAM | F_COLLIDE | F_SHELL | F_PIPE>;
  }
  return nullptr;
}

StreamKernel stream_kernel(int flags) {
  // substeps run overlapped (F_PIPE; the last one's binning is k_bin); the set-up
  // pass stands alone; the routine-by-routine substep streams (F_STREAM) and tests
  // for wall collisions (F_COLLIDE) in passes of their own
  switch (flags) {
    case F_STREAM | F_COLLIDE | F_PIPE: return k_stream<F_STREAM | F_COLLIDE | F_PIPE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT | F_PIPE:
      return k_stream<F_STREAM | F_COLLIDE | F_SHELL | F_PIPE>;
    case F_SHELL | F_BINROT: return k_stream<F_SHELL | F_BINROT>;
    case F_STREAM: return k_stream<F_STREAM>;
    case F_COLLIDE: return k_stream<F_COLLIDE>;
  }
  return nullptr;
}

// colloid_aux of substep l (1..n_sub) as a kernel of its own (blocks of
// S.aux_nw warps, one colloid each); `act`: with the pending orientation update
// of substep l-1
static __device__ __forceinline__ void k_aux_body(const SysF64 &S, const int VB, const int NVB, int l, int act,
                                                  bool vlist = false) {
  const long long gs = S.ss->step * S.n_sub + (l - 1);
  if ((int)VB < S.Nc) colloid_aux(S, gs, VB, act != 0, threadIdx.x >> 5, S.aux_nw, vlist);
}

// (vl: the forces from the step's pair list, the free-flight schedule)
__global__ void __launch_bounds__(256) k_aux(__grid_constant__ const SysF64 S, int l, int act, int vl) {
  k_aux_body(S, blockIdx.x, gridDim.x, l, act, vl != 0);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_aux_b(const SysF64 *Ss, const int *boff, int nrep, int l, int act) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_aux_body(sS, VB, NVB, l, act); });
}

EventKernel event_kernel(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE | F_PIPE: return k_events<F_COLLIDE | F_PIPE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT | F_PIPE: return k_events<F_COLLIDE | F_SHELL | F_BINROT | F_PIPE>;
    case F_SHELL | F_BINROT: return k_events<F_SHELL | F_BINROT>;
    case F_COLLIDE: return k_events<F_COLLIDE>;
  }
  return nullptr;
}

// ------------------------------------------------------------- SRD collision

// Per cell: the SRD collision of rotation_mpcd (cpp/rotation_mpcd.cpp:14-49) as
// one affine map of the cell's displacements, w' = u + s R (w - u) = A w + b,
// A = s R, b = u - A u.  u is the cell mean, R the rotation by theta about the
// cell's random axis (rho, phi), s the thermostat factor; the variance the
// reference computes after rotating equals sum|w - u|^2 = S2 - n|u|^2 before.
// Consumes (and clears) the exact sums k_stream accumulated.
__global__ void __launch_bounds__(256) k_cell_prep(const SysF64 S, int sort) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  CellAcc a = CellAcc{0, 0, 0, 0, 0, 0};
  if (c < S.Cpad) {
    a = S.acc[c];
    S.acc[c] = CellAcc{0, 0, 0, 0, 0, 0};
    if (sort) S.cursor[c] = 0;
  }
  // counting sort, first half: exclusive prefix of the occupancy within this block
  // of 256 cells, and the block's total
  if (sort) {
    __shared__ int wsum[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v = a.n, incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int before = 0, total = 0;
    for (int q = 0; q < 8; ++q) {
      before += q < w ? wsum[q] : 0;
      total += wsum[q];
    }
    if (c < S.Cpad) S.cell_off[c] = before + incl - v;
    if (threadIdx.x == 0) S.blk_off[blockIdx.x] = total;
  }
  if (c >= S.C) return;
  double *ab = S.cell_ab + (size_t)c * 12;
  int n = a.n;
  if (n > S.max_per_cell) atomicOr(&S.ss->err, ERRB_OCCUPANCY);
  if (n <= 1 || n > S.max_per_cell) {
    ab[0] = 1; ab[1] = 0; ab[2] = 0; ab[3] = 0; ab[4] = 1; ab[5] = 0; ab[6] = 0; ab[7] = 0; ab[8] = 1;
    ab[9] = 0; ab[10] = 0; ab[11] = 0;
    return;
  }
  // (sx 2^-kw) / n in one product: the power-of-two scaling is exact, so this is the same
  // rounding of the same exact product
  const double insw = S.insw_n[n];
  double ux = (double)a.sx * insw, uy = (double)a.sy * insw, uz = (double)a.sz * insw;
  double s2 = (double)a.s2 * S.inv_sw;
  double var = s2 - (double)n * (ux * ux + uy * uy + uz * uz);
  // sqrt(cs (n - 1) / var) as sqrt(cs (n - 1)) (per n, from the host) times 1/sqrt(var): within
  // a few ulp of the quotient's root, and no double division on the FP64 pipe
  double s = var > 0 ? S.sqcs_n[n] * rsqrt(var) : 1.0;
  // rotation axis: rho = 2 ran - 1, phi = 4 asin(1) ran (cpp/rotation_mpcd.cpp:19-20); the sine
  // and cosine of phi = pi (2 ran) from sincospi (2 ran is exact), within an ulp of sincos(phi)
  uint4 r = draw4(S.key, DOM_AXIS, 0, (uint32_t)(c + 1), 0, (uint32_t)(S.ss->step + 1));
  double rho = pm1(r.x);
  double sp, cp;
  sincospi(2.0 * u01(r.y), &sp, &cp);
  double sq = sqrt(1.0 - rho * rho);
  double r1 = cp * sq, r2 = sp * sq, r3 = rho;
  double ct = S.ct, st = S.st, ict = S.ict;
  double i1 = ict * r1, i2 = ict * r2, i3 = ict * r3;
  double R[9] = {i1 * r1 + ct, i1 * r2 - st * r3, i1 * r3 + st * r2,
                 i2 * r1 + st * r3, i2 * r2 + ct, i2 * r3 - st * r1,
                 i3 * r1 - st * r2, i3 * r2 + st * r1, i3 * r3 + ct};
#pragma unroll
  for (int k = 0; k < 9; ++k) ab[k] = s * R[k];
  ab[9] = ux - (ab[0] * ux + ab[1] * uy + ab[2] * uz);
  ab[10] = uy - (ab[3] * ux + ab[4] * uy + ab[5] * uz);
  ab[11] = uz - (ab[6] * ux + ab[7] * uy + ab[8] * uz);
}

// counting sort, second half: exclusive prefix of the block totals (one block)
static __device__ __forceinline__ void k_scan_blocks_body(const SysF64 &S, const int VB, const int NVB, int nblk) {
  __shared__ int wsum[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nblk; base += 1024) {
    int i = base + threadIdx.x;
    int v = i < nblk ? S.blk_off[i] : 0, incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int before = carry, total = 0;
    for (int q = 0; q < 32; ++q) {
      before += q < w ? wsum[q] : 0;
      total += wsum[q];
    }
    __syncthreads();
    if (i < nblk) S.blk_off[i] = before + incl - v;
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024) k_scan_blocks(__grid_constant__ const SysF64 S, int nblk) {
  k_scan_blocks_body(S, blockIdx.x, gridDim.x, nblk);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(1024) k_scan_blocks_b(const SysF64 *Ss, const int *boff, int nrep, int nblk) {
  __shared__ SysF64 sS;
  // each system's own block count
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_scan_blocks_body(sS, VB, NVB, (sS.Cpad + 255) / 256); });
}

// The SRD collision applied to each particle, w' = A w + b of its cell, and the
// particle written, rotated, to its slot of the other buffer in cell order (the
// slot within a cell is taken with one atomic per group of equal cells in a warp).
__global__ void __launch_bounds__(256) k_rotate_sort(const SysF64 S, int src, int dst) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= S.N) return;
  S.pend[p] = 0;  // no particle is pending at the start of a step
  const Fluid F = fluid_at(S, src), G = fluid_at(S, dst);
  const int c = S.rotcell[p];
  double wx = F.wx[p], wy = F.wy[p], wz = F.wz[p];
  if (c < S.C) {
    const double2 *ab = reinterpret_cast<const double2 *>(S.cell_ab + (size_t)c * 12);
    double2 a01 = ab[0], a23 = ab[1], a45 = ab[2], a67 = ab[3], a8b0 = ab[4], b12 = ab[5];
    double nx = fma(a01.x, wx, fma(a01.y, wy, fma(a23.x, wz, a8b0.y)));
    double ny = fma(a23.y, wx, fma(a45.x, wy, fma(a45.y, wz, b12.x)));
    double nz = fma(a67.x, wx, fma(a67.y, wy, fma(a8b0.x, wz, b12.y)));
    wx = nx; wy = ny; wz = nz;
  }
  const unsigned act = __activemask();
  const unsigned grp = __match_any_sync(act, c);
  const int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&S.cursor[c], __popc(grp));
  base = __shfl_sync(grp, base, leader);
  const int slot = S.blk_off[c >> 8] + S.cell_off[c] + base + __popc(grp & ((1u << lane) - 1u));
  const int id = F.id[p];
  // occupancy and rotcell come from the same binning pass, so slots form a
  // permutation of 0..N-1; anything else is reported, never written
  if (slot < 0 || slot >= S.N || id < 0 || id >= S.N) {
    atomicOr(&S.ss->err, ERRB_OCCUPANCY);
    return;
  }
  G.x[slot] = F.x[p]; G.y[slot] = F.y[p]; G.z[slot] = F.z[p];
  G.wx[slot] = wx; G.wy[slot] = wy; G.wz[slot] = wz;
  G.id[slot] = id;
  S.newpos[id] = slot;
}

// The SRD collision applied in place, w' = A w + b of the particle's cell (the
// steps between two sorts).
__global__ void __launch_bounds__(256) k_rotate(const SysF64 S, int fb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= S.N) return;
  S.pend[p] = 0;  // no particle is pending at the start of a step
  const int c = S.rotcell[p];
  if (c >= S.C) return;
  const Fluid F = fluid_at(S, fb);
  const double2 *ab = reinterpret_cast<const double2 *>(S.cell_ab + (size_t)c * 12);
  double2 a01 = ab[0], a23 = ab[1], a45 = ab[2], a67 = ab[3], a8b0 = ab[4], b12 = ab[5];
  double wx = F.wx[p], wy = F.wy[p], wz = F.wz[p];
  F.wx[p] = fma(a01.x, wx, fma(a01.y, wy, fma(a23.x, wz, a8b0.y)));
  F.wy[p] = fma(a23.y, wx, fma(a45.x, wy, fma(a45.y, wz, b12.x)));
  F.wz[p] = fma(a67.x, wx, fma(a67.y, wy, fma(a8b0.x, wz, b12.y)));
}

// candidates of a particle for its next `rem` substeps, packed: the colloids its straight path
// comes near, from the flight table of its cell (positions in buffer b); NEAR_WILD where that
// does not cover them
static __device__ __forceinline__ unsigned near_cand64(const SysF64 &S, long long step, int rem, int b, double x,
                                                       double y, double z, double wx, double wy, double wz) {
  const float px = d2f_trunc(x), py = d2f_trunc(y), pz = d2f_trunc(z);
  int cx = (int)px, cy = (int)py, cz = (int)pz;  // positions in (0, L]: L is cell 0
  cx -= cx == S.Lx ? S.Lx : 0; cy -= cy == S.Ly ? S.Ly : 0; cz -= cz == S.Lz ? S.Lz : 0;
  if (!(cx >= 0 && cx < S.Lx && cy >= 0 && cy < S.Ly && cz >= 0 && cz < S.Lz)) return NEAR_WILD;
  const float fr = (float)rem;
  const float fx = fr * d2f_trunc(wx), fy = fr * d2f_trunc(wy), fz = fr * d2f_trunc(wz);
  const float travel = sqrtf(fx * fx + fy * fy + fz * fz), rad = near_radius(S, S.ss->cm, rem);
  if (!(travel <= S.flight_rv) || rad + travel > S.near_img) return NEAR_WILD;
  const FlightCell *fc = S.ftab + lin_cell(S, cx, cy, cz);
  const int cnt = tcount(fc->tc, step);
  if (cnt > FLIGHT_CAP) return NEAR_WILD;
  unsigned cand = NEAR_NONE;
  for (int k = 0; k < cnt; ++k) {
    const int j = fc->id[k];
    const float4 c = S.Xf[b][j];
    const float dx = wrap_half(c.x - px, S.Lxf), dy = wrap_half(c.y - py, S.Lyf), dz = wrap_half(c.z - pz, S.Lzf);
    if (path_meets(-dx, -dy, -dz, fx, fy, fz, rad)) cand = near_add(cand, j);
  }
  return cand;
}

// --------------------------------------------------------------------- run()

// rear-shell test of run() (cpp/run.cpp:17-19) against the kicked colloid
// velocity V + v0 ra, and the shell count per colloid
__global__ void k_run_shell(const SysF64 S, int fb) {
  const int n = min(S.ss->nshell, S.shell_cap);
  const double *Xc = S.X[(int)((S.ss->step * S.n_sub - 1) & 1)];
  const Fluid F = fluid_at(S, fb);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    ShellRec rec = S.shell[i];
    int p = S.newpos[rec.p];
    d3 pos = mk(F.x[p], F.y[p], F.z[p]);
    uint8_t pass = 0;
    for (int k = 0; k < rec.n; ++k) {
      int j = rec.j[k];
      d3 r = mk(ref_img(__dsub_rn(pos.x, Xc[3 * j]), S.dx), ref_img(__dsub_rn(pos.y, Xc[3 * j + 1]), S.dy),
                ref_img(__dsub_rn(pos.z, Xc[3 * j + 2]), S.dz));
      d3 V = add3(mk(S.V[3 * j], S.V[3 * j + 1], S.V[3 * j + 2]),
                  mul3s(mk(S.ra[3 * j], S.ra[3 * j + 1], S.ra[3 * j + 2]), S.v0));
      if (dot_ref(r, V) <= 0) {
        pass |= (uint8_t)(1u << k);
        atomicAdd(&S.shell_cnt[j], 1);
      }
    }
    S.shell[i].pass = pass;
  }
}

// vel_fl -= v0 ra M / (m cnt) for each rear shell the particle is in, in colloid
// order (cpp/run.cpp:20-24)
// (split: a near particle whose kicked path may meet a sphere becomes active)
__global__ void k_run_kick(const SysF64 S, int fb, int split) {
  const int n = min(S.ss->nshell, S.shell_cap);
  const Fluid F = fluid_at(S, fb);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    ShellRec rec = S.shell[i];
    if (!rec.pass) continue;
    int p = S.newpos[rec.p];
    // v = w (1/dt): within an ulp of w / dt, without a double division per component
    d3 v = mk(__dmul_rn(F.wx[p], S.inv_dt), __dmul_rn(F.wy[p], S.inv_dt), __dmul_rn(F.wz[p], S.inv_dt));
    for (int k = 0; k < rec.n; ++k) {
      if (!((rec.pass >> k) & 1)) continue;
      int j = rec.j[k];
      d3 del = mul3s(mk(S.ra[3 * j], S.ra[3 * j + 1], S.ra[3 * j + 2]), S.v0);
      double f = __ddiv_rn(S.mass_colloid, __dmul_rn(S.mass_fl, (double)S.shell_cnt[j]));
      v = sub3(v, mul3s(del, f));
    }
    F.wx[p] = __dmul_rn(v.x, S.dt); F.wy[p] = __dmul_rn(v.y, S.dt); F.wz[p] = __dmul_rn(v.z, S.dt);
    if (!split) continue;
    // an active particle's candidates are looked up anew (k_near_step64); another may become active
    if (S.fnear[p] == FN_ACTIVE) {
      S.fnear[p] = FN_KICKED;
    } else if (S.fnear[p] == FN_NEAR) {
      const unsigned cand = near_cand64(S, S.ss->step, S.n_sub, (int)((S.ss->step * S.n_sub - 1) & 1), F.x[p], F.y[p],
                                        F.z[p], F.wx[p], F.wy[p], F.wz[p]);
      if (cand == NEAR_NONE) continue;
      S.fnear[p] = FN_ACTIVE;
      const int i = atomicAdd(&S.ss->nact, 1);
      S.act[i] = p;
      S.actc[i] = cand;
    }
  }
}

// ------------------------------------------------------------------ colloids

// One warp per colloid (warp w of block b holds colloid b + gridDim.x * w), its
// vector components on separate lanes so the FP64 latency chains run side by
// side: lane k < 3 the linear component k (V, f, X), lane 3 + k the angular
// component k (Omega); the orientation update draws the three sines and cosines
// on lanes 0-2.  `l` is the substep (1..n_sub) that M_FINISH / M_ACT end, or 0
// before the first substep of a step.  With M_ADVANCE the colloid then moves to
// the following substep (update_pos_md, cpp/update.cpp:48-54).  In the fused step
// the orientation update of substeps 1..n-1 runs in the next streaming pass
// instead (colloid_aux), off the critical path.
static __device__ __forceinline__ void k_fin_colloid(const SysF64 &S, int j, int lane, int mode, long long g,
                                                     long long gn);

static __device__ __forceinline__ void k_fin_body(const SysF64 &S, const int VB, const int NVB, int mode, int l) {
  const int lane = threadIdx.x & 31;
  // with fin_table a block per colloid (warp 0 the colloid, all warps its cell
  // table), else a warp per colloid
  const int j = S.fin_table ? VB : VB + NVB * (threadIdx.x >> 5);
  const long long step = S.ss->step;
  const long long g = step * S.n_sub + (l - 1);  // substep finished (l >= 1)
  const long long gn = g + 1;                    // substep advanced to
  if (VB == 0 && threadIdx.x == 0 && (mode & M_FLIGHT)) {
    // events a pass before this step listed (the set-up's), which no list takes over
    S.ss->ev_total += S.ss->nnew[0] + S.ss->nnew[1] + S.ss->nevents;
    S.ss->nnew[0] = S.ss->nnew[1] = S.ss->nevents = 0;
  } else if (VB == 0 && threadIdx.x == 0) {
    if (S.precision == MPCD_FP64) {
      // the list substep g's streaming pass filled has been taken over by the event
      // pass (into the pending list, empty again after the last substep); its
      // buffer serves substep g+2.  The grid shift of the next step's binning is
      // drawn two substeps ahead: the last streaming pass bins with it and runs
      // beside the finish of the substep before it.
      const int b = (int)(g & 1);
      const int nn = S.ss->nnew[b];
      S.ss->ev_total += nn;
      S.ss->nnew[b] = 0;
      if (mode & M_FINISH) {
        const int np = S.ss->npend + (nn < S.events_cap ? nn : S.events_cap);
        S.ss->npend = l >= S.n_sub ? 0 : (np < S.pend_cap ? np : S.pend_cap);
      }
      const int ahead = S.n_sub >= 2 ? S.n_sub - 2 : 0;
      if ((mode & M_ADVANCE) && (gn % S.n_sub) == ahead) set_shift(S, step + 2);
    } else {
      S.ss->ev_total += S.ss->nevents;
      S.ss->nevents = 0;  // the event list of the coming streaming pass
      if ((mode & M_ADVANCE) && (gn % S.n_sub) == S.n_sub - 1) set_shift(S, step + 2);  // it bins for the next step
    }
  }
  if (j >= S.Nc) return;  // (j is the block's or the warp's)
  if (!S.fin_table) {
    if (lane < 6) k_fin_colloid(S, j, lane, mode, g, gn);
    if ((mode & M_FLIGHT) && S.ss->crowd == step + 1) {
      // a crowded flight cell: the cell tables of the step's first two substeps
      __syncwarp();
      if (S.ss->tab != gn) table_of(S, j, gn, lane, 32);
      table_of(S, j, gn + 1, lane, 32);
    }
    return;
  }
  if (threadIdx.x < 6) k_fin_colloid(S, j, lane, mode, g, gn);
  if (mode & M_ADVANCE) {
    // the cell table of substep gn+1 from the new position, by the whole block: the
    // streaming pass of gn+1 then needs this kernel only, not the side kernel of gn
    __syncthreads();
    const int nxt = (int)(gn & 1);
    const long long e = gn + 1;
    unsigned long long *Tc = S.Tcnt[e & 1];
    uint16_t *Tl = S.Tlist[e & 1];
    int *err = &S.ss->err;
    for_reach_cells(S, S.cbox[nxt][j], S.Xf[nxt][j], table_reach(S, e), threadIdx.x, blockDim.x,
                    [&](int cell) { tappend(Tc, Tl, cell, e, j, err); });
  }
}

// the per-colloid part of k_fin on lanes 0-5
static __device__ __forceinline__ void k_fin_colloid(const SysF64 &S, int j, int lane, int mode, long long g,
                                                     long long gn) {
  const unsigned grp = 0x3Fu;  // lanes 0-5
  const int k = lane < 3 ? lane : lane - 3;
  const bool lin = lane < 3;
  double v = lin ? S.V[3 * j + k] : S.W[3 * j + k];
  double f = lin ? S.f[3 * j + k] : 0.0;

  if (mode & (M_FINISH | M_COLL)) {
    // end of fluid_colloid_collision: V += vc m/M, Omega += omega m/I (cpp/fluid_colloid_collision.cpp:46-47)
    ExchAcc *e = S.exch + j;
    const double x = __dadd_rn((double)e->hi[lane] * 0x1p-20, (double)e->lo[lane] * 0x1p-72);
    e->hi[lane] = 0;
    e->lo[lane] = 0;
    const double dp = __dmul_rn(x, S.mass_fl);
    S.xacc[6 * j + lane] += dp;  // the exchange record (mpcd_exchange_read)
    v = __dadd_rn(v, __dmul_rn(dp, lin ? S.inv_mc : S.inv_ic));  // (within an ulp of dp / M)
    if (lin && (mode & M_FINISH)) {
      // compute_force_md at X_g (done by the streaming pass) and update_velocity_colloid
      const double fn = S.fnew[3 * j + k];
      v = __dadd_rn(v, __dmul_rn(__dadd_rn(f, fn), S.dtb2));
      f = fn;
    }
  }
  double ra = lin ? S.ra[3 * j + k] : 0.0;
  if (mode & M_ACT) {
    // update_activity_direction (its noise xi was drawn by the streaming pass):
    // Omega moves to lanes 0-2, each takes one sine and cosine, all gather them
    const double w = __shfl_sync(grp, v, lin ? lane + 3 : lane);
    double s = 0, co = 0;
    if (lin) sincos_small(__dmul_rn(w, S.dt), &s, &co);
    const d3 sb = mk(__shfl_sync(grp, s, 0), __shfl_sync(grp, s, 1), __shfl_sync(grp, s, 2));
    const d3 cb = mk(__shfl_sync(grp, co, 0), __shfl_sync(grp, co, 1), __shfl_sync(grp, co, 2));
    const d3 r3 = mk(__shfl_sync(grp, ra, 0), __shfl_sync(grp, ra, 1), __shfl_sync(grp, ra, 2));
    if (lin) {
      const d3 rn = activity_rot(S, r3, sb, cb, ldv(S.xi, j));
      ra = k == 0 ? rn.x : (k == 1 ? rn.y : rn.z);
    }
  }
  if (!lin) {
    S.W[3 * j + k] = v;
    return;
  }
  if (mode & M_KICK) v = __dadd_rn(v, __dmul_rn(ra, S.v0));  // run(): vel_colloid += ra v0 (cpp/run.cpp:13)

  if (mode & M_ADVANCE) {
    // update_pos_md (cpp/update.cpp:48-54)
    const int cur = (int)(g & 1), nxt = (int)(gn & 1);
    const Dim &D = k == 0 ? S.dx : (k == 1 ? S.dy : S.dz);
    const double xo = S.X[cur][3 * j + k];
    // (the division of mod in line: a call would cost this chain 2 us)
    const double xn = ref_mod<true>(__dadd_rn(xo, __dadd_rn(__dmul_rn(v, S.dt), __dmul_rn(f, S.ddt))), D);
    // the cell table of gn was built from Xo with a margin for this move
    const double ex = ref_img<true>(__dsub_rn(xn, xo), D);
    const unsigned g3 = 0x7u;
    const double e2 = __dmul_rn(ex, ex);
    const double d2 = __shfl_sync(g3, e2, 0) + __shfl_sync(g3, e2, 1) + __shfl_sync(g3, e2, 2);
    const d3 Xn = mk(__shfl_sync(g3, xn, 0), __shfl_sync(g3, xn, 1), __shfl_sync(g3, xn, 2));
    S.X[nxt][3 * j + k] = xn;
    if (k == 0) {
      if (d2 > S.ss->cm2) atomicOr(&S.ss->err, ERRB_DISPLACE);
      S.Xf[nxt][j] = make_float4((float)Xn.x, (float)Xn.y, (float)Xn.z, 0.f);
      S.cbox[nxt][j] = colloid_cell(S, Xn);
      if (mode & M_FLIGHT) S.ccell[nxt][j] = cell_coords(S, S.cbox[nxt][j]);  // (for the cooperative substeps)
      colloid_q(S, nxt, j, Xn);
    }
  }
  S.V[3 * j + k] = v;
  S.f[3 * j + k] = f;
  S.ra[3 * j + k] = ra;
}

__global__ void __launch_bounds__(256) k_fin(__grid_constant__ const SysF64 S, int mode, int l) {
  k_fin_body(S, blockIdx.x, gridDim.x, mode, l);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(128) k_fin_b(const SysF64 *Ss, const int *boff, int nrep, int mode, int l) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_fin_body(sS, VB, NVB, mode, l); });
}

// Set-up (the prologue of main, cpp/active_brownian.cpp:17-20): forces at the
// current positions (compute_force_md), the cell table for the run() candidates
// of the first step (substep g0-1) and the table of the first substep g0.
__global__ void __launch_bounds__(128) k_colloid_setup(const SysF64 S) {
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long step = S.ss->step;
  const long long g0 = step * S.n_sub;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    set_shift(S, step + 1);
    S.ss->nevents = 0;
    S.ss->nnew[0] = S.ss->nnew[1] = 0;
    S.ss->npend = 0;
    S.ss->crowd = 0;
    S.ss->tab = g0;
    S.ss->cm = S.cmarginf;  // the static bound until a step has measured the colloids
    S.ss->cm2 = S.cmargin2;
  }
  if (j >= S.Nc) return;
  const int b = (int)((g0 - 1) & 1);
  double pot;
  d3 fn = wca_force(S, S.X[b], S.Xf[b], j, lane, false, pot);
  if (lane == 0) {
    stv(S.f, j, fn);
    colloid_q(S, b, j, ldv(S.X[b], j));
  }
  int *err = &S.ss->err;
  const int cb = S.cbox[b][j];
  const float4 xc = S.Xf[b][j];
  for_reach_cells(S, cb, xc, S.rT_shell, lane, 32,
                  [&](int cell) { tappend(S.Tcnt[b], S.Tlist[b], cell, g0 - 1, j, err); });
  for_reach_cells(S, cb, xc, table_reach(S, g0), lane, 32,
                  [&](int cell) { tappend(S.Tcnt[b ^ 1], S.Tlist[b ^ 1], cell, g0, j, err); });
}

// WCA potential of the configuration in position buffer b, per colloid (pairs k > j),
// for the diagnostics (cpp/update.cpp:24)
__global__ void __launch_bounds__(128) k_colloid_pot(const SysF64 S, int b) {
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= S.Nc) return;
  double pot;
  wca_force(S, S.X[b], S.Xf[b], j, lane, true, pot);
  if (lane == 0) S.pot_part[j] = pot;
}

__global__ void k_end_step(__grid_constant__ const SysF64 S) {
  k_end_step_body(S, blockIdx.x, true);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void k_end_step_b(const SysF64 *Ss, const int *boff, int nrep) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int) { k_end_step_body(sS, VB, true); });
}

// fluid diagnostics from the exact cell sums of the last binning: per block the
// sums of S(w) (3), S(|w|^2) and the count, as doubles, in a fixed order
__global__ void __launch_bounds__(256) k_diag_fluid(const SysF64 S, double *part) {
  __shared__ double sh[5][256];
  double a[5] = {0, 0, 0, 0, 0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < S.Cpad; c += gridDim.x * blockDim.x) {
    CellAcc q = S.acc[c];
    a[0] += (double)q.sx * S.inv_sw; a[1] += (double)q.sy * S.inv_sw; a[2] += (double)q.sz * S.inv_sw;
    a[3] += (double)q.s2 * S.inv_sw; a[4] += (double)q.n;
  }
  for (int k = 0; k < 5; ++k) sh[k][threadIdx.x] = a[k];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s)
      for (int k = 0; k < 5; ++k) sh[k][threadIdx.x] += sh[k][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 5; ++k) part[blockIdx.x * 5 + k] = sh[k][0];
}

// ------------------------------------------------- active particles' substeps (FP64 form)

// what the FP32 tests need of a colloid
struct __align__(16) NearCol64 {
  float4 x;
  int4 c;
  static __device__ __forceinline__ NearCol64 get(const SysF64 &S, int b, int j) { return {S.Xf[b][j], S.ccell[b][j]}; }
  static __device__ __forceinline__ void copy(const SysF64 &S, int b, int j, NearCol64 *to) {
    near_copy16(&to->x, &S.Xf[b][j]);
    near_copy16(&to->c, &S.ccell[b][j]);
  }
};

// A pending particle of k_near_step64: its state streamed to the substep in flight, the colloids
// it can be inside of (ascending; none: nc = 0), and, prepared while the colloids move, what its
// reflection off the first of them (jc) needs that no colloid position enters: the point half a
// substep back, the random point seen from there, the Rayleigh speed and the Gaussians.
struct NearEv : EvState {
  double bx, by, bz, tx, ty, tz, val, v1, v2;
  NearCell c;
  int jc, nc;
  unsigned cand;  // the slots of the colloids its path comes near; NEAR_STALE after a collision
  uint16_t cd[4];
  bool slow;  // more than four of them, or an aliased or overflowing cell: searched anew
};
static_assert(sizeof(NearEv) <= EV_STATE_BYTES, "records of SysF64::evx");

static __device__ __forceinline__ NearCell near_cell64(const SysF64 &S, double x, double y, double z) {
  NearCell c;
  c.lin = cell_of_pos(S, x, y, z, c.alias);
  c.ix = trunc_nonneg(x); c.iy = trunc_nonneg(y); c.iz = trunc_nonneg(z);
  return c;
}

// The colloids a streamed particle may be inside of in this substep (prev: the buffer of the
// positions before it): jc, the first in order that its boxes, the sphere and the colloid's move
// (mg) alone allow, among the ones its path comes near; where there is one, all those within a
// wall collision's displacement of that as well (a second sphere is reached through a collision
// with the first).
static __device__ __forceinline__ void near_spheres64(const SysF64 &S, long long step, long long gs, NearEv &e, int prev,
                                                      float mg, const NearCols<NearCol64> &cols) {
  const float px = d2f_trunc(e.x), py = d2f_trunc(e.y), pz = d2f_trunc(e.z);
  const float ch = S.r_coll + 1e-3f + mg, far = ch + S.disp_marginf + 1e-3f;
  auto dist2 = [&](float4 c) {
    const float dx = wrap_half(c.x - px, S.Lxf), dy = wrap_half(c.y - py, S.Lyf), dz = wrap_half(c.z - pz, S.Lzf);
    return dx * dx + dy * dy + dz * dz;
  };
  e.jc = -1;
  e.nc = 0;
  e.slow = e.c.alias;
  if (e.slow) return;
  if (e.cand != NEAR_WILD) {
    bool any = false;
    for (unsigned r = e.cand; (r & 0xFFFFu) != 0xFFFFu && !any; r = (r >> 16) | 0xFFFF0000u)
      any = dist2(cols.d[r & 0xFFFFu].x) <= ch * ch;
    if (!any) return;
  }
  const NearList q = near_list(S, step, gs, e.c.lin, e.c.alias);
  e.slow = q.brute;
  for (int k = 0; k < q.cnt && !e.slow; ++k) {
    const int j = q.ids[k];
    const NearCol64 o = cols.at(S, prev, j);
    const float d2 = dist2(o.x);
    if (d2 > far * far || !in_block3(S, o.c, e.c.ix, e.c.iy, e.c.iz)) continue;
    if (e.nc == 4) {
      e.slow = true;
      return;
    }
    int at = e.nc++;
    for (; at > 0 && e.cd[at - 1] > j; --at) e.cd[at] = e.cd[at - 1];
    e.cd[at] = (uint16_t)j;
    if (d2 <= ch * ch && (e.jc < 0 || j < e.jc)) e.jc = j;
  }
  if (e.jc < 0) e.nc = 0;  // no first collision
}

// the collisions of a particle, one after another, by the general routine: the rare cases that
// nothing was listed for
static __device__ __noinline__ void near_collide_rest(const SysF64 &S, NearEv &e, long long step, long long gs,
                                                      int buf) {
  const NearList q = near_list(S, step, gs, e.c.lin, e.c.alias);
  int j = near_next(S, q, -1, e.c, buf ^ 1);
  while (j >= 0) {
    if (within(S, S.X[buf], S.Xf[buf][j], j, e.x, e.y, e.z, S.r_coll, S.sig2q)) ev_collide(S, e, j, gs, buf);
    j = near_next(S, q, j, e.c, buf ^ 1);
  }
}

// the same over the colloids listed for it, from number m on: they are all it can reach (a
// displacement beyond the margin fails the step)
static __device__ __noinline__ void near_collide_listed(const SysF64 &S, NearEv &e, int m, long long gs, int buf) {
#pragma unroll 1
  for (; m < e.nc; ++m) {
    const int j = e.cd[m];
    if (within(S, S.X[buf], S.Xf[buf][j], j, e.x, e.y, e.z, S.r_coll, S.sig2q)) ev_collide(S, e, j, gs, buf);
  }
}

// run() candidate record of a particle (id) at x, y, z after the last substep: the colloids, in
// ascending order, whose boxes (of the substep before, buffer buf ^ 1) hold cell c and whose
// run() shell holds it; *band: the FP32 test against the positions of the substep before
// (margin mg) leaves the shell membership open, which the streaming pass counts as an event
static __device__ __forceinline__ void near_shell64(const SysF64 &S, long long step, int buf, float mg, double x,
                                                    double y, double z, const NearCell &c, int id, ShellRec &rec,
                                                    bool *band) {
  const NearList q = near_list(S, step, step * S.n_sub + S.n_sub - 1, c.lin, c.alias);
  const float px = d2f_trunc(x), py = d2f_trunc(y), pz = d2f_trunc(z);
  const float sl = S.r_shell - 1e-3f - mg, sh = S.r_shell + 1e-3f + mg;
  rec.p = id;
  rec.n = 0;
  rec.pass = 0;
  *band = c.alias;
  // (an unordered walk, the ids inserted in order; a colloid beyond the band is no member)
  int last = -1;
  for (int k = 0;; ++k) {
    int j;
    if (q.brute) {
      j = last = near_next(S, q, last, c, buf ^ 1);
      if (j < 0) break;
    } else {
      if (k >= q.cnt) break;
      j = q.ids[k];
    }
    const float4 f = S.Xf[buf ^ 1][j];
    const float dx = wrap_half(f.x - px, S.Lxf), dy = wrap_half(f.y - py, S.Lyf), dz = wrap_half(f.z - pz, S.Lzf);
    const float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 > sh * sh || !near_in_block(S, j, c, buf ^ 1)) continue;
    if (!(d2 < sl * sl)) *band = true;
    if (!within(S, S.X[buf], S.Xf[buf][j], j, x, y, z, S.r_shell, S.rsh2)) continue;
    if (rec.n == SHELL_J) {
      atomicOr(&S.ss->err, ERRB_SHELLSLOTS);
      continue;
    }
    int at = rec.n++;
    for (; at > 0 && rec.j[at - 1] > j; --at) rec.j[at] = rec.j[at - 1];
    rec.j[at] = (uint16_t)j;
  }
}

// Particles per block kept in shared memory: NEAR64_ACT active ones (52 bytes each; more stay
// in the other fluid buffer, which is free between sorts) and NEAR64_EV pending ones.
constexpr int NEAR64_EV = 160;
struct Near64 {
  double st[6][NEAR64_ACT];
  unsigned cand[NEAR64_ACT];
  NearEv ev[NEAR64_EV];
  NearCols<NearCol64> col;
};

// see near_step.cuh.  A particle the FP32 test cannot clear is pending for the rest of the step,
// as in the overlapped substeps.  An FP64 instruction takes a warp about 60 cycles, and the SM's
// FP64 unit 16 of them however many lanes are active, so a substep's collisions run one per lane
// on as few warps as hold them, and everything that does not wait for the colloids (the
// logarithms of the draws above all) is prepared beside the colloids' finish.
// (128 registers: with the free-flight pass's two blocks of 64 beside it all that an SM has)
__global__ void __launch_bounds__(NEAR64_BLOCK, 2) k_near_step64(__grid_constant__ const SysF64 S, int fb) {
  constexpr int NT = NEAR64_BLOCK - 32 * (NEAR_CW + 1), NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Near64 &sm = *reinterpret_cast<Near64 *>(smem_raw);
  __shared__ double s_hx[NT][6];  // the exchanges of a round's collisions, and their colloids
  __shared__ int s_hj[NT];
  __shared__ int s_nh, s_np, s_nx, s_fin;  // (s_np: pending particles; s_nx: of them, beyond NEAR64_EV)
  __shared__ int s_flag[2];
  __shared__ NearPairs s_pairs;
  const int t = threadIdx.x, VB = blockIdx.x, G = gridDim.x;
  const int n = S.n_sub;
  if (t == 0) s_np = s_nx = s_nh = s_fin = 0;
  sm.col.clear(S, t, NEAR64_BLOCK);
  if (VB == 0 && t == NT) set_shift(S, S.ss->step + 2);  // (the records of this step are all kicked)
  near_let_dependents();
  __syncthreads();
  if (t >= NT + 32 * NEAR_CW) {
    near_orient(S, VB, G, t & 31, &s_fin);
    return;
  }
  if (t >= NT) {
    near_colloids(S, s_pairs, VB, G, t - NT, 2, &s_flag[1], &s_fin);
    return;
  }
  const long long step = S.ss->step, g0 = step * n;
  const float mg = S.ss->cm;
  const Fluid F = fluid_at(S, fb), O = fluid_at(S, 1 - fb);
  const int nact = min(S.ss->nact, S.N);
  const int a0 = (int)((long long)VB * nact / G), cnt = (int)((long long)(VB + 1) * nact / G) - a0;
  const int w = t >> 5, lane = t & 31;
  auto sync = [] { group_sync(1, NT); };
  // active particle k of the block: its state in shared memory or in the other fluid buffer
  auto ptr = [&](int c, int k) -> double * {
    if (k < NEAR64_ACT) return &sm.st[c][k];
    double *o = c == 0 ? O.x : c == 1 ? O.y : c == 2 ? O.z : c == 3 ? O.wx : c == 4 ? O.wy : O.wz;
    return o + a0 + k;
  };
  auto ev = [&](int i) -> NearEv & {
    return i < NEAR64_EV ? sm.ev[i]
                         : *reinterpret_cast<NearEv *>((char *)S.evx + (size_t)EV_STATE_BYTES * O.id[a0 + i]);
  };
#pragma unroll 2
  for (int k = t; k < cnt; k += NT) {
    const int p = S.act[a0 + k];
    const double x = F.x[p], y = F.y[p], z = F.z[p], wx = F.wx[p], wy = F.wy[p], wz = F.wz[p];
    unsigned cand = S.actc[a0 + k];
    if (S.fnear[p] == FN_KICKED) {
      cand = near_cand64(S, step, n, (int)((g0 - 1) & 1), x, y, z, wx, wy, wz);
      S.fnear[p] = FN_ACTIVE;
    }
    *ptr(0, k) = x; *ptr(1, k) = y; *ptr(2, k) = z;
    *ptr(3, k) = wx; *ptr(4, k) = wy; *ptr(5, k) = wz;
    if (k < NEAR64_ACT) {
      sm.cand[k] = cand;
      sm.col.note(cand);
    }
  }
  sync();
  sm.col.load(S, (int)((g0 - 1) & 1), t, NT);
  for (int k = t; k < min(cnt, NEAR64_ACT); k += NT) sm.cand[k] = sm.col.slots(sm.cand[k]);
  sync();

  // update_pos_mpcd of substep l and the FP32 test against the positions of l - 1 with the
  // displacement bound as margin (np: pending particles of the substeps before), then what the
  // pending ones' collisions can be given in advance
  auto advance = [&](int l, int np) {
    const long long gs = g0 + (l - 1);
    const int xb = (int)(gs & 1) ^ 1;
    const float ch = S.r_coll + 1e-3f + mg;
    // active particle k by the general path
    auto one = [&](int k, unsigned cand) {
      double *px = ptr(0, k), *py = ptr(1, k), *pz = ptr(2, k);
      const double wx = *ptr(3, k), wy = *ptr(4, k), wz = *ptr(5, k);
      const double x = ref_mod(__dadd_rn(*px, wx), S.dx), y = ref_mod(__dadd_rn(*py, wy), S.dy),
                   z = ref_mod(__dadd_rn(*pz, wz), S.dz);
      const float fx = d2f_trunc(x), fy = d2f_trunc(y), fz = d2f_trunc(z);
      auto close = [&](float4 c) {
        const float dx = wrap_half(c.x - fx, S.Lxf), dy = wrap_half(c.y - fy, S.Lyf), dz = wrap_half(c.z - fz, S.Lzf);
        return dx * dx + dy * dy + dz * dz <= ch * ch;
      };
      const NearCell c = near_cell64(S, x, y, z);
      auto block = [&](int4 cc, int j) { return c.alias ? near_in_block(S, j, c, xb) : in_block3(S, cc, c.ix, c.iy, c.iz); };
      bool e = c.alias;
      if (cand == NEAR_WILD) {
        const NearList q = near_list(S, step, gs, c.lin, c.alias);
        for (int m = 0; m < (q.brute ? S.Nc : q.cnt) && !e; ++m) {
          const int j = q.brute ? m : q.ids[m];
          e = close(sm.col.at(S, xb, j).x) && near_in_block(S, j, c, xb);
        }
      } else {
        for (unsigned r = cand; (r & 0xFFFFu) != 0xFFFFu && !e; r = (r >> 16) | 0xFFFF0000u) {
          const NearCol64 &o = sm.col.d[r & 0xFFFFu];
          e = close(o.x) && block(o.c, sm.col.id[r & 0xFFFFu]);
        }
      }
      if (!e) {
        *px = x; *py = y; *pz = z;
        return;
      }
      *px = x; *py = y; *pz = z;
      int i = atomicAdd(&s_np, 1);
      const int p = S.act[a0 + k];
      if (i >= NEAR64_EV) {
        const unsigned o = atomicAdd(S.bar + BAR_EVX, 1u);
        if (o >= (unsigned)S.evx_cap) {
          // no record left: the step fails, and the particle goes on unlisted (a record of two particles
          // would be changed by both their blocks)
          atomicOr(&S.ss->err, ERRB_EVENTS);
          atomicSub(S.bar + BAR_EVX, 1u);
          atomicSub(&s_np, 1);
          return;
        }
        i = NEAR64_EV + atomicAdd(&s_nx, 1);  // (s_np also counts those that find none)
        O.id[a0 + i] = (int)o;
      }
      NearEv &v = ev(i);
      v.j = k;  // (the record is made below)
      v.p = p;
      v.cand = cand;
      S.fnear[p] = FN_PENDING;
      if (k < NEAR64_ACT) sm.cand[k] = NEAR_GONE;
    };
    // The active ones, two at a time and without a branch where they stay inside the box (so the
    // additions need no mod) and have one or two candidates, which are not near: about 75 instructions
    // each, interleaved.  Everything else takes the general path.
    const int kept = min(cnt, NEAR64_ACT);
    for (int k0 = t; k0 < kept; k0 += 2 * NT) {
      unsigned cand[2];
      bool far[2];
      double x[2][3];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = min(k0 + u * NT, kept - 1);
        cand[u] = k0 + u * NT < kept ? sm.cand[k] : NEAR_GONE;
        const unsigned top = NearCols<NearCol64>::MAX - 1, j2 = cand[u] >> 16;
        const float4 o = sm.col.d[min(cand[u] & 0xFFFFu, top)].x, o2 = sm.col.d[min(j2, top)].x;
        float d2 = 0.f, e2 = 0.f;
        far[u] = j2 - (NEAR_STALE >> 16) > 2u;  // (none of the marks)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const Dim &D = a == 0 ? S.dx : (a == 1 ? S.dy : S.dz);
          const float L = a == 0 ? S.Lxf : (a == 1 ? S.Lyf : S.Lzf);
          x[u][a] = __dadd_rn(sm.st[a][k], sm.st[3 + a][k]);
          const long long b = dbits(x[u][a]);
          far[u] = far[u] && b >= D.lo_bits && b < D.L_bits;
          const float f = d2f_box(x[u][a]), d = wrap_half((a == 0 ? o.x : a == 1 ? o.y : o.z) - f, L),
                      e = wrap_half((a == 0 ? o2.x : a == 1 ? o2.y : o2.z) - f, L);
          d2 = a == 0 ? d * d : fmaf(d, d, d2);
          e2 = a == 0 ? e * e : fmaf(e, e, e2);
        }
        const float lim = (ch + 1e-4f) * (ch + 1e-4f);  // (the general path's rounding may differ)
        far[u] = far[u] && d2 > lim && (j2 == 0xFFFFu || e2 > lim);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = k0 + u * NT;
        if (far[u]) {
          sm.st[0][k] = x[u][0]; sm.st[1][k] = x[u][1]; sm.st[2][k] = x[u][2];
        } else if (cand[u] != NEAR_GONE) {
          one(k, cand[u]);
        }
      }
    }
    for (int k = NEAR64_ACT + t; k < cnt; k += NT)  // beyond shared memory
      if (S.fnear[S.act[a0 + k]] == FN_ACTIVE) one(k, NEAR_WILD);
    sync();
    // the pending ones, old and new, one per thread: what they read of global memory (the flight
    // table, ids) is one latency for all
    const int np1 = s_np;
    for (int i = t; i < np1; i += NT) {
      NearEv &e = ev(i);
      unsigned cand = e.cand;
      if (i < np) {
        if (cand == NEAR_STALE)
          cand = e.cand = sm.col.slots(near_cand64(S, step, n - l + 1, xb, e.x, e.y, e.z, e.wx, e.wy, e.wz));
        e.x = ref_mod(__dadd_rn(e.x, e.wx), S.dx);
        e.y = ref_mod(__dadd_rn(e.y, e.wy), S.dy);
        e.z = ref_mod(__dadd_rn(e.z, e.wz), S.dz);
      } else {
        const int k = e.j;
        e.x = *ptr(0, k); e.y = *ptr(1, k); e.z = *ptr(2, k);
        e.wx = *ptr(3, k); e.wy = *ptr(4, k); e.wz = *ptr(5, k);
        e.vdx = e.vdy = e.vdz = 0.0;
        e.id = F.id[e.p]; e.last = -1; e.cnt = 0; e.j = -1;
        e.changed = false;
      }
      e.c = near_cell64(S, e.x, e.y, e.z);
      e.lin = e.c.lin;
      e.alias = e.c.alias;
      e.x0 = e.x; e.y0 = e.y; e.z0 = e.z;
      e.dumped = false;
      near_spheres64(S, step, gs, e, xb, mg, sm.col);
    }
    sync();
    // the preparations of 32 pending particles at a time, the three independent FP64 chains on
    // different warps (SM schedulers)
    for (int q = w; q < 3 * ((np1 + 31) / 32); q += NW) {
      const int i = (q / 3) * 32 + lane, what = q % 3;
      if (i >= np1) continue;
      NearEv &e = ev(i);
      if (e.slow || e.nc == 0) continue;
      const uint32_t a = (uint32_t)(e.id + 1), b = (uint32_t)(e.jc + 1), tt = (uint32_t)gs;
      const uint4 r = draw4_loop(S.key, DOM_COLL, what == 2 ? 1 : 0, a, b, tt);
      if (what == 0) {
        const double x = ref_mod(__dsub_rn(e.x, __dmul_rn(e.wx, 0.5)), S.dx);
        const double y = ref_mod(__dsub_rn(e.y, __dmul_rn(e.wy, 0.5)), S.dy);
        const double z = ref_mod(__dsub_rn(e.z, __dmul_rn(e.wz, 0.5)), S.dz);
        const d3 tp = refl_point(S, r, mk(x, y, z));
        e.bx = x; e.by = y; e.bz = z;
        e.tx = tp.x; e.ty = tp.y; e.tz = tp.z;
        continue;
      }
      // the Rayleigh speed sqrt(-log((1 - u)^2) kT/m), or the Gaussians' sqrt(-2 log(z) / z)
      // (refl_speed, refl_gauss: one logarithm and one root in the code for both)
      double x1 = 0, x2 = 0, z, iz = 1.0;
      if (what == 1) {
        const double om = __dsub_rn(1.0, u01(r.x));
        z = __dmul_rn(om, om);
      } else {
        z = refl_try(S, r, a, b, tt, x1, x2);
        iz = __drcp_rn(z);
      }
      const double lz = log(z);
      const double g = __dsqrt_rn(what == 1 ? __dmul_rn(-lz, S.inv_m_beta) : __dmul_rn(__dmul_rn(-2.0, lz), iz));
      if (what == 1) {
        e.val = g;
      } else {
        e.v1 = __dmul_rn(__dmul_rn(x1, g), S.sqrt_kt_m);
        e.v2 = __dmul_rn(__dmul_rn(x2, g), S.sqrt_kt_m);
      }
    }
    if (t == 0) s_nh = 0;
  };

  advance(1, 0);
  for (int l = 1; l <= n; ++l) {
    const long long gs = g0 + (l - 1);
    const int buf = (int)(gs & 1);
    if (l > 1) {
      const unsigned Gm = (unsigned)(G < S.Nc ? G : S.Nc);
      if (!group_wait(S, BAR_MOVE, Gm * (unsigned)(l - 1), t, 1, NT, &s_flag[0])) return;
    } else {
      sync();
    }
    if (l < n) sm.col.copy(S, buf, t, NT);  // (for the tests of l + 1; it arrives meanwhile)
    // the pending particles' wall collisions at X(l), one per lane
    const int np = s_np;
    for (int base = 0;; base += NT) {
      const int i = base + t;
      const bool last_round = base + NT >= np;
      bool hit = false;
      d3 vn = mk(0, 0, 0), xb = vn;
      NearEv *e = nullptr;
      // the particle after its collision
      auto settle = [&] {
        const double wx = __dmul_rn(vn.x, S.dt), wy = __dmul_rn(vn.y, S.dt), wz = __dmul_rn(vn.z, S.dt);
        // step forward half a substep with the new velocity
        const double x = ref_mod(__dadd_rn(xb.x, __dmul_rn(wx, 0.5)), S.dx);
        const double y = ref_mod(__dadd_rn(xb.y, __dmul_rn(wy, 0.5)), S.dy);
        const double z = ref_mod(__dadd_rn(xb.z, __dmul_rn(wz, 0.5)), S.dz);
        // the candidates are looked up with a margin; a move beyond it could hide a colloid
        const double ex = ref_img(__dsub_rn(x, e->x0), S.dx), ey = ref_img(__dsub_rn(y, e->y0), S.dy),
                     ez = ref_img(__dsub_rn(z, e->z0), S.dz);
        if (norm2_ref(ex, ey, ez) > S.disp_margin2) atomicOr(&S.ss->err, ERRB_DISPLACE);
        e->x = x; e->y = y; e->z = z; e->wx = wx; e->wy = wy; e->wz = wz;
      };
      if (i < np) {
        e = &ev(i);
        if (e->slow) {
          near_collide_rest(S, *e, step, gs, buf);
          if (e->dumped) e->cand = NEAR_STALE;
        } else if (e->nc > 0) {
          int j = -1, c = 0;
          // (the colloid prepared for, loaded beside the test)
          const d3 Vj = ldv(S.V, e->jc), Wj = ldv(S.W, e->jc), Xj = ldv(S.X[buf], e->jc);
          for (; c < e->nc; ++c) {
            j = e->cd[c];
            if (within(S, S.X[buf], S.Xf[buf][j], j, e->x, e->y, e->z, S.r_coll, S.sig2q)) break;
          }
          if (c < e->nc && j != e->jc) {
            near_collide_listed(S, *e, c, gs, buf);  // (not the colloid that was prepared for)
            if (e->dumped) e->cand = NEAR_STALE;
          } else if (c < e->nc) {
            hit = true;
            xb = mk(e->bx, e->by, e->bz);
            const d3 rs = mk(ref_img(__dsub_rn(xb.x, Xj.x), S.dx), ref_img(__dsub_rn(xb.y, Xj.y), S.dy),
                             ref_img(__dsub_rn(xb.z, Xj.z), S.dz));
            const d3 u = refl_combine(S, refl_unit(rs), e->val, mk(e->tx, e->ty, e->tz), e->v1, e->v2);
            // dump_vel_fl: the velocity when the collision routine began
            const d3 vd = mk(__dmul_rn(e->wx, S.inv_dt), __dmul_rn(e->wy, S.inv_dt), __dmul_rn(e->wz, S.inv_dt));
            vn = add3(add3(u, Vj), cross_ref(Wj, rs));
            const d3 dv = sub3(vd, vn), dl = cross_ref(rs, dv);
            const int h = atomicAdd(&s_nh, 1);
            s_hj[h] = j;
            s_hx[h][0] = dv.x; s_hx[h][1] = dv.y; s_hx[h][2] = dv.z;
            s_hx[h][3] = dl.x; s_hx[h][4] = dl.y; s_hx[h][5] = dl.z;
            e->vdx = vd.x; e->vdy = vd.y; e->vdz = vd.z;
            e->dumped = e->changed = true;
            e->cand = NEAR_STALE;
            if (c + 1 < e->nc) {  // a second sphere may hold it now
              settle();
              hit = false;
              near_collide_listed(S, *e, c + 1, gs, buf);
            }
          }
        }
      }
      sync();
      // the round's exchanges, a component per thread
      const int nh = s_nh;
      for (int q = t; q < 6 * nh; q += NT) exch_add1(S.exch + s_hj[q / 6], q % 6, s_hx[q / 6][q % 6], &S.ss->err);
      sync();
      if (t == 0) {
        if (last_round) bar_arrive(S.bar + BAR_COLL);
        else s_nh = 0;
      }
      if (hit) settle();
      if (last_round) break;
      sync();
    }
    near_copy_wait();
    sync();
    if (l < n) advance(l + 1, np);
  }

  // after the last substep: the state back to the fluid arrays (the run() candidate records and
  // the binning are the end kernel's, except of what collided in this substep)
  sync();
  const int np = s_np, buf = (int)((g0 + n - 1) & 1);
  for (int base = 0; base < np; base += NT) {
    const int i = base + t;
    BinTerm b{-1, 0, 0, 0, 0};
    ShellRec rec;
    rec.n = 0;
    if (i < np) {
      const NearEv &e = ev(i);
      const int p = e.p;
      if (e.dumped) {
        bool band;
        near_shell64(S, step, buf, mg, e.x, e.y, e.z, e.c, e.id, rec, &band);
        b = bin_term(S, S.ss->rrn, p, e.x, e.y, e.z, e.wx, e.wy, e.wz);
        S.fnear[p] = FN_DONE;
      }
      F.x[p] = e.x; F.y[p] = e.y; F.z[p] = e.z;
      F.wx[p] = e.wx; F.wy[p] = e.wy; F.wz[p] = e.wz;
    }
    near_record(S, rec, rec.n != 0);
    bin_add_warp(S.acc, b.c, b.fx, b.fy, b.fz, b.f2);
  }
  for (int k = t; k < cnt; k += NT) {
    const int p = S.act[a0 + k];
    if (k < NEAR64_ACT ? sm.cand[k] == NEAR_GONE : S.fnear[p] != FN_ACTIVE) continue;
    F.x[p] = *ptr(0, k); F.y[p] = *ptr(1, k); F.z[p] = *ptr(2, k);
  }
  if (t == 0 && np) atomicAdd((unsigned long long *)&S.ss->ev_total, (unsigned long long)np);
}

size_t near_step64_smem() { return sizeof(Near64); }

__global__ void __launch_bounds__(256) k_rotdiff_step(__grid_constant__ const SysF64 S) {
  rotdiff_step(S, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_rotdiff_step_b(const SysF64 *Ss, const int *boff, int nrep) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int) { rotdiff_step(sS, (long long)VB * blockDim.x + threadIdx.x); });
}

// the cell table of a step's first substep at the present positions (the free-flight steps
// leave none, unless a flight cell is crowded; the per-substep passes read it), one block per colloid
__global__ void __launch_bounds__(256) k_table_next(__grid_constant__ const SysF64 S) {
  const int j = blockIdx.x;
  const long long g = S.ss->step * S.n_sub;
  if (j < S.Nc && S.ss->tab != g) table_of(S, j, g, threadIdx.x, blockDim.x);
}

// (behind it: the table is built)
__global__ void k_table_mark(__grid_constant__ const SysF64 S) { S.ss->tab = S.ss->step * S.n_sub; }

// The end of a free-flight step: the step counter and the next step's margin (block 0), and, in
// the other blocks, the run() candidate records of the near particles and the binning of the
// active ones among them (k_near_step64 wrote their final state).
__global__ void __launch_bounds__(256) k_end_flight64(__grid_constant__ const SysF64 S, int fb) {
  if (blockIdx.x == 0) {
    k_end_step_body(S, 0, S.ss->crowd == S.ss->step + 1);
    return;
  }
  const long long step = S.ss->step_f;
  const float mg = S.ss->cm_f;
  const int buf = (int)((step * S.n_sub + S.n_sub - 1) & 1);
  const Fluid F = fluid_at(S, fb);
  const int count = min(S.ss->nnear, S.N), lane = threadIdx.x & 31;
  const int stride = (gridDim.x - 1) * 256;
  int i = (blockIdx.x - 1) * 256 + threadIdx.x;
  int next = i < count ? S.near[i] : 0;
  for (int base = (blockIdx.x - 1) * 256; base < count; base += stride, i += stride) {
    ShellRec rec;
    rec.n = 0;
    bool band = false;
    BinTerm b{-1, 0, 0, 0, 0};
    const int p = next;
    if (i + stride < count) next = S.near[i + stride];
    if (i < count) {
      const uint8_t fn = S.fnear[p];
      if (fn != FN_DONE) {
        const double x = F.x[p], y = F.y[p], z = F.z[p];
        near_shell64(S, step, buf, mg, x, y, z, near_cell64(S, x, y, z), F.id[p], rec, &band);
        if (fn == FN_PENDING) band = false;  // (counted when it became pending)
        if (fn != FN_NEAR) b = bin_term(S, S.ss->rrn, p, x, y, z, F.wx[p], F.wy[p], F.wz[p]);
      }
    }
    if (__any_sync(FULL, b.c >= 0)) bin_add_warp(S.acc, b.c, b.fx, b.fy, b.fz, b.f2);
    const unsigned mb = __ballot_sync(FULL, band);
    if (lane == 0 && mb) atomicAdd((unsigned long long *)&S.ss->ev_total, (unsigned long long)__popc(mb));
    const unsigned m = __ballot_sync(FULL, rec.n != 0);
    const int at = block_base(&S.ss->nshell, m, lane) + __popc(m & ((1u << lane) - 1u));
    if (rec.n) {
      if (at < S.shell_cap) S.shell[at] = rec;
      else atomicOr(&S.ss->err, ERRB_SHELL);
    }
  }
}

// error bits of every system of a batch, for one read-back
__global__ void k_gather_err(const SysF64 *Ss, int nrep, int *out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < nrep) out[r] = Ss[r].ss->err;
}

}  // namespace bgb
