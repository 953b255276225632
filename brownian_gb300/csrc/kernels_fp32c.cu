// FP32-compensated form of the MPCD + active-colloid step (sm_103a).
//
// The fluid is stored per particle as one 16-byte record {packed cell, offset x,
// offset y, offset z} (a single 128-bit load) plus FP32 velocities: 28 bytes where
// the FP64 form keeps 48, and all fluid arithmetic runs on the FP32 pipe.  A
// position is its integer cell plus an FP32 offset in [0, 1), so it is resolved to
// 2^-24 of a cell everywhere in the box, and a particle-colloid distance is an
// exact integer cell difference plus an FP32 offset difference.  What stays in
// FP64 / exact: the colloids (shared with the FP64 form), the per-cell sums
// (exact fixed-point integers, so the cell momentum is summed without rounding),
// the thermostat factor of each cell, the colloid momentum exchange (exact
// fixed-point) and every diagnostic.
//
// Kernels mirror the FP64 form: k_stream32 (stream, FP32 scan of nearby colloids,
// event list, last-substep binning), k_events32 (wall collisions in FP32, one per
// lane), k_cell_prep32, k_rotate32 / k_rotate_sort32, k_run_shell32 / k_run_kick32.
#include "near_step.cuh"

namespace bgb {

__device__ __forceinline__ void unpack(uint4 r, int &cx, int &cy, int &cz, float &ox, float &oy, float &oz) {
  cx = (int)(r.x & 1023u); cy = (int)((r.x >> 10) & 1023u); cz = (int)((r.x >> 20) & 1023u);
  ox = __uint_as_float(r.y); oy = __uint_as_float(r.z); oz = __uint_as_float(r.w);
}

__device__ __forceinline__ uint4 pack(int cx, int cy, int cz, float ox, float oy, float oz) {
  return make_uint4((unsigned)cx | ((unsigned)cy << 10) | ((unsigned)cz << 20), __float_as_uint(ox),
                    __float_as_uint(oy), __float_as_uint(oz));
}

// the SRD collision of one particle: v' = A v + b, the cell's FP32 affine map (A row-major, b)
__device__ __forceinline__ void apply_map32(const float *ab, float &vx, float &vy, float &vz) {
  const float4 *m = reinterpret_cast<const float4 *>(ab);
  float4 a = m[0], b = m[1], c = m[2];
  float nx = fmaf(a.x, vx, fmaf(a.y, vy, fmaf(a.z, vz, c.y)));
  float ny = fmaf(a.w, vx, fmaf(b.x, vy, fmaf(b.y, vz, c.z)));
  float nz = fmaf(b.z, vx, fmaf(b.w, vy, fmaf(c.x, vz, c.w)));
  vx = nx; vy = ny; vz = nz;
}

// keep the offset in [0, 1), carrying whole cells into the periodic cell index
__device__ __forceinline__ void carry(int &c, float &o, int L) {
  if (o >= 0.f && o < 1.f) return;
  float f = floorf(o);
  o -= f;
  if (o >= 1.f) { o = 0.f; f += 1.f; }
  if (!(f == f) || fabsf(f) > 1e6f) { o = 0.f; f = 0.f; }  // NaN / runaway: stays put (flagged by the range test)
  c += (int)f;
  c %= L;
  if (c < 0) c += L;
}

// particle minus colloid along one axis, minimum image: integer cell difference
// (exact) plus offset difference
__device__ __forceinline__ float rel(int c, float o, float cq, float co, int L) {
  int d = c - (int)cq;
  if (d > (L >> 1)) d -= L;
  else if (d < -(L >> 1)) d += L;
  return (float)d + (o - co);
}

// uniform in (0,1) from the top 23 bits: (k + 1/2) 2^-23 is exact in FP32, so the
// value is never 0 or 1 (with 24 bits the top value would round to 1 and a
// reflection would take log(0))
__device__ __forceinline__ float u01f(uint32_t w) { return ((float)(w >> 9) + 0.5f) * 1.1920928955078125e-7f; }

// round(v * 2^k) of an FP32 value from its bits (exact when the scale covers the
// value's last bit)
__device__ __forceinline__ long long to_fix_f(float v, int k) {
  unsigned b = __float_as_uint(v);
  int e = (int)((b >> 23) & 0xFF);
  if (e == 0) return 0;
  long long m = (long long)((b & 0x7FFFFFu) | 0x800000u);
  int sh = e - 150 + k;
  long long r;
  if (sh >= 0) r = m << (sh < 62 ? sh : 62);
  else if (sh > -40) {
    int s = -sh;
    r = m >> s;
    long long rem = m & ((1ll << s) - 1), half = 1ll << (s - 1);
    if (rem > half || (rem == half && (r & 1))) r += 1;
  } else r = 0;
  return (b >> 31) ? -r : r;
}

// one particle's part of the SRD binning for the next step (rotation_mpcd bins by the
// shifted position: cell + floor(offset + rr) per axis): its cell (recorded in rotcell)
// and the fixed-point v and |v|^2 the exact cell sums add up
struct BinTerm32 {
  int c;
  long long fx, fy, fz, f2;
};

// round(v^2 2^k) from the significand m of v (24 bits, so m^2 is exact in 64 bits):
// v^2 2^k = m^2 2^(2 (e - 150) + k); the same value as sq_fix of to_fix_f(v, k) whenever
// v 2^k is an integer (every |v| >= 2^(23 - k)), and within one unit below that
__device__ __forceinline__ long long sq_fix_f(float v, int k) {
  const unsigned b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xFF);
  if (e == 0) return 0;
  const unsigned m = (b & 0x7FFFFFu) | 0x800000u;
  const unsigned long long q = (unsigned long long)m * m;
  const int sh = 2 * (e - 150) + k;
  if (sh >= 0) return (long long)(q << (sh < 16 ? sh : 16));
  if (sh <= -63) return 0;
  const int s = -sh;
  unsigned long long r = q >> s;
  const unsigned long long rem = q & ((1ull << s) - 1ull), half = 1ull << (s - 1);
  if (rem > half || (rem == half && (r & 1ull))) r += 1ull;
  return (long long)r;
}

struct Fix2 { long long f, f2; };
static __device__ __noinline__ Fix2 fix2_far(float v, int k) { return {to_fix_f(v, k), sq_fix_f(v, k)}; }

// to_fix_f and sq_fix_f together, in 32-bit steps where the shifts allow it (2^(23 - k) <= |v| and about
// 2^-11 <= |v| < 2^5 at the k of a usual system: 99.9 % of a thermal fluid's components): v 2^k as one
// product of the significand with a power of two, v^2 2^k from m^2 2^8 by one funnel shift, the dropped
// bits compared with one half in a word of their own.  About 20 instructions a component instead of 70.
__device__ __forceinline__ void fix2(float v, int k, long long &f, long long &f2) {
  const unsigned b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xFF), sh = e - 150 + k, s = 158 - e - sh;  // (s = 8 - (2 (e - 150) + k))
  if ((unsigned)sh <= 30u && (unsigned)(s - 1) <= 30u) {
    const unsigned m = (b & 0x7FFFFFu) | 0x800000u;
    f = (long long)((int)b < 0 ? -(int)m : (int)m) * (long long)(1 << sh);
    const unsigned long long q = (unsigned long long)m * (m << 8);
    const unsigned lo = (unsigned)q, hi = (unsigned)(q >> 32), low = __funnelshift_r(lo, hi, s), rem = lo << (32 - s);
    const unsigned long long r = ((unsigned long long)(hi >> s) << 32) | low;
    f2 = (long long)(r + (rem > 0x80000000u - (low & 1u) ? 1ull : 0ull));
  } else {
    const Fix2 t = fix2_far(v, k);
    f = t.f;
    f2 = t.f2;
  }
}

__device__ __forceinline__ BinTerm32 bin32_term(const SysF64 &S, const float *rr, int p, int cx, int cy, int cz,
                                                float ox, float oy, float oz, float vx, float vy, float vz) {
  float tx = ox + rr[0], ty = oy + rr[1], tz = oz + rr[2];
  int bx = cx + (tx < 0.f ? -1 : (tx >= 1.f ? 1 : 0));
  int by = cy + (ty < 0.f ? -1 : (ty >= 1.f ? 1 : 0));
  int bz = cz + (tz < 0.f ? -1 : (tz >= 1.f ? 1 : 0));
  bx += bx < 0 ? S.Lx : 0; bx -= bx >= S.Lx ? S.Lx : 0;
  by += by < 0 ? S.Ly : 0; by -= by >= S.Ly ? S.Ly : 0;
  bz += bz < 0 ? S.Lz : 0; bz -= bz >= S.Lz ? S.Lz : 0;
  const int c = bx + S.Lx * (by + S.Ly * bz);
  S.rotcell[p] = c;
  if (!(fabsf(vx) <= S.vmaxf && fabsf(vy) <= S.vmaxf && fabsf(vz) <= S.vmaxf)) atomicOr(&S.ss->err, ERRB_VRANGE);
  BinTerm32 t;
  t.c = c;
  long long x2, y2, z2;
  fix2(vx, S.kw, t.fx, x2);
  fix2(vy, S.kw, t.fy, y2);
  fix2(vz, S.kw, t.fz, z2);
  t.f2 = x2 + y2 + z2;
  return t;
}

__device__ __forceinline__ void bin32(const SysF64 &S, int p, int cx, int cy, int cz, float ox, float oy, float oz,
                                      float vx, float vy, float vz) {
  const BinTerm32 t = bin32_term(S, S.ss->rrf, p, cx, cy, cz, ox, oy, oz, vx, vy, vz);
  bin_add(S.acc + t.c, 1, t.fx, t.fy, t.fz, t.f2);
}

struct f3 { float x, y, z; };
__device__ __forceinline__ f3 fm(float x, float y, float z) { f3 r; r.x = x; r.y = y; r.z = z; return r; }

// One wall collision of a particle in two halves.  bounce32_draw: everything that the colloid's
// state does not enter, into Bounce32: the point half a substep back (cell and offset) and, from
// stochastic_reflection (cpp/fluid_colloid_collision.cpp:7-24, in FP32 with the same keyed draws
// as the FP64 form), the random point seen from there (part 0), the Rayleigh normal speed (part
// 1), the tangential Gaussians (part 2; the second only for the fixed rules).  bounce32_apply: the
// reflection in the colloid's frame, Rayleigh normal speed along rs plus the Gaussian along
// unit(un x t), the exchange (dv, dl), half a substep forward.
struct Bounce32 {
  int cx, cy, cz;
  float ox, oy, oz;
  f3 tt;
  float val, v1, v2;
};

// (explicitly rounded: the collisions run in several kernels, and left to the compiler the
// products and sums would be fused differently from one to the next)
static __device__ __forceinline__ float xd2(f3 a) {
  return __fmaf_rn(a.z, a.z, __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y)));
}
static __device__ __forceinline__ float xdet(float a, float b, float c, float d) {  // a b - c d
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}
static __device__ __forceinline__ f3 xcross(f3 a, f3 b) {
  return fm(xdet(a.y, b.z, a.z, b.y), xdet(a.z, b.x, a.x, b.z), xdet(a.x, b.y, a.y, b.x));
}
// (r: the first block of draws for parts 0 and 1, the second for part 2)
static __device__ __forceinline__ void bounce32_part(const SysF64 &S, uint32_t a, uint32_t b, uint32_t t, int part, uint4 r,
                                                     int cx, int cy, int cz, float ox, float oy, float oz, float vx,
                                                     float vy, float vz, Bounce32 &o) {
  if (part == 0) {
    ox = __fmaf_rn(__fmul_rn(-0.5f, vx), S.dtf, ox); oy = __fmaf_rn(__fmul_rn(-0.5f, vy), S.dtf, oy);
    oz = __fmaf_rn(__fmul_rn(-0.5f, vz), S.dtf, oz);
    carry(cx, ox, S.Lx); carry(cy, oy, S.Ly); carry(cz, oz, S.Lz);
    const f3 rf = fm(__fadd_rn((float)cx, ox), __fadd_rn((float)cy, oy), __fadd_rn((float)cz, oz));
    const float t0 = u01f(r.y), t1 = u01f(r.z), t2 = u01f(r.w);
    f3 tt = fm(__fmaf_rn(t0, S.Lxf, -rf.x), __fmaf_rn(t1, S.Lyf, -rf.y), __fmaf_rn(t2, S.Lzf, -rf.z));
    tt.x = __fmaf_rn(-S.Lxf, rintf(tt.x / S.Lxf), tt.x); tt.y = __fmaf_rn(-S.Lyf, rintf(tt.y / S.Lyf), tt.y); tt.z = __fmaf_rn(-S.Lzf, rintf(tt.z / S.Lzf), tt.z);
    o.cx = cx; o.cy = cy; o.cz = cz;
    o.ox = ox; o.oy = oy; o.oz = oz;
    o.tt = tt;
  } else if (part == 1) {
    const float u = u01f(r.x);
    const float om = 1.f - u;
    o.val = sqrtf(-logf(om * om) * (float)S.inv_m_beta);
  } else {
    // pairs of Box-Muller tries from the second block of draws on
    float x1 = 0.f, x2 = 0.f, z = 2.f;
    for (int it = 0; z > 1.f && it < 256; ++it) {
      if (it > 0 && (it & 1) == 0) r = draw4_loop(S.key, DOM_COLL, 1u + (uint32_t)(it >> 1), a, b, t);
      x1 = __fmaf_rn(2.f, u01f((it & 1) ? r.z : r.x), -1.f);
      x2 = __fmaf_rn(2.f, u01f((it & 1) ? r.w : r.y), -1.f);
      z = __fmaf_rn(x1, x1, __fmul_rn(x2, x2));
    }
    z = sqrtf(-2.f * logf(z) / z);
    o.v1 = x1 * z * (float)S.sqrt_kt_m;
    o.v2 = x2 * z * (float)S.sqrt_kt_m;
  }
}

static __device__ __noinline__ void bounce32_draw(const SysF64 &S, long long gs, int j, int id, int part, int cx,
                                                     int cy, int cz, float ox, float oy, float oz, float vx, float vy,
                                                     float vz, Bounce32 &o) {
  const uint32_t a = (uint32_t)(id + 1), b = (uint32_t)(j + 1), t = (uint32_t)gs;
  bounce32_part(S, a, b, t, part, draw4_loop(S.key, DOM_COLL, part == 2 ? 1 : 0, a, b, t), cx, cy, cz, ox, oy, oz, vx, vy,
                vz, o);
}

static __device__ __forceinline__ void bounce32_apply(const SysF64 &S, int j, float4 cq, float4 co, f3 vdump,
                                                      const Bounce32 &o, int &cx, int &cy, int &cz, float &ox,
                                                      float &oy, float &oz, float &vx, float &vy, float &vz, f3 &dv,
                                                      f3 &dl) {
  cx = o.cx; cy = o.cy; cz = o.cz;
  ox = o.ox; oy = o.oy; oz = o.oz;
  const f3 rs = fm(rel(cx, ox, cq.x, co.x, S.Lx), rel(cy, oy, cq.y, co.y, S.Ly), rel(cz, oz, cq.z, co.z, S.Lz));
  const float ir = rsqrtf(xd2(rs));
  const f3 n = fm(__fmul_rn(rs.x, ir), __fmul_rn(rs.y, ir), __fmul_rn(rs.z, ir));
  const f3 un = fm(__fmul_rn(n.x, o.val), __fmul_rn(n.y, o.val), __fmul_rn(n.z, o.val));
  const f3 ut = xcross(un, o.tt);
  const float iu = rsqrtf(xd2(ut));
  const f3 ti = fm(__fmul_rn(ut.x, iu), __fmul_rn(ut.y, iu), __fmul_rn(ut.z, iu));
  f3 u = fm(__fmaf_rn(ti.x, o.v1, un.x), __fmaf_rn(ti.y, o.v1, un.y), __fmaf_rn(ti.z, o.v1, un.z));
  if (S.physics) {  // the fixed rules: the second tangential component along n x unit(ut)
    const f3 t2 = xcross(n, ti);
    u = fm(__fmaf_rn(t2.x, o.v2, u.x), __fmaf_rn(t2.y, o.v2, u.y), __fmaf_rn(t2.z, o.v2, u.z));
  }
  const f3 V = fm((float)S.V[3 * j], (float)S.V[3 * j + 1], (float)S.V[3 * j + 2]);
  const f3 W = fm((float)S.W[3 * j], (float)S.W[3 * j + 1], (float)S.W[3 * j + 2]);
  const f3 wr = xcross(W, rs);
  vx = __fadd_rn(__fadd_rn(u.x, V.x), wr.x); vy = __fadd_rn(__fadd_rn(u.y, V.y), wr.y); vz = __fadd_rn(__fadd_rn(u.z, V.z), wr.z);
  dv = fm(vdump.x - vx, vdump.y - vy, vdump.z - vz);
  dl = xcross(rs, dv);
  ox = __fmaf_rn(__fmul_rn(0.5f, vx), S.dtf, ox); oy = __fmaf_rn(__fmul_rn(0.5f, vy), S.dtf, oy);
  oz = __fmaf_rn(__fmul_rn(0.5f, vz), S.dtf, oz);
  carry(cx, ox, S.Lx); carry(cy, oy, S.Ly); carry(cz, oz, S.Lz);
}

// both halves at once, with the exchange added: in line, the draws shared, for the event pass (whose time is
// that of a few collisions in a row: 20^3, 20 colloids, 10.4 us, with the other form 13.7)
static __device__ __forceinline__ void bounce32_all(const SysF64 &S, long long gs, int j, float4 cq, float4 co, int id,
                                                    f3 vdump, int &cx, int &cy, int &cz, float &ox, float &oy,
                                                    float &oz, float &vx, float &vy, float &vz) {
  const uint32_t a = (uint32_t)(id + 1), b = (uint32_t)(j + 1), t = (uint32_t)gs;
  const uint4 r0 = draw4(S.key, DOM_COLL, 0, a, b, t), r1 = draw4(S.key, DOM_COLL, 1, a, b, t);
  Bounce32 o;
#pragma unroll
  for (int part = 0; part < 3; ++part)
    bounce32_part(S, a, b, t, part, part == 2 ? r1 : r0, cx, cy, cz, ox, oy, oz, vx, vy, vz, o);
  f3 dv, dl;
  bounce32_apply(S, j, cq, co, vdump, o, cx, cy, cz, ox, oy, oz, vx, vy, vz, dv, dl);
  exch_add6(S.exch + j, mk(dv.x, dv.y, dv.z), mk(dl.x, dl.y, dl.z), &S.ss->err);
}

// out of line, for the cooperative substeps' rare cases
static __device__ __noinline__ void bounce32(const SysF64 &S, long long gs, int j, float4 cq, float4 co, int id, f3 vdump, int &cx,
                                int &cy, int &cz, float &ox, float &oy, float &oz, float &vx, float &vy, float &vz) {
  Bounce32 o;
  for (int part = 0; part < 3; ++part) bounce32_draw(S, gs, j, id, part, cx, cy, cz, ox, oy, oz, vx, vy, vz, o);
  f3 dv, dl;
  bounce32_apply(S, j, cq, co, vdump, o, cx, cy, cz, ox, oy, oz, vx, vy, vz, dv, dl);
  exch_add6(S.exch + j, mk(dv.x, dv.y, dv.z), mk(dl.x, dl.y, dl.z), &S.ss->err);
}

// One warp's wall collisions (cpp/fluid_colloid_collision.cpp:26-49) of the particles its
// lanes hold (act: the lane has one): each lane takes its colloids in ascending order, the
// ones whose sphere holds the particle, and the body of a collision (back half a substep,
// the FP32 stochastic reflection, the exact exchange sums, forward half a substep) runs
// once for all lanes that hit a colloid at that rank.  The whole warp calls it.
template <int FLAGS>
__device__ __forceinline__ void collide32_warp(const SysF64 &S, long long gs, int buf, bool act, int id, int cnt,
                                               const uint16_t *lst, int &cx, int &cy, int &cz, float &ox, float &oy,
                                               float &oz, float &vx, float &vy, float &vz) {
  const float4 *Xq = S.Xcq[buf], *Xo = S.Xco[buf];
  const float rc2 = S.r_coll * S.r_coll;
  const f3 vdump = fm(vx, vy, vz);
  bool more = act;
  int last = -1;
  while (__any_sync(FULL, more)) {
    int j = 0x7FFFFFFF;
    float4 cq = make_float4(0.f, 0.f, 0.f, 0.f), co = cq;
    if (more) {
      for (;;) {
        j = 0x7FFFFFFF;
        for (int k = 0; k < cnt; ++k) {
          int c = lst[k];
          if (c > last && c < j) j = c;
        }
        if (j == 0x7FFFFFFF) break;
        last = j;
        cq = Xq[j]; co = Xo[j];
        f3 r = fm(rel(cx, ox, cq.x, co.x, S.Lx), rel(cy, oy, cq.y, co.y, S.Ly), rel(cz, oz, cq.z, co.z, S.Lz));
        if (r.x * r.x + r.y * r.y + r.z * r.z <= rc2) break;
      }
      more = j != 0x7FFFFFFF;
    }
    __syncwarp();
    if (j == 0x7FFFFFFF) continue;
    bounce32_all(S, gs, j, cq, co, id, vdump, cx, cy, cz, ox, oy, oz, vx, vy, vz);
  }
}

// A particle after its wall collisions: the displacement check against the cell-table
// margin, on the last substep its run() record and its binning (from its state after
// the collisions), and its state written back.
template <int FLAGS>
__device__ __forceinline__ void finish32(const SysF64 &S, const Fluid32 &F, int p, int id, int buf, int cnt,
                                         const uint16_t *lst, int cx0, int cy0, int cz0, float ox0, float oy0,
                                         float oz0, int cx, int cy, int cz, float ox, float oy, float oz, float vx,
                                         float vy, float vz) {
  constexpr int flags = FLAGS;
  {
    // the cell table is built with a margin; a move beyond it could hide a colloid
    const float ex = rel(cx, ox, (float)cx0, ox0, S.Lx), ey = rel(cy, oy, (float)cy0, oy0, S.Ly),
                ez = rel(cz, oz, (float)cz0, oz0, S.Lz);
    if (ex * ex + ey * ey + ez * ez > (float)S.disp_margin2) atomicOr(&S.ss->err, ERRB_DISPLACE);
  }
  if (flags & F_SHELL) {
    const float4 *Xq = S.Xcq[buf], *Xo = S.Xco[buf];
    const float rs2 = S.r_shell * S.r_shell;
    ShellRec rec;
    rec.p = id;
    rec.n = 0;
    rec.pass = 0;
    for (int last = -1; rec.n < SHELL_J;) {
      int j = 0x7FFFFFFF;
      for (int k = 0; k < cnt; ++k) {
        int c = lst[k];
        if (c > last && c < j) j = c;
      }
      if (j == 0x7FFFFFFF) break;
      last = j;
      float4 cq = Xq[j], co = Xo[j];
      float dx = rel(cx, ox, cq.x, co.x, S.Lx), dy = rel(cy, oy, cq.y, co.y, S.Ly), dz = rel(cz, oz, cq.z, co.z, S.Lz);
      if (dx * dx + dy * dy + dz * dz <= rs2) rec.j[rec.n++] = (uint16_t)j;
    }
    if (rec.n) {
      int idx = atomicAdd(&S.ss->nshell, 1);
      if (idx < S.shell_cap) S.shell[idx] = rec;
      else atomicOr(&S.ss->err, ERRB_SHELL);
    }
  }
  if (flags & F_BINROT) bin32(S, p, cx, cy, cz, ox, oy, oz, vx, vy, vz);
  F.q[p] = pack(cx, cy, cz, ox, oy, oz);
  F.vx[p] = vx; F.vy[p] = vy; F.vz[p] = vz;
}

// STREAM32_U particles per thread (thread t of block b: particles b * 256 U + t +
// 256 u), their loads issued together so more memory requests are in flight
#ifndef STREAM32_U
#define STREAM32_U 2
#endif
// the pass that also records run() candidates and bins keeps one particle per thread
// (its register count, and so its occupancy)
#ifndef STREAM32_U_SHELL
#define STREAM32_U_SHELL 1
#endif
static constexpr __host__ __device__ int stream32_u(int flags) { return (flags & F_SHELL) ? STREAM32_U_SHELL : STREAM32_U; }
// One chunk of 256 U particles: the particles i = chunk * 256 U + threadIdx.x + 256 u
// below `count` of the fluid (NEAR false: slot i) or of the near list (NEAR true: slot
// near[i], the free-flight schedule's per-substep passes).  The whole block calls it.
template <int FLAGS, bool NEAR>
static __device__ __forceinline__ void stream32_chunk(const SysF64 &S, const int chunk, const int count, int l,
                                                      int fb) {
  constexpr int flags = FLAGS;
  constexpr int U = stream32_u(FLAGS);
  const long long step = S.ss->step;
  const long long gs = step * S.n_sub + (l - 1);
  const Fluid32 F = fluid32_at(S, fb);
  const int i0 = chunk * (256 * U) + threadIdx.x;
  const int buf = (int)(gs & 1);
  int cx[U], cy[U], cz[U], pp[U];
  float ox[U], oy[U], oz[U], vx[U], vy[U], vz[U];
  bool valid[U], ev[U];
  unsigned members[U];
  int cnt[U], lin[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int i = i0 + 256 * u;
    valid[u] = i < count;
    ev[u] = false;
    members[u] = 0;
    cnt[u] = 0;
    lin[u] = 0;
    pp[u] = i;
    if (valid[u]) {
      const int p = NEAR ? S.near[i] : i;
      pp[u] = p;
      unpack(F.q[p], cx[u], cy[u], cz[u], ox[u], oy[u], oz[u]);
      vx[u] = F.vx[p]; vy[u] = F.vy[p]; vz[u] = F.vz[p];
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!valid[u]) continue;
    if (flags & F_STREAM) {
      ox[u] = fmaf(vx[u], S.dtf, ox[u]); oy[u] = fmaf(vy[u], S.dtf, oy[u]); oz[u] = fmaf(vz[u], S.dtf, oz[u]);
      carry(cx[u], ox[u], S.Lx); carry(cy[u], oy[u], S.Ly); carry(cz[u], oz[u], S.Lz);
    }
    lin[u] = cx[u] + S.Lx * (cy[u] + S.Ly * cz[u]);
    if (flags & (F_COLLIDE | F_SHELL)) cnt[u] = tcount(S.Tcnt[buf][lin[u]], gs);
  }
  float rr[3] = {0.f, 0.f, 0.f};
  if (flags & F_BINROT)
    for (int k = 0; k < 3; ++k) rr[k] = S.ss->rrf[k];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    BinTerm32 bt{-1, 0, 0, 0, 0};
    if (valid[u] && (flags & (F_COLLIDE | F_SHELL)) && cnt[u] > 0) {
      cnt[u] = cnt[u] < TCAP ? cnt[u] : TCAP;
      const uint16_t *lst = S.Tlist[buf] + (size_t)lin[u] * TCAP;
      const float4 *Xq = S.Xcq[buf], *Xo = S.Xco[buf];
      const float rc2 = S.r_coll * S.r_coll, rs2 = S.r_shell * S.r_shell;
      for (int k = 0; k < cnt[u]; ++k) {
        const int j = lst[k];
        const float4 cq = Xq[j], co = Xo[j];
        const float dx = rel(cx[u], ox[u], cq.x, co.x, S.Lx), dy = rel(cy[u], oy[u], cq.y, co.y, S.Ly),
                    dz = rel(cz[u], oz[u], cq.z, co.z, S.Lz);
        const float d2 = dx * dx + dy * dy + dz * dz;
        if (flags & F_COLLIDE) ev[u] |= d2 <= rc2;
        if ((flags & F_SHELL) && d2 <= rs2) members[u] |= 1u << k;
      }
    }
    const int p = pp[u];
    if (valid[u] && !ev[u] && (flags & F_BINROT))
      bt = bin32_term(S, rr, p, cx[u], cy[u], cz[u], ox[u], oy[u], oz[u], vx[u], vy[u], vz[u]);
    if (flags & F_BINROT) bin_add_warp(S.acc, bt.c, bt.fx, bt.fy, bt.fz, bt.f2);  // the whole warp
    if (valid[u] && (flags & F_STREAM)) F.q[p] = pack(cx[u], cy[u], cz[u], ox[u], oy[u], oz[u]);
  }
  // appends: events one atomic per warp (no block barrier), run() candidate
  // records (last substep) one atomic per block for all U rounds
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  unsigned mrecs[U];
  int nrec = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    mrecs[u] = __ballot_sync(FULL, (flags & F_SHELL) && valid[u] && !ev[u] && members[u] != 0);
    nrec += __popc(mrecs[u]);
  }
  int brec = 0;
  if (flags & F_SHELL) brec = block_base_n(&S.ss->nshell, nrec, lane);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int p = pp[u];
    const unsigned mrec = mrecs[u];
    const bool has_rec = (mrec >> lane) & 1u;
    const unsigned mev = __ballot_sync(FULL, ev[u]);
    int bev = 0;
    if (lane == 0 && mev) bev = atomicAdd(&S.ss->nevents, __popc(mev));
    bev = __shfl_sync(FULL, bev, 0);
    if (ev[u]) {
      const int i = bev + __popc(mev & lt);
      if (i < S.events_cap) S.events[i] = p;
      else atomicOr(&S.ss->err, ERRB_EVENTS);
    }
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
    brec += __popc(mrec);
  }
}

template <int FLAGS>
static __device__ __forceinline__ void k_stream32_body(const SysF64 &S, const int VB, const int NVB, int l, int fb) {
  stream32_chunk<FLAGS, false>(S, VB, S.N, l, fb);
}

template <int FLAGS>
__global__ void __launch_bounds__(256) k_stream32(__grid_constant__ const SysF64 S, int l, int fb) {
  k_stream32_body<FLAGS>(S, blockIdx.x, gridDim.x, l, fb);
}

// the same over a batch of systems (persistent: batch_for)
template <int FLAGS>
__global__ void __launch_bounds__(256) k_stream32_b(const SysF64 *Ss, const int *boff, int nrep, int l, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_stream32_body<FLAGS>(sS, VB, NVB, l, fb); });
}

int stream32_per_thread(int flags) { return stream32_u(flags); }

// ------------------------------------------------------------ free-flight schedule
//
// Between two SRD collisions a fluid particle moves in a straight line unless a colloid
// wall reflects it or run() kicks it, and both need a colloid within the run() shell
// radius r_shell.  A particle farther than r_shell + (its travel in the step) + (the
// colloids' largest move in the step) + slack from every colloid at the start of the
// step can meet neither in any substep: the per-substep passes would only stream it and,
// on the last substep, bin it.  The free-flight pass does that for such a particle
// (k_free_flight32: the same FP32 operations substep by substep, so the same bits), beside
// the substeps of the other particles, which the rotation pass lists (k_rotate_classify32)
// and the per-substep passes walk (k_stream32_near).  The colloids' move is bounded by
// n_sub cm (the colloid finish fails a step in which one moves further in a substep); a
// particle's travel by n_sub dt |v| (particles faster than the table allows are near);
// the slack of 0.01 covers the FP32 rounding of the distances and offsets.

// reach of the flight table: colloids within it of a cell's box can come within a
// particle's near radius of a particle in the cell
static __device__ __forceinline__ float flight_reach(const SysF64 &S) {
  return S.r_shell + S.flight_rx + (float)S.n_sub * S.ss->cm + 0.02f;
}

// the flight table of this step (both forms: the colloids' cell + offset copies are kept by
// both): colloid j (its position at the start of the step) in every cell whose box comes
// within the flight reach of it, the own box included.  A cell
// with more than FLIGHT_CAP colloids keeps counting; its particles are all near (near_list).  Block 0
// also empties the near list and draws the next step's grid shift for the free pass.
static __device__ __forceinline__ void k_flight_table32_body(const SysF64 &S, const int j) {
  const long long step = S.ss->step;
  if (j == 0 && threadIdx.x == 0) {
    S.ss->nnear = 0;
    S.ss->nact = 0;
    S.ss->cm_f = S.ss->cm;
    S.ss->step_f = step;
    S.bar[BAR_COLL] = S.bar[BAR_MOVE] = S.bar[BAR_EVX] = 0;
    shift_of(S, step + 2, S.ss->rrn);
  }
  if (j >= S.Nc) return;
  const int b0 = (int)((step * S.n_sub - 1) & 1);
  const float reach = flight_reach(S);
  if (threadIdx.x == 0) S.ccell[b0][j] = cell_coords(S, S.cbox[b0][j]);
  const float4 cq = S.Xcq[b0][j], co = S.Xco[b0][j];
  const int K = (int)ceilf(reach) + 1, side = 2 * K + 1;
  const int tot = side * side * side;
  // Along a side of L cells below 2 K + 1 the walk comes to a cell from both sides: of the offsets L apart
  // that lead to it the one counts whose cell's centre is the nearest, in [lo, lo + L).
  auto low = [](float c, int L) { return (int)floorf(c + 0.5f * (float)(L - 1)) - L + 1; };
  const int lx = low(co.x, S.Lx), ly = low(co.y, S.Ly), lz = low(co.z, S.Lz);
  const unsigned long long tag = (unsigned long long)(unsigned)(step + 1) << 32;
  for (int q = threadIdx.x; q < tot; q += blockDim.x) {
    const int ox = q % side - K, oy = (q / side) % side - K, oz = q / (side * side) - K;
    // gap from the colloid (its cell + offset co) to the box of cell (its cell + o)
    const float ex = ox > 0 ? (float)ox - co.x : (ox < 0 ? co.x - (float)ox - 1.f : 0.f);
    const float ey = oy > 0 ? (float)oy - co.y : (oy < 0 ? co.y - (float)oy - 1.f : 0.f);
    const float ez = oz > 0 ? (float)oz - co.z : (oz < 0 ? co.z - (float)oz - 1.f : 0.f);
    if (ex * ex + ey * ey + ez * ez > reach * reach) continue;
    if ((unsigned)(ox - lx) >= (unsigned)S.Lx || (unsigned)(oy - ly) >= (unsigned)S.Ly || (unsigned)(oz - lz) >= (unsigned)S.Lz)
      continue;
    int bx = ((int)cq.x + ox) % S.Lx, by = ((int)cq.y + oy) % S.Ly, bz = ((int)cq.z + oz) % S.Lz;
    bx += bx < 0 ? S.Lx : 0; by += by < 0 ? S.Ly : 0; bz += bz < 0 ? S.Lz : 0;
    FlightCell *fc = S.ftab + (bx + S.Lx * (by + S.Ly * bz));
    atomicMax(&fc->tc, tag);
    const int slot = (int)(unsigned)atomicAdd(&fc->tc, 1ull);
    if (slot < FLIGHT_CAP) fc->id[slot] = (uint16_t)j;
    // the particles of a crowded cell find their colloids in the cell tables (near_list), which are built in
    // this step; one may overflow, too
    if (slot == FLIGHT_CAP) S.ss->crowd = step + 1;
  }
}

__global__ void __launch_bounds__(128) k_flight_table32(__grid_constant__ const SysF64 S) {
  k_flight_table32_body(S, blockIdx.x);
}

// the same over a batch of systems (persistent: batch_for; max(Nc, 1) virtual blocks each)
// (32 registers, so that it leaves the cell pass beside it its place: with the 40 it would take, three
// systems of 16^3 to 32^3 273 us a step instead of 268)
__global__ void __launch_bounds__(128, 16) k_flight_table32_b(const SysF64 *Ss, const int *boff, int nrep) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int) { k_flight_table32_body(sS, VB); });
}

// rotation_mpcd of one particle (the SRD map of its cell; ROT false: a counting-sort step,
// whose scatter rotated it) and its classification: a near particle is flagged and appended to
// the near list (one atomic per block).
// U particles per thread (thread t of virtual block b: particles b 256 U + t + 256 u), their
// loads issued together so that more gathers are in flight
// SPLIT: of the near ones, those whose straight path may meet a sphere are also listed as
// active (k_near_step32)
template <bool ROT, bool SPLIT, int U>
static __device__ __forceinline__ void k_rotate_classify32_body(const SysF64 &S, const int VB, int fb) {
  const Fluid32 F = fluid32_at(S, fb);
  const long long step = S.ss->step;
  const int b0 = (int)((step * S.n_sub - 1) & 1);
  int pp[U], cc[U];
  bool valid[U], near[U];
  unsigned cand[U];  // (SPLIT: the colloids its path comes near)
  float vx[U], vy[U], vz[U];
  uint4 qq[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    pp[u] = VB * (256 * U) + (int)threadIdx.x + 256 * u;
    valid[u] = pp[u] < S.N;
    near[u] = false;
    cand[u] = NEAR_NONE;
    if (valid[u]) {
      const int p = pp[u];
      cc[u] = ROT ? S.rotcell[p] : S.C;
      vx[u] = F.vx[p]; vy[u] = F.vy[p]; vz[u] = F.vz[p];
      qq[u] = F.q[p];
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!valid[u]) continue;
    const int p = pp[u];
    int cx, cy, cz;
    float ox, oy, oz;
    unpack(qq[u], cx, cy, cz, ox, oy, oz);
    const bool inb = cx < S.Lx && cy < S.Ly && cz < S.Lz;  // (a record within the box)
    const FlightCell *fc = S.ftab + (inb ? cx + S.Lx * (cy + S.Ly * cz) : 0);
    const uint4 w0 = reinterpret_cast<const uint4 *>(fc)[0];
    if (ROT) {
      if (cc[u] < S.C) apply_map32(S.cell_ab32 + (size_t)cc[u] * 12, vx[u], vy[u], vz[u]);
      F.vx[p] = vx[u]; F.vy[p] = vy[u]; F.vz[p] = vz[u];
    }
    const float travel = (float)S.n_sub * S.dtf * sqrtf(vx[u] * vx[u] + vy[u] * vy[u] + vz[u] * vz[u]);
    int cnt = tcount(((unsigned long long)w0.y << 32) | w0.x, step);
    bool nr = false;
    if (!inb || !(travel <= S.flight_rv) || cnt > FLIGHT_CAP) {
      nr = true;  // faster than the table allows (or not finite), or a crowded cell
      cand[u] = NEAR_WILD;
    } else if (cnt > 0) {
      const float rad = near_radius(S, S.ss->cm, S.n_sub), T = (float)S.n_sub * S.dtf;
      const float r = S.r_shell + travel + (float)S.n_sub * S.ss->cm + 0.01f, r2 = r * r;
      if (r > S.near_img) {  // (a box as narrow as that: other copies of the spheres matter)
        nr = true;
        cand[u] = NEAR_WILD;
        cnt = 0;
      }
      // (four ids lie in the first half of the record)
      const uint4 w1 = cnt > 4 ? reinterpret_cast<const uint4 *>(fc)[1] : make_uint4(0, 0, 0, 0);
      const unsigned ids[6] = {w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      const float4 *Xq = S.Xcq[b0], *Xo = S.Xco[b0];
      for (int k = 0; k < cnt; ++k) {
        const int j = (int)((ids[k >> 1] >> (16 * (k & 1))) & 0xFFFFu);
        const float4 cq = Xq[j], co = Xo[j];
        const float dx = rel(cx, ox, cq.x, co.x, S.Lx), dy = rel(cy, oy, cq.y, co.y, S.Ly),
                    dz = rel(cz, oz, cq.z, co.z, S.Lz);
        if (!(dx * dx + dy * dy + dz * dz > r2)) {
          nr = true;
          if (SPLIT && path_meets(dx, dy, dz, T * vx[u], T * vy[u], T * vz[u], rad)) cand[u] = near_add(cand[u], j);
        }
      }
    }
    near[u] = nr;
    S.fnear[p] = nr ? (SPLIT && cand[u] != NEAR_NONE ? FN_ACTIVE : FN_NEAR) : FN_FREE;
  }
  // the near list: one atomic per block for all U rounds
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  unsigned m[U];
  int tot = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    m[u] = __ballot_sync(FULL, near[u]);
    tot += __popc(m[u]);
  }
  int base, ba = 0;
  unsigned ma[U];
  if (SPLIT) {
    int tota = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      ma[u] = __ballot_sync(FULL, cand[u] != NEAR_NONE);
      tota += __popc(ma[u]);
    }
    block_base2(&S.ss->nnear, tot, tota, lane, &base, &ba);
  } else {
    base = block_base_n(&S.ss->nnear, tot, lane);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (near[u]) S.near[base + __popc(m[u] & lt)] = pp[u];
    base += __popc(m[u]);
    if (!SPLIT) continue;
    if (cand[u] != NEAR_NONE) {
      S.act[ba + __popc(ma[u] & lt)] = pp[u];
      S.actc[ba + __popc(ma[u] & lt)] = cand[u];
    }
    ba += __popc(ma[u]);
  }
}

template <bool ROT, bool SPLIT>
__global__ void __launch_bounds__(256) k_rotate_classify32(__grid_constant__ const SysF64 S, int fb) {
  k_rotate_classify32_body<ROT, SPLIT, CLASSIFY32_U>(S, blockIdx.x, fb);
}

// the same over a batch of systems (persistent: batch_for)
template <bool ROT, bool SPLIT>
__global__ void __launch_bounds__(256) k_rotate_classify32_b(const SysF64 *Ss, const int *boff, int nrep, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int) { k_rotate_classify32_body<ROT, SPLIT, CLASSIFY32_U>(sS, VB, fb); });
}

// n streaming substeps along one axis: the streaming passes' o = fma(v, dt, o) and carry, n
// times, without a branch: carry's floor leaves an offset in [0, 1) as it is, so it is taken
// every time, and the cells carried are added up and wrapped into the box once at the end
// (integer sums, the same cell).  What carry does with a NaN or runaway offset is left out: its
// particle fails the range test of the binning.
static __device__ __noinline__ float2 free_axis32(float o, float v, float dt, int n) {
  float k = 0.f;
#pragma unroll 1
  for (int l = 0; l < n; ++l) {
    o = fmaf(v, dt, o);
    const float f = floorf(o);
    o -= f;
    k += f;
    if (o >= 1.f) { o = 0.f; k += 1.f; }
  }
  return make_float2(o, k);
}

// The same for the three axes where no substep's move reaches a cell's width (slow), without rounding
// instructions: the offset leaves [0, 1) only on the side it moves to, by less than 1, so carry adds a =
// -1 or 1 there (exactly floor's result); the cells carried are the whole number nearest to what the n
// moves sum up to less what the offset shows.  An offset that rounds up to 1 on its way back
// (carry makes it 0 and carries less) is left to free_axis32.  The unsigned comparison of the bits is true
// for every offset outside [0, 1).
static __device__ __forceinline__ void free_axes32(int &cx, int &cy, int &cz, float &ox, float &oy, float &oz, float vx,
                                                   float vy, float vz, float dt, int n, bool slow, int Lx, int Ly,
                                                   int Lz) {
  const float x0 = ox, y0 = oy, z0 = oz;
  float kx, ky, kz;
  bool redo = !slow;
  if (slow) {
    const float ax = vx < 0.f ? 1.f : -1.f, ay = vy < 0.f ? 1.f : -1.f, az = vz < 0.f ? 1.f : -1.f;
    float top = 0.f;
    auto move = [&](float &o, float v, float a) {
      o = fmaf(v, dt, o);
      if (__float_as_uint(o) >= 0x3f800000u) o = __fadd_rn(o, a);
      top = fmaxf(top, o);
    };
#pragma unroll 2
    for (int l = 0; l < n; ++l) {
      move(ox, vx, ax);
      move(oy, vy, ay);
      move(oz, vz, az);
    }
    const float T = (float)n * dt;
    kx = rintf(fmaf(vx, T, x0) - ox);
    ky = rintf(fmaf(vy, T, y0) - oy);
    kz = rintf(fmaf(vz, T, z0) - oz);
    redo = !(top < 1.f);
  }
  if (redo) {
    const float2 a = free_axis32(x0, vx, dt, n), b = free_axis32(y0, vy, dt, n), c = free_axis32(z0, vz, dt, n);
    ox = a.x; oy = b.x; oz = c.x;
    kx = a.y; ky = b.y; kz = c.y;
  }
  auto wrap = [](int c, int L) {
    if (c < 0 || c >= L) {
      c %= L;
      if (c < 0) c += L;
    }
    return c;
  };
  cx = wrap(cx + (int)kx, Lx);
  cy = wrap(cy + (int)ky, Ly);
  cz = wrap(cz + (int)kz, Lz);
}

// the free particles' whole step: n_sub streaming substeps (update_pos_mpcd, the
// streaming passes' operations in order) and the binning of the last substep with the
// next step's grid shift.  Runs beside the near particles' substeps, which touch none of
// its particles; a grid of a few blocks per SM walks the fluid (it shares the SMs with the
// substeps' latency-bound chain), each thread's next particle loaded while this one is worked on.
// (thr: the flag from which on a particle is not this pass's: 1, or 2 where the near ones that
// no sphere can reach are streamed here too)
// Particles p, p + stride, ... below end.
static __device__ __forceinline__ void k_free_flight32_body(const SysF64 &S, int p, const int stride, const int end,
                                                            int fb, int thr) {
  const Fluid32 F = fluid32_at(S, fb);
  const float rr[3] = {(float)S.ss->rrn[0], (float)S.ss->rrn[1], (float)S.ss->rrn[2]};
  const int n = S.n_sub;
  // (a free particle's moves of a step sum up to flight_rv at most)
  const bool slow = S.flight_rv <= 0.5f * (float)n;
  uint4 q = make_uint4(0, 0, 0, 0);
  float wx = 0.f, wy = 0.f, wz = 0.f;
  int fn = 255;
  auto load = [&](int i) {
    fn = 255;
    if (i < end) {
      fn = S.fnear[i];
      q = F.q[i];
      wx = F.vx[i]; wy = F.vy[i]; wz = F.vz[i];
    }
  };
  load(p);
  for (int p0 = p - (int)threadIdx.x; p0 < end; p0 += stride, p += stride) {
    const bool free = fn < thr;
    const float vx = wx, vy = wy, vz = wz;
    int cx, cy, cz;
    float ox, oy, oz;
    unpack(q, cx, cy, cz, ox, oy, oz);
    load(p + stride);
    BinTerm32 bt{-1, 0, 0, 0, 0};
    if (free) {
      free_axes32(cx, cy, cz, ox, oy, oz, vx, vy, vz, S.dtf, n, slow, S.Lx, S.Ly, S.Lz);
      bt = bin32_term(S, rr, p, cx, cy, cz, ox, oy, oz, vx, vy, vz);
      F.q[p] = pack(cx, cy, cz, ox, oy, oz);
    }
    bin_add_warp(S.acc, bt.c, bt.fx, bt.fy, bt.fz, bt.f2);  // the whole warp
  }
}

__global__ void __launch_bounds__(256) k_free_flight32(__grid_constant__ const SysF64 S, int fb, int thr) {
  k_free_flight32_body(S, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, S.N, fb, thr);
}

// the same over a batch of systems (persistent: batch_runs; a virtual block per FREE32_CHUNK particles)
__global__ void __launch_bounds__(256, 5) k_free_flight32_b(const SysF64 *Ss, const int *boff, int nrep, int fb,
                                                         int thr) {
  __shared__ SysF64 sS;
  batch_runs(Ss, boff, nrep, sS, [&](int v0, int v1, int) {
    k_free_flight32_body(sS, v0 * FREE32_CHUNK + (int)threadIdx.x, 256, min(sS.N, v1 * FREE32_CHUNK), fb, thr);
  });
}

// the per-substep pass over the near list (stride over chunks of 256 U)
template <int FLAGS>
static __device__ __forceinline__ void k_stream32_near_body(const SysF64 &S, const int VB, const int NVB, int l,
                                                            int fb) {
  const int count = S.ss->nnear;
  constexpr int per = 256 * stream32_u(FLAGS);
  for (int chunk = VB; chunk * per < count; chunk += NVB) stream32_chunk<FLAGS, true>(S, chunk, count, l, fb);
}

template <int FLAGS>
__global__ void __launch_bounds__(256) k_stream32_near(__grid_constant__ const SysF64 S, int l, int fb) {
  k_stream32_near_body<FLAGS>(S, blockIdx.x, gridDim.x, l, fb);
}

// the same over a batch of systems (persistent: batch_for)
template <int FLAGS>
__global__ void __launch_bounds__(256) k_stream32_near_b(const SysF64 *Ss, const int *boff, int nrep, int l, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_stream32_near_body<FLAGS>(sS, VB, NVB, l, fb); });
}

ClassifyKernel classify_kernel32(bool rotate, bool split) {
  return rotate ? (split ? k_rotate_classify32<true, true> : k_rotate_classify32<true, false>)
                : (split ? k_rotate_classify32<false, true> : k_rotate_classify32<false, false>);
}

ClassifyKernelB classify_kernel32_b(bool rotate, bool split) {
  return rotate ? (split ? k_rotate_classify32_b<true, true> : k_rotate_classify32_b<true, false>)
                : (split ? k_rotate_classify32_b<false, true> : k_rotate_classify32_b<false, false>);
}

StreamKernelB stream_kernel32_near_b(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_stream32_near_b<F_STREAM | F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_stream32_near_b<F_STREAM | F_COLLIDE | F_SHELL | F_BINROT>;
  }
  return nullptr;
}

StreamKernel stream_kernel32_near(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_stream32_near<F_STREAM | F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_stream32_near<F_STREAM | F_COLLIDE | F_SHELL | F_BINROT>;
  }
  return nullptr;
}

// wall collisions of the listed particles in colloid order, then (last substep)
// their run() record and binning; one particle per lane
template <int FLAGS>
static __device__ __forceinline__ void k_events32_body(const SysF64 &S, const int VB, const int NVB, int l, int fb) {
  constexpr int flags = FLAGS;
  const long long step = S.ss->step;
  const long long gs = step * S.n_sub + (l - 1);
  const int buf = (int)(gs & 1);
  const Fluid32 F = fluid32_at(S, fb);
  const int n = min(S.ss->nevents, S.events_cap);
  const int k0 = (threadIdx.x & 31) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (int base = 0;; base += blockDim.x) {
    const int i = VB + NVB * (k0 + base);
    const bool valid = i < n;
    if (!__any_sync(FULL, valid)) break;
    const int p = valid ? S.events[i] : 0;
    int cx = 0, cy = 0, cz = 0;
    float ox = 0.f, oy = 0.f, oz = 0.f, vx = 0.f, vy = 0.f, vz = 0.f;
    int cnt = 0, id = 0;
    if (valid) {
      unpack(F.q[p], cx, cy, cz, ox, oy, oz);
      vx = F.vx[p]; vy = F.vy[p]; vz = F.vz[p];
      id = F.id[p];
    }
    const int lin = cx + S.Lx * (cy + S.Ly * cz);
    if (valid) {
      cnt = tcount(S.Tcnt[buf][lin], gs);
      cnt = cnt < TCAP ? cnt : TCAP;
    }
    const uint16_t *lst = S.Tlist[buf] + (size_t)lin * TCAP;
    const int cx0 = cx, cy0 = cy, cz0 = cz;
    const float ox0 = ox, oy0 = oy, oz0 = oz;
    if (flags & F_COLLIDE) collide32_warp<FLAGS>(S, gs, buf, valid, id, cnt, lst, cx, cy, cz, ox, oy, oz, vx, vy, vz);
    if (!valid) continue;
    finish32<FLAGS>(S, F, p, id, buf, cnt, lst, cx0, cy0, cz0, ox0, oy0, oz0, cx, cy, cz, ox, oy, oz, vx, vy, vz);
  }
}

template <int FLAGS>
__global__ void __launch_bounds__(128) k_events32(__grid_constant__ const SysF64 S, int l, int fb) {
  k_events32_body<FLAGS>(S, blockIdx.x, gridDim.x, l, fb);
}

// the same over a batch of systems (persistent: batch_for)
template <int FLAGS>
__global__ void __launch_bounds__(128) k_events32_b(const SysF64 *Ss, const int *boff, int nrep, int l, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_events32_body<FLAGS>(sS, VB, NVB, l, fb); });
}

StreamKernel stream_kernel32(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_stream32<F_STREAM | F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_stream32<F_STREAM | F_COLLIDE | F_SHELL | F_BINROT>;
    case F_SHELL | F_BINROT: return k_stream32<F_SHELL | F_BINROT>;
  }
  return nullptr;
}

EventKernel event_kernel32(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_events32<F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_events32<F_COLLIDE | F_SHELL | F_BINROT>;
    case F_SHELL | F_BINROT: return k_events32<F_SHELL | F_BINROT>;
  }
  return nullptr;
}

StreamKernelB stream_kernel32_b(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_stream32_b<F_STREAM | F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_stream32_b<F_STREAM | F_COLLIDE | F_SHELL | F_BINROT>;
    case F_SHELL | F_BINROT: return k_stream32_b<F_SHELL | F_BINROT>;
  }
  return nullptr;
}

EventKernelB event_kernel32_b(int flags) {
  switch (flags) {
    case F_STREAM | F_COLLIDE: return k_events32_b<F_COLLIDE>;
    case F_STREAM | F_COLLIDE | F_SHELL | F_BINROT: return k_events32_b<F_COLLIDE | F_SHELL | F_BINROT>;
    case F_SHELL | F_BINROT: return k_events32_b<F_SHELL | F_BINROT>;
  }
  return nullptr;
}

// SRD collision per cell (cpp/rotation_mpcd.cpp:14-49): cell mean from the exact
// sums, thermostat factor in FP64, rotation about the random axis in FP32, stored
// as the FP32 affine map v' = A v + b; plus the occupancy prefix of the counting sort.
static __device__ __forceinline__ void k_cell_prep32_body(const SysF64 &S, const int VB, int sort) {
  const int c = VB * blockDim.x + threadIdx.x;
  __shared__ __align__(16) CellAcc cells[256];
  take_cells(S, VB * 256, cells);
  CellAcc a = CellAcc{0, 0, 0, 0, 0, 0};
  if (c < S.Cpad) {
    a = cells[threadIdx.x];
    if (sort) S.cursor[c] = 0;
  }
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
    if (threadIdx.x == 0) S.blk_off[VB] = total;
  }
  if (c >= S.C) return;
  float4 *ab4 = reinterpret_cast<float4 *>(S.cell_ab32 + (size_t)c * 12);
  const int n = a.n;
  if (n > S.max_per_cell) atomicOr(&S.ss->err, ERRB_OCCUPANCY);
  if (n <= 1 || n > S.max_per_cell) {
    ab4[0] = make_float4(1.f, 0.f, 0.f, 0.f);
    ab4[1] = make_float4(1.f, 0.f, 0.f, 0.f);
    ab4[2] = make_float4(1.f, 0.f, 0.f, 0.f);
    return;
  }
  // mean and thermostat factor in FP64 from the exact sums
  // (2^-kw / n in one factor: the power-of-two scaling is exact)
  const double insw = S.insw_n[n];
  const double ux = (double)a.sx * insw, uy = (double)a.sy * insw, uz = (double)a.sz * insw;
  const double var = (double)a.s2 * S.inv_sw - (double)n * (ux * ux + uy * uy + uz * uz);
  // The factor sqrt(3 kT (n - 1) / (m var)) scales FP32 velocities, so it is needed to FP32
  // precision only: the variance in FP64 (from the exact sums, where the cancellation
  // happens), its reciprocal root in FP32 times sqrt(3 kT (n - 1) / m) (per n, from the host)
  const float s = var > 0 ? S.sq3kt_n32[n] * rsqrtf((float)var) : 1.f;
  // rotation axis rho = 2 ran - 1, phi = 2 pi ran (cpp/rotation_mpcd.cpp:19-20)
  uint4 r = draw4(S.key, DOM_AXIS, 0, (uint32_t)(c + 1), 0, (uint32_t)(S.ss->step + 1));
  const float rho = 2.f * u01f(r.x) - 1.f;
  float sp, cp;
  sincospif(2.f * u01f(r.y), &sp, &cp);
  const float sq = sqrtf(fmaxf(1.f - rho * rho, 0.f));
  const float r1 = cp * sq, r2 = sp * sq, r3 = rho;
  const float ct = (float)S.ct, st = (float)S.st, ict = (float)S.ict;
  const float i1 = ict * r1, i2 = ict * r2, i3 = ict * r3;
  const float R[9] = {i1 * r1 + ct, i1 * r2 - st * r3, i1 * r3 + st * r2,
                      i2 * r1 + st * r3, i2 * r2 + ct, i2 * r3 - st * r1,
                      i3 * r1 - st * r2, i3 * r2 + st * r1, i3 * r3 + ct};
  const float fx = (float)ux, fy = (float)uy, fz = (float)uz;
  float A[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) A[k] = s * R[k];
  const float b0 = fx - (A[0] * fx + A[1] * fy + A[2] * fz);
  const float b1 = fy - (A[3] * fx + A[4] * fy + A[5] * fz);
  const float b2 = fz - (A[6] * fx + A[7] * fy + A[8] * fz);
  ab4[0] = make_float4(A[0], A[1], A[2], A[3]);
  ab4[1] = make_float4(A[4], A[5], A[6], A[7]);
  ab4[2] = make_float4(A[8], b0, b1, b2);
}

__global__ void __launch_bounds__(256) k_cell_prep32(__grid_constant__ const SysF64 S, int sort) {
  k_cell_prep32_body(S, blockIdx.x, sort);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_cell_prep32_b(const SysF64 *Ss, const int *boff, int nrep, int sort) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int) { k_cell_prep32_body(sS, VB, sort); });
}

static __device__ __forceinline__ void k_rotate32_body(const SysF64 &S, const int VB, const int NVB, int fb) {
  const int p = VB * blockDim.x + threadIdx.x;
  if (p >= S.N) return;
  const int c = S.rotcell[p];
  if (c >= S.C) return;
  const Fluid32 F = fluid32_at(S, fb);
  float vx = F.vx[p], vy = F.vy[p], vz = F.vz[p];
  apply_map32(S.cell_ab32 + (size_t)c * 12, vx, vy, vz);
  F.vx[p] = vx; F.vy[p] = vy; F.vz[p] = vz;
}

__global__ void __launch_bounds__(256) k_rotate32(__grid_constant__ const SysF64 S, int fb) {
  k_rotate32_body(S, blockIdx.x, gridDim.x, fb);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_rotate32_b(const SysF64 *Ss, const int *boff, int nrep, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_rotate32_body(sS, VB, NVB, fb); });
}

static __device__ __forceinline__ void k_rotate_sort32_body(const SysF64 &S, const int VB, const int NVB, int src, int dst) {
  const int p = VB * blockDim.x + threadIdx.x;
  if (p >= S.N) return;
  const Fluid32 F = fluid32_at(S, src), G = fluid32_at(S, dst);
  const int c = S.rotcell[p];
  float vx = F.vx[p], vy = F.vy[p], vz = F.vz[p];
  if (c < S.C) apply_map32(S.cell_ab32 + (size_t)c * 12, vx, vy, vz);
  const unsigned act = __activemask();
  const unsigned grp = __match_any_sync(act, c);
  const int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&S.cursor[c], __popc(grp));
  base = __shfl_sync(grp, base, leader);
  const int slot = S.blk_off[c >> 8] + S.cell_off[c] + base + __popc(grp & ((1u << lane) - 1u));
  const int id = F.id[p];
  if (slot < 0 || slot >= S.N || id < 0 || id >= S.N) {
    atomicOr(&S.ss->err, ERRB_OCCUPANCY);
    return;
  }
  G.q[slot] = F.q[p];
  G.vx[slot] = vx; G.vy[slot] = vy; G.vz[slot] = vz;
  G.id[slot] = id;
  S.newpos[id] = slot;
}

__global__ void __launch_bounds__(256) k_rotate_sort32(__grid_constant__ const SysF64 S, int src, int dst) {
  k_rotate_sort32_body(S, blockIdx.x, gridDim.x, src, dst);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_rotate_sort32_b(const SysF64 *Ss, const int *boff, int nrep, int src, int dst) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_rotate_sort32_body(sS, VB, NVB, src, dst); });
}

// candidates of a particle for its next `rem` substeps, packed: the colloids its straight path
// comes near, from the flight table of its cell (positions in buffer b); NEAR_WILD where that
// does not cover them
static __device__ __forceinline__ unsigned near_cand32(const SysF64 &S, long long step, int rem, int b, int cx,
                                                       int cy, int cz, float ox, float oy, float oz, float vx,
                                                       float vy, float vz) {
  if (!(cx < S.Lx && cy < S.Ly && cz < S.Lz)) return NEAR_WILD;
  const float T = (float)rem * S.dtf;
  const float wx = T * vx, wy = T * vy, wz = T * vz;
  const float travel = sqrtf(wx * wx + wy * wy + wz * wz), rad = near_radius(S, S.ss->cm, rem);
  if (!(travel <= S.flight_rv) || rad + travel > S.near_img) return NEAR_WILD;
  const FlightCell *fc = S.ftab + lin_cell(S, cx, cy, cz);
  const int cnt = tcount(fc->tc, step);
  if (cnt > FLIGHT_CAP) return NEAR_WILD;
  unsigned cand = NEAR_NONE;
  for (int k = 0; k < cnt; ++k) {
    const int j = fc->id[k];
    const float4 cq = S.Xcq[b][j], co = S.Xco[b][j];
    if (path_meets(rel(cx, ox, cq.x, co.x, S.Lx), rel(cy, oy, cq.y, co.y, S.Ly), rel(cz, oz, cq.z, co.z, S.Lz), wx,
                   wy, wz, rad))
      cand = near_add(cand, j);
  }
  return cand;
}

// run() (cpp/run.cpp:17-24) on the FP32 fluid: rear-shell test against V + v0 ra
static __device__ __forceinline__ void k_run_shell32_body(const SysF64 &S, const int VB, const int NVB, int fb) {
  const int n = min(S.ss->nshell, S.shell_cap);
  const int b = (int)((S.ss->step * S.n_sub - 1) & 1);
  const float4 *Xq = S.Xcq[b], *Xo = S.Xco[b];
  const Fluid32 F = fluid32_at(S, fb);
  for (int i = VB * blockDim.x + threadIdx.x; i < n; i += NVB * blockDim.x) {
    ShellRec rec = S.shell[i];
    int p = S.newpos[rec.p];
    int cx, cy, cz;
    float ox, oy, oz;
    unpack(F.q[p], cx, cy, cz, ox, oy, oz);
    uint8_t pass = 0;
    for (int k = 0; k < rec.n; ++k) {
      int j = rec.j[k];
      float4 cq = Xq[j], co = Xo[j];
      float rx = rel(cx, ox, cq.x, co.x, S.Lx), ry = rel(cy, oy, cq.y, co.y, S.Ly), rz = rel(cz, oz, cq.z, co.z, S.Lz);
      double Vx = S.V[3 * j] + S.ra[3 * j] * S.v0, Vy = S.V[3 * j + 1] + S.ra[3 * j + 1] * S.v0,
             Vz = S.V[3 * j + 2] + S.ra[3 * j + 2] * S.v0;
      if (rx * (float)Vx + ry * (float)Vy + rz * (float)Vz <= 0.f) {
        pass |= (uint8_t)(1u << k);
        atomicAdd(&S.shell_cnt[j], 1);
      }
    }
    S.shell[i].pass = pass;
  }
}

__global__ void k_run_shell32(__grid_constant__ const SysF64 S, int fb) {
  k_run_shell32_body(S, blockIdx.x, gridDim.x, fb);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void k_run_shell32_b(const SysF64 *Ss, const int *boff, int nrep, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_run_shell32_body(sS, VB, NVB, fb); });
}

// (split: a near particle whose kicked path may meet a sphere becomes active)
static __device__ __forceinline__ void k_run_kick32_body(const SysF64 &S, const int VB, const int NVB, int fb,
                                                         bool split) {
  const int n = min(S.ss->nshell, S.shell_cap);
  const Fluid32 F = fluid32_at(S, fb);
  for (int i = VB * blockDim.x + threadIdx.x; i < n; i += NVB * blockDim.x) {
    ShellRec rec = S.shell[i];
    if (!rec.pass) continue;
    int p = S.newpos[rec.p];
    float vx = F.vx[p], vy = F.vy[p], vz = F.vz[p];
    for (int k = 0; k < rec.n; ++k) {
      if (!((rec.pass >> k) & 1)) continue;
      int j = rec.j[k];
      // M v0 / (m cnt) in FP32 (the velocity it changes is FP32): no double division
      const float f = S.kick32 / (float)S.shell_cnt[j];
      vx -= (float)S.ra[3 * j] * f; vy -= (float)S.ra[3 * j + 1] * f; vz -= (float)S.ra[3 * j + 2] * f;
    }
    F.vx[p] = vx; F.vy[p] = vy; F.vz[p] = vz;
    if (!split) continue;
    // an active particle's candidates are looked up anew (k_near_step32); another may become active
    if (S.fnear[p] == FN_ACTIVE) {
      S.fnear[p] = FN_KICKED;
    } else if (S.fnear[p] == FN_NEAR) {
      int cx, cy, cz;
      float ox, oy, oz;
      unpack(F.q[p], cx, cy, cz, ox, oy, oz);
      const int b0 = (int)((S.ss->step * S.n_sub - 1) & 1);
      const unsigned cand = near_cand32(S, S.ss->step, S.n_sub, b0, cx, cy, cz, ox, oy, oz, vx, vy, vz);
      if (cand == NEAR_NONE) continue;
      S.fnear[p] = FN_ACTIVE;
      const int at = atomicAdd(&S.ss->nact, 1);
      S.act[at] = p;
      S.actc[at] = cand;
    }
  }
}

__global__ void k_run_kick32(__grid_constant__ const SysF64 S, int fb, int split) {
  k_run_kick32_body(S, blockIdx.x, gridDim.x, fb, split != 0);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void k_run_kick32_b(const SysF64 *Ss, const int *boff, int nrep, int fb, int split) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_run_kick32_body(sS, VB, NVB, fb, split != 0); });
}

// ------------------------------------------------- active particles' substeps (FP32 form)

constexpr int NEAR32_CHK = 128, NEAR32_IDX = 1024;

// what the tests need of a colloid
struct __align__(16) NearCol32 {
  float4 q, o;
  int4 c;
  static __device__ __forceinline__ NearCol32 get(const SysF64 &S, int b, int j) {
    return {S.Xcq[b][j], S.Xco[b][j], S.ccell[b][j]};
  }
  static __device__ __forceinline__ void copy(const SysF64 &S, int b, int j, NearCol32 *to) {
    near_copy16(&to->q, &S.Xcq[b][j]);
    near_copy16(&to->o, &S.Xco[b][j]);
    near_copy16(&to->c, &S.ccell[b][j]);
  }
};

// A listed particle of k_near_step32 (entry k), as NearEv of the FP64 form: the colloids it can
// be inside of in the substep, and what its reflection off the first of them (jc) needs that no
// colloid position enters
struct NearChk {
  int k, id, jc, nc;
  Bounce32 b;
  uint16_t cd[4];
  bool slow;
};

// Per block: NEAR32_ACT active particles in shared memory (32 bytes each; more stay in the
// other fluid buffer, which is free between sorts), the list of those to test exactly (more
// than NEAR32_IDX: in that buffer too) and their preparations (beyond NEAR32_CHK: none).
struct Near32 {
  uint4 q[NEAR32_ACT];
  float v[3][NEAR32_ACT];
  unsigned cand[NEAR32_ACT];
  int idx[NEAR32_IDX];
  NearChk chk[NEAR32_CHK];
  NearCols<NearCol32> col;
};

// run() candidate record of a particle after the last substep: the colloids, in ascending
// order, whose boxes (of the substep before, buffer buf ^ 1) hold cell lin and whose run()
// shell holds the particle; hit: it collided in this substep (its record then ends silently at
// the first SHELL_J colloids, as the event pass's does)
static __device__ __forceinline__ void near_shell32(const SysF64 &S, long long step, int buf, int cx, int cy, int cz,
                                                    float ox, float oy, float oz, const NearCell &c, int id, bool hit,
                                                    ShellRec &rec) {
  const NearList q = near_list(S, step, step * S.n_sub + S.n_sub - 1, c.lin, false);
  const float rs2 = S.r_shell * S.r_shell;
  rec.p = id;
  rec.n = 0;
  rec.pass = 0;
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
    const float4 cq = S.Xcq[buf][j], co = S.Xco[buf][j];
    const float dx = rel(cx, ox, cq.x, co.x, S.Lx), dy = rel(cy, oy, cq.y, co.y, S.Ly), dz = rel(cz, oz, cq.z, co.z, S.Lz);
    if (!(xd2(fm(dx, dy, dz)) <= rs2) || !near_in_block(S, j, c, buf ^ 1)) continue;
    if (rec.n == SHELL_J) {
      if (!hit) atomicOr(&S.ss->err, ERRB_SHELLSLOTS);
      if (rec.j[SHELL_J - 1] < j) continue;
      --rec.n;
    }
    int at = rec.n++;
    for (; at > 0 && rec.j[at - 1] > j; --at) rec.j[at] = rec.j[at - 1];
    rec.j[at] = (uint16_t)j;
  }
}

// see near_step.cuh.  Eight particle warps; per substep the listed particles' collisions run one
// per lane, what does not wait for the colloids (Philox, logarithms) prepared beside the
// colloids' finish.
static __device__ __forceinline__ void near_step32(const SysF64 &S, const int VB, const int G, int fb) {
  constexpr int NT = NEAR32_BLOCK - 32 * (NEAR_CW + 1), NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Near32 &sm = *reinterpret_cast<Near32 *>(smem_raw);
  __shared__ double s_hx[NT][6];  // the exchanges of a round's collisions, and their colloids
  __shared__ int s_hj[NT];
  __shared__ int s_nh, s_nchk, s_hits, s_fin;
  __shared__ int s_flag[2];
  __shared__ NearPairs s_pairs;
  const int t = threadIdx.x;
  const int n = S.n_sub;
  if (t == 0) s_nh = s_nchk = s_hits = s_fin = 0;
  sm.col.clear(S, t, NEAR32_BLOCK);
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
  const float cm = S.ss->cm;
  const Fluid32 F = fluid32_at(S, fb), O = fluid32_at(S, 1 - fb);
  const int nact = min(S.ss->nact, S.N);
  const int a0 = (int)((long long)VB * nact / G), cnt = (int)((long long)(VB + 1) * nact / G) - a0;
  auto sync = [] { group_sync(1, NT); };
  auto pq = [&](int k) -> uint4 * { return k < NEAR32_ACT ? &sm.q[k] : O.q + a0 + k; };
  auto pv = [&](int c, int k) -> float * {
    if (k < NEAR32_ACT) return &sm.v[c][k];
    return (c == 0 ? O.vx : c == 1 ? O.vy : O.vz) + a0 + k;
  };
  auto idx = [&](int i) -> int * { return i < NEAR32_IDX ? &sm.idx[i] : O.id + a0 + i; };
#pragma unroll 4
  for (int k = t; k < cnt; k += NT) {
    const int p = S.act[a0 + k];
    const uint4 q = F.q[p];
    const float vx = F.vx[p], vy = F.vy[p], vz = F.vz[p];
    unsigned cand = S.actc[a0 + k];
    if (S.fnear[p] == FN_KICKED) {
      int cx, cy, cz;
      float ox, oy, oz;
      unpack(q, cx, cy, cz, ox, oy, oz);
      cand = near_cand32(S, step, n, (int)((g0 - 1) & 1), cx, cy, cz, ox, oy, oz, vx, vy, vz);
      S.fnear[p] = FN_ACTIVE;
    }
    *pq(k) = q;
    *pv(0, k) = vx; *pv(1, k) = vy; *pv(2, k) = vz;
    if (k < NEAR32_ACT) {
      sm.cand[k] = cand;
      sm.col.note(cand);
    }
  }
  sync();
  sm.col.load(S, (int)((g0 - 1) & 1), t, NT);
  for (int k = t; k < min(cnt, NEAR32_ACT); k += NT) sm.cand[k] = sm.col.slots(sm.cand[k]);
  sync();

  // update_pos_mpcd of substep l and a test against the positions of l - 1 with the
  // displacement bound as margin: the particles to test exactly at X(l) are listed and prepared
  auto advance = [&](int l) {
    const long long gs = g0 + (l - 1);
    const int xb = (int)(gs & 1) ^ 1;
    const float ch = S.r_coll + 1e-3f + cm, far = ch + S.disp_marginf + 1e-3f;
    const bool wide = ch > S.near_img;  // (a colloid's move may turn a distance into that of a nearer copy)
    // particle k by the general path
    auto one = [&](int k, unsigned cand) {
      uint4 *q = pq(k);
      const float vx = *pv(0, k), vy = *pv(1, k), vz = *pv(2, k);
      int cx, cy, cz;
      float ox, oy, oz;
      unpack(*q, cx, cy, cz, ox, oy, oz);
      ox = fmaf(vx, S.dtf, ox); oy = fmaf(vy, S.dtf, oy); oz = fmaf(vz, S.dtf, oz);
      carry(cx, ox, S.Lx); carry(cy, oy, S.Ly); carry(cz, oz, S.Lz);
      *q = pack(cx, cy, cz, ox, oy, oz);
      auto dist2 = [&](const NearCol32 &o) {
        const float dx = rel(cx, ox, o.q.x, o.o.x, S.Lx), dy = rel(cy, oy, o.q.y, o.o.y, S.Ly),
                    dz = rel(cz, oz, o.q.z, o.o.z, S.Lz);
        return dx * dx + dy * dy + dz * dz;
      };
      // (inside a sphere that its boxes leave out, a particle needs no exact test: the box rule first)
      auto reached = [&](const NearCol32 &o) {
        return (wide || dist2(o) <= ch * ch) && in_block3(S, o.c, cx, cy, cz);
      };
      bool e = false;
      if (cand == NEAR_WILD) {
        const NearList c = near_list(S, step, gs, lin_cell(S, cx, cy, cz), false);
        for (int m = 0; m < (c.brute ? S.Nc : c.cnt) && !e; ++m) e = reached(sm.col.at(S, xb, c.brute ? m : c.ids[m]));
      } else {
        for (unsigned r = cand; (r & 0xFFFFu) != 0xFFFFu && !e; r = (r >> 16) | 0xFFFF0000u)
          e = reached(sm.col.d[r & 0xFFFFu]);
      }
      if (e) *idx(atomicAdd(&s_nchk, 1)) = k;
    };
    // Two at a time and without a branch where they have one or two candidates: carry's result for an
    // offset in (-1, 2) (one that rounds up to 1 on its way back takes the general path, as do
    // candidates from the flight table), both distances, about 120 instructions each, interleaved.
    const int kept = min(cnt, NEAR32_ACT);
    const float chl = (ch + 1e-4f) * (ch + 1e-4f);
    for (int k0 = t; k0 < kept; k0 += 2 * NT) {
      unsigned cand[2];
      bool plain[2], close[2];
      uint4 q[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = min(k0 + u * NT, kept - 1);
        cand[u] = k0 + u * NT < kept ? sm.cand[k] : NEAR_GONE;
        q[u] = sm.q[k];
        int cx, cy, cz;
        float ox, oy, oz;
        unpack(q[u], cx, cy, cz, ox, oy, oz);
        ox = fmaf(sm.v[0][k], S.dtf, ox); oy = fmaf(sm.v[1][k], S.dtf, oy); oz = fmaf(sm.v[2][k], S.dtf, oz);
        plain[u] = (cand[u] >> 16) - (NEAR_STALE >> 16) > 2u;  // (none of the marks)
        auto side = [&](int &c, float &o, int L) {
          const bool up = o >= 1.f, down = o < 0.f;
          const float a = up ? -1.f : (down ? 1.f : 0.f);
          o = __fadd_rn(o, a);
          c += up ? 1 : (down ? -1 : 0);
          c = c < 0 ? L - 1 : (c >= L ? 0 : c);
          plain[u] = plain[u] && o >= 0.f && o < 1.f;
        };
        side(cx, ox, S.Lx); side(cy, oy, S.Ly); side(cz, oz, S.Lz);
        q[u] = pack(cx, cy, cz, ox, oy, oz);
        close[u] = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const unsigned j = h ? cand[u] >> 16 : cand[u] & 0xFFFFu;
          const NearCol32 &o = sm.col.d[min(j, (unsigned)(NearCols<NearCol32>::MAX - 1))];
          const float dx = rel(cx, ox, o.q.x, o.o.x, S.Lx), dy = rel(cy, oy, o.q.y, o.o.y, S.Ly),
                      dz = rel(cz, oz, o.q.z, o.o.z, S.Lz);
          if (j != 0xFFFFu && dx * dx + dy * dy + dz * dz <= chl) close[u] = close[u] || in_block3(S, o.c, cx, cy, cz);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = k0 + u * NT;
        if (plain[u]) {
          sm.q[k] = q[u];
          if (close[u]) *idx(atomicAdd(&s_nchk, 1)) = k;
        } else if (cand[u] != NEAR_GONE) {
          one(k, cand[u]);
        }
      }
    }
    for (int k = NEAR32_ACT + t; k < cnt; k += NT) one(k, NEAR_WILD);  // beyond shared memory
    sync();
    // the listed ones, one per thread (what they read of global memory is one latency for all):
    // the colloids each may be inside of (a second sphere is reached through a collision with the
    // first), ascending; jc: the first one the sphere and the colloid's move alone reach
    const int nchk = min(s_nchk, NEAR32_CHK);
    for (int i = t; i < nchk; i += NT) {
      NearChk &v = sm.chk[i];
      const int k = *idx(i);
      int cx, cy, cz;
      float ox, oy, oz;
      unpack(*pq(k), cx, cy, cz, ox, oy, oz);
      const NearList c = near_list(S, step, gs, lin_cell(S, cx, cy, cz), false);
      v.k = k;
      v.id = F.id[S.act[a0 + k]];
      v.jc = -1;
      v.nc = 0;
      v.slow = c.brute || far > S.near_img;
      for (int m = 0; m < c.cnt && !v.slow; ++m) {
        const int j = c.ids[m];
        const NearCol32 o = sm.col.at(S, xb, j);
        const float dx = rel(cx, ox, o.q.x, o.o.x, S.Lx), dy = rel(cy, oy, o.q.y, o.o.y, S.Ly),
                    dz = rel(cz, oz, o.q.z, o.o.z, S.Lz);
        const float d2 = dx * dx + dy * dy + dz * dz;
        if (d2 > far * far || !in_block3(S, o.c, cx, cy, cz)) continue;
        if (v.nc == 4) {
          v.slow = true;
          break;
        }
        int at = v.nc++;
        for (; at > 0 && v.cd[at - 1] > j; --at) v.cd[at] = v.cd[at - 1];
        v.cd[at] = (uint16_t)j;
        if (d2 <= ch * ch && (v.jc < 0 || j < v.jc)) v.jc = j;
      }
      if (v.jc < 0) v.nc = 0;
    }
    sync();
    // the preparations, 32 particles at a time, in three parts on different warps
    for (int q = t >> 5; q < 3 * ((nchk + 31) / 32); q += NW) {
      const int i = (q / 3) * 32 + (t & 31);
      if (i >= nchk) continue;
      NearChk &v = sm.chk[i];
      if (v.slow || v.nc == 0) continue;
      int cx, cy, cz;
      float ox, oy, oz;
      unpack(*pq(v.k), cx, cy, cz, ox, oy, oz);
      bounce32_draw(S, gs, v.jc, v.id, q % 3, cx, cy, cz, ox, oy, oz, *pv(0, v.k), *pv(1, v.k), *pv(2, v.k), v.b);
    }
    if (t == 0) s_nh = 0;
  };

  advance(1);
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
    // the listed particles' wall collisions at X(l), one per lane
    const int nchk = s_nchk;
    for (int base = 0;; base += NT) {
      const int i = base + t;
      const bool last_round = base + NT >= nchk;
      int hit = -1;
      if (i < nchk) {
        const int k = *idx(i);
        NearChk *v = i < NEAR32_CHK ? &sm.chk[i] : nullptr;
        if (!v || v->slow || v->nc) {
          int cx, cy, cz;
          float ox, oy, oz;
          unpack(*pq(k), cx, cy, cz, ox, oy, oz);
          float vx = *pv(0, k), vy = *pv(1, k), vz = *pv(2, k);
          const int cx0 = cx, cy0 = cy, cz0 = cz;
          const float ox0 = ox, oy0 = oy, oz0 = oz;
          const f3 vdump = fm(vx, vy, vz);
          const NearCell c{lin_cell(S, cx, cy, cz), cx, cy, cz, false};
          const float4 *Xq = S.Xcq[buf], *Xo = S.Xco[buf];
          const float rc2 = S.r_coll * S.r_coll;
          auto inside = [&](int j) {
            const float4 cq = Xq[j], co = Xo[j];
            return xd2(fm(rel(cx, ox, cq.x, co.x, S.Lx), rel(cy, oy, cq.y, co.y, S.Ly),
                          rel(cz, oz, cq.z, co.z, S.Lz))) <= rc2;
          };
          int hits = 0;
          int id = v ? v->id : -1;
          if (!v || v->slow) {  // nothing listed: by the general routine
            const NearList q = near_list(S, step, gs, c.lin, false);
#pragma unroll 1
            for (int j = near_next(S, q, -1, c, buf ^ 1); j >= 0; j = near_next(S, q, j, c, buf ^ 1)) {
              if (!inside(j)) continue;
              if (id < 0) id = F.id[S.act[a0 + k]];
              ++hits;
              bounce32(S, gs, j, Xq[j], Xo[j], id, vdump, cx, cy, cz, ox, oy, oz, vx, vy, vz);
            }
          } else {
            // the listed colloids that hold it, one after another (they are all it can reach: a
            // displacement beyond the margin fails the step)
            int m = 0, j = -1;
            auto next = [&] {
              for (; m < v->nc; ++m) {
                j = v->cd[m];
                if (inside(j)) break;
              }
            };
            next();
#pragma unroll 1
            while (m < v->nc) {
              if (j != v->jc) {
                // not the colloid that was prepared for, or a second sphere (one in a few substeps
                // somewhere, on one lane, with every block waiting for it): prepared now, by the
                // instructions that every substep runs
                v->jc = j;
#pragma unroll 1
                for (int part = 0; part < 3; ++part)
                  bounce32_draw(S, gs, j, id, part, cx, cy, cz, ox, oy, oz, vx, vy, vz, v->b);
              }
              ++hits;
              f3 dv, dl;
              bounce32_apply(S, j, Xq[j], Xo[j], vdump, v->b, cx, cy, cz, ox, oy, oz, vx, vy, vz, dv, dl);
              const int h = atomicAdd(&s_nh, 1);
              if (h < NT) {
                s_hj[h] = j;
                s_hx[h][0] = dv.x; s_hx[h][1] = dv.y; s_hx[h][2] = dv.z;
                s_hx[h][3] = dl.x; s_hx[h][4] = dl.y; s_hx[h][5] = dl.z;
              } else {
                exch_add6(S.exch + j, mk(dv.x, dv.y, dv.z), mk(dl.x, dl.y, dl.z), &S.ss->err);
              }
              ++m;
              next();
            }
          }
          if (hits) {
            atomicAdd(&s_hits, 1);
            // the candidates are looked up with a margin; a move beyond it could hide a colloid
            const float ex = rel(cx, ox, (float)cx0, ox0, S.Lx), ey = rel(cy, oy, (float)cy0, oy0, S.Ly),
                        ez = rel(cz, oz, (float)cz0, oz0, S.Lz);
            if (ex * ex + ey * ey + ez * ez > (float)S.disp_margin2) atomicOr(&S.ss->err, ERRB_DISPLACE);
            *pq(k) = pack(cx, cy, cz, ox, oy, oz);
            *pv(0, k) = vx; *pv(1, k) = vy; *pv(2, k) = vz;
            hit = k;
            const int p = S.act[a0 + k];
            F.vx[p] = vx; F.vy[p] = vy; F.vz[p] = vz;
            if (l == n) {
              // its run() record (by the cell it collided in) and binning
              ShellRec rec;
              near_shell32(S, step, buf, cx, cy, cz, ox, oy, oz, c, id, true, rec);
              if (rec.n) {
                const int at = atomicAdd(&S.ss->nshell, 1);
                if (at < S.shell_cap) S.shell[at] = rec;
                else atomicOr(&S.ss->err, ERRB_SHELL);
              }
              const float rr[3] = {(float)S.ss->rrn[0], (float)S.ss->rrn[1], (float)S.ss->rrn[2]};
              const BinTerm32 b = bin32_term(S, rr, p, cx, cy, cz, ox, oy, oz, vx, vy, vz);
              bin_add(S.acc + b.c, 1, b.fx, b.fy, b.fz, b.f2);
              S.fnear[p] = FN_DONE;
            }
          }
        }
      }
      sync();
      // the round's exchanges, a component per thread
      const int nh = min(s_nh, NT);
      for (int q = t; q < 6 * nh; q += NT) exch_add1(S.exch + s_hj[q / 6], q % 6, s_hx[q / 6][q % 6], &S.ss->err);
      sync();
      if (t == 0) {
        if (last_round) {
          bar_arrive(S.bar + BAR_COLL);
          s_nchk = 0;
        } else {
          s_nh = 0;
        }
      }
      if (hit >= 0 && hit < NEAR32_ACT && l < n) {  // its candidates from here on
        int cx, cy, cz;
        float ox, oy, oz;
        unpack(sm.q[hit], cx, cy, cz, ox, oy, oz);
        sm.cand[hit] = sm.col.slots(near_cand32(S, step, n - l, buf, cx, cy, cz, ox, oy, oz, sm.v[0][hit],
                                                sm.v[1][hit], sm.v[2][hit]));
      }
      if (last_round) break;
      sync();
    }
    near_copy_wait();
    sync();
    if (l < n) advance(l + 1);
  }

  // after the last substep: the positions back to the fluid arrays (the run() candidate records
  // and the binning are the end kernel's, except of what collided in this substep)
  for (int k = t; k < cnt; k += NT) F.q[S.act[a0 + k]] = *pq(k);
  if (t == 0 && s_hits) atomicAdd((unsigned long long *)&S.ss->ev_total, (unsigned long long)s_hits);
}

// (104 registers: the free-flight pass's two blocks fit beside it)
__global__ void __maxnreg__(104) k_near_step32(__grid_constant__ const SysF64 S, int fb) {
  near_step32(S, blockIdx.x, gridDim.x, fb);
}

// The same over a batch of systems, each on blocks of its own (boff: where they begin; the launch
// covers the blocks from `first` on), which meet only at their system's counters.
__global__ void __maxnreg__(104) k_near_step32_b(const SysF64 *Ss, const int *boff, int nrep, int first, int fb) {
  __shared__ SysF64 sS;
  __shared__ int s_r;
  const int v = first + blockIdx.x;
  for (int r = threadIdx.x; r < nrep; r += blockDim.x)
    if (boff[r] <= v && v < boff[r + 1]) s_r = r;
  __syncthreads();
  const int r = s_r;
  const int *src = reinterpret_cast<const int *>(Ss + r);
  int *dst = reinterpret_cast<int *>(&sS);
  for (int k = threadIdx.x; k < (int)(sizeof(SysF64) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
  __syncthreads();
  near_step32(sS, v - boff[r], boff[r + 1] - boff[r], fb);
}

size_t near_step32_smem() { return sizeof(Near32); }

// The end of a free-flight step, as k_end_flight64: the step counter and the next step's margin
// (block 0); the run() candidate records of the near particles and the binning of the active
// ones among them (the others)
static __device__ __forceinline__ void k_end_flight32_body(const SysF64 &S, const int VB, const int NVB, int fb) {
  if (VB == 0) {
    k_end_step_body(S, 0, S.ss->crowd == S.ss->step + 1);
    return;
  }
  const long long step = S.ss->step_f;
  const int buf = (int)((step * S.n_sub + S.n_sub - 1) & 1);
  const Fluid32 F = fluid32_at(S, fb);
  const float rr[3] = {(float)S.ss->rrn[0], (float)S.ss->rrn[1], (float)S.ss->rrn[2]};
  const int count = min(S.ss->nnear, S.N), lane = threadIdx.x & 31;
  const int stride = (NVB - 1) * 256;
  int i = (VB - 1) * 256 + threadIdx.x;
  int next = i < count ? S.near[i] : 0;
  for (int base = (VB - 1) * 256; base < count; base += stride, i += stride) {
    ShellRec rec;
    rec.n = 0;
    BinTerm32 b{-1, 0, 0, 0, 0};
    const int p = next;
    if (i + stride < count) next = S.near[i + stride];
    if (i < count) {
      const uint8_t fn = S.fnear[p];
      if (fn != FN_DONE) {
        int cx, cy, cz;
        float ox, oy, oz;
        unpack(F.q[p], cx, cy, cz, ox, oy, oz);
        const NearCell c{lin_cell(S, cx, cy, cz), cx, cy, cz, false};
        near_shell32(S, step, buf, cx, cy, cz, ox, oy, oz, c, F.id[p], false, rec);
        if (fn != FN_NEAR) b = bin32_term(S, rr, p, cx, cy, cz, ox, oy, oz, F.vx[p], F.vy[p], F.vz[p]);
      }
    }
    if (__any_sync(FULL, b.c >= 0)) bin_add_warp(S.acc, b.c, b.fx, b.fy, b.fz, b.f2);
    const unsigned m = __ballot_sync(FULL, rec.n != 0);
    const int at = block_base(&S.ss->nshell, m, lane) + __popc(m & ((1u << lane) - 1u));
    if (rec.n) {
      if (at < S.shell_cap) S.shell[at] = rec;
      else atomicOr(&S.ss->err, ERRB_SHELL);
    }
  }
}

__global__ void __launch_bounds__(256) k_end_flight32(__grid_constant__ const SysF64 S, int fb) {
  k_end_flight32_body(S, blockIdx.x, gridDim.x, fb);
}

// the same over a batch of systems (persistent: batch_for)
__global__ void __launch_bounds__(256) k_end_flight32_b(const SysF64 *Ss, const int *boff, int nrep, int fb) {
  __shared__ SysF64 sS;
  batch_for(Ss, boff, nrep, sS, [&](int VB, int NVB) { k_end_flight32_body(sS, VB, NVB, fb); });
}

// AoS doubles (particle order) -> FP32 records; download scatters back by id
__global__ void __launch_bounds__(256) k_aos_to_q(const SysF64 S, const double *pos, const double *vel, int fb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.N) return;
  const Fluid32 F = fluid32_at(S, fb);
  int c[3];
  float o[3];
  const int L[3] = {S.Lx, S.Ly, S.Lz};
  for (int k = 0; k < 3; ++k) {
    double x = pos[3 * (size_t)i + k];
    double fl = floor(x);
    double off = x - fl;
    long long ci = (long long)fl;
    float of = (float)off;
    if (of >= 1.f) { of = 0.f; ci += 1; }
    ci %= L[k];
    if (ci < 0) ci += L[k];
    c[k] = (int)ci;
    o[k] = of;
  }
  F.q[i] = pack(c[0], c[1], c[2], o[0], o[1], o[2]);
  F.vx[i] = (float)vel[3 * (size_t)i]; F.vy[i] = (float)vel[3 * (size_t)i + 1]; F.vz[i] = (float)vel[3 * (size_t)i + 2];
  F.id[i] = i;
  S.newpos[i] = i;
}

__global__ void __launch_bounds__(256) k_q_to_aos(const SysF64 S, double *pos, double *vel, int fb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.N) return;
  const Fluid32 F = fluid32_at(S, fb);
  int cx, cy, cz;
  float ox, oy, oz;
  unpack(F.q[i], cx, cy, cz, ox, oy, oz);
  const size_t o = 3 * (size_t)F.id[i];
  if (pos) { pos[o] = (double)cx + (double)ox; pos[o + 1] = (double)cy + (double)oy; pos[o + 2] = (double)cz + (double)oz; }
  if (vel) { vel[o] = F.vx[i]; vel[o + 1] = F.vy[i]; vel[o + 2] = F.vz[i]; }
}

}  // namespace bgb
