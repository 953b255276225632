// Colloid-only dynamics with the learned closure: the fluid is not simulated;
// each MPCD step the closure network predicts, from every colloid's features,
// the mean and log-variance of the momentum and angular momentum the fluid would
// give it, a Gaussian draw of that exchange is applied as an impulse, and the
// colloids then take the step's n_sub velocity-Verlet substeps with the WCA
// forces, the active kick (run(), cpp/run.cpp:13) and the orientation update
// (cpp/update.cpp:34-46, plus rotational diffusion Dr), in FP32.
//
// Per step, two kernels (CUDA graphs of one and of eight steps):
//   k_sur_net, one block per 16 colloids over the whole GPU (16 compute warps, one
//     producer warp): each colloid's neighbours (from candidate lists kept with a
//     skin, all pairs when they expire), its 81 network inputs and its force partners
//     for the step, the whole network (four layers, BF16 mma.sync with FP32
//     accumulation, activations in shared memory, the weights streamed through a
//     ring of shared-memory stages by bulk copies while the block computes) and the
//     Gaussian draw of the exchange;
//   the substeps, k_sur_md1 (one block) or k_sur_md (one cluster of 8 blocks): the active
//     kick and the n_sub velocity-Verlet substeps (each needs every colloid's new position: a
//     block barrier, or distributed shared memory and one cluster barrier, per substep); beside
//     them, on blocks of their own, the rotational-diffusion draws and the orientations.
// Within a graph each kernel is launched before the one before it has ended: its blocks are then
// placed, its weights and constants loaded, and it waits only for the state.
// Bound: the latency of that chain (500 colloids: 12 us of network, half of it the layers' shared-memory
// traffic, 13 us of substeps).  Measured, us a step, 500 / 2,000 colloids at volume fractions
// 0.1 / 0.2: 39.8 / 50.5 -> 28.4 / 41.5 (the orientation behind the network and the
// substeps behind its whole end: 37.7 / 48.4; a branch per pair in contact before that).
// The packed weights (the layout k_sur_net reads) are rebuilt from the network at
// every mpcd_surrogate_step call.  k_sur_features computes the inputs of the
// current state on request.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/brownian_gb300.h"
#include "traj_internal.h"
#include "common.cuh"
#include "mlp_internal.h"

namespace {

using namespace bgb;
typedef __nv_bfloat16 bf16;

constexpr int NF = MPCD_MLP_IN, NO = MPCD_MLP_OUT, KNEAR = 12, MAXC = MPCD_SURROGATE_MAX_COLLOIDS, CAND = 64;
constexpr int H = MPCD_MLP_HIDDEN, INP = MLP_IN_PADDED, OUTP = MLP_OUT_PADDED;
constexpr uint32_t DOM_SUR_KICK = 20, DOM_SUR_ROT = 21;
// Colloids up to which the substeps run in one block, else in a cluster of eight: the block's barrier
// is 0.6 us a substep cheaper, but its SM shares the pair forces among few schedulers.  Measured,
// us a step, block / cluster: 30 colloids 22.9 / 24.8, 200 26.1 / 27.0, 300 (volume fraction 0.2)
// 30.9 / 29.3, 500 37.7 / 36.3, 1,024 55.6 / 41.2 (the last two before the kernels overlapped).
constexpr int kMdBlockMax = 256;
constexpr int MAXF = 32;  // force partners per colloid (within the WCA cutoff plus the skin)

struct Sur {
  int Nc, n_sub;
  float L[3], iL[3];
  float M, I, dt, v0, rotdiff_s, ct_feat2;
  float sig6, sig12, eps, rc2, fc, rscan2, rlist2, half_skin2;
  float rc;          // WCA cutoff
  float *vmax;       // the largest colloid speed at the end of the last step
  long long *fast;   // steps in which a colloid moved more than half the step's partner skin
  uint2 key;
  long long *step;  // device step counter
  float4 *X, *V, *W, *ra, *f;
  float *feat;      // the last step's network inputs [Nc][81]
  float *out;       // the last step's normalised network outputs [Nc][16]
  float4 *imp;      // per-substep linear impulse of the drawn exchange [Nc], orientation at the step's start [Nc],
                    // per-substep share of the angular exchange [Nc] (w: the step's number)
  uint16_t *fpart;  // force partners [Nc][MAXF], ascending index
  uint8_t *fpn;     // their count
  uint16_t *nbl;    // candidate neighbours [Nc][CAND] (within rlist at the last rebuild), ascending index
  int *nbn;         // their count
  float4 *xref;     // positions at the last rebuild
  int *rebuild;     // a colloid moved more than half the skin since (or no lists yet)
  int *err;
  int drop_chunk;   // fault injection for tests: the producer does not issue this weight chunk (-1: none)
  float noise;      // scale of the drawn exchange's fluctuation (1: the network's variance, 0: its mean only)
  const uint4 *wpk;                   // the packed BF16 weights (k_sur_pack)
  const float *bias;                  // the network's biases [256][256][256][16]
  const float *xmean, *xistd;         // input normalisation
  const float *ymean, *yistd;         // output normalisation
};

// rintf and floorf of |t| < 2^22 by additions: the conversion unit that rounds takes four times as
// long, and the pair loops round three times a pair
__device__ __forceinline__ float rint_add(float t) { return __fadd_rn(__fadd_rn(t, 12582912.f), -12582912.f); }
__device__ __forceinline__ float floor_add(float t) {
  const float r = rint_add(t);
  return r > t ? r - 1.f : r;
}

// minimum image of a difference of two positions inside the box
__device__ __forceinline__ float wrapd(float d, float L, float iL) { return d - L * rint_add(__fmul_rn(d, iL)); }
// back into the box after a substep's move
__device__ __forceinline__ float boxed(float x, float L, float iL) { return x - L * floor_add(__fmul_rn(x, iL)); }

// the skin of a step's force partners (pairs within the cutoff plus it): 2.5 times the
// largest displacement the last step's speeds give, within [0.5, 2]; the candidate lists
// cover the largest
__device__ __forceinline__ float partner_skin(const Sur &S) {
  return fminf(fmaxf(2.5f * *S.vmax * S.dt * S.n_sub, 0.5f), 2.0f);
}


__device__ __forceinline__ float u01f(uint32_t w) { return ((float)(w >> 9) + 0.5f) * 1.1920928955078125e-7f; }

// Box-Muller pair from two draws
__device__ __forceinline__ float2 normal2(uint32_t a, uint32_t b) {
  const float r = sqrtf(-2.f * __logf(u01f(a)));
  float s, c;
  __sincosf(6.283185307179586f * u01f(b), &s, &c);
  return make_float2(__fmul_rn(r, c), __fmul_rn(r, s));  // (rounded, whatever they are added to)
}

// features of colloid j (one warp): V, Omega, ra, then the 12 nearest colloids
// within three radii (relative position, relative velocity), nearest first,
// ties by index, zero padded - the layout of brownian_gb300.closure.features
__global__ void __launch_bounds__(128) k_sur_features(const Sur S) {
  __shared__ float sd[4][64];
  __shared__ int sk[4][64];
  __shared__ int scnt[4];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * 4 + w;
  if (j >= S.Nc) return;
  if (lane == 0) scnt[w] = 0;
  __syncwarp();
  const float4 xj = S.X[j], vj = S.V[j];
  for (int k0 = 0; k0 < S.Nc; k0 += 32) {
    const int k = k0 + lane;
    float d2 = 1e30f;
    if (k < S.Nc && k != j) {
      const float4 xk = S.X[k];
      const float dx = wrapd(xk.x - xj.x, S.L[0], S.iL[0]), dy = wrapd(xk.y - xj.y, S.L[1], S.iL[1]),
                  dz = wrapd(xk.z - xj.z, S.L[2], S.iL[2]);
      d2 = dx * dx + dy * dy + dz * dz;
    }
    const bool in = d2 < S.ct_feat2;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, in);
    int base = 0;
    if (m) {
      const int leader = __ffs(m) - 1;
      if (lane == leader) base = atomicAdd(&scnt[w], __popc(m));
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
    }
    if (in) {
      const int slot = base + __popc(m & ((1u << lane) - 1u));
      if (slot < 64) {
        sd[w][slot] = d2;
        sk[w][slot] = k;
      }
    }
  }
  __syncwarp();
  const int cnt = min(scnt[w], 64);
  float *o = S.feat + (size_t)j * NF;
  const float4 wj = S.W[j], aj = S.ra[j];
  for (int c = lane; c < NF; c += 32) o[c] = 0.f;
  __syncwarp();
  if (lane == 0) {
    o[0] = vj.x; o[1] = vj.y; o[2] = vj.z; o[3] = wj.x; o[4] = wj.y; o[5] = wj.z; o[6] = aj.x; o[7] = aj.y; o[8] = aj.z;
  }
  for (int c = lane; c < cnt; c += 32) {
    const float d2 = sd[w][c];
    const int k = sk[w][c];
    int rank = 0;
    for (int e = 0; e < cnt; ++e) rank += (sd[w][e] < d2) || (sd[w][e] == d2 && sk[w][e] < k);
    if (rank < KNEAR) {
      const float4 xk = S.X[k], vk = S.V[k];
      float *q = o + 9 + 6 * rank;
      q[0] = wrapd(xk.x - xj.x, S.L[0], S.iL[0]);
      q[1] = wrapd(xk.y - xj.y, S.L[1], S.iL[1]);
      q[2] = wrapd(xk.z - xj.z, S.L[2], S.iL[2]);
      q[3] = vk.x - vj.x; q[4] = vk.y - vj.y; q[5] = vk.z - vj.z;
    }
  }
}

// ---- the network block ---------------------------------------------------------
// Weights in fragment order: chunk g holds, for every 8-column tile t of a layer and
// lane l, one 16-byte word with the lane's mma.sync B fragments of two consecutive
// 16-deep K steps (k0 = 32 c + 2 (l & 3), rows k0 + {0, 1}, + 8, + 16, + 24 of column
// 8 t + (l >> 2)), so that a warp's fragments are one conflict-free 16-byte shared
// load each.  Chunks 0-2: layer 1 (K 96), 3-10: layer 2, 11-18: layer 3 (32 K rows
// x 256 columns, 16 KB each), 19: layer 4 (K 256 x 16 columns, 8 KB).
constexpr int ROWS = 16, NCW = 16, TPW = 32 / NCW, NET_THREADS = 32 * (NCW + 1), CHUNK_U4 = 1024, NCHUNK = 20, NSTAGE = 8,
              LDA = H + 8;
constexpr int FAULT_FIRST = 6;  // the first weight chunk that the tests' fault may leave out
constexpr int PACK_U4 = 19 * CHUNK_U4 + 512;
static_assert(ROWS == NCW, "one row per compute warp");

constexpr int CPW = 4;  // weight chunks per wait of a compute warp (at most half the ring)

constexpr int MAXSUB = 32;  // substeps per MPCD step the colloid-only step supports

struct __align__(128) NetSmem {
  uint4 ring[NSTAGE][CHUNK_U4];
  union {
    float4 xall[MAXC];  // every colloid's position (candidate-list rebuilds)
    struct {
      float4 cx[ROWS][CAND], cv[ROWS][CAND];  // the candidates' positions and velocities
    } c;
  } u;
  float4 row[4][ROWS];       // the rows' X, V, Omega, ra at the step's start
  float dp[ROWS][NO / 2];    // the drawn exchange (momentum, angular momentum)
  bf16 act[2][ROWS][LDA];
  float cd[ROWS][CAND];      // candidates within the scan distance: squared distance,
  int ck[ROWS][CAND];        // colloid,
  int ce[ROWS][CAND];        // slot in the candidate list
  alignas(16) uint16_t lst[ROWS][CAND];  // candidate lists
  int lstn[ROWS];
  int cn[ROWS];              // candidates within the scan distance per row
  float feat[ROWS][NF];
  float out[ROWS][OUTP];
  alignas(16) float bias[3 * H + OUTP];
  float xi[ROWS][NO / 2];  // the exchange's Gaussians
  float xm[NF], xs[NF], ym[NO / 2], ys[NO / 2];
  unsigned long long full[NSTAGE], empty[NSTAGE];  // a chunk landed / every compute warp is done with it
  int abort;
};

__device__ __forceinline__ uint32_t bf16_bits(const bf16 *w, long long i) {
  return (uint32_t)__bfloat16_as_ushort(w[i]);
}

// the fragment-order copy of the BF16 weights ([k][n] matrices of 256 / 16 columns)
__global__ void k_sur_pack(const bf16 *w0, const bf16 *w1, const bf16 *w2, const bf16 *w3, uint4 *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= PACK_U4) return;
  const bf16 *W;
  int npad, k0, n;
  if (i < 19 * CHUNK_U4) {
    const int g = i / CHUNK_U4, within = i % CHUNK_U4, t = within >> 5, lane = within & 31;
    const int c = g < 3 ? g : (g < 11 ? g - 3 : g - 11);
    W = g < 3 ? w0 : (g < 11 ? w1 : w2);
    npad = H;
    k0 = 32 * c + 2 * (lane & 3);
    n = 8 * t + (lane >> 2);
  } else {
    const int within = i - 19 * CHUNK_U4, kp = within >> 6, t = (within >> 5) & 1, lane = within & 31;
    W = w3;
    npad = OUTP;
    k0 = 32 * kp + 2 * (lane & 3);
    n = 8 * t + (lane >> 2);
  }
  uint32_t word[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const long long kb = k0 + 8 * h;
    word[h] = bf16_bits(W, kb * npad + n) | (bf16_bits(W, (kb + 1) * npad + n) << 16);
  }
  out[i] = make_uint4(word[0], word[1], word[2], word[3]);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait for phase `parity` of a stage's barrier: gives up after 100 ms (a
// chunk arrives in microseconds) or 2^24 tries
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, uint32_t parity) {
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (int it = 0; it < (1 << 24); ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > 100000000ull) break;
  }
  return false;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// weight chunk g into its stage, one bulk copy counted on the stage's full barrier
__device__ __forceinline__ void issue_chunk(const Sur &S, NetSmem &sm, int g) {
  const uint32_t bytes = g < 19 ? CHUNK_U4 * 16 : 512 * 16;
  unsigned long long *bar = &sm.full[g % NSTAGE];
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(sm.ring[g % NSTAGE])),
               "l"(S.wpk + (size_t)g * CHUNK_U4), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// a compute warp's wait for chunk g (lane 0, bounded).  After a wait that gave up
// (or once any wait has) the warp goes on without the chunk and without releasing
// its stage, so the producer stops too; the results are then flagged, not used.
__device__ __forceinline__ bool chunk_ready(const Sur &S, NetSmem &sm, int g) {
  int ok = 0;
  if ((threadIdx.x & 31) == 0) {
    unsigned long long *bar = &sm.full[g % NSTAGE];
    const uint32_t parity = (uint32_t)((g / NSTAGE) & 1);
    ok = mbar_try_wait(bar, parity);
    if (!ok) {
      volatile int *ab = &sm.abort;
      ok = !*ab && mbar_wait_bounded(bar, parity);
      if (!ok && !*ab) {
        atomicOr(S.err, 4);
        *ab = 1;
      }
    }
  }
  return __shfl_sync(0xFFFFFFFFu, ok, 0) != 0;
}

__device__ __forceinline__ void chunk_release(NetSmem &sm, int g, bool ok) {
  __syncwarp();
  if (ok && (threadIdx.x & 31) == 0) mbar_arrive(&sm.empty[g % NSTAGE]);
}

__device__ __forceinline__ void compute_barrier() {  // the compute warps only
  asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the A fragment of K step kk (16 rows of the activations), one ldmatrix.x4: lane l
// gives the address of row l % 16 at column kk + 8 (l / 16)
__device__ __forceinline__ void a_frag(const bf16 (*A)[LDA], int kk, uint32_t a[4]) {
  const int lane = threadIdx.x & 31;
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(&A[lane & 15][kk + 8 * (lane >> 4)]);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(addr)
               : "memory");
}

// A step's kernels are launched before the one before them has ended (each then finds its blocks
// placed and its constants loaded): wait_before holds until that one has ended and its writes are
// visible, let_dependents lets the next one start
__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float sigm(float z) { return __fdividef(1.f, 1.f + __expf(-z)); }  // as mlp.cu

// One block per 16 colloids: sixteen compute warps (a colloid each in the
// neighbour and feature phases, 16 columns each in the network) and one producer
// warp that streams the weights.
//   neighbours within max(three radii, the force cutoff plus the skin): from each
//   colloid's candidate list (colloids within that distance plus a skin of 2 at the
//   last rebuild, ascending index), or, when k_sur_md has flagged that a colloid
//   moved more than half the skin since then, from all pairs (and the lists rebuilt);
//   the features (V, Omega, ra, then the 12 nearest within three radii, nearest first,
//   ties by index, zero padded: the layout of brownian_gb300.closure.features), raw
//   to S.feat and normalised (clipped to six standard deviations) as the BF16 input
//   rows; the force partners (within the cutoff plus the skin, ascending index);
//   the exchange's Gaussians;
//   the four layers (the mlp.cu forward pass: K steps in ascending order into one
//   FP32 accumulator, bias, SiLU, BF16 between layers), the weights streamed by bulk
//   copies NSTAGE chunks ahead (full / empty barriers per stage); from the outputs
//   the Gaussian draw of the exchange (per-substep shares for the substeps' kernel).
__global__ void __launch_bounds__(NET_THREADS) k_sur_net(const Sur S) {
  extern __shared__ __align__(128) unsigned char net_smem[];
  NetSmem &sm = *reinterpret_cast<NetSmem *>(net_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, q = lane & 3;
  const unsigned lt = (1u << lane) - 1u;
  const int j0 = blockIdx.x * ROWS;
  const bool producer = warp == NCW;
  if (tid == NCW * 32) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], NCW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    sm.abort = 0;
    // the first weight chunks stream in while the neighbours are found
    for (int g = 0; g < NSTAGE; ++g)
      if (g != S.drop_chunk) issue_chunk(S, sm, g);
  }
  // what no step changes
  static_assert((3 * H + OUTP) / 4 <= NET_THREADS && NF <= NET_THREADS, "one load per thread");
  if (tid < (3 * H + OUTP) / 4) reinterpret_cast<uint4 *>(sm.bias)[tid] = reinterpret_cast<const uint4 *>(S.bias)[tid];
  if (tid < NF) {
    sm.xm[tid] = S.xmean[tid];
    sm.xs[tid] = S.xistd[tid];
  }
  if (tid < NO / 2) {
    sm.ym[tid] = S.ymean[tid];
    sm.ys[tid] = S.yistd[tid];
  }
  // the substeps of the step before have ended, and what they wrote is here
  wait_before();
  let_dependents();
  // the rows' state and the candidate lists (or every position, for a rebuild): independent loads,
  // all in flight together
  const int err = *S.err;
  const uint32_t step = (uint32_t)*S.step;
  const float rfp = S.rc + partner_skin(S), rforce2 = rfp * rfp;
  const bool rebuild = *S.rebuild != 0;
  if (tid < 4 * ROWS) {
    const int r = tid % ROWS, f = tid / ROWS, j = j0 + r;
    const float4 *src = f == 0 ? S.X : (f == 1 ? S.V : (f == 2 ? S.W : S.ra));
    if (j < S.Nc) sm.row[f][r] = src[j];
  }
  // the lists (read on every step, so that no load waits for the flag; a rebuild replaces them)
  static_assert(ROWS * CAND / 8 <= NET_THREADS, "one 16-byte piece of the lists per thread");
  if (tid < ROWS * CAND / 8) {
    const int r = tid / (CAND / 8), qv = tid % (CAND / 8), j = j0 + r;
    if (j < S.Nc)
      reinterpret_cast<uint4 *>(sm.lst[r])[qv] = reinterpret_cast<const uint4 *>(S.nbl + (size_t)j * CAND)[qv];
  }
  if (tid < ROWS) sm.lstn[tid] = j0 + tid < S.Nc ? S.nbn[j0 + tid] : 0;
  if (err & 4) {
    // a weight copy of an earlier step of this call did not arrive: no more steps (the copies in
    // flight land first)
    if (tid == NCW * 32)
      for (int g = 0; g < NSTAGE; ++g)
        if (g != S.drop_chunk) mbar_wait_bounded(&sm.full[g], 0);
    return;
  }
  if (rebuild) {
    for (int i0 = tid; i0 < S.Nc; i0 += 8 * NET_THREADS) {  // eight loads in flight per thread
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u * NET_THREADS < S.Nc) v[u] = S.X[i0 + u * NET_THREADS];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u * NET_THREADS < S.Nc) sm.u.xall[i0 + u * NET_THREADS] = v[u];
    }
  }
  __syncthreads();
  if (rebuild) {
    // all pairs: colloids within the list distance, ascending index (compute warp w: row w)
    const int r = warp, j = j0 + r;
    if (!producer && j < S.Nc) {
      const float4 xj = sm.row[0][r];
      int nl = 0;
      for (int k0 = 0; k0 < S.Nc; k0 += 32) {
        const int k = k0 + lane;
        float d2 = 1e30f;
        if (k < S.Nc && k != j) {
          const float4 xk = sm.u.xall[k];
          const float dx = wrapd(xk.x - xj.x, S.L[0], S.iL[0]), dy = wrapd(xk.y - xj.y, S.L[1], S.iL[1]),
                      dz = wrapd(xk.z - xj.z, S.L[2], S.iL[2]);
          d2 = dx * dx + dy * dy + dz * dz;
        }
        const bool inl = d2 < S.rlist2;
        const unsigned ml = __ballot_sync(0xFFFFFFFFu, inl);
        if (inl) {
          const int slot = nl + __popc(ml & lt);
          if (slot < CAND) {
            S.nbl[(size_t)j * CAND + slot] = (uint16_t)k;
            sm.lst[r][slot] = (uint16_t)k;
          }
        }
        nl += __popc(ml);
      }
      if (lane == 0) {
        sm.lstn[r] = min(nl, CAND);
        S.nbn[j] = min(nl, CAND);
        S.xref[j] = xj;
        if (nl > CAND) atomicOr(S.err, 1);
      }
    } else if (!producer && lane == 0) {
      sm.lstn[r] = 0;
    }
    __syncthreads();  // (the candidates' positions below overwrite xall)
  }
  // the candidates' positions and velocities, all loads in flight together
  {
    constexpr int PT = (ROWS * CAND + NET_THREADS - 1) / NET_THREADS;
    float4 px[PT], pv[PT];
#pragma unroll
    for (int u = 0; u < PT; ++u) {
      const int i = tid + NET_THREADS * u, r = i / CAND, e = i % CAND;
      if (i < ROWS * CAND && e < sm.lstn[r]) {
        const int k = sm.lst[r][e];
        px[u] = S.X[k];
        pv[u] = S.V[k];
      }
    }
#pragma unroll
    for (int u = 0; u < PT; ++u) {
      const int i = tid + NET_THREADS * u, r = i / CAND, e = i % CAND;
      if (i < ROWS * CAND && e < sm.lstn[r]) {
        sm.u.c.cx[r][e] = px[u];
        sm.u.c.cv[r][e] = pv[u];
      }
    }
  }
  __syncthreads();
  if (!producer) {  // compute warp w: row w
    const int r = warp, j = j0 + r;
    float *o = sm.feat[r];
    for (int col = lane; col < NF; col += 32) o[col] = 0.f;
    __syncwarp();
    if (j < S.Nc) {
    const float4 xj = sm.row[0][r], vj = sm.row[1][r];
    // neighbours within the scan distance, ascending index
    const int nlst = sm.lstn[r];
    int n = 0;
    for (int e0 = 0; e0 < nlst; e0 += 32) {
      const int e = e0 + lane;
      float d2 = 1e30f;
      if (e < nlst) {
        const float4 xk = sm.u.c.cx[r][e];
        const float dx = wrapd(xk.x - xj.x, S.L[0], S.iL[0]), dy = wrapd(xk.y - xj.y, S.L[1], S.iL[1]),
                    dz = wrapd(xk.z - xj.z, S.L[2], S.iL[2]);
        d2 = dx * dx + dy * dy + dz * dz;
      }
      const bool in = d2 < S.rscan2;
      const unsigned m = __ballot_sync(0xFFFFFFFFu, in);
      if (in) {
        const int slot = n + __popc(m & lt);  // slot <= e < CAND
        sm.cd[r][slot] = d2;
        sm.ck[r][slot] = sm.lst[r][e];
        sm.ce[r][slot] = e;
      }
      n += __popc(m);
    }
    __syncwarp();
    if (lane == 0) {
      o[0] = vj.x; o[1] = vj.y; o[2] = vj.z;
      const float4 wj = sm.row[2][r], aj = sm.row[3][r];
      o[3] = wj.x; o[4] = wj.y; o[5] = wj.z; o[6] = aj.x; o[7] = aj.y; o[8] = aj.z;
    }
    // the 12 nearest within three radii: each candidate's rank by (distance, index)
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = e0 + lane;
      const bool have = e < n;
      const float d2 = have ? sm.cd[r][e] : 3.0e38f;
      const int k = have ? sm.ck[r][e] : 0x7FFFFFFF;
      int rank = 0;
      if (n <= 32) {
        for (int f = 0; f < n; ++f) {
          const float df = __shfl_sync(0xFFFFFFFFu, d2, f);
          const int kf = __shfl_sync(0xFFFFFFFFu, k, f);
          rank += (df < S.ct_feat2) && (df < d2 || (df == d2 && kf < k));
        }
      } else {
        for (int f = 0; f < n; ++f) {
          const float df = sm.cd[r][f];
          rank += (df < S.ct_feat2) && (df < d2 || (df == d2 && sm.ck[r][f] < k));
        }
      }
      if (have && d2 < S.ct_feat2 && rank < KNEAR) {
        const int ce = sm.ce[r][e];
        const float4 xk = sm.u.c.cx[r][ce], vk = sm.u.c.cv[r][ce];
        float *qf = o + 9 + 6 * rank;
        qf[0] = wrapd(xk.x - xj.x, S.L[0], S.iL[0]);
        qf[1] = wrapd(xk.y - xj.y, S.L[1], S.iL[1]);
        qf[2] = wrapd(xk.z - xj.z, S.L[2], S.iL[2]);
        qf[3] = vk.x - vj.x; qf[4] = vk.y - vj.y; qf[5] = vk.z - vj.z;
      }
    }
    // the force partners, ascending index
    int m = 0;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = e0 + lane;
      const bool in = e < n && sm.cd[r][e] < rforce2;
      const unsigned b = __ballot_sync(0xFFFFFFFFu, in);
      if (in) {
        const int slot = m + __popc(b & lt);
        if (slot < MAXF) S.fpart[(size_t)j * MAXF + slot] = (uint16_t)sm.ck[r][e];
      }
      m += __popc(b);
    }
    if (lane == 0) {
      S.fpn[j] = (uint8_t)min(m, MAXF);
      if (m > MAXF) atomicOr(S.err, 2);
    }
    }
  }
  // the exchange's six Gaussians, on the producer's lanes meanwhile
  if (producer && lane < ROWS && j0 + lane < S.Nc) {
    const int r = lane, j = j0 + r;
    const uint4 r0 = draw4(S.key, DOM_SUR_KICK, 0, (uint32_t)(j + 1), 0, step);
    const uint4 r1 = draw4(S.key, DOM_SUR_KICK, 1, (uint32_t)(j + 1), 0, step);
    const float2 g0 = normal2(r0.x, r0.y), g1 = normal2(r0.z, r0.w), g2 = normal2(r1.x, r1.y);
    sm.xi[r][0] = g0.x; sm.xi[r][1] = g0.y; sm.xi[r][2] = g1.x;
    sm.xi[r][3] = g1.y; sm.xi[r][4] = g2.x; sm.xi[r][5] = g2.y;
  }
  static_assert(ROWS <= 32, "a lane per row");
  __syncthreads();
  // raw inputs to S.feat, normalised BF16 rows to act[0]
  for (int i = tid; i < ROWS * INP; i += NET_THREADS) {
    const int r = i / INP, c = i % INP, j = j0 + r;
    float z = 0.f;
    if (c < NF) {
      const float x = sm.feat[r][c];
      if (j < S.Nc) S.feat[(size_t)j * NF + c] = x;
      z = (x - sm.xm[c]) * sm.xs[c];
    }
    sm.act[0][r][c] = __float2bfloat16(fminf(fmaxf(z, -MLP_INPUT_CLIP), MLP_INPUT_CLIP));
  }
  __syncthreads();
  if (producer) {
    if (lane == 0) {
      // chunk g into its stage once every compute warp is done with chunk g - NSTAGE
      volatile int *ab = &sm.abort;
      int issued = NSTAGE;
      for (int g = NSTAGE; g < NCHUNK && !*ab; ++g) {
        if (!mbar_wait_bounded(&sm.empty[g % NSTAGE], (uint32_t)((g / NSTAGE - 1) & 1))) {
          atomicOr(S.err, 4);
          *ab = 1;
          break;
        }
        if (g == S.drop_chunk) continue;  // injected fault: the consumers' bounded waits give up
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_chunk(S, sm, g);
        issued = g + 1;
      }
      // every copy issued (the last one into each stage) lands before the block exits
      for (int c = issued > NSTAGE ? issued - NSTAGE : 0; c < issued; ++c)
        if (c != S.drop_chunk) mbar_wait_bounded(&sm.full[c % NSTAGE], (uint32_t)((c / NSTAGE) & 1));
    }
  } else {
    // three hidden layers: compute warp w takes columns 8 TPW w .. 8 TPW (w + 1) - 1, four
    // weight chunks per wait (their fragments and the rows' loaded together, then a chain of
    // eight products per tile)
    int g = 0;
#pragma unroll 1
    for (int layer = 0; layer < 3; ++layer) {
      const bf16(*A)[LDA] = sm.act[layer & 1];
      bf16(*Z)[LDA] = sm.act[(layer + 1) & 1];
      const int nch = layer == 0 ? INP / 32 : H / 32;
      float acc[TPW][4];
#pragma unroll
      for (int t = 0; t < TPW; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[t][e] = 0.f;
#pragma unroll 1
      for (int c = 0; c < nch; c += CPW) {
        bool ok[CPW];
        uint4 b[CPW][TPW];
        uint32_t a[CPW][2][4];
#pragma unroll
        for (int u = 0; u < CPW; ++u) {
          if (c + u >= nch) continue;
          a_frag(A, 32 * (c + u), a[u][0]);
          a_frag(A, 32 * (c + u) + 16, a[u][1]);
          ok[u] = chunk_ready(S, sm, g + u);
          const uint4 *B = sm.ring[(g + u) % NSTAGE];
#pragma unroll
          for (int t = 0; t < TPW; ++t) b[u][t] = B[(TPW * warp + t) * 32 + lane];
        }
#pragma unroll
        for (int u = 0; u < CPW; ++u) {
          if (c + u >= nch) continue;
#pragma unroll
          for (int t = 0; t < TPW; ++t) mma_bf16(acc[t], a[u][0], b[u][t].x, b[u][t].y);
#pragma unroll
          for (int t = 0; t < TPW; ++t) mma_bf16(acc[t], a[u][1], b[u][t].z, b[u][t].w);
        }
#pragma unroll
        for (int u = 0; u < CPW; ++u)
          if (c + u < nch) chunk_release(sm, g + u, ok[u]);
        g += min(CPW, nch - c);
      }
      const float *bias = sm.bias + H * layer;
#pragma unroll
      for (int t = 0; t < TPW; ++t) {
        const int n0 = 8 * (TPW * warp + t) + 2 * q;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float v0 = acc[t][2 * h] + bias[n0], v1 = acc[t][2 * h + 1] + bias[n0 + 1];
          v0 = v0 * sigm(v0);
          v1 = v1 * sigm(v1);
          __nv_bfloat162 pr;
          pr.x = __float2bfloat16(v0);
          pr.y = __float2bfloat16(v1);
          *reinterpret_cast<__nv_bfloat162 *>(&Z[gq + 8 * h][n0]) = pr;
        }
      }
      compute_barrier();
    }
    // the output layer (16 columns, 12 used): compute warps 0 and 1, one 8-column tile each
    if (warp < 2) {
      const bool ok = chunk_ready(S, sm, g);
      (void)ok;
      const uint4 *B = sm.ring[g % NSTAGE];
      const bf16(*A)[LDA] = sm.act[1];
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int kp = 0; kp < H / 32; ++kp) {
        const uint4 b = B[(2 * kp + warp) * 32 + lane];
        uint32_t a[4];
        a_frag(A, 32 * kp, a);
        mma_bf16(acc, a, b.x, b.y);
        a_frag(A, 32 * kp + 16, a);
        mma_bf16(acc, a, b.z, b.w);
      }
      const float *bias = sm.bias + 3 * H;
      const int n0 = 8 * warp + 2 * q;
      sm.out[gq][n0] = acc[0] + bias[n0];
      sm.out[gq][n0 + 1] = acc[1] + bias[n0 + 1];
      sm.out[gq + 8][n0] = acc[2] + bias[n0];
      sm.out[gq + 8][n0 + 1] = acc[3] + bias[n0 + 1];
    }
  }
  __syncthreads();
  for (int i = tid; i < ROWS * OUTP; i += NET_THREADS) {
    const int r = i / OUTP, j = j0 + r;
    if (j < S.Nc) S.out[(size_t)j * OUTP + i % OUTP] = sm.out[r][i % OUTP];
  }
  // the exchange, one (row, component) per thread: the network's normalised outputs ->
  // mean and standard deviation in physical units, and the Gaussian draw
  if (tid < ROWS * (NO / 2)) {
    const int r = tid / (NO / 2), k = tid % (NO / 2);
    const float *o = sm.out[r];
    const float lv = fminf(fmaxf(o[6 + k], -MLP_LOGVAR_CLAMP), MLP_LOGVAR_CLAMP);
    sm.dp[r][k] = (o[k] + S.noise * __expf(0.5f * lv) * sm.xi[r][k]) / sm.ys[k] + sm.ym[k];
  }
  __syncthreads();
  // for the substeps: the exchange in equal shares (the fluid collides every substep), and the
  // orientation run()'s kick uses
  const float fm = 1.f / (S.M * S.n_sub), fi = 1.f / (S.I * S.n_sub);
  if (tid < ROWS && j0 + tid < S.Nc) {
    const int r = tid, j = j0 + r;
    S.imp[j] = make_float4(sm.dp[r][0] * fm, sm.dp[r][1] * fm, sm.dp[r][2] * fm, 0.f);
    S.imp[S.Nc + j] = sm.row[3][r];
    S.imp[2 * S.Nc + j] =
        make_float4(sm.dp[r][3] * fi, sm.dp[r][4] * fi, sm.dp[r][5] * fi, __uint_as_float(step));
  }
}

// Omega and orientation of colloid j through the step's substeps: Omega takes its share of the
// angular exchange each substep, and the orientation the Euler rotation by Omega dt, then the
// rotational diffusion (update_activity_direction plus Dr).  Neither depends on positions or forces,
// so it runs on blocks of its own beside the substeps.  (Every rounding is written out: the bits do
// not depend on what the compiler fuses.)
__device__ __noinline__ void orient(const Sur &S, int j) {
  const float4 pa = S.imp[2 * S.Nc + j];
  const uint32_t step = __float_as_uint(pa.w);
  float4 w = S.W[j], a = S.ra[j];
#pragma unroll 2
  for (int l = 0; l < S.n_sub; ++l) {
    w.x += pa.x; w.y += pa.y; w.z += pa.z;
    float sx, cx, sy, cy, sz, cz;
    __sincosf(w.x * S.dt, &sx, &cx); __sincosf(w.y * S.dt, &sy, &cy); __sincosf(w.z * S.dt, &sz, &cz);
    const float ss = __fmul_rn(sx, sy), cs = __fmul_rn(cx, sy);
    const float4 m0 = make_float4(__fmul_rn(cy, cz), -__fmul_rn(cy, sz), sy, 0.f);
    const float4 m1 = make_float4(__fmaf_rn(cx, sz, __fmul_rn(ss, cz)), __fmaf_rn(-ss, sz, __fmul_rn(cx, cz)),
                                  -__fmul_rn(sx, cy), 0.f);
    const float4 m2 = make_float4(__fmaf_rn(sx, sz, -__fmul_rn(cs, cz)), __fmaf_rn(cs, sz, __fmul_rn(sx, cz)),
                                  __fmul_rn(cx, cy), 0.f);
    auto row = [&](const float4 &m) { return __fmaf_rn(m.z, a.z, __fmaf_rn(m.y, a.y, __fmul_rn(m.x, a.x))); };
    auto dot = [](float x, float y, float z, float p, float q, float r) {
      return __fmaf_rn(z, r, __fmaf_rn(x, p, __fmul_rn(y, q)));
    };
    float ax = row(m0), ay = row(m1), az = row(m2);
    if (S.rotdiff_s > 0.f) {
      const uint4 d4 = draw4(S.key, DOM_SUR_ROT, 0, (uint32_t)(j + 1), 0, step * S.n_sub + l);
      const float2 g0 = normal2(d4.x, d4.y), g1 = normal2(d4.z, d4.w);
      const float d = dot(g0.x, g0.y, g1.x, ax, ay, az);
      ax = __fmaf_rn(S.rotdiff_s, __fmaf_rn(-d, ax, g0.x), ax);
      ay = __fmaf_rn(S.rotdiff_s, __fmaf_rn(-d, ay, g0.y), ay);
      az = __fmaf_rn(S.rotdiff_s, __fmaf_rn(-d, az, g1.x), az);
    }
    const float in = rsqrtf(dot(ax, ay, az, ax, ay, az));
    a = make_float4(ax * in, ay * in, az * in, 0.f);
  }
  S.W[j] = w;
  S.ra[j] = a;
}

// ---- the substeps ---------------------------------------------------------------
// squared displacement from xs to x (minimum image)
__device__ __forceinline__ float step_moved2(const Sur &S, float4 x, float4 xs) {
  const float dx = wrapd(x.x - xs.x, S.L[0], S.iL[0]), dy = wrapd(x.y - xs.y, S.L[1], S.iL[1]),
              dz = wrapd(x.z - xs.z, S.L[2], S.iL[2]);
  return dx * dx + dy * dy + dz * dz;
}

// the WCA forces on a colloid at x from its n partners (ids in row, ascending; positions
// in P): the force-shifted WCA pair force (cpp/update.cpp:14-32) in FP32 for the pairs
// within the cutoff (1/r by the fast reciprocal square root, 1/r^6 from 1/r^2), summed in
// partner order.  Four partners at a time without a branch (a pair beyond the cutoff gets the
// factor 0, which leaves the sums as they are): the four chains of some 40 dependent operations
// run beside one another, where a branch per pair in contact made them wait in turn.
__device__ __forceinline__ float3 partner_forces(const Sur &S, float4 x, const float4 *P, const uint16_t *row, int n,
                                                 int self) {
  float3 fn = make_float3(0.f, 0.f, 0.f);
#pragma unroll 1
  for (int e = 0; e < n; e += 4) {
    const uint2 kk = *reinterpret_cast<const uint2 *>(row + e);
    const int k4[4] = {(int)(kk.x & 0xFFFFu), (int)(kk.x >> 16), (int)(kk.y & 0xFFFFu), (int)(kk.y >> 16)};
    float f[4], dx[4], dy[4], dz[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 xk = P[e + i < n ? k4[i] : self];
      dx[i] = wrapd(x.x - xk.x, S.L[0], S.iL[0]);
      dy[i] = wrapd(x.y - xk.y, S.L[1], S.iL[1]);
      dz[i] = wrapd(x.z - xk.z, S.L[2], S.iL[2]);
      const float r2 = dx[i] * dx[i] + dy[i] * dy[i] + dz[i] * dz[i];
      const float ir = rsqrtf(r2), ir2 = ir * ir, ir6 = ir2 * ir2 * ir2;
      const float g = (4.f * S.eps * (12.f * S.sig12 * ir6 * ir6 * ir - 6.f * S.sig6 * ir6 * ir) - S.fc) * ir;
      f[i] = e + i < n && r2 < S.rc2 ? g : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      fn.x += f[i] * dx[i]; fn.y += f[i] * dy[i]; fn.z += f[i] * dz[i];
    }
  }
  return fn;
}

// One block, a colloid per thread (position, velocity, force and the step's impulse
// in registers; positions, two copies by substep parity, and force partners in shared
// memory): run()'s kick along the orientation at the step's start, then n_sub substeps
// of update_pos_md, the substep's share of the exchange, compute_force_md at the new
// positions and update_velocity_colloid, one block barrier per substep (the copy a
// substep writes was last read two substeps before).  At the end: whether a colloid has
// moved more than half the skin since the candidate lists were built.
// Blocks 1, 2, ...: the orientations.
__global__ void __launch_bounds__(kMdBlockMax) k_sur_md1(const Sur S) {
  extern __shared__ float4 smem[];
  __shared__ unsigned s_vmax;  // the largest speed at the end (float bits, non-negative)
  uint16_t *sF = reinterpret_cast<uint16_t *>(smem + 2 * kMdBlockMax);  // [kMdBlockMax][MAXF] force partners
  const int T = blockDim.x, tid = threadIdx.x;
  wait_before();
  let_dependents();
  if (blockIdx.x > 0) {
    const int j = (blockIdx.x - 1) * T + tid;
    if (!(*S.err & 4) && j < S.Nc) orient(S, j);
    return;
  }
  if (tid == 0) s_vmax = 0u;
  const int j = tid;
  const bool own = j < S.Nc;
  const int err = *S.err;
  const float hs = 0.5f * partner_skin(S), hs2 = hs * hs;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), v = x, fo = x, pl = x;
  int n = 0;
  if (own) {
    const uint4 *src = reinterpret_cast<const uint4 *>(S.fpart + (size_t)j * MAXF);
    uint4 *dst = reinterpret_cast<uint4 *>(sF + j * MAXF);
    uint4 pp[MAXF * 2 / 16];
#pragma unroll
    for (int i = 0; i < MAXF * 2 / 16; ++i) pp[i] = src[i];
    n = S.fpn[j];
    x = S.X[j]; v = S.V[j]; fo = S.f[j]; pl = S.imp[j];
    const float4 a = S.imp[S.Nc + j];
#pragma unroll
    for (int i = 0; i < MAXF * 2 / 16; ++i) dst[i] = pp[i];
    v.x += S.v0 * a.x; v.y += S.v0 * a.y; v.z += S.v0 * a.z;
  }
  if (err & 4) return;  // the network's outputs of this step are incomplete: the state stays as it was
  const float hdt2m = 0.5f * S.dt * S.dt / S.M, hdtm = 0.5f * S.dt / S.M;
  for (int l = 0; l < S.n_sub; ++l) {
    float4 *P = (l & 1) ? smem : smem + kMdBlockMax;  // this substep's copy
    if (own) {  // update_pos_md
      x.x += v.x * S.dt + fo.x * hdt2m; x.y += v.y * S.dt + fo.y * hdt2m; x.z += v.z * S.dt + fo.z * hdt2m;
      x.x = boxed(x.x, S.L[0], S.iL[0]); x.y = boxed(x.y, S.L[1], S.iL[1]); x.z = boxed(x.z, S.L[2], S.iL[2]);
      P[j] = x;
    }
    __syncthreads();
    if (own) {
      // this substep's share of the fluid exchange (fluid_colloid_collision)
      v.x += pl.x; v.y += pl.y; v.z += pl.z;
      // compute_force_md at the new positions, update_velocity_colloid
      const float3 fn = partner_forces(S, x, P, sF + j * MAXF, n, j);
      v.x += (fo.x + fn.x) * hdtm; v.y += (fo.y + fn.y) * hdtm; v.z += (fo.z + fn.z) * hdtm;
      fo = make_float4(fn.x, fn.y, fn.z, 0.f);
    }
  }
  int moved = 0, fast = 0;
  if (own) {
    const float4 x0 = S.xref[j], xs = S.X[j];
    S.X[j] = x; S.V[j] = v; S.f[j] = fo;
    moved = step_moved2(S, x, x0) > S.half_skin2;
    fast = step_moved2(S, x, xs) > hs2;
    atomicMax(&s_vmax, __float_as_uint(sqrtf(v.x * v.x + v.y * v.y + v.z * v.z)));
  }
  moved = __syncthreads_or(moved);
  fast = __syncthreads_or(fast);
  if (tid == 0) {
    *S.rebuild = moved;
    if (fast) *S.fast += 1;
    *S.vmax = __uint_as_float(s_vmax);
    *S.step += 1;
  }
}

// One cluster of MDC blocks, one colloid per thread (block b takes colloids
// [b per, (b + 1) per)): position, velocity, force and the step's impulse in
// registers, force partners in shared memory.  run()'s kick along the orientation at
// the step's start, then n_sub substeps of update_pos_md, the substep's share of the
// exchange, compute_force_md at the new positions and update_velocity_colloid.  Each
// substep's new positions go to every block's copy (distributed shared memory, two
// copies by substep parity), then one cluster barrier: the copy a substep writes was
// last read two substeps before, behind the barrier in between.  At the end: whether
// a colloid has moved more than half the skin since the candidate lists were built.
constexpr int MDC = 8, MD_MAXT = MAXC / MDC;

// The second cluster: the orientations.
__global__ void __cluster_dims__(MDC, 1, 1) __launch_bounds__(MD_MAXT) k_sur_md(const Sur S) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ float4 smem[];
  uint16_t *sF = reinterpret_cast<uint16_t *>(smem + 2 * MAXC);          // [MD_MAXT][MAXF] force partners
  uint8_t *sFn = reinterpret_cast<uint8_t *>(sF + MD_MAXT * MAXF);       // [MD_MAXT] their count
  int *sMoved = reinterpret_cast<int *>(sFn + MD_MAXT);                  // [MDC] (block 0)
  unsigned *sVmax = reinterpret_cast<unsigned *>(sMoved + MDC);         // [MDC] (block 0)
  __shared__ unsigned s_vmax;
  const int tid = threadIdx.x, rank = (int)cl.block_rank();
  const int per = (S.Nc + MDC - 1) / MDC, j = rank * per + tid;
  const bool own = tid < per && j < S.Nc;
  if (tid == 0) s_vmax = 0u;
  cl.sync();  // every block has started before any writes to its copies
  wait_before();
  let_dependents();
  if (blockIdx.x >= MDC) {
    if (own && !(*S.err & 4)) orient(S, j);
    return;
  }
  const int err = *S.err;
  const float hs = 0.5f * partner_skin(S), hs2 = hs * hs;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), v = x, fo = x, pl = x;
  int n = 0;
  if (own) {
    const uint4 *src = reinterpret_cast<const uint4 *>(S.fpart + (size_t)j * MAXF);
    uint4 *dst = reinterpret_cast<uint4 *>(sF + tid * MAXF);
    uint4 pp[MAXF * 2 / 16];
#pragma unroll
    for (int i = 0; i < MAXF * 2 / 16; ++i) pp[i] = src[i];
    n = S.fpn[j];
    x = S.X[j]; v = S.V[j]; fo = S.f[j]; pl = S.imp[j];
    const float4 a = S.imp[S.Nc + j];
#pragma unroll
    for (int i = 0; i < MAXF * 2 / 16; ++i) dst[i] = pp[i];
    v.x += S.v0 * a.x; v.y += S.v0 * a.y; v.z += S.v0 * a.z;
  }
  if (err & 4) return;  // the network's outputs of this step are incomplete: the state stays as it was
  const float hdt2m = 0.5f * S.dt * S.dt / S.M, hdtm = 0.5f * S.dt / S.M;
  for (int l = 0; l < S.n_sub; ++l) {
    const int nb = (l + 1) & 1;
    if (own) {  // update_pos_md
      x.x += v.x * S.dt + fo.x * hdt2m; x.y += v.y * S.dt + fo.y * hdt2m; x.z += v.z * S.dt + fo.z * hdt2m;
      x.x = boxed(x.x, S.L[0], S.iL[0]); x.y = boxed(x.y, S.L[1], S.iL[1]); x.z = boxed(x.z, S.L[2], S.iL[2]);
      float4 *mine = (nb ? smem + MAXC : smem) + j;
#pragma unroll
      for (int b = 0; b < MDC; ++b) *cl.map_shared_rank(mine, b) = x;
    }
    cl.sync();
    if (own) {
      const float4 *P = nb ? smem + MAXC : smem;  // positions, by substep parity
      // this substep's share of the fluid exchange (fluid_colloid_collision)
      v.x += pl.x; v.y += pl.y; v.z += pl.z;
      // compute_force_md at the new positions, update_velocity_colloid
      const float3 fn = partner_forces(S, x, P, sF + tid * MAXF, n, j);
      v.x += (fo.x + fn.x) * hdtm; v.y += (fo.y + fn.y) * hdtm; v.z += (fo.z + fn.z) * hdtm;
      fo = make_float4(fn.x, fn.y, fn.z, 0.f);
    }
  }
  int moved = 0;
  if (own) {
    const float4 x0 = S.xref[j], xs = S.X[j];
    S.X[j] = x; S.V[j] = v; S.f[j] = fo;
    moved = (step_moved2(S, x, x0) > S.half_skin2 ? 1 : 0) | (step_moved2(S, x, xs) > hs2 ? 2 : 0);
    atomicMax(&s_vmax, __float_as_uint(sqrtf(v.x * v.x + v.y * v.y + v.z * v.z)));
  }
  moved = __syncthreads_or(moved & 1) | (__syncthreads_or(moved & 2) ? 2 : 0);
  if (tid == 0) {
    *cl.map_shared_rank(sMoved + rank, 0) = moved;
    *cl.map_shared_rank(sVmax + rank, 0) = s_vmax;
  }
  cl.sync();  // (also: no block leaves while another may still write its copies)
  if (rank == 0 && tid == 0) {
    int any = 0;
    unsigned vm = 0u;
    for (int b = 0; b < MDC; ++b) {
      any |= sMoved[b];
      vm = max(vm, sVmax[b]);
    }
    *S.rebuild = any & 1;
    if (any & 2) *S.fast += 1;
    *S.vmax = __uint_as_float(vm);
    *S.step += 1;
  }
}

// normalised outputs -> physical units (the arithmetic of mpcd_mlp_forward)
__global__ void k_sur_denorm(const Sur S, float *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.Nc * NO) return;
  const int r = i / NO, k = i % NO, ny = NO / 2;
  const float v = S.out[(size_t)r * OUTP + k];
  out[i] = k < ny ? v / S.yistd[k] + S.ymean[k]
                  : fminf(fmaxf(v, -MLP_LOGVAR_CLAMP), MLP_LOGVAR_CLAMP) - 2.f * __logf(S.yistd[k - ny]);
}

__global__ void k_sur_forces(const Sur S) {
  // forces at the current positions (the set-up's compute_force_md), all pairs
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= S.Nc) return;
  float3 fj = make_float3(0.f, 0.f, 0.f);
  const float4 xj = S.X[j];
  for (int k = 0; k < S.Nc; ++k) {
    if (k == j) continue;
    const float4 xk = S.X[k];
    const float dx = wrapd(xj.x - xk.x, S.L[0], S.iL[0]), dy = wrapd(xj.y - xk.y, S.L[1], S.iL[1]),
                dz = wrapd(xj.z - xk.z, S.L[2], S.iL[2]);
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 < S.rc2) {
      const float r = sqrtf(r2), ir = 1.f / r, ir6 = 1.f / (r2 * r2 * r2);
      const float mag = 4.f * S.eps * (12.f * S.sig12 * ir6 * ir6 * ir - 6.f * S.sig6 * ir6 * ir) - S.fc;
      fj.x += mag * dx * ir; fj.y += mag * dy * ir; fj.z += mag * dz * ir;
    }
  }
  S.f[j] = make_float4(fj.x, fj.y, fj.z, 0.f);
}

}  // namespace

struct mpcd_surrogate {
  Sur S;
  mpcd_mlp *net = nullptr;
  cudaStream_t stream = nullptr;
  cudaGraphExec_t exec[2] = {nullptr, nullptr};  // one step; GRAPH_STEPS steps
  uint4 *wpk = nullptr;
  float *outd = nullptr;  // the outputs in physical units (mpcd_surrogate_outputs)
  std::vector<void *> allocs;
  std::string err;
};

namespace {

int sfail(mpcd_surrogate *s, int code, const std::string &e) {
  if (s) s->err = e;
  return code;
}

constexpr int GRAPH_STEPS = 8;  // steps of a graph: within one, a kernel's start hides behind the kernel before it

void drop_graphs(mpcd_surrogate *s) {
  for (cudaGraphExec_t &g : s->exec)
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
}

template <typename T>
T *salloc(mpcd_surrogate *s, size_t n) {
  void *p = nullptr;
  if (cudaMalloc(&p, n * sizeof(T) + 64) != cudaSuccess) {
    s->err = "out of device memory";
    return nullptr;
  }
  cudaMemset(p, 0, n * sizeof(T) + 64);
  s->allocs.push_back(p);
  return static_cast<T *>(p);
}

constexpr size_t kMd1Smem = 2 * kMdBlockMax * sizeof(float4) + kMdBlockMax * MAXF * sizeof(uint16_t);
constexpr size_t kMdSmem = 2 * MAXC * sizeof(float4) + MD_MAXT * MAXF * sizeof(uint16_t) + MD_MAXT + 2 * MDC * sizeof(int);
constexpr size_t kNetSmem = sizeof(NetSmem);

// a launch that may start before the kernel before it on the stream has ended (early)
template <typename K>
cudaError_t launch_early(mpcd_surrogate *s, K *k, int grid, int block, size_t smem, bool early) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s->stream;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, s->S);
}

// n steps
int enqueue_steps(mpcd_surrogate *s, int n) {
  const Sur &S = s->S;
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < n && e == cudaSuccess; ++i) {
    e = launch_early(s, k_sur_net, (S.Nc + ROWS - 1) / ROWS, NET_THREADS, kNetSmem, i > 0);
    if (e != cudaSuccess) break;
    if (S.Nc <= kMdBlockMax) {
      const int block = (S.Nc + 31) / 32 * 32;
      e = launch_early(s, k_sur_md1, 2, block, kMd1Smem, true);
    } else {
      e = launch_early(s, k_sur_md, 2 * MDC, ((S.Nc + MDC - 1) / MDC + 31) / 32 * 32, kMdSmem, true);
    }
  }
  return e == cudaSuccess ? MPCD_OK : sfail(s, MPCD_ERR_CUDA, "step launch");
}

// the network's current weights in the order k_sur_net reads them
int pack_weights(mpcd_surrogate *s) {
  const MlpIO io = mlp_io(s->net);
  s->S.bias = io.bias;
  s->S.xmean = io.xmean; s->S.xistd = io.xistd;
  s->S.ymean = io.ymean; s->S.yistd = io.yistd;
  k_sur_pack<<<(PACK_U4 + 255) / 256, 256, 0, s->stream>>>(
      static_cast<const bf16 *>(io.w[0]), static_cast<const bf16 *>(io.w[1]), static_cast<const bf16 *>(io.w[2]),
      static_cast<const bf16 *>(io.w[3]), s->wpk);
  return cudaGetLastError() == cudaSuccess ? MPCD_OK : sfail(s, MPCD_ERR_CUDA, "weight packing");
}

}  // namespace

extern "C" int mpcd_surrogate_create(const mpcd_params *p, mpcd_mlp *net, mpcd_surrogate **out) {
  if (!p || !net || !out) return MPCD_ERR_PARAM;
  *out = nullptr;
  if (p->n_colloid < 1 || p->n_colloid > MAXC || p->n_sub < 1 || p->n_sub > MAXSUB || !(p->ndt > 0) || !(p->mass_colloid > 0) ||
      !(p->I_colloid > 0) || p->Lx < 1 || p->Ly < 1 || p->Lz < 1)
    return MPCD_ERR_PARAM;
  mpcd_surrogate *s = new mpcd_surrogate();
  s->net = net;
  Sur &S = s->S;
  memset(&S, 0, sizeof S);
  S.Nc = p->n_colloid;
  S.n_sub = p->n_sub;
  const int Ls[3] = {p->Lx, p->Ly, p->Lz};
  for (int k = 0; k < 3; ++k) {
    S.L[k] = (float)Ls[k];
    S.iL[k] = 1.f / (float)Ls[k];
  }
  S.M = (float)p->mass_colloid;
  S.I = (float)p->I_colloid;
  const double dt = p->ndt / p->n_sub;
  S.dt = (float)dt;
  S.v0 = (float)p->v0;
  S.rotdiff_s = (float)std::sqrt(2.0 * p->Dr * dt);
  const double radius = 0.5 * p->sigma;
  S.ct_feat2 = (float)(9.0 * radius * radius);
  const double rc = std::pow(2.0, 1.0 / 6.0) * p->sig_colloid;  // cpp/update.cpp:3
  S.rc2 = (float)(rc * rc);
  S.sig6 = (float)std::pow(p->sig_colloid, 6);
  S.sig12 = (float)std::pow(p->sig_colloid, 12);
  S.eps = (float)p->eps;
  S.fc = (float)(4.0 * p->eps * (12.0 * (std::pow(p->sig_colloid, 12) / std::pow(rc, 13)) -
                                 6.0 * (std::pow(p->sig_colloid, 6) / std::pow(rc, 7))));  // cpp/update.cpp:4
  // force partners within the cutoff plus a skin of 0.5 to 2 (partner_skin; k_sur_md counts
  // the steps in which a colloid moves more than half of it), features within three radii
  S.rc = (float)rc;
  const float rfmax2 = (float)((rc + 2.0) * (rc + 2.0));
  S.rscan2 = rfmax2 > S.ct_feat2 ? rfmax2 : S.ct_feat2;
  // candidate lists: within that distance plus a skin of 2, rebuilt once a colloid has
  // moved half the skin
  const double rl = std::sqrt((double)S.rscan2) + 2.0;
  S.rlist2 = (float)(rl * rl);
  S.half_skin2 = 1.0f;
  S.key = make_uint2((uint32_t)p->seed, (uint32_t)(p->seed >> 32));
  const size_t Nc = S.Nc;
  S.step = salloc<long long>(s, 1);
  S.X = salloc<float4>(s, Nc); S.V = salloc<float4>(s, Nc); S.W = salloc<float4>(s, Nc);
  S.ra = salloc<float4>(s, Nc); S.f = salloc<float4>(s, Nc);
  S.feat = salloc<float>(s, Nc * NF); S.out = salloc<float>(s, Nc * OUTP);
  S.imp = salloc<float4>(s, 3 * Nc);
  S.nbl = salloc<uint16_t>(s, Nc * CAND); S.nbn = salloc<int>(s, Nc);
  S.xref = salloc<float4>(s, Nc); S.rebuild = salloc<int>(s, 1);
  if (S.rebuild) cudaMemset(S.rebuild, 1, sizeof(int));  // no candidate lists yet
  S.fpart = salloc<uint16_t>(s, Nc * MAXF); S.fpn = salloc<uint8_t>(s, Nc);
  S.err = salloc<int>(s, 1);
  S.drop_chunk = -1;
  S.noise = 1.f;
  S.fast = salloc<long long>(s, 1);
  S.vmax = salloc<float>(s, 1);
  s->wpk = salloc<uint4>(s, PACK_U4);
  S.wpk = s->wpk;
  s->outd = salloc<float>(s, Nc * NO);
  if (!s->err.empty() || cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaFuncSetAttribute(k_sur_net, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNetSmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_sur_md, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMdSmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_sur_md1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMd1Smem) != cudaSuccess ||
      pack_weights(s) != MPCD_OK) {
    mpcd_surrogate_destroy(s);
    return MPCD_ERR_NOMEM;
  }
  *out = s;
  return MPCD_OK;
}

extern "C" int mpcd_surrogate_destroy(mpcd_surrogate *s) {
  if (!s) return MPCD_ERR_PARAM;
  if (s->stream) cudaStreamSynchronize(s->stream);
  drop_graphs(s);
  for (void *a : s->allocs) cudaFree(a);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return MPCD_OK;
}

extern "C" const char *mpcd_surrogate_last_error(const mpcd_surrogate *s) { return s ? s->err.c_str() : "null"; }

extern "C" int mpcd_surrogate_set_state(mpcd_surrogate *s, const double *pos, const double *vel, const double *ang_vel,
                                        const double *ra) {
  if (!s || !pos || !vel || !ang_vel || !ra) return MPCD_ERR_PARAM;
  const Sur &S = s->S;
  const double *src[4] = {pos, vel, ang_vel, ra};
  float4 *dst[4] = {S.X, S.V, S.W, S.ra};
  std::vector<float4> h(S.Nc);
  for (int a = 0; a < 4; ++a) {
    for (int j = 0; j < S.Nc; ++j) {
      double v[3] = {src[a][3 * j], src[a][3 * j + 1], src[a][3 * j + 2]};
      if (a == 0)
        for (int k = 0; k < 3; ++k) v[k] -= S.L[k] * std::floor(v[k] / S.L[k]);
      h[j] = make_float4((float)v[0], (float)v[1], (float)v[2], 0.f);
    }
    if (cudaMemcpyAsync(dst[a], h.data(), sizeof(float4) * S.Nc, cudaMemcpyHostToDevice, s->stream) != cudaSuccess ||
        cudaStreamSynchronize(s->stream) != cudaSuccess)
      return sfail(s, MPCD_ERR_CUDA, "state upload");
  }
  float vm = 0.f;  // the largest speed: the first step's partner skin
  for (int j = 0; j < S.Nc; ++j)
    vm = std::max(vm, (float)std::sqrt(vel[3 * j] * vel[3 * j] + vel[3 * j + 1] * vel[3 * j + 1] +
                                       vel[3 * j + 2] * vel[3 * j + 2]));
  if (cudaMemcpyAsync(S.vmax, &vm, sizeof vm, cudaMemcpyHostToDevice, s->stream) != cudaSuccess)
    return sfail(s, MPCD_ERR_CUDA, "set-up");
  k_sur_forces<<<(S.Nc + 127) / 128, 128, 0, s->stream>>>(S);
  k_sur_features<<<(S.Nc + 3) / 4, 128, 0, s->stream>>>(S);
  if (cudaMemsetAsync(S.rebuild, 1, sizeof(int), s->stream) != cudaSuccess) return sfail(s, MPCD_ERR_CUDA, "set-up");
  return cudaStreamSynchronize(s->stream) == cudaSuccess ? MPCD_OK : sfail(s, MPCD_ERR_CUDA, "set-up forces");
}

extern "C" int mpcd_surrogate_get_state(mpcd_surrogate *s, double *pos, double *vel, double *ang_vel, double *ra) {
  if (!s) return MPCD_ERR_PARAM;
  const Sur &S = s->S;
  double *dst[4] = {pos, vel, ang_vel, ra};
  const float4 *src[4] = {S.X, S.V, S.W, S.ra};
  std::vector<float4> h(S.Nc);
  for (int a = 0; a < 4; ++a) {
    if (!dst[a]) continue;
    if (cudaMemcpyAsync(h.data(), src[a], sizeof(float4) * S.Nc, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
        cudaStreamSynchronize(s->stream) != cudaSuccess)
      return sfail(s, MPCD_ERR_CUDA, "state download");
    for (int j = 0; j < S.Nc; ++j) {
      dst[a][3 * j] = h[j].x; dst[a][3 * j + 1] = h[j].y; dst[a][3 * j + 2] = h[j].z;
    }
  }
  return MPCD_OK;
}

// a trajectory frame of the colloid-only step's state
extern "C" int mpcd_traj_record_surrogate(mpcd_traj *t, mpcd_surrogate *s) {
  if (!s || !t || traj_colloids(t) != s->S.Nc) return MPCD_ERR_PARAM;
  const int r = traj_record_f4(t, s->S.X, s->S.V, s->S.ra, s->stream);
  return r ? sfail(s, r, mpcd_traj_last_error(t)) : MPCD_OK;
}

extern "C" int mpcd_surrogate_features(mpcd_surrogate *s, float *out, int recompute) {
  if (!s || !out) return MPCD_ERR_PARAM;
  const Sur &S = s->S;
  if (recompute) k_sur_features<<<(S.Nc + 3) / 4, 128, 0, s->stream>>>(S);
  if (cudaMemcpyAsync(out, S.feat, sizeof(float) * NF * S.Nc, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return sfail(s, MPCD_ERR_CUDA, "features");
  return MPCD_OK;
}

extern "C" int mpcd_surrogate_fast_steps(mpcd_surrogate *s, int64_t *count) {
  if (!s || !count) return MPCD_ERR_PARAM;
  long long c = 0;
  if (cudaMemcpyAsync(&c, s->S.fast, sizeof c, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return sfail(s, MPCD_ERR_CUDA, "fast-step count");
  *count = c;
  return MPCD_OK;
}

// the network's outputs of the last step in physical units (n_colloid x 12, host)
extern "C" int mpcd_surrogate_outputs(mpcd_surrogate *s, float *out) {
  if (!s || !out) return MPCD_ERR_PARAM;
  const Sur &S = s->S;
  k_sur_denorm<<<(S.Nc * NO + 255) / 256, 256, 0, s->stream>>>(S, s->outd);
  if (cudaMemcpyAsync(out, s->outd, sizeof(float) * NO * S.Nc, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return sfail(s, MPCD_ERR_CUDA, "outputs");
  return MPCD_OK;
}

extern "C" int mpcd_surrogate_set_fault(mpcd_surrogate *s, int drop_chunk) {
  if (!s || drop_chunk < -1 || drop_chunk >= NCHUNK || (drop_chunk >= 0 && drop_chunk < FAULT_FIRST))
    return sfail(s, MPCD_ERR_PARAM, "drop_chunk: -1, or a weight chunk the producer loop issues");
  s->S.drop_chunk = drop_chunk;
  drop_graphs(s);  // the kernels take the parameters by value: capture again
  return MPCD_OK;
}

extern "C" int mpcd_surrogate_set_noise(mpcd_surrogate *s, double scale) {
  if (!s || !(scale >= 0.0) || !(scale <= 1e3)) return sfail(s, MPCD_ERR_PARAM, "noise scale: 0 .. 1000");
  s->S.noise = (float)scale;
  drop_graphs(s);  // the kernels take the parameters by value: capture again
  return MPCD_OK;
}

extern "C" int mpcd_surrogate_step(mpcd_surrogate *s, int nsteps) {
  if (!s || nsteps < 0) return MPCD_ERR_PARAM;
  // each call starts with the error bits clear: a failed call leaves the state as it was
  // before its failing step, and the next call may go on from there
  if (cudaMemsetAsync(s->S.err, 0, sizeof(int), s->stream) != cudaSuccess) return sfail(s, MPCD_ERR_CUDA, "step");
  if (nsteps > 0 && pack_weights(s) != MPCD_OK) return MPCD_ERR_CUDA;
  for (int left = nsteps; left > 0;) {
    const int many = left >= GRAPH_STEPS ? 1 : 0, n = many ? GRAPH_STEPS : 1;
    if (!s->exec[many]) {
      cudaGraph_t g;
      if (cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        return sfail(s, MPCD_ERR_CUDA, "capture");
      int r = enqueue_steps(s, n);
      cudaError_t e = cudaStreamEndCapture(s->stream, &g);
      if (r) return r;
      if (e != cudaSuccess) return sfail(s, MPCD_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
      e = cudaGraphInstantiate(&s->exec[many], g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return sfail(s, MPCD_ERR_CUDA, std::string("instantiate: ") + cudaGetErrorString(e));
    }
    if (cudaGraphLaunch(s->exec[many], s->stream) != cudaSuccess) return sfail(s, MPCD_ERR_CUDA, "graph launch");
    left -= n;
  }
  int bits = 0;
  if (cudaMemcpyAsync(&bits, s->S.err, sizeof(int), cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return sfail(s, MPCD_ERR_CUDA, std::string("step: ") + cudaGetErrorString(cudaGetLastError()));
  if (bits & 3)
    return sfail(s, MPCD_ERR_CAPACITY, "a colloid has more neighbours than its lists hold (64 within three radii "
                                       "or the force cutoff plus 4, 32 within the force cutoff plus 2)");
  if (bits) return sfail(s, MPCD_ERR_CUDA, "a weight copy of the network kernel did not arrive");
  return MPCD_OK;
}
