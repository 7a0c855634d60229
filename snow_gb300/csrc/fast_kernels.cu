// SNOW_MODE_FAST kernels for sm_103a: the explicit snow-MPM step of the
// reference (shader/compute/mpm/*.glsl) in FP32 without fixed-point
// quantisation, on a blocked grid.
//
// Grid layout in HBM. The grid is cut into 4x4x4-node blocks.
//   acc      dense, one 3584-byte record per block: the P2G sums (m, p, f)
//            as fixed-point integers (seven int64 words per node,
//            word-major), so that they do not depend on the order they are
//            added in. All zero between steps: the grid update clears what
//            it consumes.
//   blk_flag blocks that received P2G sums (set by the P2G tile flush).
//   compact  turns the flags into the active-block list and gives each
//            active block a slot (its place in the list).
//   gout     dense over the nodes, x fastest: the grid update's output v* and
//            d = v* - alpha p/m, one 6-float record per node; zero in blocks
//            that are not active.
//
// Kernels of one step (every scene of a batch in one launch each):
//   compact      flags -> slots, active list; the step's start (counters,
//                scales, colliders)                (thread per four blocks)
//   grid         per active block: v* = p/m + dt (f/m + g), colliders, d
//   g2p2g        per work item (<= 256 particles binned to one home block):
//                bulk-copy (TMA) the 81 rows of nodes around the home block
//                into shared memory, gather v* and d (G2P), update F_E with
//                the SVD clamp, J_p, velocity, colliders, position (particle
//                advance), then scatter the updated particles (P2G of the
//                next step) into a 9^3-node shared tile, cell by cell, and
//                add the tile to acc. The items of one home block (a run)
//                share
//                the staged grid rows and the tile, which is added to acc
//                once per run.
// Separate P2G and G2P kernels serve the first step after set-up and the
// per-kernel dispatch entry point.
#include <algorithm>

#include "snow_internal.h"
#include "snow_math.cuh"
#include "snow_stats.cuh"
#include "snow_tma.cuh"
#include "fast_item.cuh"

namespace snow {
namespace {

// ===========================================================================
// Item and active-block prefixes of the scenes, by one full warp; the slots
// handed out become the scenes' active blocks.
__device__ __forceinline__ void form_prefixes(const SceneDev* __restrict__ scenes, int nscenes, int* items,
                                              int* active) {
  const int lane = threadIdx.x & 31;
  int items0 = 0, active0 = 0;
  for (int s0 = 0; s0 < nscenes; s0 += 32) {
    int ni = 0, na = 0;
    if (s0 + lane < nscenes) {
      const SceneDev& S = scenes[s0 + lane];
      ni = *(volatile int*)&S.counters[CNT_ITEMS];
      na = *(volatile int*)&S.counters[CNT_SLOTS];
      S.counters[CNT_ACTIVE] = na;
      S.counters[CNT_SLOTS] = 0;
      S.counters[CNT_OVERFLOW] = max(0, na - S.pool_cap);
      na = min(na, S.pool_cap);
    }
    int ei = ni, ea = na;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int vi = __shfl_up_sync(0xffffffffu, ei, o), va = __shfl_up_sync(0xffffffffu, ea, o);
      if (lane >= o) {
        ei += vi;
        ea += va;
      }
    }
    if (s0 + lane < nscenes) {
      items[s0 + lane] = items0 + ei - ni;
      active[s0 + lane] = active0 + ea - na;
    }
    items0 += __shfl_sync(0xffffffffu, ei, 31);
    active0 += __shfl_sync(0xffffffffu, ea, 31);
  }
  if (lane == 0) {
    items[nscenes] = items0;
    active[nscenes] = active0;
  }
}

// rigidAdvance.glsl:14-18, by one warp.
__device__ __forceinline__ void advance_colliders(const SceneDev& S, int lane) {
  for (int i = lane; i < S.ncoll; i += 32)
    for (int k = 0; k < 3; k++) S.coll[i].pos[k] = S.coll[i].pos[k] + S.dt * S.coll[i].vel[k];
}

// The start of a step for scene S, by one warp: counters reset, the magnitudes
// moved on and the scales of this step's P2G formed from them, colliders
// advanced, the solve's scalars cleared.
__device__ __forceinline__ void begin_scene(const SceneDev& S, bool rigid, bool binned, bool set_up) {
  const int lane = threadIdx.x & 31;
  if (rigid) advance_colliders(S, lane);
  if (lane == 0) {
    S.counters[CNT_WORK] = 0;
    if (!binned) S.counters[CNT_BINNED] = 0;
    // the magnitudes of the particles the pending P2G scattered become the
    // ones this step's P2G chooses its fixed-point scales from
    FixState& f = *S.fix;
    f.m_prev = f.m_cur;
    f.v_prev = f.v_cur;
    f.a_prev = f.a_cur;
    f.m_cur = f.v_cur = f.a_cur = 0u;
    const FixScale sc = step_scales(S);
    f.next[0] = sc.m;
    f.next[1] = sc.p;
    f.next[2] = sc.f;
  }
  if (S.crs) {  // the semi-implicit solve's scalars start from zero each step
    int* c = reinterpret_cast<int*>(S.crs);
    for (int i = lane; i < (int)(offsetof(CrScalars, skipping) / sizeof(int)); i += 32) c[i] = 0;
    if (lane == 0) {  // a step within kCrSkipSteps of a start below kCrSkipFactor * tol skips the solve
      CrScalars& cs = *S.crs;
      if (set_up) cs.skip_left = 0;
      cs.skipping = cs.skip_left > 0 ? 1 : 0;
      if (cs.skip_left > 0) cs.skip_left--;
    }
  }
}

// The rigid advance alone (per-kernel dispatches): it starts no step, so what the
// start of one moves on (the magnitudes, the solve's count of steps to skip) stays.
__global__ void k_rigid(const SceneDev* __restrict__ sd) { advance_colliders(*sd, threadIdx.x); }

__global__ void k_gather_counters(const SceneDev* __restrict__ scenes, int nscenes, int* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nscenes * kCounterStride; i += gridDim.x * blockDim.x)
    out[i] = scenes[i / kCounterStride].counters[i % kCounterStride];
  __threadfence_system();
}

// The outputs of a block that is no longer active read as zero.
__device__ __noinline__ void clear_block(const SceneDev& S, int b) {
  int bx, by, bz;
  home_coords(S, b, bx, by, bz);
  for (int r = 0; r < 16; r++) {
    const size_t row = node_index(S, 4 * bx, 4 * by + (r & 3), 4 * bz + (r >> 2));
    float4* o = reinterpret_cast<float4*>(S.gout + row * kOutFields);
    for (int k = 0; k < kOutFields; k++) o[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!S.crs) continue;
    float4* u = reinterpret_cast<float4*>(S.cru + row * kImpFields);
    for (int k = 0; k < kImpFields; k++) u[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// Flags -> active-block list and slots, four blocks per thread; a block that
// was active before and is not now has its outputs cleared (few blocks a
// step). The first CTAs start the step of the scenes instead (a launch of its own
// for that took 3 us of a step), and the CTA that takes its slots last forms
// the item and active-block prefixes. Bound by a chain of round trips to L2
// (flags, slots, count of the CTAs, prefixes) in small grids and by the 8 bytes a
// block it reads in large ones. The scenes' start in CTAs of its own, the CTAs
// counted before they write their lists and the prefixes formed by a warp:
// 5.1 to 3.9 us on 64^3 nodes, 7.5 to 5.7 on 256^3, 17.0 to 15.6 on 512^3.
// BINNED: the step's binning has left the particles in the binned copies.
constexpr int kCompactThreads = 256;
__global__ void __launch_bounds__(kCompactThreads) k_compact(const SceneDev* __restrict__ scenes, const int* quad_prefix,
                                                             int nscenes, long long total, int* items_prefix,
                                                             int* active_prefix, int rigid, int binned, int set_up) {
  constexpr int kWarps = kCompactThreads / 32;
  const int begin_ctas = (nscenes + kWarps - 1) / kWarps;
  chain_next();
  chain_wait();
  if ((int)blockIdx.x < begin_ctas) {
    const int s = (int)blockIdx.x * kWarps + (int)(threadIdx.x >> 5);
    if (s < nscenes) begin_scene(scenes[s], rigid != 0, binned != 0, set_up != 0);
    return;
  }
  const long long u = ((long long)blockIdx.x - begin_ctas) * kCompactThreads + threadIdx.x;
  const int s = find_scene(quad_prefix, nscenes, min(u, total - 1));
  const SceneDev& S = scenes[s];
  const int q = (int)(min(u, total - 1) - (nscenes == 1 ? 0 : quad_prefix[s]));
  // (the arrays are whole 256-byte units long)
  const int4 f4 = reinterpret_cast<const int4*>(S.blk_flag)[q], o4 = reinterpret_cast<const int4*>(S.blk_slot)[q];
  const int flag[4] = {f4.x, f4.y, f4.z, f4.w}, old[4] = {o4.x, o4.y, o4.z, o4.w};
  int want = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) want += u < total && 4 * q + k < S.nblocks && flag[k] != 0;
  int slot = want ? atomicAdd(&S.counters[CNT_SLOTS], want) : 0;
  // the CTA's slots are taken: counted before the lists are written
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&scenes[0].counters[CNT_DONE], 1) == (int)gridDim.x - begin_ctas - 1;
  }
  if (u < total && (want || (old[0] & old[1] & old[2] & old[3]) != -1)) {  // active now or before
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int b = 4 * q + k;
      if (b >= S.nblocks) break;
      int now = -1;
      if (flag[k]) {
        S.blk_flag[b] = 0;
        now = slot++;
        if (now >= S.pool_cap)
          now = -1;  // (counted by form_prefixes)
        else
          S.active[now] = b;
      }
      if (now != old[k]) S.blk_slot[b] = now;
      if (now < 0 && old[k] >= 0) clear_block(S, b);
    }
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  form_prefixes(scenes, nscenes, items_prefix, active_prefix);
  if (threadIdx.x == 0) scenes[0].counters[CNT_DONE] = 0;
}

// Largest mass, |v|, force-term bound and initial volume of the particles a
// P2G of the stored state scatters (with_stress: A from an SVD of F_E, as
// that P2G computes it), into FixState's *_prev and *_cur (zeroed before).
__global__ void __launch_bounds__(256) k_fix_measure(const SceneDev* __restrict__ sd, int with_stress) {
  const SceneDev& S = *sd;
  float mm = 0.0f, vm = 0.0f, am = 0.0f, v0 = 0.0f;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.n; p += gridDim.x * blockDim.x) {
    const float4 xm = S.xm[p];
    if (!(fabsf(xm.w) <= 100.0f)) continue;  // not scattered (p2gTransfer.glsl:64-66)
    const float4 vv = S.vv[p];
    mm = fmaxf(mm, fabsf(xm.w));
    vm = fmaxf(vm, sqrtf(vv.x * vv.x + vv.y * vv.y + vv.z * vv.z));
    v0 = fmaxf(v0, vv.w);
    if (with_stress) am = fmaxf(am, p2g_particle(S, p, xm, false).a);
  }
  // one warp's maxima per block, and only those above what is recorded: the
  // same seven words for every warp of the GPU (39 us at 262k particles,
  // now 12)
  __shared__ unsigned best[4];
  if (threadIdx.x < 4) best[threadIdx.x] = 0u;
  __syncthreads();
  const unsigned b[4] = {__reduce_max_sync(0xffffffffu, __float_as_uint(mm)), __reduce_max_sync(0xffffffffu, __float_as_uint(vm)),
                         __reduce_max_sync(0xffffffffu, __float_as_uint(am)), __reduce_max_sync(0xffffffffu, __float_as_uint(v0))};
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < 4; k++) atomicMax(&best[k], b[k]);
  __syncthreads();
  if (threadIdx.x < 7) {
    FixState& f = *S.fix;
    uint32_t* to[7] = {&f.m_prev, &f.m_cur, &f.v_prev, &f.v_cur, &f.a_prev, &f.a_cur, &f.v0max};
#pragma unroll
    for (int k = 0; k < 7; k++)
      if ((int)threadIdx.x == k && best[k / 2] > *(volatile uint32_t*)to[k]) atomicMax(to[k], best[k / 2]);
  }
}

// P2G of the stored particle state (p2gTransfer.glsl:44-151, or
// gMassCompute.glsl:33-84 when MASS_ONLY), at the scales k_fix_measure's
// magnitudes give; the CTA that takes a scene's first item records them for
// the grid update.
template <bool MASS_ONLY>
__global__ void __launch_bounds__(kItemMax, kItemCtas) k_p2g(const SceneDev* __restrict__ scenes,
                                                  const int* __restrict__ item_prefix, int nscenes) {
  extern __shared__ float4 smem_raw[];
  ItemShared& sh = *reinterpret_cast<ItemShared*>(smem_raw);
  tile_init(sh);
  constexpr int KIND = MASS_ONLY ? kP2gMass : kP2gFull;
  const int total = item_prefix[nscenes];
  for (int u = blockIdx.x; u < total; u += gridDim.x) {
    const int s = find_scene(item_prefix, nscenes, u);
    const SceneDev& S = scenes[s];
    const int4 it = S.items[u - item_prefix[s]];
    const FixScale sc = measured_scales(S);
    if (u == item_prefix[s] && threadIdx.x == 0) {
      S.fix->scale[0] = sc.m;
      S.fix->scale[1] = sc.p;
      S.fix->scale[2] = sc.f;
    }
    tile_zero(sh, P2gFields<KIND>::nf);
    int bx, by, bz;
    home_coords(S, it.x, bx, by, bz);
    const int i = threadIdx.x;
    bool have = false;
    P2GParticle q;
    q.force = false;
    q.a = 0.0f;
    AxisW w;
    int base[3] = {0, 0, 0};
    if (i < min(it.z, kItemMax)) {
      const int p = it.y + i;
      const float4 xm = S.xm[p];
      if (fabsf(xm.w) <= 100.0f) {  // p2gTransfer.glsl:64-66
        float pg[3];
        grid_coords(S, xm, pg, base);
        all_weights(pg, base, w);
        q = p2g_particle(S, p, xm, MASS_ONLY);
        have = true;
      }
    }
    P2GStored stored;
    p2g_count<KIND>(sh, S, bx, by, bz, have, q, w, base, sc, stored);
    __syncthreads();
    p2g_sum<KIND>(sh, S, bx, by, bz, stored, w);
    p2g_tile_flush<KIND>(sh, S, bx, by, bz);
    __syncthreads();
  }
}

// gForceCompute.glsl:57-103 for one node of active block b (pool slot
// `slot`) from its seven fixed-point sums w.
__device__ __forceinline__ void grid_node(const SceneDev& S, int slot, int b, int node,
                                          const unsigned long long (&w)[kAccWords]) {
  // the fixed-point sums back to floats (the scales are powers of two)
  const FixState& fx = *S.fix;
  const float ism = 1.0f / fx.scale[0], isp = 1.0f / fx.scale[1], isf = 1.0f / fx.scale[2];
  const long long mq = (long long)w[0];
  const float v[kAccFields] = {(float)mq * ism,
                               (float)(long long)w[1] * isp,
                               (float)(long long)w[2] * isp,
                               (float)(long long)w[3] * isp,
                               (float)(long long)w[4] * isf,
                               (float)(long long)w[5] * isf,
                               (float)(long long)w[6] * isf};
  int bx, by, bz;
  home_coords(S, b, bx, by, bz);
  const int gi = 4 * bx + (node & 3), gj = 4 * by + ((node >> 2) & 3), gk = 4 * bz + (node >> 4);
  const size_t ni = node_index(S, gi, gj, gk);
  float2* out = reinterpret_cast<float2*>(S.gout + ni * kOutFields);
  const float mi = v[0];
  float vs[3] = {0.0f, 0.0f, 0.0f}, d[3] = {0.0f, 0.0f, 0.0f};
  if (mq > 0) {
    const float inv = 1.0f / mi;
    const float vold[3] = {v[1] * inv, v[2] * inv, v[3] * inv};
#pragma unroll
    for (int k = 0; k < 3; k++) vs[k] = vold[k] + S.dt * (v[4 + k] * inv + S.grav[k]);
    // node position as Grid::initSSBO forms it: x_off + h * (float)i
    const float xi[3] = {__fadd_rn(S.gpos[0], __fmul_rn(S.h, (float)gi)),
                         __fadd_rn(S.gpos[1], __fmul_rn(S.h, (float)gj)),
                         __fadd_rn(S.gpos[2], __fmul_rn(S.h, (float)gk))};
    collide(S.coll, S.ncoll, xi, vs);
#pragma unroll
    for (int k = 0; k < 3; k++) d[k] = vs[k] - S.alpha * vold[k];
  }
  out[0] = make_float2(vs[0], vs[1]);
  out[1] = make_float2(vs[2], d[0]);
  out[2] = make_float2(d[1], d[2]);
  if (S.crs && !S.crs->skipping) {  // semi-implicit: the solve starts from x = v* and applies K to v* first
    const size_t i = (size_t)slot * kBlockNodes + node;
    S.crv[i] = make_float4(vs[0], vs[1], vs[2], mi > 0.0f ? mi : 0.0f);
    float* u = S.cru + ni * kImpFields;
    u[0] = vs[0];
    u[1] = vs[1];
    u[2] = vs[2];
  }
}

// The grid update on the active blocks, one 64-thread group per block (a
// warp lies inside one group, so inside one scene). Each group's blocks are
// staged by TMA: a block's fixed-point record is one contiguous 3,584-byte
// bulk copy into the group's shared buffer, and the group's next block is
// copied while it converts, updates and writes the current one. The P2G
// sums are consumed (zeroed) here. clear_only: the sums are zeroed and
// nothing is staged or written (scene set-up).
constexpr int kGridGroups = 4;  // 64-thread groups per CTA
__global__ void __launch_bounds__(kGridGroups * kBlockNodes) k_grid(const SceneDev* __restrict__ scenes,
                                                                    const int* active_prefix, int nscenes,
                                                                    int clear_only) {
  __shared__ __align__(128) unsigned long long buf[kGridGroups][kAccBlockWords];
  __shared__ uint64_t bar[kGridGroups];
  __shared__ int gabort[kGridGroups];
  const int g = threadIdx.x / kBlockNodes, node = threadIdx.x % kBlockNodes;
  chain_next();
  if (node == 0) {
    mbar_init(&bar[g], 1);
    gabort[g] = 0;
  }
  __syncthreads();
  chain_wait();
  const long long total = active_prefix[nscenes];
  const long long stride = (long long)gridDim.x * kGridGroups;
  long long u = (long long)blockIdx.x * kGridGroups + g;
  if (clear_only) {
    for (; u < total; u += stride) {
      const int s = find_scene(active_prefix, nscenes, u);
      const SceneDev& S = scenes[s];
      unsigned long long* acc = S.acc + (size_t)S.active[(int)(u - active_prefix[s])] * kAccBlockWords + node;
#pragma unroll
      for (int k = 0; k < kAccWords; k++) acc[k * kBlockNodes] = 0ull;
    }
    return;
  }
  constexpr uint32_t kBytes = kAccBlockWords * sizeof(unsigned long long);
  static_assert(kBytes % 16 == 0, "bulk copies move multiples of 16 bytes");
  // the block of work unit uu: its scene, pool slot and block id
  auto locate = [&](long long uu, int& s, int& slot, int& b) {
    s = find_scene(active_prefix, nscenes, uu);
    slot = (int)(uu - active_prefix[s]);
    b = scenes[s].active[slot];
  };
  auto issue = [&](long long uu) {  // by the group's thread 0
    int s, slot, b;
    locate(uu, s, slot, b);
    const SceneDev& S = scenes[s];
    mbar_arrive_expect_tx(&bar[g], kBytes + S.tx_unsent);
    fence_proxy_async_smem();
    bulk_g2s(buf[g], S.acc + (size_t)b * kAccBlockWords, kBytes, &bar[g]);
  };
  if (u < total && node == 0) issue(u);
  uint32_t phase = 0;
  for (; u < total; u += stride) {
    int s, slot, b;
    locate(u, s, slot, b);
    const SceneDev& S = scenes[s];
    unsigned long long w[kAccWords];
    const bool landed = mbar_wait(&bar[g], phase, S.wait_ns);
    if (landed) {
#pragma unroll
      for (int k = 0; k < kAccWords; k++) w[k] = buf[g][k * kBlockNodes + node];
    } else {
      gabort[g] = 1 + (int)phase;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(kBlockNodes) : "memory");  // the group has read its buffer
    if (gabort[g]) {
      // the copy did not land in time: counted, one more bounded wait for it
      // (the CTA must not exit while it may still land), and the group stops
      if (node == 0) {
        atomicAdd(&S.counters[CNT_TIMEOUT], 1);
        mbar_wait(&bar[g], (uint32_t)(gabort[g] - 1), S.wait_ns);
      }
      return;
    }
    phase ^= 1u;
    if (node == 0 && u + stride < total) issue(u + stride);
    unsigned long long* acc = S.acc + (size_t)b * kAccBlockWords + node;
#pragma unroll
    for (int k = 0; k < kAccWords; k++) acc[k * kBlockNodes] = 0ull;
    grid_node(S, slot, b, node, w);
  }
}

// pVolumeCompute.glsl:32-83: rho0 = sum_i m_i w_ip / h^3 from the grid mass,
// stored as V0 = m / rho0 (0 when rho0 <= 0, which disables the force as
// p2gTransfer.glsl:126 does). Per work item: the masses of its tile's nodes go to
// shared memory once instead of being read (as int64 words) 64 times a particle:
// 167 us at 1M particles, now 51. A particle whose stencil leaves the
// tile (outside the grid, binned to its border) reads them from the grid.
__device__ __forceinline__ float node_mass(const SceneDev& S, int g0, int g1, int g2, float scale_inv) {
  if (!node_in_grid(S, g0, g1, g2)) return 0.0f;
  const int blk = block_id(S, g0 >> 2, g1 >> 2, g2 >> 2);
  const long long mq = (long long)S.acc[(size_t)blk * kAccBlockWords + (g0 & 3) + 4 * (g1 & 3) + 16 * (g2 & 3)];
  return (float)mq * scale_inv;  // the scale is a power of two
}
__global__ void __launch_bounds__(256) k_volume(const SceneDev* __restrict__ sd, const int* __restrict__ item_prefix) {
  __shared__ float mass[kTile3];
  const SceneDev& S = *sd;
  const float si = 1.0f / S.fix->scale[0];
  const int total = item_prefix[1];
  for (int u = blockIdx.x; u < total; u += gridDim.x) {
    const int4 it = S.items[u];
    int bx, by, bz;
    home_coords(S, it.x, bx, by, bz);
    for (int t = threadIdx.x; t < kTile3; t += blockDim.x)
      mass[t] = node_mass(S, 4 * bx - 2 + t % kTile, 4 * by - 2 + (t / kTile) % kTile, 4 * bz - 2 + t / (kTile * kTile), si);
    __syncthreads();
    for (int i = threadIdx.x; i < it.z; i += blockDim.x) {
      const int p = it.y + i;
      const float4 xm = S.xm[p];
      float pg[3];
      int base[3], t[3];
      grid_coords(S, xm, pg, base);
      AxisW w;
      all_weights(pg, base, w);
      const bool inside = stencil_in_tile(bx, by, bz, base, t);
      float rho = 0.0f;
#pragma unroll
      for (int c = 0; c < 4; c++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
          for (int a = 0; a < 4; a++) {
            const float mi = inside ? mass[t[0] + a + kTile * (t[1] + b) + kTile * kTile * (t[2] + c)]
                                    : node_mass(S, base[0] - 1 + a, base[1] - 1 + b, base[2] - 1 + c, si);
            rho += mi * (w.wx[a] * w.wy[b] * w.wz[c]);
          }
      rho = rho / (S.h * S.h * S.h);
      float4 vv = S.vv[p];
      vv.w = rho > 0.0f ? xm.w / rho : 0.0f;
      S.vv[p] = vv;
    }
    __syncthreads();
  }
}

// g2pTransfer.glsl:53-143 fused with particleAdvance.glsl:75-217 (no P2G).
__global__ void __launch_bounds__(kItemMax) k_g2p_advance(const SceneDev* __restrict__ scenes,
                                                          const int* __restrict__ item_prefix, int nscenes) {
  extern __shared__ float4 smem_raw[];
  ItemShared& sh = *reinterpret_cast<ItemShared*>(smem_raw);
  tile_init(sh);
  const int total = item_prefix[nscenes];
  uint32_t phase = 0;
  for (int u = blockIdx.x; u < total; u += gridDim.x) {
    const int s = find_scene(item_prefix, nscenes, u);
    const SceneDev& S = scenes[s];
    const int4 it = S.items[u - item_prefix[s]];
    int bx, by, bz;
    home_coords(S, it.x, bx, by, bz);
    stage_issue<kOutFields>(sh, S, S.gout, it.x);
    load_colliders(sh, S);
    stage_wait(sh, S, phase);
    __syncthreads();
    if (sh.abort) {
      stage_abort(sh, S);
      return;
    }
    for (int i = threadIdx.x; i < it.z; i += blockDim.x) {
      const int p = it.y + i;
      const PState ps = load_state(S, p, false);  // per-kernel dispatches: binned in place
      float pg[3];
      int base[3];
      grid_coords(S, ps.xm, pg, base);
      AxisW w;
      all_weights(pg, base, w);
      float dv[3], L[3][3];
      g2p_gather(sh, S, bx, by, bz, base, w, dv, L);
      Advanced adv;
      advance_particle(S, p, ps, load_def(S, p, false), dv, L, sh, adv);
    }
    __syncthreads();
  }
}

// One explicit step per particle: G2P + particle advance of this step and
// P2G of the next, in one pass over the item's particles. The P2G stress uses
// the rotation R = W V^T of the advance's SVD: F_E' = W S' V^T with S'
// diagonal up to the Jacobi residual, whose polar rotation is W V^T.
// The CTAs take units of work from a counter: the items of a home block (a run)
// or some of them. The items of a unit share
// the staged grid rows (copied once, by bulk copies issued while the
// previous run's last item sums its P2G) and the P2G tile (added to acc
// once, at the run's end). The P2G sums are fixed
// point at the scales step_scales gives; the CTA that takes a scene's first
// item records them for the next grid update, and every CTA records the
// magnitudes of its particles for the next step's scales. BINNED: a step that
// re-binned some scene; such a scene's particles are read from its binned
// copies (CNT_BINNED) and, like every scene's, written to its streams. WIDE: with
// the sums of kCellWide particles (in shared memory; else by atomics on acc).
constexpr int kSingleRounds = 3, kUnitShare = 4;
template <bool BINNED, bool WIDE>
__global__ void __launch_bounds__(kItemMax, kItemCtas) k_g2p2g(const SceneDev* __restrict__ scenes,
                                                       const int* item_prefix, int nscenes) {
  extern __shared__ float4 smem_raw[];
  ItemShared& sh = *reinterpret_cast<ItemShared*>(smem_raw);
  chain_next();
  tile_zero(sh, kAccFields);
  tile_init(sh);
  chain_wait();
  const int total = item_prefix[nscenes];
  // A unit is a run, or unit_most of its items at a time; in the last round of the CTAs
  // (runs that start in the last gridDim.x items), and in launches of up to three
  // rounds, a single item. A run costs one copy of the grid rows and one flush, but the
  // CTA that takes it last works on alone: with whole runs to the end 50 steps of 1M
  // particles took 15.46 ms, with single items in the last round 15.08, in the last two
  // or four 15.13 and 15.21; 16M the same. 32 steps of 262k particles (4.6 rounds): 3.97
  // ms all single, 3.85 in pairs; 20 steps of 300k (4.8): 3.16, 3.12, with whole runs
  // 3.41. unit_most is about a quarter of a CTA's items, and at least two, because snow
  // pressed together lies in fewer runs than there are CTAs: 1M particles at 300 to a
  // cell, 218 runs of up to 31 items, 480 us a step in whole runs, 232 in units of up to four.
  // The counter instead of equal shares of consecutive items: the items differ
  // (surface blocks hold few particles, compressed snow costs more), 24 steps of a
  // 1.5M-particle block on a sphere 12.0 to 11.0 ms, 50 of 1M particles 17.2 to 16.3.
  int* counter = &scenes[0].counters[CNT_WORK];
  // the length of the unit that starts at item u (`it`, of scene s); 0: none does
  auto unit_at = [&](int u, int s, const int4& it) {
    const int at = it.w > 0 ? 0 : -it.w;  // its place in its run
    if (u - at >= sh.unit_tail) return 1;
    const int most = sh.unit_most;
    if ((at & (most - 1)) != 0) return 0;
    return min(most, (at == 0 ? it.w : scenes[s].items[u - at - item_prefix[s]].w) - at);
  };
  // the first item of the unit that starts at item u or at one handed out after
  // it, and the unit's length
  auto next_unit = [&](int u, int& s, int4& it, int& len) {
    for (;;) {
      if (u >= total) return total;
      s = find_scene(item_prefix, nscenes, u);
      it = scenes[s].items[u - item_prefix[s]];
      len = unit_at(u, s, it);
      if (len > 0) return u;
      u = (int)gridDim.x + atomicAdd(counter, 1);
    }
  };
  // The last warp, which holds the fewest particles of an item (items are
  // filled from thread 0), looks up the next item and issues the copies of its
  // particles.
  const int lane = threadIdx.x & 31;
  const bool lastw = (threadIdx.x >> 5) == (blockDim.x >> 5) - 1;
  if (lastw && lane == 0) {
    const int round = (int)gridDim.x;
    sh.unit_tail = total <= kSingleRounds * round ? 0 : total - round;
    sh.unit_most = 1 << max(1, __clz(round) - __clz(total / kUnitShare | 1));
    int s0 = 0, len = 1;
    int4 it0 = make_int4(0, 0, 0, 0);
    sh.index_q[0] = next_unit((int)blockIdx.x, s0, it0, len);
    sh.unit_left = len - 1;
    sh.item_q[0] = it0;
    sh.scene_q[0] = s0;
    sh.coll_scene = -1;
    sh.next_same = 0;
  }
  __syncthreads();
  if (sh.index_q[0] >= total) return;  // uniform across the CTA
  {
    const SceneDev& S0 = scenes[sh.scene_q[0]];
    const int4 it0 = sh.item_q[0];
    stage_issue<kOutFields>(sh, S0, S0.gout, it0.x);
    if (lastw) particles_issue(sh, S0, it0.y, min(it0.z, kItemMax), BINNED && particles_binned(S0));
  }
  uint32_t phase = 0, pphase = 0;
  int par = 0;
  bool run_start = true;  // uniform across the CTA
  for (;; par ^= 1) {
    __syncthreads();  // this item's queue entry is written; the last flush is done
    const int u = sh.index_q[par];
    if (u >= total) return;  // uniform across the CTA
    const int s = sh.scene_q[par];
    const SceneDev& S = scenes[s];
    if (s != sh.coll_scene) {  // uniform across the CTA
      if (threadIdx.x == 0) {
        sh.fscale = FixScale{S.fix->next[0], S.fix->next[1], S.fix->next[2]};
        sh.seen[0] = sh.seen[1] = sh.seen[2] = 0u;
        sh.pushed[0] = sh.pushed[1] = sh.pushed[2] = 0u;
      }
      load_colliders(sh, S);  // its closing barrier publishes fscale as well
      if (threadIdx.x == 0) sh.coll_scene = s;
    }
    if (threadIdx.x == 0 && u == item_prefix[s]) {
      S.fix->scale[0] = sh.fscale.m;
      S.fix->scale[1] = sh.fscale.p;
      S.fix->scale[2] = sh.fscale.f;
    }
    if (run_start && threadIdx.x == 0) sh.run_bound = 0.0f;
    const int4 it = sh.item_q[par];
    // the next item: handed out (at the end of a unit) while this one's particles
    // and grid values are waited for, copied to its queue entry during the gather and
    // looked at after it. Looked up at the item's start, the last warp waited for the
    // atomic and the load in turn and the others for it: 12 steps of 16M particles
    // 63.0 to 62.3 ms, 24 of a 1.5M block 9.70 to 9.60, 50 of 1M 15.06 to 14.94.
    int un = u + 1;
    if (lastw && lane == 0 && sh.unit_left <= 0) un = (int)gridDim.x + atomicAdd(counter, 1);
    int bx, by, bz;
    home_coords(S, it.x, bx, by, bz);
    const int i = threadIdx.x;
    const bool mine = i < min(it.z, kItemMax);
    const int p = it.y + i;
    bool landed = particles_wait(sh, S, pphase);
    if (run_start) landed = stage_wait(sh, S, phase) && landed;
    if (lastw && lane == 0 && un < total) {
      const int sn = find_scene(item_prefix, nscenes, un);
      copy_async16(&sh.item_q[par ^ 1], &scenes[sn].items[un - item_prefix[sn]]);
      sh.scene_q[par ^ 1] = sn;
    }
    bool have = false;
    P2GParticle q;
    q.force = false;
    q.a = 0.0f;
    AxisW wn;
    int nbase[3] = {0, 0, 0};
    float rec_v = 0.0f;
    if (mine && landed) {
      PState ps;
      ps.xm = sh.pxm[i];
      float pg[3];
      int base[3];
      grid_coords(S, ps.xm, pg, base);
      AxisW w;
      all_weights(pg, base, w);
      float dv[3], L[3][3];
      g2p_gather(sh, S, bx, by, bz, base, w, dv, L);
      ps.vv = sh.pvv[i];
      const PDef def = {sh.pfa[i], sh.pfb[i], sh.pvq[i], sh.pfc[i + (it.y & 1)]};
      Advanced adv;
      advance_particle(S, p, ps, def, dv, L, sh, adv);
      if (BINNED && particles_binned(S)) S.pid[p] = S.bpid[p];
      // P2G quantities of the advanced particle
      q.m = adv.xm.w;
      if (fabsf(q.m) <= 100.0f) {  // p2gTransfer.glsl:64-66
        have = true;
        q.mv[0] = q.m * adv.vv.x;
        q.mv[1] = q.m * adv.vv.y;
        q.mv[2] = q.m * adv.vv.z;
        rec_v = sqrtf(adv.vv.x * adv.vv.x + adv.vv.y * adv.vv.y + adv.vv.z * adv.vv.z);
        if (adv.vv.w > 0.0f) p2g_stress(S, adv.fe, adv.R, adv.jp, adv.vv.w, q);
        float npg[3];
        grid_coords(S, adv.xm, npg, nbase);
        all_weights(npg, nbase, wn);
      }
    }
    {  // the magnitudes the next step's scales are chosen from (per warp, then per CTA)
      const unsigned bm = __reduce_max_sync(0xffffffffu, have ? __float_as_uint(fabsf(q.m)) : 0u);
      const unsigned bv = __reduce_max_sync(0xffffffffu, __float_as_uint(rec_v));
      const unsigned ba = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(q.a, 0.0f)));  // (0 for NaN)
      if (lane == 0) {
        atomicMax(&sh.seen[0], bm);
        atomicMax(&sh.seen[1], bv);
        atomicMax(&sh.seen[2], ba);
      }
    }
    // the rest of the queue entry: every thread read this one's at the loop
    // top, and the barriers below publish it before the flush decision
    if (lastw && lane == 0) {
      copy_async_wait();
      int sn = sh.scene_q[par ^ 1], left = sh.unit_left;
      int4 itn = sh.item_q[par ^ 1];
      if (left <= 0 && un < total) {
        left = unit_at(un, sn, itn);
        if (left == 0) un = next_unit((int)gridDim.x + atomicAdd(counter, 1), sn, itn, left);
      }
      sh.unit_left = left - 1;
      const bool same = un == u + 1 && sn == s && itn.x == it.x;  // (single items of a block may also come one after the other)
      sh.item_q[par ^ 1] = itn;
      sh.scene_q[par ^ 1] = sn;
      sh.index_q[par ^ 1] = un;
      sh.next_same = un < total && same ? 1 : 0;
      sh.next_issue = un < total && !same ? 1 : 0;
    }
    P2GStored stored;
    p2g_count<kP2gFull, true, WIDE>(sh, S, bx, by, bz, have, q, wn, nbase, sh.fscale, stored);
    __syncthreads();  // counts done; the particle buffer is read
    if (sh.abort | sh.pabort) {
      stage_abort(sh, S);  // a copy wait ran out: this item's particles keep their state, the CTA stops
      return;
    }
    if (lastw && sh.index_q[par ^ 1] < total) {
      const int4 nx = sh.item_q[par ^ 1];
      const SceneDev& N = scenes[sh.scene_q[par ^ 1]];
      particles_issue(sh, N, nx.y, min(nx.z, kItemMax), BINNED && particles_binned(N));
    }
    p2g_sum<kP2gFull, true, WIDE>(sh, S, bx, by, bz, stored, wn);
    if (sh.next_issue) {  // uniform across the CTA
      const SceneDev& N = scenes[sh.scene_q[par ^ 1]];
      stage_issue<kOutFields>(sh, N, N.gout, sh.item_q[par ^ 1].x);
    }
    if (threadIdx.x == 0) {  // only maxima above what this CTA already recorded go to HBM
      unsigned* cur[3] = {&S.fix->m_cur, &S.fix->v_cur, &S.fix->a_cur};
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (sh.seen[k] > sh.pushed[k]) {
          atomicMax(cur[k], sh.seen[k]);
          sh.pushed[k] = sh.seen[k];
        }
    }
    const bool cont = sh.next_same != 0;  // uniform across the CTA
    if (!cont) p2g_tile_flush<kP2gFull, true>(sh, S, bx, by, bz);
    run_start = !cont;
  }
}

// Bulk statistics: per-thread sums in FP32 over a dozen particles, then FP64
// across threads (FP64 arithmetic is slow on this part: the per-particle work
// stays in FP32).
__global__ void __launch_bounds__(kStatsThreads) k_stats(const SceneDev* __restrict__ sd, int n, StatsSlot* slot,
                                               StatsAccum* host) {
  const SceneDev& S = *sd;
  float acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  StatsPartial t;
  stats_init(t);
  // four particles per thread and pass, their loads issued together
  constexpr int U = 4;
  const int stride = gridDim.x * blockDim.x;
  for (int p0 = blockIdx.x * blockDim.x + threadIdx.x; p0 < n; p0 += U * stride) {
    float4 xm[U], vv[U];
    float jp[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int p = p0 + u * stride;
      if (p < n) {
        xm[u] = S.xm[p];
        vv[u] = S.vv[p];
        jp[u] = S.fc[p].y;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (p0 + u * stride >= n) break;
      const float m = xm[u].w;
      const bool ok = isfinite(xm[u].x) && isfinite(xm[u].y) && isfinite(xm[u].z) && isfinite(vv[u].x) &&
                      isfinite(vv[u].y) && isfinite(vv[u].z) && isfinite(jp[u]);
      if (!ok) {
        t.bad++;
        continue;
      }
      acc[0] += m;
      acc[1] += m * vv[u].x;
      acc[2] += m * vv[u].y;
      acc[3] += m * vv[u].z;
      acc[4] += 0.5f * m * (vv[u].x * vv[u].x + vv[u].y * vv[u].y + vv[u].z * vv[u].z);
      acc[5] += m * xm[u].x;
      acc[6] += m * xm[u].y;
      acc[7] += m * xm[u].z;
      acc[8] += jp[u];
      t.bmin[0] = fminf(t.bmin[0], xm[u].x); t.bmin[1] = fminf(t.bmin[1], xm[u].y); t.bmin[2] = fminf(t.bmin[2], xm[u].z);
      t.bmax[0] = fmaxf(t.bmax[0], xm[u].x); t.bmax[1] = fmaxf(t.bmax[1], xm[u].y); t.bmax[2] = fmaxf(t.bmax[2], xm[u].z);
    }
  }
#pragma unroll
  for (int k = 0; k < 9; k++) t.acc[k] = acc[k];
  stats_commit(t, slot, host);
}

// Upload: the caller's arrays (x, v: N x 3; m: N; FE, FP: N x 9 row-major or
// null for identity), in device or page-locked host memory, packed into the
// particle streams. J_p = det F_P in double without contraction, as the
// host formerly computed it. Bound by the CPU-GPU link (210 GB/s for reads in
// whole lines): a block's stretch of every array is read by consecutive threads
// into shared memory and picked up there per particle; each thread reading its
// own particle's 12 and 36 bytes reached 168 GB/s (624 us for 1M particles with
// F_E and F_P, now 505).
constexpr int kIoTile = 256;  // particles per block and turn
// Words [0, n) of src, which starts at any 4-byte boundary, by all threads.
__device__ __forceinline__ void io_read(float* dst, const float* __restrict__ src, int n) {
  for (int k = threadIdx.x; k < n; k += kIoTile) dst[k] = __ldcs(src + k);
}
__global__ void __launch_bounds__(kIoTile) k_pack(const float* __restrict__ x, const float* __restrict__ v,
                                                  const float* __restrict__ m, const float* __restrict__ FE,
                                                  const float* __restrict__ FP, size_t n, float4* xm, float4* vv,
                                                  float4* fa, float4* fb, float2* fc, uint32_t* pid, float4* vq) {
  __shared__ float sx[3 * kIoTile], sv[3 * kIoTile], sm[kIoTile], se[9 * kIoTile], sp[9 * kIoTile];
  for (size_t i0 = blockIdx.x * (size_t)kIoTile; i0 < n; i0 += (size_t)gridDim.x * kIoTile) {
    const int cnt = (int)min((size_t)kIoTile, n - i0);
    io_read(sx, x + 3 * i0, 3 * cnt);
    io_read(sv, v + 3 * i0, 3 * cnt);
    io_read(sm, m + i0, cnt);
    if (FE) io_read(se, FE + 9 * i0, 9 * cnt);
    if (FP) io_read(sp, FP + 9 * i0, 9 * cnt);
    __syncthreads();
    const int k = threadIdx.x;
    if (k < cnt) {
      const size_t i = i0 + k;
      xm[i] = make_float4(sx[3 * k], sx[3 * k + 1], sx[3 * k + 2], sm[k]);
      vv[i] = make_float4(sv[3 * k], sv[3 * k + 1], sv[3 * k + 2], 0.0f);
      float F[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
      if (FE)
#pragma unroll
        for (int c = 0; c < 9; c++) F[c] = se[9 * k + c];
      fa[i] = make_float4(F[0], F[3], F[6], F[1]);
      fb[i] = make_float4(F[4], F[7], F[2], F[5]);
      float jp = 1.0f;
      if (FP) {
        const float* f = sp + 9 * k;
        const double a = f[0], b = f[1], c = f[2], d = f[3], e = f[4], g = f[5], h = f[6], ii = f[7], j = f[8];
        const double t0 = __dsub_rn(__dmul_rn(e, j), __dmul_rn(g, ii));
        const double t1 = __dsub_rn(__dmul_rn(d, j), __dmul_rn(g, h));
        const double t2 = __dsub_rn(__dmul_rn(d, ii), __dmul_rn(e, h));
        jp = (float)__dadd_rn(__dsub_rn(__dmul_rn(a, t0), __dmul_rn(b, t1)), __dmul_rn(c, t2));
      }
      fc[i] = make_float2(F[8], jp);
      pid[i] = (uint32_t)i;
      vq[i] = make_float4(1.0f, 0.0f, 0.0f, 0.0f);  // no previous SVD: identity frame
    }
    __syncthreads();
  }
}

// Download: the particle streams back to the caller's layout and order (slot i
// holds upload index pid[i]); any output may be null, and each lies in device or
// page-locked host memory. k_invert finds the slot of every upload index; a
// block then gathers its stretch of upload indices into shared memory and
// writes it out by consecutive threads, which fills whole lines of the CPU-GPU
// link (190 GB/s, what a DMA reaches), so that pinned arrays are written in
// place: 374 us for 1M particles instead of 107 for unpacking to a staging
// buffer and 386 for five copies; a viewer's frame of 4k particles 79 to 60 us.
__global__ void __launch_bounds__(256) k_invert(const SceneDev* __restrict__ sd, size_t n, uint32_t* slot) {
  chain_next();
  const SceneDev& S = *sd;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t j = S.pid[i];
    if (j < n) slot[j] = (uint32_t)i;  // (always: pid is a permutation)
  }
}
__device__ __forceinline__ void io_write(float* dst, const float* src, int n) {
  if (!dst) return;
  for (int k = threadIdx.x; k < n; k += kIoTile) __stcs(dst + k, src[k]);
}
__global__ void __launch_bounds__(kIoTile) k_unpack(const SceneDev* __restrict__ sd, size_t n,
                                                    const uint32_t* slot, float* x, float* v, float* FE,
                                                    float* Jp, float* volume) {
  chain_wait();
  const SceneDev& S = *sd;
  __shared__ float sx[3 * kIoTile], sv[3 * kIoTile], se[9 * kIoTile], sj[kIoTile], so[kIoTile];
  for (size_t j0 = blockIdx.x * (size_t)kIoTile; j0 < n; j0 += (size_t)gridDim.x * kIoTile) {
    const int cnt = (int)min((size_t)kIoTile, n - j0);
    const int k = threadIdx.x;
    if (k < cnt) {
      const uint32_t i = slot[j0 + k];
      if (x) {
        const float4 xm = S.xm[i];
        sx[3 * k] = xm.x;
        sx[3 * k + 1] = xm.y;
        sx[3 * k + 2] = xm.z;
      }
      if (v || volume) {
        const float4 vv = S.vv[i];
        sv[3 * k] = vv.x;
        sv[3 * k + 1] = vv.y;
        sv[3 * k + 2] = vv.z;
        so[k] = vv.w;
      }
      if (FE || Jp) {
        const float2 c = S.fc[i];
        sj[k] = c.y;
        if (FE) {
          // fa = (m00, m01, m02, m10), fb = (m11, m12, m20, m21), fc = (m22, Jp); m[c][r]
          const float4 a = S.fa[i], b = S.fb[i];
          const float mcr[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x};
#pragma unroll
          for (int r = 0; r < 3; r++)
#pragma unroll
            for (int q = 0; q < 3; q++) se[9 * k + 3 * r + q] = mcr[3 * q + r];
        }
      }
    }
    __syncthreads();
    io_write(x ? x + 3 * j0 : nullptr, sx, 3 * cnt);
    io_write(v ? v + 3 * j0 : nullptr, sv, 3 * cnt);
    io_write(FE ? FE + 9 * j0 : nullptr, se, 9 * cnt);
    io_write(Jp ? Jp + j0 : nullptr, sj, cnt);
    io_write(volume ? volume + j0 : nullptr, so, cnt);
    __syncthreads();
  }
}

// Dense copies of the P2G sums (acc) and of v* of the active blocks.
__global__ void k_download_grid(const SceneDev* __restrict__ sd, float* mass, float* mom, float* force, float* vstar) {
  const SceneDev& S = *sd;
  const int count = min(S.counters[CNT_ACTIVE], S.pool_cap);
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < (long long)count * kBlockNodes;
       u += (long long)gridDim.x * blockDim.x) {
    const int slot = (int)(u / kBlockNodes), node = (int)(u % kBlockNodes);
    const int b = S.active[slot];
    const int bx = b % S.bdim[0], by = (b / S.bdim[0]) % S.bdim[1], bz = b / (S.bdim[0] * S.bdim[1]);
    const int gi = 4 * bx + (node & 3), gj = 4 * by + ((node >> 2) & 3), gk = 4 * bz + (node >> 4);
    if (gi >= S.dim[0] || gj >= S.dim[1] || gk >= S.dim[2]) continue;
    const long long g = gi + (long long)S.dim[0] * (gj + (long long)S.dim[1] * gk);
    const float* out = S.gout + node_index(S, gi, gj, gk) * kOutFields;
    if (vstar)
      for (int k = 0; k < 3; k++) vstar[3 * g + k] = out[k];
  }
  // acc is dense: every block, every node
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
       g < (long long)S.dim[0] * S.dim[1] * S.dim[2]; g += (long long)gridDim.x * blockDim.x) {
    const int gi = (int)(g % S.dim[0]), gj = (int)((g / S.dim[0]) % S.dim[1]),
              gk = (int)(g / ((long long)S.dim[0] * S.dim[1]));
    const int blk = block_id(S, gi >> 2, gj >> 2, gk >> 2);
    const unsigned long long* acc = S.acc + (size_t)blk * kAccBlockWords + (gi & 3) + 4 * (gj & 3) + 16 * (gk & 3);
    const FixState& fx = *S.fix;
    if (mass) mass[g] = (float)(long long)acc[0] / fx.scale[0];
    for (int k = 0; k < 3; k++) {
      if (mom) mom[3 * g + k] = (float)(long long)acc[(1 + k) * kBlockNodes] / fx.scale[1];
      if (force) force[3 * g + k] = (float)(long long)acc[(4 + k) * kBlockNodes] / fx.scale[2];
    }
  }
}

template <class K>
void smem_opt_in(K kernel, int bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Shared-memory opt-in of the work-item kernels, once per device (the
// attribute belongs to the function in each device's context).
int item_smem() {
  static bool configured[kMaxDevices] = {};
  const int bytes = (int)sizeof(ItemShared);
  const int dev = current_device();
  if (!configured[dev]) {
    smem_opt_in(k_p2g<true>, bytes);
    smem_opt_in(k_p2g<false>, bytes);
    smem_opt_in(k_g2p_advance, bytes);
    smem_opt_in(k_g2p2g<false, false>, bytes);
    smem_opt_in(k_g2p2g<true, false>, bytes);
    smem_opt_in(k_g2p2g<true, true>, bytes);
    configured[dev] = true;
  }
  return bytes;
}

}  // namespace

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  return dev;
}

// SM count of the current device (cached per device: launch grids are sized
// for the GPU the launch goes to).
int num_sms() {
  static int n[kMaxDevices] = {};
  const int dev = current_device();
  if (n[dev] == 0) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n[dev] = v > 0 ? v : 1;
  }
  return n[dev];
}


void fast_rigid(const SceneDev* sd_dev, cudaStream_t st) { k_rigid<<<1, 32, 0, st>>>(sd_dev); }

void fast_gather_counters(const SceneDev* scenes, int nscenes, int* out, cudaStream_t st) {
  const int n = nscenes * kCounterStride;
  k_gather_counters<<<(n + 255) / 256, 256, 0, st>>>(scenes, nscenes, out);
}

void fast_compact(const WorkSpace& w, bool rigid, bool binned, bool chained, cudaStream_t st, bool set_up) {
  const long long g = std::max(1ll, (w.total_quads + kCompactThreads - 1) / kCompactThreads);
  const int begin_ctas = (w.nscenes + kCompactThreads / 32 - 1) / (kCompactThreads / 32);
  launch_after(chained, k_compact, (int)g + begin_ctas, kCompactThreads, 0, st, w.scenes, w.quads, w.nscenes,
               w.total_quads, w.items, w.active, rigid ? 1 : 0, binned ? 1 : 0, set_up ? 1 : 0);
}

void fast_p2g(const SceneDev* scenes, const SceneDev& sd_host, const int* item_prefix, int nscenes, int grid_ctas,
              bool mass_only, cudaStream_t st) {
  const int smem = item_smem();
  // the magnitudes of the particles, from which k_p2g chooses its scales
  cudaMemsetAsync(&sd_host.fix->m_prev, 0, offsetof(FixState, wide) - offsetof(FixState, m_prev), st);
  if (sd_host.n > 0) {
    int g = (sd_host.n + 255) / 256;
    if (g > num_sms() * 8) g = num_sms() * 8;
    k_fix_measure<<<g, 256, 0, st>>>(scenes, mass_only ? 0 : 1);
  }
  if (mass_only)
    k_p2g<true><<<grid_ctas, kItemMax, smem, st>>>(scenes, item_prefix, nscenes);
  else
    k_p2g<false><<<grid_ctas, kItemMax, smem, st>>>(scenes, item_prefix, nscenes);
}

void fast_grid(const SceneDev* scenes, const int* active_prefix, int nscenes, int grid_ctas, bool clear_only,
               bool chained, cudaStream_t st) {
  launch_after(chained, k_grid, grid_ctas, kGridGroups * kBlockNodes, 0, st, scenes, active_prefix, nscenes,
               clear_only ? 1 : 0);
}

void fast_volume(const SceneDev* sd_dev, const int* item_prefix, int n, cudaStream_t st) {
  if (n <= 0) return;
  const int g = std::min(n / 32 + 1, num_sms() * 8);
  k_volume<<<g, 256, 0, st>>>(sd_dev, item_prefix);
}

void fast_g2p_advance(const SceneDev* scenes, const int* item_prefix, int nscenes, int grid_ctas, cudaStream_t st) {
  k_g2p_advance<<<grid_ctas, kItemMax, item_smem(), st>>>(scenes, item_prefix, nscenes);
}

void fast_g2p2g(const SceneDev* scenes, const int* item_prefix, int nscenes, int grid_ctas, bool binned,
                bool wide, bool chained, cudaStream_t st) {
  launch_after(chained, wide ? k_g2p2g<true, true> : binned ? k_g2p2g<true, false> : k_g2p2g<false, false>, grid_ctas,
               kItemMax, item_smem(), st, scenes, item_prefix, nscenes);
}

void fast_stats(const SceneDev* sd_dev, int n, StatsSlot* slot, StatsAccum* host, cudaStream_t st) {
  int g = (n + kStatsThreads - 1) / kStatsThreads;  // at least one block: it publishes the empty sums
  if (g > num_sms()) g = num_sms();  // one block per SM: measured fastest (fixed costs dominate)
  if (g > kStatsMaxBlocks) g = kStatsMaxBlocks;
  if (g < 1) g = 1;
  k_stats<<<g, kStatsThreads, 0, st>>>(sd_dev, n < 0 ? 0 : n, slot, host);
}


void fast_pack(const float* x, const float* v, const float* m, const float* FE, const float* FP, size_t n,
               const SceneDev& sd, cudaStream_t st) {
  if (n == 0) return;
  const size_t g = std::min((n + kIoTile - 1) / kIoTile, (size_t)num_sms() * 8);
  k_pack<<<(int)g, kIoTile, 0, st>>>(x, v, m, FE, FP, n, sd.xm, sd.vv, sd.fa, sd.fb, sd.fc, sd.pid, sd.vq);
}

void fast_unpack(const SceneDev* sd_dev, size_t n, uint32_t* slot, float* x, float* v, float* FE, float* Jp,
                 float* volume, cudaStream_t st) {
  if (n == 0) return;
  const size_t g = std::min((n + kIoTile - 1) / kIoTile, (size_t)num_sms() * 8);
  k_invert<<<(int)g, 256, 0, st>>>(sd_dev, n, slot);
  // (chained: the positions of 4k particles to pageable memory took 26.5 us with one
  // kernel, 30.8 with two, 24.6 now)
  launch_after(true, k_unpack, (int)g, kIoTile, 0, st, sd_dev, n, slot, x, v, FE, Jp, volume);
}

void fast_download_grid(const SceneDev* sd_dev, float* mass, float* mom, float* force, float* vstar,
                        cudaStream_t st) {
  k_download_grid<<<num_sms() * 8, 256, 0, st>>>(sd_dev, mass, mom, force, vstar);
}

}  // namespace snow
