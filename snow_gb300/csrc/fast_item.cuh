// Device helpers of the FAST path shared by its kernel files
// (fast_kernels.cu: the explicit step; implicit.cu: the semi-implicit
// velocity solve): B-spline weights, colliders, the P2G quantities of a
// particle, the shared memory of a work item with its bulk copies (TMA) of
// grid rows and particles, the G2P gather, the particle advance and the P2G tile pass.
#pragma once
#include "snow_internal.h"
#include "snow_math.cuh"
#include "snow_tma.cuh"

namespace snow {
namespace {

constexpr int kTile = 9;  // tile nodes per axis: [4b-2, 4b+6]
constexpr int kTile3 = kTile * kTile * kTile;
// A work item holds up to kItemMax particles (one per thread) binned to one home block b. A
// particle whose base cell lies in [4b-1, 4b+4] (the home block plus one
// cell of drift each way) has its whole stencil inside the tile; its base
// cell has tile-local coordinates lc = base - (4b-2) - 1 in [0, 5]^3.
// What a P2G tile pass accumulates: the grid mass alone (gMassCompute.glsl),
// mass, momentum and stress force (p2gTransfer.glsl), or only a force-like
// 3-vector per node (the semi-implicit solve's K u, into the force slots).
enum P2gKind { kP2gMass = 0, kP2gFull = 1, kP2gForce = 2 };
template <int KIND> struct P2gFields {
  static constexpr int nf = KIND == kP2gMass ? 1 : (KIND == kP2gFull ? kAccFields : 3);
  static constexpr int acc_first = KIND == kP2gForce ? 4 : 0;  // first acc field written
};
constexpr int kCellsPerAxis = kTile - 3;  // 6
constexpr int kCells = kCellsPerAxis * kCellsPerAxis * kCellsPerAxis;
// P2G data in shared memory: two particles share one record, their values
// interleaved word by word (first particle's in the even word), so that a
// 16-byte load fills two operand pairs of the packed FP32 instructions and one
// instruction serves both particles. Order of the 38 pairs: A22, m, mv (3),
// A00, A01, A02, A10, A11, A12, A20, A21, unused, wx[4], gx[4], (wy, gy)[4],
// (wz, gz)[4].
constexpr int kPdPairs = 38;
constexpr int kPdStride = 2 * kPdPairs;  // words per record (304 bytes: 16-byte loads stay aligned)
enum { kPdA22 = 0, kPdM = 1, kPdMv = 2, kPdA = 5, kPdWx = 14, kPdGx = 18, kPdY = 22, kPdZ = 30 };
constexpr int kShColliders = 16;  // colliders cached in shared memory

__device__ __forceinline__ int find_scene(const int* prefix, int nscenes, long long u) {
  int lo = 0, hi = nscenes;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((long long)prefix[mid] <= u)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ float sel4(int i, float a0, float a1, float a2, float a3) {
  return i == 0 ? a0 : (i == 1 ? a1 : (i == 2 ? a2 : a3));
}

// ---- packed FP32 pairs -----------------------------------------------------
// Two floats in one 64-bit register pair; each half rounds as the scalar
// instruction does.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, unsigned& lo, unsigned& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float lo2(f32x2 v) {
  unsigned a, b;
  unpack2(v, a, b);
  return __uint_as_float(a);
}
__device__ __forceinline__ float hi2(f32x2 v) {
  unsigned a, b;
  unpack2(v, a, b);
  return __uint_as_float(b);
}

// Axis weights of the 4 stencil nodes base-1 .. base+2 (cubic.include.glsl):
// w[a] = N(d_a), g[a] = N'(-d_a) with d_a = node - x/h, as the shaders
// evaluate weighting(d) and weightingGradient(-d).
__device__ __forceinline__ void axis_weights_general(float pg, int base, float w[4], float g[4]) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const float d = (float)(base + a - 1) - pg;
    w[a] = bspline(d);
    g[a] = bspline_d(-d);
  }
}

// The same weights without branches for pg >= 0, where base = floor(pg) and
// f = pg - base is in [0, 1): the stencil distances are |d| = 1+f, f, 1-f,
// 2-f, each on a known piece of the spline. With u = 1 - f:
//   w = (u^3/6, f^3/2 - f^2 + 2/3, u^3/2 - u^2 + 2/3, f^3/6)
//   g = (-u^2/2, 3f^2/2 - 2f, -3u^2/2 + 2u, f^2/2)
// Particles below the grid origin (pg < 0, truncated toward zero) take the
// general path.
__device__ __forceinline__ void axis_weights(float pg, int base, float w[4], float g[4]) {
  if (pg < 0.0f) {
    axis_weights_general(pg, base, w, g);
    return;
  }
  const float f = pg - (float)base;
  const float u = 1.0f - f;
  const float f2 = f * f, u2 = u * u;
  const float f3 = f2 * f, u3 = u2 * u;
  w[0] = u3 * (1.0f / 6.0f);
  w[1] = 0.5f * f3 - f2 + 2.0f / 3.0f;
  w[2] = 0.5f * u3 - u2 + 2.0f / 3.0f;
  w[3] = f3 * (1.0f / 6.0f);
  g[0] = -0.5f * u2;
  g[1] = 1.5f * f2 - 2.0f * f;
  g[2] = -1.5f * u2 + 2.0f * u;
  g[3] = 0.5f * f2;
}

struct AxisW {
  float wx[4], gx[4], wy[4], gy[4], wz[4], gz[4];
};

// Grid coordinates (x - gGridPos) / h. Multiplying by 1/h can move a value
// by an ulp against the shaders' division; at a cell boundary that only
// swaps which stencil end carries the (zero) weight, so the sums agree.
__device__ __forceinline__ void grid_coords(const SceneDev& S, float4 xm, float pg[3], int base[3]) {
  pg[0] = (xm.x - S.gpos[0]) * S.inv_h;
  pg[1] = (xm.y - S.gpos[1]) * S.inv_h;
  pg[2] = (xm.z - S.gpos[2]) * S.inv_h;
#pragma unroll
  for (int k = 0; k < 3; k++) base[k] = (int)pg[k];  // ivec3(): truncation toward zero
}

__device__ __forceinline__ void all_weights(const float pg[3], const int base[3], AxisW& w) {
  axis_weights(pg[0], base[0], w.wx, w.gx);
  axis_weights(pg[1], base[1], w.wy, w.gy);
  axis_weights(pg[2], base[2], w.wz, w.gz);
}

// Whether this step's binning left the particles in the binned copies.
__device__ __forceinline__ bool particles_binned(const SceneDev& S) { return S.counters[CNT_BINNED] != 0; }

__device__ __forceinline__ void load_fe(const SceneDev& S, int p, M3& F, float& jp, bool binned = false) {
  const float4 a = (binned ? S.bfa : S.fa)[p];
  const float4 b = (binned ? S.bfb : S.fb)[p];
  const float2 c = (binned ? S.bfc : S.fc)[p];
  F.m[0][0] = a.x; F.m[0][1] = a.y; F.m[0][2] = a.z;
  F.m[1][0] = a.w; F.m[1][1] = b.x; F.m[1][2] = b.y;
  F.m[2][0] = b.z; F.m[2][1] = b.w; F.m[2][2] = c.x;
  jp = c.y;
}
__device__ __forceinline__ void store_fe(const SceneDev& S, int p, const M3& F, float jp) {
  __stcs(&S.fa[p], make_float4(F.m[0][0], F.m[0][1], F.m[0][2], F.m[1][0]));
  __stcs(&S.fb[p], make_float4(F.m[1][1], F.m[1][2], F.m[2][0], F.m[2][1]));
  __stcs(&S.fc[p], make_float2(F.m[2][2], jp));
}

__device__ __forceinline__ int block_id(const SceneDev& S, int bx, int by, int bz) {
  return (bz * S.bdim[1] + by) * S.bdim[0] + bx;
}

__device__ __forceinline__ bool node_in_grid(const SceneDev& S, int g0, int g1, int g2) {
  return g0 >= 0 && g1 >= 0 && g2 >= 0 && g0 < S.dim[0] && g1 < S.dim[1] && g2 < S.dim[2];
}

// Collider projection of gForceCompute.glsl:72-93 / particleAdvance.glsl:182-204
// for one collider that the point x hits: the velocity relative to the
// collider loses its normal inward part, with Coulomb friction.
__device__ __forceinline__ void collide_hit(const snow_collider& c, const float x[3], float v[3]) {
  float n[3] = {c.normal[0], c.normal[1], c.normal[2]};
  if (c.type == 1) {
    const float d[3] = {x[0] - c.pos[0], x[1] - c.pos[1], x[2] - c.pos[2]};
    const float len = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    n[0] = d[0] / len;
    n[1] = d[1] / len;
    n[2] = d[2] / len;
  }
  const float vrel[3] = {v[0] - c.vel[0], v[1] - c.vel[1], v[2] - c.vel[2]};
  const float vn = vrel[0] * n[0] + vrel[1] * n[1] + vrel[2] * n[2];
  if (vn < 0.0f) {
    const float vt[3] = {vrel[0] - n[0] * vn, vrel[1] - n[1] * vn, vrel[2] - n[2] * vn};
    const float muvn = c.friction * vn;
    const float lvt = sqrtf(vt[0] * vt[0] + vt[1] * vt[1] + vt[2] * vt[2]);
    if (lvt <= -muvn) {
      v[0] = c.vel[0];
      v[1] = c.vel[1];
      v[2] = c.vel[2];
    } else {
      const float s = muvn / lvt;
#pragma unroll
      for (int k = 0; k < 3; k++) v[k] = vt[k] + s * vt[k] + c.vel[k];
    }
  }
}

// All colliders in order (half-plane: dot(x - c, n) <= 0; sphere: |x - c| < r).
// A record is three 16-byte words, (pos, type), (vel, radius), (normal,
// friction): the test reads the first and the one it needs, the projection
// the whole record, only for a hit.
__device__ __forceinline__ void collide(const snow_collider* coll, int ncoll, const float x[3], float v[3]) {
  static_assert(sizeof(snow_collider) == 48, "three 16-byte words per collider");
  for (int i = 0; i < ncoll; i++) {
    const float4* c4 = reinterpret_cast<const float4*>(coll + i);
    const float4 a = c4[0];
    const int type = __float_as_int(a.w);
    bool hit = false;
    if (type == 0) {
      const float4 nf = c4[2];
      hit = (x[0] - a.x) * nf.x + (x[1] - a.y) * nf.y + (x[2] - a.z) * nf.z <= 0.0f;
    } else if (type == 1) {
      const float r = c4[1].w;
      const float d[3] = {x[0] - a.x, x[1] - a.y, x[2] - a.z};
      hit = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) < r;
    }
    if (hit) collide_hit(coll[i], x, v);
  }
}

// The same with the hit tests on a packed form of the colliders (half-plane:
// (n, n . c), tested as n . x <= n . c; sphere: (c, r^2), tested as
// |x - c|^2 < r^2): one 16-byte shared load per collider, the full record
// only for the rare hit.
__device__ __forceinline__ void collide_packed(const snow_collider* coll, const float4* hitf, const int* type,
                                               int ncoll, const float x[3], float v[3]) {
  for (int i = 0; i < ncoll; i++) {
    const float4 h = hitf[i];
    const int t = type[i];
    bool hit = false;
    if (t == 0) {
      hit = fmaf(h.z, x[2], fmaf(h.y, x[1], h.x * x[0])) <= h.w;
    } else if (t == 1) {
      const float d0 = x[0] - h.x, d1 = x[1] - h.y, d2 = x[2] - h.z;
      hit = fmaf(d2, d2, fmaf(d1, d1, d0 * d0)) < h.w;
    }
    if (hit) collide_hit(coll[i], x, v);
  }
}

// ---- fixed-point P2G sums ------------------------------------------------------
// Every contribution of a particle to a grid node (mass m w, momentum m v w,
// force A grad w) is rounded to an integer at a per-scene power-of-two scale
// (s_m, s_p, s_f), and integers are summed: in registers and in the shared
// tile as int32 (modulo 2^32; each particle adds a bound of its largest
// contribution to its item, and a tile is added to acc before the bounds of
// the particles it holds could reach 2^31, so its sums never wrap), into
// acc as int64. Integer sums do not depend on the
// order in which they are formed, so the grid a particle state produces does
// not depend on how particles are grouped into work items, on the binning
// schedule, on CTA scheduling or on the other scenes of a batch. The rounding
// of one contribution is the same on every path that forms it: the tile path
// and the per-node scatter of a particle outside its work item's tile both
// compute it with the same pinned (_rn) operations.
//
// A contribution y (|y| < 2^22 after scaling) is rounded by one FMA against
// kMagic = 1.5 * 2^23: fma(w, x, kMagic) lies in [2^23, 2^24), where floats
// are spaced by 1, so its bits minus kMagicBits are round(w x). A force
// contribution g_x kk + w_x hh is rounded as round(g_x kk + round(w_x hh));
// with a = max over rows r of |A_r0| + |A_r1| + |A_r2|, both terms and their
// sum are at most a (2/3)^3 s_f. The mass scale puts the largest
// contribution near 2^21; the momentum and force scales put bounds that
// already carry a growth margin (1.25 max|v| + margins, twice the largest
// stress term) into [2^21, 2^22), the fast range's limit. A particle whose
// contributions reach the limit (it outgrew the magnitudes the scales were
// chosen from) is scattered with exactly rounded int64 contributions ("wide"),
// which depends only on the particle itself, so it is
// as deterministic.
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kMagicBits = 0x4B400000;
constexpr float kWmax = 0.2962963f;       // (2/3)^3 >= any weight or weight-gradient product
constexpr float kFastLimit = 4190208.0f;       // 2^22 (1 - 2^-11): bound of a fast-path contribution
constexpr float kTileSumBound = 2126008832.0f;  // 0.99 * 2^31: bound of a tile's sums of contribution bounds

// The largest power of two s with x s <= 2^bits (1 for x <= 0 or not finite).
__device__ __forceinline__ float pow2_scale(float x, int bits) {
  if (!(x > 0.0f) || !isfinite(x)) return 1.0f;
  int e;
  frexpf(x, &e);  // x = f 2^e, f in [0.5, 1): x 2^(bits - e) in [2^(bits-1), 2^bits)
  return ldexpf(1.0f, max(-126, min(127, bits - e)));
}

struct FixScale {
  float m, p, f;
};

__device__ __forceinline__ float bits_float(uint32_t b) { return __uint_as_float(b); }

// Scales of a P2G that follows a grid update in the same step (the fused
// kernel): from the magnitudes of the particles the previous P2G scattered
// (FixState::*_prev). The momentum scale allows particle speeds up to
// 1.25 max|v_p| + 2 max|v_collider| + 2 |g| dt (a collider projection adds
// at most twice the collider's speed; the last term keeps the scale finite
// for a scene at rest, which gravity moves by |g| dt a step).
// It is taken from particle speeds alone: v* = p/m + dt (f/m + g) of a node
// that holds a sliver of mass can exceed every particle's speed by orders of
// magnitude, while the G2P weights such a node by as small a sliver. The
// force scale allows twice the previous largest stress term (the floor
// 1e-9 E0 V0max keeps it finite for a scene without stress). A particle
// beyond either takes the wide path.
__device__ __forceinline__ FixScale step_scales(const SceneDev& S) {
  const FixState& f = *S.fix;
  const float mmax = bits_float(f.m_prev);
  float vcoll = 0.0f;
  for (int i = 0; i < S.ncoll; i++) {
    const float* cv = S.coll[i].vel;
    vcoll = fmaxf(vcoll, sqrtf(cv[0] * cv[0] + cv[1] * cv[1] + cv[2] * cv[2]));
  }
  const float g = sqrtf(S.grav[0] * S.grav[0] + S.grav[1] * S.grav[1] + S.grav[2] * S.grav[2]);
  const float vb = 1.25f * bits_float(f.v_prev) + 2.0f * vcoll + 2.0f * g * S.dt;
  const float afloor = 1e-9f * S.young * bits_float(f.v0max);
  FixScale sc;
  sc.m = pow2_scale(mmax * kWmax, 21);
  sc.p = pow2_scale(mmax * vb * kWmax, 22);
  sc.f = pow2_scale(fmaxf(2.0f * bits_float(f.a_prev), afloor) * kWmax, 22);
  return sc;
}

// Scales of a P2G of the stored state (set-up, per-kernel dispatches): from
// the exact magnitudes a pass over the particles just measured (k_fix_measure).
__device__ __forceinline__ FixScale measured_scales(const SceneDev& S) {
  const FixState& f = *S.fix;
  const float mmax = bits_float(f.m_prev);
  const float afloor = 1e-9f * S.young * bits_float(f.v0max);
  FixScale sc;
  sc.m = pow2_scale(mmax * kWmax, 21);
  sc.p = pow2_scale(mmax * bits_float(f.v_prev) * kWmax, 22);
  sc.f = pow2_scale(fmaxf(bits_float(f.a_prev), afloor) * kWmax, 22);
  return sc;
}

// Adds one node's integer sums v[0..6] (m, p, f; mass_only: v[0]) into acc
// (two's complement adds: a sum of int64 values, whatever the order).
__device__ __forceinline__ void acc_add(const SceneDev& S, int blk, int node, const long long v[7], bool mass_only) {
  unsigned long long* a = S.acc + (size_t)blk * kAccBlockWords + node;
  const int nw = mass_only ? 1 : kAccWords;
  for (int f = 0; f < nw; f++)
    if (v[f]) atomicAdd(a + f * kBlockNodes, (unsigned long long)v[f]);
}

// ---- P2G quantities of one particle -----------------------------------------
__device__ __forceinline__ float max_nan(float a, float b) {  // (fmaxf drops NaN)
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// mass, momentum and A = -V0 * stress, stress = 2 mu(Jp) (FE - R) FE^T +
// lambda(Jp) (JE - 1) JE I with R the polar rotation of FE
// (p2gTransfer.glsl:109-141); V0 = m / rho0. `a` = max over rows r of
// |A_r0| + |A_r1| + |A_r2| bounds a force contribution and both its terms
// (in units of the weight products' bound (2/3)^3); NaN if any term is.
struct P2GParticle {
  float m, mv[3];
  float A[3][3];  // A[r][c]
  float a;
  bool force;
};

__device__ __forceinline__ void p2g_stress(const SceneDev& S, const M3& F, const M3& R, float jp, float vol,
                                           P2GParticle& q) {
  const float je = m3_det(F);
  const float e = expf(S.hardening * (1.0f - jp));
  const float mu = S.mu0 * e;
  const float lam = S.lambda0 * e;
  M3 D;
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int r = 0; r < 3; r++) D.m[c][r] = F.m[c][r] - R.m[c][r];
  const M3 P = m3_mul_bt(D, F);  // (FE - R) FE^T
  const float s2 = lam * (je - 1.0f) * je;
  float a = 0.0f;
#pragma unroll
  for (int r = 0; r < 3; r++) {
#pragma unroll
    for (int c = 0; c < 3; c++) q.A[r][c] = -vol * (2.0f * mu * P.m[c][r] + (r == c ? s2 : 0.0f));
    a = max_nan(a, fabsf(q.A[r][0]) + fabsf(q.A[r][1]) + fabsf(q.A[r][2]));
  }
  q.a = a;
  q.force = true;
}

// From the stored state: R by an SVD of F_E.
__device__ __forceinline__ P2GParticle p2g_particle(const SceneDev& S, int p, float4 xm, bool mass_only) {
  P2GParticle q;
  q.m = xm.w;
  q.force = false;
  q.a = 0.0f;
  q.mv[0] = q.mv[1] = q.mv[2] = 0.0f;
  if (mass_only) return q;
  const float4 vv = S.vv[p];
  q.mv[0] = q.m * vv.x;
  q.mv[1] = q.m * vv.y;
  q.mv[2] = q.m * vv.z;
  if (vv.w > 0.0f) {
    M3 F;
    float jp;
    load_fe(S, p, F, jp);
    M3 W, Sg, V;
    svd3<false>(F, W, Sg, V);
    p2g_stress(S, F, m3_mul_bt(W, V), jp, vv.w, q);
  }
  return q;
}

// The largest magnitude any of the particle's scaled contributions (and
// contribution terms) can take at scales sc (KIND kP2gMass: the mass alone);
// not finite for a non-finite particle.
template <int KIND>
__device__ __forceinline__ float fix_bound(const P2GParticle& q, const FixScale& sc) {
  float b = fabsf(q.m) * sc.m;
  if (KIND == kP2gFull) {
    const float mv = max_nan(fabsf(q.mv[0]), max_nan(fabsf(q.mv[1]), fabsf(q.mv[2])));
    b = max_nan(b, mv * sc.p);
    if (q.force) b = max_nan(b, q.a * sc.f);
  }
  return b * kWmax;
}
// The size of a force-like particle's A (K u): not finite if any term is not.
__device__ __forceinline__ float force_size(const P2GParticle& q) {
  float sum = 0.0f;
#pragma unroll
  for (int r = 0; r < 3; r++) sum += fabsf(q.A[r][0]) + fabsf(q.A[r][1]) + fabsf(q.A[r][2]);
  return q.force ? sum : 0.0f;
}

// The per-lane factors of one particle's contributions in stencil row
// (b, c), the same operations on every path: t1 = wy wz, t2 = gy wz,
// t3 = wy gz; mw = m_s t1, pv = mv_s t1, kk = A_s[r][0] t1,
// hh = A_s[r][1] t2 + A_s[r][2] t3 (scaled quantities, _s).
struct RowFactors {
  float mw, pv[3], kk[3], hh[3];
};
__device__ __forceinline__ void row_factors(float ms, const float mvs[3], const float As[3][3], float wyb, float gyb,
                                            float wzc, float gzc, bool mass_only, RowFactors& f) {
  const float t1 = __fmul_rn(wyb, wzc);
  f.mw = __fmul_rn(ms, t1);
  if (mass_only) return;
  const float t2 = __fmul_rn(gyb, wzc), t3 = __fmul_rn(wyb, gzc);
#pragma unroll
  for (int r = 0; r < 3; r++) {
    f.pv[r] = __fmul_rn(mvs[r], t1);
    f.kk[r] = __fmul_rn(As[r][0], t1);
    f.hh[r] = __fmaf_rn(As[r][1], t2, __fmul_rn(As[r][2], t3));
  }
}
// Rounded contributions (as magic-offset bits) at node x-weights (wxa, gxa).
__device__ __forceinline__ int fix_mass(float wxa, const RowFactors& f) {
  return __float_as_int(__fmaf_rn(wxa, f.mw, kMagic));
}
__device__ __forceinline__ int fix_mom(float wxa, const RowFactors& f, int r) {
  return __float_as_int(__fmaf_rn(wxa, f.pv[r], kMagic));
}
__device__ __forceinline__ int fix_force(float wxa, float gxa, const RowFactors& f, int r) {
  return __float_as_int(__fmaf_rn(gxa, f.kk[r], __fmaf_rn(wxa, f.hh[r], kMagic)));
}

// round(a b + h) to an integer, ties to even, with one rounding, in integer
// arithmetic (a 24 x 24 bit product and a shift): this GPU's double precision is
// 64 times slower than its single. 0 for what is not finite or reaches 4e18.
__device__ __forceinline__ long long round_product(float a, float b, long long h) {
  const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
  const int xa = (int)(ua >> 23 & 255u), xb = (int)(ub >> 23 & 255u);
  if (xa == 255 || xb == 255) return 0;
  const uint32_t ma = (ua & 0x7fffffu) | (xa ? 0x800000u : 0u), mb = (ub & 0x7fffffu) | (xb ? 0x800000u : 0u);
  const unsigned long long p = (unsigned long long)ma * mb;
  const int e = max(xa, 1) + max(xb, 1) - 300;  // |a b| = p 2^e
  const bool neg = ((ua ^ ub) >> 31) != 0u;
  constexpr long long kLimit = 4000000000000000000ll;
  long long q;
  if (e >= 0) {
    if (p != 0 && (e > 62 || (p >> (62 - e)) != 0)) return 0;
    const long long v = e > 62 ? 0ll : (long long)(p << e);
    q = h + (neg ? -v : v);
  } else if (e <= -50) {
    q = h;  // below a quarter
  } else {
    const int s = -e;
    const long long t = neg ? -(long long)p : (long long)p;
    const long long fl = t >> s, rem = t - (fl << s), half = 1ll << (s - 1);
    q = h + fl;
    if (rem > half || (rem == half && (q & 1))) q++;
  }
  return q < kLimit && q > -kLimit ? q : 0;
}

// The same for finite a and b with |a b| < 2^46, without branches.
__device__ __forceinline__ long long round_bounded(float a, float b, long long h) {
  const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
  const int xa = (int)(ua >> 23 & 255u), xb = (int)(ub >> 23 & 255u);
  const uint32_t ma = (ua & 0x7fffffu) | (xa ? 0x800000u : 0u), mb = (ub & 0x7fffffu) | (xb ? 0x800000u : 0u);
  const long long p = (long long)((unsigned long long)ma * mb);
  const int s = min(300 - max(xa, 1) - max(xb, 1), 50);  // |a b| = p 2^-s, s > 0; rounds to 0 from 50 on
  const long long t = ((ua ^ ub) >> 31) != 0u ? -p : p;
  const long long odd = (h + (t >> s)) & 1;
  return h + ((t + (1ll << (s - 1)) - 1 + odd) >> s);
}

// Scatter of the 64 stencil nodes of a warp's particles that do not go to the
// tile straight into acc (global atomics), one particle at a time with two nodes
// per lane, whose words lie in whole sectors. FAR_FAST: the particle lies outside
// its work item's tile; its contributions are rounded exactly as the tile path
// rounds them. FAR_WIDE: it outgrew the fast path's range or is not finite; each
// contribution is rounded exactly to int64. K u (kP2gForce): float sums into the
// low 4 bytes of acc's force words (free between the grid update and the next
// P2G; the solve's node passes read and clear them), in active blocks alone.
// A thread per particle took the 448 atomics of each in turn, those of a cell's
// particles to the same words, and rounded the wide ones in double precision: 8
// steps of half a cell without a binning (300k particles) took 0.69 ms each, now
// 0.36; a step whose 131k particles are all wide 1.44, now 0.85.
enum { kFarNone = 0, kFarFast = 1, kFarWide = 2, kFarTile = 3 };
struct FarParticle {
  float wx[4], gx[4], wy[4], gy[4], wz[4], gz[4];
  float ms, mvs[3], As[9];
  int base[3];
};
template <int KIND>
__device__ __noinline__ void scatter_far(const SceneDev& S, const FarParticle& f, int kind) {
  constexpr bool mo = KIND == kP2gMass;
  const int lane = threadIdx.x & 31;
  float As[3][3];
#pragma unroll
  for (int k = 0; k < 9; k++) As[k / 3][k % 3] = f.As[k];
  const int a = lane & 3, b = (lane >> 2) & 3;
  const float wxa = f.wx[a], gxa = f.gx[a], wyb = f.wy[b], gyb = f.gy[b];
  const int g0 = f.base[0] - 1 + a, g1 = f.base[1] - 1 + b;
#pragma unroll 1
  for (int c = lane >> 4; c < 4; c += 2) {
    const int g2 = f.base[2] - 1 + c;
    if (!node_in_grid(S, g0, g1, g2)) continue;
    const int blk = block_id(S, g0 >> 2, g1 >> 2, g2 >> 2), node = (g0 & 3) + 4 * (g1 & 3) + 16 * (g2 & 3);
    const float wzc = f.wz[c], gzc = f.gz[c];
    if constexpr (KIND == kP2gForce) {
      if (__ldg(&S.blk_slot[blk]) < 0) continue;  // only active blocks' words are read and cleared by the solve
      const float gw[3] = {gxa * wyb * wzc, wxa * gyb * wzc, wxa * wyb * gzc};
      float* dst = reinterpret_cast<float*>(S.acc + (size_t)blk * kAccBlockWords + 4 * kBlockNodes + node);
#pragma unroll
      for (int r = 0; r < 3; r++) atomicAdd(dst + 2 * r * kBlockNodes, As[r][0] * gw[0] + As[r][1] * gw[1] + As[r][2] * gw[2]);
    } else {
      RowFactors rf;
      row_factors(f.ms, f.mvs, As, wyb, gyb, wzc, gzc, mo, rf);
      long long v[7] = {0, 0, 0, 0, 0, 0, 0};
      if (kind == kFarFast) {
        v[0] = fix_mass(wxa, rf) - kMagicBits;
        if (!mo)
#pragma unroll
          for (int r = 0; r < 3; r++) {
            v[1 + r] = fix_mom(wxa, rf, r) - kMagicBits;
            v[4 + r] = fix_force(wxa, gxa, rf, r) - kMagicBits;
          }
      } else {
        v[0] = round_product(wxa, rf.mw, 0);
        if (!mo)
#pragma unroll
          for (int r = 0; r < 3; r++) {
            v[1 + r] = round_product(wxa, rf.pv[r], 0);
            v[4 + r] = round_product(gxa, rf.kk[r], round_product(wxa, rf.hh[r], 0));
          }
      }
      if (!(v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6])) continue;
      acc_add(S, blk, node, v, mo);
      S.blk_flag[blk] = 1;
    }
  }
}

// ---- shared memory of one work item --------------------------------------
// The staged grid values: the tile's 9 x 9 rows of nodes, each row copied from
// the dense array in one piece that starts and ends on a 16-byte boundary.
// gout: rows of 10 nodes from x = 4b - 2; u of the solve: 12 nodes from
// 4b - 4. The planes' stride is padded so that a step in z and one in y lie in
// different banks.
template <int FIELDS> struct StageShape {
  static constexpr int x0 = FIELDS == kOutFields ? 2 : 4;    // first node of a row is 4b - x0
  static constexpr int row_nodes = FIELDS == kOutFields ? 10 : 12;
  static constexpr int row = FIELDS * row_nodes;             // floats: 60 / 36
  static constexpr int plane = kTile * row + (FIELDS == kOutFields ? 8 : 4);
  static_assert(row * sizeof(float) % 16 == 0 && plane * sizeof(float) % 16 == 0, "rows of whole 16-byte words");
};
constexpr int kStageFloats = kTile * StageShape<kOutFields>::plane;
static_assert(kTile * StageShape<kImpFields>::plane <= kStageFloats, "the solve's rows fit the same buffer");

// The shares that a cell's particles are summed in: one up to kShareWhole, beyond
// it one for each kShare, so that an item whose particles lie in a few cells keeps
// all half-warps at work.
constexpr int kShareWhole = 32, kShare = 16;
constexpr int kShares = kCells + kItemMax / kShare + kItemMax / kShareWhole;

struct ItemShared {
  __align__(16) float stage[kStageFloats];             // G2P: the grid values of the tile's nodes
  // the item's particles: its stretch of each stream (fc from an even particle on)
  float4 pxm[kItemMax], pvv[kItemMax], pfa[kItemMax], pfb[kItemMax], pvq[kItemMax];
  float2 pfc[kItemMax + 2];
  __align__(16) float pd[kItemMax / 2 * kPdStride];  // P2G: particle data in tile-cell order, by pairs
  union {
    int tilei[kAccFields * kTile3];  // P2G sums of the tile's nodes (fixed point: mass, momentum, force) ...
    float tile[kAccFields * kTile3]; // ... or float (the semi-implicit solve's K u)
  };
  int cstart[kCells + 1];            // first pd slot of each tile cell
  int ccount[kCells];                // particles per tile cell (zero between items)
  short cells[kCells];               // occupied tile cells
  int shares[kShares + 1];           // ... crowded ones once for each share, with its first pd slot above
  int4 item_q[2];                    // this and the next work item of the CTA
  int scene_q[2];                    // ... and their scenes
  int index_q[2];                    // ... and their indices (total: no item)
  int coll_scene;                    // scene whose colliders sit in coll
  FixScale fscale;                   // fixed-point scales of coll_scene's P2G in this launch
  unsigned seen[3];                  // largest mass, |v|, force-term bound of coll_scene's particles (bits) ...
  unsigned pushed[3];                // ... and the part of them already recorded in FixState
  int next_same;                     // the CTA's next work item continues this item's home-block run
  int next_issue;                    // ... or starts a run whose grid rows the last warp copies
  int unit_left;                     // items of the unit in hand after the one looked up last
  int unit_tail;                     // runs from this item on are handed out item by item
  int unit_most;                     // the others as many items at a time (a power of two)
  float run_bound;                   // sum of the contribution bounds of the particles in the tile's sums
  float item_bound;                  // ... and of this item's particles headed for the tile
  int crowded;                       // a cell holds more of the item's particles than kShareWhole
  int wide;                          // some of the item's particles go through wide_scatter
  int abort;                         // 1 + parity of a wait for grid rows that ran out, else 0
  int pabort;                        // ... for particles
  uint64_t bar, pbar;                // completion of the grid rows' copies, of the particles'
  snow_collider coll[kShColliders];
  float4 chit[kShColliders];         // packed hit tests of the colliders
  int ctype[kShColliders];
};

__device__ __forceinline__ void home_coords(const SceneDev& S, int blk, int& bx, int& by, int& bz) {
  bx = blk % S.bdim[0];
  by = (blk / S.bdim[0]) % S.bdim[1];
  bz = blk / (S.bdim[0] * S.bdim[1]);
}

// Index of node (x, y, z) of the blocked grid in gout and cru.
__device__ __forceinline__ size_t node_index(const SceneDev& S, int x, int y, int z) {
  return ((size_t)z * (4 * S.bdim[1]) + y) * (4 * S.bdim[0]) + x;
}

// Every thread of the CTA calls it: issues the bulk copies (TMA) of the rows,
// one per thread, of the tile around home block `home` from the dense array `grid` into `stage` and zero-fills
// what lies outside the grid; completion lands on sh.bar, which expects
// `unsent` bytes more than are copied (0 except in tests of the timeout
// path). The caller guarantees nobody reads `stage` until the barrier's phase
// completes and that all earlier reads of `stage` are done. Rows instead of
// the 27 whole blocks around the home block: 19 KB of shared memory instead
// of 41 (the rest holds the next item's particles), and every stencil node at
// a constant offset from the particle's first instead of through twelve
// address registers.
template <int FIELDS>
__device__ __forceinline__ void stage_issue(ItemShared& sh, const SceneDev& S, const float* grid, int home) {
  using T = StageShape<FIELDS>;
  int bx, by, bz;
  home_coords(S, home, bx, by, bz);
  const int nx = 4 * S.bdim[0], ny = 4 * S.bdim[1], nz = 4 * S.bdim[2];
  const int xs = 4 * bx - T::x0, xa = max(xs, 0), xe = min(xs + T::row_nodes, nx);  // multiples of 16 bytes: x0 and nx are
  const uint32_t bytes = (uint32_t)((xe - xa) * FIELDS * (int)sizeof(float));
  const int y0 = max(0, 2 - 4 * by), y1 = min(kTile, ny - (4 * by - 2));  // rows inside the grid
  const int z0 = max(0, 2 - 4 * bz), z1 = min(kTile, nz - (4 * bz - 2));
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&sh.bar, (uint32_t)((y1 - y0) * (z1 - z0)) * bytes + S.tx_unsent);
  static_assert(kTile * kTile <= kItemMax, "a row per thread");
  if (threadIdx.x < kTile * kTile) {
    fence_proxy_async_smem();
    const int y = threadIdx.x % kTile, z = threadIdx.x / kTile;
    float* dst = sh.stage + z * T::plane + y * T::row;
    bool copied = false;
    if (y >= y0 && y < y1 && z >= z0 && z < z1) {
      bulk_g2s(dst + (xa - xs) * FIELDS, grid + node_index(S, xa, 4 * by - 2 + y, 4 * bz - 2 + z) * FIELDS, bytes, &sh.bar);
      copied = true;
      if (xe - xa == T::row_nodes) return;
    }
    for (int x = 0; x < T::row_nodes; x++)
      if (!copied || x < xa - xs || x >= xe - xs)
#pragma unroll
        for (int f = 0; f < FIELDS; f++) dst[x * FIELDS + f] = 0.0f;
  }
}

// One full warp issues the bulk copies of the particles [first, first + count)
// (a stretch of each stream, or of the binned copies) into the CTA's particle
// buffer; completion lands on sh.pbar. The caller guarantees that all earlier
// reads of the buffer are done. The loads of an item's particles are then
// under way while the CTA sums the previous item, instead of being waited for
// at the item's start and again before its advance.
__device__ __forceinline__ void particles_issue(ItemShared& sh, const SceneDev& S, int first, int count, bool binned) {
  const int lane = threadIdx.x & 31;
  const int f0 = first & ~1, fn = (first + count - f0 + 1) & ~1;  // fc: whole 16-byte words (the streams' allocations are whole 256-byte units)
  if (lane == 0) mbar_arrive_expect_tx(&sh.pbar, (uint32_t)(count * 5 * sizeof(float4) + fn * sizeof(float2)));
  __syncwarp();
  if (lane < 6) {
    fence_proxy_async_smem();
    const float4* src4[5] = {binned ? S.bxm : S.xm, binned ? S.bvv : S.vv, binned ? S.bfa : S.fa, binned ? S.bfb : S.fb,
                             binned ? S.bvq : S.vq};
    float4* dst4[5] = {sh.pxm, sh.pvv, sh.pfa, sh.pfb, sh.pvq};
#pragma unroll
    for (int k = 0; k < 5; k++)
      if (lane == k) bulk_g2s(dst4[k], src4[k] + first, (uint32_t)(count * sizeof(float4)), &sh.pbar);
    if (lane == 5) bulk_g2s(sh.pfc, (binned ? S.bfc : S.fc) + f0, (uint32_t)(fn * sizeof(float2)), &sh.pbar);
  }
}
// Waits for them, as stage_wait does for the grid rows.
__device__ __forceinline__ bool particles_wait(ItemShared& sh, const SceneDev& S, uint32_t& phase) {
  if (!mbar_wait(&sh.pbar, phase, S.wait_ns)) {
    sh.pabort = 1 + (int)phase;
    return false;
  }
  phase ^= 1u;
  return true;
}

// Every thread waits for the stage copies of the current phase, at most
// S.wait_ns. Returns false if the wait ran out; the thread then records the
// phase in sh.abort (1 + parity), and the CTA stops at its next barrier that
// checks it (stage_abort) without reading the stage.
__device__ __forceinline__ bool stage_wait(ItemShared& sh, const SceneDev& S, uint32_t& phase) {
  if (!mbar_wait(&sh.bar, phase, S.wait_ns)) {
    sh.abort = 1 + (int)phase;
    return false;
  }
  phase ^= 1u;
  return true;
}

// The end of a CTA whose copy wait ran out (every thread calls it, after a
// barrier that made sh.abort visible): the timeout is counted once (the host
// returns SNOW_ETIMEDOUT) and thread 0 gives the copies still in flight one
// more bounded wait, so the CTA does not exit while bulk copies into its
// shared memory may still land. Issues no copies.
__device__ __forceinline__ void stage_abort(ItemShared& sh, const SceneDev& S) {
  if (threadIdx.x == 0) {
    atomicAdd(&S.counters[CNT_TIMEOUT], 1);
    if (sh.abort) mbar_wait(&sh.bar, (uint32_t)(sh.abort - 1), S.wait_ns);
    if (sh.pabort) mbar_wait(&sh.pbar, (uint32_t)(sh.pabort - 1), S.wait_ns);
  }
}

// Colliders of scene S into shared memory (when they fit). Ends with
// __syncthreads.
__device__ __forceinline__ void load_colliders(ItemShared& sh, const SceneDev& S) {
  if (S.ncoll <= kShColliders && threadIdx.x < S.ncoll) {
    const snow_collider c = S.coll[threadIdx.x];
    sh.coll[threadIdx.x] = c;
    sh.ctype[threadIdx.x] = c.type;
    float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (c.type == 0)
      h = make_float4(c.normal[0], c.normal[1], c.normal[2],
                      fmaf(c.normal[2], c.pos[2], fmaf(c.normal[1], c.pos[1], c.normal[0] * c.pos[0])));
    else if (c.type == 1)
      h = make_float4(c.pos[0], c.pos[1], c.pos[2], c.radius * c.radius);
    sh.chit[threadIdx.x] = h;
  }
  __syncthreads();
}

// Zeroes the first nf fields of the P2G tile (at the start of each item,
// after the previous item's flush has read it).
__device__ __forceinline__ void tile_zero(ItemShared& sh, int nf) {
  static_assert(offsetof(ItemShared, tile) % 16 == 0, "tile must be 16-byte aligned");
  float4* t4 = reinterpret_cast<float4*>(sh.tile);
  const int n4 = nf * kTile3 / 4;
  for (int i = threadIdx.x; i < n4; i += blockDim.x) t4[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int i = 4 * n4 + threadIdx.x; i < nf * kTile3; i += blockDim.x) sh.tile[i] = 0.0f;
}

// Kernel start: cell counts, flags, the bulk-copy barrier and finite values in
// the P2G records (the half of an item's last record that holds no particle
// is multiplied by zero weights). Ends with __syncthreads.
__device__ __forceinline__ void tile_init(ItemShared& sh) {
  for (int i = threadIdx.x; i < kCells; i += blockDim.x) sh.ccount[i] = 0;
  static_assert(offsetof(ItemShared, pd) % 16 == 0 && sizeof(sh.pd) % 16 == 0, "records are cleared in 16-byte words");
  float4* pd4 = reinterpret_cast<float4*>(sh.pd);
  for (int i = threadIdx.x; i < (int)(sizeof(sh.pd) / 16); i += blockDim.x) pd4[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (threadIdx.x == 0) {
    mbar_init(&sh.bar, 1);
    mbar_init(&sh.pbar, 1);
    sh.abort = sh.pabort = 0;
    sh.run_bound = sh.item_bound = 0.0f;
    sh.wide = sh.crowded = 0;
  }
  __syncthreads();
}

// G2P sums of one particle: dv = sum_i w_ip d_i (PIC/FLIP increment,
// g2pTransfer.glsl:99-104) and L = sum_i v*_i (grad w_ip)^T (velocity
// gradient, :121-129), contracted along x first for each (y, z) row.
// node(a, b, c, p) fills the 6 values (v*, d) of stencil node (a, b, c) as
// three pairs (v0, v1), (v2, d0), (d1, d2) or returns false for a node that
// contributes nothing. Bound by shared loads and instruction issue: the packed
// instructions take 5 where the 9 sums along x take 9, and round each sum as
// those do. The z loop is not unrolled: the code of the fused kernel does not
// fit the instruction cache (0.234 against 0.237 ms, 1M particles, 256^3).
template <class Node>
__device__ __forceinline__ void g2p_sums(const AxisW& w, Node node, float dv[3], float L[3][3]) {
  f32x2 dv12 = 0ull, L0[3] = {0ull, 0ull, 0ull};  // (dv1, dv2); (L0k, L1k)
  float dv0 = 0.0f, L2[3] = {0.0f, 0.0f, 0.0f};
  f32x2 wx[4], gx[4];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    wx[a] = pack2(w.wx[a], w.wx[a]);
    gx[a] = pack2(w.gx[a], w.gx[a]);
  }
  float wz = w.wz[0], gz = w.gz[0], wzn[3] = {w.wz[1], w.wz[2], w.wz[3]}, gzn[3] = {w.gz[1], w.gz[2], w.gz[3]};
#pragma unroll 1
  for (int c = 0; c < 4; c++) {
#pragma unroll
    for (int b = 0; b < 4; b++) {
      f32x2 S1 = 0ull, SD = 0ull, D = 0ull, S2 = 0ull;  // sum wx (v0, v1), wx (v2, d0), wx (d1, d2), gx (v0, v1)
      float S22 = 0.0f;                                  // sum gx v2
#pragma unroll
      for (int a = 0; a < 4; a++) {
        f32x2 p[3];
        if (!node(a, b, c, p)) continue;
        S1 = fma2(wx[a], p[0], S1);
        SD = fma2(wx[a], p[1], SD);
        D = fma2(wx[a], p[2], D);
        S2 = fma2(gx[a], p[0], S2);
        S22 += w.gx[a] * lo2(p[1]);
      }
      const float t1 = w.wy[b] * wz, t2 = w.gy[b] * wz, t3 = w.wy[b] * gz;
      const float S12 = lo2(SD);
      dv0 += t1 * hi2(SD);
      dv12 = fma2(pack2(t1, t1), D, dv12);
      L0[0] = fma2(pack2(t1, t1), S2, L0[0]);
      L0[1] = fma2(pack2(t2, t2), S1, L0[1]);
      L0[2] = fma2(pack2(t3, t3), S1, L0[2]);
      L2[0] += t1 * S22;
      L2[1] += t2 * S12;
      L2[2] += t3 * S12;
    }
    wz = wzn[0]; wzn[0] = wzn[1]; wzn[1] = wzn[2];
    gz = gzn[0]; gzn[0] = gzn[1]; gzn[1] = gzn[2];
  }
  dv[0] = dv0;
  dv[1] = lo2(dv12);
  dv[2] = hi2(dv12);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    L[0][k] = lo2(L0[k]);
    L[1][k] = hi2(L0[k]);
    L[2][k] = L2[k];
  }
}

// Whether the stencil of base cell `base` lies in the tile of home block
// (bx, by, bz); t = its first node in tile coordinates.
__device__ __forceinline__ bool stencil_in_tile(int bx, int by, int bz, const int base[3], int t[3]) {
  t[0] = base[0] - 1 - (4 * bx - 2);
  t[1] = base[1] - 1 - (4 * by - 2);
  t[2] = base[2] - 1 - (4 * bz - 2);
  return t[0] >= 0 && t[1] >= 0 && t[2] >= 0 && t[0] <= kTile - 4 && t[1] <= kTile - 4 && t[2] <= kTile - 4;
}

// Gather for particle at base cell `base` of the item at home block
// (bx, by, bz): from the staged tile when the stencil lies in it, else from
// global memory.
__device__ __forceinline__ void g2p_gather(const ItemShared& sh, const SceneDev& S, int bx, int by, int bz,
                                           const int base[3], const AxisW& w, float dv[3], float L[3][3]) {
  using T = StageShape<kOutFields>;
  int t[3];
  if (stencil_in_tile(bx, by, bz, base, t)) {
    const float* st = sh.stage + t[2] * T::plane + t[1] * T::row + t[0] * kOutFields;
    g2p_sums(w,
             [&](int a, int b, int c, f32x2 p[3]) {
               const f32x2* o = reinterpret_cast<const f32x2*>(st + c * T::plane + b * T::row + a * kOutFields);
               p[0] = o[0];
               p[1] = o[1];
               p[2] = o[2];
               return true;
             },
             dv, L);
  } else {
    g2p_sums(w,
             [&](int a, int b, int c, f32x2 p[3]) {
               const int g0 = base[0] - 1 + a, g1 = base[1] - 1 + b, g2 = base[2] - 1 + c;
               if (!node_in_grid(S, g0, g1, g2)) return false;
               const f32x2* o = reinterpret_cast<const f32x2*>(S.gout + node_index(S, g0, g1, g2) * kOutFields);
               p[0] = o[0];
               p[1] = o[1];
               p[2] = o[2];
               return true;
             },
             dv, L);
  }
}

// Position and velocity of one particle, loaded ahead of the gather.
struct PState {
  float4 xm, vv;
};

__device__ __forceinline__ PState load_state(const SceneDev& S, int p, bool binned) {
  PState t;
  t.xm = __ldcs((binned ? S.bxm : S.xm) + p);
  t.vv = __ldcs((binned ? S.bvv : S.vv) + p);
  return t;
}

// particleAdvance.glsl:87-210 for particle p given its G2P sums; stores the
// new state and returns it with the rotation R = W V^T of the SVD.
struct Advanced {
  float4 xm, vv;
  M3 fe, R;
  float jp;
};

// F_E, J_p and the previous SVD frame of one particle.
struct PDef {
  float4 fa, fb, vq;
  float2 fc;
};

__device__ __forceinline__ PDef load_def(const SceneDev& S, int p, bool binned) {
  PDef d;
  d.fa = __ldcs((binned ? S.bfa : S.fa) + p);
  d.fb = __ldcs((binned ? S.bfb : S.fb) + p);
  d.vq = __ldcs((binned ? S.bvq : S.vq) + p);
  d.fc = __ldcs((binned ? S.bfc : S.fc) + p);
  return d;
}

__device__ __forceinline__ void advance_particle(const SceneDev& S, int p, const PState& ps, const PDef& def,
                                                 const float dv[3], const float L[3][3], const ItemShared& sh,
                                                 Advanced& out) {
  M3 FE;
  FE.m[0][0] = def.fa.x; FE.m[0][1] = def.fa.y; FE.m[0][2] = def.fa.z;
  FE.m[1][0] = def.fa.w; FE.m[1][1] = def.fb.x; FE.m[1][2] = def.fb.y;
  FE.m[2][0] = def.fb.z; FE.m[2][1] = def.fb.w; FE.m[2][2] = def.fc.x;
  const float jp = def.fc.y;
  float4 xm = ps.xm, vv = ps.vv;
  M3 step;
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int r = 0; r < 3; r++) step.m[c][r] = (c == r ? 1.0f : 0.0f) + S.dt * L[r][c];
  const M3 fe_trial = m3_mul(step, FE);
  M3 V;
  float lam[3];
  float q[4] = {def.vq.x, def.vq.y, def.vq.z, def.vq.w};
  eigen_warm(fe_trial, q, V, lam);
  __stcs(&S.vq[p], make_float4(q[0], q[1], q[2], q[3]));
  // With FE_trial = W S V^T and B = FE_trial V = W S (columns of norm
  // sigma_i), the clamped F_E' = W clamp(S) V^T = B diag(clamp(sigma)/sigma) V^T
  // and the polar rotation R = W V^T = B diag(1/sigma) V^T: the sort and QR
  // of the shader's SVD (which only serve to find W) are not needed here.
  const M3 B = m3_mul(fe_trial, V);
  M3 Br, Bc;
  float ratio = 1.0f;
  bool clamped = false;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float inv = rsqrt_nr(fmaxf(lam[c], 1e-30f));
    const float sig = lam[c] * inv;
    const float cl = fminf(fmaxf(sig, S.crit_lo), S.crit_hi);
    clamped = clamped || cl != sig;
    ratio *= __fdividef(sig, cl);
    const float sc = cl * inv;
#pragma unroll
    for (int r = 0; r < 3; r++) {
      Br.m[c][r] = B.m[c][r] * inv;
      Bc.m[c][r] = B.m[c][r] * sc;
    }
  }
  out.R = m3_mul_bt(Br, V);
  // no singular value clamped: F_E' = FE_trial exactly, J_p unchanged
  out.fe = clamped ? m3_mul_bt(Bc, V) : fe_trial;
  // det F_P' = det F_P * det(FE_trial) / det(FE'): the shader's
  // F_P' = V S^-1 W^T (I + dt L) FE FP (particleAdvance.glsl:132) has this
  // determinant; only det F_P is ever read (p2gTransfer.glsl:119).
  out.jp = clamped ? jp * ratio : jp;
  float v[3] = {S.alpha * vv.x + dv[0], S.alpha * vv.y + dv[1], S.alpha * vv.z + dv[2]};
  const float xold[3] = {xm.x, xm.y, xm.z};
  if (S.ncoll <= kShColliders)
    collide_packed(sh.coll, sh.chit, sh.ctype, S.ncoll, xold, v);
  else
    collide(S.coll, S.ncoll, xold, v);
  xm.x += S.dt * v[0];
  xm.y += S.dt * v[1];
  xm.z += S.dt * v[2];
  vv.x = v[0];
  vv.y = v[1];
  vv.z = v[2];
  __stcs(&S.xm[p], xm);
  __stcs(&S.vv[p], vv);
  store_fe(S, p, out.fe, out.jp);
  out.xm = xm;
  out.vv = vv;
  bool finite = isfinite(xm.x) && isfinite(xm.y) && isfinite(xm.z) && isfinite(v[0]) && isfinite(v[1]) &&
                isfinite(v[2]) && isfinite(out.jp);
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int r = 0; r < 3; r++) finite = finite && isfinite(out.fe.m[c][r]);
  if (!finite) atomicAdd(&S.counters[CNT_NONFINITE], 1);
}

// Clears the halves of v outside the list slots [j0, j1) of the pair at slots (j, j + 1).
__device__ __forceinline__ f32x2 mask2(f32x2 v, bool lo, bool hi) {
  unsigned a, b;
  unpack2(v, a, b);
  return pack2(__uint_as_float(lo ? a : 0u), __uint_as_float(hi ? b : 0u));
}

// Adds the particles of one tile cell (list slots j0..j1) to this lane's
// x-row (b, c) of the cell's 4x4x4 stencil: acc[a] holds node x = lx + a. The
// slots are taken two at a time (one record of sh.pd); a cell that starts or
// ends inside a record clears the other cell's half by its y weights, on which
// every term depends. Fixed point (mass alone, or mass, momentum and force):
// each contribution is rounded by the magic-offset FMA with the operations of
// row_factors, fix_mass, fix_mom and fix_force, and its bits are added to the
// unsigned accumulators, so every accumulator gains kMagicBits per slot; np
// counts the slots summed. K u (KIND kP2gForce): float sums of A grad w, the
// two halves apart in facc.
// Bound by the 128 bytes a cycle that shared memory returns to registers (the
// 16 lanes of a cell each load the particle's values). Two particles per
// packed instruction: 20 FMAs and 14 three-input adds per particle and lane
// instead of 40 and 28; with the packed gather above it took 23% of the fused
// kernel's instructions (162.6 to 125.3 million, 1M particles, 256^3).
template <int KIND>
__device__ __forceinline__ void cell_sums(const ItemShared& sh, int j0, int j1, int b, int c,
                                          unsigned (&acc)[4][kAccFields], f32x2 (&facc)[4][3], unsigned& np) {
  const f32x2 magic = pack2(kMagic, kMagic);
  for (int j = j0 & ~1; j < j1; j += 2, np += 2) {
    const float* rec = sh.pd + (j >> 1) * kPdStride;
    const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rec);
    const ulonglong2 yw = q[(kPdY >> 1) + b], zw = q[(kPdZ >> 1) + c];
    f32x2 wy = yw.x, gy = yw.y;
    const bool lo = j >= j0, hi = j + 1 < j1;
    if (!(lo && hi)) {
      wy = mask2(wy, lo, hi);
      gy = mask2(gy, lo, hi);
    }
    const f32x2 t1 = mul2(wy, zw.x);
    const ulonglong2 q0 = q[0];  // A22, m
    const ulonglong2 wx01 = q[kPdWx >> 1], wx23 = q[(kPdWx >> 1) + 1];
    const f32x2 wx[4] = {wx01.x, wx01.y, wx23.x, wx23.y};
    if (KIND != kP2gForce) {
      const f32x2 mw = mul2(q0.y, t1);
#pragma unroll
      for (int a = 0; a < 4; a++) {
        unsigned u, v;
        unpack2(fma2(wx[a], mw, magic), u, v);
        acc[a][0] += u + v;
      }
    }
    if (KIND == kP2gMass) continue;
    const f32x2 t2 = mul2(gy, zw.x), t3 = mul2(wy, zw.y);
    const ulonglong2 q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6];
    if (KIND == kP2gFull) {
      const f32x2 mv[3] = {q1.x, q1.y, q2.x};
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const f32x2 pv = mul2(mv[r], t1);
#pragma unroll
        for (int a = 0; a < 4; a++) {
          unsigned u, v;
          unpack2(fma2(wx[a], pv, magic), u, v);
          acc[a][1 + r] += u + v;
        }
      }
    }
    const ulonglong2 gx01 = q[kPdGx >> 1], gx23 = q[(kPdGx >> 1) + 1];
    const f32x2 gx[4] = {gx01.x, gx01.y, gx23.x, gx23.y};
    const f32x2 A[3][3] = {{q2.y, q3.x, q3.y}, {q4.x, q4.y, q5.x}, {q5.y, q6.x, q0.x}};
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const f32x2 kk = mul2(A[r][0], t1);
      const f32x2 hh = fma2(A[r][1], t2, mul2(A[r][2], t3));
#pragma unroll
      for (int a = 0; a < 4; a++) {
        if (KIND == kP2gFull) {
          unsigned u, v;
          unpack2(fma2(gx[a], kk, fma2(wx[a], hh, magic)), u, v);
          acc[a][4 + r] += u + v;
        } else {
          facc[a][r] = fma2(gx[a], kk, fma2(wx[a], hh, facc[a][r]));
        }
      }
    }
  }
}

__device__ __forceinline__ float sum2(f32x2 v) { return lo2(v) + hi2(v); }

// Adds the 4 nodes of this lane's row (tile nodes t0 .. t0 + 3) to the
// shared tile and clears them (float sums).
__device__ __forceinline__ void row_flush(ItemShared& sh, int t0, f32x2 (&acc)[4][3]) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
#pragma unroll
    for (int f = 0; f < 3; f++) {
      atomicAdd(&sh.tile[f * kTile3 + t0 + a], sum2(acc[a][f]));
      acc[a][f] = 0ull;
    }
  }
}
// ... fixed-point sums: `base` = np kMagicBits, the offset every accumulator
// carries (a cleared accumulator restarts at it).
template <int NF>
__device__ __forceinline__ void row_flush_fix(ItemShared& sh, int t0, unsigned (&acc)[4][kAccFields], unsigned base) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
#pragma unroll
    for (int f = 0; f < NF; f++) {
      atomicAdd(&sh.tilei[f * kTile3 + t0 + a], (int)(acc[a][f] - base));
      acc[a][f] = base;
    }
  }
}

__device__ __forceinline__ int cell_row_node(int ci, int b, int c) {
  const int lx = ci % kCellsPerAxis, ly = (ci / kCellsPerAxis) % kCellsPerAxis, lz = ci / (kCellsPerAxis * kCellsPerAxis);
  return lx + kTile * (ly + b) + kTile * kTile * (lz + c);
}

// P2G of the item's particles into the shared tile (every thread of the CTA
// calls it; thread i holds particle i of the item when `have`):
//   1. each particle inside the tile whose contributions fit the fast path's
//      range counts itself in its base cell (p2g_count); the others are
//      scattered straight to acc (scatter_far);
//   2. every warp scans the cell counts for itself: the first slot of each
//      cell and the list of the occupied cells; each particle stores its
//      (scaled) mass, momentum, A and axis weights at its slot, so the
//      particles lie in tile-cell order;
//   3. each half-warp owns one occupied cell at a time: lane l sums the
//      x-row (b, c) = (l & 3, l >> 2) of the cell's stencil over the cell's
//      particles in registers and adds the row to the shared tile.
// The tile keeps accumulating until p2g_tile_flush adds it to acc, so the
// items of one home block can share it. A barrier separates p2g_count from
// p2g_sum (2 and 3), at which the caller stops the CTA if a copy wait ran out
// (sh.abort, sh.pabort; nothing but the cell counts and the straight scatters
// has been written then).
// RUN: the tile may already hold earlier items' sums (sh.run_bound bounds
// them); when this item's particles could take a sum past kTileSumBound, the
// tile is first added to acc and cleared. p2g_sum ends with a barrier.
template <int KIND, bool CLEAR = false>
__device__ __forceinline__ void p2g_tile_flush(ItemShared& sh, const SceneDev& S, int bx, int by, int bz);

// A particle's quantities as the tile stores them (fixed point: scaled).
struct P2GStored {
  float ms, mvs[3], As[3][3];
  int cell, rank;  // its tile cell (-1: not in the tile) and its place among the cell's particles;
                   // kCellWide: its contributions outgrew 32 bits, and its stencil's first tile node
};
constexpr int kCellWide = -2;

__device__ __forceinline__ void far_put(FarParticle* f, const P2GStored& st, const AxisW& w) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
    f->wx[a] = w.wx[a];
    f->gx[a] = w.gx[a];
    f->wy[a] = w.wy[a];
    f->gy[a] = w.gy[a];
    f->wz[a] = w.wz[a];
    f->gz[a] = w.gz[a];
  }
  f->ms = st.ms;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    f->mvs[r] = st.mvs[r];
#pragma unroll
    for (int c = 0; c < 3; c++) f->As[3 * r + c] = st.As[r][c];
  }
}

// Particles in the tile whose force outgrew the scale (the first steps from
// rest: the scale follows the largest force of the step before): summed in shared
// memory, each force contribution as its low 20 bits and the rest, in two words of
// a tile of their own in pd, which is not in use yet. Not the mass and momentum,
// which stay in the fast range for these (wide_force) and round there to the
// same integers. 256 contributions below 2^42 fit both words. At kWideWarp such
// particles in a warp the zeroing and the flush cost less than their 448
// atomics each on 64-bit words in HBM: a step whose 131k particles are all wide
// took 544 us, now 220; the first of 32k particles from rest 115, now 53. WIDE: in an
// instantiation of its own, which a single scene's first step after its set-up takes:
// in every step's it cost 1% (registers).
constexpr int kWideWarp = 8;
constexpr int kWideShift = 20;
constexpr int kWideWords = 10 * kTile3;  // mass, momentum, force (low), force (rest)
static_assert(kWideWords + (int)(kItemMax / 32 * sizeof(FarParticle) / sizeof(float)) <= kItemMax / 2 * kPdStride,
              "the wide tile and a particle per warp fit pd");
__device__ __forceinline__ bool wide_force(const P2GParticle& q, const FixScale& sc, float bound) {
  const float mv = fmaxf(fabsf(q.mv[0]), fmaxf(fabsf(q.mv[1]), fabsf(q.mv[2])));
  return fmaxf(fabsf(q.m) * sc.m, mv * sc.p) * kWmax < kFastLimit && bound < 4.0e12f;  // 2^42 = 4.4e12
}
__device__ __noinline__ void wide_scatter(ItemShared& sh, const FarParticle& f, int origin) {
  int* const sum = reinterpret_cast<int*>(sh.pd);
  const int lane = threadIdx.x & 31;
  float As[3][3];
#pragma unroll
  for (int k = 0; k < 9; k++) As[k / 3][k % 3] = f.As[k];
  const int a = lane & 3, b = (lane >> 2) & 3;
  const float wxa = f.wx[a], gxa = f.gx[a], wyb = f.wy[b], gyb = f.gy[b];
#pragma unroll 1
  for (int c = lane >> 4; c < 4; c += 2) {
    RowFactors rf;
    row_factors(f.ms, f.mvs, As, wyb, gyb, f.wz[c], f.gz[c], false, rf);
    int* const at = sum + origin + a + kTile * b + kTile * kTile * c;
    atomicAdd(at, fix_mass(wxa, rf) - kMagicBits);
#pragma unroll
    for (int r = 0; r < 3; r++) {
      atomicAdd(at + (1 + r) * kTile3, fix_mom(wxa, rf, r) - kMagicBits);
      const long long v = round_bounded(gxa, rf.kk[r], round_bounded(wxa, rf.hh[r], 0));
      atomicAdd(at + (4 + r) * kTile3, (int)(v & ((1 << kWideShift) - 1)));
      atomicAdd(at + (7 + r) * kTile3, (int)(v >> kWideShift));
    }
  }
}
// The wide tile into acc; pd is left zero (finite) for the records.
__device__ __noinline__ void wide_flush(ItemShared& sh, const SceneDev& S, int bx, int by, int bz) {
  int* const sum = reinterpret_cast<int*>(sh.pd);
  for (int t = threadIdx.x; t < kTile3; t += blockDim.x) {
    long long v[7];
    bool any = false;
#pragma unroll
    for (int k = 0; k < 7; k++) {
      v[k] = sum[k * kTile3 + t];
      sum[k * kTile3 + t] = 0;
      if (k >= 4) {
        v[k] += (long long)sum[(k + 3) * kTile3 + t] * (1 << kWideShift);
        sum[(k + 3) * kTile3 + t] = 0;
      }
      any = any || v[k] != 0;
    }
    const int g0 = 4 * bx - 2 + t % kTile, g1 = 4 * by - 2 + t / kTile % kTile, g2 = 4 * bz - 2 + t / (kTile * kTile);
    if (!any || !node_in_grid(S, g0, g1, g2)) continue;
    const int blk = block_id(S, g0 >> 2, g1 >> 2, g2 >> 2);
    acc_add(S, blk, (g0 & 3) + 4 * (g1 & 3) + 16 * (g2 & 3), v, false);
    S.blk_flag[blk] = 1;
  }
}
// By the whole CTA after the counts' barrier, when the item has such particles.
__device__ __forceinline__ void wide_sums(ItemShared& sh, const SceneDev& S, int bx, int by, int bz,
                                          const P2GStored& st, const AxisW& w) {
  for (int k = threadIdx.x; k < kWideWords; k += blockDim.x) sh.pd[k] = 0.0f;
  __syncthreads();
  if (threadIdx.x == 0) sh.wide = 0;  // every thread has read it
  FarParticle* f = reinterpret_cast<FarParticle*>(sh.pd + kWideWords) + (threadIdx.x >> 5);
  uint32_t todo = __ballot_sync(0xffffffffu, st.cell == kCellWide);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    __syncwarp();
    if ((int)(threadIdx.x & 31) == src) far_put(f, st, w);
    __syncwarp();
    wide_scatter(sh, *f, __shfl_sync(0xffffffffu, st.rank, src));
  }
  __syncthreads();
  wide_flush(sh, S, bx, by, bz);
  __syncthreads();
}

// Whether a binning would bring a particle at this base cell into its item's tile:
// not one well outside the grid, which is binned to the border.
__device__ __forceinline__ bool binning_helps(const SceneDev& S, const int base[3]) {
  bool in = true;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int home = min(max(base[k], 0), S.dim[k] - 1) & ~3;
    in = in && base[k] >= home - 1 && base[k] <= home + kCellsPerAxis - 2;
  }
  return in;
}

template <int KIND, bool RUN = false, bool WIDE = false>
__device__ __forceinline__ void p2g_count(ItemShared& sh, const SceneDev& S, int bx, int by, int bz, bool have,
                                          const P2GParticle& q, const AxisW& w, const int base[3], const FixScale& sc,
                                          P2GStored& st) {
  constexpr bool fix = KIND != kP2gForce;
  const int ox = 4 * bx - 2, oy = 4 * by - 2, oz = 4 * bz - 2;
  st.cell = -1;
  st.rank = 0;
  st.ms = 0.0f;
  float tile_bound = 0.0f;  // the particle's contribution bound, if it goes to the tile
  int far = kFarNone;       // ... or how it is scattered
#pragma unroll
  for (int r = 0; r < 3; r++) {
    st.mvs[r] = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) st.As[r][c] = q.force ? (fix ? q.A[r][c] * sc.f : q.A[r][c]) : 0.0f;
  }
  if (fix) {
    st.ms = q.m * sc.m;
#pragma unroll
    for (int r = 0; r < 3; r++) st.mvs[r] = q.mv[r] * sc.p;
  }
  if (have) {
    // what is not finite stays out of the records: cell_sums multiplies the
    // particle that shares a record by zero weights, be it of the cell beside, of an
    // item before or of another scene. It is scattered straight to its own nodes,
    // where what is not finite counts as nothing (K u: stays what it is). A NaN position
    // lies in cell 0 of the grid
    const float bound = fix ? fix_bound<KIND>(q, sc) : force_size(q);
    const bool fast = bound < (fix ? kFastLimit : INFINITY);  // false for NaN and infinite values as well
    const int lx = base[0] - 1 - ox, ly = base[1] - 1 - oy, lz = base[2] - 1 - oz;
    const bool inside = lx >= 0 && ly >= 0 && lz >= 0 && lx < kCellsPerAxis && ly < kCellsPerAxis && lz < kCellsPerAxis;
    const bool finite_w = w.wx[1] + w.wy[1] + w.wz[1] < 4.0f;
    if (inside && fast && finite_w) {
      st.cell = lx + kCellsPerAxis * ly + kCellsPerAxis * kCellsPerAxis * lz;
      st.rank = atomicAdd(&sh.ccount[st.cell], 1);
      if (st.rank == kShareWhole) sh.crowded = 1;
      tile_bound = bound;
    } else {
      // the particle drifted out of its home block's tile since the last
      // binning, outgrew the fast path's range or is not finite
      if (!inside && binning_helps(S, base)) atomicAdd(&S.counters[CNT_FALLBACK], 1);
      far = fast && finite_w ? kFarFast : kFarWide;
      if (KIND != kP2gForce && far == kFarWide) atomicAdd(&S.fix->wide, 1u);
      if (KIND == kP2gForce && !q.force) far = kFarNone;
      if (WIDE && inside && finite_w && wide_force(q, sc, bound)) {
        far = kFarTile;
        st.rank = lx + kTile * ly + kTile * kTile * lz;
      }
    }
  }
  if (WIDE) {
    const int n = __popc(__ballot_sync(0xffffffffu, far == kFarTile));
    if (far == kFarTile) {
      far = n >= kWideWarp ? kFarNone : kFarWide;
      if (n >= kWideWarp) {
        st.cell = kCellWide;
        sh.wide = 1;
      }
    }
  }
  uint32_t todo = __ballot_sync(0xffffffffu, far != kFarNone);
  if (todo) {
    // through the warp's part of the particle buffer, which its lanes have read
    static_assert(sizeof(FarParticle) <= 32 * sizeof(float4), "one particle in the warp's part of a stream");
    FarParticle* f = reinterpret_cast<FarParticle*>(sh.pfa + (threadIdx.x & ~31u));
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      __syncwarp();
      if ((int)(threadIdx.x & 31) == src) {
        far_put(f, st, w);
#pragma unroll
        for (int r = 0; r < 3; r++) f->base[r] = base[r];
      }
      __syncwarp();
      scatter_far<KIND>(S, *f, __shfl_sync(0xffffffffu, far, src));
    }
  }
  if (RUN) {  // per warp: its tile particles times their largest bound (no lower than their sum)
    const uint32_t in = __ballot_sync(0xffffffffu, st.cell >= 0);
    const float bmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(tile_bound)));
    if ((threadIdx.x & 31) == 0 && in) atomicAdd(&sh.item_bound, (float)__popc(in) * bmax);
  }
}

// Sums the shares [k0, k1) of the half-warp's slice into the tile. Cells of a
// slice often follow each other along x: the row's sums then slide one node
// instead of being flushed, so only the node that leaves the window goes to the
// shared tile. share(k, ci, j0, j1): the k-th share's cell and pd slots.
template <int KIND, class Share>
__device__ __forceinline__ void sum_shares(ItemShared& sh, int k0, int k1, Share share) {
  constexpr int NF = P2gFields<KIND>::nf;
  constexpr bool fix = KIND != kP2gForce;
  const int l16 = threadIdx.x & 15, b = l16 & 3, c = l16 >> 2;
  int cur = -1;
  unsigned acc[4][kAccFields];
  f32x2 facc[4][3];
#pragma unroll
  for (int a = 0; a < 4; a++) {
#pragma unroll
    for (int f = 0; f < kAccFields; f++) acc[a][f] = 0u;
#pragma unroll
    for (int f = 0; f < 3; f++) facc[a][f] = 0ull;
  }
  unsigned np = 0;
  for (int k = k0; k < k1; k++) {
    int ci, j0, j1;
    share(k, ci, j0, j1);
    if (cur >= 0) {
      const int row = cell_row_node(cur, b, c);
      const unsigned base_bits = np * (unsigned)kMagicBits;
      if (ci == cur + 1 && ci % kCellsPerAxis != 0) {
        // only node 0 leaves the window: flush it, slide the rest
#pragma unroll
        for (int f = 0; f < NF; f++) {
          if (fix) {
            atomicAdd(&sh.tilei[f * kTile3 + row], (int)(acc[0][f] - base_bits));
            acc[0][f] = acc[1][f];
            acc[1][f] = acc[2][f];
            acc[2][f] = acc[3][f];
            acc[3][f] = base_bits;
          } else {
            atomicAdd(&sh.tile[f * kTile3 + row], sum2(facc[0][f]));
            facc[0][f] = facc[1][f];
            facc[1][f] = facc[2][f];
            facc[2][f] = facc[3][f];
            facc[3][f] = 0ull;
          }
        }
      } else if (fix) {
        row_flush_fix<NF>(sh, row, acc, base_bits);
      } else {
        row_flush(sh, row, facc);
      }
    }
    cell_sums<KIND>(sh, j0, j1, b, c, acc, facc, np);
    cur = ci;
  }
  if (cur >= 0) {
    if (fix)
      row_flush_fix<NF>(sh, cell_row_node(cur, b, c), acc, np * (unsigned)kMagicBits);
    else
      row_flush(sh, cell_row_node(cur, b, c), facc);
  }
}

// An item with a cell of more than kShareWhole particles: its cells in shares (which
// start at a record's first particle), listed by every warp for itself. With whole
// cells an item of snow pressed to 300 particles a cell kept one half-warp of sixteen
// at work, on a chain of 128 pairs: 880 us a step of 1M such particles, 480 in shares.
template <int KIND>
__device__ __noinline__ void sum_crowded(ItemShared& sh) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int c0 = 0; c0 < kCells; c0 += 32) {
    const int ci = min(c0 + lane, kCells - 1), first = sh.cstart[ci];
    const int count = c0 + lane < kCells ? sh.cstart[ci + 1] - first : 0;
    const int parts = count > kShareWhole ? (count + kShare - 1) / kShare : (count > 0 ? 1 : 0);
    int incl = parts;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    for (int q = 0; q < parts; q++)
      sh.shares[n + incl - parts + q] = ci | (q ? (first + count * q / parts) & ~1 : first) << 16;
    n += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) sh.shares[n] = sh.cstart[kCells] << 16;
  __syncwarp();
  const int hw = threadIdx.x >> 4, nhw = blockDim.x >> 4;
  sum_shares<KIND>(sh, (n * hw) / nhw, (n * (hw + 1)) / nhw, [&](int k, int& ci, int& j0, int& j1) {
    ci = sh.shares[k] & 0xffff;
    j0 = sh.shares[k] >> 16;
    j1 = sh.shares[k + 1] >> 16;
  });
}

template <int KIND, bool RUN = false, bool WIDE = false>
__device__ __forceinline__ void p2g_sum(ItemShared& sh, const SceneDev& S, int bx, int by, int bz, const P2GStored& st,
                                        const AxisW& w) {
  constexpr int nf = P2gFields<KIND>::nf;
  const int lane = threadIdx.x & 31;
  const int my_cell = st.cell;
  if (WIDE && sh.wide) wide_sums(sh, S, bx, by, bz, st, w);  // uniform across the CTA
  if (RUN && sh.run_bound + sh.item_bound > kTileSumBound) {  // uniform across the CTA
    // this item's sums could wrap the tile's int32 sums: the earlier items'
    // go to acc first (integer sums: the split changes no bit of the result)
    p2g_tile_flush<KIND>(sh, S, bx, by, bz);
    __syncthreads();
    if (threadIdx.x == 0) sh.run_bound = 0.0f;
    tile_zero(sh, nf);
  }
  // exclusive scan of the cell counts and list of the occupied cells, seven
  // cells per lane. Every warp forms all of it and writes the same values, so
  // that no barrier lies between the scan and the stores that use it.
  constexpr int kPer = (kCells + 31) / 32;
  int ncells;
  {
    int cnt[kPer], sum = 0, occ = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const int ci = lane * kPer + k;
      cnt[k] = ci < kCells ? sh.ccount[ci] : 0;
      sum += cnt[k] + (cnt[k] > 0 ? 1 << 16 : 0);  // particles below, occupied cells above
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    ncells = sh.crowded ? -1 : __shfl_sync(0xffffffffu, incl, 31) >> 16;  // uniform across the CTA
    int at = (incl - sum) & 0xffff;
    occ = (incl - sum) >> 16;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const int ci = lane * kPer + k;
      if (ci <= kCells) sh.cstart[ci] = at;  // cstart[kCells]: the count of all
      if (cnt[k] > 0) sh.cells[occ++] = (short)ci;
      at += cnt[k];
    }
    static_assert(32 * kPer > kCells, "the lane past the last cell writes the end");
    __syncwarp();
  }
  if (my_cell >= 0) {
    // the particle's P2G data, stored in tile-cell order
    const int slot = sh.cstart[my_cell] + st.rank;
    float* d = sh.pd + (slot >> 1) * kPdStride + (slot & 1);
    d[2 * kPdM] = st.ms;
    if (KIND != kP2gMass) {
#pragma unroll
      for (int r = 0; r < 3; r++) {
        d[2 * (kPdMv + r)] = st.mvs[r];
#pragma unroll
        for (int c = 0; c < 3; c++) d[2 * (r == 2 && c == 2 ? kPdA22 : kPdA + 3 * r + c)] = st.As[r][c];
      }
    }
#pragma unroll
    for (int a = 0; a < 4; a++) {
      d[2 * (kPdWx + a)] = w.wx[a];
      d[2 * (kPdGx + a)] = w.gx[a];
      d[2 * (kPdY + 2 * a)] = w.wy[a];
      d[2 * (kPdY + 2 * a + 1)] = w.gy[a];
      d[2 * (kPdZ + 2 * a)] = w.wz[a];
      d[2 * (kPdZ + 2 * a + 1)] = w.gz[a];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kCells; i += blockDim.x) sh.ccount[i] = 0;  // every warp has scanned them
  if (threadIdx.x == 0) sh.crowded = 0;
  if (RUN && threadIdx.x == 0) {  // every thread has read both bounds
    sh.run_bound += sh.item_bound;
    sh.item_bound = 0.0f;
  }
  if (ncells < 0) {
    sum_crowded<KIND>(sh);
  } else {
    // half-warp h takes a contiguous slice of the list (the two halves of a warp get
    // neighbouring slices, whose particle counts are alike)
    const int hw = threadIdx.x >> 4, nhw = blockDim.x >> 4;
    sum_shares<KIND>(sh, (ncells * hw) / nhw, (ncells * (hw + 1)) / nhw, [&](int k, int& ci, int& j0, int& j1) {
      ci = sh.cells[k];
      j0 = sh.cstart[ci];
      j1 = sh.cstart[ci + 1];
    });
  }
  __syncthreads();
}

// Adds the tile's non-zero nodes that lie in the grid to acc and flags
// their blocks (fixed point: each node's non-zero sums into its int64
// words; K u: three float adds into the force words of blocks active in
// this step). One tile node per thread, x fastest, so consecutive threads
// add to consecutive words. Every thread of the CTA calls it after
// p2g_sum's closing barrier; the caller separates it from the
// next use of the tile with a barrier.
// CLEAR: the tile's nodes that are not zero are cleared as they are read (cleared
// whole at each run's start instead, 50 steps of 1M particles took 14.92 ms, now 14.84,
// 24 of a 1.5M block 9.60 and 9.53).
template <int KIND, bool CLEAR>
__device__ __forceinline__ void p2g_tile_flush(ItemShared& sh, const SceneDev& S, int bx, int by, int bz) {
  constexpr int nf = P2gFields<KIND>::nf;
  const int ox = 4 * bx - 2, oy = 4 * by - 2, oz = 4 * bz - 2;
  for (int t = threadIdx.x; t < kTile3; t += blockDim.x) {
    const int x = t % kTile, y = (t / kTile) % kTile, z = t / (kTile * kTile);
    const int g0 = ox + x, g1 = oy + y, g2 = oz + z;
    if (!CLEAR && (g0 < 0 || g1 < 0 || g2 < 0 || g0 >= S.dim[0] || g1 >= S.dim[1] || g2 >= S.dim[2])) continue;
    int v[nf];
    int any = 0;
#pragma unroll
    for (int f = 0; f < nf; f++) {
      v[f] = sh.tilei[f * kTile3 + t];  // float K u: its bits (zero for 0.0f)
      any |= v[f];
    }
    if (!any) continue;
    if (CLEAR) {
#pragma unroll
      for (int f = 0; f < nf; f++) sh.tilei[f * kTile3 + t] = 0;
      if (g0 < 0 || g1 < 0 || g2 < 0 || g0 >= S.dim[0] || g1 >= S.dim[1] || g2 >= S.dim[2]) continue;
    }
    const int blk = block_id(S, g0 >> 2, g1 >> 2, g2 >> 2);
    unsigned long long* a = S.acc + (size_t)blk * kAccBlockWords + (g0 & 3) + 4 * (g1 & 3) + 16 * (g2 & 3);
    if constexpr (KIND == kP2gForce) {
      // K u goes only to blocks active in this step: the solve's node passes
      // read and clear the words of those alone (a block whose fixed-point
      // sums all rounded to zero is not active, although its K u may not be)
      if (__ldg(&S.blk_slot[blk]) < 0) continue;
      float* fw = reinterpret_cast<float*>(a + 4 * kBlockNodes);
#pragma unroll
      for (int f = 0; f < 3; f++) atomicAdd(fw + 2 * f * kBlockNodes, __int_as_float(v[f]));
    } else {
#pragma unroll
      for (int f = 0; f < nf; f++)
        if (v[f]) atomicAdd(a + f * kBlockNodes, (unsigned long long)(long long)v[f]);
      S.blk_flag[blk] = 1;
    }
  }
}
}  // namespace
}  // namespace snow
