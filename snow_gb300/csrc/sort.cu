// Particle binning for SNOW_MODE_FAST on sm_103a: the particle streams in the
// order of their cell keys and the P2G work items (home block, particle range);
// and a stable LSD radix sort of (key, particle index) pairs for the callers
// who ask for the sorted keys themselves.
//
// The reference has no sort (it scatters every (particle, neighbour) pair with
// global int atomics, p2gTransfer.cpp:22-23); binning is what makes the
// shared-memory tiling of this implementation possible. Cell of a particle: ivec3((x - gGridPos) /
// gridSpacing) as p2gTransfer.glsl:76-81 computes it (truncation toward
// zero), clamped into the grid. Key: block-major cell index
//   key = block(i>>2, j>>2, k>>2) * 64 + (i&3) + 4 (j&3) + 16 (k&3)
// with blocks numbered x fastest. The sort is stable, so the permutation is
// the one std::stable_sort gives on the same keys.
//
// Radix sort: 8-bit digits; per pass an upsweep (per-tile digit histograms,
// digit-major), an exclusive scan of the histograms and a downsweep that ranks
// each tile's keys stably with warp match/ballot and per-warp digit counters,
// then scatters.
#include <mutex>

#include "snow_internal.h"
#include "snow_tma.cuh"

namespace snow {
namespace {

constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsKpt = 16;                         // keys per thread
constexpr int kRsTile = kRsThreads * kRsKpt;       // 4096 keys per tile
constexpr int kRsPerWarp = kRsTile / kRsWarps;     // 512
constexpr int kScanChunk = 4096;                   // entries per scan CTA

__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const uint32_t* __restrict__ keys, size_t n, int shift,
                                                        uint32_t* __restrict__ hist, int ntiles) {
  __shared__ uint32_t h[256];
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    h[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)tile * kRsTile;
    for (int i = threadIdx.x; i < kRsTile; i += kRsThreads) {
      const size_t idx = base + i;
      if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + tile] = h[threadIdx.x];
    __syncthreads();
  }
}

// ---- exclusive scan of a uint32 array, three phases ----------------------
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t wsum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? wsum[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) wsum[lane] = s;
  }
  __syncthreads();
  const uint32_t before = (w > 0 ? wsum[w - 1] : 0u) + x - v;
  if (total) *total = wsum[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(256) k_scan_reduce(const uint32_t* __restrict__ a, size_t len,
                                                     uint32_t* __restrict__ partial) {
  const size_t base = (size_t)blockIdx.x * kScanChunk;
  uint32_t s = 0;
  for (int i = threadIdx.x; i < kScanChunk; i += blockDim.x) {
    const size_t idx = base + i;
    if (idx < len) s += a[idx];
  }
  uint32_t total;
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_partials(uint32_t* __restrict__ partial, int np) {
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < np; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < np ? partial[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, &total);
    if (i < np) partial[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_scan_down(uint32_t* __restrict__ a, size_t len,
                                                   const uint32_t* __restrict__ partial) {
  constexpr int per = kScanChunk / 256;
  const size_t base = (size_t)blockIdx.x * kScanChunk + (size_t)threadIdx.x * per;
  uint32_t v[per];
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < per; j++) {
    v[j] = (base + j < len) ? a[base + j] : 0u;
    s += v[j];
  }
  uint32_t run = partial[blockIdx.x] + block_exclusive_scan(s, nullptr);
#pragma unroll
  for (int j = 0; j < per; j++) {
    if (base + j < len) a[base + j] = run;
    run += v[j];
  }
}

void exclusive_scan(uint32_t* a, size_t len, uint32_t* partial, cudaStream_t st) {
  const int chunks = (int)((len + kScanChunk - 1) / kScanChunk);
  k_scan_reduce<<<chunks, 256, 0, st>>>(a, len, partial);
  k_scan_partials<<<1, 1024, 0, st>>>(partial, chunks);
  k_scan_down<<<chunks, 256, 0, st>>>(a, len, partial);
}

__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const uint32_t* __restrict__ kin,
                                                           const uint32_t* __restrict__ vin,
                                                           uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                           size_t n, int shift,
                                                           const uint32_t* __restrict__ offsets, int ntiles) {
  __shared__ uint32_t wcount[kRsWarps][256];
  __shared__ uint32_t gbase[256];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    for (int i = threadIdx.x; i < kRsWarps * 256; i += kRsThreads) (&wcount[0][0])[i] = 0u;
    gbase[threadIdx.x] = offsets[(size_t)threadIdx.x * ntiles + tile];
    __syncthreads();
    const size_t base = (size_t)tile * kRsTile + (size_t)w * kRsPerWarp;
    uint32_t key[kRsKpt], val[kRsKpt], rank[kRsKpt];
#pragma unroll
    for (int j = 0; j < kRsKpt; j++) {
      const size_t idx = base + (size_t)j * 32 + lane;
      const bool valid = idx < n;
      key[j] = valid ? kin[idx] : 0u;
      val[j] = valid ? vin[idx] : 0u;
      const uint32_t d = valid ? ((key[j] >> shift) & 255u) : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const uint32_t before = d < 256u ? wcount[w][d] : 0u;
      __syncwarp();
      if (d < 256u && (peers & lt) == 0u) wcount[w][d] = before + __popc(peers);
      __syncwarp();
      rank[j] = valid ? before + __popc(peers & lt) : 0xffffffffu;
    }
    __syncthreads();
    {
      const int d = threadIdx.x;  // one thread per digit
      uint32_t run = 0;
#pragma unroll
      for (int ww = 0; ww < kRsWarps; ww++) {
        const uint32_t t = wcount[ww][d];
        wcount[ww][d] = run;
        run += t;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRsKpt; j++) {
      if (rank[j] == 0xffffffffu) continue;
      const uint32_t d = (key[j] >> shift) & 255u;
      const uint32_t pos = gbase[d] + wcount[w][d] + rank[j];
      kout[pos] = key[j];
      vout[pos] = val[j];
    }
    __syncthreads();
  }
}

// ---- cell keys ---------------------------------------------------------------
__device__ __forceinline__ uint32_t cell_key(const SceneDev& S, float4 xm) {
  const float x[3] = {xm.x, xm.y, xm.z};
  int c[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    int v = (int)((x[k] - S.gpos[k]) / S.h);
    v = v < 0 ? 0 : (v > S.dim[k] - 1 ? S.dim[k] - 1 : v);
    c[k] = v;
  }
  const uint32_t b =
      ((uint32_t)(c[2] >> 2) * (uint32_t)S.bdim[1] + (uint32_t)(c[1] >> 2)) * (uint32_t)S.bdim[0] + (uint32_t)(c[0] >> 2);
  return b * 64u + (uint32_t)(c[0] & 3) + 4u * (uint32_t)(c[1] & 3) + 16u * (uint32_t)(c[2] & 3);
}

__global__ void k_keys(const SceneDev* __restrict__ sd, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  const SceneDev& S = *sd;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.n; p += gridDim.x * blockDim.x) {
    keys[p] = cell_key(S, S.xm[p]);
    vals[p] = (uint32_t)p;
  }
}

// ---- binning -----------------------------------------------------------------
// The order of the stable sort by cell key, in six kernels over all scenes of
// a step instead of the radix sort's passes (five launches each, three or four
// passes a scene): the particles are counted per grid block, the blocks' starts
// are scanned, the particle indices are put into their blocks, a group of threads
// per block orders its few hundred by (cell, index) (a CTA's groups together those
// of a crowded block), and the streams are moved. Bound by
// launches in small scenes and by the 184 bytes a particle that the streams'
// move reads and writes in large ones. A binning of 32k / 262k / 1M particles
// took 67 / 81 / 126 us in 20 launches, now 20 / 28 / 69 in 6.
__device__ __forceinline__ int scene_of(const int* prefix, int nscenes, long long u) {
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

// Keys, and each particle's place among those of its block (in no particular
// order): the lanes of a warp that share a block take their places with one
// atomic.
__global__ void __launch_bounds__(256) k_bin_count(const WorkSpace w) {
  chain_next();
  chain_wait();
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long u0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; u0 < w.total_particles;
       u0 += warps * 32) {
    const bool valid = u0 + lane < w.total_particles;
    const long long u = valid ? u0 + lane : w.total_particles - 1;
    const int s = scene_of(w.particles, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int p = (int)(u - w.particles[s]);
    const uint32_t key = cell_key(S, S.xm[p]);
    const int b = (int)(key >> 6);
    const unsigned long long id = valid ? (unsigned long long)s << 32 | (unsigned)b : ~0ull;
    const uint32_t peers = __match_any_sync(0xffffffffu, id);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (valid && lane == leader) base = atomicAdd(&S.bcount[b], __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!valid) continue;
    S.bkey[p] = key;
    S.brank[p] = (uint32_t)(base + __popc(peers & ((1u << lane) - 1u)));
    if (p == 0) S.counters[CNT_ITEMS] = 0;
  }
}

// Particles per chunk of blocks.
__global__ void __launch_bounds__(kBinChunk / 2) k_bin_reduce(const WorkSpace w) {
  chain_next();
  chain_wait();
  for (long long u = blockIdx.x; u < w.total_chunks; u += gridDim.x) {
    const int s = scene_of(w.chunks, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int c = (int)(u - w.chunks[s]), b0 = c * kBinChunk + 2 * (int)threadIdx.x;
    int2 n = make_int2(0, 0);
    if (b0 + 1 < S.nblocks)
      n = *reinterpret_cast<const int2*>(S.bcount + b0);
    else if (b0 < S.nblocks)
      n.x = S.bcount[b0];
    const int any = __syncthreads_or(n.x | n.y);
    uint32_t sum = 0;
    if (any) block_exclusive_scan((uint32_t)(n.x + n.y), &sum);
    if (threadIdx.x == 0) S.bchunk[c] = (int)sum;
    if (w.fit && any)
#pragma unroll
      for (int k = 0; k < kSizeChoices; k++) {
        const int z = size_choice(k);
        const int items = __reduce_add_sync(0xffffffffu, (n.x + z - 1) / z + (n.y + z - 1) / z);
        if ((threadIdx.x & 31) == 0 && items) atomicAdd(&w.sizes[k], items);
      }
  }
}

// The most particles of a work item (size_choice).
__device__ __forceinline__ int item_size(const WorkSpace& w, int items_max) {
  if (!w.fit) return items_max;
  const int rounds = (w.sizes[kSizeChoices - 1] + w.fit - 1) / w.fit;
  if (rounds > kFitRounds) return items_max;
  int size = items_max;
#pragma unroll
  for (int k = kSizeChoices - 1; k >= 0; k--)
    if (w.sizes[k] <= rounds * w.fit) size = size_choice(k);
  return size;
}

// Block ranges and work items, a CTA per chunk of blocks: the chunk starts
// after the particles of the chunks before it. Each block's particles are split
// into near-equal items of at most item_size.
__global__ void __launch_bounds__(kBinChunk / 2) k_bin_scan(const WorkSpace w) {
  __shared__ int first_item;
  chain_next();
  chain_wait();
  for (long long u = blockIdx.x; u < w.total_chunks; u += gridDim.x) {
    const int s = scene_of(w.chunks, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int c = (int)(u - w.chunks[s]);
    if (S.bchunk[c] == 0) continue;  // uniform across the CTA
    uint32_t sum = 0, before;
    for (int k = threadIdx.x; k < c; k += blockDim.x) sum += (uint32_t)S.bchunk[k];
    block_exclusive_scan(sum, &before);
    const int b0 = c * kBinChunk + 2 * (int)threadIdx.x;
    const int most = item_size(w, S.items_max);
    int cnt[2], nit[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      cnt[k] = b0 + k < S.nblocks ? S.bcount[b0 + k] : 0;
      nit[k] = (cnt[k] + most - 1) / most;
    }
    uint32_t items;
    uint32_t at = before + block_exclusive_scan((uint32_t)(cnt[0] + cnt[1]), nullptr);
    const uint32_t ahead = block_exclusive_scan((uint32_t)(nit[0] + nit[1]), &items);
    if (threadIdx.x == 0) first_item = atomicAdd(&S.counters[CNT_ITEMS], (int)items);
    __syncthreads();
    int it = first_item + (int)ahead;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      if (cnt[k] == 0) continue;
      const int b = b0 + k;
      S.bcount[b] = 0;
      S.bstart[b] = (int)at;
      S.bend[b] = (int)at + cnt[k];
      for (int j = 0; j < nit[k]; j++, it++) {
        if (it >= S.item_cap) break;  // cannot happen: item_cap covers the bound
        const int first = (int)(((long long)j * cnt[k]) / nit[k]), last = (int)(((long long)(j + 1) * cnt[k]) / nit[k]);
        S.items[it] = make_int4(b, (int)at + first, last - first, j == 0 ? nit[k] : -j);
      }
      at += (uint32_t)cnt[k];
    }
    __syncthreads();
  }
}

// Particle indices and keys into block order. The CTA that finishes last forms
// the item prefix.
__global__ void __launch_bounds__(256) k_bin_place(const WorkSpace w) {
  chain_next();
  chain_wait();
  const long long stride = (long long)gridDim.x * blockDim.x, u0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long u = u0; u < w.total_particles; u += stride) {
    const int s = scene_of(w.particles, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int p = (int)(u - w.particles[s]);
    const uint32_t key = S.bkey[p];
    const int d = S.bstart[key >> 6] + (int)S.brank[p];
    S.bidx[d] = (uint32_t)p;
    S.bskey[d] = key;
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&w.scenes[0].counters[CNT_DONE], 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    int a = 0;
    for (int s = 0; s < w.nscenes; s++) {
      w.items[s] = a;
      a += *(volatile int*)&w.scenes[s].counters[CNT_ITEMS];
    }
    w.items[w.nscenes] = a;
    for (int k = 0; k < kSizeChoices; k++) w.sizes[k] = 0;
    w.scenes[0].counters[CNT_DONE] = 0;
  }
}

// A group of 128 threads per occupied block (by its first work item): its particle
// indices in the order of their cells, and of the indices within a cell. The moves
// that follow have a thread per particle: done here, by the few hundred threads of a
// block's CTA, they took 69 us at 1M particles against 35. A particle's place in its
// cell is counted against all the cell's others; where a block of more than
// kCellThreads * kCellHeld particles has a cell of more than kMaxRanked, whose square
// that would cost, and where it has more than kMaxBlock, the CTA's groups together
// sort the whole block afterwards (order_crowded).
constexpr int kCellThreads = 128;
constexpr int kCellGroups = 4;
constexpr int kCellCta = kCellThreads * kCellGroups;
constexpr int kCellCtas = 3;  // per SM (40 registers)
constexpr int kCellHeld = 6;  // particles a thread holds in registers: blocks up to 768 are read once
constexpr int kMaxRanked = 128;
constexpr int kMaxBlock = 4096;
struct CellGroup {
  int count[64], start[64], cursor[64];
  uint32_t idx[kCellThreads * kCellHeld];
};
struct CrowdCounts {
  uint32_t next[4 * 256];                   // [digits + 1][values]: where the next index of each value goes
  uint32_t warps[kCellCta / 32 * 256];      // [warps][values]: the warps' counts in a tile, then their starts
};

// The n particle indices at S.bidx[n0 ..] into the order of their cells, and of the
// indices within a cell: a stable radix sort by the CTA, three digits of the index
// (five, beyond 2^24 particles) and then the cell, between bidx and brank (whose
// places are no longer needed). Bound by the latency of its reads and of the counts,
// and by one SM's scattered writes. A binning of 3.2M particles in 1,000 blocks with
// 200 to a cell takes 365 us, of 1M in 16 blocks 734, in one 9,230 (without any order
// in such cells 263, 688 and 7,980; by one group of 128 threads 465, 1,760 and 27,000;
// in a kernel of its own with 1,024 threads 351, 505 and 7,190, but then all binnings
// take a launch more: 20 steps of 300k with a binning in most 3.08 ms, 3.095).
constexpr int kCrowdedHeld = 8;  // indices of a thread under way
__device__ __noinline__ void order_crowded(CrowdCounts& sh, const SceneDev& S, int n0, int n) {
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int bits = 32 - __clz(S.n - 1), digits = bits <= 24 ? 3 : 5, width = max(6, (bits + digits - 1) / digits);
  const int values = 1 << width;  // of a digit: at most 256, and 128 where there are five
  auto digit = [&](uint32_t p, int k) { return k == digits ? S.bkey[p] & 63u : p >> (k * width) & (uint32_t)(values - 1); };
  for (int k = threadIdx.x; k < (digits + 1) * values; k += kCellCta) sh.next[k] = 0u;
  __syncthreads();
  for (int t = 0; t < n; t += kCellCta * kCrowdedHeld) {  // all digits are counted in one read
    uint32_t p[kCrowdedHeld];
#pragma unroll
    for (int j = 0; j < kCrowdedHeld; j++) {
      const int i = t + j * kCellCta + (int)threadIdx.x;
      p[j] = i < n ? S.bidx[n0 + i] : ~0u;
    }
#pragma unroll
    for (int j = 0; j < kCrowdedHeld; j++) {
      const uint32_t in = __ballot_sync(0xffffffffu, p[j] != ~0u);
      if (p[j] == ~0u) continue;
      for (int k = 0; k <= digits; k++) {  // often one value for the whole warp
        const uint32_t d = digit(p[j], k);
        int same;
        __match_all_sync(in, d, &same);
        if (!same)
          atomicAdd(&sh.next[k * values + d], 1u);
        else if (lane == 0)
          atomicAdd(&sh.next[k * values + d], (uint32_t)__popc(in));
      }
    }
  }
  __syncthreads();
  for (int k = wi; k <= digits; k += (kCellCta / 32)) {  // a warp scans a digit's counts: where its values start
    uint32_t run = 0u;
    for (int v = k * values + lane; v < (k + 1) * values; v += 32) {
      const uint32_t c = sh.next[v];
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      sh.next[v] = run + incl - c;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncthreads();
  uint32_t* const mine = sh.warps + wi * values;
#pragma unroll 1
  for (int pass = 0; pass <= digits; pass++) {  // an even number of passes: the last ends in bidx
    const uint32_t* const from = (pass & 1 ? S.brank : S.bidx) + n0;
    uint32_t* const to = (pass & 1 ? S.bidx : S.brank) + n0;
    uint32_t* const base = sh.next + pass * values;
    const int mine0 = wi * 32 * kCrowdedHeld + lane;  // the warp's stretch of a tile
    for (int t = 0; t < n; t += kCellCta * kCrowdedHeld) {
      uint32_t p[kCrowdedHeld], d[kCrowdedHeld], rank[kCrowdedHeld];
#pragma unroll
      for (int j = 0; j < kCrowdedHeld; j++) {
        const int i = t + mine0 + 32 * j;
        p[j] = i < n ? from[i] : ~0u;
      }
#pragma unroll
      for (int j = 0; j < kCrowdedHeld; j++) d[j] = p[j] != ~0u ? digit(p[j], pass) : ~0u;
      for (int v = lane; v < values; v += 32) mine[v] = 0u;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kCrowdedHeld; j++) {  // stable within the stretch
        const uint32_t peers = __match_any_sync(0xffffffffu, d[j]), below = peers & ((1u << lane) - 1u);
        const uint32_t before = d[j] != ~0u ? mine[d[j]] : 0u;
        __syncwarp();
        if (d[j] != ~0u && below == 0u) mine[d[j]] = before + __popc(peers);
        __syncwarp();
        rank[j] = before + __popc(below);
      }
      __syncthreads();
      for (int v = threadIdx.x; v < values; v += kCellCta) {  // the warps' counts become their starts
        uint32_t at = base[v];
#pragma unroll
        for (int k = 0; k < (kCellCta / 32); k++) {
          const uint32_t c = sh.warps[k * values + v];
          sh.warps[k * values + v] = at;
          at += c;
        }
        base[v] = at;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kCrowdedHeld; j++)
        if (d[j] != ~0u) to[mine[d[j]] + rank[j]] = p[j];
      __syncthreads();
    }
  }
}

__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kCellThreads) : "memory");
}
__global__ void __launch_bounds__(kCellCta, kCellCtas) k_bin_cells(const WorkSpace w, int in_step) {
  chain_next();
  chain_wait();
  __shared__ union {
    CellGroup group[kCellGroups];
    CrowdCounts crowd;
  } sh;
  __shared__ int crowded;
  if (threadIdx.x == 0) crowded = 0;
  __syncthreads();
  const int g = threadIdx.x / kCellThreads, tid = threadIdx.x % kCellThreads;
  CellGroup& cg = sh.group[g];
  auto leave = [&](const SceneDev& S, int n0) {  // a block to order_crowded
    S.bskey[n0] |= 0x80000000u;
    crowded = 1;
  };
  const int total = w.items[w.nscenes];
  for (int u = blockIdx.x * kCellGroups + g; u < total; u += gridDim.x * kCellGroups) {
    const int s = scene_of(w.items, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    if (in_step && u == w.items[s] && tid == 0) S.counters[CNT_BINNED] = 1;
    const int4 it = S.items[u - w.items[s]];
    const int n0 = S.bstart[it.x], n = S.bend[it.x] - n0;
    if (it.y != n0) continue;  // uniform across the group
    if (n > kMaxBlock) {
      if (tid == 0) leave(S, n0);
      continue;
    }
    const bool small = n <= kCellThreads * kCellHeld;
    uint32_t p[kCellHeld];
    int c[kCellHeld];
    if (tid < 64) cg.count[tid] = 0;
    group_sync(g);
    if (small) {
#pragma unroll
      for (int k = 0; k < kCellHeld; k++) {
        const int i = k * kCellThreads + tid;
        if (i < n) {
          p[k] = S.bidx[n0 + i];
          c[k] = (int)(S.bskey[n0 + i] & 63u);
          atomicAdd(&cg.count[c[k]], 1);
        }
      }
    } else {
      for (int i = tid; i < n; i += kCellThreads) atomicAdd(&cg.count[S.bskey[n0 + i] & 63u], 1);
    }
    group_sync(g);
    bool crowd = false;
    if (tid < 32) {
      const int c0 = cg.count[2 * tid], c1 = cg.count[2 * tid + 1];
      int incl = c0 + c1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (tid >= o) incl += v;
      }
      const int at = incl - c0 - c1;
      cg.start[2 * tid] = cg.cursor[2 * tid] = at;
      cg.start[2 * tid + 1] = cg.cursor[2 * tid + 1] = at + c0;
    }
    if (!small) {
      const int most = __reduce_max_sync(0xffffffffu, max(cg.count[2 * (tid & 31)], cg.count[2 * (tid & 31) + 1]));
      crowd = most > kMaxRanked;  // uniform across the group
    }
    group_sync(g);
    if (crowd) {
      if (tid == 0) leave(S, n0);
    } else if (small) {
#pragma unroll
      for (int k = 0; k < kCellHeld; k++)
        if (k * kCellThreads + tid < n) cg.idx[atomicAdd(&cg.cursor[c[k]], 1)] = p[k];
      group_sync(g);
#pragma unroll
      for (int k = 0; k < kCellHeld; k++) {
        if (k * kCellThreads + tid >= n) break;
        const int a = cg.start[c[k]], m = cg.count[c[k]];
        int r = 0;
        for (int j = a; j < a + m; j++) r += cg.idx[j] < p[k];
        S.bidx[n0 + a + r] = p[k];
      }
    } else {
      uint32_t* far = S.brank + n0;  // the places are no longer needed
      for (int i = tid; i < n; i += kCellThreads) far[atomicAdd(&cg.cursor[S.bskey[n0 + i] & 63u], 1)] = S.bidx[n0 + i];
      group_sync(g);
      for (int i = tid; i < n; i += kCellThreads) {
        const uint32_t q = far[i];
        const int cell = (int)(S.bkey[q] & 63u), a = cg.start[cell], m = cg.count[cell];
        int r = 0;
        for (int j = a; j < a + m; j++) r += far[j] < q;
        S.bidx[n0 + a + r] = q;
      }
    }
    group_sync(g);
  }
  __syncthreads();
  if (!crowded) return;
  for (int k = 0; k < kCellGroups; k++)  // the groups' blocks again, those that were left
    for (int u = blockIdx.x * kCellGroups + k; u < total; u += gridDim.x * kCellGroups) {
      const int s = scene_of(w.items, w.nscenes, u);
      const SceneDev& S = w.scenes[s];
      const int4 it = S.items[u - w.items[s]];
      const int n0 = S.bstart[it.x], n = S.bend[it.x] - n0;
      if (it.y == n0 && S.bskey[n0] >> 31 != 0u) order_crowded(sh.crowd, S, n0, n);
    }
}

// The particle streams into the binned copies, in the order bidx.
__global__ void __launch_bounds__(256) k_bin_move(const WorkSpace w) {
  chain_next();
  chain_wait();
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < w.total_particles;
       u += (long long)gridDim.x * blockDim.x) {
    const int s = scene_of(w.particles, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int i = (int)(u - w.particles[s]);
    const uint32_t p = S.bidx[i];
    const float4 xm = S.xm[p], vv = S.vv[p], fa = S.fa[p], fb = S.fb[p], vq = S.vq[p];
    const float2 fc = S.fc[p];
    const uint32_t pid = S.pid[p];
    S.bxm[i] = xm;
    S.bvv[i] = vv;
    S.bfa[i] = fa;
    S.bfb[i] = fb;
    S.bfc[i] = fc;
    S.bvq[i] = vq;
    S.bpid[i] = pid;
  }
}

// The binned copies back into the streams.
__global__ void __launch_bounds__(256) k_bin_back(const WorkSpace w) {
  chain_next();
  chain_wait();
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < w.total_particles;
       u += (long long)gridDim.x * blockDim.x) {
    const int s = scene_of(w.particles, w.nscenes, u);
    const SceneDev& S = w.scenes[s];
    const int i = (int)(u - w.particles[s]);
    S.xm[i] = S.bxm[i];
    S.vv[i] = S.bvv[i];
    S.fa[i] = S.bfa[i];
    S.fb[i] = S.bfb[i];
    S.fc[i] = S.bfc[i];
    S.vq[i] = S.bvq[i];
    S.pid[i] = S.bpid[i];
  }
}

int grid_for(size_t n, int threads, int per_sm) {
  size_t g = (n + threads - 1) / threads;
  const size_t cap = (size_t)num_sms() * per_sm;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

}  // namespace

size_t radix_tiles(size_t n) { return (n + kRsTile - 1) / kRsTile; }

void radix_sort_pairs(uint32_t* k[2], uint32_t* v[2], size_t n, int key_bits, uint32_t* hist, uint32_t* scan_tmp,
                      cudaStream_t st, int start) {
  if (n == 0) return;
  const int ntiles = (int)radix_tiles(n);
  const int passes = (key_bits + 7) / 8;
  int cur = start;
  const int g = grid_for((size_t)ntiles * kRsThreads, kRsThreads, 8);
  for (int pass = 0; pass < passes; pass++) {
    const int shift = 8 * pass;
    k_rs_hist<<<g, kRsThreads, 0, st>>>(k[cur], n, shift, hist, ntiles);
    exclusive_scan(hist, (size_t)256 * ntiles, scan_tmp, st);
    k_rs_scatter<<<g, kRsThreads, 0, st>>>(k[cur], v[cur], k[cur ^ 1], v[cur ^ 1], n, shift, hist, ntiles);
    cur ^= 1;
  }
  if (cur == 1) {
    cudaMemcpyAsync(k[0], k[1], n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(v[0], v[1], n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
  }
}

void fast_sort_keys(const SceneDev& sd, const SceneDev* sd_dev, BinScratch& b, int key_bits, cudaStream_t st) {
  if (sd.n <= 0) return;
  // an odd number of passes starts from the second buffer so that the
  // result lands in the first without a copy
  const int start = ((key_bits + 7) / 8) & 1;
  k_keys<<<grid_for(sd.n, 256, 8), 256, 0, st>>>(sd_dev, b.keys[start], b.vals[start]);
  radix_sort_pairs(b.keys, b.vals, (size_t)sd.n, key_bits, b.hist, b.scan_tmp, st, start);
}

void fast_bin_scenes(const WorkSpace& w, bool copy_back, bool chained, cudaStream_t st) {
  if (w.total_particles <= 0) return;
  const size_t n = (size_t)w.total_particles;
  const bool chain = w.total_particles <= kChainParticles;
  launch_after(chain && chained, k_bin_count, grid_for(n, 256, 8), 256, 0, st, w);
  launch_after(chain, k_bin_reduce, grid_for((size_t)w.total_chunks, 1, 8), kBinChunk / 2, 0, st, w);
  launch_after(chain, k_bin_scan, grid_for((size_t)w.total_chunks, 1, 8), kBinChunk / 2, 0, st, w);
  launch_after(chain, k_bin_place, grid_for(n, 256, 8), 256, 0, st, w);
  // an occupied block holds some hundred particles; at most a group for each 64
  launch_after(chain, k_bin_cells, grid_for(n, 64 * kCellGroups, kCellCtas), kCellCta, 0, st, w, copy_back ? 0 : 1);
  launch_after(chain, k_bin_move, grid_for(n, 256, 8), 256, 0, st, w);
  if (copy_back) launch_after(chain, k_bin_back, grid_for(n, 256, 8), 256, 0, st, w);
}

}  // namespace snow

// ---------------------------------------------------------------------------
// snow_sort_keys_static: a stable radix sort for callers that cannot allocate
// device memory. One cooperative launch: every CTA holds its tile of keys and
// values in registers through all passes of 8 bits, so that a pass scatters
// into the output arrays themselves once all CTAs have read them, and only the
// digit counts of the tiles (and the barriers' counters) need scratch, which
// lies in one file-scope __device__ array; every GPU that loads the library
// holds it (about 130 KB) until the process exits.
// Bound by launches and barriers: 262,144 keys of 24 bits took 140 us as 19
// launches and copies (86 us of them on the GPU), now 47 (32): 1,024 threads of
// two keys against 256 of eight, 48 us on the GPU.
// ---------------------------------------------------------------------------
namespace snow {
namespace {

constexpr size_t kStaticKeys = SNOW_SORT_STATIC_MAX_KEYS;
constexpr int kOneThreads = 1024;
constexpr int kOneWarps = kOneThreads / 32;
constexpr int kOneKpt = 2;                            // keys per thread
constexpr int kOneTile = kOneThreads * kOneKpt;       // 2048 keys per CTA
constexpr int kOneSplit = kOneThreads / 256;          // threads per digit where the digits are summed
constexpr int kOneCtas = (int)(kStaticKeys / kOneTile);  // 128: all resident at once
static_assert(kStaticKeys % kOneTile == 0, "whole tiles");
constexpr int kOneBarriers = 8;                       // two per pass, four passes
// layout: [digit counts kOneCtas x 256][barrier counters][CTAs whose wait ran out, until it is read]
constexpr size_t kStaticWords = (size_t)kOneCtas * 256 + kOneBarriers + 1;

__device__ __align__(256) uint32_t g_sort_scratch[kStaticWords];

// All CTAs of the (cooperative) launch meet at counter `bar`, zero before it.
// The wait is bounded like the copy waits; a CTA that runs out of it is counted,
// returns false and does no more work. LIMITED: with the limit and the arrivals of
// `wait`, in an instantiation of its own: as parameters of the one in use they
// took 262,144 keys from 47 to 54 us (its loads are scheduled otherwise).
constexpr int kSortExpired = kOneCtas * 256 + kOneBarriers;
struct SortWait {
  uint32_t limit_ns;
  uint32_t absent;  // arrivals waited for beyond those of the CTAs (a test of the timeout path)
};
template <bool LIMITED>
__device__ __forceinline__ bool grid_meet(uint32_t* bar, const SortWait& wait) {
  __shared__ bool met;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const uint64_t t0 = global_ns();
    met = true;
    for (uint32_t round = 0; *(volatile uint32_t*)bar < gridDim.x + (LIMITED ? wait.absent : 0u); round++)
      if ((round & 63u) == 63u && (round > (1u << 26) || global_ns() - t0 > (uint64_t)(LIMITED ? wait.limit_ns : kDefaultWaitNs))) {
        met = false;
        atomicAdd(&g_sort_scratch[kSortExpired], 1u);
        break;
      }
    __threadfence();
  }
  __syncthreads();
  return met;
}

template <bool LIMITED>
__global__ void __launch_bounds__(kOneThreads) k_sort_one(const uint32_t* keys, uint32_t* sorted, uint32_t* perm,
                                                          uint32_t n, int passes, uint32_t* hist, uint32_t* bars,
                                                          const SortWait wait) {
  __shared__ uint32_t wcount[kOneWarps][256];
  __shared__ uint32_t part[kOneSplit][256], ahead[kOneSplit][256], wsum[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int digit = threadIdx.x & 255, split = threadIdx.x >> 8;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t first = blockIdx.x * kOneTile + w * (kOneTile / kOneWarps) + lane;
  for (int pass = 0; pass < passes; pass++) {
    const int shift = 8 * pass;
    uint32_t key[kOneKpt], val[kOneKpt], rank[kOneKpt];
#pragma unroll
    for (int j = 0; j < kOneKpt; j++) {
      const uint32_t i = first + 32 * j;
      key[j] = i < n ? __ldcg((pass == 0 ? keys : sorted) + i) : 0u;
      val[j] = i < n ? (pass == 0 ? i : __ldcg(perm + i)) : 0u;
    }
#pragma unroll
    for (int d = lane; d < 256; d += 32) wcount[w][d] = 0u;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kOneKpt; j++) {  // stable within the warp's keys
      const bool valid = first + 32 * j < n;
      const uint32_t d = valid ? (key[j] >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const uint32_t before = valid ? wcount[w][d] : 0u;
      __syncwarp();
      if (valid && (peers & lt) == 0u) wcount[w][d] = before + __popc(peers);
      __syncwarp();
      rank[j] = before + __popc(peers & lt);
    }
    __syncthreads();
    // the warps' counts of each digit become their starts among the tile's
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < kOneWarps / kOneSplit; k++) {
      const int ww = split * (kOneWarps / kOneSplit) + k;
      const uint32_t t = wcount[ww][digit];
      wcount[ww][digit] = run;
      run += t;
    }
    part[split][digit] = run;
    __syncthreads();
    uint32_t tile = 0, mine = 0;
#pragma unroll
    for (int k = 0; k < kOneSplit; k++) {
      if (k == split) mine = tile;
      tile += part[k][digit];
    }
    if (split == 0) __stcg(hist + blockIdx.x * 256 + digit, tile);
    if (!grid_meet<LIMITED>(bars + 2 * pass, wait)) return;
    uint32_t total = 0, before = 0;
#pragma unroll 8
    for (int c = split; c < (int)gridDim.x; c += kOneSplit) {
      const uint32_t t = __ldcg(hist + c * 256 + digit);
      total += t;
      if (c < (int)blockIdx.x) before += t;
    }
    part[split][digit] = total;
    ahead[split][digit] = before;
    __syncthreads();
    // exclusive scan of the digits' totals (by the first 256 threads) plus what
    // the tiles before this one hold of the digit
    uint32_t sum = 0, lead = 0, incl = 0;
    if (split == 0) {
#pragma unroll
      for (int k = 0; k < kOneSplit; k++) {
        sum += part[k][digit];
        lead += ahead[k][digit];
      }
      incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) wsum[w] = incl;
    }
    __syncthreads();
    if (split == 0) {
      uint32_t off = 0;
      for (int k = 0; k < w; k++) off += wsum[k];
      part[0][digit] = off + incl - sum + lead;
    }
    __syncthreads();
    // the starts: of the digit, of the tile's share, of the warp's
    {
      const uint32_t base = part[0][digit] + mine;
#pragma unroll
      for (int k = 0; k < kOneWarps / kOneSplit; k++) wcount[split * (kOneWarps / kOneSplit) + k][digit] += base;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kOneKpt; j++) {
      if (first + 32 * j >= n) continue;
      const uint32_t pos = wcount[w][(key[j] >> shift) & 255u] + rank[j];
      __stcg(sorted + pos, key[j]);
      __stcg(perm + pos, val[j]);
    }
    if (pass + 1 < passes && !grid_meet<LIMITED>(bars + 2 * pass + 1, wait)) return;
  }
}

// The driver's id of the calling thread's current context (0 if none). Ids
// are never reused in a process, so a context created after a reset (which
// reloads the module and moves g_sort_scratch) gets a new id.
unsigned long long current_context_id() {
  using GetCurrent = int (*)(void**);
  using GetId = int (*)(void*, unsigned long long*);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static bool looked_up = false;
  if (!looked_up) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f);
    looked_up = true;
  }
  void* c = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&c) != 0 || !c || get_id(c, &id) != 0) return 0;
  return id;
}

// Device address of g_sort_scratch in the current context. Host code only
// sees a host-side stand-in for the symbol, so the address is looked up
// (cudaGetSymbolAddress) and cached per context: a reset of the device's
// primary context reloads the module at another address, and the new
// context's different id makes the cache look the address up again.
cudaError_t static_scratch(uint32_t** out) {
  static std::mutex mu;
  static unsigned long long ctx_id[64] = {};
  static uint32_t* addr[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  const unsigned long long id = current_context_id();
  if (!addr[dev] || id == 0 || id != ctx_id[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_sort_scratch);  // also makes the primary context current
    if (e != cudaSuccess) return e;
    addr[dev] = static_cast<uint32_t*>(p);
    ctx_id[dev] = current_context_id();
  }
  *out = addr[dev];
  return cudaSuccess;
}

// Whether the byte ranges [a, a + n) and [b, b + n) of 32-bit words overlap.
bool ranges_overlap(const void* a, const void* b, size_t n) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  const uintptr_t bytes = n * sizeof(uint32_t);
  return x < y + bytes && y < x + bytes;
}

snow_status sort_static(const uint32_t* keys, uint32_t* sorted_keys, uint32_t* perm, size_t n, int key_bits, void* stream,
                        const SortWait* limited) {
  if (!keys || !sorted_keys || !perm || key_bits < 1 || key_bits > 32) return SNOW_EINVAL;
  if (n > kStaticKeys) return SNOW_EINVAL;
  if (n == 0) return SNOW_OK;
  // every CTA reads its keys before any writes (keys and sorted_keys may
  // coincide, but then exactly); perm may share memory with neither
  if (ranges_overlap(perm, keys, n) || ranges_overlap(perm, sorted_keys, n) ||
      (keys != sorted_keys && ranges_overlap(keys, sorted_keys, n)))
    return SNOW_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* scratch = nullptr;
  if (static_scratch(&scratch) != cudaSuccess) {
    cudaGetLastError();
    return SNOW_ECUDA;
  }
  uint32_t* bars = scratch + (size_t)kOneCtas * 256;
  uint32_t count = (uint32_t)n;
  int passes = (key_bits + 7) / 8;
  SortWait wait = limited ? *limited : SortWait{};
  const void* kernel = limited ? reinterpret_cast<const void*>(&k_sort_one<true>) : reinterpret_cast<const void*>(&k_sort_one<false>);
  void* args[] = {&keys, &sorted_keys, &perm, &count, &passes, &scratch, &bars, &wait};
  const unsigned ctas = (unsigned)((n + kOneTile - 1) / kOneTile);
  if (cudaMemsetAsync(bars, 0, kOneBarriers * sizeof(uint32_t), st) != cudaSuccess ||
      cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(kOneThreads), args, 0, st) != cudaSuccess) {
    cudaGetLastError();
    return SNOW_ECUDA;
  }
  if (cudaGetLastError() != cudaSuccess) return SNOW_ECUDA;
  return SNOW_OK;
}

}  // namespace
}  // namespace snow

extern "C" snow_status snow_sort_keys_static(const uint32_t* keys, uint32_t* sorted_keys, uint32_t* perm, size_t n,
                                             int key_bits, void* stream) {
  return snow::sort_static(keys, sorted_keys, perm, n, key_bits, stream, nullptr);
}

extern "C" snow_status snow_sort_keys_static_limited(const uint32_t* keys, uint32_t* sorted_keys, uint32_t* perm,
                                                     size_t n, int key_bits, void* stream, uint32_t wait_ns,
                                                     uint32_t absent) {
  const snow::SortWait wait = {wait_ns ? wait_ns : snow::kDefaultWaitNs, absent};
  return snow::sort_static(keys, sorted_keys, perm, n, key_bits, stream, &wait);
}

extern "C" snow_status snow_sort_static_check(void* stream) {
  using namespace snow;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* scratch = nullptr;
  uint32_t expired = 0;
  cudaError_t e = static_scratch(&scratch);
  uint32_t* word = scratch + kSortExpired;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&expired, word, sizeof expired, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && expired) e = cudaMemsetAsync(word, 0, sizeof expired, st);
  if (e == cudaSuccess && expired) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return SNOW_ECUDA;
  }
  return expired ? SNOW_ETIMEDOUT : SNOW_OK;
}
