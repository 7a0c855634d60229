// Internal interfaces between the host runtime (snow_api.cpp) and the CUDA
// kernel files (ref_kernels.cu, fast_kernels.cu, sort.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/snow_mpm.h"

namespace snow {

// ---------------------------------------------------------------------------
// Reference mode: the shaders' buffers, byte for byte (std140).
// ---------------------------------------------------------------------------
struct RefArgs {
  float gpos[3];
  int dim[3];
  float h;
  float young, poisson, hardening, crit_c, crit_s, alpha;
  float grav[3];
  int ncoll;
  snow_collider* coll;
  int n;
  float4* pxm;   // (x, m)
  int4* pv;      // (v * 1e8, rho0 * 1e6)
  float4* pfe;   // mat4 per particle, 4 columns
  float4* pfp;
  int4* pvn;     // G2P accumulators (g2pTransfer.glsl bindings 6, 13-15)
  int4* pd0;
  int4* pd1;
  int4* pd2;
  long long G;
  int4* gv;      // (p * 1e8, m * 1e8)
  int4* gf;      // (f * 1e6, 0)
  float4* gvn;   // (v*, 0)
};

void ref_rigid(snow_collider* coll, int ncoll, float dt, cudaStream_t st);
void ref_reset(const RefArgs& a, cudaStream_t st);
void ref_p2g(const RefArgs& a, bool mass_only, cudaStream_t st);
void ref_volume(const RefArgs& a, cudaStream_t st);
void ref_grid(const RefArgs& a, float dt, cudaStream_t st);
void ref_g2p(const RefArgs& a, cudaStream_t st);
void ref_advance(const RefArgs& a, float dt, cudaStream_t st);

// ---------------------------------------------------------------------------
// Fast mode.
// ---------------------------------------------------------------------------
constexpr int kBlockNodes = 64;            // 4 x 4 x 4 nodes per grid block
constexpr int kAccFields = 7;              // m, p (3), f (3)
constexpr int kOutFields = 6;              // v* (3), d = v* - alpha p/m (3)
// acc holds the P2G sums as integers (fixed point at per-scene power-of-two
// scales): per node seven int64 words (m, p_x, p_y, p_z, f_x, f_y, f_z),
// stored word-major per block. No node sum can leave the int64 range (each
// contribution is below 2^22 or, on the wide path, 2^62), however many
// particles pile into a cell.
constexpr int kAccWords = kAccFields;
constexpr int kAccBlockWords = kAccWords * kBlockNodes;    // 448 (3584 bytes)
constexpr int kOutBlockFloats = kOutFields * kBlockNodes;  // 384: a block's share of gout

// Fixed-point state of one scene's P2G sums. Magnitudes are the bits of
// non-negative floats (they order like unsigned ints, so atomicMax records
// maxima); every value here is an order-independent function of the state.
struct FixState {
  float scale[3];     // s_m, s_p, s_f of the sums now in acc (integer = round(contribution * s))
  uint32_t m_prev;    // largest particle mass, |v| and force-term bound a of the particles the
  uint32_t v_prev;    //   previous P2G scattered (a = max over rows r of |A_r0| + |A_r1| + |A_r2|)
  uint32_t a_prev;
  uint32_t m_cur;     // the same, recorded by the P2G in flight (moved to *_prev at each step's start)
  uint32_t v_cur;
  uint32_t a_cur;
  uint32_t v0max;     // largest initial particle volume
  uint32_t wide;      // particles scattered with int64 contributions (outgrew the fast range), cumulative
  float next[3];      // s_m, s_p, s_f of the step's P2G, formed at the step's start
};

// Per-scene counters (int32), one row of kCounterStride per scene.
enum {
  CNT_ACTIVE = 0,     // active grid blocks this step
  CNT_OVERFLOW = 1,   // blocks that found no slot in the pool
  CNT_ITEMS = 2,      // P2G work items since the last binning
  CNT_NONFINITE = 3,  // particles with a non-finite field (cumulative since the set-up)
  CNT_HOME = 4,       // unused
  CNT_FALLBACK = 5,   // particles that left their P2G tile and that a binning would help (cumulative)
  CNT_TIMEOUT = 6,    // bounded waits that ran out (cumulative)
  CNT_DONE = 7,       // CTAs of the compaction finished (the last forms the prefixes)
  CNT_BINNED = 8,     // 1: this step's binning left the particles in the binned copies
  CNT_WORK = 9,       // hands out the fused kernel's work to its CTAs (scene 0's)
  CNT_SLOTS = 10,     // slots the compaction has given out (zero between compactions)
  kCounters = 11,
  kFixOffset = 16,    // a scene's FixState follows its counters (one copy reads both)
  kCounterStride = 32
};

// Semi-implicit velocity solve: conjugate residuals on the mass-scaled form
// of (M + beta dt^2 K) v = M v* over the active nodes, one record per scene,
// cleared (up to `skipping`) at the start of each step. Iteration k
// (1-based) forms rAr[k] = (r_{k-1}, A r_{k-1}), ApAp[k] = |A p_{k-1}|^2 and
// rr[k] = |r_k|^2. A step whose initial residual is below
// kCrSkipFactor * tolerance makes the next steps skip the solve: they take
// v = v*, which is what a solve that exits at iteration 0 gives, without
// evaluating K v*; the step after them checks again. The skip lasts
// kCrSkipSteps steps, doubled for each further factor of 10 the residual
// lies below the threshold, up to kCrSkipSteps * 2^kCrSkipDoublings.
constexpr int kCrMaxIters = 128;
constexpr int kCrSkipSteps = 15;
constexpr int kCrSkipDoublings = 4;
constexpr double kCrSkipFactor = 1e-3;
struct CrScalars {
  double bb;                   // |M^1/2 v*|^2
  double rr[kCrMaxIters + 1];  // rr[0]: the initial residual
  double rAr[kCrMaxIters + 1];
  double ApAp[kCrMaxIters + 1];
  int iters;                   // iterations taken
  int skipping;                // 1: this step skips the solve
  int skip_left;               // steps still to skip (kept across steps)
  int pad;
};
constexpr int kImpFields = 3;                              // u of the solve: one 3-vector per node
constexpr int kImpBlockFloats = kImpFields * kBlockNodes;  // 192: a block's share of cru
constexpr uint32_t kDefaultWaitNs = 1000000000u;   // one second

// Device-resident description of one FAST scene (read by every kernel).
struct SceneDev {
  float gpos[3];
  float h;
  float inv_h;  // 1 / h (FAST kernels multiply instead of dividing)
  int dim[3];
  int bdim[3];
  int nblocks;
  float young, poisson, hardening, crit_lo, crit_hi, alpha;
  float mu0, lambda0;  // Lame parameters at J_p = 1 (lame.include.glsl:11-27)
  float grav[3];
  float dt;
  int ncoll;
  snow_collider* coll;
  int n;
  // particle streams (SoA): xm = (x, m), vv = (v, V0),
  // fa = (FE00, FE10, FE20, FE01), fb = (FE11, FE21, FE02, FE12),
  // fc = (FE22, Jp); FE stored column-major (m[c][r]).
  float4* xm;
  float4* vv;
  float4* fa;
  float4* fb;
  float2* fc;
  float4* vq;       // FAST: the Jacobi frame (quaternion) of each particle's last SVD
  uint32_t* pid;    // upload index of the particle now stored at each slot
  // the binning's permuted copies of xm, vv, fa, fb, fc, vq: a binning inside
  // a step leaves the particles there (counters[CNT_BINNED] = 1), and the
  // kernels of that step read them from there until the fused kernel, which
  // writes every particle, has put them back into the streams above
  float4* bxm;
  float4* bvv;
  float4* bfa;
  float4* bfb;
  float2* bfc;
  float4* bvq;
  uint32_t* bpid;
  // binning (k_bin_*): per particle its key and its place among its block's,
  // and the block-ordered particle indices and keys; per block its count (zero
  // between binnings) and range; per kBinChunk blocks their count; most
  // particles per work item
  uint32_t* bkey;
  uint32_t* brank;
  uint32_t* bidx;
  uint32_t* bskey;
  int* bcount;
  int* bstart;
  int* bend;
  int* bchunk;
  int nchunks;
  int items_max;
  // blocked grid
  int* blk_slot;    // nblocks: pool slot of the block this step, -1 if inactive
  int* blk_flag;    // nblocks: block received P2G sums since the last compaction
  unsigned long long* acc;  // nblocks x 448 words: the fixed-point P2G sums, word-major per block (dense)
  FixState* fix;            // their scales and the magnitudes the next scales are chosen from
  int* active;      // pool_cap: block id of each slot
  // grid-update output, dense over the nodes of the blocked grid (4 bdim per
  // axis, x fastest), per node (v*, d) as 6 floats; zero in blocks that are
  // not active, so that a node without mass reads as zero
  float* gout;
  int pool_cap;
  // P2G work items: (home block, first particle, count, and in a block's first
  // item the number of its items, else minus its place among them)
  int4* items;
  int item_cap;
  int* counters;    // kCounterStride ints
  // bounded waits for bulk copies into shared memory: give up after wait_ns
  // nanoseconds; tx_unsent (0 in normal use) is added to the bytes each such
  // wait expects, so that it runs out (a test of the timeout path)
  uint32_t wait_ns;
  uint32_t tx_unsent;
  // semi-implicit velocity solve (crs == nullptr: the scene steps explicitly)
  float imp_beta;   // beta of (M + beta dt^2 K) v = M v*
  float imp_tol;    // stop once |r| <= imp_tol |M^1/2 v*| (r of the mass-scaled system)
  int imp_maxit;    // at most this many iterations per step
  float4* crv;      // 3 planes of pool_cap x 64 float4 per node: (v, m), (p, 0), (A p, 0)
  float* cru;       // u = M^-1/2 r (the vector K is applied to), 3 floats per node, dense as gout
  CrScalars* crs;
};

// Re-binning intervals when the caller names none, and the steps between the
// host's looks at the device counters.
constexpr int kAutoInterval = 32;
constexpr int kCheckSteps = 8;
struct FastTuning {
  int sort_interval = kAutoInterval;  // re-bin particles at least every k steps ...
  bool chosen = false;                // ... asked for by the caller (else chosen from the speeds, up to kAutoInterval)
  int items_max = 256;    // most particles per work item (kMinItemMax .. kItemMax) ...
  bool items_chosen = false;  // ... asked for by the caller (else fewer where all items then run at once, size_choice)
  int ctas_per_sm = 2;    // work-item CTAs launched per SM (1 .. kItemCtas)
};
constexpr int kMinItemMax = 64;
// Threads of a work-item CTA (one particle each) and CTAs resident per SM:
// registers (128 a thread) fit 16 warps an SM in any shape. 2 x 256 threads
// against 3 x 160, 3 x 192 (96 registers, 0.4 KB of spills a thread) and
// 2 x 320 (the same): 0.237 ms a step's fused kernel at 1M particles, 256^3,
// against 0.26, 0.27 and 0.28.
constexpr int kItemMax = 256;
constexpr int kItemCtas = 2;

// Work spaces over nscenes scenes: prefix[s] .. prefix[s+1] are scene s's units
// (P2G work items, active blocks, particles, quads and chunks of grid
// blocks), in one device array of five prefixes of nscenes + 1 entries. Item
// and active-block counts are only known on the device; the binning and the
// compaction form those two prefixes there. The binning's item counts at each
// size follow them.
struct WorkSpace {
  const SceneDev* scenes;
  int nscenes;
  int* items;
  int* active;
  const int* particles;
  const int* quads;
  const int* chunks;
  long long total_particles, total_quads, total_chunks;
  int fit;     // CTAs that the items are fitted to (0: the scenes' items_max as it is)
  int* sizes;  // items there would be at each size_choice (zero between binnings)
};
constexpr int kWorkPrefixes = 5;
// Item sizes that a binning of few particles chooses from: the smallest at which
// the items take no more rounds of the fused kernel's CTAs than at the largest, if
// those are at most kFitRounds. A round lasts as long as its largest items, whose
// time falls with their size down to about 96 (below, their fixed part outweighs
// it), and a size that needs a round more loses 5 to 25%. A step with items of up
// to 256 and as chosen: 4k particles 26.8 to 23.3 us, 32k 33.2 to 29.9, 65k 49.9
// to 42.3, 80k 50.7 to 46.5, 131k 63.7 to 60.4, the same from 160k on.
constexpr int kSizeChoices = 8;
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int size_choice(int k) { return k <= 4 ? 96 + 16 * k : 160 + 32 * (k - 4); }
constexpr int kFitRounds = 3;
// Whether a binning of n particles over `ctas` CTAs looks for one.
inline bool fits_items(long long n, int ctas) { return n <= (long long)kFitRounds * ctas * size_choice(kSizeChoices - 1); }
constexpr int kBinChunk = 512;  // grid blocks per chunk of the binning's scan
// Moves a scene's colliders by dt * velocity (rigidAdvance.glsl:14-18). A step's
// compaction does the same in its first CTAs.
void fast_rigid(const SceneDev* sd_dev, cudaStream_t st);
// Copies every scene's counters and FixState into out[s * kCounterStride ...] (mapped
// pinned memory: a batch reads them one re-binning interval later, without
// draining the stream).
void fast_gather_counters(const SceneDev* scenes, int nscenes, int* out, cudaStream_t st);
// Flags -> active list and slots; its first CTAs start the step of every scene
// (counters, scales of the step's P2G; rigid: the colliders), and the CTA that takes
// its slots last forms the item and active-block prefixes. binned: the step's binning
// ran before and left the particles in the binned copies. set_up: of a new state, for
// which no solve may be skipped on account of the last.
void fast_compact(const WorkSpace& w, bool rigid, bool binned, bool chained, cudaStream_t st, bool set_up = false);
// P2G of the stored particle state (set-up, per-kernel dispatches), after a
// pass over the particles that measures the magnitudes its fixed-point
// scales are chosen from.
void fast_p2g(const SceneDev* scenes, const SceneDev& sd_host, const int* item_prefix, int nscenes, int grid_ctas,
              bool mass_only, cudaStream_t st);
void fast_grid(const SceneDev* scenes, const int* active_prefix, int nscenes, int grid_ctas, bool clear_only,
               bool chained, cudaStream_t st);
void fast_volume(const SceneDev* sd_dev, const int* item_prefix, int n, cudaStream_t st);
void fast_g2p_advance(const SceneDev* scenes, const int* item_prefix, int nscenes, int grid_ctas, cudaStream_t st);
// binned: some scene of the launch was re-binned in this step (its particles
// are in its binned copies)
void fast_g2p2g(const SceneDev* scenes, const int* item_prefix, int nscenes, int grid_ctas, bool binned,
                bool wide, bool chained, cudaStream_t st);
// The semi-implicit velocity solve between the grid update (which leaves
// v*, m and u = v* in the solver planes) and G2P: iterations of conjugate
// residuals (each a K u pass over the items and three passes over the active
// nodes) until every scene has converged or reached its cap, then the
// colliders on v and v, d written back into gout. Scenes without a solver
// record are left alone. d_iter is a device int (the iteration counter).
// When `st` is capturing a graph the whole solve is the body of a
// conditional IF node (captured on `gate`), taken when any scene solves in
// this step, and its iterations a conditional WHILE node inside it (body
// captured on `body`; both streams not otherwise in use); otherwise
// max_iters iterations are launched.
void fast_implicit_solve(const SceneDev* scenes, const int* item_prefix, const int* active_prefix, int nscenes,
                         int max_iters, int item_ctas, int grid_ctas, int* d_iter, cudaStream_t body,
                         cudaStream_t gate, cudaStream_t st);
// Kernel attributes of the solve (outside any stream capture).
void fast_implicit_setup();

// Launches k after the kernel launched before it in st. chained: that kernel is
// one that calls chain_next and chain_wait, and nothing lies between the two; k's
// CTAs then start once all of that kernel's have started (as far as there is
// room) and set themselves up while it runs. Every thread of such a kernel calls
// chain_wait before it reads or writes global memory: it returns when the kernel
// before has finished, which by then has waited for the one before it. What these
// kernels read and another of them wrote is read by plain loads, through pointers
// that are not __restrict__ (a load of read-only memory could move above the
// wait); the scenes' descriptors are written by copies, which nothing is chained to.
// It takes launches and the kernels' set-up out of a short step: one step of 4k
// particles with its download 56 to 54 us, 100 steps of 32k 3.70 to 3.64 ms, 20
// steps of 300k with a binning in most 3.20 to 3.16. The gain ends near the limit, and
// longer steps lose (plain to chained, as many steps as take about 15 ms): 524k
// particles 8.97 to 8.91 ms, 1M 16.42 to 16.37, 1.5M 15.25 both, 2M 15.07 to 15.12, 4M
// 14.70 to 14.76, 8M 14.45 both, 16M 28.73 to 28.81; batches of 1.6M, 4M and 8M
// particles in all the same either way.
constexpr long long kChainParticles = 1 << 20;
template <typename... P, typename... A>
inline void launch_after(bool chained, void (*k)(P...), int grid, int block, int smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = (size_t)smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

// While `st` captures a graph: appends a conditional node (IF or WHILE) on
// `cond` after the work captured so far, and captures `fill`'s launches on
// `body` (a stream not otherwise capturing) as the node's body. Returns
// false when `st` is not capturing or a call failed (a failure also
// invalidates the capture, which then fails at its end).
template <class Fill>
bool capture_conditional(cudaStream_t st, cudaGraphConditionalHandle cond, cudaGraphConditionalNodeType type,
                         cudaStream_t body, Fill fill) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t ndeps = 0;
  if (cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, nullptr, &ndeps) != cudaSuccess ||
      cs != cudaStreamCaptureStatusActive)
    return false;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = cond;
  p.conditional.type = type;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if (cudaGraphAddNode(&node, g, deps, nullptr, ndeps, &p) != cudaSuccess ||
      cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies) != cudaSuccess ||
      cudaStreamBeginCaptureToGraph(body, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                    cudaStreamCaptureModeThreadLocal) != cudaSuccess)
    return false;
  fill(body);
  cudaGraph_t out = nullptr;
  return cudaStreamEndCapture(body, &out) == cudaSuccess;
}
// A conditional handle on the graph `st` is capturing (false if none).
inline bool capture_handle(cudaStream_t st, cudaGraphConditionalHandle* cond) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaGraph_t g = nullptr;
  if (cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr, nullptr) != cudaSuccess ||
      cs != cudaStreamCaptureStatusActive)
    return false;
  return cudaGraphConditionalHandleCreate(cond, g, 0, cudaGraphCondAssignDefault) == cudaSuccess;
}

// Scratch of a scene's binning and of the radix sort of its cell keys.
struct BinScratch {
  uint32_t* keys[2];
  uint32_t* vals[2];
  uint32_t* hist;      // 256 x tiles
  uint32_t* scan_tmp;  // partial sums of the scan
  float4* tmp4[5];     // permutation targets for xm, vv, fa, fb, vq
  float2* tmp2;        // ... and fc
  uint32_t* tmp_pid;   // ... and pid
  size_t n_cap;
};
size_t radix_tiles(size_t n);
// Sorts (key, index) pairs for the first n particles of scene `sd` (a host
// copy of the device descriptor) and leaves the sorted keys in keys[0] and
// the permutation in vals[0].
void fast_sort_keys(const SceneDev& sd, const SceneDev* sd_dev, BinScratch& b, int key_bits, cudaStream_t st);
// Binning of every scene of the work space: particles into the order of the
// stable sort by cell key, work items, the item prefix. copy_back false: the
// particles stay in the binned copies (CNT_BINNED) for the step's fused kernel,
// which must follow in the same step.
void fast_bin_scenes(const WorkSpace& w, bool copy_back, bool chained, cudaStream_t st);

// Radix sort of arbitrary (key, value) pairs; the result lands in k[0]/v[0].
void radix_sort_pairs(uint32_t* k[2], uint32_t* v[2], size_t n, int key_bits, uint32_t* hist, uint32_t* scan_tmp,
                      cudaStream_t st, int start = 0);  // start: the buffer holding the input

// Bulk statistics of one scene.
struct StatsAccum {
  double mass, mom[3], ke, com[3], jp;
  int bmin_key[3], bmax_key[3];  // order-preserving int keys of the bbox floats
  unsigned long long nonfinite;
};
// Per-block partial sums of one statistics read and the counter of blocks
// that have written theirs. The kernel's last block sums the partials in
// block order (the result does not depend on which block finished when),
// writes the totals to `host` (mapped pinned memory, read after the stream
// passes the kernel) and resets the counter, so a read needs no copy in
// either direction.
constexpr int kStatsMaxBlocks = 1024;
struct StatsBlockSum {
  double acc[9];  // mass, momentum x3, kinetic energy, mass-weighted position x3, sum J_p
  float bmin[3], bmax[3];
  unsigned long long bad;
};
struct StatsSlot {
  StatsBlockSum part[kStatsMaxBlocks];
  unsigned int done;
};
void fast_stats(const SceneDev* sd_dev, int n, StatsSlot* slot, StatsAccum* host, cudaStream_t st);
void ref_stats(const RefArgs& a, StatsSlot* slot, StatsAccum* host, cudaStream_t st);
void fast_download_grid(const SceneDev* sd_dev, float* mass, float* mom, float* force, float* vstar, cudaStream_t st);
void fast_pack(const float* x, const float* v, const float* m, const float* FE, const float* FP, size_t n,
               const SceneDev& sd, cudaStream_t st);
// slot: n words of scratch
void fast_unpack(const SceneDev* sd_dev, size_t n, uint32_t* slot, float* x, float* v, float* FE, float* Jp,
                 float* volume, cudaStream_t st);

constexpr int kMaxDevices = 64;
// The calling thread's current device (0 .. kMaxDevices - 1).
int current_device();
int num_sms();

}  // namespace snow
