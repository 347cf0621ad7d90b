// small.cu -- the unbinding loop of small subhaloes, one thread block or one warp
// per subhalo.
//
// Subhalo_t::Unbind (src/subhalo_unbind.cpp:263-431) iterates until the bound
// count converges.  The batch path (loop.cu, tree.cu, walk.cu) advances every
// active subhalo of a call by one pass per round of ~40 launches, so the round
// count is set by the slowest subhalo, and a round costs its launches however
// little it holds.  This kernel runs a subhalo's passes to the end on the device:
// tree, walk, partition, averages and decisions, one step after another with
// barriers between them.  It is used
//   * for a whole call whose subhaloes all hold at most `cap` particles
//     (launch_small_call): the kernel also sets the lists up and writes the
//     results, so the call is one copy of the states and one launch;
//   * from the first round of a larger call at which every active energy list
//     holds at most `cap` particles (launch_small): in the 2000-subhalo workload
//     the larger subhaloes converge in 2-3 passes, and a few dozen of under 512
//     particles need 4-7.
//
// Split.  Sizes fall as N^-0.9, so most lists hold a few dozen particles: a list of
// up to kSmallWarpCap particles takes a warp (two or four when there are few), one of
// up to kSmallMediumCap four warps (or eight), a longer one a block of kSB threads,
// or a cluster of blocks when the chip has room: its first block does every step but
// the walk, whose targets are spread over all of them.  Each class has a
// queue in size order (an atomic counter hands out the next list).  A block of 256
// threads per list, one per SM, spent its time in barriers and latency with
// most lanes idle: 20,000 subhaloes of 20-500 particles took 16.7 ms in this
// kernel and 19.8 ms in all, now 3.1 and 3.4; 400 of 20-1200: 1.93 -> 0.69 ms; one of
// 380: 0.52 -> 0.33 ms; one of 1,920: 2.9 -> 0.75 ms.
//
// Registers.  Two blocks of 512 threads per SM leave 64 per thread, and the kernel
// spills (404 bytes stored, 496 loaded in FP32 and 492 in FP64; 440 and 448 bytes of
// stack).  Many lists need both blocks; a call of few lists has the spills on its
// chain for nothing (another budget for those: not measured).
//
// Double arithmetic (frames, moments, divisions) runs at 1/64 of the FP32 rate
// and a dependent double add takes about 150 cycles, so the steps keep it
// off the serial chains: the moments go from the leaves up, every cell as
// soon as its child cells are done (as many steps as the tree is high, not as
// it is deep), and a warp's lanes share divisions.
//
// The steps are the batch kernels' own per-element functions (tree_ops.cuh,
// walk_ops.cuh, loop_ops.cuh) on the subhalo's slice of the same buffers, so
// every result is bit for bit the batch path's:
//   * the tree keys and the energy keys are sorted with the list index in their low
//     bits: the order of the batch path's stable radix sort;
//   * the frame and final sums are block_sum's: per chunk of 1024, the partial sums
//     of 8 groups of 32 list positions, added in order.
#include "loop_ops.cuh"
#include "tree_ops.cuh"
#include "walk_ops.cuh"

#include <algorithm>
#include <cstddef>

namespace hbtu {
namespace {

typedef unsigned long long ull;

constexpr int kSB = 512;  // threads of a block: one round of targets for most lists
constexpr int kWarps = kSB / 32;
constexpr int kMT = 128;  // threads that share a medium list
constexpr int kPer = 4;   // list positions a thread holds while permuting
static_assert(kSmallCap <= kPer * kSB && kSmallMediumCap <= kPer * kMT && kSmallWarpCap <= kPer * 32,
              "a group's threads hold its longest list");
constexpr int kMaxCluster = 8;
constexpr int kSumGroups = kLB / 32;  // the warps of a chunk-sum block

__host__ __device__ constexpr int pow2_at_least(int n)
{
  int p = 32;
  while (p < n) p <<= 1;
  return p;
}

// Shared memory of one subhalo's group of T threads, for lists of up to `cap`.
struct SmallLayout {
  size_t key0, key1, val0, val1, part, seg, ctr, bytes;
  explicit __host__ __device__ SmallLayout(int cap, bool warp = false)
  {
    // the bitonic sort pads to a power of two
    const size_t n1 = (size_t)(warp ? (cap + 1) / 2 * 2 : pow2_at_least(cap)) + 1;
    const size_t groups = cap > kChunk ? 2 * kSumGroups
                                       : (cap + 31) / 32 < kSumGroups ? (cap + 31) / 32 : kSumGroups;
    key0 = 0;
    key1 = key0 + 8 * n1;
    part = key1 + 8 * n1;
    seg = part + 8 * 18 * groups;
    val0 = seg + (sizeof(SegState) + 7) / 8 * 8;
    val1 = val0 + 4 * n1;
    ctr = val1 + 4 * n1;
    bytes = (ctr + 16 * sizeof(int) + 15) / 16 * 16;
  }
};

// One subhalo's group of T threads: 32 (a warp), kMT (four warps) or kSB (the
// block).  T is a runtime value: with one instance of the code per T the kernel
// outgrew the instruction cache (a quarter of the warps' stalls).
struct Group {
  int T, tid, bar;
  ull *key0, *key1;
  int *val0, *val1, *ctr;
  double *part;
  SegState *sg;
  __device__ __forceinline__ Group(int threads, unsigned char *mem, const SmallLayout &L)
  {
    T = threads;
    tid = threadIdx.x & (T - 1);
    bar = T == kSB ? 0 : 1 + threadIdx.x / T;
    key0 = reinterpret_cast<ull *>(mem + L.key0);
    key1 = reinterpret_cast<ull *>(mem + L.key1);
    part = reinterpret_cast<double *>(mem + L.part);
    sg = reinterpret_cast<SegState *>(mem + L.seg);
    val0 = reinterpret_cast<int *>(mem + L.val0);
    val1 = reinterpret_cast<int *>(mem + L.val1);
    ctr = reinterpret_cast<int *>(mem + L.ctr);
  }
  __device__ __forceinline__ void sync() const
  {
    if (T == 32)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(T) : "memory");
  }
};

// Shared memory of four warps: a medium list's group, or a short list each.
__host__ __device__ inline size_t quad_bytes(int cap)
{
  const size_t a = SmallLayout(cap < kSmallMediumCap ? cap : kSmallMediumCap).bytes;
  const size_t b = 4 * SmallLayout(cap < kSmallWarpCap ? cap : kSmallWarpCap, true).bytes;
  return a > b ? a : b;
}

// The size classes of a call, from its numbers of lists longer than kSmallMediumCap,
// of medium ones and of short ones (at most kSmallWarpCap), for a chip that holds
// `blocks` blocks: bound[k]: lists longer than bound[0] are large, than bound[1] medium;
// T[k]: threads of a group.  Many lists: the fewest threads that hold one,
// since groups wait for their own chains of steps and many of them hide that.  Fewer
// lists than the chip has room for: more threads each.  A handful: a block or a
// cluster for any but the shortest.
struct SmallClasses {
  int bound[2], T[3];
};
__host__ __device__ inline SmallClasses small_classes_of(int large, int medium, int small, int blocks)
{
  SmallClasses q = {{kSmallMediumCap, kSmallWarpCap}, {kSB, kMT, 32}};
  if (large + medium + small <= blocks / 8) q.bound[0] = 64;
  if (medium <= 2 * blocks) q.T[1] = 2 * kMT;
  if (small <= 4 * blocks)
    q.T[2] = 128;
  else if (small <= 8 * blocks)
    q.T[2] = 64;
  if (q.bound[0] < q.bound[1]) q.bound[1] = q.bound[0];
  return q;
}

struct SmallJobs {
  const int *list[3];  // large, medium, short
};

// Exclusive scan of in[0..n1) in place, each thread taking a contiguous run.
__device__ void group_scan(const Group &g, long long *x, int n1)
{
  __shared__ long long ws[kWarps];
  const int per = (n1 + g.T - 1) / g.T;
  const int b = g.tid * per, e = min(n1, b + per);
  long long loc = 0;
  for (int k = b; k < e; k++) loc += x[k];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long inc = loc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  long long run = inc - loc;
  if (g.T != 32) {
    if (lane == 31) ws[w] = inc;
    g.sync();
    for (int k = w & ~(g.T / 32 - 1); k < w; k++) run += ws[k];
  }
  for (int k = b; k < e; k++) {
    const long long v = x[k];
    x[k] = run;
    run += v;
  }
  g.sync();
}

// n distinct keys of a sorted ascending; the result is in the array returned
// (a or b).  Few keys: the rank of each by counting; else a bitonic network.
__device__ ull *group_sort(const Group &g, ull *a, ull *b, int n)
{
  if (g.T == 32 || n <= 160) {
    for (int i = g.tid; i < n; i += g.T) {
      const ull ki = a[i];
      int r = 0;
      for (int j = 0; j < n; j++) r += a[j] < ki;
      b[r] = ki;
    }
    g.sync();
    return b;
  }
  const int m = pow2_at_least(n);
  for (int i = n + g.tid; i < m; i += g.T) a[i] = ~0ull;
  g.sync();
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int q = g.tid; q < m / 2; q += g.T) {
        const int i = 2 * q - (q & (j - 1));
        const ull x = a[i], y = a[i + j];
        if ((x > y) == ((i & k) == 0)) {
          a[i] = y;
          a[i + j] = x;
        }
      }
      g.sync();
    }
  return a;
}

// List positions [lo, hi) of the subhalo sorted by the energies in src,
// stable (the batch path's k_blk_* with the radix sort).
__device__ void sort_block(const Group &g, const Ctx &c, int P0, int lo, int hi,
                           const float *src)
{
  const int m = hi - lo;
  if (m <= 0) return;
  for (int i = g.tid; i < m; i += g.T)
    g.key0[i] = ((ull)float_key(src[P0 + lo + i]) << 32) | (unsigned)i;
  g.sync();
  const ull *s = group_sort(g, g.key0, g.key1, m);
  int pid[kPer];
  float E[kPer];
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int i = g.tid + k * g.T;
    if (i >= m) break;
    const int from = P0 + lo + (int)(unsigned)s[i];
    pid[k] = c.epid[from];
    E[k] = c.eE[from];
  }
  g.sync();
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int i = g.tid + k * g.T;
    if (i >= m) break;
    c.epid[P0 + lo + i] = pid[k];
    c.eE[P0 + lo + i] = E[k];
    c.epos_of_pid[pid[k]] = P0 + lo + i;
  }
  g.sync();
}

// One pass's octree over list positions [t0, t0 + ntree), in the element arrays
// from P0 and node slots from 2*P0.  First the cube and the keys in Morton order;
// the list positions in that order go to val1.  Returns the array of the sorted
// keys, key0 or key1.
__device__ __forceinline__ ull *tree_keys(const Group &g, const Ctx &c, int P0)
{
  SegState &sg = *g.sg;
  const int n = sg.ntree, t0 = sg.t0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int i = g.tid; i < n; i += g.T) {
    const float4 a = c.pm[c.epid[P0 + t0 + i]];
    mn[0] = fminf(mn[0], a.x);
    mn[1] = fminf(mn[1], a.y);
    mn[2] = fminf(mn[2], a.z);
    mx[0] = fmaxf(mx[0], a.x);
    mx[1] = fmaxf(mx[1], a.y);
    mx[2] = fmaxf(mx[2], a.z);
    const int e = P0 + i;
    c.mask[e] = 0ull;
    c.pending[e] = 0;
    int4 *slot = reinterpret_cast<int4 *>(c.cslot + first_slot(e));
    slot[0] = make_int4(-1, -1, -1, -1);
    slot[1] = make_int4(-1, -1, -1, -1);
  }
#pragma unroll
  for (int j = 0; j < 3; j++)
    for (int o = 16; o > 0; o >>= 1) {
      mn[j] = fminf(mn[j], __shfl_xor_sync(0xffffffffu, mn[j], o));
      mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], o));
    }
  if (g.T != 32) {
    __shared__ float bb[6][kWarps];
    if (lane == 0)
      for (int j = 0; j < 3; j++) {
        bb[j][w] = mn[j];
        bb[3 + j][w] = mx[j];
      }
    g.sync();
    if (g.tid == 0)
      for (int j = 0; j < 3; j++)
        for (int k = 1; k < g.T / 32; k++) {
          mn[j] = fminf(mn[j], bb[j][w + k]);
          mx[j] = fmaxf(mx[j], bb[3 + j][w + k]);
        }
  }
  if (g.tid == 0) seg_cube(sg, mn, mx, n == 0, c.P);
  g.sync();
  // keys in Morton order: the key's unused low bits hold the list index (where
  // they are too few, ranks by key and index)
  ull *sk = g.key1;
  const int ibits = 32 - __clz(max(n - 1, 1));
  const ull imask = (1ull << ibits) - 1ull;
  if (64 - 3 * sg.levels >= ibits) {
    for (int i = g.tid; i < n; i += g.T)
      g.key0[i] = seg_key(sg, c.pm[c.epid[P0 + t0 + i]]) | (ull)i;
    g.sync();
    sk = group_sort(g, g.key0, g.key1, n);
    for (int i = g.tid; i < n; i += g.T) {
      const ull k = sk[i];
      g.val1[i] = P0 + t0 + (int)(k & imask);
      sk[i] = k & ~imask;
    }
  } else {
    for (int i = g.tid; i < n; i += g.T) g.key0[i] = seg_key(sg, c.pm[c.epid[P0 + t0 + i]]);
    g.sync();
    for (int i = g.tid; i < n; i += g.T) {
      const ull ki = g.key0[i];
      int r = 0;
      for (int j = 0; j < n; j++) {
        const ull kj = g.key0[j];
        r += (kj < ki) | ((kj == ki) & (j < i));
      }
      g.key1[r] = ki;
      g.val1[r] = P0 + t0 + i;
    }
  }
  g.sync();
  return sk;
}

// Its nodes; xs: the free key array.
__device__ __forceinline__ void tree_nodes(const Group &g, const Ctx &c, int P0, const ull *sk,
                                           long long *xs)
{
  SegState &sg = *g.sg;
  const int n = sg.ntree;
  for (int i = g.tid; i < n - 1; i += g.T) karras_elem(c, sk, P0, n, i);
  g.sync();
  for (int i = g.tid; i < n; i += g.T) cells_elem(c, P0, n, P0 + i, sg.levels);
  g.sync();
  // prefix counts of the cells starting at each key (the batch path's k_popc +
  // scan), kept in shared memory: entry n of this subhalo's scan would be
  // entry 0 of the next subhalo's in the global array
  for (int i = g.tid; i <= n; i += g.T) xs[i] = i < n ? __popcll(c.mask[P0 + i]) : 0;
  g.sync();
  group_scan(g, xs, n + 1);
  for (int i = g.tid; i < n; i += g.T) {
    const int e = P0 + i;
    leaves_elem(c, sg, P0, n, e, c.pm[c.epid[g.val1[i]]], sk[i], xs);
    if (c.iscell[e]) cellnodes_elem(c, sg, P0, n, e, sk, xs);
  }
  if (g.tid < 2) g.ctr[g.tid] = 0;
  g.sync();
}

// Its moments from the leaves up: the list of cells whose child cells are all
// done (at `list`), and how many each other cell still waits for.
__device__ __forceinline__ void tree_moments(const Group &g, const Ctx &c, int P0, int *list)
{
  const SegState &sg = *g.sg;
  const int n = sg.ntree;
  int *rem = g.val0, *next = list + n;
  for (int i = g.tid; i < n; i += g.T)
    if (c.iscell[P0 + i]) {
      const int k = c.pending[P0 + i];
      rem[i] = k;
      if (k == 0) list[atomicAdd(&g.ctr[0], 1)] = i;
    }
  g.sync();
  for (int cur = 0;; cur ^= 1) {  // each step takes at least one cell off
    const int count = g.ctr[cur];
    if (count == 0) break;
    for (int k = g.tid; k < count; k += g.T) {
      const int i = list[k], e = P0 + i;
      cell_moment<false>(c, sg, e, c.cdepth[e]);
      const int p = c.pcell[e];
      if (p >= 0 && atomicSub(&rem[p - P0], 1) == 1) next[atomicAdd(&g.ctr[cur ^ 1], 1)] = p - P0;
    }
    g.sync();
    if (g.tid == 0) g.ctr[cur] = 0;
    int *t = list;
    list = next;
    next = t;
    g.sync();
  }
}

// The pass's energies: targets first, first + step, ... of the pass; val1 or, in
// the other blocks of a cluster, sval holds their list positions.
template <bool kFP64>
__device__ void walk_targets(const Group &g, const Ctx &c, int s, int P0, const int *sval,
                             int first, int step)
{
  const SegState &sg = *g.sg;
  const int tm = sg.tgt_mode;
  const int count = tm == 1 ? sg.coh_n : sg.ntgt;
  int total = 0;
  const int lane = threadIdx.x & 31;
  for (int w = first; w - lane < count; w += step) {  // whole warps
    int epos = 0, pid = 0;
    bool active = w < count;
    if (!active) {
    } else if (tm == 0) {  // full pass: tree leaves in Morton order
      epos = sval[w];
      pid = c.epid[epos];
      c.coh_pid[P0 + w] = pid;
    } else if (tm == 1) {  // correction pass: the last full pass's order, still bound
      pid = c.coh_pid[P0 + w];
      epos = c.epos_of_pid[pid];
      active = (epos - P0) < sg.ntgt;
    } else {
      epos = P0 + w;
      pid = c.epid[epos];
    }
    Target t;
    init_target<!kFP64>(c, sg, s, epos, pid, active, 2 * P0, t);
    int ninter = 0;
    const double pot =
        kFP64 ? walk_fp64(c, t, &ninter) : walk_lean<false, true>(c.nd, t, c.P, &ninter);
    finish_target(c, sg, t, pot);
    total += ninter;
  }
  total = __reduce_add_sync(0xffffffffu, total);
  if ((threadIdx.x & 31) == 0 && total)
    atomicAdd((ull *)&c.seg[s].interactions, (ull)total);
}

// PartitionBindingEnergy (src/subhalo_unbind.cpp:21-58) in closed form, as
// k_part_codes .. k_part_copyback do; returns Nbound.
__device__ int partition(const Group &g, const Ctx &c, int P0)
{
  int *const F = g.ctr, *const G = g.ctr + 1, *const info = g.ctr + 2;
  long long *px = reinterpret_cast<long long *>(g.key0);
  int *Pk = g.val0, *Qk = g.val1;
  const int nl = g.sg->nlast;
  if (g.tid == 0) {
    *F = 0x7fffffff;
    *G = 0x7fffffff;
  }
  for (int l = g.tid; l <= nl; l += g.T) {
    long long code = 0;
    if (l >= 1 && l < nl) {
      const float e = c.eE[P0 + l];
      code = (e < 0.f ? (1ll << 32) : 0ll) | (e > 0.f ? 1ll : 0ll);
    }
    px[l] = code;
  }
  g.sync();
  group_scan(g, px, nl + 1);
  const long long x1 = nl >= 2 ? px[1] : 0, xe = nl >= 2 ? px[nl] : 0;
  const int nPos = (int)((xe - x1) & 0xffffffffll), nNeg = (int)((xe - x1) >> 32);
  if (nl >= 2)
    for (int l = 1 + g.tid; l < nl; l += g.T) {
      const float e = c.eE[P0 + l];
      if (e > 0.f) Pk[(int)((px[l] - x1) & 0xffffffffll)] = l;
      if (e < 0.f) Qk[(int)((xe - px[l]) >> 32) - 1] = l;
    }
  g.sync();
  if (nl >= 2)
    for (int l = 1 + g.tid; l < nl; l += g.T) {
      if (!(c.eE[P0 + l] > 0.f)) continue;
      const int k = (int)((px[l] - x1) & 0xffffffffll) + 1;
      if (k > min(nPos, nNeg)) continue;
      const int qk = Qk[k - 1];
      if (l >= qk) atomicMin(F, k);
      if (k + 1 > nNeg || l >= Qk[k]) atomicMin(G, k);
    }
  g.sync();
  if (g.tid == 0) {
    const float e0 = c.eE[P0];
    int mb = 0, mf = 0, vd = 0, nb;
    if (nl < 2) {
      nb = nl == 1 ? (e0 < 0.f) : 0;
    } else {
      const int mn = min(nPos, nNeg);
      const int Fk = min(*F, mn + 1) - 1;
      const int Gk = min(*G - 1, Fk);
      if (nNeg > 0) {
        mb = 1 + Gk;
        mf = Gk + (Gk + 1 <= Fk ? 1 : 0);
        vd = (mf == mb) ? Pk[mf - 1] : Qk[mb - 1];
      }
      nb = vd + (e0 < 0.f);
    }
    info[0] = mb;
    info[1] = mf;
    info[2] = vd;
    info[3] = nb;
  }
  g.sync();
  const int mb = info[0], mf = info[1], vd = info[2], nb = info[3];
  int pid[kPer];
  float E[kPer];
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int l = g.tid + k * g.T;
    if (l >= nl) break;
    int src = l;
    if (nl >= 2) {
      const float e = c.eE[P0 + l];
      if (l == vd) {
        src = 0;
      } else if (l == 0) {
        src = nNeg >= 1 ? Qk[0] : 0;
      } else if (e < 0.f) {
        const int kq = (int)((xe - px[l]) >> 32);
        if (kq <= mf) src = Pk[kq - 1];
      } else if (e > 0.f) {
        const int kp = (int)((px[l] - x1) & 0xffffffffll) + 1;
        if (kp <= mb - 1) src = Qk[kp];
      }
    }
    pid[k] = c.epid[P0 + src];
    E[k] = c.eE[P0 + src];
  }
  g.sync();
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int l = g.tid + k * g.T;
    if (l >= nl) break;
    c.epid[P0 + l] = pid[k];
    c.eE[P0 + l] = E[k];
    c.epos_of_pid[pid[k]] = P0 + l;
  }
  g.sync();
  return nb;
}

// Sums of K values over list positions [0, nb), as block_sum takes them per chunk
// of kChunk and the batch path adds the chunks: a chunk's positions
// 32 w + lane + 256 j belong to its group w, one warp each here.  sums(first,
// hi, out) leaves a group's sums in out[0..K); returns sum `lane` in the lanes
// of the first warp.
template <int K, class Sums>
__device__ __forceinline__ double list_sums(const Group &g, int nb, Sums sums)
{
  const int nw = g.T / 32;
  const int lane = threadIdx.x & 31, w = g.tid >> 5;
  const int nch = (nb + kChunk - 1) / kChunk;
  for (int q = w; q < kSumGroups * nch; q += nw) {
    const int lo = (q / kSumGroups) * kChunk, grp = q % kSumGroups;
    const int hi = min(lo + kChunk, nb);
    if (32 * grp < hi - lo) sums(lo + 32 * grp + lane, hi, g.part + K * q);
  }
  g.sync();
  double total = 0.;
  if (w == 0 && lane < K)
    for (int ch = 0; ch < nch; ch++) {
      const int groups = min(kSumGroups, (min(kChunk, nb - ch * kChunk) + 31) / 32);
      double t = 0.;
      for (int k = 0; k < groups; k++) t += g.part[K * (ch * kSumGroups + k) + lane];
      total += t;
    }
  g.sync();
  return total;
}

// AverageVelocity / AveragePosition of the bound block [0, nb) and the decisions.
__device__ void decide(const Group &g, const Ctx &c, int P0, int nb, int max_passes)
{
  SegState &sg = *g.sg;
  double sum = 0.;
  if (nb > 1) {
    const float4 o = c.pm[c.epid[P0]];
    const double od[3] = {f2d(o.x), f2d(o.y), f2d(o.z)};
    sum = list_sums<7>(g, nb, [&](int p, int hi, double *out) {
      double v[7] = {0., 0., 0., 0., 0., 0., 0.}, one;
      for (; p < hi; p += kLB) {
        const int pid = c.epid[P0 + p];
        frame_terms(c.pm[pid], c.vel[pid], o, od, c.P, v);
      }
      const int k = warp_sums<7>(v, &one);
      if (k >= 0) out[k] = one;
    });
  }
  if (g.tid < 32) {
    double mean[6];
    const double mass = frame_means(sum, g.tid, nb, mean);
    if (g.tid == 0) control_segment(c, sg, nb, mass, mean, max_passes);
  }
  g.sync();
}

// A call's lists of one subhalo and its loop state, as k_init and the batch
// path's host set-up make them.
__device__ void load_subhalo(const Group &g, const Ctx &c, const SmallCall &io, int s)
{
  SegState &sg = *g.sg;
  const int off = (int)io.off[s], n = (int)(io.off[s + 1] - io.off[s]);
  if (g.tid == 0) {
    init_segment(sg, off, n, io.st[s], c.P.maxsample);
    c.seg[s].interactions = 0;
  }
  g.sync();
  int first = 0x7fffffff;
  for (int i = g.tid; i < n; i += g.T) {
    const int p = off + i;
    c.pm[p] = make_float4(io.pos[3 * (size_t)p], io.pos[3 * (size_t)p + 1],
                          io.pos[3 * (size_t)p + 2], io.mass[p]);
    c.vel[p] = make_float4(io.vel[3 * (size_t)p], io.vel[3 * (size_t)p + 1],
                           io.vel[3 * (size_t)p + 2], 0.f);
    c.epid[p] = p;
    c.eE[p] = 0.f;
    c.epos_of_pid[p] = p;
    if (c.id[p] == sg.mb_id) first = min(first, i);
  }
  first = __reduce_min_sync(0xffffffffu, first);
  if ((threadIdx.x & 31) == 0) atomicMin(&sg.first_mb, first);
  g.sync();
}

// The final sums and the outputs of one subhalo, its bound block sorted.
__device__ void finish_subhalo(const Group &g, const Ctx &c, const SmallCall &io, int s, int P0)
{
  SegState &sg = *g.sg;
  double sum = 0.;
  if (sg.status == SEG_CONVERGED || sg.status == SEG_FAILED)
    sum = list_sums<18>(g, sg.nbound, [&](int p, int hi, double *out) {
      kin_warp_sums(c, sg, sg.nbound, p, hi, out, 1);
    });
  if (g.tid < 32) {
    if (g.tid == 0) sg.interactions = __ldcg(&c.seg[s].interactions);
    __syncwarp();
    write_result(c, sg, sum, g.tid, io.res + s);
  }
  for (int p = P0 + g.tid; p < P0 + sg.n; p += g.T)
    write_position(c, sg, p, io.order_out, io.energy_out);
  g.sync();
}

__device__ __forceinline__ void cluster_sync()
{
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}

// Every field of a subhalo's state but the interaction count, which the walks
// add to in global memory.
__device__ void copy_state(const Group &g, const SegState *from, SegState *to)
{
  constexpr int skip = offsetof(SegState, interactions) / 4;
  const volatile int *a = reinterpret_cast<const volatile int *>(from);
  int *b = reinterpret_cast<int *>(to);
  for (int k = g.tid; k < (int)(sizeof(SegState) / 4); k += g.T)
    if (k != skip && k != skip + 1) b[k] = a[k];
}

// The sorts between two passes: the unbound block of the last one (the batch path
// sorts it at the start of the next round, also after convergence); at the end of
// a whole call the bound block (src/subhalo_unbind.cpp:405), and after
// RefineBindingEnergyOrder's extra pass (:234-262, :406-407) the refined positions
// by its energies.  Sets that pass up where it applies.
__device__ __forceinline__ void sort_between(const Group &g, const Ctx &c, bool whole, bool refined)
{
  SegState &sg = *g.sg;
  int lo = refined ? 0 : sg.ub_lo, hi = refined ? sg.ntgt : sg.ub_hi;
#pragma unroll 1
  for (int k = 0; k < 2; k++) {
    sort_block(g, c, sg.off, lo, hi, refined ? c.eR : c.eE);
    const bool end = sg.status == SEG_CONVERGED || sg.status == SEG_FAILED;
    if (k == 1 || refined || !whole || !end) break;
    lo = 0;
    hi = sg.nbound;
  }
  g.sync();
  if (g.tid == 0) {
    sg.ub_lo = sg.ub_hi = 0;
    if (whole && sg.refine && !refined && sg.status == SEG_CONVERGED) {
      sg.status = SEG_ACTIVE;
      sg.mode = MODE_REFINE;
      sg.t0 = 0;
      sg.ntree = sg.ntgt = (int)min((long long)sg.nbound, c.P.maxsample);
      sg.mfac = 1.f;
      sg.tgt_mode = 0;
      sg.evals += sg.ntgt;
    }
  }
  g.sync();
}

// c.small_next: the three queues' next job, their counts, and the classes' threads.
//
// The groups of a block advance their subhaloes step by step together, with a
// block barrier between the steps (a group whose subhalo ends takes the next
// one): groups that ran apart, each in its own part of the code, missed the
// instruction cache more often than they waited for anything else (14 of 26 stalls
// per instruction; the queues are in size order, so a block's groups have like
// work).
template <bool kFP64>
__global__ void __launch_bounds__(kSB, 2)
    k_unbind_small(Ctx c, SmallCall io, SmallJobs jobs, int whole, int cap, int max_passes)
{
  HBTU_KERNEL_PROLOGUE();
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned rank, blocks, cluster;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(blocks));
  asm("mov.u32 %0, %%clusterid.x;" : "=r"(cluster));
  const int w = threadIdx.x >> 5;
#pragma unroll 1
  for (int cls = 0; cls < 3; cls++) {  // large lists, medium, short
    const int n = c.small_next[3 + cls], T = c.small_next[6 + cls];
    // a cluster per large list (there are as many): the first block leads, the
    // others take part in the walk
    const bool shared = cls == 0 && blocks > 1;
    const bool lead = !shared || rank == 0;
    // over all blocks first, so only as many groups of each as that takes
    bool more = shared ? (int)cluster < n
                       : (int)threadIdx.x / T < (n + (int)gridDim.x - 1) / (int)gridDim.x;
    const SmallLayout L(min(cap, cls == 0 ? kSmallCap : cls == 1 ? kSmallMediumCap : kSmallWarpCap),
                        cls == 2);
    // four warps' memory is one medium group's or four short lists'
    const Group g(T,
                  smem + (cls == 0 ? 0 : (w / 4 & ~(T > kMT ? 1 : 0)) * quad_bytes(cap)) +
                      (cls == 2 ? (w % 4) / (T / 32) * L.bytes : 0),
                  L);
    SegState &sg = *g.sg;
    bool have = false, refined = false;
    int s = 0;
    for (;;) {
      if (!have && more) {
        int k = cluster;
        if (!shared) {
          g.sync();
          if (g.tid == 0) g.ctr[15] = atomicAdd(&c.small_next[cls], 1);
          g.sync();
          k = g.ctr[15];
        }
        have = k < n;
        more = have && !shared;
        refined = false;
        if (have) {
          s = jobs.list[cls][k];
          if (lead) {
            if (whole)
              load_subhalo(g, c, io, s);
            else
              copy_state(g, &c.seg[s], &sg);
            g.sync();
          }
        }
      }
      if (!__syncthreads_or(have)) break;
      if (have && lead) sort_between(g, c, whole, refined);
      bool act = have && lead && sg.status == SEG_ACTIVE;
      ull *sk = g.key0;
      if (act) sk = tree_keys(g, c, sg.off);
      ull *other = sk == g.key0 ? g.key1 : g.key0;
      __syncthreads();
      if (act) tree_nodes(g, c, sg.off, sk, reinterpret_cast<long long *>(other));
      __syncthreads();
      if (act) tree_moments(g, c, sg.off, reinterpret_cast<int *>(other));
      __syncthreads();
      const int *sval = g.val1;
      if (have && shared) {
        if (lead) {
          copy_state(g, &sg, &c.seg[s]);
          if (act && sg.tgt_mode == 0)
            for (int i = g.tid; i < sg.ntree; i += T) c.sb.val_a[sg.off + i] = g.val1[i];
        }
        cluster_sync();
        if (!lead) {
          copy_state(g, &c.seg[s], &sg);
          g.sync();
          sval = c.sb.val_a + sg.off;
          act = sg.status == SEG_ACTIVE;
        }
      }
      if (act)
        // a cluster's warps take targets in turn over its blocks
        walk_targets<kFP64>(g, c, s, sg.off, sval,
                            shared ? (w * blocks + rank) * 32 + (threadIdx.x & 31) : g.tid,
                            shared ? blocks * T : T);
      if (act && shared) cluster_sync();
      __syncthreads();
      if (act && lead) {
        if (sg.mode == MODE_REFINE) {
          refined = true;
          g.sync();
          if (g.tid == 0) sg.status = SEG_CONVERGED;
          g.sync();
        } else {
          const int nb = partition(g, c, sg.off);
          decide(g, c, sg.off, nb, max_passes);
        }
      }
      if (have && !act) {  // ended
        have = false;
        if (lead && whole) {
          finish_subhalo(g, c, io, s, sg.off);
        } else if (!shared) {
          copy_state(g, &sg, &c.seg[s]);
          g.sync();
        }
      }
    }
  }
}

// The active subhaloes in size order, by class: class k from small_list[k S] on,
// their counts to small_next.
__global__ void __launch_bounds__(1024) k_small_list(Ctx c, int blocks)
{
  HBTU_KERNEL_PROLOGUE();
  __shared__ int ws[3][32], base[3], count[3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 3) base[threadIdx.x] = count[threadIdx.x] = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < c.S; s += 1024)
    if (c.seg[s].status == SEG_ACTIVE) {
      const int n = c.seg[s].nlast;
      atomicAdd(&count[n > kSmallMediumCap ? 0 : n > kSmallWarpCap ? 1 : 2], 1);
    }
  __syncthreads();
  const SmallClasses classes = small_classes_of(count[0], count[1], count[2], blocks);
  for (int b = 0; b < c.S; b += 1024) {
    const int k = b + threadIdx.x;
    const int s = k < c.S ? c.seg_order[k] : 0;
    const bool act = k < c.S && c.seg[s].status == SEG_ACTIVE;
    const int n = act ? c.seg[s].nlast : 0;
    const int cls = !act ? -1 : n > classes.bound[0] ? 0 : n > classes.bound[1] ? 1 : 2;
    unsigned m[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      m[q] = __ballot_sync(0xffffffffu, cls == q);
      if (lane == 0) ws[q][w] = __popc(m[q]);
    }
    __syncthreads();
    int at[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      at[q] = base[q];
      for (int v = 0; v < w; v++) at[q] += ws[q][v];
      if (cls == q) c.small_list[q * c.S + at[q] + __popc(m[q] & ((1u << lane) - 1u))] = s;
    }
    __syncthreads();
    if (threadIdx.x == 1023)
#pragma unroll
      for (int q = 0; q < 3; q++) base[q] = at[q] + __popc(m[q]);
    __syncthreads();
  }
  if (threadIdx.x < 3) {
    c.small_next[threadIdx.x] = 0;
    c.small_next[3 + threadIdx.x] = base[threadIdx.x];
    c.small_next[6 + threadIdx.x] = classes.T[threadIdx.x];
  }
}

// Resident blocks of the kernel (two per SM, by its launch bounds and memory).
int resident_blocks()
{
  int dev = 0, sms = 0;
  HBTU_CUDA(cudaGetDevice(&dev));
  HBTU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return 2 * sms;
}

// Shared memory of a block, for lists of up to `cap`, with or without large ones.
size_t block_bytes(int cap, bool large)
{
  const size_t quads = (kSB / kMT) * quad_bytes(cap);
  return large ? std::max(quads, SmallLayout(cap).bytes) : quads;
}

// n[k]: upper bounds of the jobs of each class.
void launch(Ctx &c, const SmallCall &io, int whole, const SmallJobs &jobs, int cap,
            const int (&n)[3], int max_passes)
{
  const size_t smem = block_bytes(cap, n[0] > 0);
  void (*kernel)(Ctx, SmallCall, SmallJobs, int, int, int) =
      c.P.precision == HBTU_PRECISION_FP64 ? k_unbind_small<true> : k_unbind_small<false>;
  // The attribute is the kernel's, not the launch's: set to what a call's own lists need, it
  // could fall below another thread's need between that thread's setting and
  // its launch.  Every call sets the largest.
  HBTU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)block_bytes(kSmallCap, true)));
  const int resident = resident_blocks();
  // few large lists: a cluster of blocks each, while half the chip holds them and
  // each block has a warp per scheduler
  int cluster = 1;
  while (n[0] > 0 && cluster < kMaxCluster && 128 * cluster < cap &&
         2 * cluster * n[0] <= resident / 2)
    cluster *= 2;
  // the groups of each class, at one per block if the chip has room
  int grid = std::max(cluster * n[0], std::max(n[1], n[2]));
  grid = std::max(1, std::min(grid, resident));
  grid = (grid + cluster - 1) / cluster * cluster;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = launch_overlap() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = kSB;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c.st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  HBTU_CUDA(cudaLaunchKernelEx(&cfg, kernel, c, io, jobs, whole, cap, max_passes));
  HBTU_LAUNCHED();
}

}  // namespace

void launch_small(Ctx &c, int cap, int nactive, int max_passes)
{
  if (nactive <= 0) return;
  launch_k(k_small_list, 1, 1024, 0, c.st, c, resident_blocks());
  HBTU_LAUNCHED();
  // the classes' sizes are known on the device alone
  const SmallJobs jobs = {{c.small_list, c.small_list + c.S, c.small_list + 2 * (size_t)c.S}};
  const int most[3] = {nactive, nactive, nactive};
  launch(c, SmallCall(), 0, jobs, cap, most, max_passes);
}

void small_classes(const int64_t *offsets, const int *order, int S, int (&n)[3], int (&T)[3])
{
  auto longer = [&](int cap) {  // lists longer than cap: order is by size
    int lo = 0, hi = S;
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (offsets[order[mid] + 1] - offsets[order[mid]] > cap)
        lo = mid + 1;
      else
        hi = mid;
    }
    return lo;
  };
  const int a = longer(kSmallMediumCap), b = longer(kSmallWarpCap);
  const SmallClasses q = small_classes_of(a, b - a, S - b, resident_blocks());
  n[0] = longer(q.bound[0]);
  n[1] = longer(q.bound[1]) - n[0];
  n[2] = S - n[0] - n[1];
  for (int k = 0; k < 3; k++) T[k] = q.T[k];
}

void launch_small_call(Ctx &c, const SmallCall &io, int cap, int max_passes)
{
  const SmallJobs jobs = {
      {io.order, io.order + io.jobs[0], io.order + io.jobs[0] + io.jobs[1]}};
  launch(c, io, 1, jobs, cap, io.jobs, max_passes);
}

}  // namespace hbtu
