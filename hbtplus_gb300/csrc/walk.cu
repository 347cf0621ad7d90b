// walk.cu -- binding energies by Barnes-Hut walk (the hot loop).
//
// Reference: GravityTree_t::EvaluatePotential (src/gravity_tree.cpp:79-164),
// BindingEnergy (:166-175), and the two energy loops of Subhalo_t::Unbind
// (src/subhalo_unbind.cpp:319-328 correction, :341-354 full pass).
//
// Each target performs exactly the reference's stackless walk: at a cell it
// opens (goes to the first child, preorder index + 1) when
// len*len > r*r*theta^2, otherwise it takes the cell's monopole and jumps to
// the skip pointer; particles are never opened.  Targets are taken in Morton
// order, subhaloes largest first, so a warp holds neighbouring targets.
//
// FP32 (default): coordinates relative to the subhalo frame centre, wrapped
// once in double, so the per-interaction periodic wrap disappears; opening
// decisions within 1e-5 of the threshold are re-taken in double exactly as
// the reference takes them; the potential is summed in float with
// compensation and formed in double once per target (no double arithmetic in
// the loop: this GPU's FP64 rate is 1/64 of its FP32 rate).  Two schedules:
//   lane (default): every lane walks its own target, or in large launches two
//     neighbouring ones at once, one 32-byte node record per step; large blocks
//     keep a block's neighbouring targets on one SM, so the walks share L1;
//   warp: the warp visits the smallest index any of its targets waits at, so
//     each node is a broadcast load (kept as an option for comparison).
// FP64: absolute float coordinates, NEAREST per interaction, every operation
// in the reference's order without fused multiply-add; one walk per lane.
// The per-target walks live in walk_ops.cuh (shared with small.cu).
#include "walk_ops.cuh"
#include <algorithm>

namespace hbtu {
namespace {

constexpr int kWB = 128;

// Target w of this pass: segment, list position, particle, walk range.
template <bool kRel, bool kWarp = false>
__device__ __forceinline__ void load_target(const Ctx &c, int w, int total, Target &t)
{
  if (w >= total) {
    t.s = 0;
    t.epos = -1;
    t.pid = -1;
    t.active = false;
    t.nxt = kDone;
    t.end = 0;
    t.mself = 0.f;
    t.q[0] = t.q[1] = t.q[2] = 0.f;
    return;
  }
  const int k = upper_bound_i(c.tgt_base, c.S + 1, w) - 1;
  const int s = c.seg_order[k];
  const SegState &sg = c.seg[s];
  const int local = w - c.tgt_base[k];
  const int tm = sg.tgt_mode;
  int epos, pid;
  bool active;
  if (tm == 0) {  // full pass: tree leaves in Morton order
    epos = c.sb.val_a[c.tree_base[s] + local];
    pid = c.epid[epos];
    c.coh_pid[sg.off + local] = pid;
    active = true;
  } else if (kWarp && tm == 1) {  // correction pass: the last full pass's order, still bound
    pid = c.coh_pid[sg.off + local];
    epos = c.epos_of_pid[pid];
    active = (epos - sg.off) < sg.ntgt;
  } else if (tm == 1 || sg.coh_n > 0) {  // launch_bound_order, launch_list_order
    pid = c.epid2[sg.off + local];
    epos = c.epos_of_pid[pid];
    c.coh_pid[sg.off + local] = pid;
    active = true;
  } else {  // list order
    epos = sg.off + local;
    pid = c.epid[epos];
    active = true;
  }
  init_target<kRel>(c, sg, s, epos, pid, active, 2 * c.tree_base[s], t);
}

// Correction passes walk the particles still bound, in the Morton order of the
// last full pass.  That pass's list is first rid of the particles removed since,
// which left lanes idle and kept the neighbours of a pair apart (correction pass
// of a 2.7e7-particle host: 94 ms with the removed ones in the list, one target
// per lane; 93 without them, 92 in pairs with them, 65 in pairs without).  The new
// list goes to epid2, free between the tree build and the partition; the walk
// copies it to coh_pid (load_target).  Bandwidth- and gather-bound: 56 us for the
// 1.3e6 particles of a tracking step.
// k_order_count leaves per 32 list positions x the bits of the still bound and y
// how many come before them in the block, and per block their count (scanned next).
constexpr int kOrderBlock = 1024;

__global__ void __launch_bounds__(kOrderBlock) k_order_count(Ctx c)
{
  HBTU_KERNEL_PROLOGUE();
  __shared__ int wsum[32];
  const int p = blockIdx.x * kOrderBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  bool keep = false;
  if (p < c.N) {
    const SegState &sg = c.seg[c.pseg[p]];
    keep = sg.status == SEG_ACTIVE && sg.tgt_mode == 1 && p - sg.off < sg.coh_n &&
           c.epos_of_pid[c.coh_pid[p]] - sg.off < sg.ntgt;
  }
  const unsigned bits = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) wsum[w] = __popc(bits);
  __syncthreads();
  if (w == 0) {
    const int own = wsum[lane];
    int x = own;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    wsum[lane] = x - own;
    if (lane == 31) c.pX[blockIdx.x] = x;
  }
  __syncthreads();
  if (lane == 0 && p < c.N)
    reinterpret_cast<uint2 *>(c.pcode)[p >> 5] = make_uint2(bits, wsum[w]);
}

__global__ void __launch_bounds__(kWB) k_order_write(Ctx c)
{
  HBTU_KERNEL_PROLOGUE();
  const int p = blockIdx.x * kWB + threadIdx.x;
  if (p >= c.N) return;
  const uint2 *words = reinterpret_cast<const uint2 *>(c.pcode);
  SegState &sg = c.seg[c.pseg[p]];
  const uint2 x = words[p >> 5];
  if (p == sg.off && sg.status == SEG_ACTIVE && sg.tgt_mode == 1) sg.coh_n = sg.ntgt;
  if (!(x.x >> (p & 31) & 1u)) return;
  const int o = sg.off;
  const uint2 y = words[o >> 5];
  const int at = (int)c.pX[p / kOrderBlock] + x.y + __popc(x.x & ((1u << (p & 31)) - 1u));
  const int at0 = (int)c.pX[o / kOrderBlock] + y.y + __popc(y.x & ((1u << (o & 31)) - 1u));
  c.epid2[o + at - at0] = c.coh_pid[p];
}

void launch_bound_order(Ctx &c)
{
  const int nb = (c.N + kOrderBlock - 1) / kOrderBlock;
  launch_k(k_order_count, nb, kOrderBlock, 0, c.st, c);
  HBTU_LAUNCHED();
  exclusive_scan_i64(c.pX, c.pX, nb, c.scan_tmp, c.st);
  launch_k(k_order_write, (c.N + kWB - 1) / kWB, kWB, 0, c.st, c);
  HBTU_LAUNCHED();
}

// Targets of subhaloes with sampled potentials come in list order at first (their
// trees hold a few of them), and a warp's walks then share no nodes.  They are sorted
// along the Morton curve of the tree's root cell, 2^bits cells a side (four passes of
// the sort for up to 2048 subhaloes); later passes keep that order
// (launch_bound_order).  First passes of 2000 subhaloes, 1000 particles per tree:
// 758 -> 607 us, second 494 -> 414 us, for 90 us of sorting; one of 1.2e6 particles
// takes 4.4 ms, not 6.3.
__global__ void __launch_bounds__(kWB) k_list_keys(Ctx c, int bits)
{
  HBTU_KERNEL_PROLOGUE();
  const int p = blockIdx.x * kWB + threadIdx.x;
  if (p >= c.N) return;
  const int s = c.pseg[p];
  const SegState &sg = c.seg[s];
  const unsigned top = (1u << (3 * bits)) - 1u;  // after every target of the subhalo
  unsigned key = top;
  if (sg.status == SEG_ACTIVE && sg.tgt_mode == 2 && p - sg.off < sg.ntgt) {
    const float4 a = c.pm[c.epid[p]];
    const float x[3] = {a.x, a.y, a.z};
    const float side = (float)(1 << bits), inv = __fdividef(side, (float)sg.len);
    unsigned cell[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const float u = rel_coord(x[j], sg.fc[j], c.P) * inv + 0.5f * side;
      cell[j] = (unsigned)fminf(fmaxf(u, 0.f), side - 1.f);  // NaN: cell 0
    }
    key = 0;
    for (int b = bits - 1; b >= 0; b--)
      key = key << 3 | (cell[0] >> b & 1u) << 2 | (cell[1] >> b & 1u) << 1 | (cell[2] >> b & 1u);
    key = min(key, top - 1u);
  }
  c.sb.lo_a[p] = (unsigned long long)s << (3 * bits) | key;
  c.sb.hi_a[p] = 0;
  c.sb.val_a[p] = p;
}

__global__ void __launch_bounds__(kWB) k_list_write(Ctx c)
{
  HBTU_KERNEL_PROLOGUE();
  const int p = blockIdx.x * kWB + threadIdx.x;
  if (p >= c.N) return;
  SegState &sg = c.seg[c.pseg[p]];
  if (sg.status != SEG_ACTIVE || sg.tgt_mode != 2 || p - sg.off >= sg.ntgt) return;
  if (p == sg.off) sg.coh_n = sg.ntgt;
  c.epid2[p] = c.epid[c.sb.val_a[p]];
}

// The warp schedule's squared distance: with the compiler's own choice of fused
// multiply-adds, which is not dist2's (the lane schedule's) everywhere.
__device__ __forceinline__ float dist2_warp(float4 na, const float q[3])
{
  const float dx = na.x - q[0], dy = na.y - q[1], dz = na.z - q[2];
  return dx * dx + dy * dy + dz * dz;
}

// FP32 walk, warp schedule.  Leaf runs: when targets open a cell
// whose children are all particles, each of those targets takes every child
// in order (particles are never opened) -- the warp streams the children
// through a loop with no opening test and no scheduling per node.
template <bool kLeafRuns>
__global__ void __launch_bounds__(kWB) k_walk_fp32(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  const DevParams &P = c.P;
  const unsigned full = 0xffffffffu;
  Target t;
  load_target<true, true>(c, blockIdx.x * kWB + threadIdx.x, total, t);
  PotAcc acc;
  const float theta2 = P.theta2;
  const float hf = P.hf, hinvf = P.hinvf, h2f = P.h2f;
  const double th2d = P.theta2d;
  int ninter = 0;
  unsigned steps = 0;

  int cur = __reduce_min_sync(full, t.nxt);
  float4 na = make_float4(0.f, 0.f, 0.f, 0.f);
  int2 nm = make_int2(0, 0);
  if (cur != kDone) {
    load_node(c.nd, cur, na, nm);
  }
  while (cur != kDone) {
    float4 pa;  // speculative; a spare slot follows the last node
    int2 pmeta;
    load_node(c.nd, cur + 1, pa, pmeta);
    const float l2 = __int_as_float(nm.x & 0x7fffffff);
    const bool bottom = kLeafRuns && nm.x < 0;
    const int sk = nm.y;
    bool run = false;
    if (t.nxt == cur) {
      const float r2 = dist2_warp(na, t.q);
      if (opens(na, t.q, l2, r2, theta2, th2d)) {
        if (bottom)
          run = true;
        else
          t.nxt = cur + 1 < t.end ? cur + 1 : kDone;
      } else {
        t.nxt = (unsigned)(sk - cur - 1) < (unsigned)(t.end - cur - 1) ? sk : kDone;
        ninter++;
        interact(na, r2, acc.f, hf, h2f, hinvf);
      }
    }
    const unsigned runners = kLeafRuns ? __ballot_sync(full, run) : 0u;
    if (runners) {
      // children cur+1 .. sk-1 are particles: stream them (every runner is at
      // cur, in one tree, so the bound is the same for all of them)
      const int last = __shfl_sync(full, min(sk, t.end), __ffs(runners) - 1);
      int j = cur + 1;
      for (; j + 1 < last; j += 2) {
        const float4 a0 = c.nd[j].p, a1 = c.nd[j + 1].p;
        if (run) {
          interact(a0, dist2_warp(a0, t.q), acc.f, hf, h2f, hinvf);
          interact(a1, dist2_warp(a1, t.q), acc.f, hf, h2f, hinvf);
        }
      }
      if (j < last) {
        const float4 a0 = c.nd[j].p;
        if (run) interact(a0, dist2_warp(a0, t.q), acc.f, hf, h2f, hinvf);
      }
      if (run) {
        ninter += last - cur - 1;
        t.nxt = (unsigned)(sk - cur - 1) < (unsigned)(t.end - cur - 1) ? sk : kDone;
      }
      acc.flush();
      cur = __reduce_min_sync(full, t.nxt);
      if (cur != kDone) {
        load_node(c.nd, cur, na, nm);
      }
    } else if (__any_sync(full, t.nxt == cur + 1)) {
      cur = cur + 1;
      na = pa;
      nm = pmeta;
    } else {
      cur = __reduce_min_sync(full, t.nxt);
      if (cur != kDone) {
        load_node(c.nd, cur, na, nm);
      }
    }
    if ((++steps & 7u) == 0u) acc.flush();
  }
  finish_target(c, c.seg[t.s], t, acc.total((double)__fdiv_rn(t.mself, P.eps)));  // + cancels the self term
  count_interactions(c, t.s, ninter);
}

// FP32 walk, lane schedule (walk_lean): blocks of kB neighbouring targets.
template <int kB, bool kSib, bool kFlat>
__global__ void __launch_bounds__(kB) k_walk_fp32_lean(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  Target t;
  load_target<true>(c, blockIdx.x * kB + threadIdx.x, total, t);
  int ninter = 0;
  const double pot = walk_lean<kSib, kFlat>(kSib ? c.nd2 : c.nd, t, c.P, &ninter);
  finish_target(c, c.seg[t.s], t, pot);
  count_interactions(c, t.s, ninter);
}

// Two neighbouring targets per lane (walk_pair).
constexpr int kPB = 256;
inline unsigned pair_blocks(int n) { return ((unsigned)n + 2 * kPB - 1) / (2 * kPB); }

// Loads the lane's targets and walks them, first those of the first one's tree,
// then, where the second is of another subhalo, that one.  The targets are loaded
// again for the second round and the results, so that the walk holds no more of them
// than it needs (63 registers, 2.7e7 targets: 122.5 -> 120.0 ms, their correction pass
// 65.3 -> 63.1).  At 48 registers the walk spills and gains nothing (122.4, 63.6), at 79
// it loses (129.8, 70.9).
__device__ __forceinline__ void walk_targets_pair(const Ctx &c, int total, Target (&t)[2],
                                                  double (&pot)[2], int (&ninter)[2])
{
  const float zero[2] = {0.f, 0.f};
  PairSums sums = {f2_pack(zero), f2_pack(zero), {0, 0}};
#pragma unroll 1
  for (int round = 0; round < 2; round++) {
    int w = 2 * (blockIdx.x * kPB + threadIdx.x);
    asm volatile("" : "+r"(w));
    load_target<true>(c, w, total, t[0]);
    load_target<true>(c, w + 1, total, t[1]);
    const bool a0 = t[0].end > t[0].nxt, a1 = t[1].end > t[1].nxt;
    const bool apart = a0 && t[1].nxt != t[0].nxt;
    const bool here[2] = {round == 0 && a0, a1 && apart == (round == 1)};
    if (here[0] || here[1])
      walk_pair(c.nd, t, here, here[0] ? t[0].nxt : t[1].nxt, here[0] ? t[0].end : t[1].end, c.P,
                sums);
  }
  float h[2], e[2];
  f2_unpack(sums.hi, h);
  f2_unpack(sums.comp, e);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double base = f2d(__fdiv_rn(t[k].mself, c.P.eps));  // cancels the self term
    pot[k] = dadd(dadd(base, f2d(h[k])), -f2d(e[k]));
    ninter[k] = sums.ninter[k];
  }
}

__global__ void __launch_bounds__(kPB, 3) k_walk_fp32_pair(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  Target t[2];
  int ninter[2];
  double pot[2];
  walk_targets_pair(c, total, t, pot, ninter);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    finish_target(c, c.seg[t[k].s], t[k], pot[k]);
    count_interactions(c, t[k].s, ninter[k]);
  }
}

// The lane schedule's energy walks (these and k_walk_fp32_pair) are launched after all
// of the kernel before them: blocks placed while its blocks still hold their SMs
// gather on the other SMs, and a walk of few blocks never evens that out (1e5 targets
// after 108 blocks of 1024 threads: 574 us, not 287; the unbinding of 1.1e5 particles
// 1.81 ms, 1.90 launched ahead).  The other walks (FP64, warp schedule, gradients) are
// launched ahead; for them the two ways have not been compared.
template <bool kSib>
void launch_lean(Ctx &c, int n)
{
  if (n >= 152 * 4 * 512)  // blocks of neighbouring targets share an SM's L1
    launch_after(k_walk_fp32_lean<512, kSib, false>, (n + 511) / 512, 512, 0, c.st, c, n);
  else if (n >= 152 * 4 * 256)
    launch_after(k_walk_fp32_lean<256, kSib, true>, (n + 255) / 256, 256, 0, c.st, c, n);
  else
    launch_after(k_walk_fp32_lean<128, kSib, true>, (n + 127) / 128, 128, 0, c.st, c, n);
}

// FP64: the reference's arithmetic, operation by operation (walk_fp64), one
// walk per lane.
__global__ void __launch_bounds__(kWB) k_walk_fp64(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  Target t;
  load_target<false>(c, blockIdx.x * kWB + threadIdx.x, total, t);
  int ninter = 0;
  const double pot = walk_fp64(c, t, &ninter);
  finish_target(c, c.seg[t.s], t, pot);
  count_interactions(c, t.s, ninter);
}

// ---------------------------------------------------------------------------
// Adjoint: gradient of the total binding energy over a fixed particle set,
//   E_tot = sum_i m_i |dv_i|^2 / 2 + (1/2) sum_i m_i phi_i,
// with dv_i the velocity relative to the frame (RelativeVelocity, Hubble flow
// included) and phi_i the walk potential (self term cancelled).  The frame is
// the set's centre of mass, so its dependence on x, v, m cancels (sum m dv = 0):
//   dE/dv_k = m_k dv_k,
//   dE/dx_k = m_k (H a dv_k + grad phi(x_k)),
//   dE/dm_k = |dv_k|^2 / 2 + phi_k.
// grad phi is recomputed by a walk with the reference's opening rule on the same
// tree (nothing of the energy walk is stored); per accepted node
//   far  (r >= h): d(-m/r)/dx_t = -m dx / r^3,
//   near (r < h):  d(m wp(u)/h)/dx_t = -m wp'(u) dx / (h^2 r),  u = r/h,
// with wp' the derivative of the cubic-spline kernel; dx = x_node - x_target.
// The walk is walk_lean's (one target per lane, the same nodes in the same
// order, the potential in the same compensated float sum); the gradient
// terms go into compensated float sums, one per lane, so a target's results do
// not depend on the other targets of the call.  kGrad =
// false computes only the energies (the forward pass of the autograd function).
// s += v in a compensated float sum (Kahan): s - c carries the sum.
__device__ __forceinline__ void kahan_add(float &s, float &c, float v)
{
  const float y = __fsub_rn(v, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}

// As in walk_lean the next node's load is issued before the node's terms are
// computed (1e6 targets: 5.74 -> 5.60 ms; 2000 subhaloes, 6e5 targets: 1.73 -> 1.64).
template <bool kSib, bool kGrad>
__device__ __forceinline__ double walk_grad(const WNode *nodes, const Target &t,
                                            const DevParams &P, double (&acc)[3])
{
  const float hf = P.hf, hinvf = P.hinvf, h2f = P.h2f;
  const double th2d = P.theta2d;
  float hi = 0.f, comp = 0.f;  // Kahan sum of the potential
  // compensated (Kahan) float sums of the gradient: no double arithmetic in the
  // loop, where the lanes of a warp drift apart and a double instruction would
  // issue once per drifting group of lanes
  float ax = 0.f, ay = 0.f, az = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  const int root = t.nxt;
  const unsigned nn = t.end > root ? (unsigned)(t.end - root) : 0u;
  if (nn > 0u) {
    unsigned left = nn;  // steps left
    int cur = root;
    float4 na;
    int4 nm;
    load_node(nodes, cur, na, nm);
    bool go;
    do {
      const float dx = na.x - t.q[0], dy = na.y - t.q[1], dz = na.z - t.q[2];
      const float r2 = dist2(na, t.q);
      const float lo = __int_as_float(nm.z);
      const float up = kSib ? lo * kBandRatio : __int_as_float(nm.w);
      bool open = r2 < lo;
      if (r2 >= lo && r2 <= up)
        open = exact_open(na, t.q[0], t.q[1], t.q[2], __int_as_float(nm.x & 0x7fffffff), th2d);
      const int next = open ? (kSib ? nm.w : cur + 1) : nm.y;
      go = --left > 0u && (unsigned)(next - root) < nn;
      cur = go ? next : root;          // the last load is not used
      const float mass = fabsf(na.w);  // cells carry their mass with the sign bit set
      load_node(nodes, cur, na, nm);
      const float rinv = rsqrt_normal(fmaxf(r2, 1e-30f));
      float contrib = -mass * rinv;
      if (r2 < h2f) contrib = softened_fp32(mass, r2, rinv, hf, hinvf);
      contrib = open ? 0.f : contrib;
      const float y = __fsub_rn(contrib, comp);
      const float sum = __fadd_rn(hi, y);
      comp = __fsub_rn(__fsub_rn(sum, hi), y);
      hi = sum;
      if (kGrad && !open) {
        float w;  // gradient weight: grad phi -= m * w * dx
        if (r2 >= h2f) {
          w = rinv * rinv * rinv;
        } else {
          const float u = r2 * rinv * hinvf;
          const float iu = hf * rinv;  // 1/u
          const float dwp = u < 0.5f
                                ? u * (10.666666666667f + u * u * (32.0f * u - 38.4f))
                                : -0.066666666667f * iu * iu +
                                      u * (21.333333333333f +
                                           u * (-48.0f + u * (38.4f - 10.666666666667f * u)));
          w = r2 > 0.f ? hinvf * hinvf * dwp * rinv : 0.f;
        }
        const float mw = mass * w;
        kahan_add(ax, cx, mw * dx);
        kahan_add(ay, cy, mw * dy);
        kahan_add(az, cz, mw * dz);
      }
    } while (go);
  }
  acc[0] = dsub((double)ax, (double)cx);
  acc[1] = dsub((double)ay, (double)cy);
  acc[2] = dsub((double)az, (double)cz);
  const double base = (double)__fdiv_rn(t.mself, P.eps);  // cancels the self term
  return dadd(dadd(base, (double)hi), -(double)comp);
}

// The target's gradient and its term of the total energy.
template <bool kGrad>
__device__ __forceinline__ void finish_grad(const Ctx &c, const Target &t, double pot_sum,
                                            const double (&acc)[3])
{
  if (!t.active) return;
  const DevParams &P = c.P;
  const SegState &sg = c.seg[t.s];
  const double ga = ddiv((double)P.G, (double)P.a);
  const double pot = dmul(pot_sum, ga);
  const float4 a = c.pm[t.pid], v = c.vel[t.pid];
  const float tp[3] = {a.x, a.y, a.z}, tv[3] = {v.x, v.y, v.z};
  float dv[3];
  relvel(tp, tv, sg.ref_pos, sg.ref_vel, dv, P);
  const double m = (double)a.w;
  const double k2 = (double)dv[0] * dv[0] + (double)dv[1] * dv[1] + (double)dv[2] * dv[2];
  const double ha = (double)P.Hz * (double)P.a;
  const int i = t.pid;  // no list permutation in this call: input position
  if (kGrad) {
    if (c.grad_pos)
      for (int j = 0; j < 3; j++)
        c.grad_pos[first_coord(i) + j] = (float)(m * (ha * dv[j] - ga * acc[j]));
    if (c.grad_vel)
      for (int j = 0; j < 3; j++) c.grad_vel[first_coord(i) + j] = (float)(m * dv[j]);
    if (c.grad_mass) c.grad_mass[i] = (float)(0.5 * k2 + pot);
  }
  c.e_part[i] = 0.5 * m * k2 + 0.5 * m * pot;
}

template <int kB, bool kSib, bool kGrad>
__global__ void __launch_bounds__(kB) k_grad_walk(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  Target t;
  load_target<true>(c, blockIdx.x * kB + threadIdx.x, total, t);
  double acc[3];
  const double pot = walk_grad<kSib, kGrad>(kSib ? c.nd2 : c.nd, t, c.P, acc);
  finish_grad<kGrad>(c, t, pot, acc);
}

// The energies alone, two neighbouring targets per lane (walk_pair).
__global__ void __launch_bounds__(kPB, 3) k_grad_walk_pair(Ctx c, int total)
{
  HBTU_KERNEL_PROLOGUE();
  Target t[2];
  int ninter[2];
  double pot[2];
  const double acc[3] = {0., 0., 0.};
  walk_targets_pair(c, total, t, pot, ninter);
#pragma unroll
  for (int k = 0; k < 2; k++) finish_grad<false>(c, t[k], pot[k], acc);
}

template <bool kSib, bool kGrad>
void launch_grad(Ctx &c, int n)
{
  if (n >= 152 * 4 * 512)
    launch_k(k_grad_walk<512, kSib, kGrad>, (n + 511) / 512, 512, 0, c.st, c, n);
  else if (n >= 152 * 4 * 256)
    launch_k(k_grad_walk<256, kSib, kGrad>, (n + 255) / 256, 256, 0, c.st, c, n);
  else
    launch_k(k_grad_walk<128, kSib, kGrad>, (n + 127) / 128, 128, 0, c.st, c, n);
}

}  // namespace

void launch_list_order(Ctx &c, const PassPlan &pl)
{
  if (!list_order(c, pl)) return;
  int sbits = 0;
  while ((1 << sbits) < c.S) sbits++;
  const int bits = std::min(7, (40 - sbits) / 3);
  launch_k(k_list_keys, (c.N + kWB - 1) / kWB, kWB, 0, c.st, c, bits);
  HBTU_LAUNCHED();
  int words[8], shifts[8], np = 0;
  for (int b = 0; b < sbits + 3 * bits; b += 8) {
    words[np] = 0;
    shifts[np++] = b;
  }
  radix_sort(c.sb, c.N, words, shifts, np, c.st);
  launch_k(k_list_write, (c.N + kWB - 1) / kWB, kWB, 0, c.st, c);
  HBTU_LAUNCHED();
}

void launch_walk(Ctx &c, const PassPlan &pl)
{
  const int n = pl.ntgt_total;
  if (n <= 0) return;
  if (pl.norder > 0) launch_bound_order(c);
  const unsigned blocks = (n + kWB - 1) / kWB;
  if (c.P.precision == HBTU_PRECISION_FP64)
    launch_k(k_walk_fp64, blocks, kWB, 0, c.st, c, n);
  else if (c.opt_schedule == 1 && c.opt_leaf_runs)
    launch_k(k_walk_fp32<true>, blocks, kWB, 0, c.st, c, n);
  else if (c.opt_schedule == 1)
    launch_k(k_walk_fp32<false>, blocks, kWB, 0, c.st, c, n);
  else if (pair_walk(c, pl))
    launch_after(k_walk_fp32_pair, pair_blocks(n), kPB, 0, c.st, c, n);
  else if (sibling_walk(c, pl))  // the tree build made the sibling-block records
    launch_lean<true>(c, n);
  else
    launch_lean<false>(c, n);
  HBTU_LAUNCHED();
}

void launch_grad_walk(Ctx &c, const PassPlan &pl)
{
  const int n = pl.ntgt_total;
  if (n <= 0) return;
  const bool grad = c.grad_pos || c.grad_vel || c.grad_mass;
  const bool sib = sibling_walk(c, pl);  // the tree build made the sibling-block records
  if (pair_walk(c, pl))  // no gradient asked for
    launch_k(k_grad_walk_pair, pair_blocks(n), kPB, 0, c.st, c, n);
  else if (sib && grad)
    launch_grad<true, true>(c, n);
  else if (sib)
    launch_grad<true, false>(c, n);
  else if (grad)
    launch_grad<false, true>(c, n);
  else
    launch_grad<false, false>(c, n);
  HBTU_LAUNCHED();
}

}  // namespace hbtu
