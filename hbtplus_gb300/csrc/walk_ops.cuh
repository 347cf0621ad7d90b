// walk_ops.cuh -- one target's Barnes-Hut walk and its binding energy, shared
// by the batch walks (walk.cu: one launch per pass over every active
// subhalo's targets) and the per-subhalo loop (small.cu).
//
// Reference: GravityTree_t::EvaluatePotential (src/gravity_tree.cpp:79-164),
// BindingEnergy (:166-175) and the two energy loops of Subhalo_t::Unbind
// (src/subhalo_unbind.cpp:319-328 correction, :341-354 full pass).  A target
// performs exactly the reference's stackless walk: at a cell it opens (goes to
// the first child) when len*len > r*r*theta^2, otherwise it takes the cell's
// monopole and jumps to the skip pointer; particles are never opened.
#pragma once
#include "device_common.cuh"

namespace hbtu {

struct Target {
  int s, epos, pid, nxt, end;
  bool active;
  float q[3];  // position used by the walk (relative for FP32, absolute for FP64)
  float mself;
};

// The walk of particle `pid` at list position `epos` of subhalo s in the
// coming pass: its position (relative to the frame centre for kRel, else
// absolute), the self term it cancels (full and refine passes, if it is in
// the tree), and the node range of the subhalo's tree.
template <bool kRel>
__device__ __forceinline__ void init_target(const Ctx &c, const SegState &sg, int s, int epos,
                                            int pid, bool active, int root, Target &t)
{
  t.s = s;
  t.epos = epos;
  t.pid = pid;
  t.active = active;
  t.nxt = kDone;
  t.end = 0;
  t.mself = 0.f;
  t.q[0] = t.q[1] = t.q[2] = 0.f;
  if (!active) return;
  const float4 a = c.pm[pid];
  if (sg.mode != MODE_CORRECTION && epos - sg.off < sg.ntree) t.mself = fmul(a.w, sg.mfac);
  if (kRel) {
    t.q[0] = rel_coord(a.x, sg.fc[0], c.P);
    t.q[1] = rel_coord(a.y, sg.fc[1], c.P);
    t.q[2] = rel_coord(a.z, sg.fc[2], c.P);
  } else {
    t.q[0] = a.x;
    t.q[1] = a.y;
    t.q[2] = a.z;
  }
  const int nn = sg.ntree > 0 ? min(sg.nnodes, 2 * sg.ntree) : 0;  // node slots of this subhalo
  t.end = root + nn;
  t.nxt = nn > 0 ? root : kDone;
}

// x / a for the scale factor a, correctly rounded: a quotient from the
// rounded reciprocal, corrected twice by its exact remainder (Markstein 1990:
// the first correction brings it within a unit in the last place, the second
// rounds it correctly).  Five double operations; a quotient or remainder that
// could leave the normal range takes the division.
__device__ __forceinline__ double over_scale(double x, const DevParams &P)
{
  if (P.a == 1.f) return x;
  const unsigned ex = (unsigned)((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ffu;
  if (ex - 200u > 1600u) return ddiv(x, P.ad);
  double q = dmul(x, P.a_inv);
  q = __fma_rn(__fma_rn(-P.ad, q, x), P.a_inv, q);
  return __fma_rn(__fma_rn(-P.ad, q, x), P.a_inv, q);
}

// BindingEnergy (full pass) or the correction update, and the store.
__device__ __forceinline__ void finish_target(const Ctx &c, const SegState &sg, const Target &t,
                                              double pot_sum)
{
  if (!t.active) return;
  const DevParams &P = c.P;
  const double pot = over_scale(dmul(pot_sum, P.Gd), P);
  const float4 a = c.pm[t.pid], v = c.vel[t.pid];
  const float tp[3] = {a.x, a.y, a.z}, tv[3] = {v.x, v.y, v.z};
  float E;
  if (sg.mode != MODE_CORRECTION) {
    float dv[3];
    relvel(tp, tv, sg.ref_pos, sg.ref_vel, dv, P);
    E = d2f(dadd(half_of(f2d(vdot(dv, dv))), pot));
  } else {
    float ov[3];
    relvel(tp, tv, sg.old_pos, sg.old_vel, ov, P);
    const float tt = fadd(vdot(ov, sg.dV), sg.dK);
    E = d2f(dadd(f2d(c.eE[t.epos]), dsub(f2d(tt), pot)));
  }
  if (sg.mode == MODE_REFINE)
    c.eR[t.epos] = E;
  else
    c.eE[t.epos] = E;
  if (c.pot_out) c.pot_out[t.epos] = pot;
}

// Adds a warp's interaction counts to its subhaloes' totals (one atomic per
// warp when the warp holds one subhalo).
__device__ __forceinline__ void count_interactions(const Ctx &c, int s, int n)
{
  const unsigned full = 0xffffffffu;
  const int s0 = __shfl_sync(full, s, 0);
  if (__all_sync(full, s == s0)) {
    const int sum = __reduce_add_sync(full, n);
    if ((threadIdx.x & 31) == 0 && sum)
      atomicAdd((unsigned long long *)&c.seg[s0].interactions, (unsigned long long)sum);
  } else if (n) {
    atomicAdd((unsigned long long *)&c.seg[s].interactions, (unsigned long long)n);
  }
}

// Opening test of the reference, len*len > r*r*theta^2: float first, and in
// double with the reference's operation order when within 1e-5 of the edge.
__device__ __forceinline__ bool opens(float4 na, const float q[3], float l2, float r2, float theta2,
                                      double th2d)
{
  const float thr = r2 * theta2;
  bool open = l2 > thr;
  if (l2 > 0.f && fabsf(l2 - thr) <= 1e-5f * thr) {  // particles (l2 = 0) never open
    const double ex = dsub((double)na.x, (double)q[0]);
    const double ey = dsub((double)na.y, (double)q[1]);
    const double ez = dsub((double)na.z, (double)q[2]);
    const double er2 = dadd(dadd(dmul(ex, ex), dmul(ey, ey)), dmul(ez, ez));
    open = (double)l2 > dmul(er2, th2d);
  }
  return open;
}

__device__ __forceinline__ float dist2(float4 na, const float q[3])
{
  const float dx = na.x - q[0], dy = na.y - q[1], dz = na.z - q[2];
  return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// FP32 potential sum without double arithmetic in the walk loop (this GPU's
// FP64 rate is 1/64 of its FP32 rate): interactions go into a short float
// partial sum `f`, which is flushed every few steps into a compensated
// (Kahan) float total hi - c.  The total is formed in double once per target.
struct PotAcc {
  float f = 0.f, hi = 0.f, c = 0.f;
  __device__ __forceinline__ void flush()
  {
    const float y = __fsub_rn(f, c);
    const float t = __fadd_rn(hi, y);
    c = __fsub_rn(__fsub_rn(t, hi), y);
    hi = t;
    f = 0.f;
  }
  __device__ __forceinline__ double total(double base) const
  {
    return dadd(dadd(base, (double)hi), dsub((double)f, (double)c));
  }
};

// Softened potential without a division: 1/u = h/r = h * rinv.
__device__ __forceinline__ float softened_fp32(float m, float r2, float rinv, float hf, float hinvf)
{
  const float r = r2 * rinv;
  const float u = r * hinvf;
  float wp;
  if (u < 0.5f)
    wp = -2.8f + u * u * (5.333333333333f + u * u * (6.4f * u - 9.6f));
  else
    wp = -3.2f + 0.066666666667f * (hf * rinv) +
         u * u * (10.666666666667f + u * (-16.0f + u * (9.6f - 2.133333333333f * u)));
  return m * hinvf * wp;
}

// One monopole interaction in FP32: -m/r outside the softening length h,
// the cubic-spline potential inside it (Springel, Yoshida & White 2001).
__device__ __forceinline__ void interact(float4 na, float r2, float &pot_f, float hf, float h2f,
                                         float hinvf)
{
  const float rinv = rsqrtf(fmaxf(r2, 1e-30f));
  const float m = fabsf(na.w);  // cells carry their mass with the sign bit set
  if (r2 >= h2f)
    pot_f = fmaf(-m, rinv, pot_f);
  else
    pot_f += softened_fp32(m, r2, rinv, hf, hinvf);
}

// The reference's opening decision in double, for a target whose float test
// fell within 1e-5 of the threshold.
__device__ __forceinline__ bool opens_double(float4 na, float qx, float qy, float qz, float l2,
                                             double th2d)
{
  const double ex = dsub(f2d(na.x), f2d(qx));
  const double ey = dsub(f2d(na.y), f2d(qy));
  const double ez = dsub(f2d(na.z), f2d(qz));
  const double er2 = dadd(dadd(dmul(ex, ex), dmul(ey, ey)), dmul(ez, ez));
  return f2d(l2) > dmul(er2, th2d);
}

// As a call, so that a walk's steps issue no double instruction otherwise.
static __device__ __noinline__ bool exact_open(float4 na, float qx, float qy, float qz, float l2,
                                               double th2d)
{
  return opens_double(na, qx, qy, qz, l2, th2d);
}

// FP32 walk of one target, lane schedule: the opening test is two compares
// against per-cell thresholds precomputed from len^2/theta^2 (the
// reference's double test decides the rare cases in between), every
// interaction goes straight into a compensated float sum, and the walk ends
// when the index leaves the tree (skip pointers that leave it are kDone).
//   kSib = false: preorder records; the next node is cur + 1 on opening, the
//     skip pointer otherwise.
//   kSib = true: the sibling-block records (nd2): a cell's children sit in
//     consecutive slots, so the sibling an accepted cell hands on to is
//     usually in the same cache line; the next node is the first-child
//     pointer (m.w) on opening and the skip pointer otherwise, and the upper
//     threshold is recomputed from the lower one.  Same nodes, same order,
//     same sums as the preorder walk.
// Both stop after as many steps as the tree has nodes, whatever its pointers.
//
// A step's chain is load, distance, decision, next load; the interaction hangs
// off it.  The next node's load is therefore issued as soon as the decision is
// known, before the interaction is computed.  With few targets the chip waits on
// that chain, and kFlat keeps the interaction from stretching it: the softened
// potential is computed on every step and selected, without a branch that the
// lanes of a warp take apart (first pass of a 1.1e5-particle subhalo: 925 -> 657
// us, 5e4 particles 732 -> 474 us).  With many targets the instructions count, and
// the branch is the better form (867,289 targets: 2 to 4% faster than kFlat).
// Returns the potential sum (self term cancelled, before G/a); *ninter counts
// the interactions.
constexpr float kBandRatio = 1.0000200002f;  // (1 + 1e-5) / (1 - 1e-5), rounded up

// 1/sqrt(x) for x >= 1e-30: without the subnormal inputs' scaling, which such an
// x never needs, the result is rsqrtf's.
__device__ __forceinline__ float rsqrt_normal(float x)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// softened_fp32 without a branch: both polynomials (the fused multiply-adds
// that softened_fp32 contracts to), then one is taken.
__device__ __forceinline__ float softened_select(float m, float r2, float rinv, float hf,
                                                 float hinvf)
{
  const float u = __fmul_rn(__fmul_rn(r2, rinv), hinvf);
  const float uu = __fmul_rn(u, u);
  const float in = __fmaf_rn(
      uu, __fmaf_rn(uu, __fmaf_rn(6.4f, u, -9.6f), 5.333333333333f), -2.8f);
  const float out = __fmaf_rn(
      uu,
      __fmaf_rn(u, __fmaf_rn(u, __fmaf_rn(-2.133333333333f, u, 9.6f), -16.0f), 10.666666666667f),
      __fmaf_rn(0.066666666667f, __fmul_rn(hf, rinv), -3.2f));
  return __fmul_rn(__fmul_rn(m, hinvf), u < 0.5f ? in : out);
}

template <bool kSib, bool kFlat>
__device__ __forceinline__ double walk_lean(const WNode *nodes, const Target &t,
                                            const DevParams &P, int *ninter)
{
  const float hf = P.hf, hinvf = P.hinvf, h2f = P.h2f;
  float hi = 0.f, comp = 0.f;  // Kahan sum
  int nacc = 0;
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
      const float r2 = dist2(na, t.q);
      const float lo = __int_as_float(nm.z);
      const float up = kSib ? lo * kBandRatio : __int_as_float(nm.w);
      bool open = r2 < lo;
      if (r2 >= lo && r2 <= up)
        open = exact_open(na, t.q[0], t.q[1], t.q[2], __int_as_float(nm.x & 0x7fffffff),
                          P.theta2d);
      const int next = open ? (kSib ? nm.w : cur + 1) : nm.y;
      go = --left > 0u && (unsigned)(next - root) < nn;
      cur = go ? next : root;  // the last load is not used
      const float mass = fabsf(na.w);
      load_node(nodes, cur, na, nm);
      const float rinv = rsqrt_normal(fmaxf(r2, 1e-30f));
      float contrib = __fmul_rn(-mass, rinv);
      if (kFlat) {
        const float near = softened_select(mass, r2, rinv, hf, hinvf);
        contrib = r2 < h2f ? near : contrib;
      } else if (r2 < h2f) {
        contrib = softened_fp32(mass, r2, rinv, hf, hinvf);
      }
      // an opened node adds zero, which can still settle the compensation
      const float y = __fsub_rn(open ? 0.f : contrib, comp);
      const float s = __fadd_rn(hi, y);
      comp = __fsub_rn(__fsub_rn(s, hi), y);
      hi = s;
      nacc += open ? 0 : 1;
    } while (go);
  }
  *ninter = nacc;
  const double base = f2d(__fdiv_rn(t.mself, P.eps));  // cancels the self term
  return dadd(dadd(base, f2d(hi)), -f2d(comp));
}

// Two floats in one 64-bit register: each half rounds as the float operation
// does, and the two take one issue slot.
using Float2 = unsigned long long;
__device__ __forceinline__ Float2 f2_pack(const float (&v)[2])
{
  Float2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v[0]), "f"(v[1]));
  return r;
}
__device__ __forceinline__ void f2_unpack(Float2 x, float (&v)[2])
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(x));
}
__device__ __forceinline__ Float2 f2_add(Float2 a, Float2 b)
{
  Float2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Float2 f2_sub(Float2 a, Float2 b)
{
  Float2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Float2 f2_mul(Float2 a, Float2 b)
{
  Float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Float2 f2_fma(Float2 a, Float2 b, Float2 c)
{
  Float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct PairSums {
  Float2 hi, comp;  // Kahan sums
  int ninter[2];
};

// FP32 walks of two neighbouring targets by one lane, over the union of the
// nodes they visit (1.18 per node of one walk): each node is loaded once for
// both.  A target that accepts a cell the other opens waits at the cell's skip
// pointer.  Preorder records: indices only grow along a walk, so a target is at
// the current node when the index it waits at has been reached, and the walk
// ends when the index leaves the tree (a skip pointer that did not grow would
// count as the next index).  Each target visits its walk_lean nodes in their
// order and takes the same float operations, so its sum is the same bit for bit.
//
// walk_lean's large launches wait for L1 (16.4 data wavefronts per load of 32
// records, 84 to 90% of the cycles).  This loop takes 76 instructions per node of
// the union against 2 x 49, two fifths of the loads away, and issues on 71% of the
// cycles at 74% of L1's wavefronts (79% of the sectors hit); dropping a tenth of its
// instructions did not change the time.  What made it pay: pairs of float operations
// in one instruction (distances and sums; the spline's constants stay immediates, as
// pairs they cost 20 registers), and the rare double test and the near branch as
// loops, which the compiler does not predicate.  The sibling-block records brought
// nothing here (2.7e7 targets: 124 ms with them, 122 without), and their layout is
// not built.
// With walk_grad's sums the same loop gained nothing (1e6 targets: 5.9 ms against
// 5.7): 12 more registers and selects.
//
// The walks of those of t[0], t[1] with here[k], in the tree of nodes root .. end - 1.
__device__ __forceinline__ void walk_pair(const WNode *nodes, const Target (&t)[2],
                                          const bool (&here)[2], int root, int end,
                                          const DevParams &P, PairSums &sums)
{
  int at[2] = {here[0] ? root : kDone, here[1] ? root : kDone};
  Float2 hi = sums.hi, comp = sums.comp;
  int cur = root;
  float4 na;
  int4 nm;
  load_node(nodes, cur, na, nm);
  bool go;
  do {
    bool open[2], vis[2];
    float r2[2], neg[2], rinv[2], dx[2], dy[2], dz[2];
    const int child = cur + 1, skip = max(nm.y, child);
    const float lo = __int_as_float(nm.z), up = __int_as_float(nm.w);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      dx[k] = na.x - t[k].q[0];
      dy[k] = na.y - t[k].q[1];
      dz[k] = na.z - t[k].q[2];
    }
    const Float2 x = f2_pack(dx), y = f2_pack(dy), z = f2_pack(dz);
    f2_unpack(f2_fma(z, z, f2_fma(x, x, f2_mul(y, y))), r2);  // dist2
#pragma unroll
    for (int k = 0; k < 2; k++) open[k] = r2[k] < lo;
    int band = (!open[0] && r2[0] <= up) || (!open[1] && r2[1] <= up);
    while (__builtin_expect(band, 0)) {
#pragma unroll
      for (int k = 0; k < 2; k++)
        if (!open[k] && r2[k] <= up)
          open[k] = opens_double(na, t[k].q[0], t[k].q[1], t[k].q[2],
                                 __int_as_float(nm.x & 0x7fffffff), P.theta2d);
      asm volatile("mov.u32 %0, 0;" : "=r"(band));
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      vis[k] = at[k] <= cur;
      const bool take = vis[k] && !open[k];
      neg[k] = take ? -fabsf(na.w) : 0.f;
      if (take) {
        sums.ninter[k]++;
        at[k] = skip;
      }
    }
    cur = (vis[0] && open[0]) || (vis[1] && open[1]) ? child : skip;
    go = cur < end;
    if (go) load_node(nodes, cur, na, nm);
#pragma unroll
    for (int k = 0; k < 2; k++) rinv[k] = rsqrt_normal(fmaxf(r2[k], 1e-30f));
    Float2 contrib = f2_mul(f2_pack(neg), f2_pack(rinv));
    int near = fminf(r2[0], r2[1]) < P.h2f;
    while (near) {
      float v[2];
      f2_unpack(contrib, v);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const float soft = softened_select(-neg[k], r2[k], rinv[k], P.hf, P.hinvf);
        v[k] = r2[k] < P.h2f ? soft : v[k];
      }
      contrib = f2_pack(v);
      asm volatile("mov.u32 %0, 0;" : "=r"(near));
    }
    // an opened node adds zero, which can still settle the compensation
    const Float2 add = f2_sub(contrib, comp), sum = f2_add(hi, add);
    float h[2], c[2], s[2], e[2];
    f2_unpack(hi, h);
    f2_unpack(comp, c);
    f2_unpack(sum, s);
    f2_unpack(f2_sub(f2_sub(sum, hi), add), e);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      h[k] = vis[k] ? s[k] : h[k];
      c[k] = vis[k] ? e[k] : c[k];
    }
    hi = f2_pack(h);
    comp = f2_pack(c);
  } while (go);
  sums.hi = hi;
  sums.comp = comp;
}

// The softened FP64 interaction with the reference's arithmetic, operation by operation
// (src/gravity_tree.cpp:136-160).
static __device__ __noinline__ double fp64_softened(double r, double mass, double h_inv)
{
  const double u = dmul(r, h_inv);
  const double uu = dmul(u, u);
  double wp;
  if (u < 0.5)
    wp = dadd(-2.8, dmul(uu, dadd(5.333333333333, dmul(uu, dsub(dmul(6.4, u), 9.6)))));
  else
    wp = dadd(dadd(-3.2, ddiv(0.066666666667, u)),
              dmul(uu, dadd(10.666666666667,
                            dmul(u, dadd(-16.0, dmul(u, dsub(9.6, dmul(2.133333333333, u))))))));
  return dmul(dmul(mass, h_inv), wp);
}

static __device__ __noinline__ double fp64_contrib_any(double r2, double mass, double h, double h_inv)
{
  const double r = __dsqrt_rn(r2);
  if (r >= h) return -ddiv(mass, r);
  return fp64_softened(r, mass, h_inv);
}

// Whether a correction x / y, taken with a reciprocal of y good to a few units in the last
// place, may have rounded the corrected value the wrong way: only where x / y is within
// 2^-46 of half a unit of that value, a power of two, so where the mantissas of x and y
// agree to 64 units.  (The bits of x = 0 count as mantissa zero: then exact, and
// perhaps reported.)
__device__ __forceinline__ bool near_half(double x, double y)
{
  const unsigned long long d =
      (unsigned long long)__double_as_longlong(x) - (unsigned long long)__double_as_longlong(y);
  return ((d + 64ull) & 0xfffffffffffffull) <= 128ull;
}

// The interaction at squared distance r2: -mass / r outside the softening length, r
// the rounded root, both operations correctly rounded as the reference's are.
// Root and reciprocal together, from one float approximation of 1/sqrt(r2): the
// coupled Newton iteration g -> sqrt(r2), k -> 1 / (2 sqrt(r2)), then the root
// corrected by its exact remainder, and the quotient from 2k corrected twice by
// its own (Markstein 1990; Cornea, Harrison & Tang 2002): 14 double operations, where
// the two library operations took about 20 of the FP64 pipe, which is what
// bounds this walk.  The corrections are taken with k, not with a correctly rounded
// reciprocal, so a root or quotient within 2^-50 of a unit of the midpoint of two
// doubles could fall on its other side (58 of 1622 quotients built to lie that close
// did); where the last remainder says that it may be (near_half: integer code),
// and outside the range where no step can leave the normal doubles or floats,
// the library operations.
__device__ __forceinline__ double fp64_contrib(double r2, float mass, const DevParams &P)
{
  const unsigned ex = (unsigned)((unsigned long long)__double_as_longlong(r2) >> 52);
  const unsigned em = __float_as_uint(mass) >> 23;
  if (ex - (1023u - 100u) > 200u || em - 27u > 200u)
    return fp64_contrib_any(r2, f2d(mass), P.h, P.h_inv);
  const double y = f2d(rsqrt_normal(d2f(r2)));
  double g = dmul(r2, y), k = half_of(y);
  double e = __fma_rn(-g, k, 0.5);
  g = __fma_rn(g, e, g);
  k = __fma_rn(k, e, k);
  e = __fma_rn(-g, k, 0.5);
  g = __fma_rn(g, e, g);
  k = __fma_rn(k, e, k);
  const double rem = __fma_rn(-g, g, r2);  // r = g + rem / 2g
  const double r = __fma_rn(rem, k, g);
  const double m = f2d(mass);
  // positive doubles compare as their bits do
  if (__double_as_longlong(r) < __double_as_longlong(P.h) && !near_half(rem, g))
    return fp64_softened(r, m, P.h_inv);
  const double inv = __longlong_as_double(__double_as_longlong(k) + (1ll << 52));
  double q = dmul(m, inv);
  q = __fma_rn(__fma_rn(-q, r, m), inv, q);
  const double qrem = __fma_rn(-q, r, m);
  if (near_half(rem, g) || near_half(qrem, r)) return fp64_contrib_any(r2, m, P.h, P.h_inv);
  return -__fma_rn(qrem, inv, q);
}

// r^2 of a collected node (walk_fp64).
__device__ __forceinline__ double fp64_r2(float4 item)
{
  if (item.x != item.x) return __hiloint2double(__float_as_int(item.y), __float_as_int(item.z));
  const double dx = f2d(item.x), dy = f2d(item.y), dz = f2d(item.z);
  return __fma_rn(dz, dz, __fma_rn(dx, dx, dmul(dy, dy)));
}

// NEAREST((double)x - (double)q) for float coordinates, as the reference
// forms a node-target separation.  When the float difference s is exact (a
// float TwoSum with a zero error term) it is the double difference, and for
// |s| < box its wrap is exact in float as well (Sterbenz), so the separation is
// a float; exact: whether that is so.  Otherwise the double path.
__device__ __forceinline__ float sep_float(float x, float q, const DevParams &P, bool &exact)
{
  const float s = __fsub_rn(x, q);
  const float bb = __fsub_rn(s, x);
  const float err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(-q, bb));
  exact = exact && err == 0.f && (!P.periodic || fabsf(s) < P.box);
  return P.periodic ? nearest_f(s, P) : s;
}

static __device__ __noinline__ double sep_fp64(float x, float q, int periodic, float box,
                                               float boxhalf)
{
  const double d = dsub(f2d(x), f2d(q));
  if (!periodic) return d;
  return d > f2d(boxhalf) ? dsub(d, f2d(box)) : d < -f2d(boxhalf) ? dadd(d, f2d(box)) : d;
}

// r^2 in the reference's order from double separations.
static __device__ __noinline__ double dist2_fp64(float4 na, float qx, float qy, float qz, int periodic,
                                                 float box, float boxhalf)
{
  const double dx = sep_fp64(na.x, qx, periodic, box, boxhalf);
  const double dy = sep_fp64(na.y, qy, periodic, box, boxhalf);
  const double dz = sep_fp64(na.z, qz, periodic, box, boxhalf);
  return dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
}

static __device__ __noinline__ bool opens_fp64(double r2, float l2, double th2d)
{
  return f2d(l2) > dmul(r2, th2d);
}

// FP64 walk of one target, lane schedule, over the preorder records: absolute
// float coordinates (nd_abs), NEAREST per interaction, the reference's
// arithmetic and summation order.  The double pipe bounds it, so
//   * a step that opens its cell uses none of it: the separations are floats where
//     exact (nearly always), and their float r^2 decides by the record's
//     thresholds (l^2/theta^2 (1 -+ 1e-5)); in between the reference's comparison
//     is made in double;
//   * the accepted nodes are collected, kFp64Queue at a time, and then
//     evaluated by all lanes of a warp together: a double instruction costs the
//     same however few lanes run it, and of the lanes of a step a third opens
//     its cell;
//   * the squares of float separations are exact in double, so the two additions of
//     r^2 are fused with them.
// All lanes of a warp call it together (lanes without a target with an empty
// range).  Returns the potential sum (self term cancelled, before G/a).  400
// subhaloes of up to 24,000 particles: 13.0 -> 9.2 ms a call (12.6 -> 8.9 with other
// sizes of the same law); 1000 of up to 1900, in the per-subhalo kernel: 27 -> 8.7 ms.
// (Two nodes' chains interleaved: no gain.)
constexpr int kFp64Queue = 8;

__device__ __forceinline__ double walk_fp64(const Ctx &c, const Target &t, int *ninter)
{
  const DevParams &P = c.P;
  double pot_d = f2d(__fdiv_rn(t.mself, P.eps));
  int n = 0;
  int cur = t.nxt;
  const int end = t.end;
  float4 queue[kFp64Queue];  // separation and mass; or a NaN and r^2 as two words
  while (__any_sync(0xffffffffu, cur < end)) {
    int cnt = 0;
    while (cur < end && cnt < kFp64Queue) {
      const float4 na = c.nd_abs[cur];
      const int4 nm = c.nd[cur].m;
      bool exact = true;
      float4 item = make_float4(sep_float(na.x, t.q[0], P, exact), sep_float(na.y, t.q[1], P, exact),
                                sep_float(na.z, t.q[2], P, exact), na.w);
      const float r2f = item.x * item.x + item.y * item.y + item.z * item.z;
      bool open = r2f < __int_as_float(nm.z);
      if (!exact || (!open && r2f <= __int_as_float(nm.w))) {
        const double r2 = dist2_fp64(na, t.q[0], t.q[1], t.q[2], P.periodic, P.box, P.boxhalf);
        open = opens_fp64(r2, __int_as_float(nm.x & 0x7fffffff), P.theta2d);
        item.x = __int_as_float(0x7fffffff);
        item.y = __int_as_float(__double2hiint(r2));
        item.z = __int_as_float(__double2loint(r2));
      }
      if (open) {
        cur = cur + 1;
      } else {
        const int sk = nm.y;
        cur = (unsigned)(sk - cur - 1) < (unsigned)(end - cur - 1) ? sk : end;
        queue[cnt++] = item;
      }
    }
    n += cnt;
    __syncwarp();  // evaluate together
#pragma unroll 1
    for (int k = 0; k < cnt; k++) {
      const float4 item = queue[k];
      pot_d = dadd(pot_d, fp64_contrib(fp64_r2(item), item.w, P));
    }
  }
  *ninter = n;
  return pot_d;
}

}  // namespace hbtu
