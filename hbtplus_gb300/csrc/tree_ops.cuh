// tree_ops.cuh -- the per-element steps of the octree build, shared by the
// batch kernels (tree.cu: one thread per element of every active subhalo) and
// the per-subhalo loop (small.cu: one block walks one subhalo through them).
//
// Reference: OctTree_t::Build (src/oct_tree.tpp:16-144) and
// GravityTree_t::UpdateInternalNodes / ProcessNode / FillNodeCenter
// (src/gravity_tree.cpp:18-77).  The steps:
//   seg_cube       bounding cube and depth of geometric subdivision;
//   seg_key        octal key of one particle (the reference's comparisons
//                  x > centre with centres halved in double);
//   karras_elem    one internal node of the Karras (2012) radix tree over a
//                  subhalo's sorted keys;
//   cells_elem     whether an internal node is an octree cell;
//   leaves_elem    preorder slot and record of one particle leaf;
//   cellnodes_elem preorder slot, skip pointer and side of one cell;
//   cell_moment    mass and centre of mass of one cell from its children,
//                  in octant order, in double, rounded to float per cell.
// Element e of a subhalo's tree is its e-th key in sorted order; `base` is the
// index of its first element in the element arrays, and its node slots are
// [2*base, 2*base + 2*n).
#pragma once
#include "device_common.cuh"

namespace hbtu {

__device__ __forceinline__ int ll_tz(long long v) { return v ? __ffsll(v) - 1 : 64; }

// A double in units of 2^-E, if an integer below 2^62 there (else false).
__device__ __forceinline__ bool double_fixed(double d, int E, long long &X)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const int ex = (int)((b >> 52) & 0x7ffull);
  unsigned long long v = b & 0xfffffffffffffull;
  if (ex == 0) {  // zero (a subnormal is no multiple of any unit used here)
    X = 0;
    return v == 0ull;
  }
  if (ex == 0x7ff) return false;
  v |= 1ull << 52;
  const int sh = ex - 1075 + E;
  if (sh >= 0) {
    if (sh > 9) return false;
    v <<= sh;
  } else {
    if (-sh > 52 || (v & ((1ull << -sh) - 1ull)) != 0ull) return false;
    v >>= -sh;
  }
  X = (long long)(b >> 63 ? 0ull - v : v);
  return true;
}

// Fixed-point form of the key computation.  The reference halves the cube in
// double: centre_k = centre_{k-1} +- len / 2^(k+1).  When the centre, len/4
// and every later increment are integers in units of 2^-E, and every centre
// fits in 53 significant bits, none of those double operations rounds, so the
// same comparisons x > centre_k can be made exactly on 64-bit integers
// (a tenth of the cost: double runs at 1/64 of the FP32 rate on this GPU).
__device__ __forceinline__ void fixed_point_cube(SegState &sg, int levels)
{
  sg.kfast = 0;
  if (levels <= 0 || !(sg.len > 0.)) return;
  long long M = 0;  // largest |centre| + len, as the bits of a positive double
  for (int j = 0; j < 3; j++)
    M = max(M, __double_as_longlong(dadd(fabs(sg.center[j]), sg.len)));
  const int top = (int)(M >> 52) - 1022;  // the largest is below 2^top
  const int E = 61 - top;                 // |values| < 2^61 in fixed point
  long long inc, least;
  if (!double_fixed(sg.len, E - 2, inc) || !double_fixed(sg.len, E - levels - 1, least)) return;
  int g = ll_tz(inc >> (levels - 1));  // trailing zeros of the smallest increment
  for (int j = 0; j < 3; j++) {
    if (!double_fixed(sg.center[j], E, sg.kc[j])) return;
    g = min(g, ll_tz(sg.kc[j]));
  }
  if (top + E - g > 53) return;  // some centre would need more than 53 bits
  sg.kinc = inc;
  sg.kscale = E;
  sg.kfast = 1;
}

// A float position in units of 2^-E, if exact (else false).
__device__ __forceinline__ bool float_fixed(float x, int E, long long &X)
{
  const unsigned b = __float_as_uint(x);
  const int ex = (int)((b >> 23) & 255u);
  if (ex == 0) {  // zero (denormals take the double path)
    X = 0;
    return (b & 0x7fffffffu) == 0u;
  }
  if (ex == 255) return false;
  const long long mant = (long long)((b & 0x7fffffu) | 0x800000u);
  const int sh = ex - 150 + E;  // x = mant * 2^(ex - 150)
  long long v;
  if (sh >= 0) {
    if (sh > 37) return false;  // would pass 2^61
    v = mant << sh;
  } else {
    if (-sh > 24 || (mant & ((1ll << -sh) - 1)) != 0) return false;
    v = mant >> -sh;
  }
  X = (b >> 31) ? -v : v;
  return true;
}

// Depth of geometric subdivision of a cube of side len: the number of
// halvings until the side is below res (the len halving rule of
// src/gravity_tree.cpp:37-40), at most kMaxLevels, from exponents and mantissas.
__device__ __forceinline__ int cube_levels(double len, float res)
{
  const unsigned long long a = (unsigned long long)__double_as_longlong(len);
  const unsigned long long r = (unsigned long long)__double_as_longlong(f2d(res));
  const int ea = (int)(a >> 52), er = (int)(r >> 52);
  if (ea > 0 && ea < 0x7ff && er > 0 && er < 0x7ff) {
    const unsigned long long low = 0xfffffffffffffull;
    return min(kMaxLevels, max(0, ea - er + ((a & low) >= (r & low) ? 1 : 0)));
  }
  int levels = 0;
  while (len >= (double)res && levels < kMaxLevels) {
    len = dmul(len, 0.5);
    levels++;
  }
  return levels;
}

// Root cube of a subhalo from the float bounding box of its tree particles
// (src/oct_tree.tpp:30-51; an empty box gives a cube of side 0) and its depth
// of geometric subdivision.  One thread does this per subhalo and pass, so the
// few double operations left (the sums and differences) matter: the halvings,
// comparisons and fixed-point forms are integer operations.
// The frame centre of the relative coordinates is the subhalo's frame.
__device__ __forceinline__ int seg_cube(SegState &sg, const float mn[3], const float mx[3],
                                        bool empty, const DevParams &P)
{
  double Len = 0.;
  for (int j = 0; j < 3; j++) {
    const double lo = f2d(mn[j]), hi = f2d(mx[j]);
    const double e = dsub(hi, lo);
    if (j == 0 || __double_as_longlong(e) > __double_as_longlong(Len)) Len = e;  // e >= 0
    sg.center[j] = half_of(dadd(hi, lo));
  }
  if (empty) Len = 0.;
  sg.len = Len;
  const int levels = cube_levels(Len, P.res);
  sg.levels = levels;
  fixed_point_cube(sg, levels);
  for (int j = 0; j < 3; j++) sg.fc[j] = sg.ref_pos[j];
  return levels;
}

// Octal key: digit k (k = 1..levels) is the octant at depth k, found with the
// reference's comparisons against centres halved in double (tpp:67-95).
// Left-aligned in 64 bits.
__device__ __forceinline__ unsigned long long seg_key(const SegState &sg, float4 a)
{
  const float x[3] = {a.x, a.y, a.z};
  unsigned long long key = 0;
  long long X[3];
  if (sg.kfast && float_fixed(x[0], sg.kscale, X[0]) && float_fixed(x[1], sg.kscale, X[1]) &&
      float_fixed(x[2], sg.kscale, X[2])) {
    long long cen[3] = {sg.kc[0], sg.kc[1], sg.kc[2]};
    long long inc = sg.kinc;
    for (int k = 0; k < sg.levels; k++) {
      unsigned d = 0;
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const bool gt = X[j] > cen[j];
        cen[j] += gt ? inc : -inc;
        d |= (unsigned)gt << j;
      }
      inc >>= 1;
      key = (key << 3) | d;
    }
    if (sg.levels > 0) key <<= (64 - 3 * sg.levels);
    return key;
  }
  double cen[3] = {sg.center[0], sg.center[1], sg.center[2]};
  double lenhalf = dmul(0.5, sg.len);
  for (int k = 0; k < sg.levels; k++) {
    lenhalf = dmul(lenhalf, 0.5);
    unsigned d = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if ((double)x[j] > cen[j]) {
        cen[j] = dadd(cen[j], lenhalf);
        d |= 1u << j;
      } else {
        cen[j] = dsub(cen[j], lenhalf);
      }
    }
    key = (key << 3) | d;
  }
  if (sg.levels > 0) key <<= (64 - 3 * sg.levels);
  return key;
}

// Longest common prefix of sorted keys i and j (index tie-break for equal keys).
__device__ __forceinline__ int kdelta(const unsigned long long *keys, int n, int i, int j)
{
  if (j < 0 || j >= n) return -1;
  const unsigned long long a = keys[i], b = keys[j];
  if (a != b) return __clzll(a ^ b);
  return 64 + __clz((unsigned)(i ^ j));
}

// Internal node i (0 <= i < n-1) of the Karras (2012) binary radix tree over
// a subhalo's sorted keys: its key range, split depth, and the parent links of
// its two children (parentI for an internal child, parentL for a leaf).
__device__ __forceinline__ void karras_elem(const Ctx &c, const unsigned long long *keys, int base,
                                            int n, int i)
{
  const int e = base + i;
  const int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = kdelta(keys, n, i, i - d);
  int lmax = 2;
  while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dn = kdelta(keys, n, i, j);
  int sp = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (kdelta(keys, n, i, i + (sp + t) * d) > dn) sp += t;
  } while (t > 1);
  const int gamma = i + sp * d + min(d, 0);
  const int first = min(i, j), last = max(i, j);
  c.rfirst[e] = first;
  c.rlast[e] = last;
  c.dnode[e] = dn;
  if (first == gamma)  // the left child is a leaf (key gamma) or internal node gamma
    c.parentL[base + gamma] = e;
  else
    c.parentI[base + gamma] = e;
  if (last == gamma + 1)  // the right child: leaf or internal node gamma + 1
    c.parentL[base + gamma + 1] = e;
  else
    c.parentI[base + gamma + 1] = e;
  if (i == 0) c.parentI[e] = -1;
}

__device__ __forceinline__ int oct_depth(int dn, int levels) { return min(dn / 3, levels); }

// Octant digit at depth k (1-based) of a left-aligned key.
__device__ __forceinline__ int octant_at(unsigned long long key, int k)
{
  return (int)(key >> (64 - 3 * k)) & 7;
}

// An internal node is an octree cell when its octal depth exceeds its
// parent's (the root always is).  Records the depth bits per first key.
__device__ __forceinline__ void cells_elem(const Ctx &c, int base, int n, int e, int levels)
{
  if (e - base >= n - 1) {
    c.iscell[e] = 0;
    return;
  }
  const int od = oct_depth(c.dnode[e], levels);
  const int p = c.parentI[e];
  const int odp = p < 0 ? -1 : oct_depth(c.dnode[p], levels);
  const int cell = od > odp;
  c.iscell[e] = cell;
  if (cell) atomicOr(&c.mask[base + c.rfirst[e]], 1ull << od);
}

// Walk record meta of a cell with side^2 = l2 (float, as the reference
// computes len*len): the squared distances below which the cell surely opens
// and above which it surely does not, l2/theta^2 (1 -+ 1e-5); in between the
// walk takes the reference's decision in double, so these need be no better
// than a small part of 1e-5 and are formed in float.  Particles (never opened)
// get -1 for both.
__device__ __forceinline__ int4 cell_meta(float l2, int skip, const DevParams &P)
{
  const float q = __fdiv_rn(l2, P.theta2);
  return make_int4(__float_as_int(l2), skip, __float_as_int(q * (1.f - 1e-5f)),
                   __float_as_int(q * (1.f + 1e-5f)));
}

// Side of a cell at octal depth od, as float: the root's side halved od times
// in double.  Every cell's depth is at most the subhalo's depth of geometric
// subdivision, so each halving applies; it is exact, and taken on the
// exponent (double arithmetic runs at 1/64 of the FP32 rate on this GPU).
__device__ __forceinline__ float cell_side(double len, int od)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(len);
  const int ex = (int)(b >> 52);
  if (ex - od > 1023 - 120 && ex < 0x7ff)
    return d2f(__longlong_as_double((long long)(b - ((unsigned long long)od << 52))));
  for (int k = 0; k < od; k++) len = dmul(len, 0.5);
  return __double2float_rn(len);
}

__device__ __forceinline__ int4 particle_meta(int skip)
{
  return make_int4(0, skip, __float_as_int(-1.f), __float_as_int(-1.f));
}

__device__ __forceinline__ float4 make_rel(float4 a, const float fc[3], const DevParams &P)
{
  return make_float4(rel_coord(a.x, fc[0], P), rel_coord(a.y, fc[1], P), rel_coord(a.z, fc[2], P),
                     a.w);
}

// Particle leaf j of a subhalo's tree (element e = base + j): preorder index
// j + #cells starting at or before key j; a0 is its particle {x, y, z, m}
// (mass not yet scaled by the sampling factor).  Xs[0..n]: the exclusive scan
// of the cells starting at each of the subhalo's keys (any common offset).
// The subhalo of one particle gets a root cell of side 0 holding it
// (tpp:56-102 with one particle).
__device__ __forceinline__ void leaves_elem(const Ctx &c, SegState &sg, int base, int n, int e,
                                            float4 a0, unsigned long long key,
                                            const long long *Xs)
{
  const int j = e - base;
  const int nb = 2 * base;
  const float4 a = make_float4(a0.x, a0.y, a0.z, fmul(a0.w, sg.mfac));
  if (n == 1) {
    const float4 r = make_rel(a, sg.fc, c.P);
    c.nd_abs[nb] = a;
    c.nd[nb].p = make_float4(r.x, r.y, r.z, -r.w);  // the sign bit marks a cell
    c.nd[nb].m = cell_meta(fmul((float)sg.len, (float)sg.len), kDone, c.P);
    c.nd_abs[nb + 1] = a;
    c.nd[nb + 1].p = r;
    c.nd[nb + 1].m = particle_meta(kDone);
    sg.nnodes = 2;
    return;
  }
  const long long xb = Xs[0];
  const int idx = j + (int)(Xs[j + 1] - xb);
  const int nnodes = n + (int)(Xs[n] - xb);
  c.nd_abs[nb + idx] = a;
  c.nd[nb + idx].p = make_rel(a, sg.fc, c.P);
  c.nd[nb + idx].m = particle_meta(idx + 1 < nnodes ? nb + idx + 1 : kDone);
  if (j == 0) sg.nnodes = nnodes;
  // the octant slot in the lowest cell holding this particle (none in a bucket)
  int p = c.parentL[e];
  for (int guard = 0; p >= 0 && !c.iscell[p] && guard < 256; guard++) p = c.parentI[p];
  if (p >= 0 && c.iscell[p]) {
    const int odp = oct_depth(c.dnode[p], sg.levels);
    if (odp < sg.levels) c.cslot[first_slot(p) + octant_at(key, odp + 1)] = nb + idx;
  }
}

// Cell e (an internal node with iscell[e] set): preorder index, skip pointer,
// side (len*len in float), octal depth, and a count of child cells on the
// parent.  keys: the subhalo's sorted keys, element-indexed from `base`; Xs
// as for leaves_elem.
__device__ __forceinline__ void cellnodes_elem(const Ctx &c, const SegState &sg, int base, int n,
                                               int e, const unsigned long long *keys,
                                               const long long *Xs)
{
  const int nb = 2 * base;
  const int od = oct_depth(c.dnode[e], sg.levels);
  const int lo = c.rfirst[e], hi = c.rlast[e];
  const unsigned long long m = c.mask[base + lo];
  const int rank = __popcll(m & ((1ull << od) - 1ull));
  const long long xb = Xs[0];
  const int idx = lo + (int)(Xs[lo] - xb) + rank;
  const int skip = hi + 1 + (int)(Xs[hi + 1] - xb);
  const float lf = cell_side(sg.len, od);
  c.nd[nb + idx].m = cell_meta(fmul(lf, lf), hi + 1 < n ? nb + skip : kDone, c.P);
  c.cidx[e] = nb + idx;
  c.cskip[e] = nb + skip;
  c.cdepth[e] = od;
  int p = c.parentI[e];
  for (int guard = 0; p >= 0 && !c.iscell[p] && guard < 256; guard++) p = c.parentI[p];
  if (p >= 0 && !c.iscell[p]) p = -1;  // malformed tree: never climb past it
  c.pcell[e] = p;
  if (p >= 0) {
    atomicAdd(&c.pending[p], 1);
    const int odp = oct_depth(c.dnode[p], sg.levels);
    c.cslot[first_slot(p) + octant_at(keys[lo], odp + 1)] = nb + idx;
  }
}

// 1/m for the quotients below, m > 0: the float reciprocal approximation,
// refined by one Newton-Raphson step r <- r + r (1 - m r) in double, which
// squares its relative error (at most 2^-22.4, with the rounding of m to float)
// to below 2^-44.  ok: m lies in the range where none of this can overflow or
// lose bits to subnormals (else r is not used).
__device__ __forceinline__ double recip_refined(double m, bool &ok)
{
  const float mf = d2f(m);
  const unsigned ex = __float_as_uint(mf) >> 23;  // the sign bit too: a negative m is not ok
  ok = ex - (127u - 100u) <= 200u;
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(mf));
  const double r = f2d(r0);
  return __fma_rn(r, __fma_rn(-m, r, 1.0), r);
}

// float(c / m) with the quotient first rounded to double, as the reference
// rounds its double centre of mass to float, given r ~ 1/m (ok as above).
// q = c * r is within 2^-44 of c / m, at most 512 of its units in the last
// place, so both round to the same float unless q lies that close to a
// point M halfway between two floats (its low 29 mantissa bits near 2^28).
// There (always, for instance, at the midpoint of two equal masses) the side
// of M follows from rho = c - M m, one fused multiply-add: its sign and a zero
// are exact.  c / m = M: a tie, to even.  |rho| at least 4 times the half
// unit of M times m: the double quotient lies on rho's side of M.  In between,
// and outside the range of normal floats, the exact division.  A cell of two
// equal masses takes 12 to 15 double operations in all, where the
// division's own (per axis, for the whole warp when one lane needs it)
// more than doubled that: double runs at 1/64 of the FP32 rate on this GPU.
static __device__ __noinline__ float quot_float_divided(double c, double m)
{
  return d2f(ddiv(c, m));
}

__device__ __forceinline__ float quot_float(double c, double m, double r, bool ok)
{
  const double q = dmul(c, r);
  const unsigned long long b = (unsigned long long)__double_as_longlong(q);
  const int ex = (int)((b >> 52) & 0x7ffull);
  const unsigned rem = (unsigned)(b & 0x1fffffffull);
  if (ok && ex >= 1023 - 125 && ex <= 1023 + 126) {
    if (rem - (0x10000000u - 512u) > 1024u) return d2f(q);
    const unsigned long long mid = (b & ~0x1fffffffull) | 0x10000000ull;
    const unsigned long long rho = (unsigned long long)__double_as_longlong(
        __fma_rn(-__longlong_as_double((long long)mid), m, c));
    // 4 * (half a unit of M) * m, by its exponent: 2^(ex - 1023 - 53 + 2) m
    const unsigned long long far = (unsigned long long)__double_as_longlong(m) +
                                   ((unsigned long long)(long long)(ex - 1023 - 51) << 52);
    const unsigned long long arho = rho & 0x7fffffffffffffffull;
    if (arho == 0ull || arho >= far) {
      const unsigned long long down = (mid & 0x7fffffffffffffffull) >> 29;  // towards zero
      const bool up = arho == 0ull ? (down & 1ull) != 0ull : (rho >> 63) == (mid >> 63);
      const unsigned bits =
          (unsigned)(down - ((unsigned long long)(1023 - 127) << 23)) + (up ? 1u : 0u);
      return __uint_as_float(bits | ((unsigned)(mid >> 63) << 31));
    }
  }
  return quot_float_divided(c, m);
}

// Bottom-up moments of one cell: mass and centre of mass over its children in
// octant order, in double, rounded to float as the reference does.  The
// children come from the cell's eight octant slots; the children of a bucket
// cell (particles sharing the whole key, depth == levels) hold the slots that
// follow it, in preorder, so they are read one after another.  src(k) gives
// the moment {x, y, z, m} of node slot k (global memory, or a block's copy).
// A product of two floats is exact in double, so one fused multiply-add
// rounds exactly as the reference's multiply-then-add.
// The same with the cell's octant slots s0, s1 (cslot) already loaded;
// bucket: the cell is a bucket (depth == levels).
template <class Src>
__device__ __forceinline__ float4 cell_moment_slots(bool bucket, int idx, int end, int4 s0,
                                                    int4 s1, Src src)
{
  double m = 0., cx = 0., cy = 0., cz = 0.;
  auto add = [&](float4 a) {
    const double w = f2d(a.w);
    m = dadd(m, w);
    cx = __fma_rn(f2d(a.x), w, cx);
    cy = __fma_rn(f2d(a.y), w, cy);
    cz = __fma_rn(f2d(a.z), w, cz);
  };
  if (!bucket) {
    // the occupied octants in ascending order; a warp then issues as many
    // (double) additions as its lanes' largest number of children, not eight.
    // Two at a time, so that both moments are on their way before the first
    // is added.
    const int sl[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    unsigned occ = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) occ |= (sl[j] > idx && sl[j] < end ? 1u : 0u) << j;
    auto take = [&]() {
      const int j = __ffs(occ) - 1;
      occ &= occ - 1;
      const int4 h = j < 4 ? s0 : s1;
      const int q = j & 3;
      return q == 0 ? h.x : (q == 1 ? h.y : (q == 2 ? h.z : h.w));
    };
    while (occ) {
      const int k0 = take();
      const int k1 = occ ? take() : -1;
      const float4 a0 = src(k0), a1 = src(k1 >= 0 ? k1 : k0);
      add(a0);
      if (k1 >= 0) add(a1);
    }
  } else {
#pragma unroll 4
    for (int k = idx + 1; k < end; k++) add(src(k));
  }
  bool ok;
  const double r = recip_refined(m, ok);
  return make_float4(quot_float(cx, m, r, ok), quot_float(cy, m, r, ok), quot_float(cz, m, r, ok),
                     d2f(m));
}

template <bool kCG, class Src>
__device__ __forceinline__ float4 cell_moment_of(const Ctx &c, const SegState &sg, int e,
                                                 int depth, int idx, int end, Src src)
{
  int4 s0 = make_int4(-1, -1, -1, -1), s1 = s0;
  const bool bucket = depth >= sg.levels;
  if (!bucket) {
    const int4 *slot = reinterpret_cast<const int4 *>(c.cslot + first_slot(e));
    s0 = kCG ? __ldcg(slot) : slot[0];
    s1 = kCG ? __ldcg(slot + 1) : slot[1];
  }
  return cell_moment_slots(bucket, idx, end, s0, s1, src);
}

// The walk record's position and mass of a cell from its moment (fc: the
// subhalo's frame centre).
__device__ __forceinline__ void store_cell_rel(const Ctx &c, const float fc[3], int idx, float4 r)
{
  float4 rel = make_rel(r, fc, c.P);
  rel.w = -rel.w;  // the sign bit marks a cell for the walks
  c.nd[idx].p = rel;
}

// cell_moment_of over the moments in global memory (kCG: through L2, for
// callers whose children were written by other blocks during the same
// launch); stores the cell's moment and record.
template <bool kCG>
__device__ __forceinline__ void cell_moment(const Ctx &c, const SegState &sg, int e, int depth)
{
  const int idx = c.cidx[e], end = c.cskip[e];
  const float4 r = cell_moment_of<kCG>(c, sg, e, depth, idx, end, [&](int k) {
    return kCG ? __ldcg(&c.nd_abs[k]) : c.nd_abs[k];
  });
  if (kCG)
    __stcg(&c.nd_abs[idx], r);
  else
    c.nd_abs[idx] = r;
  store_cell_rel(c, sg.fc, idx, r);
}

}  // namespace hbtu
