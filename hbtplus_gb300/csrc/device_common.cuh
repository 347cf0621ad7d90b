// device_common.cuh -- device helpers and the per-call context.
//
// Arithmetic that decides the bound set follows the reference's float
// (HBTReal) / double split operation by operation.  nvcc contracts a*b+c into
// FMA by default, which rounds differently from the reference's separate
// multiply and add, so every such operation is spelled with an explicit
// round-to-nearest intrinsic (__fmul_rn, __dadd_rn, ...).
#pragma once
#include "hbtu_internal.h"

namespace hbtu {

constexpr int kChunk = 1024;  // elements per reduction chunk
// Chunks from which on a subhalo's chunk sums are added by k_fold_chunks: with fewer,
// the loop of sum_chunks (145 cycles a chunk) costs less than one more launch.
constexpr int kLongSum = 64;
constexpr int kDone = 0x7fffffff;

// One tree node as the walks read it (32 bytes, one sector): p = {x, y, z,
// mass} relative to the frame centre (sign bit of the mass set on cells),
// m = {len*len bits with the all-particle-children flag in the sign bit, skip
// pointer, sure-open and sure-accept squared distances as float bits}.
struct __align__(32) WNode {
  float4 p;
  int4 m;
};

// Both halves of node i in one 256-bit load.
__device__ __forceinline__ void load_node(const WNode *nd, int i, float4 &p, int4 &m)
{
  asm("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w), "=r"(m.x), "=r"(m.y), "=r"(m.z), "=r"(m.w)
      : "l"(nd + i));
}

__device__ __forceinline__ void load_node(const WNode *nd, int i, float4 &p, int2 &m)
{
  int4 q;
  load_node(nd, i, p, q);
  m = make_int2(q.x, q.y);
}

// First octant slot of the cell of element e (Ctx::cslot) and first coordinate of particle
// i in an array of triples: a call holds up to 2^30 of them, and an int's product
// overflows from 2^28 and 2^31 / 3 on.
__host__ __device__ inline size_t first_slot(int e) { return 8 * (size_t)e; }
__host__ __device__ inline size_t first_coord(int i) { return 3 * (size_t)i; }

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// Exact float -> double and round-to-nearest-even double -> float, built
// from the IEEE-754 fields with integer operations: the conversion
// instructions run on the FP64 unit, at 1/64 of the FP32 rate on this GPU.
// The special cases are integer code too; the results are the instructions', bit for
// bit (f2d leaves it to the next operation to quiet a signalling NaN).  A double
// instruction behind a condition is no way out: the compiler predicates short
// branches, and a predicated-off double instruction holds the FP64 unit as long as
// an executed one (measured: 20 of them per step in a walk took it from 1.5 to 25 ms).
// Rare double paths in this library are calls for the same reason.
__device__ __forceinline__ double f2d(float x)
{
  unsigned u = __float_as_uint(x);
  unsigned bias = 1023 - 127;
  const unsigned sign = u & 0x80000000u;
  const unsigned e = (u >> 23) & 0xffu;
  if (e == 0u) {  // zero or subnormal: 2^64 x is exact
    u = __float_as_uint(__fmul_rn(x, 0x1p64f));
    bias = (u & 0x7fffffffu) ? bias - 64 : 0;
  }
  if (e == 0xffu) bias = 0x7ff - 0xff;
  const unsigned hi = sign | ((((u >> 23) & 0xffu) + bias) << 20) | ((u & 0x7fffffu) >> 3);
  return __hiloint2double((int)hi, (int)(u << 29));
}

__device__ __forceinline__ float d2f(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ffull) - 1023 + 127;
  const unsigned long long mant = b & 0xfffffffffffffull;
  // round half to even; a carry bumps the exponent
  unsigned bits = ((unsigned)e << 23) + (unsigned)(mant >> 29) +
                  ((b & 0x1fffffffull) + ((mant >> 29) & 1ull) > (1ull << 28) ? 1u : 0u);
  if (e <= 0) {  // a subnormal result, or zero
    const int s = min(30 - e, 63);
    const unsigned long long m = mant | (1ull << 52);
    const unsigned long long q = m >> s, rem = m & ((1ull << s) - 1ull), half = 1ull << (s - 1);
    bits = s > 53 ? 0u : (unsigned)q + (rem + (q & 1ull) > half ? 1u : 0u);
  } else if (e >= 255 || bits >= 0x7f800000u) {  // overflow, infinity or NaN (quiet, payload kept)
    bits = e == 0x7ff - 1023 + 127 && mant ? 0x7fc00000u | (unsigned)(mant >> 29) : 0x7f800000u;
  }
  return __uint_as_float(bits | ((unsigned)(b >> 63) << 31));
}

// x / 2, on the exponent where that is exact.
__device__ __forceinline__ double half_of(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned ex = (unsigned)(b >> 52) & 0x7ffu;
  if (ex - 2u < 0x7ffu - 2u) return __longlong_as_double((long long)(b - (1ull << 52)));
  return dmul(0.5, x);
}

// NEAREST (src/config_parser.h:142) on a double / a float operand.
__device__ __forceinline__ double nearest_d(double x, const DevParams &P)
{
  return x > (double)P.boxhalf ? dsub(x, (double)P.box)
                               : (x < -(double)P.boxhalf ? dadd(x, (double)P.box) : x);
}
__device__ __forceinline__ float nearest_f(float x, const DevParams &P)
{
  return x > P.boxhalf ? fsub(x, P.box) : (x < -P.boxhalf ? fadd(x, P.box) : x);
}

// Snapshot_t::RelativeVelocity (src/snapshot.h:100-111), float arithmetic.
__device__ __forceinline__ void relvel(const float tp[3], const float tv[3], const float rp[3],
                                       const float rv[3], float dv[3], const DevParams &P)
{
  const float ha = fmul(P.Hz, P.a);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    float dx = fsub(tp[j], rp[j]);
    if (P.periodic) dx = nearest_f(dx, P);
    dv[j] = fadd(fsub(tv[j], rv[j]), fmul(ha, dx));
  }
}

// VecNorm / VecDot (src/mymath.h:20-21) in float.
__device__ __forceinline__ float vdot(const float a[3], const float b[3])
{
  return fadd(fadd(fmul(a[0], b[0]), fmul(a[1], b[1])), fmul(a[2], b[2]));
}

// Relative coordinate of an absolute float coordinate: wrapped once in
// double, then rounded to float.  When the float difference s = x - c is
// exact (a float TwoSum with a zero error term) it equals the double one, and
// for |s| < box the wrap s -+ box is exact in float as in double (Sterbenz:
// box/2 < |s| < 2 box), so the float arithmetic gives the same bits without
// the FP64 pipe (1/64 of the FP32 rate on this GPU); otherwise the double path.
static __device__ __noinline__ float rel_coord_double(float x, float c, int periodic, float box,
                                                      float boxhalf)
{
  double d = dsub(f2d(x), f2d(c));
  if (periodic) d = d > f2d(boxhalf) ? dsub(d, f2d(box)) : d < -f2d(boxhalf) ? dadd(d, f2d(box)) : d;
  return d2f(d);
}

__device__ __forceinline__ float rel_coord(float x, float c, const DevParams &P)
{
  const float s = __fsub_rn(x, c);
  const float bb = __fsub_rn(s, x);
  const float err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(-c, bb));
  if (err == 0.f && !P.periodic) return s;
  if (err == 0.f && fabsf(s) < P.box) return nearest_f(s, P);
  return rel_coord_double(x, c, P.periodic, P.box, P.boxhalf);
}

// Order-preserving 32-bit key of a float (ascending); -0 sorts as +0.
__device__ __forceinline__ unsigned float_key(float e)
{
  unsigned u = __float_as_uint(e == 0.f ? 0.f : e);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k)
{
  return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k);
}
// A subhalo's bounding box before any particle: keys above / below every float's.
constexpr unsigned kBoxLow = 0xffffffffu, kBoxHigh = 0u;

__device__ __forceinline__ int upper_bound_i(const int *a, int n, int x)
{
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] <= x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// The per-call device context: every buffer of the workspace.
struct Ctx {
  DevParams P;
  int N, S;
  cudaStream_t st;
  // particles
  float4 *pm, *vel;
  long long *id;
  int *type, *pseg;
  int *epid, *epid2;
  float *eE, *eE2, *eR;
  int *epos_of_pid, *coh_pid;
  // per segment
  SegState *seg;
  PassPlan *plan, *plan_host;
  int *tree_base, *tgt_base;                 // S+1 each
  int *tchunk_base, *bchunk_base, *ub_base;  // S+1 each
  int4 *plan_cnt, *plan_cnt2;                // S each: gathered plan counters
  long long *plan_inter;                     // S: gathered interaction counts
  int *seg_off;                              // S+1
  int *seg_order;                            // S: subhaloes by size, largest first
  int opt_leaf_runs;                         // warp schedule streams all-particle cells
  int opt_schedule;                          // FP32 walk: 0 one walk per lane, 1 warp schedule
  int *part_info;                            // 8 ints per segment
  unsigned *seg_bbox;                        // 6 per segment: float_key of the box's low and high corners
  double *chunk_sums;                        // 16 per chunk
  // sort
  SortBuffers sb;
  // tree construction
  int *parentI, *parentL, *rfirst, *rlast, *dnode;
  int *iscell, *cidx, *cskip, *cdepth, *pcell, *pending, *pending0;  // pending: child cells
  int *cslot;  // 8 per cell: node index of the child in each octant, -1 if none
  // moment work lists: cell_list holds the large chunk roots from the front and
  // the top cells from the back, chunk_list the small chunk roots; lvl[0..3]:
  // their counts (large, top), the job counter, the small count
  int *cell_list, *chunk_list, *lvl;
  unsigned long long *mask;
  long long *X;
  // nodes (2 per tree particle)
  float4 *nd_abs;
  WNode *nd;
  // the FP32 walk's layout: the same records with each cell's children in
  // consecutive slots (m.w = first child's slot instead of the upper
  // threshold); null when the workspace has no room for it
  WNode *nd2;
  int *newidx;
  long long *X2;
  void *scan_tmp2;
  int opt_layout;  // 1: the FP32 lane walk uses nd2
  // partition
  long long *pcode, *pX;
  int *Pk, *Qk;
  void *scan_tmp;
  double *pot_out;  // optional: potentials of a full pass (hbtu_binding_energies)
  // adjoint outputs (hbtu_energy_gradient), by input position; grads may be null
  float *grad_pos, *grad_vel, *grad_mass;
  double *e_part;
  // the per-subhalo loop (small.cu): it takes over once every active
  // subhalo's list holds at most small_cap particles (0: never)
  int *small_next;   // three work queues (large, medium, short lists): next jobs, counts, threads
  int *small_list;   // 3 S: their jobs, S each
  int small_cap;
  int nlong;  // subhaloes whose chunk sums k_fold_chunks adds, the first of seg_order
};

// launchers (tree.cu)
void launch_bbox_cube(Ctx &c, int max_chunks);
void launch_tree_build(Ctx &c, const PassPlan &pl);
// launchers (walk.cu)
void launch_walk(Ctx &c, const PassPlan &pl);
// sorts the targets that come in list order, before the tree build
void launch_list_order(Ctx &c, const PassPlan &pl);
void launch_sibling_layout(Ctx &c, const PassPlan &pl);
// The FP32 walk's warp schedule sums a target's terms in parts that depend on the warp's other
// targets: its passes take them as they come, without the orders below.
__host__ __device__ inline bool warp_schedule(const Ctx &c)
{
  return c.opt_schedule == 1 && c.P.precision != HBTU_PRECISION_FP64;
}
// Targets in list order are sorted along a space-filling curve (launch_list_order)
// when a pass has at least kListMin of them: the sort's dozen launches take longer
// than they save below (one subhalo of 7.2e4 particles, 1000 in the tree: the call
// takes 1.20 ms without, 1.23 with; 2.4e5: 1.78 and 1.48), and when they are half of
// the call's particles, all of which the sort moves.
constexpr int kListMin = 1 << 17;
inline bool list_order(const Ctx &c, const PassPlan &pl)
{
  return pl.nlist >= kListMin && pl.nlist >= c.N / 2 && !warp_schedule(c);
}
// The FP32 lane walk of two neighbouring targets per lane (walk_pair): from
// kPairMin targets on, 5 warps of pairs per scheduler.  Fewer lanes than that leave
// the chip waiting on each walk's chain of loads (first pass of a subhalo of 1.1e5
// particles: 937 us in pairs, 623 one by one; 1.6e5: 1014 and 967; 2.2e5: 1174 and
// 1228; 3.4e5: 1607 and 2278; 1.1e6: 4.5 and 5.5 ms; 2.7e7: 122 and 160 ms).
// Targets in list order are no neighbours: 780,000 of them took 810 us against 765,
// sorted 607 against 637.  A pass that has some of them, unsorted, takes one target per
// lane; where they are the fewer this is the slower side (704,198 targets, 41% of them in
// list order: first walk 2.1 ms, in pairs 1.77; from 50% on they are sorted).
// The gradient's walk stays with one target per lane.
constexpr int kPairMin = 152 * 4 * 5 * 64;
inline bool pair_walk(const Ctx &c, const PassPlan &pl)
{
  return c.P.precision != HBTU_PRECISION_FP64 && c.opt_schedule == 0 &&
         (pl.nlist == 0 || list_order(c, pl)) &&
         pl.ntgt_total >= kPairMin && !(c.grad_pos || c.grad_vel || c.grad_mass);
}
// The FP32 lane walk over the sibling-block records (the tree build then makes
// them): for trees of at least kSiblingMinTree particles in all, where the
// faster walk pays for the extra pass over the nodes (the small trees of
// correction passes do not), unless walk_pair takes the pass.
constexpr int kSiblingMinTree = 1 << 16;
inline bool sibling_walk(const Ctx &c, const PassPlan &pl)
{
  return c.P.precision != HBTU_PRECISION_FP64 && c.opt_schedule == 0 && c.opt_layout && c.nd2 &&
         pl.ntree_total >= kSiblingMinTree && !pair_walk(c, pl);
}
void launch_grad_walk(Ctx &c, const PassPlan &pl);
// per-subhalo sums of a per-particle double array (input positions), deterministic
void launch_segment_sums(Ctx &c, const double *x, double *out);
// (direct.cu) exact FP64 potentials of particles tidx[0..nt) from all n particles
void direct_potential_fp64(const DevParams &P, const float4 *pm, int n, const int *tidx, int nt,
                           double *out, double *partial, int nsplit, cudaStream_t st);
// (small.cu) the remaining passes of every active subhalo, one block or warp
// per subhalo; `cap` bounds their energy lists (at most kSmallCap particles)
constexpr int kSmallCap = 2048;
constexpr int kSmallDefault = 2048;
void launch_small(Ctx &c, int cap, int nactive, int max_passes);
// A whole call whose subhaloes all hold at most kSmallCap particles, in the
// same kernel: set-up, every pass and the results.
struct SmallCall {
  const float *pos, *vel, *mass;
  const hbtu_state *st;    // per subhalo
  const long long *off;    // S + 1
  const int *order;        // subhaloes by size, largest first
  int jobs[3];             // lists of each size class (small_classes)
  int64_t *order_out;
  float *energy_out;
  hbtu_result *res;
};
constexpr int kSmallWarpCap = 128;    // lists up to this long: one warp each
constexpr int kSmallMediumCap = 512;  // lists up to this long: four warps, longer ones a block
// The lists of each size class and the threads of its groups.
void small_classes(const int64_t *offsets, const int *order, int S, int (&n)[3], int (&T)[3]);
void launch_small_call(Ctx &c, const SmallCall &io, int cap, int max_passes);
// launchers (loop.cu)
void launch_init(Ctx &c, const float *pos, const float *vel, const float *mass,
                 const long long *id);
void launch_plan(Ctx &c, int mode);  // 0 pass, 1 bound chunks, 2 final
void launch_partition(Ctx &c);
void launch_averages_control(Ctx &c, int max_passes);
// which: 0 unbound blocks, 1 bound parts, 2 refined prefixes (keyed by eR)
void launch_block_sort(Ctx &c, int total, int which);
void launch_refine_mode(Ctx &c, int enter);
void launch_finalize(Ctx &c, int64_t *order_out, float *energy_out, hbtu_result *res_dev);

}  // namespace hbtu
