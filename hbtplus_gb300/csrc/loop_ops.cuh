// loop_ops.cuh -- steps of the unbinding loop shared by the batch kernels
// (loop.cu) and the per-subhalo loop (small.cu):
//   block_sum        deterministic FP64 sums of a 1024-element chunk by a block
//                    of kLB threads (fixed association, so both callers round
//                    alike);
//   control_segment  one subhalo's decisions after a pass: disruption
//                    (src/subhalo_unbind.cpp:361-379), the sticky correction
//                    flag (:383-392), the frame (AverageVelocity /
//                    AveragePosition from the chunk sums, :108-188),
//                    convergence on the particle count (:395) and the set-up
//                    of the next full (:331-356) or correction (:312-330)
//                    pass.
#pragma once
#include "device_common.cuh"

namespace hbtu {

constexpr int kLB = 256;  // threads of a chunk-sum block
constexpr int kSums = 24;  // doubles per reduction chunk

// One step of a warp reduce-scatter of N doubles: the lanes of each pair
// (lane, lane ^ o) add the same two values as an xor butterfly would, but
// each keeps only half of them (the lane with bit o set keeps the upper
// half, indices h .. N-1 with h = ceil(N/2), padded by one zero when N is
// odd).  Five steps (o = 16 .. 1) leave each sum in one lane, bit-identical
// to the butterfly's result (same pairs, same order of association).
template <int N>
__device__ __forceinline__ void rs_step(const double (&cur)[N], double (&nxt)[(N + 1) / 2], int o,
                                        bool upper)
{
  constexpr int h = (N + 1) / 2;
#pragma unroll
  for (int j = 0; j < h; j++) {
    const double lo = cur[j], hi = (j + h < N) ? cur[j + h] : 0.;
    const double recv = __shfl_xor_sync(0xffffffffu, upper ? lo : hi, o);
    nxt[j] = (upper ? hi : lo) + recv;
  }
}

// A warp's sums of K values by that reduce-scatter: returns the index of the sum
// this lane then holds in *sum, or -1.
template <int K>
__device__ __forceinline__ int warp_sums(const double (&v)[K], double *sum)
{
  static_assert(K >= 1 && K <= 32, "one sum per lane at most");
  const int lane = threadIdx.x & 31;
  constexpr int n1 = (K + 1) / 2, n2 = (n1 + 1) / 2, n3 = (n2 + 1) / 2, n4 = (n3 + 1) / 2,
                n5 = (n4 + 1) / 2;
  double a1[n1], a2[n2], a3[n3], a4[n4], a5[n5];
  rs_step<K>(v, a1, 16, lane & 16);
  rs_step<n1>(a1, a2, 8, lane & 8);
  rs_step<n2>(a2, a3, 4, lane & 4);
  rs_step<n3>(a3, a4, 2, lane & 2);
  rs_step<n4>(a4, a5, 1, lane & 1);
  // the index of the sum this lane holds: the split follows the padded
  // sizes N; n counts the lane's real (unpadded) values
  int base = 0, n = K, N = K;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int h = (N + 1) / 2;
    if (lane & o) {
      base += h;
      n = max(0, n - h);
    } else {
      n = min(n, h);
    }
    N = h;
  }
  *sum = a5[0];
  return n >= 1 ? base : -1;
}

// Sums of K values over a block of kLB threads into out[0 .. K).  The
// chunk's elements p = threadIdx.x + j*kLB (0 <= p < nvalid) are spread over
// the warps in order, so a warp with 32*w >= nvalid holds only zeros and
// writes them without reducing (small subhaloes leave most warps empty).
template <int K>
__device__ void block_sum(double (&v)[K], double *out, int nvalid)
{
  __shared__ double sh[K][kLB / 32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (32 * w < nvalid) {
    double sum;
    const int k = warp_sums<K>(v, &sum);
    if (k >= 0) sh[k][w] = sum;
  } else if (lane < K) {
    sh[lane][w] = 0.;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0.;
    for (int j = 0; j < kLB / 32; j++) t += sh[threadIdx.x][j];
    out[threadIdx.x] = t;
  }
}

// x[0] + x[kSums] + x[2 kSums] + .. (n terms), rounded after each addition as a loop
// of double additions from zero rounds: the order fixes the result.  Such a loop takes
// about 145 cycles a term on this GPU (2.7e7 particles, 26,657 chunks: 1.9 ms).  By a
// warp, 32 terms at a time, in integers: while the sum stays within one binade it is a
// whole number of its last places, and adding a term adds floor(x), plus one if the
// term's fraction rounds up: a prefix sum over the lanes.  A fraction of exactly one
// half rounds the sum to even, so the parity after it is zero, and the parity before
// the next such term is that of what came in between.  32 terms among which the sum
// leaves the binade, or whose terms are larger than the sum, or not finite, are added
// by the loop.  7 sums of 26,657 chunks: 1.9 ms -> 0.47 ms; 18: 1.9 -> 1.26; one of 977:
// 143 -> 26 us.
__device__ __forceinline__ double sum_in_order(const double *x, int n, int lane)
{
  constexpr unsigned kFull = 0xffffffffu;
  constexpr long long kHidden = 1ll << 52;
  double t = 0.;
  double next = lane < n ? x[(size_t)lane * kSums] : 0.;
  for (int g = 0; g < n; g += 32) {
    const double v = next;
    next = g + 32 + lane < n ? x[(size_t)(g + 32 + lane) * kSums] : 0.;
    const long long tb = __double_as_longlong(t), vb = __double_as_longlong(v);
    const int te = (int)(tb >> 52) & 0x7ff, ve = (int)(vb >> 52) & 0x7ff;
    long long sum = (tb & (kHidden - 1)) | kHidden;
    sum = tb < 0 ? -sum : sum;
    long long q = (vb & (kHidden - 1)) | (ve ? kHidden : 0ll);
    q = vb < 0 ? -q : q;
    const int d = te - max(ve, 1);
    bool ok = te > 64 && te < 2046 && d >= 0;
    const int sh = min(max(d, 0), 62);  // beyond: floor -1 or 0 and the same rounding
    const unsigned long long unit = 1ull << sh;
    const unsigned long long frac2 = ((unsigned long long)q & (unit - 1ull)) << 1;
    q >>= sh;
    const bool tie = frac2 == unit;
    int up = frac2 > unit;
    const unsigned ties = __ballot_sync(kFull, tie);
    const unsigned odd = __ballot_sync(kFull, !tie && ((q + up) & 1));
    if (tie) {
      const unsigned below = (1u << lane) - 1u, prev = ties & below;
      const int first = prev ? 32 - __clz(prev) : 0;  // the lane after the last tie
      const int parity = __popc(odd & below & ~((1u << first) - 1u)) + (prev ? 0 : (int)(sum & 1));
      up = (parity + (int)(q & 1)) & 1;
    }
    const long long inc = q + up;
    long long pre = inc;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(kFull, pre, o);
      if (lane >= o) pre += y;
    }
    const long long at = sum + pre - up;  // floor of the exact sum after this term
    ok = ok && ((at ^ (at >> 63)) >> 52) == 1;
    if (__all_sync(kFull, ok)) {
      sum += __shfl_sync(kFull, pre, 31);
      const long long mag = sum < 0 ? -sum : sum;
      t = __longlong_as_double((((long long)te << 52) + (mag - kHidden)) |
                               (sum < 0 ? (long long)(1ull << 63) : 0ll));
    } else {
      const int m = min(32, n - g);
      for (int i = 0; i < m; i++) t += __shfl_sync(kFull, v, i);
    }
  }
  return t;
}

// The first K sums of the subhaloes of at least kLongSum chunks (of the nlong largest),
// to their first chunk's place: warp w takes one of them.
__device__ __forceinline__ void fold_chunks(const Ctx &c, int K, int w, int lane)
{
  if (w >= c.nlong * K) return;
  const int s = c.seg_order[w / K];
  const int b0 = c.bchunk_base[s], n = c.bchunk_base[s + 1] - b0;
  if (n < kLongSum) return;
  double *x = c.chunk_sums + (size_t)b0 * kSums + w % K;
  const double t = sum_in_order(x, n, lane);
  if (lane == 0) x[0] = t;
}

// NEAREST(x - o) * m in double (AveragePosition's term, src/subhalo_unbind.cpp:
// 139-188), bit for bit, mostly without double arithmetic.  When the float
// difference s = x - o is exact (a float TwoSum with a zero error term) and
// |s| < box, the wrap s -+ box is exact in float too (Sterbenz: box/2 < |s| <
// 2 box), and the product of the two floats is exact as a float product plus
// its fma remainder, added exactly in double: one FP64 add instead of the
// double subtract, wrap and multiply (FP64 runs at 1/64 of the FP32 rate on
// this GPU).  Otherwise the double path.
static __device__ __noinline__ double rel_times_mass_double(float x, double od, double md,
                                                            float box, float boxhalf)
{
  const double d = dsub(f2d(x), od);
  return dmul(d > f2d(boxhalf) ? dsub(d, f2d(box)) : d < -f2d(boxhalf) ? dadd(d, f2d(box)) : d, md);
}

__device__ __forceinline__ double rel_times_mass(float x, float o, double od, float m, double md,
                                                 const DevParams &P)
{
  const float s = __fsub_rn(x, o);
  const float bb = __fsub_rn(s, x);
  const float err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(-o, bb));
  if (err == 0.f && fabsf(s) < P.box) {
    const float q = s > P.boxhalf ? __fsub_rn(s, P.box) : (s < -P.boxhalf ? __fadd_rn(s, P.box) : s);
    const float p = __fmul_rn(q, m);
    const float r = __fmaf_rn(q, m, -p);  // q*m - p, exact
    return dadd(f2d(p), f2d(r));
  }
  return rel_times_mass_double(x, od, md, P.box, P.boxhalf);
}

// One bound particle's terms of the frame sums: w[0] += m, w[1..3] += v*m
// (float products), w[4..6] += NEAREST(x - o)*m about the origin o (periodic)
// or x*m (float products).
__device__ __forceinline__ void frame_terms(float4 a, float4 u, float4 o, const double (&od)[3],
                                            const DevParams &P, double (&w)[7])
{
  const float m = a.w;
  const double md = f2d(m);
  w[0] += md;
  w[1] += f2d(fmul(u.x, m));
  w[2] += f2d(fmul(u.y, m));
  w[3] += f2d(fmul(u.z, m));
  if (P.periodic) {
    w[4] += rel_times_mass(a.x, o.x, od[0], m, md, P);
    w[5] += rel_times_mass(a.y, o.y, od[1], m, md, P);
    w[6] += rel_times_mass(a.z, o.z, od[2], m, md, P);
  } else {
    w[4] += f2d(fmul(a.x, m));
    w[5] += f2d(fmul(a.y, m));
    w[6] += f2d(fmul(a.z, m));
  }
}

// The bound block's mass-weighted means of a frame, by one warp: lanes 0..6
// hold its sums (mass, mass-weighted velocity, mass-weighted position about
// Elist[0]; v * m and x * m over m), and each lane divides one of them, so that
// the warp issues one double division, not six.  Returns the mass.
__device__ __forceinline__ double frame_means(double sum, int lane, int nb, double (&mean)[6])
{
  const double mass = __shfl_sync(0xffffffffu, sum, 0);
  const double q = ddiv(sum, nb > 1 && lane < 7 ? mass : 1.);
#pragma unroll
  for (int k = 0; k < 6; k++) mean[k] = __shfl_sync(0xffffffffu, q, k + 1);
  return mass;
}

// The decisions of subhalo s after a pass whose partition kept nb particles
// bound; msum and mean are the bound block's mass and means (frame_means)
// when nb > 1.
__device__ __forceinline__ void control_segment(const Ctx &c, SegState &sg, int nb, double msum,
                                                const double (&mean)[6], int max_passes)
{
  const DevParams &P = c.P;
  const int nl = sg.nlast;
  sg.passes++;
  sg.evals += sg.ntgt;
  if (sg.tgt_mode == 0) sg.coh_n = sg.ntgt;
  if (nb < P.minpart) {  // disruption (src/subhalo_unbind.cpp:361-379)
    sg.status = SEG_DISRUPTED;
    sg.e0 = c.eE[sg.off];
    sg.nbound = 1;
    sg.nlast = 1;
    for (int j = 0; j < 3; j++) {
      sg.ref_pos[j] = sg.mb_pos[j];
      sg.ref_vel[j] = sg.mb_vel[j];
    }
    const int k = sg.first_mb < sg.n ? sg.first_mb : 0;
    sg.mbound = c.pm[sg.off + k].w;
    sg.ub_lo = sg.ub_hi = 0;
    return;
  }
  sg.ub_lo = nb;
  sg.ub_hi = nl;
  const int ndiff = nl - nb;
  if (ndiff < nb && (P.maxsample <= 0 || ndiff < P.maxsample)) {  // :383-392
    sg.corr = 1;
    for (int j = 0; j < 3; j++) {
      sg.old_pos[j] = sg.ref_pos[j];
      sg.old_vel[j] = sg.ref_vel[j];
    }
  }
  if (nb == 1) {  // AverageVelocity / AveragePosition with one particle
    const int pid = c.epid[sg.off];
    const float4 a = c.pm[pid], u = c.vel[pid];
    sg.mbound = a.w;
    sg.ref_vel[0] = u.x;
    sg.ref_vel[1] = u.y;
    sg.ref_vel[2] = u.z;
    sg.ref_pos[0] = a.x;
    sg.ref_pos[1] = a.y;
    sg.ref_pos[2] = a.z;
  } else if (nb > 1) {
    sg.mbound = d2f(msum);
    for (int j = 0; j < 3; j++) sg.ref_vel[j] = d2f(mean[j]);
    const float4 o = c.pm[c.epid[sg.off]];
    const double org[3] = {f2d(o.x), f2d(o.y), f2d(o.z)};
    for (int j = 0; j < 3; j++) {
      double x = mean[3 + j];
      if (P.periodic) x = dadd(x, org[j]);
      sg.ref_pos[j] = d2f(x);
    }
  } else {
    sg.mbound = 0.f;
  }
  if (__int2float_rn(nb) >= fmul(__int2float_rn(nl), P.prec)) {  // :395
    sg.status = SEG_CONVERGED;
    sg.nbound = nb;
    sg.refine = P.refine && nb > P.maxsample;  // :406-407
    return;
  }
  sg.nbound = nb;
  if (sg.corr) {  // correction pass over the removed block (:312-330)
    sg.mode = MODE_CORRECTION;
    sg.t0 = nb;
    sg.ntree = nl - nb;
    sg.ntgt = nb;
    sg.mfac = 1.f;
    relvel(sg.old_pos, sg.old_vel, sg.ref_pos, sg.ref_vel, sg.dV, P);
    sg.dK = d2f(half_of(f2d(vdot(sg.dV, sg.dV))));
    sg.tgt_mode = sg.coh_n > 0 ? 1 : 2;
  } else {  // full pass (:331-356)
    sg.mode = MODE_FULL;
    sg.t0 = 0;
    sg.ntgt = nb;
    if (P.maxsample > 0 && nb > P.maxsample) {
      sg.ntree = (int)P.maxsample;
      sg.mfac = __fdiv_rn(__int2float_rn(nb), (float)P.maxsample);
      sg.tgt_mode = sg.coh_n > 0 ? 1 : 2;
    } else {
      sg.ntree = nb;
      sg.mfac = 1.f;
      sg.tgt_mode = 0;
    }
  }
  sg.nlast = nb;
  if (sg.passes >= max_passes) sg.status = SEG_FAILED;
}

static __device__ __noinline__ double nearest_double(double x, float box, float boxhalf)
{
  return x > f2d(boxhalf) ? dsub(x, f2d(box)) : x < -f2d(boxhalf) ? dadd(x, f2d(box)) : x;
}

// Type of bound particle pid for the per-type sums, -1: not counted
// (CountParticleTypes, src/subhalo.cpp:400-444); nb: Nbound.
__device__ __forceinline__ int counted_type(const Ctx &c, int nb, int pid)
{
  const int t = c.type ? c.type[pid] : 1;
  return (nb <= 100 && c.id[pid] == -1) || t < 0 || t > 5 ? -1 : t;
}

// One bound particle's terms of the final sums (list position p of nb):
// binding energy, kinetic energy, angular momentum and mass (AverageKinematics,
// src/subhalo_unbind.cpp:189-232).
__device__ __forceinline__ void kin_terms(const Ctx &c, const SegState &sg, int pid, float E,
                                          double (&v)[7])
{
  const DevParams &P = c.P;
  const float4 a = c.pm[pid], u = c.vel[pid];
  const float m = a.w;
  const float x[3] = {a.x, a.y, a.z}, w[3] = {u.x, u.y, u.z};
  const double md = f2d(m);
  v[0] += f2d(fmul(E, m));
  double dx[3], dv[3];
  for (int j = 0; j < 3; j++) {
    // the wrap of a float difference below the box size is exact in float
    // (Sterbenz), so it gives the double wrap's bits without the FP64 pipe
    const float d = fsub(x[j], sg.ref_pos[j]);
    if (!P.periodic)
      dx[j] = f2d(d);
    else if (fabsf(d) < P.box)
      dx[j] = f2d(nearest_f(d, P));
    else
      dx[j] = nearest_double(f2d(d), P.box, P.boxhalf);
    dx[j] = dmul(dx[j], P.ad);
    dv[j] = dadd(f2d(fsub(w[j], sg.ref_vel[j])), dmul(P.Hzd, dx[j]));
    v[1] += dmul(dmul(dv[j], dv[j]), md);
  }
  v[2] += dmul(dsub(dmul(dx[1], dv[2]), dmul(dx[2], dv[1])), md);
  v[3] += dmul(dsub(dmul(dx[2], dv[0]), dmul(dx[0], dv[2])), md);
  v[4] += dmul(dsub(dmul(dx[0], dv[1]), dmul(dx[1], dv[0])), md);
  v[5] += md;
}

// A warp's final sums over the list positions first, first + kLB, ... < hi of each
// lane (Nbound nb), in the association of block_sum<18>: sums 0..5 are
// kin_terms', 6..11 the counts of each type and 12..17 their masses; sum k to
// out[k * stride].  Almost always a warp's particles are of one type: then five of
// the masses' sums are zero, and seven sums are reduced instead of 18.
__device__ __forceinline__ void kin_warp_sums(const Ctx &c, const SegState &sg, int nb, int first,
                                              int hi, double *out, int stride)
{
  const int lane = threadIdx.x & 31;
  double v[7] = {0., 0., 0., 0., 0., 0., 0.};
  int cnt[6] = {0, 0, 0, 0, 0, 0};
  int lo_t = 6, hi_t = -1;  // the types met
  for (int p = first; p < hi; p += kLB) {
    const int pid = c.epid[sg.off + p];
    kin_terms(c, sg, pid, c.eE[sg.off + p], v);
    const int t = counted_type(c, nb, pid);
    if (t >= 0) {
      lo_t = min(lo_t, t);
      hi_t = max(hi_t, t);
      v[6] += f2d(c.pm[pid].w);
    }
#pragma unroll
    for (int q = 0; q < 6; q++) cnt[q] += t == q;
  }
  const int t0 = __reduce_min_sync(0xffffffffu, lo_t), t1 = __reduce_max_sync(0xffffffffu, hi_t);
  double sum;
  const int k = warp_sums<7>(v, &sum);
  if (k >= 0 && k < 6) out[k * stride] = sum;
#pragma unroll
  for (int q = 0; q < 6; q++) cnt[q] = __reduce_add_sync(0xffffffffu, cnt[q]);
  if (lane < 6) {
    int n = cnt[0];
#pragma unroll
    for (int q = 1; q < 6; q++) n = lane == q ? cnt[q] : n;
    out[(6 + lane) * stride] = (double)n;  // exact
    if (t0 >= t1 && lane != t0) out[(12 + lane) * stride] = 0.;
  }
  if (t0 >= t1) {
    if (k == 6 && t1 >= 0) out[(12 + t0) * stride] = sum;
    return;
  }
  double w[6] = {0., 0., 0., 0., 0., 0.};  // several types
  for (int p = first; p < hi; p += kLB) {
    const int pid = c.epid[sg.off + p];
    const int t = counted_type(c, nb, pid);
    const double md = f2d(c.pm[pid].w);
#pragma unroll
    for (int q = 0; q < 6; q++) w[q] += t == q ? md : 0.;
  }
  const int q = warp_sums<6>(w, &sum);
  if (q >= 0) out[(12 + q) * stride] = sum;
}

// A subhalo's result record, by one warp: lanes 0..17 hold the sums of
// kin_terms (v[6..11] the type counts) when it is neither trivial nor disrupted.
__device__ __forceinline__ void write_result(const Ctx &c, const SegState &sg, double part,
                                             int lane, hbtu_result *res)
{
  const DevParams &P = c.P;
  const bool summed = sg.status != SEG_TRIVIAL && sg.status != SEG_DISRUPTED;
  double v[18];
#pragma unroll
  for (int k = 0; k < 18; k++) v[k] = __shfl_sync(0xffffffffu, part, k);
  // the divisions by the mass, one per lane: E, 1/2 (for K), the angular momentum
  const double num = lane == 0 ? v[0] : (lane == 1 ? 0.5 : (lane < 5 ? part : 1.));
  const double quot = ddiv(num, summed && sg.nbound > 1 && lane < 5 ? v[5] : 1.);
  double over_m[5];
#pragma unroll
  for (int k = 0; k < 5; k++) over_m[k] = __shfl_sync(0xffffffffu, quot, k);
  if (lane != 0) return;
  hbtu_result r;
  memset(&r, 0, sizeof(r));
  r.too_few = sg.n < P.minpart;
  r.iterations = sg.passes;
  r.evaluations = sg.evals;
  r.interactions = sg.interactions;
  for (int j = 0; j < 3; j++) {
    r.ref_pos[j] = sg.ref_pos[j];
    r.ref_vel[j] = sg.ref_vel[j];
    r.mostbound_pos[j] = sg.mb_pos[j];
    r.mostbound_vel[j] = sg.mb_vel[j];
  }
  if (sg.status == SEG_TRIVIAL) {  // src/subhalo_unbind.cpp:275-293 + CountParticles
    r.nbound = sg.n;
    if (sg.n == 1) {
      const int t = c.type ? c.type[sg.off] : 1;
      const float m = c.pm[sg.off].w;
      if (t >= 0 && t <= 5) {
        r.nbound_type[t] = 1;
        r.mbound_type[t] = m;
      }
      float acc = 0.f;
      for (int k = 0; k < 6; k++) acc = fadd(acc, r.mbound_type[k]);
      r.mbound = acc;
    }
  } else if (sg.status == SEG_DISRUPTED) {
    r.disrupted = 1;
    r.nbound = 1;
    r.mbound = sg.mbound;
    const int k = sg.first_mb < sg.n ? sg.first_mb : 0;
    const int t = c.type ? c.type[sg.off + k] : 1;
    const bool skip = c.id[sg.off + k] == -1 || t < 0 || t > 5;
    if (!skip) {
      r.nbound_type[t] = 1;
      r.mbound_type[t] = c.pm[sg.off + k].w;
    }
  } else {
    r.converged = sg.status == SEG_CONVERGED;
    if (sg.status == SEG_FAILED) r.status = HBTU_ERR_NOT_CONVERGED;
    r.nbound = sg.nbound;
    r.mbound = sg.mbound;
    if (sg.nbound > 0) {
      const int pid = c.epid[sg.off];
      const float4 a = c.pm[pid], u = c.vel[pid];
      r.mostbound_pos[0] = a.x;
      r.mostbound_pos[1] = a.y;
      r.mostbound_pos[2] = a.z;
      r.mostbound_vel[0] = u.x;
      r.mostbound_vel[1] = u.y;
      r.mostbound_vel[2] = u.z;
    }
    if (sg.nbound > 1) {
      const double E = over_m[0];
      const double K = dmul(v[1], over_m[1]);
      r.specific_potential = d2f(dsub(E, K));
      r.specific_kinetic = d2f(K);
      for (int j = 0; j < 3; j++) r.specific_angmom[j] = d2f(over_m[2 + j]);
    }
    for (int t = 0; t < 6; t++) {
      r.nbound_type[t] = (int64_t)v[6 + t];
      r.mbound_type[t] = d2f(v[12 + t]);
    }
  }
  *res = r;
}

// Order and energy at global list position p of subhalo sg.
__device__ __forceinline__ void write_position(const Ctx &c, const SegState &sg, int p,
                                               int64_t *order, float *energy)
{
  const int l = p - sg.off;
  if (sg.status == SEG_TRIVIAL) {
    order[p] = l;
    energy[p] = 0.f;
  } else if (sg.status == SEG_DISRUPTED) {
    const int k = sg.first_mb < sg.n ? sg.first_mb : 0;
    order[p] = l == 0 ? k : (l == k ? 0 : l);
    energy[p] = l == 0 ? sg.e0 : __int_as_float(0x7fc00000);
  } else {
    order[p] = c.epid[p] - sg.off;
    energy[p] = c.eE[p];
  }
}

}  // namespace hbtu
