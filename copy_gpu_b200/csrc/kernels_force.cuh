// kernels_force.cuh -- near-field pair force (LJ 12-6 + real-space erfc Coulomb), the RBE
// k-space force fused into the same per-atom pass, RBE structure factors, the RBE k-sampler,
// and the EAM density / force passes.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "kernels_bonded.cuh"

namespace rbmd {

// ------------------------------------------------------------------------------------------
// k-sample record: integer m vector plus the per-sample force coefficient w*k (w folds S/P,
// qqr2e, -4 pi / (V k^2), the importance weight and the sign of the phase convention) and the
// structure factor rho = sum_j q_j e^{i k.r_j}.  32 B (FP32) so that a record is two 16-byte
// shared-memory loads; the owning replica of record g is krep[g].
// ------------------------------------------------------------------------------------------
struct KRec32 { int mx, my, mz; float wx, wy, wz, re, im; };                 // 32 B
struct KRec64 { int mx, my, mz, pad; double wx, wy, wz, re, im, pad2; };     // 64 B

// phase -> (cos, sin) of 2*pi*(t - 1/2) for a 32-bit fixed-point turn t: the top 23 bits form a
// float in [1, 2), so tf - 1.5 lies in [-0.5, 0.5); MUFU sin/cos are accurate on [-pi, pi].
__device__ __forceinline__ void turn_sincos(uint32_t ph, float& s, float& c) {
  float tf = __uint_as_float((ph >> 9) | 0x3F800000u) - 1.5f;
  float th = tf * 6.28318530717958647692f;
  __sincosf(th, &s, &c);
}
// 64-bit fixed-point turn -> exact double angle 2*pi*(t - 1/2) with t - 1/2 in [-0.5, 0.5)
__device__ __forceinline__ void turn_sincos(unsigned long long ph, double& s, double& c) {
  long long sg = (long long)(ph ^ 0x8000000000000000ull);   // (t - 1/2) * 2^64 as signed
  double t = (double)sg * 5.42101086242752217e-20;           // 2^-64
  sincospi(2.0 * t, &s, &c);
}

struct LJTable {
  float lj24_f[kMaxReplicaTypes * kMaxReplicaTypes];    // -24 sqrt(eps_i eps_j)  (float)
  float sig6_f[kMaxReplicaTypes * kMaxReplicaTypes];    // ((sig_i + sig_j)/2)^6   (float)
  double lj24_d[kMaxReplicaTypes * kMaxReplicaTypes];
  double sig6_d[kMaxReplicaTypes * kMaxReplicaTypes];
};

struct NearParams {
  int n, stride, ntypes, cap;
  int with_lj, with_coul, molecular;
  double rc, alpha, coul_scale;   // coul_scale multiplies the erfc Coulomb pair force
  double sqrt_alpha, two_sqrt_alpha_over_sqrt_pi;
  int kstage;                     // records of shared memory available for k staging
  int orig;                       // neighbour type "ORIGINAL": pairs with d^2 < rc^2 (no 1e-4 margin)
  SpecialDev sp;                  // molecular == 2: special-bond partner lists
};

template <class R> struct KRec;
template <> struct KRec<float> { using T = KRec32; };
template <> struct KRec<double> { using T = KRec64; };
// e^x, 1/sqrt(x) and 1/x by one MUFU operation each.  The flush-to-zero forms leave out the
// rescaling of denormals, which the arguments here never are: x = -alpha d^2 above -100, d^2 > 1e-4.
__device__ __forceinline__ float exp_r(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.44269504088896340736f));
  return r;
}
__device__ __forceinline__ double exp_r(double x) { return exp(x); }
__device__ __forceinline__ float rsqrt_r(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_r(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_r(double x) { return sqrt(x); }
__device__ __forceinline__ double rsqrt_r(double x) { return 1.0 / sqrt(x); }

// approximate reciprocal (one MUFU op, about 1 ulp): the pair terms carry a 1e-5 budget
__device__ __forceinline__ float rcp_r(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The same with one Newton step, to within about an ulp (the IEEE form takes a dozen instructions).
__device__ __forceinline__ float rcp_nr(float x) {
  const float t = rcp_r(x);
  return fmaf(t, fmaf(-x, t, 1.0f), t);
}

// erfc(x) for x >= 0 given e = exp(-x^2).  FP32: Abramowitz & Stegun, Handbook of Mathematical
// Functions, eq. 7.1.26 (rational approximation in t = 1/(1 + p x), |error| <= 1.5e-7), which
// reuses the Gaussian factor the real-space force needs anyway.  FP64: the library erfc.
__device__ __forceinline__ float erfc_shared(float x, float e) {
  const float t = rcp_nr(fmaf(0.3275911f, x, 1.0f));   // an ulp of t leaves the formula's 1.5e-7 as it is
  float poly = fmaf(1.061405429f, t, -1.453152027f);
  poly = fmaf(poly, t, 1.421413741f);
  poly = fmaf(poly, t, -0.284496736f);
  poly = fmaf(poly, t, 0.254829592f);
  return poly * t * e;
}
__device__ __forceinline__ double erfc_shared(double x, double) { return erfc(x); }

// the same for two arguments side by side: e^(-a d2), and erfc with its Gaussian factors
__device__ __forceinline__ Pair<float> exp_neg2(float a, Pair<float> d2) {
  const Pair<float> m = mul2(mul2(both<float>(-a), d2), both<float>(1.44269504088896340736f));
  Pair<float> r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(m.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(m.y));
  return r;
}
__device__ __forceinline__ Pair<double> exp_neg2(double a, Pair<double> d2) { return {exp(-a * d2.x), exp(-a * d2.y)}; }
__device__ __forceinline__ Pair<float> erfc_shared2(Pair<float> x, Pair<float> e) {
  const Pair<float> one = both<float>(1.0f), u = fma2(both<float>(0.3275911f), x, one);
  const Pair<float> w{rcp_r(u.x), rcp_r(u.y)};
  const Pair<float> t = fma2(w, fma2(mul2(both<float>(-1.0f), u), w, one), w);
  Pair<float> poly = fma2(both<float>(1.061405429f), t, both<float>(-1.453152027f));
  poly = fma2(poly, t, both<float>(1.421413741f));
  poly = fma2(poly, t, both<float>(-0.284496736f));
  poly = fma2(poly, t, both<float>(0.254829592f));
  return mul2(mul2(poly, t), e);
}
__device__ __forceinline__ Pair<double> erfc_shared2(Pair<double> x, Pair<double>) { return {erfc(x.x), erfc(x.y)}; }

template <class R> __host__ __device__ __forceinline__ R lj24(const LJTable& t, int k);
template <> __host__ __device__ __forceinline__ float lj24<float>(const LJTable& t, int k) { return t.lj24_f[k]; }
template <> __host__ __device__ __forceinline__ double lj24<double>(const LJTable& t, int k) { return t.lj24_d[k]; }
template <class R> __host__ __device__ __forceinline__ R sig6(const LJTable& t, int k);
template <> __host__ __device__ __forceinline__ float sig6<float>(const LJTable& t, int k) { return t.sig6_f[k]; }
template <> __host__ __device__ __forceinline__ double sig6<double>(const LJTable& t, int k) { return t.sig6_d[k]; }

// RBE force terms of one atom over the k records sub, sub + G, .. < P of `kr` (shared or global memory).
template <class R, int G>
__device__ __forceinline__ void rbe_terms(const typename FracT<R>::T& fr, const typename KRec<R>::T* kr,
                                          int P, int sub, R& ax, R& ay, R& az) {
#pragma unroll 4
  for (int l = sub; l < P; l += G) {
    const typename KRec<R>::T k = kr[l];
    R s, c;
    if constexpr (sizeof(R) == 4) {
      const uint32_t ph = (uint32_t)k.mx * fr.x + (uint32_t)k.my * fr.y + (uint32_t)k.mz * fr.z;
      turn_sincos(ph, s, c);
    } else {
      const unsigned long long ph = (unsigned long long)(long long)k.mx * fr.x +
                                    (unsigned long long)(long long)k.my * fr.y +
                                    (unsigned long long)(long long)k.mz * fr.z;
      turn_sincos(ph, s, c);
    }
    const R val = c * (R)k.im - s * (R)k.re;
    ax += val * (R)k.wx;
    ay += val * (R)k.wy;
    az += val * (R)k.wz;
  }
}

// Minimum-image handling of the pair vector in the near pass:
//   kMiNone  every replica has >= 3 cells per axis and the list is rebuilt every step: listed
//            pairs have |r_d| < rc < L/2, MinDistanceVec is the identity;
//   kMiLJ    the reference's semantics for small boxes: MinDistanceVec on the LJ vector only;
//   kMiAll   Verlet skin: pairs listed at rc + skin are filtered by the list predicate at rc;
//            the cached positions are unwrapped since the build (k_regather), so the stored
//            image shift still gives the minimum-image vector.
constexpr int kMiNone = 0, kMiLJ = 1, kMiAll = 2;
// Added to MI: the LJ pairs of one bond-graph component take their special-bond weight
// (molecular == 2).  A separate instantiation, so the passes without topology carry none of it.
constexpr int kMiSpecial = 4;

template <class R>
__device__ __forceinline__ void min_image(R& q0, R& q1, R& q2, const R* box) {
  if (fabs(q0) > box[0] * (R)0.5) q0 -= (q0 > 0 ? box[0] : -box[0]);
  if (fabs(q1) > box[1] * (R)0.5) q1 -= (q1 > 0 ? box[1] : -box[1]);
  if (fabs(q2) > box[2] * (R)0.5) q2 -= (q2 > 0 ? box[2] : -box[2]);
}

__device__ __forceinline__ double rcp_r(double x) { return 1.0 / x; }

// Near force of one slot per thread over its list row.
// Pair physics: ComputeNearForceVerletWorklet / ComputeLJForceVerletWorklet
// (rbmd/framework/run/worklet/RunWorklet.cpp:170-303) with ComputeLJForce and
// ComputeNearEnergyForce (rbmd/framework/forceFunction/ExecForceFunction.h:74-140):
//   LJ on MinDistanceVec(p_j', p_i) skipped within a molecule; Coulomb on p_j' - p_i for
//   0.01 < d < rc with G = erfc(sqrt(a) d)/d^2 + 2 sqrt(a) e^{-a d^2}/(sqrt(pi) d); pairs with
//   q_i q_j = 0 skip the Coulomb term.  Under list reuse (MI == kMiAll, list built at rc + skin)
//   a pair also has to pass the list predicate at rc (rc^2 - d^2 > 1e-4 && d^2 > 1e-4), as the
//   reference's per-call list would.
// Per-type LJ coefficients are staged in shared memory.  The loop is software-pipelined: the
// list entry two iterations ahead and the neighbour position one iteration ahead are in flight
// while the current pair is evaluated.  Accumulation: groups of four pair forces are summed in
// FP32 and folded into a two-float (TwoSum) per-atom accumulator.
template <class R, bool COUL, int MI>
__global__ void __launch_bounds__(256) k_near_force(
    NearParams prm, const LJTable* __restrict__ ljt, const typename Traits<R>::V4* __restrict__ pos4,
    const int2* __restrict__ meta, const int* __restrict__ nbr, const int* __restrict__ count,
    const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot,
    const int* __restrict__ slot_atom, double* __restrict__ force,
    double* __restrict__ energy_slot, uint32_t* status) {
  using V4 = typename Traits<R>::V4;
  __shared__ R lj_a[kMaxReplicaTypes * kMaxReplicaTypes], lj_s6[kMaxReplicaTypes * kMaxReplicaTypes];
  const int nt2 = prm.ntypes * prm.ntypes;
  for (int t = threadIdx.x; t < nt2; t += blockDim.x) {
    lj_a[t] = lj24<R>(*ljt, t);
    lj_s6[t] = sig6<R>(*ljt, t);
  }
  __syncthreads();
  const bool MOLEC = prm.molecular != 0;
  constexpr bool SPW = (MI & kMiSpecial) != 0;
  const bool ENERGY = energy_slot != nullptr;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= prm.n) return;
  const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
  const V4 pi = pos4[i];
  const bool typed = MOLEC || prm.ntypes > 1;
  const int2 mi = typed ? meta[i] : make_int2(0, 0);
  const R rc = (R)prm.rc;
  const R cut2 = rc * rc;
  const R box[3] = {Traits<R>::box(rp, 0), Traits<R>::box(rp, 1), Traits<R>::box(rp, 2)};
  const R wrap[3] = {Traits<R>::wrap(rp, 0), Traits<R>::wrap(rp, 1), Traits<R>::wrap(rp, 2)};
  const R sa = (R)prm.sqrt_alpha, aa = (R)prm.alpha, c2 = (R)prm.two_sqrt_alpha_over_sqrt_pi;
  const R cs = (R)prm.coul_scale;
  const R qi = pi.w;
  const int trow = prm.ntypes > 1 ? mi.x * prm.ntypes : 0;   // one LJ type when all types agree
  const int st = prm.stride;
  Acc<R> fx, fy, fz;
  R gx = 0, gy = 0, gz = 0;   // FP32 group sum folded into the accumulators every 4 pairs
  R e_lj = 0, e_coul = 0;
  const int cnt = min(count[i], prm.cap);   // an overflowed row is redone after regrowth
  // pipeline prologue
  int e_cur = cnt > 0 ? __ldg(nbr + nbr_at(0, i, st)) : 0;
  int e_nxt = cnt > 1 ? __ldg(nbr + nbr_at(1, i, st)) : 0;
  V4 pj_cur = pos4[cnt > 0 ? (e_cur >> kShiftBits) : i];
  for (int p = 0; p < cnt; ++p) {
    const int e = e_cur;
    const V4 pj = pj_cur;
    // issue the loads of the next iterations before the arithmetic of this one
    e_cur = e_nxt;
    if (p + 1 < cnt) pj_cur = pos4[e_cur >> kShiftBits];
    if (p + 2 < cnt) e_nxt = __ldg(nbr + nbr_at(p + 2, i, st));
    R px = pj.x, py = pj.y, pz = pj.z;
    if (e & 63) {   // periodic image: p_j - offset (PeriodicCoordOffset)
      const int c0 = e & 3, c1 = (e >> 2) & 3, c2b = (e >> 4) & 3;
      px = px - (c0 == 1 ? wrap[0] : (c0 == 2 ? -wrap[0] : (R)0));
      py = py - (c1 == 1 ? wrap[1] : (c1 == 2 ? -wrap[1] : (R)0));
      pz = pz - (c2b == 1 ? wrap[2] : (c2b == 2 ? -wrap[2] : (R)0));
    }
    const R r0 = px - pi.x, r1 = py - pi.y, r2 = pz - pi.z;
    const R d2 = r0 * r0 + r1 * r1 + r2 * r2;
    if ((MI & 3) == kMiAll && !((prm.orig ? cut2 - d2 > (R)0 : cut2 - d2 > (R)1.0e-4) && d2 > (R)1.0e-4)) continue;
    R f = 0;
    if (COUL) {
      const R qq = qi * pj.w;
      if (qq != (R)0) {
        const R inv = rsqrt_r(d2);
        const R dis = d2 * inv;
        if (dis < rc && dis > (R)0.01) {
          const R ex = exp_r(-aa * d2);
          const R erfcv = erfc_shared(sa * dis, ex);
          const R g = (erfcv * inv + c2 * ex) * inv;
          f = -qq * g * inv * cs;
          if (ENERGY) e_coul += qq * erfcv * inv * cs;
        }
      }
    }
    R fl0 = 0, fl1 = 0, fl2 = 0;
    bool same = false;
    int tj = 0;
    R wsp = (R)1;   // special-bond LJ weight (molecular == 2: meta.y is the bond-graph component)
    if (typed) {
      const int2 mj = meta[e >> kShiftBits];
      same = MOLEC && (mj.y == mi.y);
      tj = prm.ntypes > 1 ? mj.x : 0;
      if (SPW && same) {
        wsp = special_weight<R>(prm.sp, slot_atom[i], slot_atom[e >> kShiftBits]);
        same = false;
      }
    }
    if (!same) {
      R q0 = r0, q1 = r1, q2 = r2;   // MinDistanceVec(p_j', p_i)
      R dl2 = d2;
      if ((MI & 3) == kMiLJ) {
        min_image(q0, q1, q2, box);
        dl2 = q0 * q0 + q1 * q1 + q2 * q2;
      }
      if (dl2 < cut2 && dl2 > (R)0.0001) {
        const R inv2 = rcp_r(dl2);
        const R sd6 = lj_s6[trow + tj] * inv2 * inv2 * inv2;
        const R a24 = lj_a[trow + tj];
        R scal = a24 * (((R)2 * sd6 - (R)1) * sd6) * inv2;
        if (SPW) scal *= wsp;
        fl0 = scal * q0; fl1 = scal * q1; fl2 = scal * q2;
        // 4 eps (s6 - 1) s6 with 4 eps = -lj24/6
        if (ENERGY) e_lj += (SPW ? wsp : (R)1) * (-a24 / (R)6 * (sd6 - (R)1) * sd6);
      }
    }
    gx += f * r0 + fl0;
    gy += f * r1 + fl1;
    gz += f * r2 + fl2;
    if ((p & 3) == 3) {
      fx.add(gx); fy.add(gy); fz.add(gz);
      gx = gy = gz = 0;
    }
  }
  fx.add(gx); fy.add(gy); fz.add(gz);
  const double F[3] = {fx.value(), fy.value(), fz.value()};
  if (!isfinite(F[0]) || !isfinite(F[1]) || !isfinite(F[2])) set_flag(status, kFlagNonFinite);
  const int id = slot_atom[i];
  force[3 * id] = F[0];
  force[3 * id + 1] = F[1];
  force[3 * id + 2] = F[2];
  if (ENERGY) {
    energy_slot[2 * i] = 0.5 * (double)e_lj;
    energy_slot[2 * i + 1] = 0.5 * (double)e_coul;
  }
}

// Near force, one thread per atom, for the common case of one LJ coefficient pair for every type
// pair and no molecules (the electrolyte benchmarks): the same pair set,
// predicates and pair physics as k_near_force, with less work per listed pair:
//   * the list is walked a chunk of four entries at a time: one 16-byte load per chunk, the last
//     chunk filled with the slot itself by the list build (distance 0, which the predicate
//     refuses), so no entry is tested against the row's length; the entries of the chunk after
//     next and the positions of the next are in flight while a chunk is evaluated;
//   * all lanes of a warp run the chunks of its longest row (lanes past their row hold the slot
//     itself), so the votes below are on full warps;
//   * the periodic image offsets are decoded only when some lane of the warp holds an image
//     entry in the chunk (most warps hold none), in one branch per chunk;
//   * the LJ terms of two entries are evaluated side by side in packed FP32x2 instructions,
//     branch-free, and selected by the predicate d2_lo < d^2 <= d2_max (the list predicate at rc
//     as one comparison, list_d2_max);
//   * the four pair forces of a chunk are summed in R and folded into the two-float accumulator.
// Bound by issue and the latency of the position gathers; 1,000,000 atoms, 72 listed pairs each:
// 288 -> 219 us, 512 replicas (2.2 M atoms) 685 -> 548 us against one 4-byte list load, one length
// test and one image branch per entry.
// Pair physics as k_near_force: ComputeNearForceVerletWorklet / ComputeLJForceVerletWorklet
// (rbmd/framework/run/worklet/RunWorklet.cpp:170-303), ExecForceFunction::ComputeLJForce and
// ComputeNearEnergyForce (rbmd/framework/forceFunction/ExecForceFunction.h:74-140).
// G > 1: G lanes per atom for systems with too few atoms to fill the chip; lane s takes the chunks
// s, s + G, .. and the lanes' sums are combined in FP64 by a fixed butterfly.
// FP32 is held to 64 registers (32 warps per SM; 74 without).  With that and the .ftz forms of exp_r
// and rsqrt_r: 1,000,000 atoms 219 -> 191 -> 181 us, 512 replicas 548 -> 478 -> 448 us (69 % of the
// issue slots, 28.9 of 32 lanes active).
template <class R, bool COUL, int MI, bool ENERGY, int G>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 1) k_near_lean(
    NearParams prm, R a24, R s6, R d2_max, const typename Traits<R>::V4* __restrict__ pos4,
    const int4* __restrict__ nbr4, const int* __restrict__ count, const RepDev* __restrict__ reps,
    const int* __restrict__ rep_of_slot, const int* __restrict__ slot_atom, double* __restrict__ force,
    double* __restrict__ energy_slot, uint32_t* status) {
  static_assert((MI & 3) != kMiLJ && (MI & kMiSpecial) == 0, "k_near_lean: no per-pair minimum image, no weights");
  using V4 = typename Traits<R>::V4;
  const int gid = (int)((blockIdx.x * blockDim.x + threadIdx.x) / G), sub = threadIdx.x % G;
  const bool active = gid < prm.n;   // lanes past the end run along with an empty row
  const int i = active ? gid : prm.n - 1;
  const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
  const V4 pi = pos4[i];
  const R rc = (R)prm.rc;
  const R sa = (R)prm.sqrt_alpha, aa = (R)prm.alpha, c2 = (R)prm.two_sqrt_alpha_over_sqrt_pi;
  const R cs = (R)prm.coul_scale;
  const R qi = pi.w;
  const int nch = active ? (min(count[i], prm.cap) + 3) >> 2 : 0;   // chunks of the row
  const int last = __reduce_max_sync(0xffffffffu, nch);
  const int self = i << kShiftBits;
  const int4 idle = make_int4(self, self, self, self);
  // 24 eps (2 s6 u - 1) s6 u / d^2 with u = d^-6 as (ka u - kb) d^-8
  const Pair<R> ka = both<R>((R)2 * a24 * s6 * s6), kb = both<R>(-a24 * s6);
  Acc3<R> F;
  R e_lj = 0, e_coul = 0;
  const size_t st = (size_t)prm.stride * G;
  const int4* row = nbr4 + (size_t)prm.stride * sub + i;
  int4 e = sub < nch ? __ldg(row) : idle;
  int4 e_nxt = sub + G < nch ? __ldg(row + st) : idle;
  row += 2 * st;
  V4 pj[4] = {pos4[e.x >> kShiftBits], pos4[e.y >> kShiftBits], pos4[e.z >> kShiftBits], pos4[e.w >> kShiftBits]};
  for (int c = sub; c - sub < last; c += G, row += st) {
    if (__any_sync(0xffffffffu, ((e.x | e.y | e.z | e.w) & 63) != 0)) {   // p_j - PeriodicCoordOffset
      const int ee[4] = {e.x, e.y, e.z, e.w};
      const R w0 = Traits<R>::wrap(rp, 0), w1 = Traits<R>::wrap(rp, 1), w2 = Traits<R>::wrap(rp, 2);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int k0 = ee[k] & 3, k1 = (ee[k] >> 2) & 3, k2 = (ee[k] >> 4) & 3;
        pj[k].x -= k0 == 1 ? w0 : (k0 == 2 ? -w0 : (R)0);
        pj[k].y -= k1 == 1 ? w1 : (k1 == 2 ? -w1 : (R)0);
        pj[k].z -= k2 == 1 ? w2 : (k2 == 2 ? -w2 : (R)0);
      }
    }
    Pair<R> gx = both<R>(0), gy = both<R>(0), gz = both<R>(0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const V4 &pa = pj[2 * h], &pb = pj[2 * h + 1];
      const Pair<R> rx{pa.x - pi.x, pb.x - pi.x}, ry{pa.y - pi.y, pb.y - pi.y}, rz{pa.z - pi.z, pb.z - pi.z};
      const Pair<R> d2 = fma2(rz, rz, fma2(ry, ry, mul2(rx, rx)));
      const bool in[2] = {d2.x > (R)1.0e-4 && d2.x <= d2_max, d2.y > (R)1.0e-4 && d2.y <= d2_max};
      const Pair<R> i2{rcp_r(d2.x), rcp_r(d2.y)};
      const Pair<R> i4 = mul2(i2, i2), i6 = mul2(i4, i2), i8 = mul2(i4, i4);
      const Pair<R> lj = mul2(fma2(ka, i6, kb), i8);
      Pair<R> t{in[0] ? lj.x : (R)0, in[1] ? lj.y : (R)0};
      if (ENERGY) {
        // 4 eps (sd6 - 1) sd6 with 4 eps = -a24 / 6
        const R sx = s6 * i6.x, sy = s6 * i6.y;
        if (in[0]) e_lj += -a24 / (R)6 * (sx - (R)1) * sx;
        if (in[1]) e_lj += -a24 / (R)6 * (sy - (R)1) * sy;
      }
      if (COUL) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const R qq = qi * (k ? pb.w : pa.w);
          if (in[k] && qq != (R)0) {
            const R dd = k ? d2.y : d2.x;
            const R inv = rsqrt_r(dd);
            const R dis = dd * inv;
            if (dis < rc && dis > (R)0.01) {
              const R ex = exp_r(-aa * dd);
              const R erfcv = erfc_shared(sa * dis, ex);
              const R g = (erfcv * inv + c2 * ex) * inv;
              const R f = -qq * g * inv * cs;
              if (k) t.y += f;
              else t.x += f;
              if (ENERGY) e_coul += qq * erfcv * inv * cs;
            }
          }
        }
      }
      gx = fma2(t, rx, gx);
      gy = fma2(t, ry, gy);
      gz = fma2(t, rz, gz);
    }
    F.add(gx.x + gx.y, gy.x + gy.y, gz.x + gz.y);
    // advance the pipeline: positions of the next chunk, entries of the one after
    e = e_nxt;
    pj[0] = pos4[e.x >> kShiftBits];
    pj[1] = pos4[e.y >> kShiftBits];
    pj[2] = pos4[e.z >> kShiftBits];
    pj[3] = pos4[e.w >> kShiftBits];
    e_nxt = c + 2 * G < nch ? __ldg(row) : idle;
  }
  double Fd[3] = {F.vx(), F.vy(), F.vz()}, el = (double)e_lj, ec = (double)e_coul;
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    Fd[0] += __shfl_xor_sync(0xffffffffu, Fd[0], o);
    Fd[1] += __shfl_xor_sync(0xffffffffu, Fd[1], o);
    Fd[2] += __shfl_xor_sync(0xffffffffu, Fd[2], o);
    if (ENERGY) {
      el += __shfl_xor_sync(0xffffffffu, el, o);
      ec += __shfl_xor_sync(0xffffffffu, ec, o);
    }
  }
  if (!active || sub != 0) return;
  if (!isfinite(Fd[0]) || !isfinite(Fd[1]) || !isfinite(Fd[2])) set_flag(status, kFlagNonFinite);
  const int id = slot_atom[i];
  force[3 * id] = Fd[0];
  force[3 * id + 1] = Fd[1];
  force[3 * id + 2] = Fd[2];
  if (ENERGY) {
    energy_slot[2 * i] = 0.5 * el;
    energy_slot[2 * i + 1] = 0.5 * ec;
  }
}

// Near force with G lanes per atom (G = 4 .. 32) for systems with few atoms or long lists
// (water at 10 A: ~550 neighbours, 30,000 atoms), where one thread per atom leaves most of the
// GPU idle.  Lane s of an atom's group takes the chunks s, s + G, .. of four list entries: one
// 16-byte load per chunk, the next chunk's entries and the four positions (and, with types or
// molecules, records) of the current one in flight together, the image offsets decoded in one
// branch per chunk.  The filler entries of the last chunk hold the slot itself, at distance 0,
// which no predicate accepts.  The pair terms are those of k_near_force (same predicates and
// operations), two entries side by side in packed FP32x2 instructions, branch-free and selected
// by the predicates; each lane sums the four forces of a chunk and folds them into a two-float
// accumulator, and the group combines its G partial sums in FP64 with a fixed butterfly, so the
// result does not depend on scheduling.  Bound by issue and the latency of the gathers.  Five steps
// of 30,000 water atoms at 16 lanes 1231 us with a branch per entry and predicate, 1120 packed (the
// pass 113 -> 91 us, 75.9 -> 56.2 M warp instructions, 63 % of the issue slots);
// 22,824 chain atoms with special bonds 777 -> 686 us (80 registers: 1120 and 709; the next chunk's
// positions a step ahead: 1131 and 716).  The special lists, needed only for pairs inside a
// molecule, are searched in one copy outside the unrolled entries, where they took 16 us a pass.
template <class R, bool COUL, int MI, int G>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 1) k_near_force_group(
    NearParams prm, const LJTable* __restrict__ ljt, const typename Traits<R>::V4* __restrict__ pos4,
    const int2* __restrict__ meta, const int* __restrict__ nbr, const int* __restrict__ count,
    const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot,
    const int* __restrict__ slot_atom, double* __restrict__ force,
    double* __restrict__ energy_slot, uint32_t* status) {
  using V4 = typename Traits<R>::V4;
  __shared__ R lj_a[kMaxReplicaTypes * kMaxReplicaTypes], lj_s6[kMaxReplicaTypes * kMaxReplicaTypes];
  const int nt2 = prm.ntypes * prm.ntypes;
  for (int t = threadIdx.x; t < nt2; t += blockDim.x) {
    lj_a[t] = lj24<R>(*ljt, t);
    lj_s6[t] = sig6<R>(*ljt, t);
  }
  __syncthreads();
  const bool MOLEC = prm.molecular != 0;
  constexpr bool SPW = (MI & kMiSpecial) != 0;
  const bool ENERGY = energy_slot != nullptr;
  const int gid = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) / G);
  const int sub = threadIdx.x % G;
  const bool active = gid < prm.n;   // inactive groups still join the shuffles below
  const int i = active ? gid : prm.n - 1;
  const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
  const V4 pi = pos4[i];
  const bool typed = MOLEC || prm.ntypes > 1;
  const int2 mi = typed ? meta[i] : make_int2(0, 0);
  const R rc = (R)prm.rc;
  const R cut2 = rc * rc;
  const R sa = (R)prm.sqrt_alpha, aa = (R)prm.alpha, c2 = (R)prm.two_sqrt_alpha_over_sqrt_pi;
  const R cs = (R)prm.coul_scale;
  const R qi = pi.w;
  const int trow = prm.ntypes > 1 ? mi.x * prm.ntypes : 0;
  const int tmask = prm.ntypes > 1 ? ~0 : 0;
  const R margin = prm.orig ? (R)0 : (R)1.0e-4;
  const int4* nbr4 = reinterpret_cast<const int4*>(nbr) + i;
  const int nch = active ? (min(count[i], prm.cap) + 3) >> 2 : 0;
  const int last = __reduce_max_sync(0xffffffffu, nch);
  const int self = i << kShiftBits;
  const int4 idle = make_int4(self, self, self, self);
  Acc3<R> acc;
  R e_lj = 0, e_coul = 0;
  int4 e4 = sub < nch ? __ldg(nbr4 + (size_t)sub * prm.stride) : idle;
  for (int c = sub; c - sub < last; c += G) {
    const int ee[4] = {e4.x, e4.y, e4.z, e4.w};
    V4 pj[4];
    int2 mj[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) pj[k] = pos4[ee[k] >> kShiftBits];
    if (typed)
#pragma unroll
      for (int k = 0; k < 4; ++k) mj[k] = meta[ee[k] >> kShiftBits];
    e4 = c + G < nch ? __ldg(nbr4 + (size_t)(c + G) * prm.stride) : idle;
    if (__any_sync(0xffffffffu, ((ee[0] | ee[1] | ee[2] | ee[3]) & 63) != 0)) {   // p_j - PeriodicCoordOffset
      const R w0 = Traits<R>::wrap(rp, 0), w1 = Traits<R>::wrap(rp, 1), w2 = Traits<R>::wrap(rp, 2);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int k0 = ee[k] & 3, k1 = (ee[k] >> 2) & 3, k2 = (ee[k] >> 4) & 3;
        pj[k].x -= k0 == 1 ? w0 : (k0 == 2 ? -w0 : (R)0);
        pj[k].y -= k1 == 1 ? w1 : (k1 == 2 ? -w1 : (R)0);
        pj[k].z -= k2 == 1 ? w2 : (k2 == 2 ? -w2 : (R)0);
      }
    }
    Pair<R> gx2 = both<R>(0), gy2 = both<R>(0), gz2 = both<R>(0);
    unsigned bonded = 0;   // entries of the atom's own bond-graph component (SPW)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const V4 &pa = pj[2 * h], &pb = pj[2 * h + 1];
      const Pair<R> rx{pa.x - pi.x, pb.x - pi.x}, ry{pa.y - pi.y, pb.y - pi.y}, rz{pa.z - pi.z, pb.z - pi.z};
      const Pair<R> d2 = fma2(rz, rz, fma2(ry, ry, mul2(rx, rx)));
      // the list predicate at rc (list reuse); every listed pair passes it otherwise
      bool in[2] = {d2.x > (R)1.0e-4, d2.y > (R)1.0e-4};
      if ((MI & 3) == kMiAll) {
        in[0] = in[0] && cut2 - d2.x > margin;
        in[1] = in[1] && cut2 - d2.y > margin;
      }
      Pair<R> t = both<R>(0);
      if (COUL) {
        const Pair<R> qq{qi * pa.w, qi * pb.w};
        if (qq.x != (R)0 || qq.y != (R)0) {   // the term of a pair with q_i q_j = 0 is 0
          const Pair<R> inv{rsqrt_r(d2.x), rsqrt_r(d2.y)};
          const Pair<R> dis = mul2(d2, inv);
          const Pair<R> ex = exp_neg2(aa, d2);
          const Pair<R> erfcv = erfc_shared2(mul2(both<R>(sa), dis), ex);
          const Pair<R> qi2 = mul2(mul2(qq, inv), both<R>(cs));
          const Pair<R> g = mul2(fma2(erfcv, inv, mul2(both<R>(c2), ex)), inv);
          const Pair<R> f = mul2(qi2, g);
          const bool cx = ((MI & 3) != kMiAll || in[0]) && dis.x < rc && dis.x > (R)0.01;
          const bool cy = ((MI & 3) != kMiAll || in[1]) && dis.y < rc && dis.y > (R)0.01;
          t.x = cx ? -f.x : (R)0;
          t.y = cy ? -f.y : (R)0;
          if (ENERGY) e_coul += (cx ? qi2.x * erfcv.x : (R)0) + (cy ? qi2.y * erfcv.y : (R)0);
        }
      }
      Pair<R> qx = rx, qy = ry, qz = rz, l2 = d2;
      bool lj[2] = {in[0], in[1]};
      if ((MI & 3) == kMiLJ) {   // MinDistanceVec
        const R box[3] = {Traits<R>::box(rp, 0), Traits<R>::box(rp, 1), Traits<R>::box(rp, 2)};
        min_image(qx.x, qy.x, qz.x, box);
        min_image(qx.y, qy.y, qz.y, box);
        l2 = fma2(qz, qz, fma2(qy, qy, mul2(qx, qx)));
        lj[0] = l2.x > (R)1.0e-4;
        lj[1] = l2.y > (R)1.0e-4;
      }
      if ((MI & 3) != kMiAll) {
        lj[0] = lj[0] && l2.x < cut2;
        lj[1] = lj[1] && l2.y < cut2;
      }
      int tj[2] = {0, 0};
      if (typed) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const bool same = MOLEC && mj[2 * h + k].y == mi.y;
          tj[k] = mj[2 * h + k].x & tmask;
          if (SPW && same && ((MI & 3) != kMiAll || in[k])) bonded |= 1u << (2 * h + k);
          lj[k] = lj[k] && !same;
        }
      }
      const Pair<R> i2{rcp_r(l2.x), rcp_r(l2.y)};
      const Pair<R> sd6 = mul2(mul2(mul2(Pair<R>{lj_s6[trow + tj[0]], lj_s6[trow + tj[1]]}, i2), i2), i2);
      const Pair<R> a24{lj_a[trow + tj[0]], lj_a[trow + tj[1]]};
      Pair<R> sc = mul2(mul2(a24, mul2(fma2(both<R>(2), sd6, both<R>(-1)), sd6)), i2);
      sc.x = lj[0] ? sc.x : (R)0;
      sc.y = lj[1] ? sc.y : (R)0;
      if (ENERGY) {
        if (lj[0]) e_lj += -a24.x / (R)6 * (sd6.x - (R)1) * sd6.x;
        if (lj[1]) e_lj += -a24.y / (R)6 * (sd6.y - (R)1) * sd6.y;
      }
      if ((MI & 3) == kMiLJ) {
        gx2 = fma2(sc, qx, fma2(t, rx, gx2));
        gy2 = fma2(sc, qy, fma2(t, ry, gy2));
        gz2 = fma2(sc, qz, fma2(t, rz, gz2));
      } else {
        t = add2(t, sc);
        gx2 = fma2(t, rx, gx2);
        gy2 = fma2(t, ry, gy2);
        gz2 = fma2(t, rz, gz2);
      }
    }
    R gx = gx2.x + gx2.y, gy = gy2.x + gy2.y, gz = gz2.x + gz2.y;
    if (SPW) {
      // LJ of pairs inside the component, a dozen per atom, with the special-bond weight of the
      // pair: one copy of the partner search, outside the unrolled entries
      while (bonded) {
        const int b = __ffs(bonded) - 1;
        bonded &= bonded - 1;
        const int e = b & 2 ? (b & 1 ? ee[3] : ee[2]) : (b & 1 ? ee[1] : ee[0]);
        const int k0 = e & 3, k1 = (e >> 2) & 3, k2 = (e >> 4) & 3;
        const V4 q = pos4[e >> kShiftBits];
        R q0 = (k0 == 0 ? q.x : q.x - (k0 == 1 ? Traits<R>::wrap(rp, 0) : -Traits<R>::wrap(rp, 0))) - pi.x;
        R q1 = (k1 == 0 ? q.y : q.y - (k1 == 1 ? Traits<R>::wrap(rp, 1) : -Traits<R>::wrap(rp, 1))) - pi.y;
        R q2 = (k2 == 0 ? q.z : q.z - (k2 == 1 ? Traits<R>::wrap(rp, 2) : -Traits<R>::wrap(rp, 2))) - pi.z;
        if ((MI & 3) == kMiLJ) {
          const R box[3] = {Traits<R>::box(rp, 0), Traits<R>::box(rp, 1), Traits<R>::box(rp, 2)};
          min_image(q0, q1, q2, box);
        }
        const R dl2 = q0 * q0 + q1 * q1 + q2 * q2;
        if (dl2 < cut2 && dl2 > (R)0.0001) {
          const int tj = prm.ntypes > 1 ? meta[e >> kShiftBits].x : 0;
          const R wsp = special_weight<R>(prm.sp, slot_atom[i], slot_atom[e >> kShiftBits]);
          const R inv2 = rcp_r(dl2);
          const R sd6 = lj_s6[trow + tj] * inv2 * inv2 * inv2;
          const R a24 = lj_a[trow + tj];
          const R scal = a24 * (((R)2 * sd6 - (R)1) * sd6) * inv2 * wsp;
          gx += scal * q0;
          gy += scal * q1;
          gz += scal * q2;
          if (ENERGY) e_lj += wsp * (-a24 / (R)6 * (sd6 - (R)1) * sd6);
        }
      }
    }
    acc.add(gx, gy, gz);
  }
  double F[3] = {acc.vx(), acc.vy(), acc.vz()};
  double el = (double)e_lj, ec = (double)e_coul;
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    F[0] += __shfl_xor_sync(0xffffffffu, F[0], o);
    F[1] += __shfl_xor_sync(0xffffffffu, F[1], o);
    F[2] += __shfl_xor_sync(0xffffffffu, F[2], o);
    el += __shfl_xor_sync(0xffffffffu, el, o);
    ec += __shfl_xor_sync(0xffffffffu, ec, o);
  }
  if (!active || sub != 0) return;
  if (!isfinite(F[0]) || !isfinite(F[1]) || !isfinite(F[2])) set_flag(status, kFlagNonFinite);
  const int id = slot_atom[i];
  force[3 * id] = F[0];
  force[3 * id + 1] = F[1];
  force[3 * id + 2] = F[2];
  if (ENERGY) {
    energy_slot[2 * i] = 0.5 * el;
    energy_slot[2 * i + 1] = 0.5 * ec;
  }
}

// RBE k-space force, G lanes per charged atom (compact index c, caller id qidx[c]):
// F_i = q_i sum_l w_l k_l (cos(k_l.r_i) Im rho_l - sin(k_l.r_i) Re rho_l)
// (ComputeNewRBEForceWorklet, RunWorklet.cpp:1508-1548; S/P and qqr2e are folded into the
// records).  The block stages the k records of the replicas its atoms belong to in shared
// memory (two 16-byte broadcast loads per sample) when they fit.  Runs on the k-space stream
// concurrently with the near pass and writes far_force[c]; k_add_far folds it into the force.
// Bound by MUFU (two per term) when the chip is full; the lanes of an atom take every G-th sample and
// are summed in FP64 by a fixed butterfly, so that few charged atoms still fill it (launch_rbe_force):
// 25,000 charged atoms in FP64 37 -> 27 us.
constexpr int kRbeThreads = 128;

template <class R, int G>
__global__ void __launch_bounds__(kRbeThreads) k_rbe_force(int nq, int kstage, const int* __restrict__ qidx,
                                                   const typename FracT<R>::T* __restrict__ frac,
                                                   const typename KRec<R>::T* __restrict__ krec,
                                                   const RepDev* __restrict__ reps,
                                                   const int* __restrict__ rep_of,
                                                   double* __restrict__ far_force) {
  extern __shared__ __align__(16) unsigned char ksm_raw[];
  typename KRec<R>::T* ksm = reinterpret_cast<typename KRec<R>::T*>(ksm_raw);
  const int c0 = blockIdx.x * (kRbeThreads / G);
  const int sub = threadIdx.x % G;
  const int last = min(nq, c0 + kRbeThreads / G) - 1;
  const int c = min(c0 + (int)threadIdx.x / G, last);   // lanes past the end repeat the last atom
  const bool active = c0 + (int)threadIdx.x / G < nq;
  const int ra = rep_of ? rep_of[qidx[c0]] : 0;
  const int rb = rep_of ? rep_of[qidx[last]] : 0;
  const int kfirst = reps[ra].k_begin;
  const int kcount = reps[rb].k_begin + reps[rb].P - kfirst;
  const bool staged = kcount <= kstage;
  if (staged) {
    const int nwords = kcount * (int)(sizeof(typename KRec<R>::T) / 16);
    const int4* src = reinterpret_cast<const int4*>(krec + kfirst);
    int4* dst = reinterpret_cast<int4*>(ksm);
    for (int t = threadIdx.x; t < nwords; t += blockDim.x) dst[t] = src[t];
  }
  __syncthreads();
  const RepDev& rp = reps[rep_of ? rep_of[qidx[c]] : 0];
  const typename FracT<R>::T fr = frac[c];
  R ax = 0, ay = 0, az = 0;
  if (staged) rbe_terms<R, G>(fr, ksm + (rp.k_begin - kfirst), rp.P, sub, ax, ay, az);
  else rbe_terms<R, G>(fr, krec + rp.k_begin, rp.P, sub, ax, ay, az);
  double F[3] = {(double)ax, (double)ay, (double)az};
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) F[d] += __shfl_xor_sync(0xffffffffu, F[d], o);
  if (!active || sub != 0) return;
  const double q = (double)fr.q;
  far_force[3 * c] = q * F[0];
  far_force[3 * c + 1] = q * F[1];
  far_force[3 * c + 2] = q * F[2];
}

__global__ void k_add_far(int nq, const int* __restrict__ qidx, const double* __restrict__ far_force,
                          double* __restrict__ force, uint32_t* status) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * nq) return;
  const int c = t / 3, d = t - 3 * c;
  const int id = qidx[c];
  const double v = force[3 * id + d] + far_force[t];
  if (!isfinite(v)) set_flag(status, kFlagNonFinite);
  force[3 * id + d] = v;
}

// ------------------------------------------------------------------------------------------
// RBE structure factors, one k per lane.  Work item = (replica, atom chunk, k tile of
// 32*KL*warps samples).  Lane l of warp w owns samples w*32*KL + l + 32*j (j < KL): its m
// vector and (Re, Im) accumulators live in registers.  The block stages the chunk's atoms
// (fixed-point fractional coordinates + charge) in shared memory, 256 at a time, and every lane
// reads each staged atom by a broadcast load, so one 16-byte load serves 32*KL (atom, k) pairs.
// Each (item, k) partial is owned by one lane: no cross-lane reduction.  There is no N x P
// buffer (the reference materialises rho_Re/Im[P*N] and reduces by key, ExecutionMD.cpp:412-448).
// ------------------------------------------------------------------------------------------
// Per-replica reduction layout: items are ordered (replica, chunk, tile); replica r's partials
// for tile t and chunk c sit at item_base_r + c * ntiles_r + t.
struct RhoRep { int item_base, ntiles, nchunks, pad; };

// What a finished structure factor fills in.
template <class R> struct RhoOut {
  const double* weights;           // importance weights (nullable)
  double qqr2e;
  typename KRec<R>::T* krec;
  double2* rho;
  double* ek;
};

// Sample l of a replica from its summed partials: undo the half-turn phase convention (rho = -sum)
// and fill the force coefficients of the k record, rho, and the k-space energy estimate
// (S/P) qqr2e w_l (2 pi / V) |rho_l|^2 / k_l^2.
template <class R>
__device__ __forceinline__ void rho_record(const RepDev& rp, int l, double re, double im, const RhoOut<R>& o) {
  const int g = rp.k_begin + l;
  typename KRec<R>::T k = o.krec[g];
  re = -re;
  im = -im;
  const double twopi = 6.283185307179586476925;
  const double kx = twopi * k.mx / rp.box_d[0], ky = twopi * k.my / rp.box_d[1],
               kz = twopi * k.mz / rp.box_d[2];
  const double k2 = kx * kx + ky * ky + kz * kz;
  const double wgt = o.weights ? o.weights[g] : 1.0;
  // F_i = q_i (S/P) qqr2e sum_l wgt (-4 pi /(V k^2)) k (cos Im - sin Re); the kernel evaluates
  // the angle shifted by half a turn, which flips cos and sin: store -w.
  const double w0 = -(rp.S / rp.P) * o.qqr2e * wgt * (-4.0 * 3.14159265358979323846 / (rp.volume * k2));
  k.wx = (decltype(k.wx))(w0 * kx);
  k.wy = (decltype(k.wy))(w0 * ky);
  k.wz = (decltype(k.wz))(w0 * kz);
  k.re = (decltype(k.re))re;
  k.im = (decltype(k.im))im;
  o.krec[g] = k;
  o.rho[g] = make_double2(re, im);
  o.ek[g] = (rp.S / rp.P) * o.qqr2e * wgt * (2.0 * 3.14159265358979323846 / rp.volume) *
                (re * re + im * im) / k2;
}

struct RhoItem { int atom_begin, atom_end, k_first, k_count; };
constexpr int kRhoStage = 256;

// The fixed-point coordinates are formed while staging (k tile 0 also writes them for k_rbe_force).
// rep_done: with few chunks per replica the block that finishes a replica's last item sums its
// partials in chunk order and fills the records (kFusedChunks); otherwise k_rho_finish does.  Bound by
// MUFU (two per term) when the chip is full: 25,000 charged atoms in FP64 in chunks of 64 to 256
// atoms 67 -> 28 us against chunks of 1024; 1,600 charged atoms 25 us with k_frac and k_rho_finish as
// launches of their own, 16 us in one.
constexpr int kFusedChunks = 32;

template <class R, int KL>
__global__ void __launch_bounds__(256) k_rho_lanes(
    const RhoItem* __restrict__ items, int P, const int* __restrict__ qidx, const double* __restrict__ pos,
    const double* __restrict__ charge, const RepDev* __restrict__ reps, const RhoRep* __restrict__ rr,
    typename FracT<R>::T* __restrict__ frac, R* partial, int ktile, int* __restrict__ rep_done, RhoOut<R> o) {
  using FT = typename FracT<R>::T;
  __shared__ FT stage[kRhoStage];
  __shared__ int last;
  const RhoItem it = items[blockIdx.x];
  const int r = it.k_first / P;   // replicas hold P samples each
  const RepDev& rp = reps[r];
  const bool first_tile = it.k_first == rp.k_begin;
  const typename KRec<R>::T* krec = o.krec;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  using MT = typename std::conditional<sizeof(R) == 4, uint32_t, unsigned long long>::type;
  MT mx[KL], my[KL], mz[KL];
  R re[KL], im[KL];
  int kk[KL];
  bool any = false;
#pragma unroll
  for (int j = 0; j < KL; ++j) {
    kk[j] = w * 32 * KL + j * 32 + lane;
    const bool ok = kk[j] < it.k_count;
    any |= ok;
    const typename KRec<R>::T k = ok ? krec[it.k_first + kk[j]] : typename KRec<R>::T{};
    mx[j] = (MT)(long long)k.mx;
    my[j] = (MT)(long long)k.my;
    mz[j] = (MT)(long long)k.mz;
    re[j] = 0;
    im[j] = 0;
  }
  const bool warp_any = __any_sync(0xffffffffu, any);
  for (int base = it.atom_begin; base < it.atom_end; base += kRhoStage) {
    const int cnt = min(kRhoStage, it.atom_end - base);
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
      const FT f = frac_of<R>(rp, pos, charge, qidx[base + t]);
      stage[t] = f;
      if (first_tile) frac[base + t] = f;
    }
    __syncthreads();
    if (!warp_any) continue;
#pragma unroll 4
    for (int a = 0; a < cnt; ++a) {
      const FT f = stage[a];
#pragma unroll
      for (int j = 0; j < KL; ++j) {
        const MT ph = mx[j] * (MT)f.x + my[j] * (MT)f.y + mz[j] * (MT)f.z;
        R s, c;
        turn_sincos(ph, s, c);
        re[j] = fma((R)f.q, c, re[j]);
        im[j] = fma((R)f.q, s, im[j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < KL; ++j)
    if (kk[j] < it.k_count) {
      partial[((size_t)blockIdx.x * ktile + kk[j]) * 2] = re[j];
      partial[((size_t)blockIdx.x * ktile + kk[j]) * 2 + 1] = im[j];
    }
  if (!rep_done) return;
  __threadfence();   // the partials before the count
  __syncthreads();
  const RhoRep q = rr[r];
  if (threadIdx.x == 0) last = atomicAdd(rep_done + r, 1) == q.nchunks * q.ntiles - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();   // the count before the other blocks' partials
  for (int l = threadIdx.x; l < P; l += blockDim.x) {
    const int tile = l / ktile, k = l % ktile;
    double sr = 0, si = 0;
#pragma unroll 4
    for (int c = 0; c < q.nchunks; ++c) {
      const size_t at = (((size_t)q.item_base + (size_t)c * q.ntiles + tile) * ktile + k) * 2;
      sr += (double)__ldcg(partial + at);
      si += (double)__ldcg(partial + at + 1);
    }
    rho_record<R>(rp, l, sr, si, o);
  }
  if (threadIdx.x == 0) rep_done[r] = 0;
}

// Sum of the chunk partials of 32 consecutive k samples of one tile per block: lane = sample, so a
// warp reads 32 consecutive partials, warp w takes the chunks w, w + warps, .. (FP64) and the warps
// are added in order through shared memory (deterministic).
// (One warp per sample read one 8-byte partial per 32-byte sector: 12.5 us at 390 chunks of 305 samples,
// now 10.8.  Systems of up to kFusedChunks chunks per replica, such as batches of small replicas, have no
// launch of it.)
constexpr int kFinishWarps = 16;   // at most; the launch uses as many as the longest chunk list needs

template <class R>
__global__ void __launch_bounds__(32 * kFinishWarps) k_rho_finish(
    int nrep, int groups, int P, int ktile, const RhoRep* __restrict__ rr, const RepDev* __restrict__ reps,
    const R* __restrict__ partial, RhoOut<R> o) {
  __shared__ double sre[kFinishWarps][32], sim[kFinishWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int r = blockIdx.x / groups;               // groups = ceil(P / 32) blocks per replica
  const int l = (blockIdx.x % groups) * 32 + lane;
  const RepDev& rp = reps[r];
  const RhoRep q = rr[r];
  const int tile = l / ktile, kk = l % ktile;      // ktile is a multiple of 32: one tile per block
  double re = 0, im = 0;
  if (l < P) {
#pragma unroll 4
    for (int c = w; c < q.nchunks; c += nw) {
      const size_t at = (((size_t)q.item_base + (size_t)c * q.ntiles + tile) * ktile + kk) * 2;
      re += (double)partial[at];
      im += (double)partial[at + 1];
    }
  }
  sre[w][lane] = re;
  sim[w][lane] = im;
  __syncthreads();
  if (w != 0 || l >= P) return;
  for (int k = 1; k < nw; ++k) {
    re += sre[k][lane];
    im += sim[k][lane];
  }
  rho_record<R>(rp, l, re, im, o);
}

// ------------------------------------------------------------------------------------------
// RBE k-sampler: RBEPSAMPLE::Fetch_P_Sample + MH_Algorithm (rbmd/framework/model/
// RBEPSample.h:63-173) with mu = 0, sigma_d = sqrt(alpha/2) L_d / pi.  The MH ratio
// (P(m')/P(m)) (q(m)/q(m')) is G(m')/G(m) with G = exp(-pi^2 m^2/(alpha L^2)) / q(m) tabulated
// on the host (FP64); u <= min(1, ratio) is evaluated as u * G(m) <= G(m').
// One block per replica: phase 1 draws the Gaussian proposals, their G values and the
// acceptance uniforms of the first D steps in parallel (they do not depend on the chain);
// phase 2 resolves every per-axis chain state of those D steps in parallel (a step with
// u gmax <= G(m) accepts whatever the state, and the states between two such steps are replayed
// exactly), then assigns sample indices to the states that are not all zero (the all-zero retry
// of the reference couples the axes only there) with a block scan.  Steps past D, and windows
// holding a proposal beyond the tables, run the chain sequentially on one thread as the
// reference does.  Same k-sets as the sequential chain, bit for bit.
// ------------------------------------------------------------------------------------------
struct SamplerRep {
  double sigma[3];
  double gmax[3];   // largest finite G of each axis' table
  int qmax;
  int g_offset;     // offset of this replica's G tables (3 * (qmax+1) doubles)
};

__device__ __forceinline__ double sampler_draw(uint32_t k0, uint32_t k1, long long step, int rep,
                                               int axis, long long draw, double* ua) {
  uint32_t c[4] = {(uint32_t)draw, (uint32_t)axis | ((uint32_t)rep << 2), (uint32_t)(unsigned long long)step,
                   (uint32_t)((unsigned long long)step >> 32)};
  philox4x32(c, k0, k1);
  double U1 = ((double)c[0] + 0.5) * (1.0 / 4294967296.0);
  if (U1 < 1e-6) U1 = ((double)c[3] + 0.5) * (1.0 / 4294967296.0);
  if (U1 < 1e-6) U1 = 1e-6;
  const double U2 = ((double)c[1] + 0.5) * (1.0 / 4294967296.0);
  *ua = ((double)c[2] + 0.5) * (1.0 / 4294967296.0);
  return sqrt(-2.0 * log(U1)) * cos(2.0 * 3.14159265358979323846 * U2);
}

__device__ __forceinline__ double sampler_g(const double* g, int qmax, int axis, int m) {
  m = abs(m);
  return m <= qmax ? g[axis * (qmax + 1) + m] : __longlong_as_double(0x7ff0000000000000ll);
}

template <int D>
__global__ void __launch_bounds__(256) k_sample(int nrep, const SamplerRep* __restrict__ srep,
                                                const double* __restrict__ gtab,
                                                const RepDev* __restrict__ reps, unsigned long long seed,
                                                long long step_arg, const long long* __restrict__ step_dev,
                                                int* __restrict__ kvec_out,
                                                void* __restrict__ krec, int rec_bytes,
                                                int* __restrict__ krep, uint32_t* status) {
  const int r = blockIdx.x;
  if (r >= nrep) return;
  const long long step = step_dev ? *step_dev : step_arg;   // device counter under graph replay
  const SamplerRep s = srep[r];
  const int P = reps[r].P, kb = reps[r].k_begin;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  const double* g = gtab + s.g_offset;
  __shared__ int mw[3][D];
  __shared__ double ua[3][D];
  __shared__ double gw[3][D];
  for (int t = threadIdx.x; t < 3 * D; t += blockDim.x) {
    const int axis = t / D, d = t % D;
    double u;
    const double gs = sampler_draw(k0, k1, step, r, axis, d, &u);
    const int m = (int)round(s.sigma[axis] * gs);
    mw[axis][d] = m;
    ua[axis][d] = u;
    gw[axis][d] = sampler_g(g, s.qmax, axis, m);
  }
  __syncthreads();
  auto prop = [&](int axis, long long d, double* u, double* gm) -> int {
    if (d < D) { *u = ua[axis][d]; *gm = gw[axis][d]; return mw[axis][d]; }
    const double gs = sampler_draw(k0, k1, step, r, axis, d, u);
    const int m = (int)round(s.sigma[axis] * gs);
    *gm = sampler_g(g, s.qmax, axis, m);
    return m;
  };
  auto emit = [&](int i, const int* X) {
    int* o = kvec_out + 3 * (kb + i);
    o[0] = X[0]; o[1] = X[1]; o[2] = X[2];
    int* rec = reinterpret_cast<int*>(reinterpret_cast<char*>(krec) + (size_t)(kb + i) * rec_bytes);
    rec[0] = X[0]; rec[1] = X[1]; rec[2] = X[2];
    krep[kb + i] = r;
  };
  // first sample: the first draw that is not all zero (the reference's Fetch_P_Sample do-while)
  __shared__ int s_d0, s_x0[3], s_seq, s_total;
  __shared__ double s_g0[3];
  if (threadIdx.x == 0) {
    long long draw = 0;
    int X0[3];
    double G0[3];
    for (int guard = 0;; ++guard) {
      double u;
      for (int a = 0; a < 3; ++a) X0[a] = prop(a, draw, &u, &G0[a]);
      ++draw;
      if (!(X0[0] == 0 && X0[1] == 0 && X0[2] == 0)) break;
      if (guard > 100000) { set_flag(status, kFlagSampler); X0[0] = 1; G0[0] = sampler_g(g, s.qmax, 0, 1); break; }
    }
    emit(0, X0);
    s_d0 = (int)min(draw, (long long)D);
    for (int a = 0; a < 3; ++a) { s_x0[a] = X0[a]; s_g0[a] = G0[a]; }
    // the parallel chain below needs a non-empty window and every state in it with a finite G
    s_seq = draw >= D || !(isfinite(G0[0]) && isfinite(G0[1]) && isfinite(G0[2]));
    s_total = 1;
  }
  __syncthreads();
  const int d0 = s_d0;
  // The Metropolis-Hastings chain of each axis (MH_Algorithm, RBEPSample.h:63-85) is an
  // independence sampler: proposals do not depend on the state, and a step accepts when
  // u G(X_prev) <= G(m).  A step with u gmax <= G(m) accepts whatever the state (rounding is
  // monotonic, and every state of the window has G <= gmax), so each state is resolved in
  // parallel from the nearest such step before it, replaying the few steps in between exactly as
  // the sequential chain would.  Draws whose G is infinite (proposals past the table) fall back
  // to the sequential chain.
  int bad = 0;
  for (int t = threadIdx.x; t < 3 * (D - d0); t += blockDim.x) bad |= !isfinite(gw[t / (D - d0)][d0 + t % (D - d0)]);
  if (__syncthreads_or(bad) || s_seq) {
    if (threadIdx.x != 0) return;
    // sequential chain from the first sample (the reference's loop, Fetch_P_Sample:155-172)
    int X0[3] = {s_x0[0], s_x0[1], s_x0[2]};
    double G0[3] = {s_g0[0], s_g0[1], s_g0[2]};
    long long draw = d0;
    int i = 1;
    long long guard = 0;
    while (i < P) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        double u, gm;
        const int m_w = prop(a, draw, &u, &gm);
        if (u * G0[a] <= gm) { X0[a] = m_w; G0[a] = gm; }
      }
      ++draw;
      if (++guard > 64LL * P + 100000) { set_flag(status, kFlagSampler); break; }
      if (X0[0] == 0 && X0[1] == 0 && X0[2] == 0) continue;
      emit(i, X0);
      ++i;
    }
    return;
  }
  __shared__ int chain[3][D];
  for (int t = threadIdx.x; t < 3 * (D - d0); t += blockDim.x) {
    const int a = t / (D - d0), d = d0 + t % (D - d0);
    int sidx = d;
    while (sidx >= d0 && !(ua[a][sidx] * s.gmax[a] <= gw[a][sidx])) --sidx;
    int X;
    double G;
    if (sidx < d0) { X = s_x0[a]; G = s_g0[a]; sidx = d0 - 1; }
    else { X = mw[a][sidx]; G = gw[a][sidx]; }
    for (int k = sidx + 1; k <= d; ++k)
      if (ua[a][k] * G <= gw[a][k]) { X = mw[a][k]; G = gw[a][k]; }
    chain[a][d] = X;
  }
  __syncthreads();
  // emission: samples 1, 2, ... are the states of the draws that are not all zero, in draw order
  constexpr int kPer = (D + 255) / 256;
  const int base = d0 + threadIdx.x * kPer;
  int cnt = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int d = base + j;
    if (d < D && !(chain[0][d] == 0 && chain[1][d] == 0 && chain[2][d] == 0)) ++cnt;
  }
  // block exclusive scan of cnt (blockDim.x == 256)
  __shared__ int wsum[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  int off = 0;
  for (int w = 0; w < wid; ++w) off += wsum[w];
  int i = 1 + off + incl - cnt;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int d = base + j;
    if (d < D && !(chain[0][d] == 0 && chain[1][d] == 0 && chain[2][d] == 0)) {
      if (i < P) {
        const int X[3] = {chain[0][d], chain[1][d], chain[2][d]};
        emit(i, X);
      }
      ++i;
    }
  }
  if (threadIdx.x == 255) s_total = i;   // 1 + every non-zero state of the window
  __syncthreads();
  if (threadIdx.x != 0 || s_total >= P) return;
  // more samples than the window holds: continue the chain sequentially from its last state
  int X0[3] = {chain[0][D - 1], chain[1][D - 1], chain[2][D - 1]};
  double G0[3];
  for (int a = 0; a < 3; ++a) G0[a] = sampler_g(g, s.qmax, a, X0[a]);
  long long draw = D;
  int k = s_total;
  long long guard = D - d0;
  while (k < P) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double u, gm;
      const int m_w = prop(a, draw, &u, &gm);
      if (u * G0[a] <= gm) { X0[a] = m_w; G0[a] = gm; }
    }
    ++draw;
    if (++guard > 64LL * P + 100000) { set_flag(status, kFlagSampler); break; }
    if (X0[0] == 0 && X0[1] == 0 && X0[2] == 0) continue;
    emit(k, X0);
    ++k;
  }
}

// ------------------------------------------------------------------------------------------
// EAM passes (funcfl, 7-coefficient splines): pass 1 = ComputeEAMfpVerletWorklet
// (RunWorklet.cpp:305-359) -> fp[slot]; pass 2 = ComputeEAMForceVerletWorklet (:361-417).
// Spline rows are stored as two float4 (c0..c3, c4..c6,0).  MI: MinDistanceVec on the pair
// vector, needed only when a replica has fewer than 3 cells on an axis (otherwise the stored
// image shift already gives the nearest image, also under list reuse: the slot cache is
// unwrapped since the build).  FP32 uses r = rsq * rsqrt(rsq) and 1/r = rsqrt(rsq).
// ------------------------------------------------------------------------------------------
struct EamDev {
  const float4* rows;   // value rows (c3, c4, c5, c6) of rho(r) [nr + 1], then of z2(r) [nr + 1]
  const float4* frho;   // 2 float4 per row
  const float4* rhor;
  const float4* z2r;
  int nrho, nr;
  float rdr, rdrho;
  double rdr_d, rdrho_d;
  float rhomax;
};

template <class R, bool MI>
__global__ void __launch_bounds__(128) k_eam_fp(int n, int stride, int cap, double rc, EamDev eam,
                                                const typename Traits<R>::V4* __restrict__ pos4,
                                                const int* __restrict__ nbr, const int* __restrict__ count,
                                                const RepDev* __restrict__ reps,
                                                const int* __restrict__ rep_of_slot, R* __restrict__ fp,
                                                double* __restrict__ embed_slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
  const typename Traits<R>::V4 pi = pos4[i];
  const R wrap[3] = {Traits<R>::wrap(rp, 0), Traits<R>::wrap(rp, 1), Traits<R>::wrap(rp, 2)};
  const R box[3] = {Traits<R>::box(rp, 0), Traits<R>::box(rp, 1), Traits<R>::box(rp, 2)};
  const R ibox[3] = {(R)1 / box[0], (R)1 / box[1], (R)1 / box[2]};
  const R cut2 = (R)rc * (R)rc;
  const R rdr = sizeof(R) == 4 ? (R)eam.rdr : (R)eam.rdr_d;
  Acc<R> rho;
  const int cnt = min(count[i], cap);
  for (int p = 0; p < cnt; ++p) {
    const int e = __ldg(nbr + nbr_at(p, i, stride));
    const int j = e >> kShiftBits;
    const typename Traits<R>::V4 pj = pos4[j];
    R r[3];
    const R pjv[3] = {pj.x, pj.y, pj.z}, piv[3] = {pi.x, pi.y, pi.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int cd = (e >> (2 * d)) & 3;
      const R off = cd == 1 ? wrap[d] : (cd == 2 ? -wrap[d] : (R)0);
      R v = piv[d] - (pjv[d] - off);
      if (MI) v -= box[d] * rint(v * ibox[d]);   // MinDistanceVec
      r[d] = v;
    }
    const R rsq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (rsq < cut2 && rsq > (R)0.01) {
      R pp = rsq * rsqrt_r(rsq) * rdr + (R)1;
      int m = (int)pp;
      m = min(m, eam.nr - 1);
      pp -= (R)m;
      pp = fmin(pp, (R)1);
      const float4 b = __ldg(eam.rhor + 2 * m + 0);
      const float4 c = __ldg(eam.rhor + 2 * m + 1);
      rho.add((((R)b.w * pp + (R)c.x) * pp + (R)c.y) * pp + (R)c.z);
    }
  }
  const R rr = (R)rho.value();
  R pp = rr * (sizeof(R) == 4 ? (R)eam.rdrho : (R)eam.rdrho_d) + (R)1;
  int m = (int)pp;
  m = max(1, min(m, eam.nrho - 1));
  pp -= (R)m;
  pp = fmin(pp, (R)1);
  const float4 a = __ldg(eam.frho + 2 * m + 0);
  const float4 b = __ldg(eam.frho + 2 * m + 1);
  fp[i] = ((R)a.x * pp + (R)a.y) * pp + (R)a.z;
  if (embed_slot) {
    double phi = (((double)a.w * pp + (double)b.x) * pp + (double)b.y) * pp + (double)b.z;
    if ((double)rr > eam.rhomax) phi += (double)fp[i] * ((double)rr - eam.rhomax);
    embed_slot[i] = phi;
  }
}

template <class R, bool MI>
__global__ void __launch_bounds__(128) k_eam_force(int n, int stride, int cap, double rc, EamDev eam,
                                                   const typename Traits<R>::V4* __restrict__ pos4,
                                                   const int* __restrict__ nbr, const int* __restrict__ count,
                                                   const RepDev* __restrict__ reps,
                                                   const int* __restrict__ rep_of_slot,
                                                   const R* __restrict__ fp, const int* __restrict__ slot_atom,
                                                   double* __restrict__ force, double* __restrict__ pair_slot,
                                                   uint32_t* status, int ref_sign) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
  const typename Traits<R>::V4 pi = pos4[i];
  const R wrap[3] = {Traits<R>::wrap(rp, 0), Traits<R>::wrap(rp, 1), Traits<R>::wrap(rp, 2)};
  const R box[3] = {Traits<R>::box(rp, 0), Traits<R>::box(rp, 1), Traits<R>::box(rp, 2)};
  const R ibox[3] = {(R)1 / box[0], (R)1 / box[1], (R)1 / box[2]};
  const R cut2 = (R)rc * (R)rc;
  const R rdr = sizeof(R) == 4 ? (R)eam.rdr : (R)eam.rdr_d;
  const R fpi = fp[i];
  Acc<R> fx, fy, fz;
  R epair = 0;
  const int cnt = min(count[i], cap);
  for (int p = 0; p < cnt; ++p) {
    const int e = __ldg(nbr + nbr_at(p, i, stride));
    const int j = e >> kShiftBits;
    const typename Traits<R>::V4 pj = pos4[j];
    R r[3];
    const R pjv[3] = {pj.x, pj.y, pj.z}, piv[3] = {pi.x, pi.y, pi.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int cd = (e >> (2 * d)) & 3;
      const R off = cd == 1 ? wrap[d] : (cd == 2 ? -wrap[d] : (R)0);
      // pair vector p_i - p_j' (the sign for which F = -grad E, as LAMMPS' pair_eam and the
      // reference's RBL pass, RunWorklet.cpp:1180); ref_sign: the reference's Verlet pass uses
      // MinDistanceVec(p_j, p_i) (RunWorklet.cpp:402), which reverses the force
      R v = ref_sign ? (pjv[d] - off) - piv[d] : piv[d] - (pjv[d] - off);
      if (MI) v -= box[d] * rint(v * ibox[d]);
      r[d] = v;
    }
    const R rsq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (rsq < cut2 && rsq > (R)0.01) {
      const R recip = rsqrt_r(rsq);
      const R rv = rsq * recip;
      R pp = rv * rdr + (R)1;
      int m = (int)pp;
      m = min(m, eam.nr - 1);
      pp -= (R)m;
      pp = fmin(pp, (R)1);
      const float4 ra = __ldg(eam.rhor + 2 * m + 0);
      const float4 za = __ldg(eam.z2r + 2 * m + 0);
      const float4 zb = __ldg(eam.z2r + 2 * m + 1);
      const R rhop = ((R)ra.x * pp + (R)ra.y) * pp + (R)ra.z;
      const R z2p = ((R)za.x * pp + (R)za.y) * pp + (R)za.z;
      const R z2 = (((R)za.w * pp + (R)zb.x) * pp + (R)zb.y) * pp + (R)zb.z;
      const R phi = z2 * recip;
      const R phip = z2p * recip - phi * recip;
      const R psip = fpi * rhop + fp[j] * rhop + phip;
      const R fpair = -psip * recip;
      fx.add(r[0] * fpair);
      fy.add(r[1] * fpair);
      fz.add(r[2] * fpair);
      epair += phi;
    }
  }
  const double F[3] = {fx.value(), fy.value(), fz.value()};
  if (!isfinite(F[0]) || !isfinite(F[1]) || !isfinite(F[2])) set_flag(status, kFlagNonFinite);
  const int id = slot_atom[i];
  force[3 * id] = F[0];
  force[3 * id + 1] = F[1];
  force[3 * id + 2] = F[2];
  if (pair_slot) pair_slot[i] = 0.5 * (double)epair;
}

// EAM passes in FP32 with the spline tables in shared memory, for tables whose value rows fit
// (launch_eam).  The per-pair work is a gather of 16-byte spline rows at random indexes: from L1 it
// takes a tag lookup per lane, from shared memory about 11 cycles a warp, so one block per SM copies
// the rows once and walks the atoms.  Rows hold the value polynomial alone, (c3, c4, c5, c6) of
// rho(r) and of z2(r): the derivative is (3 c3 p^2 + 2 c4 p + c5) / dr, which the seven-coefficient
// rows store rounded (their c0..c2).  G lanes per atom share a row of the list, lane s taking the
// chunks s, s + G, .. of four entries (the last chunk is filled with the slot itself, which the
// predicate 0.01 < r^2 < rc^2 refuses); each term goes into a two-float accumulator, the lanes'
// sums are combined in FP64 by a fixed butterfly.  Pass 1 also writes (x, y, z, F'(rho)) per slot, so
// that pass 2 needs one gather per neighbour.  Bound by issue and the gathers: 256,000 atoms at 4 lanes
// 80 + 165 -> 66 + 85 us (1 and 2 lanes: the step 1.5 and 1 % longer).  Pair physics as k_eam_fp and
// k_eam_force.
constexpr int kEamThreads = 1024;

template <bool MI>
__device__ __forceinline__ void eam_vec(const float4& pi, const float4& pj, int e, const float* wrap, const float* box,
                                        const float* ibox, float* r) {
  r[0] = pj.x;
  r[1] = pj.y;
  r[2] = pj.z;
  if ((e & 63) != 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int cd = (e >> (2 * d)) & 3;
      r[d] -= cd == 1 ? wrap[d] : (cd == 2 ? -wrap[d] : 0.f);
    }
  }
  r[0] = pi.x - r[0];
  r[1] = pi.y - r[1];
  r[2] = pi.z - r[2];
  if (MI) {   // MinDistanceVec
#pragma unroll
    for (int d = 0; d < 3; ++d) r[d] -= box[d] * rint(r[d] * ibox[d]);
  }
}

// spline row and offset of distance r; row 0 (for a NaN of the filler entries) exists
__device__ __forceinline__ int eam_row(float r, float rdr, int nr, float& p) {
  const float pp = r * rdr + 1.0f;
  const int m = max(0, min((int)pp, nr - 1));
  p = fminf(pp - (float)m, 1.0f);
  return m;
}

template <bool MI, int G>
__global__ void __launch_bounds__(kEamThreads, 1) k_eam_fp_smem(
    int n, int stride, int cap, float rc, EamDev eam, const float4* __restrict__ pos4, const int4* __restrict__ nbr4,
    const int* __restrict__ count, const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot,
    float4* __restrict__ posf, double* __restrict__ embed_slot) {
  extern __shared__ float4 eam_tab[];
  for (int t = threadIdx.x; t <= eam.nr; t += blockDim.x) eam_tab[t] = eam.rows[t];
  __syncthreads();
  const int sub = threadIdx.x % G;
  const float cut2 = rc * rc;
  for (long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x; (at & ~31LL) < (long long)n * G;
       at += (long long)gridDim.x * blockDim.x) {
    const bool active = at / G < n;
    const int i = active ? (int)(at / G) : n - 1;
    const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
    const float4 pi = pos4[i];
    const float box[3] = {rp.box_f[0], rp.box_f[1], rp.box_f[2]};
    const float ibox[3] = {1.f / box[0], 1.f / box[1], 1.f / box[2]};
    const int nch = active ? (min(count[i], cap) + 3) >> 2 : 0;
    const int last = __reduce_max_sync(0xffffffffu, nch);
    const int self = i << kShiftBits;
    const int4 idle = make_int4(self, self, self, self);
    Acc<float> rho;
    int4 e = sub < nch ? __ldg(nbr4 + (size_t)sub * stride + i) : idle;
    for (int c = sub; c - sub < last; c += G) {
      const int ee[4] = {e.x, e.y, e.z, e.w};
      float4 pj[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) pj[k] = pos4[ee[k] >> kShiftBits];
      e = c + G < nch ? __ldg(nbr4 + (size_t)(c + G) * stride + i) : idle;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float r[3], p;
        eam_vec<MI>(pi, pj[k], ee[k], rp.wrap_f, box, ibox, r);
        const float rsq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
        const bool in = rsq < cut2 && rsq > 0.01f;
        const float4 a = eam_tab[eam_row(rsq * rsqrt_r(rsq), eam.rdr, eam.nr, p)];
        rho.add(in ? ((a.x * p + a.y) * p + a.z) * p + a.w : 0.f);
      }
    }
    double sum = rho.value();
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (!active || sub != 0) continue;
    const float rr = (float)sum;
    float pp = rr * eam.rdrho + 1.0f;
    const int m = max(1, min((int)pp, eam.nrho - 1));
    pp = fminf(pp - (float)m, 1.0f);
    const float4 a = __ldg(eam.frho + 2 * m + 0), b = __ldg(eam.frho + 2 * m + 1);
    const float fp = (a.x * pp + a.y) * pp + a.z;
    posf[i] = make_float4(pi.x, pi.y, pi.z, fp);
    double phi = (((double)a.w * pp + (double)b.x) * pp + (double)b.y) * pp + (double)b.z;
    if ((double)rr > eam.rhomax) phi += (double)fp * ((double)rr - eam.rhomax);
    embed_slot[i] = phi;
  }
}

template <bool MI, int G>
__global__ void __launch_bounds__(kEamThreads, 1) k_eam_force_smem(
    int n, int stride, int cap, float rc, EamDev eam, const float4* __restrict__ posf, const int4* __restrict__ nbr4,
    const int* __restrict__ count, const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot,
    const int* __restrict__ slot_atom, double* __restrict__ force, double* __restrict__ pair_slot, uint32_t* status,
    int ref_sign) {
  extern __shared__ float4 eam_tab[];   // rows of rho, then of z2
  for (int t = threadIdx.x; t < 2 * (eam.nr + 1); t += blockDim.x) eam_tab[t] = eam.rows[t];
  __syncthreads();
  const float4* ztab = eam_tab + eam.nr + 1;
  const int sub = threadIdx.x % G;
  const float cut2 = rc * rc;
  // ref_sign: the reference's Verlet pass uses MinDistanceVec(p_j, p_i) (RunWorklet.cpp:402)
  const float sgn = ref_sign ? 1.f : -1.f;
  for (long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x; (at & ~31LL) < (long long)n * G;
       at += (long long)gridDim.x * blockDim.x) {
    const bool active = at / G < n;
    const int i = active ? (int)(at / G) : n - 1;
    const RepDev& rp = reps[rep_of_slot ? rep_of_slot[i] : 0];
    const float4 pi = posf[i];
    const float box[3] = {rp.box_f[0], rp.box_f[1], rp.box_f[2]};
    const float ibox[3] = {1.f / box[0], 1.f / box[1], 1.f / box[2]};
    const int nch = active ? (min(count[i], cap) + 3) >> 2 : 0;
    const int last = __reduce_max_sync(0xffffffffu, nch);
    const int self = i << kShiftBits;
    const int4 idle = make_int4(self, self, self, self);
    Acc3<float> F;
    float epair = 0.f;
    int4 e = sub < nch ? __ldg(nbr4 + (size_t)sub * stride + i) : idle;
    for (int c = sub; c - sub < last; c += G) {
      const int ee[4] = {e.x, e.y, e.z, e.w};
      float4 pj[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) pj[k] = posf[ee[k] >> kShiftBits];
      e = c + G < nch ? __ldg(nbr4 + (size_t)(c + G) * stride + i) : idle;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float r[3], p;
        eam_vec<MI>(pi, pj[k], ee[k], rp.wrap_f, box, ibox, r);
        const float rsq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
        const bool in = rsq < cut2 && rsq > 0.01f;
        const float recip = rsqrt_r(rsq);
        const int m = eam_row(rsq * recip, eam.rdr, eam.nr, p);
        const float4 a = eam_tab[m], z = ztab[m];
        const float rhop = (((a.x * 3.f) * p + (a.y + a.y)) * p + a.z) * eam.rdr;
        const float z2p = (((z.x * 3.f) * p + (z.y + z.y)) * p + z.z) * eam.rdr;
        const float z2 = ((z.x * p + z.y) * p + z.z) * p + z.w;
        const float phi = z2 * recip;
        const float phip = z2p * recip - phi * recip;
        const float psip = pi.w * rhop + pj[k].w * rhop + phip;
        const float fpair = in ? sgn * psip * recip : 0.f;
        F.add(r[0] * fpair, r[1] * fpair, r[2] * fpair);
        epair += in ? phi : 0.f;
      }
    }
    double Fd[3] = {F.vx(), F.vy(), F.vz()}, ep = (double)epair;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      Fd[0] += __shfl_xor_sync(0xffffffffu, Fd[0], o);
      Fd[1] += __shfl_xor_sync(0xffffffffu, Fd[1], o);
      Fd[2] += __shfl_xor_sync(0xffffffffu, Fd[2], o);
      ep += __shfl_xor_sync(0xffffffffu, ep, o);
    }
    if (!active || sub != 0) continue;
    if (!isfinite(Fd[0]) || !isfinite(Fd[1]) || !isfinite(Fd[2])) set_flag(status, kFlagNonFinite);
    const int id = slot_atom[i];
    force[3 * id] = Fd[0];
    force[3 * id + 1] = Fd[1];
    force[3 * id + 2] = Fd[2];
    pair_slot[i] = 0.5 * ep;
  }
}

}  // namespace rbmd
