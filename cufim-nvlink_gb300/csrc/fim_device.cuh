// fim_device.cuh -- device arithmetic shared by the kernels of the GB300 FIM
// solver: exact float/double conversions, the reference's local solvers in
// FP64 (solve_tri_cu / solve_tet_cu, cuda_fim.h:1256-1360) and the tet prefix
// program, the corner relabelling, fp16 bound packing and the bounded grid
// barrier.  Included by every CUDA translation unit of the solver; all of
// them are compiled with -fmad=false (see fim_kernels.cu).
#pragma once

#include "fim_internal.h"
#include "fim_filter.cuh"

#include <cfloat>
#include <cstdint>
#include <cuda_fp16.h>

namespace fimgb {

#define FIM_INF DBL_MAX
#define FULL_MASK 0xffffffffu

// ---------------------------------------------------------------------------
// local solver, FP64 with the reference's float-typed triangle intermediates

// Exact float <-> double conversions and FP64 sign tests from the bit
// patterns (IEEE 754 binary32 / binary64), on the integer pipes: on GB300 a
// conversion or an FP64 comparison occupies the FP64 pipe like an FP64
// multiply.  Operands outside the normal range take the hardware
// instruction.

// (double)f, exact
__device__ __forceinline__ double f2d(float f)
{
  const uint32_t u = __float_as_uint(f);
  const uint32_t e = (u >> 23) & 0xffu;
  if (e - 1u < 254u)  // normal: rebias the exponent, widen the fraction
    return __longlong_as_double((long long)(((unsigned long long)(u & 0x80000000u) << 32) |
                                            ((unsigned long long)(e + 896u) << 52) |
                                            ((unsigned long long)(u & 0x7fffffu) << 29)));
  return (double)f;  // zero, subnormal, infinity, NaN
}

// (float)x, round to nearest, ties to even
__device__ __forceinline__ float d2f(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
  if (e - 897u < 254u) {  // the float is normal, or rounds up to infinity
    const uint32_t frac = (uint32_t)(b >> 29) & 0x7fffffu;
    const uint32_t rest = (uint32_t)b & 0x1fffffffu;  // the 29 bits dropped
    uint32_t r = ((e - 896u) << 23) | frac;
    r += (rest > 0x10000000u || (rest == 0x10000000u && (frac & 1u))) ? 1u : 0u;  // carries into the exponent
    return __uint_as_float(r | ((uint32_t)(b >> 32) & 0x80000000u));
  }
  return (float)x;  // zero, subnormal result, infinity, NaN
}

// (float)(x * 2^-s) for |s| <= 60, round to nearest, ties to even: the
// scaling is an exponent change, exact whenever the scaled double is normal
__device__ __forceinline__ float d2f_pow2(double x, int s)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ffu);
  const int es = e - s;  // biased exponent of x * 2^-s
  if (e != 0 && e != 0x7ff && (uint32_t)(es - 897) < 254u) {
    const uint32_t frac = (uint32_t)(b >> 29) & 0x7fffffu;
    const uint32_t rest = (uint32_t)b & 0x1fffffffu;
    uint32_t r = ((uint32_t)(es - 896) << 23) | frac;
    r += (rest > 0x10000000u || (rest == 0x10000000u && (frac & 1u))) ? 1u : 0u;
    return __uint_as_float(r | ((uint32_t)(b >> 32) & 0x80000000u));
  }
  return (float)(x * ldexp(1.0, -s));
}

// The float copy of a time: rounded to nearest, +inf only for FIM_INF (a
// larger finite time than a float holds gives NaN, "ask the FP64 time"), so
// that a vertex without a time shows by its copy alone.
__device__ __forceinline__ float time_f(double x)
{
  const float f = (float)x;
  return f == INFINITY && x < FIM_INF ? __int_as_float(0x7fffffff) : f;
}

// x > 0 (false for zeros and NaN)
__device__ __forceinline__ bool dgt0(double x)
{
  return (unsigned long long)__double_as_longlong(x) - 1ull < 0x7ff0000000000000ull;
}
// 0 < x < 1
__device__ __forceinline__ bool din01(double x)
{
  return (unsigned long long)__double_as_longlong(x) - 1ull < 0x3fefffffffffffffull;
}
// 0 < x < inf (false for NaN)
__device__ __forceinline__ bool dpos_finite(double x)
{
  return (unsigned long long)__double_as_longlong(x) - 1ull < 0x7fefffffffffffffull;
}
// x finite (not inf, not NaN)
__device__ __forceinline__ bool dfinite(double x)
{
  return ((unsigned long long)__double_as_longlong(x) & 0x7ff0000000000000ull) != 0x7ff0000000000000ull;
}
// x < 0 (false for zeros and NaN)
__device__ __forceinline__ bool dlt0(double x)
{
  return (unsigned long long)__double_as_longlong(x) - 0x8000000000000001ull < 0x7ff0000000000000ull;
}

// solve_tri_cu, cuda_fim.h:1256-1300
__device__ __forceinline__ double tri_ref(double e12, double e13, double e23, double p1, double p2)
{
  const double a = e23;
  const double b = -0.5 * (e12 + e23 - e13);
  const double c = e12;
  const double p12 = p2 - p1;
  // the reference's float casts as d2f / f2d (same values)
  float dv = d2f(p12 * p12 - c);
  const float sv = d2f(f2d(dv) * (b * b - a * c));
  // the reference compares the float intermediates after widening them to
  // double; comparing the floats themselves gives the same answers (NaN too)
  // without the FP64 conversions
  if (dv != 0.f && sv >= 0.f) {
    dv = d2f(c * f2d(dv));
    const float st = sqrtf(sv);
    const double dst = f2d(st), ddv = f2d(dv);
    const float l1 = d2f(-(b * p12 * p12 - b * c - dst * p12) / ddv);
    const float l2 = d2f(-(b * p12 * p12 - b * c + dst * p12) / ddv);
    const double dl1 = f2d(l1), dl2 = f2d(l2);
    float r1 = d2f(p2 - dl1 * p12 + sqrt(a + 2.0 * dl1 * b + f2d(l1 * l1) * c));
    if (!((l1 >= 0.f) && (l1 <= 1.f))) r1 = (float)FIM_INF;
    float r2 = d2f(p2 - dl2 * p12 + sqrt(a + 2.0 * dl2 * b + f2d(l2 * l2) * c));
    if (!((l2 >= 0.f) && (l2 <= 1.f))) r2 = (float)FIM_INF;
    return f2d(fminf(r1, r2));
  }
  return FIM_INF;
}

// tri_ref again, its two roots separately and without FP64 divisions and
// square roots.  Both only ever reach the result rounded to float -- l is a
// float, and so is the sum that holds the square root -- and a float is
// decided by an approximation good to 2^-40 unless that lies next to a
// rounding boundary.  On GB300 the FP64 pipe takes 64 cycles per warp
// instruction, and a division or square root is nine or ten of them: tri_ref
// issues about 73 FP64 instructions for its two roots, this 38.
//   l: q = N / D by the FP32 division (2^-21 relative), its residual
//      N - q D exactly by one FP64 fma (D is a float), the correction by
//      another FP32 division: q + dl is off by less than 2^-43 |l|.
//   sum: s0 = sqrt(Q) by the FP32 reciprocal square root (2^-21), its
//      residual Q - s0^2 exactly by one FP64 fma, the correction linear:
//      s0 + d0 is off by less than 2^-42 s0; added to p2 - l p12 in FP64.
// Where the float is not decided, or an operand is far from 1 (where the
// bounds above could meet subnormals), tri_root_ref evaluates the root as
// the reference does.
//
// The conversions are plain shifts of the bit patterns, without branches:
// every operand whose exponent they cannot take raises `odd`, which also
// ends in tri_root_ref.  One warp, both roots: tri_ref 3.40 us, this 2.40 us
// (0.88 us up to the roots, 0.76 us each); 3.55 us with conversions that
// branch to the hardware's for zeros and subnormals.
__device__ __forceinline__ uint32_t dhi(double x) { return (uint32_t)__double2hiint(x); }
// (double)f for a normal f (zero becomes 2^-127)
__device__ __forceinline__ double f2d_normal(float f)
{
  const uint32_t u = __float_as_uint(f);
  return __hiloint2double((int)(((u & 0x7fffffffu) >> 3) + 0x38000000u | (u & 0x80000000u)), (int)(u << 29));
}
// whether x lies in [2^-126, 2^127) by magnitude
__device__ __forceinline__ bool d_float_range(double x) { return (dhi(x) & 0x7fffffffu) - 0x38100000u < 0x0fd00000u; }
// (float)x rounded to nearest (ties to even), for d_float_range(x)
__device__ __forceinline__ float d2f_normal(double x)
{
  const uint32_t hi = dhi(x), lo = (uint32_t)__double2loint(x);
  uint32_t r = __funnelshift_l(lo, (hi & 0x7fffffffu) - 0x38000000u, 3);
  r += (lo & 0x1fffffffu) + (r & 1u) > 0x10000000u ? 1u : 0u;
  return __uint_as_float(r | (hi & 0x80000000u));
}
// x truncated to a float, for d_float_range(x); 0 below it
__device__ __forceinline__ float d2f_trunc(double x)
{
  const uint32_t hi = dhi(x), m = hi & 0x7fffffffu;
  const uint32_t r = __funnelshift_l((uint32_t)__double2loint(x), m - 0x38000000u, 3);
  return __uint_as_float(m < 0x38100000u ? 0u : r | (hi & 0x80000000u));
}

struct TriPre {
  double a, b, c, p2, p12, bpc, stp;
  float dv;
  bool odd;
};

// The floats of an odd triangle, by the conversions that take everything
// (out of line: rare).
static __device__ __noinline__ void tri_odd(double dvd, double gram, double c, float &dv, float &sv, float &ddv)
{
  dv = d2f(dvd);
  sv = d2f(f2d(dv) * gram);
  ddv = d2f(c * f2d(dv));
}

// false: no root has a value
__device__ __forceinline__ bool tri_prepare(double e12, double e13, double e23, double p1, double p2, TriPre &t)
{
  t.a = e23;
  t.b = -0.5 * (e12 + e23 - e13);
  t.c = e12;
  t.p2 = p2;
  t.p12 = p2 - p1;
  const double dvd = t.p12 * t.p12 - t.c;
  float dv = d2f_normal(dvd);
  const double gram = t.b * t.b - t.a * t.c;
  double svd = f2d_normal(dv) * gram;
  float sv = d2f_normal(svd);
  double dd = t.c * f2d_normal(dv);
  t.dv = d2f_normal(dd);
  t.odd = !(d_float_range(dvd) && d_float_range(svd) && d_float_range(dd));
  if (t.odd) tri_odd(dvd, gram, t.c, dv, sv, t.dv);
  if (!(dv != 0.f && sv >= 0.f)) return false;
  t.bpc = t.b * t.p12 * t.p12 - t.b * t.c;
  const float st = sqrtf(sv);
  double sd = f2d_normal(st);
  if (t.odd) sd = (double)st;
  t.stp = sd * t.p12;
  return true;
}

static __device__ __noinline__ double tri_root_ref(double a, double b, double c, double p2, double p12, double n, float dv)
{
  const float l = d2f(n / f2d(dv));
  if (!((l >= 0.f) && (l <= 1.f))) return FIM_INF;
  const double ld = f2d(l);
  return f2d(d2f(p2 - ld * p12 + sqrt(a + 2.0 * ld * b + f2d(l * l) * c)));
}

__device__ __forceinline__ bool mid_range(float x) { return fabsf(x) >= 0x1p-60f && fabsf(x) <= 0x1p60f; }

// Root 1 or 2 of the triangle solve: FIM_INF (or NaN) when it has no value.
__device__ __forceinline__ double tri_root(const TriPre &t, bool second)
{
  const double n = -(t.bpc + (second ? t.stp : -t.stp));
  const float nf = d2f_trunc(n);
  const float q = __fdividef(nf, t.dv);
  const float dl = __fdividef(d2f_trunc(fma(-f2d_normal(q), f2d_normal(t.dv), n)), t.dv);
  const float l = q + dl, lr = dl - (l - q), lerr = fabsf(l) * 0x1p-42f;  // q + dl == l + lr
  bool sure = !t.odd && mid_range(t.dv) && mid_range(nf) && fabsf(q) >= 0x1p-40f && fabsf(q) <= 0x1p40f &&
              l + (lr + lerr) == l && l + (lr - lerr) == l;
  if (sure) {
    if (!((l >= 0.f) && (l <= 1.f))) return FIM_INF;
    const double ld = f2d_normal(l), l2 = __hiloint2double((int)(dhi(ld) + 0x00100000u), __double2loint(ld));  // 2 l
    const double qd = t.a + l2 * t.b + f2d_normal(l * l) * t.c;
    const float x = d2f_trunc(qd);
    const float rs = rsqrtf(x), s0 = x * rs;
    const double s0d = f2d_normal(s0);
    const float d0 = d2f_trunc(fma(-s0d, s0d, qd)) * 0.5f * rs;
    const double w = t.p2 - ld * t.p12 + s0d + f2d_normal(d0);
    // (float)w with 2^14 of the FP64 units in the last place to spare on
    // both sides of the rounding boundary: 2^-40 |w| and more while s0 is at
    // most 4 |w|
    const uint32_t hi = dhi(w), lo = (uint32_t)__double2loint(w), rest = lo & 0x1fffffffu;
    const uint32_t r = __funnelshift_l(lo, (hi & 0x7fffffffu) - 0x38000000u, 3) + (rest > 0x10000000u ? 1u : 0u);
    const float rf = __uint_as_float(r | (hi & 0x80000000u));
    sure = x >= 0x1p-60f && x <= 0x1p60f && d_float_range(w) && rest - (0x10000000u - 0x4000u) > 0x8000u &&
           s0 <= 4.f * fabsf(rf);
    if (sure) return f2d_normal(rf);
  }
  return tri_root_ref(t.a, t.b, t.c, t.p2, t.p12, n, t.dv);
}

// solve_tet_cu, cuda_fim.h:1302-1360 (the reference's closed form, term for term)
__device__ __forceinline__ double tet_ref(double e13, double e23, double e34, double e12, double e14,
                                          double e24, double p1, double p2, double p3)
{
  const double a = e13;
  const double b = 0.5 * (e23 + e13 - e12);
  const double c = -0.5 * (e34 + e13 - e14);
  const double d = e23;
  const double e = -0.5 * (e34 + e23 - e24);
  const double f = e34;
  const double q13 = p3 - p1;
  const double q23 = p3 - p2;

  const double sqt =
    -e*e*c*d*d + a*d*d*d*d - (b*b*c - a*c*c)*f*f + ((b*b - a*c)*f*f -
    (e*e*c - a*d*d - 2.*(e*c - b*d)*e)*f)*q13*q13 - 2.*(e*e*c*d -
    2.*e*b*d*d + a*d*d*d + (b*b - a*c)*d*f)*q13*q23 + (e*e*c*c -
    2.*e*b*c*d + a*c*d*d + (b*b*c - a*c*c)*f)*q23*q23 + 2.*(e*c*d*d -
    b*d*d*d)*e + (e*e*c*c + (b*b - 2.*a*c)*d*d - 2.*(e*c*c - b*c*d)*e)*f;

  if (sqt < 0.) return FIM_INF;

  const double pa = e*c*d*d - b*d*d*d + (e*c - b*d)*f*q13*q13 - 2.*(e*c*d - b*d*d)*q13*q23 +
                    (e*c*c - b*c*d)*q23*q23 - (e*c*c - b*c*d)*f;
  const double pb = (d*d*d*d - 2.*c*d*d*f + c*c*f*f + (d*d*f - c*f*f)*q13*q13 -
                     2.*(d*d*d - c*d*f)*q13*q23 + (c*d*d - c*c*f)*q23*q23);

  const double la2 = (pa + sqt*(d*q13 - c*q23))/pb;
  const double lb2 = (pa - sqt*(d*q13 - c*q23))/pb;
  const double la1 = -((f*la2 + e)*q13 - (d*la2 + b)*q23)/(d*q13 - c*q23);
  const double lb1 = -((f*lb2 + e)*q13 - (d*lb2 + b)*q23)/(d*q13 - c*q23);

  double l3 = 1 - la1 - la2, ra = FIM_INF, rb = FIM_INF;
  if ((la1 > 0. && la1 < 1.) && (la2 > 0. && la2 < 1.) && l3 > 0.)
    ra = la1*p1 + la2*p2 + l3*p3 + sqrt(a + 2.*la1*b + la1*la1*c + 2.*la1*la2*d + 2.*la2*e + la2*la2*f);
  l3 = 1 - lb1 - lb2;
  if ((lb1 > 0. && lb1 < 1.) && (lb2 > 0. && lb2 < 1.) && l3 > 0.)
    rb = lb1*p1 + lb2*p2 + l3*p3 + sqrt(a + 2.*lb1*b + lb1*lb1*c + 2.*lb1*lb2*d + 2.*lb2*e + lb2*lb2*f);
  return fmin(ra, rb);
}

// The same tet solve with its long FP64 prefix (b, c, e, q13, q23, sqt, pa,
// pb, sqt*X) spread over a group of kDagLanes lanes: the generated level
// program (gen_tet_dag.py) gives each lane one DFMA per level on operands in
// the group's scratch S, so the prefix costs kDagLevels dependent FP64
// instructions instead of one per node.  The results are bit-identical to
// tet_ref (every node is one correctly rounded operation of the source's own
// expression tree).
#include "tet_dag.inc"
// Doubles from one group's scratch to the next: half a bank row apart (mod
// 128 B), so that two groups of a half-warp write without conflicts.
constexpr int kDagStride = (kDagSlots + 15) / 16 * 16 + 8;

// x with its sign flipped where the word `flip` has its top bit set
__device__ __forceinline__ double flip_sign(double x, uint32_t flip)
{
  return __hiloint2double(__double2hiint(x) ^ (int)flip, __double2loint(x));
}

// Runs the level program on scratch S (leaves already stored); gl is the
// lane's index in its group.  All lanes of the warp take part.  A lane's
// program words are loaded three levels ahead (level by level from constant
// memory, with eight addresses per warp, they lengthened every level), and
// its operands one level ahead: the program takes a result of the level
// before only from the lane's own register.  One warp of four tets: 1.48 us
// (21 levels); 1.73 us with every operand from shared memory (20 levels),
// 1.85 us where also the groups' scratch lay on the same banks.
__device__ __forceinline__ void tet_dag_prefix(double *S, int gl)
{
  const uint4 *prog = kTetDagProg[gl];
  uint4 q = __ldg(prog);
  uint32_t w = q.x;
  double A = S[w & 255u], B = S[(w >> 8) & 255u], C = S[(w >> 16) & 255u], last = 0.0;
  double *out = S + kDagLeaves + gl;
#pragma unroll
  for (int r = 0; r < kDagLevels / kDagStep; ++r) {
    const uint4 next = __ldg(prog + (r + 1 < kDagLevels / kDagStep ? r + 1 : r));
#pragma unroll
    for (int k = 0; k < kDagStep; ++k) {
      const double x = fma(flip_sign((w & (1u << 27)) ? last : A, (w << 7) & 0x80000000u), (w & (1u << 28)) ? last : B,
                           flip_sign((w & (1u << 29)) ? last : C, (w << 5) & 0x80000000u));
      // while that runs: the next level's operands, of levels up to the last
      // (past the end: some again)
      w = k == 0 ? q.y : (k == 1 ? q.z : next.x);
      A = S[w & 255u]; B = S[(w >> 8) & 255u]; C = S[(w >> 16) & 255u];
      last = x;
      *out = last;
      out += kDagLanes;
      __syncwarp();
    }
    q = next;
  }
}

// One root of tet_ref from the prefix in S: second = false gives its "a"
// value (pa + sqt X), true its "b" value (pa - sqt X, written as
// pa + (-(sqt X)), which IEEE arithmetic rounds identically), so two lanes
// run one instruction stream and tet_ref's result is the fmin of their
// values.  The sign tests run on the integer pipes (dlt0, din01, dgt0).
__device__ __forceinline__ double tet_root_tail(const double *S, bool second)
{
  const double a = S[kDagLeafE13], d = S[kDagLeafE13 + 1], f = S[kDagLeafE13 + 2];
  const double b = S[kDagOut_b], c = S[kDagOut_c], e = S[kDagOut_e];
  const double p1 = S[kDagLeafP1], p2 = S[kDagLeafP1 + 1], p3 = S[kDagLeafP1 + 2];
  const double q13 = S[kDagOut_q13], q23 = S[kDagOut_q23];
  const double sqt = S[kDagOut_sqt];
  if (dlt0(sqt)) return FIM_INF;
  const double pa = S[kDagOut_pa], pb = S[kDagOut_pb], sx = S[kDagOut_sx], X = S[kDagOut_X];
  const double l2 = (pa + (second ? -sx : sx))/pb;
  const double l1 = -((f*l2 + e)*q13 - (d*l2 + b)*q23)/X;
  const double l3 = 1 - l1 - l2;
  double r = FIM_INF;
  if (din01(l1) && din01(l2) && dgt0(l3))
    r = l1*p1 + l2*p2 + l3*p3 + sqrt(a + 2.*l1*b + l1*l1*c + 2.*l1*l2*d + 2.*l2*e + l2*l2*f);
  return r;
}


// ---------------------------------------------------------------------------
// corner relabelling and bound packing (metric kernel and solve)

// For target slot t the other slots are relabelled "1","2","3" =
// (t+1)%4, (t+2)%4, (t+3)%4 (the reference's gray-code mapping,
// cuda_fim.h:41-48).  sel_of(t, k) is the edge index of the k-th relabelled
// edge e13, e23, e34, e12, e14, e24.
__host__ __device__ constexpr int sel_of(int t, int k)
{
  return k == 0 ? edge_index((t + 1) & 3, (t + 3) & 3)
       : k == 1 ? edge_index((t + 2) & 3, (t + 3) & 3)
       : k == 2 ? edge_index((t + 3) & 3, t)
       : k == 3 ? edge_index((t + 1) & 3, (t + 2) & 3)
       : k == 4 ? edge_index((t + 1) & 3, t)
       :          edge_index((t + 2) & 3, t);
}

// Two non-negative lower bounds as fp16 rounded towards -inf (so they stay
// lower bounds), packed low | high << 16.
__device__ __forceinline__ uint32_t half_pair_rd(float lo, float hi)
{
  return (uint32_t)__half_as_ushort(__float2half_rd(lo)) | ((uint32_t)__half_as_ushort(__float2half_rd(hi)) << 16);
}
__device__ __forceinline__ float half_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float half_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }

// ---------------------------------------------------------------------------
// bounded grid barrier

__device__ __forceinline__ uint64_t global_timer()
{
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int ld_volatile_i32(const int32_t *p)
{
  return *(const volatile int32_t *)p;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// All blocks of the (co-resident) grid meet here, for barrier k (1, 2, ...):
// each adds 1 to the low half of the phase's word (FimCtl::phase) and waits
// until all have.  *count receives the high half, the length of the list that
// the phase appended to: one L2 round trip less per phase than reading it
// after the barrier.  Every wait is bounded by timeout_ns of %globaltimer and
// by a spin cap; on expiry the block records KERR_TIMEOUT and the phase and
// sets the word's error bit, and every block leaves the kernel at its next
// barrier.  Returns false when the caller must return.
constexpr uint32_t kPhaseError = 0x80000000u;
static __device__ bool grid_sync(FimCtl *ctl, uint32_t nblocks, uint64_t timeout_ns, int k, int32_t *count)
{
  __shared__ int s_ok, s_count;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long *word = &ctl->phase[k & 3].v;
    // the word of phase k + 2, last used by barrier k - 2, which every block has left
    if (blockIdx.x == 0) ctl->phase[(k + 2) & 3].v = 0ull;
    // (a release on the arrival itself: with a full fence before a relaxed one
    // the 58k windowed slab took 4.25 ms instead of 4.17)
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(1ull) : "memory");
    const uint64_t t0 = global_timer();
    uint32_t spins = 0;
    int ok = 1;
    unsigned long long w;
    for (;;) {
      w = ld_acquire_u64(word);
      if ((uint32_t)w >= nblocks) break;  // everyone is here (or the error bit is set)
      ++spins;
      if ((spins & 255u) == 0u) {
        if (ld_volatile_i32(&ctl->error) != KERR_NONE) { ok = 0; break; }
        if (global_timer() - t0 > timeout_ns || spins > (1u << 30)) {
          if (atomicCAS(&ctl->error, KERR_NONE, KERR_TIMEOUT) == KERR_NONE) ctl->error_where = k;
          atomicOr(word, (unsigned long long)kPhaseError);
          ok = 0;
          break;
        }
      }
    }
    if ((uint32_t)w & kPhaseError) ok = 0;
    s_ok = ok;
    s_count = (int32_t)(w >> 32);
  }
  __syncthreads();
  *count = s_count;
  return s_ok != 0;
}

// Order-preserving map of doubles to unsigned integers, so that the minimum
// of a vertex's candidates can be formed with integer atomicMin.
__device__ __forceinline__ unsigned long long dkey(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dunkey(unsigned long long k)
{
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

}  // namespace fimgb
