// Device-side helpers shared by the kernels of libhdg.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "hdg_internal.h"

template <int P> struct Dims {
  static constexpr int NW = (P + 1) * (P + 2) / 2;  // scalar Dubiner functions (u)
  static constexpr int NT = P + 1;                  // Legendre functions per edge (trace)
  static constexpr int NV = 2 * NW;                 // vector functions (q)
  static constexpr int N = NV + NW;                 // local (q,u) system size
  static constexpr int M = 3 * NT;                  // trace dofs of a cell
  static constexpr int NC = N + M + 1;              // augmented columns [Me | EF | Bte]
  static constexpr int LD = NC | 1;                 // odd row stride: conflict-free FP64 column reads
};

// Field evaluation: the kinds of hdg.h (HDG_FIELD_*), parameters in device memory.
__device__ __forceinline__ double eval_field_kind(int kind, const double* __restrict__ p, double x, double y) {
  switch (kind) {
    case HDG_FIELD_CONST: return p[0];
    case HDG_FIELD_SINSIN: return p[0] * sinpi(p[1] * x) * sinpi(p[2] * y);
    case HDG_FIELD_BUMPS: {
      int K = (int)p[0];
      double s = 0.0;
      for (int k = 0; k < K; ++k) {
        const double* b = p + 1 + 4 * k;
        double dx = x - b[0], dy = y - b[1];
        s += b[3] * exp(-(dx * dx + dy * dy) / (2.0 * b[2] * b[2]));
      }
      return s;
    }
    case HDG_FIELD_FOURIER:
    case HDG_FIELD_EXP_FOURIER: {
      int K = (int)p[0];
      double g = p[1];
      for (int k = 0; k < K; ++k) {
        const double* b = p + 2 + 4 * k;
        g += b[3] * cos(6.283185307179586 * (b[0] * x + b[1] * y) + b[2]);
      }
      return kind == HDG_FIELD_EXP_FOURIER ? exp(g) : g;
    }
  }
  return 0.0;
}
// The source as the element kernels read it (CoefDev::fprep): Gaussian bumps carry -1/(2 s^2) in
// place of s, every other kind its plain parameters.
__device__ __forceinline__ double eval_source_prepared(int kind, const double* __restrict__ p, double x, double y) {
  if (kind != HDG_FIELD_BUMPS) return eval_field_kind(kind, p, x, y);
  const int K = (int)p[0];
  double s = 0.0;
  for (int k = 0; k < K; ++k) {
    const double* b = p + 1 + 4 * k;
    const double dx = x - b[0], dy = y - b[1];
    s += b[3] * exp((dx * dx + dy * dy) * b[2]);
  }
  return s;
}

// ---- fields in fixed point ------------------------------------------------------------------------
// The FP64 pipe issues a warp instruction in 16 clocks, the integer pipes one in half a clock to one, and an
// exp or a cos is some 16 to 19 FP64 instructions: the element kernels spent most of their time on the modes
// of a field.  A sum of Gaussian bumps or Fourier modes is therefore evaluated in 64-bit fixed point, with
// its parameters laid out by the host (capi.cpp: prepare_fixed):
//   coordinates  X = x 2^s with |X| <= 2^61, s of the problem (its coordinates and the centres of its bumps)
//   a mode       the phase k.x + phi / 2 pi in turns, modulo one, as a 64-bit fraction: reducing the argument is
//                the wrap-around; cos by folding to a quarter turn and a polynomial in its square
//   a bump       the exponent of two (r sqrt(log2 e / 2) / sigma)^2 with 54 fraction bits; 2^-f by a polynomial, the
//                double assembled from its bits
// The polynomials interpolate at Chebyshev nodes (errors 2^-67 and 2^-58.6).  The phase is good to 2^-57 of a turn
// and the exponent to some 2^-52, where FP64 loses 2^-53 of the argument itself (of 90 radians in the workloads): the
// sums are closer to the exact ones than before: largest error over the sum of |terms| at 2e5 points, FP64 / here: 64 modes
// up to |k| = 10 1.5e-15 / 1.1e-16, their exponential 1.7e-14 / 1.2e-15, eight bumps 5.4e-15 / 4.7e-16 (rms 1.3e-16 /
// 1.2e-16).  That is of a unit square; where the grid 2^-s costs a field digits against FP64 (a narrow bump near the
// origin of a large domain, hundreds of turns over it) the field stays in FP64, as a product of sines does: it is small
// without being a difference, at the sides of a domain, and keeps its relative accuracy there.
enum { FIX_BUMPS = 100, FIX_FOURIER = 101, FIX_EXP_FOURIER = 102 };

// cos(2 pi t / 2^64) in units of 2^-62
__device__ __forceinline__ long long cos_turns(unsigned long long t) {
  const long long h = (long long)t;
  unsigned long long w = h < 0 ? 0ull - t : t;  // half a turn is 2^63
  const bool neg = w > (1ull << 62);
  if (neg) w = (1ull << 63) - w;                // a quarter turn is 2^62: taken as 2^62 - 1, so that its square fits
  w = w < (1ull << 62) ? w : (1ull << 62) - 1;
  const unsigned long long z = __umul64hi(w << 1, w << 1) << 2;  // the square of 4 w, units of 2^-64
  // terms far below the last place of the sum need 32 bits of the square only
  const unsigned zh = (unsigned)(z >> 32);
  unsigned long long q = 302636559ull - __umulhi(2363548u, zh);
  q = 29452814462ull - __umulhi((unsigned)q, zh);
  q = 2172507397706ull - __umul64hi(q, z);
  q = 116223906387215ull - __umul64hi(q, z);
  q = 4239339756756521ull - __umul64hi(q, z);
  q = 96215822532081128ull - __umul64hi(q, z);
  q = 1169844122888618737ull - __umul64hi(q, z);
  q = 5689439577989151075ull - __umul64hi(q, z);
  const long long v = (long long)(1ull << 62) - (long long)__umul64hi(q, z);
  return neg ? -v : v;
}

// 2^-e, e in units of 2^-54
__device__ __forceinline__ double exp2_minus(unsigned long long e) {
  const unsigned n = (unsigned)(e >> 54);
  if (n > 1020u) return 0.0;  // below the smallest normal number
  const unsigned long long f = e << 10;
  const unsigned fh = (unsigned)(f >> 32);
  unsigned long long q = 62120492029ull - __umulhi(2906043853u, fh);
  q = 934447969506ull - __umul64hi(q, f);
  q = 12185082205994ull - __umul64hi(q, f);
  q = 140679108108160ull - __umul64hi(q, f);
  q = 1420723857345589ull - __umul64hi(q, f);
  q = 12298036444282079ull - __umul64hi(q, f);
  q = 88711583007090357ull - __umul64hi(q, f);
  q = 511935043784382635ull - __umul64hi(q, f);
  q = 2215698446797586272ull - __umul64hi(q, f);
  q = 6393154322601321910ull - __umul64hi(q, f);
  q = 9223372036854775787ull - __umul64hi(q, f);  // in (2^62, 2^63]
  // 53 leading bits, rounded; the implicit bit carries into the exponent
  return __longlong_as_double((long long)(((unsigned long long)(1021u - n) << 52) + ((q + 512ull) >> 10)));
}

// The angle of mode b = (kx, ky, phase, amplitude) at a point, in units of 2^-64 turn
__device__ __forceinline__ unsigned long long turns_of(long long X, long long Y, const double* __restrict__ b, int sh) {
  const __int128 t = (__int128)X * __double_as_longlong(b[0]) + (__int128)Y * __double_as_longlong(b[1]);
  const unsigned long long lo = (unsigned long long)t;
  const long long hi = (long long)(t >> 64);
  const unsigned long long turns = sh < 64 ? (lo >> sh) | ((unsigned long long)hi << 1 << (63 - sh))
                                           : (unsigned long long)(hi >> (sh - 64));
  return turns + (unsigned long long)__double_as_longlong(b[2]);
}

// The terms part, part + parts, ... of a field that is a sum (bumps, modes), so that several lanes can share a point; a
// field that is no sum is evaluated whole by part 0.  The parts add up to the field, or to what finish_parts makes it
// from.  kind and p: the prepared form (CoefDev::fkfix, ffix); X, Y: the point in fixed point.
__device__ __forceinline__ double eval_part(int kind, const double* __restrict__ p, double x, double y, long long X,
                                            long long Y, int part, int parts) {
  if (kind == FIX_BUMPS) {
    const int K = (int)__double_as_longlong(p[0]);
    double s = 0.0;
    for (int k = part; k < K; k += parts) {
      const double* b = p + 1 + 4 * k;
      const long long dx = X - __double_as_longlong(b[0]), dy = Y - __double_as_longlong(b[1]);
      const unsigned long long sg = (unsigned long long)__double_as_longlong(b[2]);  // scale, its shift in the low bits
      const int sh = (int)(sg & 63ull);
      const unsigned long long gx = __umul64hi((unsigned long long)(dx < 0 ? -dx : dx), sg);
      const unsigned long long gy = __umul64hi((unsigned long long)(dy < 0 ? -dy : dy), sg);
      if (((gx | gy) >> (63 - sh)) > 1ull) continue;  // beyond 32 sqrt(2 / log2 e) widths: below 2^-1024
      const unsigned long long ax = gx << sh, ay = gy << sh;
      const unsigned long long ex = __umul64hi(ax, ax), e = ex + __umul64hi(ay, ay);
      if (e >= ex) s = fma(b[3], exp2_minus(e), s);
    }
    return s;
  }
  if (kind == FIX_FOURIER || kind == FIX_EXP_FOURIER) {
    const unsigned long long head = (unsigned long long)__double_as_longlong(p[0]);
    const int K = (int)(head & 0xffffffffull), sh = (int)((head >> 32) & 0xffull), w = (int)(short)(head >> 48);
    long long s = 0;
    for (int k = part; k < K; k += parts) {
      const double* b = p + 2 + 4 * k;
      s += __mul64hi(cos_turns(turns_of(X, Y, b, sh)), __double_as_longlong(b[3]));
    }
    const double v = (double)s * __hiloint2double((1023 + 2 - w) << 20, 0);
    return part == 0 ? p[1] + v : v;
  }
  return part == 0 ? eval_source_prepared(kind, p, x, y) : 0.0;
}
// The field from the sum of its parts.
__device__ __forceinline__ double finish_parts(int kind, double v) { return kind == FIX_EXP_FOURIER ? exp(v) : v; }

// 1/d to an ulp from the hardware's FP64 estimate (some 20 bits, not on the FP64 pipe) by one step of third order,
// r <- r (1 + e + e^2) with e = 1 - d r, which cubes the error: three FP64 instructions.  Where the estimate or the step
// under- or overflows: the division.
__device__ __forceinline__ double recip_cubic(double d) {
  const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
  if (e < 24u || e > 2022u) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double x = fma(-d, r, 1.0);
  return fma(r, fma(x, x, x), r);
}

// 1/d by Newton-Raphson iteration from the FP32 approximate reciprocal: each step r <- r + r (1 - d r)
// squares the relative error (about 2^-22 -> 2^-44 -> below 2^-53), so two steps give the FP64
// reciprocal to within an ulp at a fraction of the cost of a correctly rounded FP64 division.
// Outside the FP32 range the FP64 division is used.
__device__ __forceinline__ double recip_newton(double d) {
  const float df = (float)d;
  if (!(fabsf(df) > 1e-30f && fabsf(df) < 1e30f)) return 1.0 / d;
  double r = (double)__fdividef(1.0f, df);
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  return r;
}

__device__ __forceinline__ double eval_field_dev(const FieldDev& f, double x, double y) {
  return eval_field_kind(f.kind, f.prm, x, y);
}



__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block reduction of one double (all threads get the result).
template <int BLOCK> __device__ __forceinline__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = (l < BLOCK / 32) ? sh[l] : 0.0;
    t = warp_sum(t);
    if (l == 0) sh[0] = t;
  }
  __syncthreads();
  t = sh[0];
  __syncthreads();
  return t;
}

// Segments: every CUDA block of a row-parallel kernel covers rows [row0, row1) of one problem.
// A per-problem sum is formed deterministically: each block writes its partial, and the last
// block of the problem to finish (atomic ticket, no waiting) adds the problem's partials in
// block order.  part holds 2 doubles per block; cnt holds one ticket per (problem, slot).
struct SegArgs {
  const int32_t* seg_prob;
  const int32_t* seg_row0;
  const int32_t* seg_row1;
  const int32_t* prob_blk0;
  const int32_t* prob_nblk;
  double* part;
  unsigned* cnt;  // [nprob][4]
};

// ---- reductions with few FP64 instructions ---------------------------------------------------
// GB300 issues FP64 at about 2 lanes per clock per SM, 1/64 of its FP32 rate, so a shuffle tree
// over every warp of a block (5 FP64 adds per warp per value) costs more than the rows it sums.
// The block sums below stage the per-thread values in shared memory and add them with 1 or 2
// warps (8 values per lane in sequence, then one shuffle tree).  Dot products of the FP32
// iteration are accumulated in float-float arithmetic on the FP32 pipe instead (FF).  All sums
// run in a fixed order, so the results are deterministic.  Results are valid in thread 0.

// Float-float accumulator: the pair (hi, lo) holds the sum to about 2^-44 relative.  a*b is split
// exactly with an FMA (Dekker's product, via fmaf) and added with Knuth's TwoSum followed by a
// renormalisation; the _rn intrinsics keep the compiler from contracting or reordering the steps.
struct FF {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add2(float h, float l) {
    const float s = __fadd_rn(hi, h);
    const float bv = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bv)), __fsub_rn(h, bv));
    const float t = __fadd_rn(__fadd_rn(lo, l), err);
    hi = __fadd_rn(s, t);
    lo = __fsub_rn(t, __fsub_rn(hi, s));
  }
  __device__ __forceinline__ void add_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    add2(p, __fmaf_rn(a, b, -p));
  }
  __device__ __forceinline__ double to_double() const { return (double)hi + (double)lo; }
};

// FP64 accumulator with the FF interface.
struct D64 {
  double v = 0.0;
  __device__ __forceinline__ void add_prod(double a, double b) { v = fma(a, b, v); }
  __device__ __forceinline__ double to_double() const { return v; }
};

template <typename T> struct DotAcc;
template <> struct DotAcc<double> { using type = D64; };
template <> struct DotAcc<float> { using type = FF; };

__device__ __forceinline__ FF warp_sum(FF v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float h = __shfl_xor_sync(0xffffffffu, v.hi, o);
    const float l = __shfl_xor_sync(0xffffffffu, v.lo, o);
    v.add2(h, l);
  }
  return v;
}

// Block sums of NV (1 or 2) doubles.
template <int BLOCK, int NV>
__device__ __forceinline__ void block_sum_lean(const double (&v)[NV], double (&out)[NV]) {
  static_assert(BLOCK % 32 == 0 && BLOCK <= 1024 && (NV == 1 || NV == 2), "block shape");
  constexpr int PER = BLOCK / 32;
  __shared__ double red[NV * BLOCK];
#pragma unroll
  for (int i = 0; i < NV; ++i) red[i * BLOCK + threadIdx.x] = v[i];
  __syncthreads();
  if (threadIdx.x < 32 * NV) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const double* src = red + w * BLOCK + l * PER;
    double t = src[0];
#pragma unroll
    for (int k = 1; k < PER; ++k) t += src[k];
    t = warp_sum(t);
    if (l == 0) red[w * BLOCK] = t;  // this warp alone read red[w*BLOCK, (w+1)*BLOCK)
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) out[i] = red[i * BLOCK];
  __syncthreads();
}

// Block sums of NV float-float values, returned as doubles.
template <int BLOCK, int NV>
__device__ __forceinline__ void block_sum_lean(const FF (&v)[NV], double (&out)[NV]) {
  static_assert(BLOCK % 32 == 0 && BLOCK <= 1024 && (NV == 1 || NV == 2), "block shape");
  __shared__ float2 red[NV][BLOCK / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const FF t = warp_sum(v[i]);
    if (l == 0) red[i][w] = make_float2(t.hi, t.lo);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      FF s;
      for (int k = 0; k < BLOCK / 32; ++k) s.add2(red[i][k].x, red[i][k].y);
      out[i] = s.to_double();
    }
  }
  __syncthreads();
}

// Cross-block stage: the block's partials (valid in thread 0) go to part[], and the last block of
// the problem adds the problem's partials (each thread its strided share, then a block sum, in a
// fixed order).  Returns true in every thread of that last block; the sums are valid in its
// thread 0.
template <int BLOCK, int NV>
__device__ __forceinline__ bool seg_combine(const SegArgs& g, int P, int slot, const double (&bp)[NV],
                                            double (&sum)[NV]) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) g.part[2 * blockIdx.x + i] = bp[i];
    __threadfence();
    const unsigned t = atomicAdd(&g.cnt[4 * P + slot], 1u);
    last = (t == (unsigned)g.prob_nblk[P] - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int b0 = g.prob_blk0[P], nb = g.prob_nblk[P];
  double s[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) s[i] = 0.0;
  for (int k = threadIdx.x; k < nb; k += BLOCK)  // every thread loads its strided partials
#pragma unroll
    for (int i = 0; i < NV; ++i) s[i] += ((volatile double*)g.part)[2 * (b0 + k) + i];
  double tot[NV];
  block_sum_lean<BLOCK, NV>(s, tot);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) sum[i] = tot[i];
    g.cnt[4 * P + slot] = 0;
  }
  return true;
}

// Per-problem sums of two (seg_finish) or one (seg_finish1) values: block sums, then the
// cross-block stage.  V is double or FF (a D64 accumulator is passed as its double).
template <int BLOCK, typename V>
__device__ __forceinline__ bool seg_finish(const SegArgs& g, int P, int slot, V v0, V v1, double* sum0,
                                           double* sum1) {
  const V v[2] = {v0, v1};
  double bp[2], s[2];
  block_sum_lean<BLOCK, 2>(v, bp);
  if (!seg_combine<BLOCK, 2>(g, P, slot, bp, s)) return false;
  *sum0 = s[0];
  *sum1 = s[1];
  return true;
}
template <int BLOCK>
__device__ __forceinline__ bool seg_finish(const SegArgs& g, int P, int slot, D64 v0, D64 v1, double* sum0,
                                           double* sum1) {
  return seg_finish<BLOCK, double>(g, P, slot, v0.v, v1.v, sum0, sum1);
}
template <int BLOCK, typename V>
__device__ __forceinline__ bool seg_finish1(const SegArgs& g, int P, int slot, V v0, double* sum0) {
  const V v[1] = {v0};
  double bp[1], s[1];
  block_sum_lean<BLOCK, 1>(v, bp);
  if (!seg_combine<BLOCK, 1>(g, P, slot, bp, s)) return false;
  *sum0 = s[0];
  return true;
}
