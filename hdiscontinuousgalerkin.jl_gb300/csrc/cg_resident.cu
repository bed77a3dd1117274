// The Jacobi CG iteration of one problem in one launch, its state resident on the chip.
//
// With two kernels per iteration (cg.cu) a small system pays for launches, reduction tails and
// re-read vectors, not for arithmetic.  Measured per iteration, two kernels / here (whole solves): 14.9 / 6.1 us at 6272
// rows (p = 1, FP64), 22 / 10 us at 142k rows (p = 4, FP32), 43 / 32.5 us at 591k rows (p = 2, FP64; 22.7 us of it are the
// FP64 pipe's 23 instructions a row).  Here every CTA owns a contiguous range of faces for the whole launch.  Its rows of x, r, p, q,
// D^-1 and z stay in shared memory (and its matrix rows too, where they fit), only z travels through L2 (the
// columns of a row belong to other CTAs), and an iteration is two phases with a reduction over all CTAs after
// each:
//   A: q = A z + beta q, p = z + beta p, p.q           | alpha
//   B: x += alpha p, r -= alpha q, z = D^-1 r, r.z, r.r | beta, convergence; z is visible to all
// Every CTA forms the same scalars from the same partials in the same order, so all leave the loop together and
// repeated solves are bit-identical.
//
// Two ways to run the reduction, chosen by size (cg_resident_plan):
//   cluster  at most 16 CTAs in one cluster: partials go through distributed shared memory and the barrier is the
//            hardware's (0.24 us at 16 CTAs), but only 16 SMs' FP64 pipes work on the rows;
//   grid     a cooperative launch of one CTA per SM: partials go through L2 and the barrier is a counter (1.3 us at
//            152 CTAs), which pays once the rows' arithmetic on 16 SMs costs more.
// A grid has the chip to itself (others of the process wait for it: res_launch), so it is for a solve that is alone: grid_turns
// in cg.cu.
// A counter barrier gives up after SPIN_LIMIT polls (seconds) and reports CG_LOST instead of waiting for ever.
//
// What bounds it: the FP64 pipe issues a warp instruction per 16 clocks whatever its active lanes, with 64 clocks of
// latency (measured), so a reduction is a chain of some 25 dependent FP64 instructions, and a scalar that every
// thread forms for itself costs 16 warps' worth of the pipe: the sums are spread over the four schedulers, the scalars
// formed by one thread, and the FP32 iteration's block sums are float-float on the FP32 pipe.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "cg_resident.cuh"
#include "cg_sync.cuh"
#include "once_per_device.h"

namespace {


template <typename T> struct ResArgs {
  CgArgs<T> a;
  float2* pairs;     // FP32: (z, p) of every row, two buffers of nf * NT
  unsigned* count;   // grid: arrivals (zeroed before the launch)
  double* part;      // grid: [2][MAX_GRID][2] partials
  int faces_per_cta, iters;
};

template <int NT> __device__ __forceinline__ void load_z(const double* __restrict__ z, int g, double (&o)[NT]) {
  const double* s = z + (int64_t)g * NT;
  if constexpr (NT % 2 == 0) {  // g NT doubles from an aligned base: 16-byte aligned
#pragma unroll
    for (int j = 0; j < NT; j += 2) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(s + j));
      o[j] = v.x;
      o[j + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < NT; ++j) o[j] = __ldcg(s + j);
  }
}

template <int NT, typename T, bool GRID, bool MAT>
__global__ void __launch_bounds__(RB, 1) k_cg_resident(ResArgs<T> q) {
  constexpr bool F64 = sizeof(T) == sizeof(double);
  const CgArgs<T>& a = q.a;
  __shared__ ResShared sh;
  extern __shared__ __align__(16) unsigned char dyn[];
  const int fpc = q.faces_per_cta, cap = fpc * NT;
  const int f0 = blockIdx.x * fpc, nfl = max(0, min(fpc, a.nf - f0)), nr = nfl * NT, row0 = f0 * NT;
  const int64_t nd = (int64_t)a.nf * NT;
  // shared arrays of the CTA's rows
  T* sr = reinterpret_cast<T*>(dyn);
  T* sp = sr + cap;
  T* sq = sp + cap;
  T* sd = sq + cap;
  T* sz = sd + cap;
  T* sx = sz + cap;          // FP64: x; FP32: xh, xl
  T* sxl = sx + cap;
  T* sm = sx + (F64 ? 1 : 2) * cap;  // matrix rows [5 NT][cap]
  int32_t* sc = reinterpret_cast<int32_t*>(sm + (MAT ? 5 * NT * cap : 0));  // block columns [5][fpc]

  // scalars of the problem: kept by thread 0, the same in every CTA
  double rz = a.sc[0], rz_old = a.sc[1], pq = a.sc[2], rr = a.sc[3], alpha = a.sc[6];
  const double beta0 = a.sc[7];
  double beta = beta0, stop_rr = 0.0, floor_rr = 0.0;
  if (threadIdx.x == 0) {
    const double bb = a.sc[4], tol2 = a.sc[5];
    stop_rr = tol2 * bb;
    floor_rr = fmax(1e-24, 100.0 * tol2) * bb;
    sh.rz = rz;
  }
  int status = a.st[0], it = a.st[1];
  const int maxit = a.st[2];
  if (status != 0) return;  // uniform over the grid

  for (int k = threadIdx.x; k < 5 * nfl; k += RB) {
    const int s = k / nfl, f = k - s * nfl;
    sc[s * fpc + f] = a.bcol5[(int64_t)s * a.nf + f0 + f];
  }
  if constexpr (MAT) {
    for (int s = 0; s < 5 * NT; ++s)
      for (int l = threadIdx.x; l < nr; l += RB) sm[s * cap + l] = a.val[s * nd + row0 + l];
  }
  for (int l = threadIdx.x; l < nr; l += RB) {
    const int row = row0 + l;
    sr[l] = a.r[row];
    sp[l] = a.p[row];
    sd[l] = a.dinv[row];
    sz[l] = a.z[row];
    if constexpr (F64) {
      sq[l] = a.q[row];
      sx[l] = a.x[row];
    } else {
      sx[l] = a.xh[row];
      sxl[l] = a.xl[row];
      q.pairs[row] = make_float2((float)sz[l], (float)sp[l]);
    }
  }
  int epoch = 0;
  if constexpr (!GRID) cluster_sync_all();  // every CTA of the cluster runs before its shared memory is written
  if constexpr (!F64) {  // the pairs of all CTAs are in place
    double none[1];
    const bool ok = all_sum<GRID, 1>(sh, q.count, q.part, epoch++, 0.0, none);
    if (threadIdx.x == 0) sh.status = ok ? 0 : CG_LOST;
  }
  __syncthreads();
  if (!F64 && sh.status != 0) {
    if (threadIdx.x == 0) a.st[0] = CG_LOST;
    return;
  }

  int n = 0;
  for (; n < q.iters && status == 0; ++n) {
    // ---- A ------------------------------------------------------------------------------------------------
    // beta: of the launch's start, then of the last B (read before sh.bc is written again: a reduction lies between)
    const T bt = n == 0 ? (T)beta0 : (F64 ? (T)sh.bc : (T)sh.bch);
    if (threadIdx.x == RB - 1) sh.rz_inv = recip(sh.rz);  // for beta: r.z of this direction is known already
    typename DotAcc<T>::type dpq;
    const float2* __restrict__ pin = F64 ? nullptr : q.pairs + (int64_t)(n & 1) * nd;
    for (int l = threadIdx.x; l < nr; l += RB) {
      const int f = l / NT;
      T w0 = T(0), w1 = T(0);  // few rows per thread (MAT): two chains, since the FP64 latency is 64 clocks
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const int g = sc[k * fpc + f];
        T zc[NT];
        if constexpr (F64) {
          load_z<NT>(a.z, g, zc);
        } else {
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const float2 v = __ldcg(pin + (int64_t)g * NT + j);
            zc[j] = v.x + bt * v.y;
          }
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int s = k * NT + j;
          const T v = MAT ? sm[s * cap + l] : __ldg(a.val + s * nd + row0 + l);
          if (MAT && (s & 1)) w1 += v * zc[j];
          else w0 += v * zc[j];
        }
      }
      const T pn = sz[l] + bt * sp[l];
      if constexpr (MAT) w0 += w1;
      const T qn = F64 ? w0 + bt * sq[l] : w0;
      sp[l] = pn;
      sq[l] = qn;
      dpq.add_prod(pn, qn);
    }
    {
      double s1[1], mine;
      if constexpr (F64) mine = cta_sum<1>(sh, {dpq.v});
      else mine = cta_sum<1>(sh, {dpq});
      const bool ok = all_sum<GRID, 1>(sh, q.count, q.part, epoch++, mine, s1);
      if (threadIdx.x == 0) {
        pq = s1[0];
        alpha = (pq > 0.0) ? rz * recip(pq) : 0.0;
        sh.bc = alpha;
        if constexpr (!F64) {
          sh.bch = (float)alpha;
          sh.bcl = (float)(alpha - (double)sh.bch);
        }
        sh.status = ok ? 0 : CG_LOST;
      }
    }
    __syncthreads();
    if (sh.status != 0) {
      status = CG_LOST;
      break;
    }
    // ---- B ------------------------------------------------------------------------------------------------
    const T at = F64 ? (T)sh.bc : (T)sh.bch;
    const float ah = sh.bch, al = sh.bcl;
    typename DotAcc<T>::type drz, drr;
    float2* pout = F64 ? nullptr : q.pairs + (int64_t)((n + 1) & 1) * nd;
    for (int l = threadIdx.x; l < nr; l += RB) {
      const T pv = sp[l];
      if constexpr (F64) {
        sx[l] += at * pv;
      } else {  // x += alpha p in float-float
        const float ph = __fmul_rn(ah, (float)pv);
        const float pe = __fmaf_rn(al, (float)pv, __fmaf_rn(ah, (float)pv, -ph));
        FF xx;
        xx.hi = sx[l];
        xx.lo = sxl[l];
        xx.add2(ph, pe);
        sx[l] = xx.hi;
        sxl[l] = xx.lo;
      }
      const T rn = sr[l] - at * sq[l];
      const T zn = sd[l] * rn;
      sr[l] = rn;
      sz[l] = zn;
      if constexpr (F64) a.z[row0 + l] = zn;
      else pout[row0 + l] = make_float2((float)zn, (float)pv);
      drz.add_prod(rn, zn);
      drr.add_prod(rn, rn);
    }
    {
      double s2[2], mine;
      if constexpr (F64) mine = cta_sum<2>(sh, {drz.v, drr.v});
      else mine = cta_sum<2>(sh, {drz, drr});
      const bool ok = all_sum<GRID, 2>(sh, q.count, q.part, epoch++, mine, s2);
      if (threadIdx.x == 0) {  // the decisions of k_cg_b
        const double rr_prev = rr;
        rz_old = rz;
        rz = s2[0];
        rr = s2[1];
        beta = rz * sh.rz_inv;
        sh.rz = rz;
        int next = 0;
        if (!(pq > 0.0) || !isfinite(rr)) {
          next = (isfinite(rr) && rr_prev <= floor_rr) ? 1 : 3;
        } else if (rr <= stop_rr) {
          next = 1;
        } else if (it + 1 >= maxit) {
          next = 2;
        }
        sh.bc = beta;
        if constexpr (!F64) sh.bch = (float)beta;
        sh.status = ok ? next : CG_LOST;
      }
    }
    __syncthreads();
    status = sh.status;
    if (status == CG_LOST) break;
    ++it;
  }
  // state back to memory (z is there already in FP64)
  for (int l = threadIdx.x; l < nr; l += RB) {
    const int row = row0 + l;
    a.r[row] = sr[l];
    a.p[row] = sp[l];
    a.q[row] = sq[l];
    if constexpr (F64) {
      a.x[row] = sx[l];
    } else {
      a.z[row] = sz[l];
      a.xh[row] = sx[l];
      a.xl[row] = sxl[l];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.sc[0] = rz;
    a.sc[1] = rz_old;
    a.sc[2] = pq;
    a.sc[3] = rr;
    a.sc[6] = alpha;
    a.sc[7] = beta;
    a.sc[9] = 0.0;  // the latest direction is in p
    a.st[1] = it;
  }
  if (threadIdx.x == 0 && (blockIdx.x == 0 || status == CG_LOST)) a.st[0] = status;
}

template <int NT, typename T> size_t res_smem(int fpc, bool mat) {
  const size_t vec = sizeof(T) == sizeof(double) ? 6 : 7;
  return sizeof(T) * (size_t)fpc * NT * (vec + (mat ? 5 * NT : 0)) + sizeof(int32_t) * 5 * (size_t)fpc;
}

template <int NT, typename T, bool GRID, bool MAT> void set_attributes(int device) {
  static OncePerDevice once;
  once(device, [] {
    auto* k = k_cg_resident<NT, T, GRID, MAT>;
    HDG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
    if (!GRID) HDG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  });
}

template <int NT, typename T, bool MAT> int max_clusters(int ctas, size_t smem, int device) {
  set_attributes<NT, T, false, MAT>(device);
  return res_max_clusters(k_cg_resident<NT, T, false, MAT>, ctas, smem);
}

// Rows up to which one cluster is the faster form: beyond, the rows' arithmetic on 16 SMs costs more than the
// counter barriers of the grid form save.  Clocks per iteration, cluster / grid: FP64 p = 1, 2480 rows 10.7k / 17.3k,
// 6272 rows 13.3k / 17.9k, 24832 rows 32.7k / 18.2k; solves of the FP32 iteration, p = 4: 15.7k rows 9.8 / 10.9 ms,
// 30.8k rows 18.0 / 15.8 ms.
template <typename T> constexpr int cluster_rows() { return sizeof(T) == sizeof(double) ? 11000 : 20000; }

template <int NT, typename T> CgResident plan_nt(int nf, int device, bool grid_allowed) {
  CgResident pl;
  const int forced = res_forced_kind();
  if (forced == CgResident::NONE) return pl;
  const int64_t rows = (int64_t)nf * NT;
  if (forced != CgResident::GRID && (rows <= cluster_rows<T>() || forced == CgResident::CLUSTER)) {
    const int c = MAX_CLUSTER, fpc = (nf + c - 1) / c;
    for (int mat = 1; mat >= 0; --mat) {
      const size_t sm = res_smem<NT, T>(fpc, mat);
      if (sm > SMEM_MAX) continue;
      if ((mat ? max_clusters<NT, T, true>(c, sm, device) : max_clusters<NT, T, false>(c, sm, device)) < 1) continue;
      return CgResident{CgResident::CLUSTER, c, fpc, mat != 0, sm};
    }
  }
  if (!grid_allowed && forced != CgResident::GRID) return pl;
  int sms = 0;
  if ((sms = res_grid_ctas(device)) == 0) return pl;
  const int fpc = (nf + sms - 1) / sms;
  for (int mat = 1; mat >= 0; --mat) {
    const size_t sm = res_smem<NT, T>(fpc, mat);
    if (sm <= SMEM_MAX) return CgResident{CgResident::GRID, sms, fpc, mat != 0, sm, forced == CgResident::GRID};
  }
  return pl;  // the vectors do not fit on the chip
}

template <int NT, typename T, bool GRID, bool MAT>
void launch_one(const CgResident& pl, ResArgs<T> q, int device, cudaStream_t st) {
  set_attributes<NT, T, GRID, MAT>(device);
  if (GRID) HDG_CUDA(cudaMemsetAsync(q.count, 0, sizeof(unsigned), st));
  res_launch<GRID>(k_cg_resident<NT, T, GRID, MAT>, pl.ctas, pl.smem, q, device, st);
}

template <int NT, typename T>
void launch_nt(const CgResident& pl, const CgArgs<T>& a, float2* pairs, void* sync, int iters, int device,
               cudaStream_t st) {
  static_assert(CG_SYNC_BYTES >= 256 + sizeof(double) * 4 * MAX_GRID, "partials of every CTA");
  ResArgs<T> q{a, pairs, (unsigned*)sync, (double*)((char*)sync + 256), pl.faces_per_cta, iters};
  const bool grid = pl.kind == CgResident::GRID;
  if (grid && pl.mat_smem) launch_one<NT, T, true, true>(pl, q, device, st);
  else if (grid) launch_one<NT, T, true, false>(pl, q, device, st);
  else if (pl.mat_smem) launch_one<NT, T, false, true>(pl, q, device, st);
  else launch_one<NT, T, false, false>(pl, q, device, st);
}

}  // namespace

template <typename T> CgResident cg_resident_plan(int nt, int nf, int device, bool grid_allowed) {
  switch (nt) {
    case 2: return plan_nt<2, T>(nf, device, grid_allowed);
    case 3: return plan_nt<3, T>(nf, device, grid_allowed);
    case 4: return plan_nt<4, T>(nf, device, grid_allowed);
    case 5: return plan_nt<5, T>(nf, device, grid_allowed);
  }
  return CgResident{};
}

template <typename T>
void cg_resident_launch(const CgResident& pl, int nt, const CgArgs<T>& a, float2* pairs, void* sync, int iters,
                        int device, cudaStream_t st) {
  switch (nt) {
    case 2: launch_nt<2, T>(pl, a, pairs, sync, iters, device, st); break;
    case 3: launch_nt<3, T>(pl, a, pairs, sync, iters, device, st); break;
    case 4: launch_nt<4, T>(pl, a, pairs, sync, iters, device, st); break;
    case 5: launch_nt<5, T>(pl, a, pairs, sync, iters, device, st); break;
  }
}

template CgResident cg_resident_plan<double>(int, int, int, bool);
template CgResident cg_resident_plan<float>(int, int, int, bool);
template void cg_resident_launch<double>(const CgResident&, int, const CgArgs<double>&, float2*, void*, int, int,
                                         cudaStream_t);
template void cg_resident_launch<float>(const CgResident&, int, const CgArgs<float>&, float2*, void*, int, int,
                                        cudaStream_t);
