// What the resident CG iterations (cg_resident.cu, lagrange.cu) share: sums over the CTAs of one cluster or of a
// cooperative grid, and their launches.
#pragma once
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "cg_resident.cuh"

constexpr int RB = 512;                 // threads per CTA
constexpr int MAX_CLUSTER = 16;
constexpr int MAX_GRID = 256;           // CTAs whose partials fit the synchronisation buffer
constexpr int SPIN_LIMIT = 1 << 22;
constexpr size_t SMEM_MAX = 216 * 1024; // dynamic; the static part (reduction staging) is below 12 KB

struct ResShared {
  double stage[2][RB];
  double part[2][RB / 4];
  float2 ff[2][RB / 32];
  double slot[2][MAX_CLUSTER][2];  // cluster: every CTA's partials, written by their owners
  double bc;                       // broadcast within the CTA: alpha, beta
  double rz, rz_inv;               // r.z and, formed off the critical path, its reciprocal
  float bch, bcl;                  // alpha as a float-float pair
  int status;
};

// The CTA's sums of NV values per thread, in lanes 0..NV-1 of warp 0.  FP64: four warps (one per scheduler) add four
// values per lane, then one warp adds the rest, its lower lanes the first value's and its upper lanes the second's: as
// few FP64 instructions as the depth of the tree allows.
template <int NV> __device__ __forceinline__ double cta_sum(ResShared& sh, const double (&v)[NV]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int i = 0; i < NV; ++i) sh.stage[i][t] = v[i];
  __syncthreads();
  if (t < RB / 4) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const double* s = sh.stage[i] + t;
      sh.part[i][t] = (s[0] + s[RB / 4]) + (s[RB / 2] + s[3 * RB / 4]);
    }
  }
  __syncthreads();
  if (t >= 32) return 0.0;
  if constexpr (NV == 1) {
    const double* s = sh.part[0] + t;
    return warp_sum((s[0] + s[32]) + (s[64] + s[96]));
  } else {
    const double* s = sh.part[t >> 4] + (t & 15);
    double x = ((s[0] + s[16]) + (s[32] + s[48])) + ((s[64] + s[80]) + (s[96] + s[112]));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return __shfl_sync(0xffffffffu, x, (t & 1) << 4);  // lane i: value i
  }
}
template <int NV> __device__ __forceinline__ double cta_sum(ResShared& sh, const FF (&v)[NV]) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const FF t = warp_sum(v[i]);
    if (l == 0) sh.ff[i][w] = make_float2(t.hi, t.lo);
  }
  __syncthreads();
  double out = 0.0;
  if (w == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      FF t;
      if (l < RB / 32) {
        t.hi = sh.ff[i][l].x;
        t.lo = sh.ff[i][l].y;
      }
      t = warp_sum(t);
      if (l == i) out = t.to_double();
    }
  }
  return out;
}

// 1/d to an ulp: the hardware's approximation (some 20 bits) and two Newton steps, each squaring the error; a third of
// a division's latency.  Outside the range where neither the estimate nor the steps under- or overflow: the division.
__device__ __forceinline__ double recip(double d) {
  if (!(fabs(d) > 1e-290 && fabs(d) < 1e290)) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  return fma(r, fma(-d, r, 1.0), r);
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The sums over all CTAs of the CTA sums `mine` (lanes 0..NV-1 of warp 0), valid in every lane of warp 0; what any
// thread wrote to global memory before is visible to every CTA after its next __syncthreads.  Returns false (in warp 0)
// when the barrier gave up.  Contains barriers: every thread calls it.
template <bool GRID, int NV>
__device__ __forceinline__ bool all_sum(ResShared& sh, unsigned* count, double* part, int epoch, double mine,
                                        double (&out)[NV]) {
  const int par = epoch & 1, l = threadIdx.x & 31;
  bool ok = true;
  if constexpr (GRID) {
    __syncthreads();  // the CTA's writes before this point are ordered before lane 0's release
    if (threadIdx.x < 32) {
      double* slot = part + (size_t)par * MAX_GRID * 2;
      if (l < NV) __stcg(slot + 2 * blockIdx.x + l, mine);
      __syncwarp();
      if (l == 0) {  // release: the CTA's writes; acquire: every other CTA's
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        const unsigned want = (unsigned)(epoch + 1) * gridDim.x;
        unsigned seen;
        int n = 0;
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
          if (++n > SPIN_LIMIT) {
            ok = false;
            break;
          }
        } while (seen < want);
      }
      __syncwarp();  // orders the other lanes' loads of the partials after lane 0's acquire (a shuffle does not)
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      // all partials are loaded before the first is added (one L2 latency)
      constexpr int PER = MAX_GRID / 32;
      double2 v[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k)
        v[k] = (l + 32 * k < (int)gridDim.x) ? __ldcg(reinterpret_cast<const double2*>(slot) + l + 32 * k)
                                             : make_double2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        double t[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) t[k] = i ? v[k].y : v[k].x;
#pragma unroll
        for (int o = PER / 2; o > 0; o >>= 1)
#pragma unroll
          for (int k = 0; k < o; ++k)
            if (32 * (k + o) < (int)gridDim.x) t[k] += t[k + o];
        out[i] = warp_sum(t[0]);
      }
    }
  } else {
    uint32_t me;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(me));
    if (threadIdx.x < 32) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const double v = __shfl_sync(0xffffffffu, mine, i);
        if (l < MAX_CLUSTER) {
          uint32_t to;
          const uint32_t at = (uint32_t)__cvta_generic_to_shared(&sh.slot[par][me][i]);
          asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(l));
          asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(v) : "memory");
        }
      }
    }
    cluster_sync_all();
    if (threadIdx.x < 32) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        double t = sh.slot[par][l & (MAX_CLUSTER - 1)][i];
#pragma unroll
        for (int o = MAX_CLUSTER / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        out[i] = t;
      }
    }
  }
  return ok;
}

// ------------------------------------------------------------------ host side
// Cooperative launches of this process on one device follow one another: two grids that each hold a part of the
// SMs would wait for the rest of them.
struct GridTurn {
  std::mutex mu;
  cudaEvent_t last = nullptr;
};
inline GridTurn& grid_turn(int device) {
  static GridTurn t[64];
  return t[device & 63];
}

// One launch of a resident kernel: a cooperative grid, or one cluster, of `ctas` CTAs.
template <bool GRID, class K, class A>
void res_launch(K* kern, int ctas, size_t smem, A args, int device, cudaStream_t st) {
  if constexpr (GRID) {
    GridTurn& turn = grid_turn(device);
    std::lock_guard<std::mutex> lk(turn.mu);
    if (!turn.last) HDG_CUDA(cudaEventCreateWithFlags(&turn.last, cudaEventDisableTiming));
    HDG_CUDA(cudaStreamWaitEvent(st, turn.last, 0));
    void* p[] = {&args};
    HDG_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)ctas), dim3(RB), p, smem, st));
    HDG_CUDA(cudaEventRecord(turn.last, st));
  } else {
    cudaLaunchConfig_t cf = {};
    cf.gridDim = dim3((unsigned)ctas);
    cf.blockDim = dim3(RB);
    cf.dynamicSmemBytes = smem;
    cf.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cf.attrs = &at;
    cf.numAttrs = 1;
    HDG_CUDA(cudaLaunchKernelEx(&cf, kern, args));
  }
}

// Clusters of `ctas` CTAs that can be resident (0: the form is not available).
template <class K> int res_max_clusters(K* kern, int ctas, size_t smem) {
  cudaLaunchConfig_t cf = {};
  cf.gridDim = dim3((unsigned)ctas);
  cf.blockDim = dim3(RB);
  cf.dynamicSmemBytes = smem;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cf.attrs = &at;
  cf.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cf) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// CTAs of the grid form, one per SM (0: not available).
inline int res_grid_ctas(int device) {
  int sms = 0, coop = 0;
  HDG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  HDG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
  return (coop && sms <= MAX_GRID) ? sms : 0;
}

inline int res_forced_kind() {  // HDG_CG_RESIDENT=none|cluster|grid (where it fits)
  const char* e = std::getenv("HDG_CG_RESIDENT");
  if (!e) return -1;
  if (std::strcmp(e, "none") == 0) return (int)CgResident::NONE;
  if (std::strcmp(e, "cluster") == 0) return (int)CgResident::CLUSTER;
  if (std::strcmp(e, "grid") == 0) return (int)CgResident::GRID;
  return -1;
}
