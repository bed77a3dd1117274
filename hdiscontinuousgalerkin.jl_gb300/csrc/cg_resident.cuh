// The Jacobi CG iteration of one problem with its state resident on the chip (cg_resident.cu), and
// what it shares with the launch-per-kernel iteration of cg.cu.
#pragma once
#include "hdg_device.cuh"

constexpr int HDG_CG_SC = 10;  // per problem: rz, rz_old, pq, rr, bb, tol2, alpha, beta, rr_true, flip
constexpr int CG_LOST = 6;     // status: a barrier of the resident iteration gave up

template <typename T> struct CgArgs {
  SegArgs g;
  const int32_t* bcol5;
  int nf;
  const T* val;
  const double* b;
  const T* dinv;
  double* x;
  T* r;
  T* z;
  T* p;
  T* q;
  T* p2;
  double* sc;
  int32_t* st;
  float* xh;  // FP32 iteration: steps since the last refinement as a float-float pair (hi, lo)
  float* xl;
};

// How a system's Jacobi iteration runs: as two kernels per iteration (none), by one cluster of CTAs,
// or by a cooperative grid of one CTA per SM.
struct CgResident {
  enum Kind { NONE, CLUSTER, GRID } kind = NONE;
  int ctas = 0, faces_per_cta = 0;
  bool mat_smem = false;  // the CTA's matrix rows are kept in shared memory
  size_t smem = 0;
  bool forced = false;  // by HDG_CG_RESIDENT
};
// The plan of a system with one problem (NONE where its state does not fit, or only a grid's would and that is not
// allowed), and one launch of at most `iters` iterations of it.  `sync`: CG_SYNC_BYTES of device memory for the barriers; `pairs`: 2 x
// rows (z, p) pairs of the FP32 iteration.
constexpr size_t CG_SYNC_BYTES = 16384;
template <typename T> CgResident cg_resident_plan(int nt, int nf, int device, bool grid_allowed);
template <typename T>
void cg_resident_launch(const CgResident& pl, int nt, const CgArgs<T>& a, float2* pairs, void* sync, int iters,
                        int device, cudaStream_t st);
